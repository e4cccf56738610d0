"""The AMS chain at every block width, against a sparse direct solve.

The transfers, first smoothing steps, coarsest solve and SpMMs of the AMS run
as overlapping kernels (programmatic dependent launch) whose lane layout
follows the block width: 1, 2 or 4 columns per load, 1 to 4 lanes per row or
vertex, padded blocks.  Each width solves CSEM right-hand sides on a mesh of
some 1000 cells; the solutions must agree with the direct solve to 1e-6 of
the largest value per column, the bar of the other solve tests (rtol 1e-8, a
factor 100 for the condition between residual and error at 0.5-4 Hz).
"""

import numpy as np
import pytest

import emfem_b200 as E
from emfem_b200 import meshgen as mg
from exact_solve import exact_solutions

pytestmark = pytest.mark.gpu


def build(cells):
    import torch
    freqs = np.array([0.5, 4.0])
    prob = mg.marine_csem(cells, freqs=freqs, n_tx=3, name="chain")
    c = E.EMContext(0)
    c.set_mesh(prob.mesh)
    c.set_model(prob.model)
    c.set_frequencies(freqs)
    c.create_linear_system(0)
    rp, ci = c.make_sparsity_patterns()
    ne = prob.mesh.n_edges
    tx = np.tile(prob.survey.tx, (2, 1))
    colf = np.repeat(freqs, 3)
    s = torch.zeros((ne, 6), dtype=torch.complex128, device="cuda")
    c.assemble_matrix(0)
    c.assemble_rhs_csem_block_dev(colf, tx, s.data_ptr())
    s = s.cpu().numpy()
    jobs = []
    for f in range(2):
        c.assemble_matrix(f)
        Cv, Mv, _ = c.get_matrices()
        jobs.append((rp, ci, Cv, Mv, np.conj(s[:, 3 * f:3 * f + 3])))
    exact = np.concatenate(exact_solutions(jobs), axis=1)
    return c, colf, s, exact


@pytest.fixture(scope="module")
def system():
    b = build(1200)
    yield b
    b[0].close()


@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("k", [1, 2, 3, 4, 8, 17])
@pytest.mark.parametrize("options", ["-emg_restrict_smooth 1 -emg_smoother chebyshev",
                                     "-emg_restrict_smooth 0 -emg_smoother chebyshev",
                                     "-emg_restrict_smooth 1 -emg_smoother l1jacobi"])
def test_block_widths(system, fp32, k, options):
    c, colf, s, exact = system
    if "l1jacobi" in options and k != 3:
        pytest.skip("one width per smoother")
    cols = np.arange(k) % 6
    # coarsest grids small enough that the hierarchy has several levels
    c.process_options("-emg_amg_max_coarse 40 " + options)
    c.assemble_matrix(0)
    x, infos = c.solve_block(colf[cols], s[:, cols], rtol=1e-8, max_it=200, inner_fp32=fp32)
    assert all(i.reason == 0 for i in infos)
    err = np.abs(x - exact[:, cols]).max(axis=0) / np.abs(exact[:, cols]).max(axis=0)
    assert err.max() <= 1e-6, err


@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("K", [8, 16, 32, 64])
@pytest.mark.parametrize("variant", [801, 802])
def test_dense_residency_layout(system, fp32, K, variant):
    """y = b - (C + w Ms) x with the 6-blocks-per-SM layout against float64: rows
    of 9 to 40 nonzeros leave every remainder of its rounds of 2 (and of 2
    lanes).  Tolerances as in test_gpu_spmm_layouts.py."""
    import scipy.sparse as sp
    import torch
    c = system[0]
    c.assemble_matrix(0)
    rp, ci = c.make_sparsity_patterns()
    Cv, Mv, _ = c.get_matrices()
    n = rp.size - 1
    Cm, Mm = sp.csr_matrix((Cv, ci, rp), shape=(n, n)), sp.csr_matrix((Mv / (2 * np.pi * 0.5), ci, rp), shape=(n, n))
    rng = np.random.default_rng(K)
    w = 2 * np.pi * np.logspace(-1, 1, K)
    if K == 16:
        w = np.repeat(w[::2], 2)  # complex columns: pairs share their frequency
    dt = torch.float32 if fp32 else torch.float64
    x = torch.from_numpy(rng.standard_normal((n, K))).to(dt).cuda()
    b = torch.from_numpy(rng.standard_normal((n, K))).to(dt).cuda()
    y = torch.full_like(x, float("nan"))
    torch.cuda.synchronize()
    v = 4 if fp32 else 2
    ok = c.spmm_layout_dev(fp32, w, x.data_ptr(), b.data_ptr(), y.data_ptr(), v, variant)
    assert ok == (K // v * (variant - 800) <= 32)
    if not ok:
        return
    c.synchronize()
    xh, bh, yh = x.double().cpu().numpy(), b.double().cpu().numpy(), y.double().cpu().numpy()
    ref = bh - Cm @ xh - (Mm @ xh) * w
    scale = np.abs(bh) + abs(Cm) @ np.abs(xh) + (abs(Mm) @ np.abs(xh)) * w
    assert (np.abs(yh - ref) / scale).max() <= (1e-5 if fp32 else 1e-13)


@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("mmax", [1, 3, 4, 5, 9])
def test_fcg_truncations(system, fp32, mmax):
    """The passes over the FCG directions go in groups of up to four: every
    group size, a second and a third group."""
    if fp32 and mmax > 4:
        pytest.skip("refused with the FP32 preconditioner")
    c, colf, s, exact = system
    c.process_options("-emg_amg_max_coarse 40 -emg_restrict_smooth 1 -emg_smoother chebyshev "
                      f"-emg_block_fcg_mmax {mmax}")
    c.assemble_matrix(0)
    x, infos = c.solve_block(colf[:4], s[:, :4], rtol=1e-8, max_it=200, inner_fp32=fp32)
    c.process_options("-emg_block_fcg_mmax 2")
    assert all(i.reason == 0 for i in infos)
    err = np.abs(x - exact[:, :4]).max(axis=0) / np.abs(exact[:, :4]).max(axis=0)
    assert err.max() <= 1e-6, err


@pytest.mark.parametrize("mmax", [2, 3])
def test_fcg_long_vectors(mmax):
    """Block vectors longer than four grids of the passes, with a remainder:
    several pairs of a thread in flight."""
    c, colf, s, exact = build(16000)
    try:
        assert s.shape[0] * 32 > 4 * 4 * 148 * 256
        cols = np.arange(32) % 6
        c.process_options(f"-emg_block_fcg_mmax {mmax}")
        x, infos = c.solve_block(colf[cols], s[:, cols], rtol=1e-8, max_it=200, inner_fp32=True)
        assert all(i.reason == 0 for i in infos)
        err = np.abs(x - exact[:, cols]).max(axis=0) / np.abs(exact[:, cols]).max(axis=0)
        assert err.max() <= 1e-6, err
    finally:
        c.close()


@pytest.mark.parametrize("power", [-520, -515, -500, 0, 480])
def test_pc_apply_scales(system, power):
    """The preconditioner is linear: b scaled by a power of two gives x scaled
    by it, also where the squares of its FCG are near the ends of the range (norms of b
    from 1e-151 to 1e150; below, the squares of a solve to 1e-2 are subnormal
    and lose its digits).  The order of the sums differs from run to run, by
    1e-10 of x: the solve tests' 1e-6."""
    c, colf, s, _ = system
    c.process_options("-emg_amg_max_coarse 40")
    c.assemble_matrix(0)
    c.create_pc()
    b = np.concatenate([s[:, 0].real, s[:, 0].imag])
    b *= 2.0 ** -int(np.floor(np.log2(np.linalg.norm(b)))) * 2.0 ** 18
    x0 = c.pc_apply_b(b)
    x = c.pc_apply_b(b * 2.0 ** power)
    x = x * 2.0 ** -(power // 2) * 2.0 ** -(power - power // 2)
    assert np.linalg.norm(x - x0) <= 1e-6 * np.linalg.norm(x0)


@pytest.mark.parametrize("fp32", [True, False])
@pytest.mark.parametrize("mmax", [1, 2, 3, 4, 5, 9])
def test_fcg_groups_are_reached(system, fp32, mmax):
    """test_fcg_truncations with inner solves long enough that the ring of directions
    fills and wraps: more than mmax + 1 inner iterations per outer one."""
    if fp32 and mmax > 4:
        pytest.skip("refused with the FP32 preconditioner")
    c, colf, s, exact = system
    c.process_options(f"-emg_amg_max_coarse 40 -emg_block_fcg_mmax {mmax} -emg_block_inner_rtol 1e-6 "
                      "-emg_block_inner_max_it 60")
    try:
        c.assemble_matrix(0)
        x, infos = c.solve_block(colf[:4], s[:, :4], rtol=1e-8, max_it=200, inner_fp32=fp32)
    finally:
        c.process_options("-emg_block_fcg_mmax 2 -emg_block_inner_rtol 1e-2 -emg_block_inner_max_it 30")
    assert all(i.reason == 0 for i in infos)
    assert min(i.inner_its / i.outer_its for i in infos) > mmax + 1, [(i.inner_its, i.outer_its) for i in infos]
    err = np.abs(x - exact[:, :4]).max(axis=0) / np.abs(exact[:, :4]).max(axis=0)
    assert err.max() <= 1e-6, err
