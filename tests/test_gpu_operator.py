"""y = (C + i w_c Ms) x on complex columns (emg_spmv_complex_dev) against float64.

Each block width has its own lane layout: one column per lane and 4, 2 or 1
lanes per row up to 8 columns, two columns per lane from 16 on, 4 nonzeros
per lane and round.  The meshes give rows of 6 to 601 nonzeros (every remainder of
a round, rows of many rounds) and row counts that end in the middle of a warp
and of a block; every column has its own frequency, which travels with the
launch.  Bar: 1e-13 of |C| |x| + w |Ms| |x| per component, as the FP64 layouts
of test_gpu_spmm_layouts.py (rows of hundreds of nonzeros are summed in order,
601 x 2^-53 = 7e-14).
"""

import numpy as np
import pytest
import scipy.sparse as sp

import emfem_b200 as E
from emfem_b200 import meshgen as mg
from test_gpu_assembly import _fan

pytestmark = pytest.mark.gpu


def _mesh(name):
    if name == "tet":
        pts = np.array([[0.0, 0, 0], [90, 0, 0], [0, 110, 0], [0, 0, 70]])
        return mg.build_topology(pts, mg.orient_positive(pts, np.array([[0, 1, 2, 3]])), np.zeros(1, dtype=np.int32))
    n = int(name[4:])
    return _fan(n, {3: 2, 40: 3, 200: 6}[n], True)


@pytest.fixture(scope="module", params=["tet", "fan-3", "fan-40", "fan-200"])
def operator(request):
    m = _mesh(request.param)
    c = E.EMContext(0)
    c.set_mesh(m)
    c.set_model(mg.Model(mg.VERTICAL, np.array([[10.0, 30.0], [1.0, 2.0], [100.0, 50.0]])))
    c.set_frequencies([1.0 / (2 * np.pi)])  # w = 1: M = Ms
    c.create_linear_system(0)
    c.assemble_matrix(0)
    rp, ci = c.make_sparsity_patterns()
    Cv, Mv, _ = c.get_matrices()
    n = rp.size - 1
    yield c, sp.csr_matrix((Cv, ci, rp), shape=(n, n)), sp.csr_matrix((Mv, ci, rp), shape=(n, n))
    c.close()


@pytest.mark.parametrize("conj", [False, True])
@pytest.mark.parametrize("k", [1, 2, 4, 8, 16, 32])
def test_widths(operator, k, conj):
    import torch
    c, Cm, Mm = operator
    n = Cm.shape[0]
    rng = np.random.default_rng(10 * k + conj)
    w = np.abs(Cm).max() / max(np.abs(Mm).max(), 1e-300) * np.logspace(-1, 1, k)  # both parts count
    xh = rng.standard_normal((n, k)) + 1j * rng.standard_normal((n, k))
    x = torch.from_numpy(xh).cuda()
    pad = 64  # around y: nothing else is written
    buf = torch.full((2 * pad + n * k,), complex("nan+nanj"), dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    c.spmv_complex_dev(w, x.data_ptr(), buf.data_ptr() + 16 * pad, conj_out=conj)
    c.synchronize()
    out = buf.cpu().numpy()
    assert np.isnan(out[:pad]).all() and np.isnan(out[pad + n * k:]).all()
    y = out[pad:pad + n * k].reshape(n, k)
    ref = Cm @ xh + 1j * w * (Mm @ xh)
    if conj:
        ref = ref.conj()
    ax = np.abs(xh.real) + np.abs(xh.imag)
    scale = abs(Cm) @ ax + w * (abs(Mm) @ ax)
    d = y - ref
    assert (np.maximum(np.abs(d.real), np.abs(d.imag)) <= 1e-13 * scale).all()


@pytest.mark.parametrize("k", [0, 3, 12, 33, 64])
def test_refused_widths(operator, k):
    import torch
    c, Cm, _ = operator
    x = torch.zeros((Cm.shape[0], max(k, 1)), dtype=torch.complex128, device="cuda")
    with pytest.raises(E.EMGError):
        c.spmv_complex_dev(np.ones(k), x.data_ptr(), x.data_ptr())
