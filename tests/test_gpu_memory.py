"""Results through the staged device-to-host copy and the context's memory pool.

Receiver fields come back through two pinned buffers of 2 MB whose contents
host threads copy in parts of 64 KB: the sizes here put the result on either
side of a part, of a buffer and of both buffers (96 bytes per receiver), and
each must equal, to the bit, the same receivers asked for 500 at a time.
The pool hands freed blocks to later calls: a context that builds its
preconditioner again, on another mesh and back, must solve to the same
result.
"""

import numpy as np
import pytest

import emfem_b200 as E
from emfem_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 682, 683, 21845, 21846, 43691, 70000])
def test_fields_of_any_size(csem_small, n):
    import torch
    m = csem_small.mesh
    rng = np.random.default_rng(n)
    with E.EMContext(0) as c:
        c.set_mesh(m)
        c.set_model(csem_small.model)
        c.set_frequencies([1.0])
        c.create_linear_system(0)
        x = torch.from_numpy(rng.standard_normal((m.n_edges, 2))).cuda()
        cells = rng.integers(0, m.n_tets, size=n).astype(np.int32)
        pts = m.points[m.tets[cells]].mean(axis=1)
        torch.cuda.synchronize()
        e, h = c.interpolate_fields_block_dev([1.0], x.data_ptr(), pts, cells)
        for i in range(0, n, 500):
            ei, hi = c.interpolate_fields_block_dev([1.0], x.data_ptr(), pts[i:i + 500], cells[i:i + 500])
            assert np.array_equal(e[i:i + 500], ei) and np.array_equal(h[i:i + 500], hi)


def test_blocks_reused_across_meshes(csem_small):
    import torch
    big = mg.marine_csem(9000, freqs=(1.0,), name="bigger")
    sols = []
    with E.EMContext(0) as c:
        for prob in (csem_small, big, csem_small):
            c.set_mesh(prob.mesh)
            c.set_model(prob.model)
            c.set_frequencies([1.0])
            c.create_linear_system(0)
            for _ in range(2):
                c.assemble_matrix(0)
                s = torch.zeros((prob.mesh.n_edges, 2), dtype=torch.complex128, device="cuda")
                x = torch.zeros_like(s)
                c.assemble_rhs_csem_block_dev([1.0, 1.0], np.repeat(prob.survey.tx[:1], 2, axis=0), s.data_ptr())
                infos = c.solve_block_dev([1.0, 1.0], s.data_ptr(), x.data_ptr(), rtol=1e-8, max_it=200)
                assert all(i.reason == 0 for i in infos)
            sols.append(x.cpu().numpy())
    # two solves to a relative residual of 1e-8: the solve tests' 1e-6
    assert np.abs(sols[2] - sols[0]).max() <= 1e-6 * np.abs(sols[0]).max()


def _fields_context(prob, c, k=2):
    import torch
    c.set_mesh(prob.mesh)
    c.set_model(prob.model)
    c.set_frequencies([1.0])
    c.create_linear_system(0)
    return torch.from_numpy(np.random.default_rng(5).standard_normal((prob.mesh.n_edges, 2 * k))).cuda()


def test_a_result_does_not_wait_for_another_context(csem_small):
    """A context whose kernels are still queued asks for its fields; the fields
    of another context, asked for at that time by another thread, come back
    long before.  (The queue is operator applications of a quarter of a million
    cells, as many as the driver queues: about 1000, 0.1 s.)"""
    import threading
    import time
    import torch
    big = mg.marine_csem(250000, freqs=(1.0,), name="busy")
    m = csem_small.mesh
    n = 2000
    rng = np.random.default_rng(11)
    with E.EMContext(0) as a, E.EMContext(0) as b:
        xa, xb = _fields_context(big, a), _fields_context(csem_small, b)
        a.assemble_matrix(0)
        v = torch.zeros((big.mesh.n_edges, 16), dtype=torch.complex128, device="cuda")
        w = torch.zeros_like(v)
        ca, cb = (rng.integers(0, p.n_tets, size=n).astype(np.int32) for p in (big.mesh, m))
        pa, pb = big.mesh.points[big.mesh.tets[ca]].mean(axis=1), m.points[m.tets[cb]].mean(axis=1)
        torch.cuda.synchronize()
        read_b = lambda: b.interpolate_fields_block_dev([1.0] * 2, xb.data_ptr(), pb, cb)  # noqa: E731
        want = read_b()
        a.interpolate_fields_block_dev([1.0] * 2, xa.data_ptr(), pa, ca)
        done = {}

        def busy():
            for _ in range(2000):
                a.spmv_complex_dev(np.ones(16), v.data_ptr(), w.data_ptr())
            done["queued"] = time.perf_counter()
            a.interpolate_fields_block_dev([1.0] * 2, xa.data_ptr(), pa, ca)
            done["a"] = time.perf_counter()

        th = threading.Thread(target=busy)
        th.start()
        while "queued" not in done:
            time.sleep(1e-3)
        time.sleep(2e-3)
        t0 = time.perf_counter()
        got = read_b()
        t1 = time.perf_counter()
        th.join()
    assert done["a"] - done["queued"] > 0.05  # the other context was busy all the while
    assert t1 - t0 < 0.5 * (done["a"] - t0)
    assert all(np.array_equal(x, y) for x, y in zip(got, want))


@pytest.mark.parametrize("n", [85, 86, 5461, 5462, 10922, 10923])
def test_fields_around_the_staging_limits(csem_small, n):
    """192 bytes per receiver: 16 KB (no staging below), one buffer of 1 MB, both."""
    m = csem_small.mesh
    rng = np.random.default_rng(n)
    with E.EMContext(0) as c:
        x = _fields_context(csem_small, c)
        cells = rng.integers(0, m.n_tets, size=n).astype(np.int32)
        pts = m.points[m.tets[cells]].mean(axis=1)
        first = c.interpolate_fields_block_dev([1.0, 1.0], x.data_ptr(), pts, cells)
        again = c.interpolate_fields_block_dev([1.0, 1.0], x.data_ptr(), pts, cells)
        for i in range(0, n, 60):
            part = c.interpolate_fields_block_dev([1.0, 1.0], x.data_ptr(), pts[i:i + 60], cells[i:i + 60])
            for full in (first, again):
                assert all(np.array_equal(f[i:i + 60], p) for f, p in zip(full, part))
