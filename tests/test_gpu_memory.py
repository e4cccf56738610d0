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
