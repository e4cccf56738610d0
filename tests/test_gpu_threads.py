"""Contexts in two threads at once, with what the process shares between them:
the layout table of the SpMM tuner (also read while it is written), the store
of freed device memory and the staging buffers.  Each must solve to what it
solves to alone; two solves to a relative residual of 1e-8 agree to the
solve tests' 1e-6."""

import threading

import numpy as np
import pytest

import emfem_b200 as E
from emfem_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def _run(prob, widths, stream):
    import torch
    out = []
    with torch.cuda.stream(stream), E.EMContext(0) as c:
        c.set_mesh(prob.mesh)
        c.set_model(prob.model)
        c.set_frequencies([1.0])
        c.create_linear_system(0)
        c.assemble_matrix(0)
        cells = np.arange(0, prob.mesh.n_tets, 7, dtype=np.int32)
        pts = prob.mesh.points[prob.mesh.tets[cells]].mean(axis=1)
        for k in widths:
            f = np.linspace(0.5, 1.5, k)
            s = torch.zeros((prob.mesh.n_edges, k), dtype=torch.complex128, device="cuda")
            x = torch.zeros_like(s)
            stream.synchronize()
            c.assemble_rhs_csem_block_dev(f, np.repeat(prob.survey.tx[:1], k, axis=0), s.data_ptr())
            infos = c.solve_block_dev(f, s.data_ptr(), x.data_ptr(), rtol=1e-8, max_it=200)
            assert all(i.reason == 0 for i in infos)
            out.append(c.interpolate_fields_block_dev(f, x.data_ptr(), pts, cells)[0])
    return out


def test_two_contexts_at_once():
    import torch
    probs = [mg.marine_csem(n, freqs=(1.0,), name="threads") for n in (9000, 14000)]
    widths = (1, 4, 2, 8)
    streams = [torch.cuda.Stream() for _ in probs]
    got, bad, stop = [None, None], [], threading.Event()

    def work(i):
        try:
            got[i] = _run(probs[i], widths, streams[i])
        except Exception as e:  # noqa: BLE001
            bad.append(e)

    def poll():
        while not stop.is_set():
            E.spmm_layouts()

    th = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    reader = threading.Thread(target=poll)
    for t in th + [reader]:
        t.start()
    for t in th:
        t.join()
    stop.set()
    reader.join()
    assert not bad, bad
    for i, p in enumerate(probs):
        for a, b in zip(got[i], _run(p, widths, streams[i])):
            assert np.abs(a - b).max() <= 1e-6 * np.abs(b).max()
