"""Row-wise assembly on fans of tets around an axis, against the oracle.

The axis edges of a fan collect a term from every tet around them: 3 and 40
tets per axis edge stay inside the record's 9-bit positions and the block's
tile of row slots, 200 tets on 5 consecutive axis edges (601 slots per row)
exceed both, so that columns are searched for and rows summed in place.
Bars of the other assembly tests: pattern and boundary cells equal, values to
1e-12 of the largest.
"""

import dataclasses

import numpy as np
import pytest

import emfem_b200 as E
from emfem_b200 import meshgen as mg
import oracle as O

pytestmark = pytest.mark.gpu


def _fan(n_ring, n_axis, shuffle):
    a = np.linspace(0, 2 * np.pi, n_ring, endpoint=False)
    ring = np.stack([1.3 * np.cos(a), np.sin(a), 0.45 + 0.02 * np.sin(3 * a)], axis=1)
    axis = np.stack([np.zeros(n_axis), np.zeros(n_axis), np.linspace(0, 1, n_axis)], axis=1)
    pts = np.concatenate([ring, axis]) * 100.0
    tets = [[n_ring + k, n_ring + k + 1, i, (i + 1) % n_ring] for k in range(n_axis - 1) for i in range(n_ring)]
    tets = np.array(tets, dtype=np.int64)
    if shuffle:  # vertex ids in another order: every orientation of the record's signs
        perm = np.random.default_rng(n_ring).permutation(pts.shape[0])
        inv = np.empty_like(perm)
        inv[perm] = np.arange(perm.size)
        pts, tets = pts[perm], inv[tets]
    tets = mg.orient_positive(pts, tets)
    attr = (np.arange(tets.shape[0]) % 3).astype(np.int32)
    return mg.build_topology(pts, tets, attr)


@pytest.mark.parametrize("n_ring,n_axis", [(3, 2), (40, 3), (200, 6)])
@pytest.mark.parametrize("shuffle", [False, True])
def test_fan_matches_oracle(n_ring, n_axis, shuffle):
    m = _fan(n_ring, n_axis, shuffle)
    model = mg.Model(mg.ARBITRARY, np.array([[10.0, 30.0, 5.0, 20.0, -35.0, 50.0], [1.0, 2.0, 4.0, 10.0, 0.0, 5.0],
                                             [100.0, 100.0, 100.0, 0.0, 0.0, 0.0]]))
    om = O.Mesh(m)
    orp, oci = O.sparsity(om)
    Co, Mo, bo = O.assemble(om, model, 2.0, orp, oci)
    with E.EMContext(0) as c:
        c.set_mesh(m)
        c.set_model(model)
        c.set_frequencies([2.0])
        c.create_linear_system(0)
        c.assemble_matrix(0)
        rp, ci = c.make_sparsity_patterns()
        C, M, bdr = c.get_matrices()
        c.assemble_matrix(0)
        C2, M2, _ = c.get_matrices()
    assert np.array_equal(rp, orp) and np.array_equal(ci, oci) and np.array_equal(bdr, bo)
    assert np.abs(C - Co).max() <= 1e-12 * np.abs(Co).max()
    assert np.abs(M - Mo).max() <= 1e-12 * max(np.abs(Mo).max(), 1e-300)
    assert np.array_equal(C, C2) and np.array_equal(M, M2)  # a fixed summation order


def _not_mirrored(rp, ci, v):
    """Entries that differ in any bit from the transposed ones."""
    n = rp.size - 1
    row = np.repeat(np.arange(n, dtype=np.int64), np.diff(rp))
    back = np.lexsort((row, ci))  # entry (j, i) in the place of (i, j): the pattern is symmetric
    assert np.array_equal(row[back], ci) and np.array_equal(ci[back], row)
    return int((v != v[back]).sum())


@pytest.mark.parametrize("mesh", ["fan-3", "fan-40", "fan-200", "csem_small", "mt_aniso"])
def test_entries_equal_their_mirror(mesh, request):
    """C and Ms are symmetric to the bit: both rows of an off-diagonal entry
    evaluate its one or two terms with the same operands in the same order
    (the preconditioned iterations assume a symmetric operator, and in the air
    rounding of C is not small against w Ms)."""
    if mesh.startswith("fan"):
        n = int(mesh[4:])
        m = _fan(n, {3: 2, 40: 3, 200: 6}[n], True)
        model = mg.Model(mg.ARBITRARY, np.array([[10.0, 30.0, 5.0, 20.0, -35.0, 50.0], [1.0, 2.0, 4.0, 10.0, 0.0, 5.0],
                                                 [1e8, 1e8, 1e8, 0.0, 0.0, 0.0]]))
    else:
        prob = request.getfixturevalue(mesh)
        m, model = prob.mesh, prob.model
    with E.EMContext(0) as c:
        c.set_mesh(m)
        c.set_model(model)
        c.set_frequencies([2.0])
        c.create_linear_system(0)
        c.assemble_matrix(0)
        rp, ci = c.make_sparsity_patterns()
        C, M, _ = c.get_matrices()
    assert _not_mirrored(rp, ci, C) == 0 and _not_mirrored(rp, ci, M) == 0


@pytest.mark.parametrize("mesh", ["fan-40", "fan-200", "csem_small"])
def test_diagonal_is_summed_in_a_fixed_order(mesh, request):
    """A diagonal entry is the sum of its tets' entries in the order (t mod 32,
    t), to the bit: the order of the tet-wise scatter (a warp per 32 tets), which
    solutions in the air depend on.  The tets' own entries come from a mesh
    of the same tets with no vertex in common."""
    if mesh.startswith("fan"):
        n = int(mesh[4:])
        m = _fan(n, {40: 3, 200: 6}[n], True)
        model = mg.Model(mg.ISOTROPIC, np.array([[10.0], [3.0], [1e8]]))
    else:
        prob = request.getfixturevalue(mesh)
        m, model = prob.mesh, prob.model
    nt = m.n_tets
    # vertex 4 t + rank keeps the order of a tet's ids, so its entries are the same numbers
    rank = np.argsort(np.argsort(m.tets, axis=1), axis=1)
    pts = np.empty((4 * nt, 3))
    alone = (4 * np.arange(nt)[:, None] + rank).astype(np.int64)
    pts[alone] = m.points[m.tets]
    apart = mg.build_topology(pts, alone, m.attr)
    diag = []
    for x in (m, apart):
        x = dataclasses.replace(x, edge_bdr=np.zeros_like(x.edge_bdr))  # no Dirichlet rows: whole entries
        with E.EMContext(0) as c:
            c.set_mesh(x)
            c.set_model(model)
            c.set_frequencies([2.0])
            c.create_linear_system(0)
            c.assemble_matrix(0)
            rp, ci = c.make_sparsity_patterns()
            C, _, _ = c.get_matrices()
        diag.append(C[ci == np.repeat(np.arange(rp.size - 1), np.diff(rp))])
    want = np.zeros(m.n_edges)
    for t in np.lexsort((np.arange(nt), np.arange(nt) % 32)):
        want[m.tet2edge[t]] += diag[1][apart.tet2edge[t]]
    assert np.array_equal(diag[0], want)
