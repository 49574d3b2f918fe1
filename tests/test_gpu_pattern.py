"""The warp-per-row sparsity pass at its edges, on fans of 2n P2 tetrahedra
around one node: its row holds 5n + 5 columns of 20n candidates.  n = 5 .. 25
cross the register sorts (32, 64, 128 columns, then shared memory and the fill
pass), n = 13 the candidates the first launch has room for.  The thread-per-row pass at its
column limit, on P1 tetrahedra that share little more than one node."""
import numpy as np
import pytest

import gtgpu as GT
import oracle as O
from test_gpu_parity import TOL64, _fan_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 6, 11, 12, 13, 24, 25, 60])
def test_fan_rows(n):
    m = _fan_mesh(n)
    V = GT.lagrange_space(GT.interior(m), 2)
    A = GT.assemble_matrix(GT.laplacian(), np.float64, V)
    rp, ci, v = A.csr()
    assert np.diff(rp).max() == 5 * n + 5
    om = dict(D=3, ctype=m.cell_type, coords=m.coords, cell_nodes=m.cell_nodes, pf0=m.corners, pf1=m.bedges,
              pf1g=None, pf2=m.bfaces, pf2g=m.bface_group, cells=(), box=())
    ref = O.lagrange_space(om, 2)
    cp, rv, nz = O.assemble_matrix(ref, O.LAPLACE, 4)
    orp, oci, ov = O.csc_to_csr(cp, rv, nz, ref["nfree"])
    assert np.array_equal(rp, orp) and np.array_equal(ci, oci)
    assert np.abs(v - ov).max() <= TOL64 * np.abs(ov).max()


@pytest.mark.parametrize("disjoint,extra", [(1, 0), (5, 0), (9, 0), (10, 0), (10, 1), (10, 2), (11, 0)])
def test_bouquet_rows(disjoint, extra):
    """Tetrahedra around node 1: 3 new nodes each, 1 for each extra one (it
    shares a face's edge with the first) -- 3 * disjoint + extra + 1 columns of
    the 32 the row-per-thread pass holds; 33 and 34 are recounted."""
    from gtgpu.mesh import Mesh
    rng = np.random.default_rng(disjoint * 10 + extra)
    n = 1 + 3 * disjoint + extra
    coords = np.vstack([[0.0, 0.0, 0.0], rng.uniform(-1.0, 1.0, (n - 1, 3))])
    cells = [[1, 2 + 3 * i, 3 + 3 * i, 4 + 3 * i] for i in range(disjoint)]
    cells += [[1, 2, 3, 2 + 3 * disjoint + j] for j in range(extra)]
    m = Mesh(D=3, cell_type=GT.api._lib.GT_TET4, coords=coords, cell_nodes=np.asarray(cells, np.int32),
             corners=np.zeros(0, np.int32), bfaces=np.zeros((0, 3), np.int32), bface_group=np.zeros(0, np.int32),
             bedges=np.zeros((0, 2), np.int32))
    V = GT.lagrange_space(GT.interior(m), 1)
    rp, ci, v = GT.assemble_matrix(GT.mass(), np.float64, V).csr()
    dofs = V.face_dofs()
    pairs = sorted({(a, b) for c in dofs for a in c for b in c})
    assert np.array_equal(ci + 1, [b for _, b in pairs])
    assert np.array_equal(np.diff(rp), np.bincount([a - 1 for a, _ in pairs], minlength=n))
    assert np.diff(rp).max() == n
    # the entries of the mass matrix add up to the volume (positive terms)
    J = coords[np.asarray(cells) - 1][:, 1:] - coords[np.asarray(cells) - 1][:, :1]
    vol = np.abs(np.linalg.det(J)).sum() / 6.0
    assert abs(v.sum() - vol) <= 1e-12 * vol


def _with_split_cells(n, nodes):
    """A grid of P2 tetrahedra whose cells around the first `nodes` interior
    nodes are split at their centroids: 48 cells at such a node."""
    m = GT.cartesian_mesh((0.0, 1.0, 0.0, 1.0, 0.0, 1.0), (n, n, n), simplexify=True)
    cn = m.cell_nodes
    inner = np.nonzero(((m.coords > 0.0) & (m.coords < 1.0)).all(axis=1))[0] + 1
    split = np.isin(cn, inner[:nodes]).any(axis=1)
    new = m.num_nodes + 1 + np.arange(split.sum())
    cells = [cn[~split]]
    for j in range(4):
        t = cn[split].copy()
        t[:, j] = new
        cells.append(t)
    m.coords = np.ascontiguousarray(np.vstack([m.coords, m.coords[cn[split] - 1].mean(axis=1)]))
    m.cell_nodes = np.ascontiguousarray(np.vstack(cells).astype(np.int32))
    return m


@pytest.mark.parametrize("n,nodes", [(3, 1), (4, 3), (5, 64)])
def test_few_rows_beyond_the_first_launch(n, nodes):
    """A few rows with more candidates than the first launch has room for: they
    alone are counted again (one launch and a scan more)."""
    m = _with_split_cells(n, nodes)
    V = GT.lagrange_space(GT.interior(m), 2)
    A = GT.assemble_matrix(GT.laplacian(), np.float64, V)
    rp, ci, v = A.csr()
    om = dict(D=3, ctype=m.cell_type, coords=m.coords, cell_nodes=m.cell_nodes, pf0=m.corners, pf1=m.bedges,
              pf1g=None, pf2=m.bfaces, pf2g=m.bface_group, cells=(), box=())
    ref = O.lagrange_space(om, 2)
    cp, rv, nz = O.assemble_matrix(ref, O.LAPLACE, 4)
    orp, oci, ov = O.csc_to_csr(cp, rv, nz, ref["nfree"])
    assert np.array_equal(rp, orp) and np.array_equal(ci, oci)
    assert np.abs(v - ov).max() <= TOL64 * np.abs(ov).max()
    ctx = V.ctx
    if n == 3:  # a scan of one launch in both
        plain = GT.cartesian_mesh((0.0, 1.0, 0.0, 1.0, 0.0, 1.0), (n, n, n), simplexify=True)
        count = []
        for mesh in (plain, m):
            W = GT.lagrange_space(GT.interior(mesh), 2)
            GT.assemble_matrix(GT.laplacian(), np.float64, W)
            l0 = ctx.launches()
            GT.assemble_matrix(GT.laplacian(), np.float64, W)
            count.append(ctx.launches() - l0)
        assert count[1] == count[0] + 2
