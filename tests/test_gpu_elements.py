"""The element kernels without a quadrature loop over node pairs
(csrc/gt_elements.cuh) against the oracle's quadrature, at cell counts around
the cells per block (16 Q1 and 4 Q2 hexahedra, 32 and 128 P2 tetrahedra).

An entry is a sum over at most 27 points (or an exact integral) of products of
about ten factors: its rounding error stays below 100 eps of the sum of the
terms' magnitudes, which is at most a few times the largest entry.  FP64: 100
eps x 8 < 2e-13 of the largest entry; FP32 (FP64 geometry): 100 eps32 x 8 <
1e-4, and 5e-6 for the 27 FP32 products of one entry added in sequence.
"""
import numpy as np
import pytest

import gtgpu as GT
import oracle as O
from test_gpu_parity import _oracle_space

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,simplex,order", [
    ((1, 1, 1), False, 1), ((2, 2, 3), False, 1), ((2, 2, 4), False, 1), ((2, 3, 3), False, 1),
    ((1, 1, 1), False, 2), ((2, 2, 2), False, 2), ((3, 3, 3), False, 2), ((5, 3, 2), False, 2),
    ((1, 1, 1), True, 2), ((2, 4, 2), True, 2), ((11, 2, 2), True, 2), ((4, 4, 4), True, 2),
])
def test_laplacian_blocks(cells, simplex, order):
    m = GT.cartesian_mesh((0.0, 1.0, -0.5, 2.0, 0.0, 0.7), cells, simplexify=simplex)
    # every node moved, also those on the boundary (single layers of cells)
    m.coords += np.random.default_rng(3).uniform(-0.1, 0.1, m.coords.shape) / max(cells)
    coef = GT.lognormal_cells(m.num_cells, 1.0, 17)
    ref, _ = _oracle_space(m, order, 1, None)
    cp, rv, nz = O.assemble_matrix(ref, O.LAPLACE, 2 * order, coef=coef)
    orp, oci, ov = O.csc_to_csr(cp, rv, nz, ref["nfree"])
    ob = O.assemble_vector(ref, 2 * order, 1.0)
    V = GT.lagrange_space(GT.interior(m), order)
    A, b = GT.assemble_matrix_and_vector(GT.laplacian(coef), GT.source(1.0), "mixed", V)
    rp, ci, v = A.csr()
    assert np.array_equal(rp, orp) and np.array_equal(ci, oci)
    scale = np.abs(ov).max()
    assert np.abs(v - ov).max() <= 2e-13 * scale
    assert np.abs(A.values32() - ov).max() <= 5e-6 * scale
    assert np.abs(b - ob).max() <= 2e-13 * np.abs(ob).max()
    # the row sums of a pure Neumann Laplacian vanish, and the matrix is symmetric
    import scipy.sparse as sp
    M = sp.csr_matrix((v, ci, rp))
    assert np.abs(M @ np.ones(M.shape[0])).max() <= 2e-12 * scale
    assert abs(M - M.T).max() <= 2e-13 * scale


def test_fp32_point_weights_of_the_load_vector_p2():
    # |det J| w is held in the matrix's type.  The shape functions sum to one at
    # every point, so the load vector of f = 1 sums to the cells' rounded point
    # weights.  det J is the product of differences of rounded coordinates (a
    # few eps off the cell volume; a point's rounding to FP32 changes for it
    # with probability ~1e-8), the sum is exact to n eps: 1e-13 against the
    # 1e-9 and more that the rounding to FP32 moves it.
    cells = (3, 5, 7)
    m = GT.cartesian_mesh((0.0, 1.0, 0.0, 1.0, 0.0, 1.0), cells, simplexify=True)
    V = GT.lagrange_space(GT.interior(m), 2)
    w = np.repeat([-74 / 5625, 343 / 45000, 56 / 2250], [1, 4, 6])
    want = m.num_cells * (w / np.prod(cells)).astype(np.float32).astype(np.float64).sum()
    assert abs(want - 1.0) > 1e-10
    _, b = GT.assemble_matrix_and_vector(GT.laplacian(None), GT.source(1.0), np.float32, V)
    assert abs(np.asarray(b, np.float64).sum() - want) <= 1e-13


@pytest.mark.parametrize("order", [1, 2])
def test_fp32_point_weights_of_the_load_vector_hex(order):
    # the same on distorted hexahedra (parallel ones take the factored path,
    # whose weights are FP64), det J from the trilinear map's gradients
    m = GT.cartesian_mesh((0.0, 1.0, 0.0, 1.0, 0.0, 1.0), (3, 5, 7))
    m.coords += np.random.default_rng(5).uniform(-0.02, 0.02, m.coords.shape)
    V = GT.lagrange_space(GT.interior(m), order)
    x1, w1 = np.polynomial.legendre.leggauss(order + 1)
    x1, w1 = 0.5 + 0.5 * x1, 0.5 * w1
    X = m.coords[m.cell_nodes.astype(np.int64) - 1]
    want = exact = 0.0
    for q in np.ndindex(order + 1, order + 1, order + 1):
        g = np.empty((8, 3))
        for v in range(8):
            for d in range(3):
                g[v, d] = np.prod([((1 if v >> t & 1 else -1) if t == d else (x1[q[t]] if v >> t & 1 else 1 - x1[q[t]]))
                                   for t in range(3)])
        dv = np.abs(np.linalg.det(np.einsum("cvi,vj->cij", X, g))) * w1[q[0]] * w1[q[1]] * w1[q[2]]
        want += dv.astype(np.float32).astype(np.float64).sum()
        exact += dv.sum()
    assert abs(want - exact) > 1e-11
    _, b = GT.assemble_matrix_and_vector(GT.laplacian(None), GT.source(1.0), np.float32, V)
    assert abs(np.asarray(b, np.float64).sum() - want) <= 1e-13


@pytest.mark.parametrize("n", [2, 9, 17])
def test_fp32_values_of_q1_hexahedra(n):
    """FP32 values of distorted Q1 hexahedra are the element entries rounded
    once and added in FP32.  With u = 2^-24, a rounding error of rms u / sqrt 3
    of each of a diagonal entry's eight about equal terms (sqrt(1/8) of the
    entry) and of its seven partial sums (sqrt(sum (j/8)^2, j = 2..8) = 1.78 of
    the entry) gives at most 1.82 u / sqrt 3 = 6.3e-8 in the 2-norm."""
    m = GT.cartesian_mesh((0.0, 1.0, 0.0, 1.0, 0.0, 1.0), (n, n, n))
    m.coords += np.random.default_rng(3).uniform(-0.15, 0.15, m.coords.shape) / n
    V = GT.lagrange_space(GT.interior(m), 1)
    A = GT.assemble_matrix(GT.laplacian(GT.lognormal_cells(m.num_cells, 0.5, 17)), "mixed", V)
    v = A.csr()[2]
    assert np.linalg.norm(A.values32() - v) <= 6.3e-8 * np.linalg.norm(v)


@pytest.mark.parametrize("cells,order", [((1, 1, 1), 1), ((2, 4, 4), 1), ((3, 11, 2), 1), ((2, 2, 2), 2), ((3, 3, 3), 2)])
def test_mass_blocks_and_vector_of_hexahedra(cells, order):
    """Mass matrices of distorted hexahedra (Q1: 32 cells a block) against the
    oracle's quadrature, with the bounds above, and the element vectors: the
    same whether a matrix is formed with them or not, and whichever."""
    m = GT.cartesian_mesh((0.0, 1.0, -0.5, 2.0, 0.0, 0.7), cells)
    m.coords += np.random.default_rng(3).uniform(-0.1, 0.1, m.coords.shape) / max(cells)
    coef = GT.lognormal_cells(m.num_cells, 1.0, 17)
    ref, _ = _oracle_space(m, order, 1, None)
    cp, rv, nz = O.assemble_matrix(ref, O.MASS, 2 * order, coef=coef)
    orp, oci, ov = O.csc_to_csr(cp, rv, nz, ref["nfree"])
    ob = O.assemble_vector(ref, 2 * order, 1.0, coef=coef)
    V = GT.lagrange_space(GT.interior(m), order)
    l = GT.source(1.0, coef)
    A, b = GT.assemble_matrix_and_vector(GT.mass(coef), l, "mixed", V)
    rp, ci, v = A.csr()
    assert np.array_equal(rp, orp) and np.array_equal(ci, oci)
    scale = np.abs(ov).max()
    assert np.abs(v - ov).max() <= 2e-13 * scale
    assert np.abs(A.values32() - ov).max() <= 5e-6 * scale
    assert np.abs(b - ob).max() <= 2e-13 * np.abs(ob).max()
    _, b2 = GT.assemble_matrix_and_vector(GT.laplacian(coef), l, np.float64, V)
    assert np.array_equal(b, b2) and np.array_equal(b, GT.assemble_vector(l, np.float64, V))
