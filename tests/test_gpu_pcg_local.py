"""The persistent solver on CTA-local vectors (csrc/gt_pcg_local.cuh) at the
edges of its placements: one row, fewer rows than CTAs, one cluster, a grid,
the sliced form, block rows of 1, 2 and 3, and a numbering whose local sets do not fit in
shared memory (solved by the kernel on global vectors).

The solver stops when its FP64 residual is at most rtol ||b||.  The same
residual formed here differs from it by rounding alone, at most
(row length + 2) eps sum |a_ij| |x_j| per entry; that bound is added to rtol.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import gtgpu as GT

pytestmark = pytest.mark.gpu

RTOL = 1e-10


def _system(cell, order, ncomp, n, T, shuffle=False):
    D = 2 if cell == "quad" else 3
    m = GT.cartesian_mesh((0.0, 1.0) * D, (n,) * D, simplexify=cell == "tet")
    if shuffle:
        m.cell_nodes = np.ascontiguousarray(m.cell_nodes[np.random.default_rng(5).permutation(m.num_cells)])
    V = GT.lagrange_space(GT.interior(m), order, tensor_size=(ncomp,) if ncomp > 1 else None,
                          dirichlet_boundary=GT.boundary(m))
    kappa = GT.lognormal_cells(m.num_cells, 0.5, 31)
    a = GT.laplacian(kappa) if ncomp == 1 else GT.elasticity(kappa, 0.3)
    f = 1.0 if ncomp == 1 else [0.5] * (ncomp - 1) + [-1.0]
    return GT.assemble_matrix_and_vector(a, GT.source(f), T, V)


def _check(A, b, x):
    rp, ci, v = A.csr()
    M = sp.csr_matrix((v, ci, rp), shape=(len(b), len(b)))
    r = np.asarray(b) - M @ np.asarray(x)
    row = np.diff(rp).max() + 2
    slack = row * np.finfo(float).eps * np.linalg.norm(abs(M) @ np.abs(x))
    assert np.linalg.norm(r) <= RTOL * np.linalg.norm(b) + slack


@pytest.mark.parametrize("T,mode", [(np.float64, "fp64"), ("mixed", "ir")])
@pytest.mark.parametrize("cell,order,ncomp,n", [
    ("quad", 1, 1, 2),    # one row
    ("quad", 1, 1, 4),    # fewer rows than a cluster has CTAs
    ("quad", 2, 1, 17), ("hex", 1, 1, 9), ("hex", 2, 1, 5), ("tet", 1, 1, 13),  # one cluster
    ("quad", 1, 1, 130), ("hex", 1, 1, 27), ("hex", 2, 1, 13), ("tet", 2, 1, 9),  # a grid
    ("quad", 1, 2, 2), ("quad", 2, 2, 11), ("quad", 1, 2, 90),  # block rows of 2
    ("hex", 1, 3, 2), ("hex", 1, 3, 5), ("hex", 2, 3, 6),  # block rows of 3
])
def test_residual_at_the_edges(cell, order, ncomp, n, T, mode):
    A, b = _system(cell, order, ncomp, n, T)
    x, info = GT.solve(A, b, rtol=RTOL, mode=mode)
    assert info["converged"]
    _check(A, b, x)
    again, _ = GT.solve(A, b, rtol=RTOL, mode=mode)
    assert np.array_equal(x, again)


@pytest.mark.parametrize("T,mode", [(np.float64, "fp64"), ("mixed", "ir")])
@pytest.mark.parametrize("cell,n", [("quad", 514), ("hex", 66), ("tet", 66)])
def test_sliced_form(cell, n, T, mode):
    """Scalar systems above 262,144 rows, streamed from the sliced copy; the
    row counts (513^2, 65^3) leave one row in the last slice of 32."""
    A, b = _system(cell, 1, 1, n, T)
    assert A.shape[0] > 262144 and A.shape[0] % 32 == 1
    x, info = GT.solve(A, b, rtol=RTOL, mode=mode)
    assert info["converged"]
    _check(A, b, x)
    again, _ = GT.solve(A, b, rtol=RTOL, mode=mode)
    assert np.array_equal(x, again)


@pytest.mark.parametrize("T,mode", [(np.float64, "fp64"), ("mixed", "ir")])
def test_scattered_numbering_takes_the_global_vectors(T, mode):
    """Cells in random order number the nodes at random: a CTA's rows touch
    columns all over the system."""
    A, b = _system("tet", 1, 1, 56, T, shuffle=True)
    x, info = GT.solve(A, b, rtol=RTOL, mode=mode)
    assert info["converged"]
    _check(A, b, x)


def test_zero_right_hand_side_and_iteration_limits():
    A, b = _system("quad", 1, 1, 40, np.float64)
    x, info = GT.solve(A, np.zeros_like(b), rtol=RTOL, mode="fp64")
    assert info["iterations"] == 0 and not np.any(x)
    with pytest.raises(Exception):
        GT.solve(A, b, rtol=RTOL, maxit=3, mode="fp64")


@pytest.mark.parametrize("cell,n", [("quad", 33), ("quad", 130), ("tet", 66)])  # a cluster, a grid, the sliced form
def test_squares_of_the_residual_below_the_normal_range(cell, n):
    """b scaled by 2^-480: ||b||^2 lies near 2^-960, ||r||^2 at convergence at
    2^-66 of it, below the smallest normal number.  The solve goes on there:
    the scaled solution has the residual of the unscaled one."""
    A, b = _system(cell, 1, 1, n, np.float64)
    s = 2.0 ** -480
    b = b / np.linalg.norm(b)
    assert RTOL ** 2 * s ** 2 < np.finfo(float).tiny
    x, info = GT.solve(A, b * s, rtol=RTOL, mode="fp64")
    assert info["converged"] and 0.0 < info["rel_residual"] <= RTOL
    _check(A, b, x / s)
