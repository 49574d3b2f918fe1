"""The persistent solver on CTA-local vectors (csrc/gt_pcg_local.cuh) at the
edges of its placements: one row, fewer rows than CTAs, one cluster, a grid,
the sliced form, block rows of 1, 2 and 3, and a numbering whose local sets do not fit in
shared memory (solved by the kernel on global vectors).

The solver stops when its FP64 residual is at most rtol ||b||.  The same
residual formed here differs from it by rounding alone, at most
(row length + 2) eps sum |a_ij| |x_j| per entry; that bound is added to rtol.
"""
import math

import numpy as np
import pytest
import scipy.sparse as sp

import gtgpu as GT
from gtgpu import _lib
from gtgpu.api import _ptr

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


def _scattered(cell, order, ncomp, n, T):
    """nodes numbered at random"""
    D = 2 if cell == "quad" else 3
    m = GT.cartesian_mesh((0.0, 1.0) * D, (n,) * D, simplexify=cell == "tet")
    new = np.random.default_rng(5).permutation(m.num_nodes)
    coords = np.empty_like(m.coords)
    coords[new] = m.coords
    m.coords = coords
    for name in ("cell_nodes", "corners", "bfaces", "bedges"):
        a = getattr(m, name)
        setattr(m, name, np.ascontiguousarray((new[a - 1] + 1).astype(np.int32)) if a.size else a)
    m.cell_nodes = np.ascontiguousarray(m.cell_nodes[np.random.default_rng(6).permutation(m.num_cells)])
    V = GT.lagrange_space(GT.interior(m), order, tensor_size=(ncomp,) if ncomp > 1 else None,
                          dirichlet_boundary=GT.boundary(m))
    k = GT.lognormal_cells(m.num_cells, 0.5, 31)
    a = GT.laplacian(k) if ncomp == 1 else GT.elasticity(k, 0.3)
    return GT.assemble_matrix_and_vector(a, GT.source(1.0 if ncomp == 1 else [0.5] * ncomp), T, V)


@pytest.mark.parametrize("T,mode", [(np.float64, "fp64"), ("mixed", "ir"), ("mixed", "fp32")])
@pytest.mark.parametrize("n", [56, 66])  # below and above 262,144 rows
def test_scattered_nodes(n, T, mode):
    """A CTA's rows touch columns all over the system, whose local sets do not
    fit in shared memory.  The kernel on global vectors, or one launch per
    phase, solves it, and a second solve goes there at once, with the same
    result."""
    A, b = _scattered("tet", 1, 1, n, T)
    rtol = RTOL if mode != "fp32" else 1e-4
    count, xs = [], []
    for _ in range(2):
        l0 = A.ctx.launches()
        x, info = GT.solve(A, b, rtol=rtol, mode=mode)
        count.append(A.ctx.launches() - l0)
        xs.append(x)
        assert info["converged"]
        if mode != "fp32":  # (stops by its recurrence residual)
            _check(A, b, x)
    assert np.array_equal(xs[0], xs[1])
    assert count[1] < count[0] or (n, mode) == (56, "fp32")  # (fits)


@pytest.mark.parametrize("mode", ["fp64", "ir"])
@pytest.mark.parametrize("cell,order,ncomp,n", [
    ("hex", 2, 1, 25), ("quad", 2, 1, 250), ("quad", 2, 2, 170), ("hex", 1, 3, 41), ("hex", 2, 3, 17)])
def test_kernel_on_global_vectors(cell, order, ncomp, n, mode):
    """its lane counts: mean rows up to and above 40 entries, block rows"""
    A, b = _scattered(cell, order, ncomp, n, "mixed")
    x, info = GT.solve(A, b, rtol=RTOL, mode=mode)
    assert info["converged"] and info["rel_residual"] <= RTOL
    _check(A, b, x)


@pytest.mark.parametrize("cell,order,ncomp,n", [
    ("quad", 1, 1, 2), ("quad", 1, 1, 4), ("quad", 2, 1, 17), ("hex", 1, 1, 9), ("tet", 1, 1, 13),  # one cluster
    ("quad", 1, 1, 130), ("hex", 2, 1, 13), ("tet", 2, 1, 9),  # a grid
    ("quad", 1, 2, 2), ("quad", 2, 2, 11), ("hex", 1, 3, 2), ("hex", 2, 3, 6),  # block rows
    ("quad", 1, 1, 514), ("hex", 1, 1, 66),  # the sliced form
])
def test_fp32_mode(cell, order, ncomp, n):
    """The FP32 iteration without residual updates stops by its recurrence
    residual, which drifts from the true one by the rounding of the k updates
    of x and r: at most (row length + 4) u sum |a_ij| |x_j| each."""
    A, b = _system(cell, order, ncomp, n, "mixed")
    x, info = GT.solve(A, b, rtol=1e-4, mode="fp32")
    assert info["converged"]
    rp, ci, v = A.csr()
    M = sp.csr_matrix((v, ci, rp), shape=(len(b), len(b)))
    u, k = 2.0 ** -24, info["iterations"]
    slack = (k + 1) * (np.diff(rp).max() + 4) * u * np.linalg.norm(abs(M) @ np.abs(x))
    r = np.linalg.norm(b - M @ x)
    assert r <= 1e-4 * np.linalg.norm(b) + slack
    assert abs(info["rel_residual"] - r / np.linalg.norm(b)) <= 1e-6 * info["rel_residual"]
    again, _ = GT.solve(A, b, rtol=1e-4, mode="fp32")
    assert np.array_equal(x, again)


def _sum(values, fp32=False, missing=0, timeout=200_000_000):
    ctx = GT.default_context()
    values = np.ascontiguousarray(values, np.float64)
    out = np.full(1, np.nan)
    st = ctx.lib.gt_ctx_sum_probe(ctx.h, values.size // 512, missing, timeout,
                                  _lib.GT_FP32 if fp32 else _lib.GT_FP64, _ptr(values), _ptr(out))
    return st, out[0]


@pytest.mark.parametrize("ctas", [1, 2, 33, 152])
@pytest.mark.parametrize("fp32", [False, True])
def test_sums_on_the_integer_pipes(ctas, fp32):
    """Over a warp's lanes, a CTA's warps and the CTAs numbers are aligned to the
    largest one and rounded 56, 56 and 53 bits below it: with at most 32, 16 and
    160 of them, the total is off by 2^-52 + 2^-53 + 2^-46 of the magnitudes' sum
    at most, and sums of whole numbers below 2^30 are exact."""
    rng = np.random.default_rng(ctas)
    n = 512 * ctas
    whole = rng.integers(-2 ** 14, 2 ** 14, n).astype(np.float64)
    assert _sum(whole, fp32) == (0, whole.sum())
    assert _sum(rng.permutation(whole), fp32) == (0, whole.sum())
    for spread in (0, 8, 30):
        v = rng.standard_normal(n) * 2.0 ** rng.uniform(-spread, spread, n)
        if fp32:
            v = v.astype(np.float32).astype(np.float64)
        st, t = _sum(v, fp32)
        assert st == 0 and abs(t - math.fsum(v)) <= 2.0 ** -45 * math.fsum(np.abs(v))
    one = np.zeros(n)
    one[n // 2] = -1.7e-42 if fp32 else -4.9e-324  # subnormal
    assert _sum(one, fp32)[1] == np.float64(np.float32(one[n // 2]) if fp32 else one[n // 2])
    tiny = rng.integers(-999, 999, n) * 2.0 ** (-149 if fp32 else -1074)
    assert _sum(tiny, fp32)[1] == math.fsum(tiny)
    assert _sum(np.zeros(n), fp32) == (0, 0.0)
    big = np.zeros(n)
    big[:3] = [1.5 * 2.0 ** (127 if fp32 else 1023), 2.0 ** (126 if fp32 else 1022), -(2.0 ** (126 if fp32 else 1022))]
    assert _sum(big, fp32)[1] == big[0]
    for bad in (np.nan, np.inf, -np.inf):
        one[n // 2] = bad
        assert np.isnan(_sum(one, fp32)[1])


def test_sum_of_a_missing_arrival_gives_up():
    v = np.ones(512 * 16)
    assert _sum(v)[0] == _lib.GT_OK
    st, _ = _sum(v, missing=1, timeout=50_000_000)
    assert st == _lib.GT_ERR_TIMEOUT
    assert _sum(v, missing=160)[0] == _lib.GT_ERR_INVALID
    assert _sum(v) == (_lib.GT_OK, 512.0 * 16)  # the context goes on
    A, b = _system("quad", 1, 1, 40, np.float64)
    assert GT.solve(A, b, rtol=RTOL, mode="fp64")[1]["converged"]


def test_quick_division():
    """within an ulp of the quotient; the division itself where an exponent is
    near the ends of the range, and for zeros, infinities and NaN"""
    rng = np.random.default_rng(1)
    n = 200_000
    e = np.concatenate([rng.uniform(-500, 500, n), [-511, -511, 511.9, 511.9] * 50])
    a = rng.uniform(1, 2, e.size) * 2.0 ** np.floor(e) * rng.choice([-1, 1], e.size)
    b = rng.uniform(1, 2, e.size) * 2.0 ** np.floor(rng.permutation(e)) * rng.choice([-1, 1], e.size)
    edge = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e-310, 1e308, 2.0 ** -512, 2.0 ** 513, 1.0, -3.0])
    A, B = (x.ravel() for x in np.meshgrid(edge, edge))
    a, b = np.concatenate([a, A]), np.concatenate([b, B])
    q = np.empty_like(a)
    ctx = GT.default_context()
    assert ctx.lib.gt_ctx_divide_probe(ctx.h, a.size, _ptr(a), _ptr(b), _ptr(q)) == 0
    with np.errstate(all="ignore"):
        want = a / b
        m = e.size
        assert np.all(np.abs(q[:m] - want[:m]) <= np.spacing(np.abs(want[:m])))
    ea, eb = (np.frexp(x[m:])[1] + 1022 for x in (a, b))
    plain = (np.minimum(ea, eb) < 512) | (np.maximum(ea, eb) > 1535) | (a[m:] == 0) | (b[m:] == 0)
    plain |= ~np.isfinite(a[m:]) | ~np.isfinite(b[m:])
    assert np.array_equal(q[m:][plain], want[m:][plain], equal_nan=True)
    assert np.all(np.abs(q[m:][~plain] - want[m:][~plain]) <= np.spacing(np.abs(want[m:][~plain])))
