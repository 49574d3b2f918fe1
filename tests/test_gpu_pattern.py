"""The warp-per-row sparsity pass at its edges, on fans of 2n P2 tetrahedra
around one node: its row holds 5n + 5 columns of 20n candidates.  n = 5 .. 25
cross the register sorts (32, 64, 128 columns, then shared memory and the fill
pass), n = 13 the candidates the first launch has room for."""
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
