"""The thread-per-block Dyson kernel of small bases, on both sides of its
block-count line, against the oracle at the tolerances of the other Dyson
tests (complex128 1e-12; complex64 / mixed 5e-5 / 2e-5)."""
import numpy as np
import pytest

from helpers import approx_err, dyson_inputs

pytestmark = pytest.mark.gpu


# (N_b, N_E, N_k): one block, warps with idle lanes, the lines at 2048 (N_b = 5) and 4096 blocks (N_b = 6)
@pytest.mark.parametrize("N,NE,Nk", [(1, 1, 1), (2, 65, 3), (3, 64, 2), (4, 129, 5), (5, 683, 3), (5, 682, 3),
                                     (6, 1366, 3), (6, 1365, 3)])
@pytest.mark.parametrize("precision,tol", [("c128", 1e-12), ("c64", 5e-5), ("mixed", 2e-5)])
def test_small_basis_matches_oracle(gpu_ops, orc, N, NE, Nk, precision, tol):
    eps, h, SR, SL, SG = dyson_inputs(300 + N, NE, Nk, N)
    GR, GL, GG, scale, trL, trG = gpu_ops.dyson_keldysh(eps, h, SR, SL, SG, precision=precision, return_traces=True)
    oGR, _, oscale, _ = orc.retarded_green(eps, h, SR)
    oGL, oGG = orc.keldysh_green(oGR, SL), orc.keldysh_green(oGR, SG)
    for got, ref in ((GR, oGR), (GL, oGL), (GG, oGG), (trL, np.trace(oGL, axis1=2, axis2=3)),
                     (trG, np.trace(oGG, axis1=2, axis2=3))):
        assert approx_err(got, ref) < tol
    np.testing.assert_allclose(scale, oscale, rtol=1e-14 if precision == "c128" else 1e-6)


@pytest.mark.parametrize("N,k", [(2, 2), (5, 3), (5, 5), (6, 1)])
def test_small_basis_singular_block(gpu_ops, N, k):
    """A zero k-th pivot (row and column k of the block zero) in one block."""
    from qclb200 import SingularException

    NE = 4500
    eps = np.linspace(1.0, 2.0, NE)
    h = np.zeros((1, N, N), dtype=complex)
    SR = np.zeros((NE, 1, N, N), dtype=complex, order="F")
    SR[77, 0, k - 1, k - 1] = eps[77]
    with pytest.raises(SingularException) as ex:
        gpu_ops.retarded_green(eps, h, SR)
    assert ex.value.k == k
