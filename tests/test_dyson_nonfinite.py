"""A block with a NaN below an exact zero on the diagonal of its first pivot
column: the NaN is the pivot (as in the warp-per-block kernel of the larger
bases), so the block's result is not finite and no block is singular.  The
other blocks keep the oracle's values at the tolerances of the other Dyson
tests (complex128 1e-12; complex64 5e-5)."""
import numpy as np
import pytest

from helpers import approx_err, dyson_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,NE", [(2, 70), (3, 64), (4, 65), (5, 2100), (5, 90), (6, 4200), (7, 90)])
@pytest.mark.parametrize("precision,tol", [("c128", 1e-12), ("c64", 5e-5)])
def test_nan_in_the_pivot_column_is_not_singular(gpu_ops, orc, N, NE, precision, tol):
    eps, h, SR, _, _ = dyson_inputs(900 + N, NE, 1, N)
    e = NE // 2
    h[:] = 0.0  # D = eps - Sigma^R exactly
    if precision == "c64":
        eps = eps.astype(np.float32).astype(float)
    SR[e, 0, :, 0] = 0.0
    SR[e, 0, 0, 0] = eps[e]
    SR[e, 0, N - 1, 0] = np.nan
    GR = gpu_ops.retarded_green(eps, h, SR, precision=precision)
    assert not np.isfinite(GR[e]).any()
    ok = np.arange(NE) != e
    ref = orc.retarded_green(eps[ok], h, np.asfortranarray(SR[ok]))[0]
    assert approx_err(GR[ok], ref) < tol
