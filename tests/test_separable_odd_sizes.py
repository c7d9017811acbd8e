"""Complex64 separable sums whose intermediate has an odd number of elements
(odd grids, bases and term counts): the tensor-core operands behind it start
on their alignment all the same.  Against numpy in complex128, at the
tolerance of the other complex64 separable contractions (2e-6)."""
import numpy as np
import pytest

from helpers import approx_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("NE,Nk,Nb,J", [(55, 9, 5, 5), (33, 3, 7, 1), (65, 5, 9, 7), (41, 3, 3, 9)])
def test_odd_intermediate(gpu_ops, NE, Nk, Nb, J):
    from qclb200.problem import Mechanism

    rng = np.random.default_rng(NE)
    N2 = Nb * Nb

    def r(*shape):
        return np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape))

    radial, block, G, wk = r(Nk, Nk, J), r(N2, N2, J), r(NE, Nk, Nb, Nb), rng.uniform(0.2, 1.0, Nk)
    got = gpu_ops.production_static_contraction(
        Mechanism("impurity", "separable_sum", 0.7, radial=radial, block=block), G, wk, precision="c64")
    A = (G * wk[None, :, None, None]).reshape(NE, Nk, N2, order="F")
    ref = np.zeros((NE, Nk, N2), complex)
    for i in range(J):
        ref += np.einsum("mn,enq->emq", radial[:, :, i], A) @ block[:, :, i].T
    assert approx_err(got, (0.7 * ref).reshape(G.shape, order="F")) < 2e-6
