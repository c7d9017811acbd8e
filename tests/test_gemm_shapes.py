"""The generic contraction products at the lines of their tile rules: every
tile shape of the complex64 and complex128 kernels, with rows, columns and K
off the tile edges, beta, and the broadcast over momenta, against the same map
in numpy (complex128 1e-13, complex64 2e-6: the tolerances of the other
contraction tests)."""
import numpy as np
import pytest

from helpers import approx_err

pytestmark = pytest.mark.gpu


def _random(rng, *shape):
    return np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape))


# one CTA; few CTAs (32-row tiles); 64-row tiles; 128-row tiles and 64 x 64 tiles; long K
@pytest.mark.parametrize("NE,Nk,Nb", [(5, 2, 3), (33, 3, 9), (300, 4, 13), (1030, 3, 23), (67, 2, 41)])
@pytest.mark.parametrize("beta", [0.0, 0.6])
@pytest.mark.parametrize("precision,tol", [("c128", 1e-13), ("c64", 2e-6)])
def test_contraction_tile_shapes(gpu_ops, NE, Nk, Nb, beta, precision, tol):
    from qclb200.problem import Mechanism

    rng = np.random.default_rng(NE)
    N2, J = Nb * Nb, 5
    G, S0 = _random(rng, NE, Nk, Nb, Nb), _random(rng, NE, Nk, Nb, Nb)
    wk = rng.uniform(0.2, 1.0, Nk)
    A = (G * wk[None, :, None, None]).reshape(NE, Nk, N2, order="F")
    block = _random(rng, N2, N2)
    left, right, radial = _random(rng, N2, J), _random(rng, J, N2), _random(rng, Nk, Nk)
    ll, lr = _random(rng, Nk * N2, J), _random(rng, J, Nk * N2)
    flat = A.reshape(NE, Nk * N2, order="F")
    cases = [
        (Mechanism("acoustic", "momentum_independent", 0.7, block=block),
         np.broadcast_to((A.sum(axis=1) @ block.T)[:, None, :], A.shape)),
        (Mechanism("IFR", "ifr", 0.7, left=left, right=right, radial=radial),
         np.einsum("mn,enj->emj", radial, A @ right.T) @ left.T),
        (Mechanism("LO", "low_rank", 0.7, left=ll, right=lr),
         ((flat @ lr.T) @ ll.T).reshape(A.shape, order="F")),
    ]
    for mech, ref in cases:
        got = gpu_ops.production_static_contraction(mech, G, wk, alpha=1.3, beta=beta, S=S0, precision=precision)
        want = 0.91 * np.asarray(ref).reshape(G.shape, order="F") + beta * S0
        assert approx_err(got, want) < tol, mech.kind
