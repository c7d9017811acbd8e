"""Row scales of the complex64 tensor-core products at the edges of the split
kernels: whole rows in one tile (up to 64 complex columns), one column more,
a last slice of a few columns, rows off a tile of 32.  Against the product in
FP64 over the rounded inputs, row by row, at the tolerance of the other
complex64 contraction tests (2e-6: two FP16 halves keep 22 bits, FP32 sums)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _random(rng, *shape):
    return np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape))


@pytest.mark.parametrize("Nk,Nb", [(1, 1), (7, 3), (16, 2), (4, 4), (65, 1), (1, 9), (2, 11), (257, 1), (5, 8)])
@pytest.mark.parametrize("NE", [1, 33, 96])
def test_row_scales(gpu_ops, NE, Nk, Nb):
    from qclb200.problem import Mechanism

    rng = np.random.default_rng(100 * Nk + Nb)
    nc = Nk * Nb * Nb
    M = _random(rng, nc, nc).astype(np.complex64)
    scale = 10.0 ** rng.integers(-20, 12, NE)
    if NE > 2:
        scale[1] = 0.0
    G = np.asfortranarray(_random(rng, NE, Nk, Nb, Nb) * scale[:, None, None, None]).astype(np.complex64)
    G = np.asfortranarray(G)
    if NE > 40:  # non-finite entries, the first and the last column, stay in their rows
        G[5, 0, 0, 0] = np.nan
        G[40, Nk - 1, Nb - 1, Nb - 1] = np.inf
    wk = np.ones(Nk)
    got = gpu_ops.production_static_contraction(Mechanism("impurity", "dense", 1.0, matrix=M.astype(complex)), G, wk,
                                                precision="c64").reshape(NE, nc, order="F")
    with np.errstate(invalid="ignore"):
        ref = G.reshape(NE, nc, order="F").astype(complex) @ M.astype(complex).T
    for e in range(NE):
        if NE > 40 and e in (5, 40):
            assert not np.isfinite(got[e]).all()
        else:
            assert np.linalg.norm(got[e] - ref[e]) <= 2e-6 * np.linalg.norm(ref[e])
