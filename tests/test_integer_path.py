"""Complex128 contractions on the integer tensor path (csrc/i8_gemm.cu).

Sizes just above the line of its dispatch rule, at the edges of its tiles,
panels and accumulation lengths, against the same product in numpy (FP64) or
the oracle.  Tolerance: the digits keep each part to 2^-61 of its row's
largest and the products left out are below 2^-64 of a product of row maxima,
which is far below the FP64 sums on the other side of the comparison, whose
relative error is bounded by sqrt(K) 2^-53 times a small constant: 1e-13, the
tolerance of the other complex128 contraction tests.
"""
import numpy as np
import pytest

from helpers import approx_err

pytestmark = pytest.mark.gpu


def _random(rng, *shape):
    return np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape))


def _dense(M, G, wk, factor):
    NE = G.shape[0]
    A = (G * wk[None, :, None, None]).reshape(NE, -1, order="F")
    return (factor * (A @ M.T)).reshape(G.shape, order="F")


# rows at and off a tile of 128, K and columns at and off blocks of 64 and tiles of 64 ... 128
@pytest.mark.parametrize("NE,Nk,Nb", [(1024, 4, 16), (641, 3, 21), (257, 5, 20), (192, 4, 24), (2050, 3, 16)])
@pytest.mark.parametrize("beta", [0.0, -0.5])
def test_dense_integer_path_matches_fp64(gpu_ops, NE, Nk, Nb, beta):
    from qclb200.problem import Mechanism

    rng = np.random.default_rng(NE)
    nc = Nk * Nb * Nb
    assert NE * nc * nc >= 1e9
    M, G, S0 = _random(rng, nc, nc), _random(rng, NE, Nk, Nb, Nb), _random(rng, NE, Nk, Nb, Nb)
    wk = rng.uniform(0.2, 1.0, Nk)
    mech = Mechanism("impurity", "dense", 0.7, matrix=M)
    got = gpu_ops.production_static_contraction(mech, G, wk, alpha=1.3, beta=beta, S=S0)
    assert approx_err(got, _dense(M, G, wk, 1.3 * 0.7) + beta * S0) < 1e-13


def test_dense_integer_path_row_scales_and_non_finite_rows(gpu_ops):
    """Rows of very different size (the scale of a row is its own), a zero row,
    operator rows of very different size, and non-finite entries, which stay in
    their row of the result."""
    from qclb200.problem import Mechanism

    rng = np.random.default_rng(4)
    NE, Nk, Nb = 260, 4, 22
    nc = Nk * Nb * Nb
    M, G = _random(rng, nc, nc), _random(rng, NE, Nk, Nb, Nb)
    scale = 10.0 ** rng.integers(-200, 60, NE)
    scale[7] = 0.0
    G = np.asfortranarray(G * scale[:, None, None, None])
    M = np.asfortranarray(M * (10.0 ** rng.integers(-30, 30, nc))[:, None])
    G[11, 2, 3, 4] = np.nan
    G[13, 0, 0, 0] = np.inf
    wk = rng.uniform(0.2, 1.0, Nk)
    got = gpu_ops.production_static_contraction(Mechanism("impurity", "dense", 1.0, matrix=M), G, wk)
    got = got.reshape(NE, nc, order="F")
    assert not np.isfinite(got[[11, 13]]).any()
    assert (got[7] == 0).all()
    ok = np.setdiff1d(np.arange(NE), [11, 13, 7])
    ref = _dense(M, G[ok], wk, 1.0).reshape(len(ok), nc, order="F")
    # every output against the size of its own row and column
    err = np.abs(got[ok] - ref) / (scale[ok][:, None] * np.linalg.norm(M, axis=1)[None, :])
    assert err.max() < 1e-13 * np.linalg.norm(wk)


@pytest.mark.parametrize("NE,Nk,Nb,J", [(900, 10, 14, 3), (101, 50, 13, 8), (30, 7, 46, 8)])
def test_separable_integer_path_matches_fp64(gpu_ops, NE, Nk, Nb, J):
    """Stage 2 of a separable sum: more rows than one panel, a full chunk, and
    a K above one int32 accumulation (8 x 46^2 = 16 928)."""
    from qclb200.problem import Mechanism

    rng = np.random.default_rng(J + Nb)
    N2 = Nb * Nb
    assert NE * Nk * N2 * J * N2 >= 1e9
    radial = _random(rng, Nk, Nk, J)
    block = np.asfortranarray(rng.random((N2, N2, J)) - 0.5 + 1j * (rng.random((N2, N2, J)) - 0.5))
    G = _random(rng, NE, Nk, Nb, Nb)
    wk = rng.uniform(0.2, 1.0, Nk)
    got = gpu_ops.production_static_contraction(
        Mechanism("impurity", "separable_sum", 0.37, radial=radial, block=block), G, wk)
    A = (G * wk[None, :, None, None]).reshape(NE, Nk, N2, order="F")
    ref = np.zeros((NE, Nk, N2), complex)
    for i in range(J):
        ref += np.einsum("mn,enq->emq", radial[:, :, i], A) @ block[:, :, i].T
    assert approx_err(got, (0.37 * ref).reshape(G.shape, order="F")) < 1e-13


def test_scba_integer_path_matches_oracle(gpu_ops, orc):
    """A solve whose dense maps take both Keldysh components through one
    product."""
    from qclb200.problem import small_problem
    from qclb200.scba import solve_scba_production

    pr = small_problem(NE=150, Nk=8, Nb=16, mechanisms=("LO", "impurity"))
    assert 2 * pr.NE * (pr.Nk * pr.Nb ** 2) ** 2 >= 1e9
    hist, solver = solve_scba_production(pr, 2)
    solver.close()
    ref, _ = orc.scba(pr, 2)
    for g, o in zip(hist, ref):
        assert abs(g["J"] - o["J"]) <= 1e-9 * abs(o["J"])
        assert np.allclose(g["populations"], o["populations"], rtol=1e-9, atol=0)
        assert abs(g["r_Sigma"] - o["rSigma"]) <= 1e-9


def test_integer_path_wait_timeout_is_reported_and_recoverable(gpu_ops):
    """With the wait limit at zero the first waits give up with copies in
    flight; the call reports QCL_TIMEOUT and the next one is correct."""
    from qclb200 import _lib
    from qclb200.problem import Mechanism

    rng = np.random.default_rng(9)
    NE, Nk, Nb = 1024, 4, 16
    nc = Nk * Nb * Nb
    M, G, wk = _random(rng, nc, nc), _random(rng, NE, Nk, Nb, Nb), rng.uniform(0.2, 1.0, Nk)
    mech = Mechanism("impurity", "dense", 1.0, matrix=M)
    lib = _lib.lib()
    _lib.check(lib.qcl_debug_set_wait_limit(0))
    try:
        with pytest.raises(_lib.QCLError) as ex:
            gpu_ops.production_static_contraction(mech, G, wk)
        assert ex.value.code == _lib.QCL_TIMEOUT
    finally:
        _lib.check(lib.qcl_debug_set_wait_limit(-1))
    assert approx_err(gpu_ops.production_static_contraction(mech, G, wk), _dense(M, G, wk, 1.0)) < 1e-13
