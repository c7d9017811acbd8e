"""Element-wise accuracy of the large complex128 contractions, against extended
precision on a sample of outputs, in units of sum_k |A[e,k]| |B[j,k]|.

An FP64 sum of 2K products stays within about sqrt(2K) 2^-53 of that sum
(random rounding; twice that is the tolerance), however the sizes of the
entries spread within a row.  The integer path keeps entries relative to their
row's largest, so it may only run where that is no worse: where it does, on
rows of one size, it is far more accurate than FP64 sums, which shows the path.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _random(rng, *shape):
    return np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape))


def _errors(A, B, got, sample, rng):
    """|got - A B^T| / sum |A| |B| at `sample` random outputs."""
    es, js = rng.integers(0, A.shape[0], sample), rng.integers(0, B.shape[0], sample)
    a, b = A[es].astype(np.clongdouble), B[js].astype(np.clongdouble)
    size = (np.abs(a) * np.abs(b)).sum(axis=1)
    keep = size > 0
    err = np.abs(got[es, js] - (a * b).sum(axis=1))[keep] / size[keep]
    assert (got[es, js][~keep] == 0).all()
    return err.astype(float)


@pytest.mark.parametrize("spread", [1e-2, 1e-4, 1e-8, 1e-12])
def test_dense_rows_of_graded_entries(gpu_ops, spread):
    """Half of every row of G is small by `spread`, and every other output
    reads only that half."""
    from qclb200.problem import Mechanism

    rng = np.random.default_rng(31)
    NE, Nk, Nb = 420, 4, 22
    nc = Nk * Nb * Nb
    assert NE * nc * nc >= 1e9
    M, G = _random(rng, nc, nc), _random(rng, NE, Nk, Nb, Nb).reshape(NE, nc, order="F")
    G[:, nc // 2:] *= spread
    M[::2, :nc // 2] = 0.0
    got = gpu_ops.production_static_contraction(Mechanism("impurity", "dense", 1.0, matrix=np.asfortranarray(M)),
                                                np.asfortranarray(G).reshape((NE, Nk, Nb, Nb), order="F"), np.ones(Nk))
    err = _errors(G, M, got.reshape(NE, nc, order="F"), 4000, rng)
    assert err.max() < 2 * np.sqrt(2 * nc) * 2.0 ** -53


@pytest.mark.parametrize("spread", [1e-4, 1e-8])
def test_separable_blocks_of_graded_entries(gpu_ops, spread):
    from qclb200.problem import Mechanism

    rng = np.random.default_rng(32)
    NE, Nk, Nb, J = 901, 10, 16, 3
    N2 = Nb * Nb
    assert NE * Nk * N2 * J * N2 >= 1e9
    radial = np.asfortranarray(np.repeat(np.eye(Nk)[:, :, None], J, axis=2).astype(complex))
    block = _random(rng, N2, N2, J)
    block[::2, :N2 // 2] = 0.0
    G = _random(rng, NE, Nk, N2)
    G[:, :, N2 // 2:] *= spread
    got = gpu_ops.production_static_contraction(
        Mechanism("impurity", "separable_sum", 1.0, radial=radial, block=block),
        np.asfortranarray(G).reshape((NE, Nk, Nb, Nb), order="F"), np.ones(Nk))
    A = np.repeat(G.reshape(NE * Nk, N2, order="F")[:, None], J, axis=1).reshape(NE * Nk, J * N2)
    B = block.transpose(0, 2, 1).reshape(N2, J * N2)
    err = _errors(A, B, got.reshape(NE * Nk, N2, order="F"), 4000, rng)
    assert err.max() < 2 * np.sqrt(2 * J * N2) * 2.0 ** -53


def test_rows_of_one_size_take_the_integer_path(gpu_ops):
    """Rows of normal entries, of sizes 1e-100 to 1e100, with zero rows on both
    sides (a row of G outside the energy window, an uncoupled output)."""
    from qclb200.problem import Mechanism

    rng = np.random.default_rng(33)
    NE, Nk, Nb = 400, 8, 16
    nc = Nk * Nb * Nb
    M, G = _random(rng, nc, nc), _random(rng, NE, nc)
    G *= 10.0 ** rng.integers(-100, 101, NE)[:, None]
    M *= 10.0 ** rng.integers(-100, 101, nc)[:, None]
    G[[0, 5, 129]] = 0.0
    M[[7, 2047]] = 0.0
    got = gpu_ops.production_static_contraction(Mechanism("impurity", "dense", 1.0, matrix=np.asfortranarray(M)),
                                                np.asfortranarray(G).reshape((NE, Nk, Nb, Nb), order="F"), np.ones(Nk))
    err = _errors(G, M, got.reshape(NE, nc, order="F"), 4000, rng)
    # the path's own rounding: six FP64 additions into C, whose parts are of the size of |C|, which for random
    # phases stays below 4.5 / sqrt(K) of the sum: 6.6e-17; sums of K FP64 products exceed 2e-16
    assert err.max() < 6 * 2.0 ** -53 * 4.5 / np.sqrt(nc)


# rows off and at a tile of 128, K off and at blocks of 32 and stages of 8 of them
@pytest.mark.parametrize("NE,Nk,Nb", [(641, 3, 22), (1024, 4, 16), (449, 5, 20), (2050, 3, 16), (385, 6, 17)])
@pytest.mark.parametrize("beta", [0.0, -0.5])
@pytest.mark.parametrize("large", [1.0, 0.1])
def test_dense_levels(gpu_ops, NE, Nk, Nb, beta, large):
    """Columns of normal entries, or one in ten of them with the others 1e-3 of
    their size: the leading bits then ask for one more diagonal of digits."""
    from qclb200.problem import Mechanism

    rng = np.random.default_rng(NE)
    nc = Nk * Nb * Nb
    assert NE * nc * nc >= 1e9
    M, G, S0 = _random(rng, nc, nc), _random(rng, NE, nc), _random(rng, NE, nc)
    for X in (M, G):
        X *= np.where(rng.random(nc) < large, 1.0, 1e-3)[None, :]
    S0 *= np.abs(G).max() * np.abs(M).max()
    f = lambda x: np.asfortranarray(x).reshape((NE, Nk, Nb, Nb), order="F")
    got = gpu_ops.production_static_contraction(Mechanism("impurity", "dense", 1.0, matrix=np.asfortranarray(M)), f(G),
                                                np.ones(Nk), beta=beta, S=f(S0)).reshape(NE, nc, order="F")
    # the term of S0 enters both sides as one more product
    A, B = np.concatenate([G, np.ones((NE, 1))], axis=1), np.concatenate([M, np.zeros((nc, 1))], axis=1)
    es, js = rng.integers(0, NE, 4000), rng.integers(0, nc, 4000)
    a, b = A[es].astype(np.clongdouble), B[js].astype(np.clongdouble)
    b[:, -1] = beta * S0[es, js]
    err = np.abs(got[es, js] - (a * b).sum(axis=1)) / (np.abs(a) * np.abs(b)).sum(axis=1)
    assert err.max() < 2 * np.sqrt(2 * nc) * 2.0 ** -53
    ref = G @ M.T + beta * S0
    assert np.linalg.norm(got - ref) < 1e-13 * np.linalg.norm(ref)
