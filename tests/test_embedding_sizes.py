"""The embedding kernel at the edges of its padded sizes and energy tiles,
against the oracle, at the tolerances of the other operator tests (complex128
1e-13, complex64 1e-5: two sums of up to 48 complex products in FP32)."""
import numpy as np
import pytest

from helpers import approx_err

pytestmark = pytest.mark.gpu


# (N_b, N_E, N_k): one energy, ragged last tiles of 1, 2, 4 and 8 energies, both sides of the padded sizes
@pytest.mark.parametrize("N,NE,Nk", [(1, 2, 1), (7, 9, 2), (8, 33, 1), (9, 13, 3), (16, 21, 2), (17, 7, 2), (23, 10, 1),
                                     (25, 5, 2), (32, 11, 2), (33, 4, 1), (48, 6, 2)])
@pytest.mark.parametrize("precision,tol", [("c128", 1e-13), ("c64", 1e-5)])
def test_embedding_sizes(gpu_ops, orc, N, NE, Nk, precision, tol):
    rng = np.random.default_rng(1000 * N + NE)
    eps = np.linspace(-1.0, 2.0, NE)
    T = rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))
    G = np.asfortranarray(rng.standard_normal((NE, Nk, N, N)) + 1j * rng.standard_normal((NE, Nk, N, N)))
    for delta in (0.37, -0.61, 0.0, 3.0 / (NE - 1)):
        got = gpu_ops.embedding_component(T, G, eps, delta, precision=precision)
        assert approx_err(got, orc.embedding_component(T, G, orc.ShiftPlan(eps, delta))) < tol
