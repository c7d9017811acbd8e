"""Host arrays staged through pinned slots: the same results as the small calls
that are copied directly, for calls of one slab, several, and a last one that
is not full, in place, for strided (Dyson) and contiguous (Hilbert) parts, and
from pinned memory, which is copied directly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _columns(rng, NE, ncols):
    return np.asfortranarray(rng.standard_normal((NE, ncols)) + 1j * rng.standard_normal((NE, ncols)))


# 8 MB over the fields starts the staging; a slab is 4 MB of a field
@pytest.mark.parametrize("NE,ncols", [(700, 250), (700, 375), (1001, 800), (513, 2049)])
def test_staged_hilbert_equals_direct_columns(gpu_ops, NE, ncols):
    rng = np.random.default_rng(ncols)
    eps = np.linspace(-1.0, 2.0, NE)
    wE = np.full(NE, eps[1] - eps[0])
    SL, SG = _columns(rng, NE, ncols), _columns(rng, NE, ncols)
    SR, Gam, r = gpu_ops.retarded_self_energy_fft(SL, SG, eps, wE, return_roundoff=True)
    assert 0 <= r < 1e-12
    for c0 in range(0, ncols, 90):  # below 8 MB: copied directly
        part = slice(c0, min(ncols, c0 + 90))
        sr, gam = gpu_ops.retarded_self_energy_fft(SL[:, part], SG[:, part], eps, wE)
        assert np.array_equal(gam, Gam[:, part])
        assert np.linalg.norm(sr - SR[:, part]) <= 1e-14 * np.linalg.norm(sr)


def test_staged_hilbert_in_place_and_pinned(gpu_ops):
    import ctypes

    import torch

    from qclb200 import _lib

    rng = np.random.default_rng(5)
    NE, ncols = 801, 900
    eps = np.linspace(-1.0, 2.0, NE)
    wE = np.full(NE, eps[1] - eps[0])
    X = _columns(rng, NE, ncols)
    want = gpu_ops.fft_hilbert_transform(X, eps, wE)
    P = ctypes.c_void_p
    lib = _lib.lib()
    pinned = torch.from_numpy(X.ravel(order="F").copy()).pin_memory()
    for src in (X.copy(order="F"), pinned.numpy()):
        ptr = P(src.ctypes.data)
        _lib.check(lib.qcl_fft_hilbert_transform(0, NE, ncols, P(eps.ctypes.data), P(wE.ctypes.data), ptr, ptr, None))
        got = src.reshape((NE, ncols), order="F")
        assert np.linalg.norm(got - want) <= 1e-14 * np.linalg.norm(want)


@pytest.mark.parametrize("NE,Nk,Nb", [(500, 9, 11), (2100, 13, 7)])
@pytest.mark.parametrize("precision", ["c128", "mixed"])
def test_staged_dyson_equals_direct_momenta(gpu_ops, NE, Nk, Nb, precision):
    from helpers import dyson_inputs

    eps, h, SR, SL, SG = dyson_inputs(3, NE, Nk, Nb)
    whole = gpu_ops.dyson_keldysh(eps, h, SR, SL, SG, precision=precision, return_traces=True)
    for m in range(Nk):  # one momentum: copied directly
        at = slice(m, m + 1)
        one = gpu_ops.dyson_keldysh(eps, np.asfortranarray(h[at]), SR[:, at], SL[:, at], SG[:, at],
                                    precision=precision, return_traces=True)
        for a, b in zip(whole, one):
            assert np.array_equal(a[:, at], b)
