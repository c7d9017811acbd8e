"""qcl_dev_dyson_keldysh with the Green functions written over the self
energies, on both sides of the dispatch lines of the small-basis kernel.

The reference is the out-of-place call of the same kernels: the same sums, or
the same sums in the order of the other kernel, whose differences the
tolerances of the other Dyson tests cover (complex128 1e-12, complex64 5e-5,
mixed 2e-5).
"""
import ctypes

import numpy as np
import pytest

from helpers import approx_err, dyson_inputs

pytestmark = pytest.mark.gpu


def _call(torch, precision, NE, Nk, N, eps, h, SR, SL, SG, GL, GG):
    from qclb200 import _lib

    p = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())
    GR, status = torch.empty_like(SR), torch.zeros(2, dtype=torch.int32, device="cuda")
    _lib.check(_lib.lib().qcl_dev_dyson_keldysh(
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), _lib.PRECISIONS[precision], NE, Nk, N, p(eps), 0.0,
        p(h), p(SR), p(SL), p(SG), p(GR), p(GL), p(GG), None, None, None, p(status)))
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0]


@pytest.mark.parametrize("N,NE,Nk", [(1, 33, 2), (2, 65, 3), (3, 64, 2), (4, 129, 5), (5, 683, 3), (5, 100, 2),
                                     (6, 1366, 3), (12, 67, 2)])
@pytest.mark.parametrize("precision,tol", [("c128", 1e-12), ("c64", 5e-5), ("mixed", 2e-5)])
def test_green_functions_over_the_self_energies(gpu_ops, N, NE, Nk, precision, tol):
    import torch

    eps, h, SR, SL, SG = dyson_inputs(700 + N, NE, Nk, N)
    dt = torch.complex128 if precision == "c128" else torch.complex64
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a.transpose(3, 2, 1, 0))).to("cuda", dt)
    SR, SL, SG = dev(SR), dev(SL), dev(SG)
    eps = torch.from_numpy(eps).cuda()
    h = torch.from_numpy(h.ravel(order="F").copy()).cuda()
    GL, GG = torch.empty_like(SL), torch.empty_like(SL)
    _call(torch, precision, NE, Nk, N, eps, h, SR, SL, SG, GL, GG)
    L, G = SL.clone(), SG.clone()
    _call(torch, precision, NE, Nk, N, eps, h, SR, L, G, L, G)
    assert approx_err(L.cpu().numpy(), GL.cpu().numpy()) < tol
    assert approx_err(G.cpu().numpy(), GG.cpu().numpy()) < tol
    # one component alone, in place
    L = SL.clone()
    _call(torch, precision, NE, Nk, N, eps, h, SR, L, None, L, None)
    assert approx_err(L.cpu().numpy(), GL.cpu().numpy()) < tol
