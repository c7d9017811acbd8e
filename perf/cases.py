"""The calls of the SCBA hot path that a host program makes, at the sizes it makes them.

Five kinds of case:

* ``dyson``: the batched Dyson solve with its Keldysh products on device
  fields (``qcl_dev_dyson_keldysh``), per (E, k) block;
* ``hilbert``: the FFT Hilbert transform of device columns
  (``qcl_dev_fft_hilbert_transform``), with or without the length-2L check;
* ``suite``: the fixed-point residual suite on device fields
  (``qcl_dev_residual_suite_noalloc``);
* ``sigma``: the operator-level drop-in on host arrays
  (``operators.retarded_self_energy_fft``), copies included;
* ``scba``: iterations of a device-resident solve (``ProductionSCBA``), then
  the coherence matrix that the outer Poisson loop reads (and, for small
  structures, the Green functions).

``exact`` restates each in 64-bit torch.  Outputs that one computes at
roundoff level (a solve's own defects) are given together with the sizes they
are small against, or left without a value.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qclnegf.jl_b200"))

from qclb200 import _lib, operators  # noqa: E402
from qclb200.problem import Mechanism, SCBAProblem, energy_grid, momentum_grid  # noqa: E402
from qclb200.scba import ProductionSCBA  # noqa: E402

PTR = ctypes.c_void_p
ALL = "LO acoustic impurity IFR alloy"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a first look at a structure: four states, a coarse grid, and its Green functions; launches and host
        # reads are all of the time
        dict(name="scba_small", kind="scba", precision="c128", NE=41, Nk=3, Nb=4, mechanisms="LO acoustic IFR",
             form="dense", terms=5, steps=5, green=True),
        # the tutorial-sized structure (3 periods x 4 states, acoustic phonons) in FP64
        dict(name="scba_tutorial", kind="scba", precision="c128", NE=400, Nk=16, Nb=12, mechanisms="acoustic",
             form="dense", terms=5, steps=5),
        # one point of a bias sweep over small structures, mixed precision, odd grid
        dict(name="scba_sweep_point", kind="scba", precision="mixed", NE=383, Nk=8, Nb=16,
             mechanisms="LO acoustic IFR", form="separable", terms=9, steps=5),
        # every mechanism, momentum-dependent kernels as dense operators: mixed bulk iterations ...
        dict(name="scba_dense_mixed", kind="scba", precision="mixed", NE=1024, Nk=32, Nb=16, mechanisms=ALL,
             form="dense", terms=5, steps=3),
        # ... and the FP64 iterations of the plain solve and of the refinement after promotion
        dict(name="scba_dense_fp64", kind="scba", precision="c128", NE=1024, Nk=32, Nb=16, mechanisms=ALL,
             form="dense", terms=5, steps=1),
        # the full-physics basis (32 states, separable kernels of 17 and 27 terms) on half its grid each way
        dict(name="scba_stack_mixed", kind="scba", precision="mixed", NE=1024, Nk=32, Nb=32, mechanisms=ALL,
             form="separable", terms=17, steps=1),
        # the reference's baseline grid and basis (2401 x 61, 5 states): G^R, G^<, G^> with scale and traces
        dict(name="dyson_baseline", kind="dyson", precision="c128", NE=2401, Nk=61, Nb=5, outputs="RLG"),
        # the operator batch of the benchmark: G^R and G^<
        dict(name="dyson_batch", kind="dyson", precision="c128", NE=4096, Nk=32, Nb=24, outputs="RL"),
        # the same solve inside a mixed iteration of the full-physics basis
        dict(name="dyson_mixed", kind="dyson", precision="mixed", NE=2048, Nk=32, Nb=32, outputs="RLG"),
        # the Hilbert transform of the benchmark's batch
        dict(name="hilbert_batch", kind="hilbert", precision="c128", NE=4096, ncols=18432, verify=False),
        # the residual suite of a mixed iteration, called by a host that owns the device memory
        dict(name="suite_mixed", kind="suite", precision="mixed", NE=1024, Nk=32, Nb=16),
        # the operator-level drop-in at the baseline grid: host arrays in and out
        dict(name="sigma_host", kind="sigma", precision="c128", NE=2401, ncols=61 * 25),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    while True:
        kind = rng.choice(["scba", "scba", "scba", "dyson", "dyson", "hilbert", "suite", "sigma"])
        precision = rng.choice(["c128", "c128", "mixed", "mixed", "c64"])
        if kind == "hilbert":
            case = dict(kind=kind, precision=rng.choice(["c128", "c64"]), NE=_log_int(rng, 100, 4096),
                        ncols=_log_int(rng, 50, 30000), verify=rng.random() < 0.5)
            size = case["NE"] * case["ncols"] / 80e6
        elif kind == "sigma":
            case = dict(kind=kind, precision=rng.choice(["c128", "c64"]), NE=_log_int(rng, 100, 4096),
                        ncols=_log_int(rng, 50, 4000))
            size = case["NE"] * case["ncols"] / 6e6
        else:
            case = dict(kind=kind, precision=precision, NE=_log_int(rng, 33, 4096), Nk=_log_int(rng, 2, 64),
                        Nb=_log_int(rng, 4, 48 if kind == "dyson" else 32))
            blocks, n = case["NE"] * case["Nk"], case["Nb"]
            if kind == "dyson":
                case["outputs"] = rng.choice(["RL", "RLG"])
                size = blocks * n ** 3 / 2e9
            elif kind == "suite":
                size = blocks * n ** 3 / 3e8
            else:
                case["mechanisms"] = rng.choice(["acoustic", "acoustic IFR", "LO acoustic IFR", ALL])
                case["form"] = rng.choice(["dense", "separable"])
                case["terms"] = rng.randint(3, 17)
                case["steps"] = rng.choice([1, 3])
                case["green"] = blocks * n * n < 60000
                k = case["steps"] * (2 if precision == "c128" else 0.5)
                size = max(k * blocks * n ** 3 / 6e8, _contraction_flops(case) * k / 3e12)
                if case["form"] == "dense" and case["Nk"] * n * n > 8192 and "LO" in case["mechanisms"]:
                    continue
        if size <= 1:
            return case


def _contraction_flops(case):
    """Real operations of one iteration's contractions, in the cheaper of each operator's forms."""
    NE, Nk, N = case["NE"], case["Nk"], case["Nb"]
    total = 0.0
    for name in case["mechanisms"].split():
        if name in ("acoustic", "alloy"):
            one = 8.0 * NE * N ** 4 + 4.0 * NE * Nk * N * N
        elif name == "IFR":
            one = 8.0 * NE * 3 * Nk * (2 * N * N + Nk)
        elif case["form"] == "dense":
            one = 8.0 * NE * (Nk * N * N) ** 2
        else:
            one = 8.0 * _terms(case, name) * NE * N * N * (Nk * Nk + Nk * N * N)
        total += 2 * one
    return total


def _terms(case, name):
    # the tabulated impurity covariance compresses to more terms than the LO kernel (27 against 17)
    return case["terms"] if name == "LO" else case["terms"] + case["terms"] * 10 // 17


def work(case):
    s = 16 if case["precision"] == "c128" else 8
    NE = case["NE"]
    L = 1 << (2 * NE - 2).bit_length()
    if case["kind"] in ("hilbert", "sigma"):
        n = NE * case["ncols"]
        fields = 2 if case["kind"] == "hilbert" else 4
        ffts = 4 if case.get("verify") else 2
        return dict(bytes=fields * s * n, flops=case["ncols"] * ffts * 5.0 * L * math.log2(L))
    blocks, N = NE * case["Nk"], case["Nb"]
    field = blocks * N * N * s
    if case["kind"] == "dyson":
        g = len(case["outputs"]) - 1
        return dict(bytes=(2 + 2 * g) * field, flops=blocks * N ** 3 * (8.0 + 16.0 * g))
    if case["kind"] == "suite":
        return dict(bytes=7 * field, flops=blocks * N ** 3 * 9 * 8.0)
    families = len(case["mechanisms"].split()) + 2
    per_step = blocks * N ** 3 * (8.0 + 2 * 16.0 + 9 * 8.0 + 6 * 16.0) + _contraction_flops(case)
    per_step += (families - 2) * case["Nk"] * N * N * 4 * 5.0 * L * math.log2(L)
    return dict(bytes=case["steps"] * 6 * families * field, flops=case["steps"] * per_step)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _cdtype(case):
    return torch.complex128 if case["precision"] == "c128" else torch.complex64


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _to_field(blocks, NE, Nk, dtype):
    """(Nk NE, N, N) blocks -> the E-fastest field, as a (N_b, N_a, Nk, NE) tensor."""
    N = blocks.shape[-1]
    return blocks.reshape(Nk, NE, N, N).permute(3, 2, 0, 1).to(dtype).contiguous()


def _to_blocks(field):
    """The E-fastest field as (Nk NE, N, N) complex128 blocks."""
    N = field.shape[0]
    return field.permute(2, 3, 1, 0).reshape(-1, N, N).to(torch.complex128)


def _positive(g, NE, Nk, N, scale, dtype):
    """A field of positive semidefinite blocks X X^H scale / N, a few momenta at a time."""
    out = torch.empty((N, N, Nk, NE), dtype=dtype, device="cuda")
    some = max(1, (1 << 23) // (NE * N * N))
    for m in range(0, Nk, some):
        n = min(some, Nk - m)
        X = torch.randn((n * NE, N, N), dtype=torch.complex128, device="cuda", generator=g)
        out[:, :, m:m + n] = _to_field((X @ X.mH) * (scale / N), NE, n, dtype)
    return out


def _hamiltonian(seed, N, Nk):
    """Hermitian blocks h[k]: subbands over 250 meV, couplings of 2 meV between neighbouring periods of 8
    states, parabolic dispersion (units of 0.1 eV)."""
    rng = np.random.default_rng(seed)
    h0 = np.diag(rng.uniform(0.0, 2.5, N)).astype(complex)
    x = 0.02 * (rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))) / math.sqrt(2)
    near = np.abs(np.arange(N)[:, None] // 8 - np.arange(N)[None, :] // 8) == 1
    x = np.triu(x, 1) * near
    kappa = np.linspace(0.0, 1.2, Nk)
    return np.asfortranarray(h0 + x + x.conj().T + 0.57 * kappa[:, None, None] ** 2 * np.eye(N))


def _device_h(h):
    return torch.from_numpy(h.ravel(order="F").copy()).cuda()


def _structure(case, seed):
    """Grids, Hamiltonian, couplings and kernel factors of a synthetic structure (solver units)."""
    rng = np.random.default_rng(seed)
    NE, Nk, N = case["NE"], case["Nk"], case["Nb"]
    eps, wE = energy_grid(-1.0, 2.0, NE)
    kappa, wk = momentum_grid(2.0, Nk)
    c = np.triu(0.05 * (rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))), 1)
    h0 = np.diag(np.linspace(-0.3, 1.2, N)) + c + c.conj().T
    h = h0 + 0.06 * kappa[:, None, None] ** 2 * np.eye(N)
    T = 0.05 * (rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N)))
    x = (np.arange(48) + 0.5) / 24.0
    centre = np.linspace(0.2, 1.8, N) + 0.02 * rng.standard_normal(N)
    width = 0.24 / max(N / 4, 1) * (1 + 0.2 * rng.random(N))
    chi = np.exp(-0.5 * ((x[:, None] - centre) / np.maximum(width, 0.06)) ** 2)
    chi /= np.sqrt((chi ** 2).sum(axis=0) / 24.0)
    strength = 0.05 * min(1.0, 16.0 / N)
    kernels = {}
    for name in case["mechanisms"].split():
        if name in ("acoustic", "alloy"):
            # K[a,c,d,b] = sum_x w chi_a chi_c chi_d chi_b
            w = rng.uniform(0.5, 1.5, 48) / 24.0
            kernels[name] = dict(chi=chi, w=w / max((w[:, None] * chi ** 4).sum(axis=0)),
                                 q=strength * (1.3 if name == "alloy" else 1.0))
        elif name == "IFR":
            v = (rng.standard_normal((N, 3)) + 0.3j * rng.standard_normal((N, 3))) / math.sqrt(6)
            radial = np.exp(-0.5 * (kappa[:, None] - kappa[None, :]) ** 2)
            kernels[name] = dict(v=v, radial=radial, q=strength * 0.6)
        else:
            # K(m,m') = sum_t R_t(m,m') F_t (x) conj F_t: form factors and screened couplings
            n = _terms(case, name) if case["form"] == "separable" else case["terms"]
            F = rng.standard_normal((n, N, N)) + 1j * rng.standard_normal((n, N, N))
            F = 0.5 * (F + F.conj().transpose(0, 2, 1))
            F /= np.sqrt((np.abs(F) ** 2).sum(axis=0)).max()
            d2 = (kappa[:, None] - kappa[None, :]) ** 2
            R = np.stack([1.0 / (1.0 + d2 + t) for t in range(n)])
            kernels[name] = dict(F=F, R=R, q=strength * (0.8 if name == "LO" else 0.5))
    return dict(eps=eps, wE=wE, wk=wk, h=h, T=T, kernels=kernels, Ep=0.3, hw=0.367, N_LO=0.25, gs=2, target=0.05,
                kBT=0.2, eta=0.02, alpha=0.3)


def _mechanism(name, k, form):
    if "chi" in k:
        pair = torch.from_numpy(np.einsum("ga,gc->gac", k["chi"], k["chi"])).cuda()
        w = torch.from_numpy(k["w"]).cuda()
        N = k["chi"].shape[1]
        # block[(a,b),(c,d)], first index fastest
        block = torch.einsum("gac,gdb->dcba", w[:, None, None] * pair, pair).reshape(N * N, N * N)
        return Mechanism(name, "momentum_independent", k["q"], block=block.to(torch.complex128).contiguous())
    if "v" in k:
        v = k["v"]
        N, J = v.shape
        left = np.einsum("aj,bj->baj", v, v.conj()).reshape(N * N, J)
        return Mechanism(name, "ifr", k["q"], left=np.asfortranarray(left), right=np.asfortranarray(left.conj().T),
                         radial=np.asfortranarray(k["radial"].astype(complex)))
    F, R = torch.from_numpy(k["F"]).cuda(), torch.from_numpy(k["R"]).cuda()
    n, N = F.shape[0], F.shape[1]
    if form == "separable":
        block = torch.einsum("tac,tbd->tdcba", F, F.conj()).reshape(n, N * N, N * N).contiguous()
        return Mechanism(name, "separable_sum", k["q"], block=block,
                         radial=np.asfortranarray(np.transpose(k["R"], (1, 2, 0)).astype(complex)))
    Nk = R.shape[1]
    # matrix[(m,a,b),(m',c,d)], first index fastest
    left = torch.einsum("tac,tbd->tdcba", F, F.conj()).reshape(n, -1)
    matrix = (left.T @ R.to(torch.complex128).reshape(n, -1)).reshape(N, N, N, N, Nk, Nk)  # d c b a m m'
    return Mechanism(name, "dense", k["q"], matrix=matrix.permute(0, 1, 5, 2, 3, 4).contiguous())


def prepare(case, seed):
    kind = case["kind"]
    if kind == "scba":
        st = _structure(case, seed)
        T = np.asfortranarray(st["T"])
        problem = SCBAProblem(
            NE=case["NE"], Nk=case["Nk"], Nb=case["Nb"], eps=st["eps"], wE=st["wE"], wk=st["wk"],
            h=np.asfortranarray(st["h"]), Tplus=T, Tminus=np.asfortranarray(T.conj().T), Ep=st["Ep"],
            hw_LO=st["hw"], N_LO=st["N_LO"], gs=st["gs"], target=st["target"], kBT=st["kBT"], eta_seed=st["eta"],
            alpha=st["alpha"], mechanisms=[_mechanism(n, k, case["form"]) for n, k in st["kernels"].items()])
        torch.cuda.synchronize()  # the operators are read on the context's own stream
        torch.cuda.empty_cache()
        solver = ProductionSCBA(problem, precision=case["precision"], use_graph=True)
        solver.seed()
        return dict(case=case, solver=solver)
    if kind in ("hilbert", "sigma"):
        eps, wE = energy_grid(-0.5, 3.5, case["NE"])
        g = _generator(seed)
        shape = (case["ncols"], case["NE"])
        # broadened lines over a smooth background, per column
        e = torch.linspace(-0.5, 3.5, case["NE"], dtype=torch.float64, device="cuda")
        cols = []
        for _ in range(1 if kind == "hilbert" else 2):
            a, c = (torch.randn((case["ncols"], 1), dtype=torch.complex128, device="cuda", generator=g) for _ in "ac")
            x0 = 3 * torch.rand((case["ncols"], 1), dtype=torch.float64, device="cuda", generator=g)
            y = a / (1 + ((e - x0) / 0.05) ** 2) + 0.1 * c * torch.cos(e)
            y += 0.01 * torch.randn(shape, dtype=torch.complex128, device="cuda", generator=g)
            cols.append(y.to(_cdtype(case)))
        if kind == "sigma":
            host = [np.asfortranarray(y.cpu().numpy().T) for y in cols]
            return dict(case=case, eps=eps, wE=wE, SL=host[0], SG=host[1])
        return dict(case=case, de=float(eps[1] - eps[0]), wE=torch.from_numpy(wE).cuda(), Gam=cols[0],
                    Lam=torch.empty_like(cols[0]), sums=torch.zeros(2, dtype=torch.float64, device="cuda"))
    NE, Nk, N, dtype = case["NE"], case["Nk"], case["Nb"], _cdtype(case)
    g = _generator(seed)
    h = _hamiltonian(seed, N, Nk)
    eps = torch.linspace(-0.5, 3.5, NE, dtype=torch.float64, device="cuda")
    SL = _positive(g, NE, Nk, N, 0.005, dtype).mul_(1j)
    SG = _positive(g, NE, Nk, N, 0.015, dtype).mul_(-1j)
    SR = 0.5 * (SG - SL)
    state = dict(case=case, eps=eps, h=_device_h(h), SR=SR, SL=SL, SG=SG)
    if kind == "dyson":
        state.update(GR=torch.empty_like(SL), GL=torch.empty_like(SL),
                     status=torch.zeros(2, dtype=torch.int32, device="cuda"))
        if case["outputs"] == "RLG":
            state.update(GG=torch.empty_like(SL), scale=torch.empty((Nk, NE), dtype=torch.float64, device="cuda"),
                         trL=torch.empty((Nk, NE), dtype=torch.complex128, device="cuda"),
                         trG=torch.empty((Nk, NE), dtype=torch.complex128, device="cuda"))
        else:
            del state["SG"]
        return state
    # an iteration's state: G of the totals, and a candidate lesser total some per cent off
    for name in ("GR", "GL", "GG"):
        state[name] = torch.empty_like(SL)
    some = max(1, (1 << 23) // (NE * N * N))
    hk = torch.from_numpy(np.ascontiguousarray(h)).cuda()
    for m in range(0, Nk, some):
        n = min(some, Nk - m)
        at = slice(m, m + n)
        GR = torch.linalg.inv(_blocks_of_D(eps, hk[at], _to_blocks(SR[:, :, at])))
        state["GR"][:, :, at] = _to_field(GR, NE, n, dtype)
        for out, S in (("GL", SL), ("GG", SG)):
            state[out][:, :, at] = _to_field(GR @ _to_blocks(S[:, :, at]) @ GR.mH, NE, n, dtype)
    state["SLc"] = SL + _positive(g, NE, Nk, N, 0.0005, dtype).mul_(1j)
    state["out"] = torch.zeros(5, dtype=torch.float64, device="cuda")
    return state


def _blocks_of_D(eps, h, SR):
    """eps - h - Sigma^R as (Nk NE, N, N) blocks, energy fastest."""
    N = h.shape[-1]
    D = eps[None, :, None, None] * torch.eye(N, dtype=torch.complex128, device=h.device) - h[:, None]
    return D.reshape(-1, N, N) - SR


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _p(t):
    return None if t is None else PTR(t.data_ptr())


def _stream():
    return PTR(torch.cuda.current_stream().cuda_stream)


def run(state):
    case = state["case"]
    kind, code = case["kind"], _lib.PRECISIONS[case["precision"]]
    s = state
    if kind == "dyson":
        _lib.check(_lib.lib().qcl_dev_dyson_keldysh(
            _stream(), code, case["NE"], case["Nk"], case["Nb"], _p(s["eps"]), 0.0, _p(s["h"]), _p(s["SR"]),
            _p(s["SL"]), _p(s.get("SG")), _p(s["GR"]), _p(s["GL"]), _p(s.get("GG")), _p(s.get("scale")),
            _p(s.get("trL")), _p(s.get("trG")), _p(s["status"])))
        return {k: s[k] for k in ("GR", "GL", "GG", "scale", "trL", "trG", "status") if k in s}
    if kind == "hilbert":
        _lib.check(_lib.lib().qcl_dev_fft_hilbert_transform(
            _stream(), code, case["NE"], case["ncols"], s["de"], _p(s["wE"]), _p(s["Gam"]), _p(s["Lam"]),
            _p(s["sums"]) if case["verify"] else None))
        return dict(Lam=s["Lam"], sums=s["sums"]) if case["verify"] else dict(Lam=s["Lam"])
    if kind == "sigma":
        return operators.retarded_self_energy_fft(s["SL"], s["SG"], s["eps"], s["wE"], precision=case["precision"])
    if kind == "suite":
        _lib.check(_lib.lib().qcl_dev_residual_suite_noalloc(
            _stream(), code, case["NE"], case["Nk"], case["Nb"], _p(s["eps"]), _p(s["h"]), _p(s["GR"]), _p(s["GL"]),
            _p(s["GG"]), _p(s["SR"]), _p(s["SL"]), _p(s["SG"]), _p(s["SLc"]), _p(s["out"])))
        return dict(out=s["out"])
    rows = s["solver"].run(case["steps"])
    # rows of a reduced-precision context are sums over complex64 fields: their type here is that of the fields
    real, cplx = (np.float64, np.complex128) if case["precision"] == "c128" else (np.float32, np.complex64)
    out = {k: np.array([r[k] for r in rows], real)
           for k in ("J", "lam", "number", "holes", "normalized_charge", "r_Sigma", "populations")}
    # the defects of the solve itself lie at roundoff: with r_K in one array, as a row holds them
    out["residuals"] = np.array([[r[k] for k in ("r_K", "r_D", "r_A", "r_PSD", "r_caus")] for r in rows], real)
    out["status"] = np.array([r["status"] for r in rows], np.int64)
    out["density_matrix"] = s["solver"].density_matrix().astype(cplx)
    if case.get("green"):
        out.update(s["solver"].green())
    return out


# ---------------------------------------------------------------------------
# the same in 64-bit torch
# ---------------------------------------------------------------------------
def _hilbert(x, wE, de):
    """Principal-value transform of x[..., e] by one zero-padded FFT convolution."""
    NE = x.shape[-1]
    L = 1 << (2 * NE - 2).bit_length()
    lag = torch.arange(L, dtype=torch.float64, device=x.device)
    lag = torch.where(lag < NE, lag, lag - L)
    k = torch.where((lag == 0) | (lag.abs() >= NE), torch.zeros_like(lag), 1 / (2 * math.pi * de * lag))
    kf = torch.fft.fft(k.to(torch.complex128))
    return torch.fft.ifft(torch.fft.fft(x * wE, n=L) * kf)[..., :NE]


def _exact_dyson(case, s):
    NE, Nk = case["NE"], case["Nk"]
    N = case["Nb"]
    h = s["h"].reshape(N, N, Nk).permute(2, 1, 0)
    D = _blocks_of_D(s["eps"], h, _to_blocks(s["SR"]))
    out = {}
    if "scale" in s:
        out["scale"] = D.abs().sum(dim=2).amax(dim=1).reshape(Nk, NE)
    GR = torch.linalg.inv(D)
    out["GR"] = _to_field(GR, NE, Nk, torch.complex128)
    for S, G, tr in (("SL", "GL", "trL"), ("SG", "GG", "trG")):
        if S in s:
            X = GR @ _to_blocks(s[S]) @ GR.mH
            out[G] = _to_field(X, NE, Nk, torch.complex128)
            if tr in s:
                out[tr] = X.diagonal(dim1=1, dim2=2).sum(dim=1).reshape(Nk, NE)
    return out


def _exact_suite(case, s):
    NE, Nk, N = case["NE"], case["Nk"], case["Nb"]
    h = s["h"].reshape(N, N, Nk).permute(2, 1, 0)
    GR, GL, GG, SR, SL, SG, SLc = (_to_blocks(s[k]) for k in ("GR", "GL", "GG", "SR", "SL", "SG", "SLc"))
    D = _blocks_of_D(s["eps"], h, SR)

    def fro(x):
        return torch.linalg.matrix_norm(x)

    def eigvals(x):  # some blocks at a time: the batched solver takes a limited number
        return torch.cat([torch.linalg.eigvalsh(y) for y in x.split(4096)])

    def positive(x):
        v = eigvals(0.5 * (x + x.mH))
        top = v.abs().amax(dim=1)
        floor = 64 * N * 2.220446049250313e-16 * top.clamp(min=1.0)
        return ((-v[:, 0] - floor).clamp(min=0) / top.clamp(min=1e-300)).max()

    rD = (fro(D @ GR - torch.eye(N, device=D.device)) / (fro(D) * fro(GR) + math.sqrt(N))).max()
    A, Gam = 1j * (GR - GR.mH), 1j * (SG - SL)
    rA = (A - GR @ Gam @ GR.mH).norm() / A.norm()
    rK = (GL - GR @ SLc @ GR.mH).norm() / GL.norm()
    rPSD = max(positive(x) for x in (A, -1j * GL, 1j * GG, Gam, -1j * (GR @ SL @ GR.mH), 1j * (GR @ SG @ GR.mH)))
    top = eigvals((SR - SR.mH) / 2j)[:, -1].clamp(min=0)
    rcaus = (top / (eigvals(SR @ SR.mH)[:, -1].sqrt() + 1e-14)).max()
    return dict(out=torch.stack([rD, rA, rK, rPSD, rcaus]))


def _exact_scba(case, seed):
    """The seed and `steps` iterations, on (Nk, NE, N, N) fields."""
    st = _structure(case, seed)
    NE, Nk, N = case["NE"], case["Nk"], case["Nb"]
    dev = {k: torch.from_numpy(np.ascontiguousarray(st[k])).cuda() for k in ("eps", "wE", "wk", "h", "T")}
    eps, wE, wk = dev["eps"], dev["wE"], dev["wk"]
    de = float(st["eps"][1] - st["eps"][0])
    eye = torch.eye(N, dtype=torch.complex128, device="cuda")
    D0 = eps[None, :, None, None] * eye - dev["h"][:, None]
    weights = (wk[:, None] * wE[None, :])[..., None, None]

    def number(G):
        return (-0.5j * st["gs"] / math.pi * (weights * G).diagonal(dim1=2, dim2=3).sum()).real.item()

    def shifted(X, delta):
        at = (eps + delta - eps[0]) / de
        ok = (eps + delta >= eps[0]) & (eps + delta <= eps[-1])
        left = at.floor().clamp(0, NE - 2).long()
        left = torch.where((left > 0) & (eps[left] > eps + delta), left - 1, left)
        th = ((eps + delta - eps[left]) / (eps[left + 1] - eps[left]))[None, :, None, None]
        return ok[None, :, None, None] * ((1 - th) * X[:, left] + th * X[:, left + 1])

    ops = {n: {k: torch.from_numpy(np.asarray(v)).cuda().to(torch.complex128) if isinstance(v, np.ndarray) else v
               for k, v in kernel.items()} for n, kernel in st["kernels"].items()}

    def mixed_over_k(R, X):
        return (R @ (wk[:, None] * X.reshape(Nk, -1))).reshape(X.shape)

    def contract(k, G):
        if "chi" in k:
            X = (wk[:, None, None, None] * G).sum(dim=0)
            x = torch.einsum("gc,ecd,gd->eg", k["chi"], X, k["chi"])
            S = torch.einsum("eg,ga,gb->eab", x * k["w"], k["chi"], k["chi"])
            return k["q"] * S[None].expand(Nk, NE, N, N)
        if "v" in k:
            x = torch.einsum("cj,mecd,dj->mej", k["v"].conj(), G, k["v"])
            return k["q"] * torch.einsum("mej,aj,bj->meab", mixed_over_k(k["radial"], x), k["v"], k["v"].conj())
        S = torch.zeros_like(G)
        for t in range(k["F"].shape[0]):
            S += k["F"][t] @ mixed_over_k(k["R"][t], G) @ k["F"][t].mH
        return S.mul_(k["q"])

    def candidates(GR, GL, GG):
        fam = []
        for name, k in ops.items():
            if name == "LO":
                n = st["N_LO"]
                SL = contract(k, (n + 1) * shifted(GL, st["hw"]) + n * shifted(GL, -st["hw"]))
                SG = contract(k, (n + 1) * shifted(GG, -st["hw"]) + n * shifted(GG, st["hw"]))
            else:
                SL, SG = contract(k, GL), contract(k, GG)
            Gam = 1j * (SG - SL)
            SR = torch.empty_like(Gam)
            for m in range(Nk):
                x = Gam[m].permute(1, 2, 0)
                SR[m] = _hilbert(x, wE, de).permute(2, 0, 1) - 0.5j * Gam[m]
            fam.append([SR, SL, SG])
        for T, d in ((dev["T"], st["Ep"]), (dev["T"].mH, -st["Ep"])):
            fam.append([T @ shifted(X, d) @ T.mH for X in (GR, GL, GG)])
        return fam

    # equilibrium seed: G^< = -f (G^R - G^A) with the Fermi level that gives the target number
    GR = torch.linalg.inv(D0 + 1j * st["eta"] * eye)
    diff = GR - GR.mH
    q = (0.5 * st["gs"] / math.pi * wE * (wk[:, None] * (1j * diff).diagonal(dim1=2, dim2=3).sum(2).real).sum(0))
    q, e = q.cpu().numpy(), st["eps"]

    def fermi(mu):
        x = (e - mu) / st["kBT"]
        return np.where(x > 40, 0.0, np.where(x < -40, 1.0, 1 / (np.exp(np.clip(x, -40, 40)) + 1)))

    lo, hi = e[0] - 50 * st["kBT"], e[-1] + 50 * st["kBT"]
    while True:
        mid = 0.5 * (lo + hi)
        if mid in (lo, hi):
            break
        lo, hi = (mid, hi) if (q * fermi(mid)).sum() < st["target"] else (lo, mid)
    f = torch.from_numpy(fermi(lo)).cuda()[None, :, None, None]
    fam = candidates(GR, -f * diff, (1 - f) * diff)

    rows = {k: [] for k in ("J", "lam", "number", "holes", "normalized_charge", "r_Sigma", "populations")}

    def change(old, new):
        return ((new - old).norm() / (new.norm() + 1e-14)).item()

    for _ in range(case["steps"]):
        tot = [sum(x[c] for x in fam) for c in range(3)]
        GR = torch.linalg.inv(D0 - tot[0])
        GL, GG = GR @ tot[1] @ GR.mH, GR @ tot[2] @ GR.mH
        n, holes, target = number(GL), -number(GG), st["target"]
        a, c = (target / n, 0.0) if n >= target else (1.0, (target - n) / holes)
        GL, GG = a * GL - c * GG, (1 - c) * GG - (1 - a) * GL
        cand = candidates(GR, GL, GG)
        flux = (fam[-2][2] @ GL - fam[-2][1] @ GG).diagonal(dim1=2, dim2=3)
        J = (0.5 * st["gs"] / math.pi * (weights[..., 0] * flux).sum()).real.item() * SCBAProblem.J0
        pairs = [(x[c], y[c]) for x, y in zip(fam, cand) for c in range(3)]
        pairs += [(fam[-2][c] + fam[-1][c], cand[-2][c] + cand[-1][c]) for c in range(3)]
        rows["J"].append(J)
        rows["lam"].append(n / target)
        rows["number"].append(n)
        rows["holes"].append(holes)
        rows["normalized_charge"].append(a * n + c * holes)
        rows["r_Sigma"].append(max(change(*p) for p in pairs))
        del pairs
        diag = (-0.5j * st["gs"] / math.pi * (weights * GL).diagonal(dim1=2, dim2=3)).sum(dim=(0, 1)).real / target
        rows["populations"].append(diag.cpu().numpy())
        for x, y in zip(fam, cand):
            for c in range(3):
                x[c] = (1 - st["alpha"]) * x[c] + st["alpha"] * y[c]
    out = {k: np.array(v, np.float64) for k, v in rows.items()}
    out["residuals"] = None
    out["density_matrix"] = (weights * GL).sum(dim=(0, 1)).cpu().numpy()
    if case.get("green"):
        out.update({k: X.transpose(0, 1).cpu().numpy() for k, X in (("GR", GR), ("GL", GL), ("GG", GG))})
    return out


def exact(case, seed):
    if case["kind"] == "scba":
        return _exact_scba(case, seed)
    s = prepare(case, seed)
    if case["kind"] == "dyson":
        return _exact_dyson(case, s)
    if case["kind"] == "suite":
        return _exact_suite(case, s)
    if case["kind"] == "hilbert":
        return dict(Lam=_hilbert(s["Gam"].to(torch.complex128), s["wE"], s["de"]))
    SL, SG = (torch.from_numpy(np.ascontiguousarray(s[k].T)).cuda().to(torch.complex128) for k in ("SL", "SG"))
    Gam = 1j * (SG - SL)
    SR = _hilbert(Gam, torch.from_numpy(s["wE"]).cuda(), float(s["eps"][1] - s["eps"][0])) - 0.5j * Gam
    return SR.T.contiguous(), Gam.T.contiguous()
