"""The residual suite with one row per lane (N_b <= 32) at the edges of its
padded sizes, against the oracle: a defect of each kind planted in a block of
its own, so that every test that has no certificate goes through the
tridiagonal path, the state without them, and a non-finite block.  Tolerances as in
the other residual-suite tests (1e-10 relative)."""
import math

import numpy as np
import pytest

from helpers import dyson_inputs

pytestmark = pytest.mark.gpu


def _state(orc, seed, NE, Nk, N):
    eps, h, SR, SL, SG = dyson_inputs(seed, NE, Nk, N)
    GR = orc.retarded_green(eps, h, SR)[0]
    return eps, h, GR, orc.keldysh_green(GR, SL), orc.keldysh_green(GR, SG), SR, SL, SG


def _compare(gpu_ops, orc, args, cand):
    ref = orc.residual_suite(*args, cand)
    got = gpu_ops.production_residual_suite(*args, cand)
    for k in ("rK", "rPSD", "rcaus"):
        assert got[k] == pytest.approx(ref[k], rel=1e-10, abs=1e-14), k
    for k in ("rD", "rA"):  # roundoff unless planted
        assert got[k] == pytest.approx(ref[k], rel=1e-10, abs=1e-14), k
    return ref, got


@pytest.mark.parametrize("N", [1, 2, 7, 8, 9, 15, 16, 17, 24, 25, 32, 33])
def test_planted_defects_match_oracle(gpu_ops, orc, N):
    NE, Nk = 11, 2
    eps, h, GR, GL, GG, SR, SL, SG = _state(orc, 40 + N, NE, Nk, N)
    rng = np.random.default_rng(N)
    cand = np.asfortranarray(SL * (1 + 0.05 * rng.standard_normal(SL.shape)))
    _compare(gpu_ops, orc, (eps, h, GR, GL, GG, (SR, SL, SG)), cand)
    last = N - 1

    def planted(X, e, m, value):
        Y = np.array(X, order="F")
        Y[e, m, last, last] += value
        return Y

    top = {k: float(np.abs(v).max()) for k, v in dict(GR=GR, GL=GL, GG=GG, SL=SL, SG=SG, SR=SR).items()}
    cases = {
        "occupied": (eps, h, GR, planted(GL, 5, 0, 2j * top["GL"]), GG, (SR, SL, SG)),
        "unoccupied": (eps, h, GR, GL, planted(GG, 6, 1, -2j * top["GG"]), (SR, SL, SG)),
        "spectral": (eps, h, planted(GR, 4, 0, 2j * top["GR"]), GL, GG, (SR, SL, SG)),
        # Sigma< and Sigma>: the broadening and both raw products
        "raw_occupied": (eps, h, GR, GL, GG, (SR, planted(SL, 2, 1, -3j * top["SL"]), SG)),
        "raw_unoccupied": (eps, h, GR, GL, GG, (SR, SL, planted(SG, 9, 0, 3j * top["SG"]))),
    }
    for name, args in cases.items():
        ref, _ = _compare(gpu_ops, orc, args, cand)
        assert ref["rPSD"] > 1e-6, name
    acausal = planted(SR, 3, 1, 3j * top["SR"])
    ref, _ = _compare(gpu_ops, orc, (eps, h, GR, GL, GG, (acausal, SL, SG)), cand)
    assert ref["rcaus"] > 1e-6


@pytest.mark.parametrize("N", [5, 16, 32])
def test_non_finite_block_is_reported(gpu_ops, orc, N):
    eps, h, GR, GL, GG, SR, SL, SG = _state(orc, 7, 9, 2, N)
    GL[4, 1, N - 1, 0] = np.nan
    got = gpu_ops.production_residual_suite(eps, h, GR, GL, GG, (SR, SL, SG), SL)
    assert got["rPSD"] == math.inf and got["rK"] == math.inf and got["rcaus"] == 0
