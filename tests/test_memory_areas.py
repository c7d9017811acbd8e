"""The optional work area of a complex128 context (the digits of the integer
tensor path): whatever a budget leaves over, a context that the estimate
admits runs."""
import pytest

pytestmark = pytest.mark.gpu


def _problem(NE, Nk, Nb, mechanisms=("impurity",)):
    from qclb200.problem import small_problem

    return small_problem(NE=NE, Nk=Nk, Nb=Nb, mechanisms=mechanisms)


@pytest.mark.parametrize("NE,Nk,Nb", [(400, 8, 16), (1024, 4, 16)])
def test_any_budget_above_the_estimate_runs(gpu_ops, NE, Nk, Nb):
    """From nothing left over to room for all the digits (24 bytes per entry of
    the operator and of both fields), in steps of a sixteenth."""
    from qclb200.scba import ProductionSCBA, estimate_memory

    pr = _problem(NE, Nk, Nb)
    nc = Nk * Nb * Nb
    assert 2 * NE * nc * nc >= 1e9  # the size that the integer path is for
    peak = estimate_memory(pr)["peak"]
    digits = 25 * nc * (nc + 2 * NE + 512)
    rows = []
    for i in range(0, 17):
        s = ProductionSCBA(pr, memory_budget_bytes=peak + digits * i // 16)
        s.seed()
        rows.append(s.step())
        s.close()
    for r in rows:
        assert r["status"] == 0
        assert abs(r["J"] - rows[0]["J"]) <= 1e-9 * abs(rows[0]["J"])
