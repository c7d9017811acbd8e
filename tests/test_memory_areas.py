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


def test_area_without_a_budget_is_bounded(gpu_ops):
    """An operator of 10 240 rows, whose digits take 2.6 GB: without a budget the
    context keeps at most 2 GiB (and the allocator's 2 MB pages) beyond its
    estimate."""
    import dataclasses

    import numpy as np
    import torch
    from qclb200.scba import ProductionSCBA, estimate_memory

    pr = _problem(192, 2, 16)
    Nk = 40
    nc = Nk * 16 * 16
    pr = dataclasses.replace(
        pr, Nk=Nk, wk=np.full(Nk, 0.1), h=np.asfortranarray(np.repeat(pr.h[:1], Nk, axis=0)),
        mechanisms=[dataclasses.replace(pr.mechanisms[0], matrix=np.asfortranarray(np.eye(nc, dtype=complex)))])
    ProductionSCBA(_problem(33, 2, 4)).close()  # the library's own memory
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    s = ProductionSCBA(pr)
    used = before - torch.cuda.mem_get_info()[0]
    s.close()
    assert used < estimate_memory(pr)["resident"] + (2 << 30) + (128 << 20)
