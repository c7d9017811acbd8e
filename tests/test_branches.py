"""Candidates built on several streams: the same rows as one mechanism after
another (phase telemetry keeps one stream), with and without graphs, for
every number of mechanisms, and with contexts opened and closed in turn (the
streams of closed contexts are used again)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("J", "lam", "number", "holes", "r_Sigma", "r_K", "r_roundoff")


@pytest.mark.parametrize("mechanisms", [(), ("acoustic",), ("LO", "acoustic", "IFR"),
                                        ("LO", "acoustic", "impurity", "IFR", "alloy")])
@pytest.mark.parametrize("use_graph", [False, True])
@pytest.mark.parametrize("precision", ["c128", "mixed"])
def test_branches_leave_rows_unchanged(gpu_ops, mechanisms, use_graph, precision):
    from qclb200.problem import small_problem
    from qclb200.scba import ProductionSCBA

    pr = small_problem(NE=41, Nk=3, Nb=4, mechanisms=mechanisms)
    rows = []
    for telemetry in (True, False, False):
        s = ProductionSCBA(pr, precision=precision, use_graph=use_graph, telemetry=telemetry)
        s.seed()
        rows.append(s.run(5))
        s.close()
    for other in rows[1:]:
        for a, b in zip(rows[0], other):
            assert [a[k] for k in KEYS] == [b[k] for k in KEYS]
            assert np.array_equal(a["populations"], b["populations"])


def test_contexts_interleaved(gpu_ops):
    """Two contexts stepped in turn while others open and close."""
    from qclb200.problem import small_problem
    from qclb200.scba import ProductionSCBA

    pr = small_problem(NE=41, Nk=3, Nb=4, mechanisms=("LO", "acoustic", "IFR"))
    a, b = (ProductionSCBA(pr, use_graph=True) for _ in range(2))
    a.seed()
    b.seed()
    ja, jb = [], []
    for _ in range(6):
        ja.append(a.step()["J"])
        c = ProductionSCBA(pr)
        c.seed()
        c.step()
        c.close()
        jb.append(b.step()["J"])
    a.close()
    b.close()
    assert ja == jb
