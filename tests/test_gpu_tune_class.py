"""A tuned launch form is for the class of case it was timed on: a case whose
pressure is solved elsewhere (in the program, where the tuned one was a kernel of
its own), with other solvers, or over another numbering keeps its own form, also
on a context that held the tuned case before."""
import pytest

import xcal as X
from xcal import _abi, cases

pytestmark = pytest.mark.gpu

LAUNCH = ("mode", "ctas", "ctas_per_sm")


def _form(s, made):
    case, keep = X.make_case(made[1], made[2], made[3])
    s.setup(case)
    s.run(1)
    f = s.last_form()
    return tuple(f[k] for k in LAUNCH)


def _fresh(made, renumber=_abi.RENUMBER_COLOR):
    s = X.Solver(made[0], renumber=renumber)
    try:
        return _form(s, made)
    finally:
        s.close()


@pytest.mark.parametrize("make", [lambda **kw: cases.cavity2d(41, **kw), lambda **kw: cases.cavity2d(83, **kw),
                                  lambda **kw: cases.bfs(8, **kw), lambda **kw: cases.cavity2d(230, **kw)],
                         ids=["7-tiles", "27-tiles", "bfs", "207-tiles"])
def test_tuned_form_stays_in_its_class(make):
    tuned_case = make()
    others = {"BiCGSTAB for p": make(p_solver=X.BicgstabSolver), "GMRES for U": make(u_solver=X.GmresSolver),
              "Jacobi": make(precon=X.Jacobi)}
    default = {k: _fresh(m) for k, m in others.items()}
    none = _fresh(tuned_case, _abi.RENUMBER_NONE)
    s = X.Solver(tuned_case[0])
    try:
        case, keep = X.make_case(tuned_case[1], tuned_case[2], tuned_case[3])
        s.setup(case)
        r = s.autotune(iterations=3)
        choice = tuple(r[k] for k in LAUNCH)
        assert _form(s, others["BiCGSTAB for p"]) == default["BiCGSTAB for p"]
        assert _form(s, tuned_case) == choice
    finally:
        s.close()
    assert _fresh(tuned_case) == choice
    for k, m in others.items():
        assert _fresh(m) == default[k], k
    assert _fresh(tuned_case, _abi.RENUMBER_NONE) == none
