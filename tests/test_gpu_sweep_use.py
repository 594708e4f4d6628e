"""Sweeps by one CTA are set up for what will sweep: runs of a narrow numbering
whose preconditioners have no levels take the build without them and reserve no
shared memory for a vector, ILU(0) sweeps in global memory and reserves none,
and DILU reserves the largest of its vectors that fits (98,304 bytes).  The
values are the oracle's in every case."""
import pytest

import xcal as X
from xcal import _abi, cases
from parity_util import assert_parity, run_oracle

pytestmark = pytest.mark.gpu


def _solver(model, which, precon):
    return X.set_solver(getattr(model, which), solver=X.BicgstabSolver if which == "U" else X.CgSolver,
                        preconditioner=precon(), convergence=1e-7, relax=0.7 if which == "U" else 0.3, itmax=100)


@pytest.mark.parametrize("geom,n,U,p,sweeps,shared", [
    ("quad", 33, X.Jacobi, X.Jacobi, False, 0), ("quad", 33, X.NormDiagonal, X.Jacobi, False, 0),
    ("quad", 33, X.ILU0, X.ILU0, True, 0), ("quad", 33, X.DILU, X.DILU, True, 33 * 33 * 2 * 8),
    ("quad", 33, X.Jacobi, X.DILU, True, 33 * 33 * 8), ("quad", 33, X.DILU, X.ILU0, True, 33 * 33 * 2 * 8),
    ("quad", 80, X.DILU, X.DILU, True, 80 * 80 * 8), ("hex", 16, X.DILU, X.DILU, False, 0),
    ("hex", 9, X.DILU, X.DILU, True, 9 * 9 * 9 * 3 * 8)])
def test_sweeps_and_shared_memory(geom, n, U, p, sweeps, shared):
    iters = 2
    make = cases.cavity3d if geom == "hex" else cases.cavity2d
    mesh, model, config, pref = make(n, iterations=iters)
    config["solvers"]["U"], config["solvers"]["p"] = _solver(model, "U", U), _solver(model, "p", p)
    case, keep = X.make_case(model, config, pref)
    s = X.Solver(mesh, renumber=_abi.RENUMBER_NONE)
    try:
        s.setup(case)
        fU, fp = cases.fields(model)
        for f, v in ((_abi.FIELD_UX, fU[0]), (_abi.FIELD_UY, fU[1]), (_abi.FIELD_UZ, fU[2]), (_abi.FIELD_P, fp)):
            s.set_field(f, v)
        dev = s.run(iters)
        form = s.last_form()
        assert form["sweeps_by_one"] == sweeps and form["shared_bytes"] == shared
        dev["U"] = [s.get_field(f) for f in (_abi.FIELD_UX, _abi.FIELD_UY, _abi.FIELD_UZ)]
        dev["p"] = s.get_field(_abi.FIELD_P)
        dev["perm"] = s.permutation() - 1
        dev["AU"], dev["bU"] = s.equation(0)
        dev["Ap"], bp = s.equation(1)
        dev["bp"] = bp[0]
    finally:
        s.close()
    orc = run_oracle(mesh, model, config, pref, iters, dev["perm"])
    assert_parity(dev, orc, nU=3 if geom == "hex" else 2)
