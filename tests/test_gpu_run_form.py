"""xcal_last_run_form: the form that a run's pressure solve took and the kernels
it launched, as the rules choose them and as XCAL_CG asks for them.  Forms that
only large meshes take by themselves are asked for on meshes of one partial
tile up to a few tiles, bitwise against the oracle, in PISO, and in a run that
converges."""
import numpy as np
import pytest

import xcal as X
from xcal import _abi, cases
from parity_util import assert_parity, run_oracle

pytestmark = pytest.mark.gpu

FIELDS = (_abi.FIELD_UX, _abi.FIELD_UY, _abi.FIELD_UZ, _abi.FIELD_P)


def _make(geom, n, iters, **kw):
    return {"quad": cases.cavity2d, "hex": cases.cavity3d, "bfs": cases.bfs}[geom](n, iterations=iters, **kw)


class _Run:
    """One context on a case; run() starts from the model's fields."""

    def __init__(self, made, prec=_abi.PREC_FP64, renumber=_abi.RENUMBER_COLOR):
        self.mesh, self.model, self.config, self.pref = made
        self.case, self.keep = X.make_case(self.model, self.config, self.pref, prec)
        self.s = X.Solver(self.mesh, renumber=renumber)
        self.s.setup(self.case)

    def run(self, iters, piso=False):
        U, p = cases.fields(self.model)
        for f, v in zip(FIELDS, (U[0], U[1], U[2], p)):
            self.s.set_field(f, v)
        out = self.s.run(iters, piso=piso)
        out["U"] = np.stack([self.s.get_field(f) for f in FIELDS[:3]])
        out["p"] = self.s.get_field(_abi.FIELD_P)
        return out


@pytest.mark.parametrize("geom,n,prec,renumber,kw,form", [
    ("quad", 2, 0, 2, {}, "cluster"), ("quad", 40, 0, 2, {}, "cluster"), ("quad", 155, 1, 2, {}, "cluster"),
    ("hex", 20, 0, 2, {}, "cluster"), ("hex", 28, 0, 2, {}, "resident"),
    ("quad", 160, 0, 2, {}, "resident"), ("quad", 200, 1, 2, {}, "resident"),
    ("bfs", 27, 0, 2, {}, "resident"), ("hex", 32, 0, 2, {}, "resident"), ("hex", 70, 0, 2, {}, "kernel"),
    ("quad", 40, 0, 0, {}, "general"), ("quad", 40, 0, 2, {"precon": X.Jacobi}, "general"),
    ("quad", 40, 0, 2, {"p_solver": X.BicgstabSolver}, "general")])
def test_form_taken(geom, n, prec, renumber, kw, form):
    r = _Run(_make(geom, n, 2, **kw), prec, renumber)
    try:
        r.run(2)
        f = r.s.last_form()
        assert f["cg"] == form
        assert f["launches"] == (5 if form in ("cluster", "kernel") else 1)
        assert f["sweeps_by_one"] == (renumber == _abi.RENUMBER_NONE)
        if form == "resident":
            assert f["shared_bytes"] >= 256 * 5 * (8 if prec else 12)
    finally:
        r.s.close()


@pytest.mark.parametrize("form", ["kernel", "streamed", "resident"])
@pytest.mark.parametrize("geom,n", [("quad", 2), ("quad", 16), ("quad", 23), ("quad", 32), ("quad", 45), ("bfs", 3),
                                    ("hex", 2), ("hex", 7), ("hex", 16)])
def test_forced_forms_match_oracle(form, geom, n, monkeypatch):
    monkeypatch.setenv("XCAL_SYNC", "grid")
    monkeypatch.setenv("XCAL_CG", "program" if form == "resident" else form)
    r = _Run(_make(geom, n, 3))
    try:
        dev = r.run(3)
        assert r.s.last_form()["cg"] == form
        dev["perm"] = r.s.permutation() - 1
        dev["AU"], dev["bU"] = r.s.equation(0)
        dev["Ap"], bp = r.s.equation(1)
        dev["bp"] = bp[0]
        orc = run_oracle(r.s.exported_mesh(), r.model, r.config, r.pref, 3, dev["perm"])
        assert_parity(dev, orc, nU=3 if geom == "hex" else 2)
    finally:
        r.s.close()


@pytest.mark.parametrize("form", ["kernel", "streamed"])
@pytest.mark.parametrize("prec", [_abi.PREC_FP64, _abi.PREC_MIXED], ids=["fp64", "mixed"])
def test_forced_forms_in_piso_and_to_convergence(form, prec, monkeypatch):
    made = _make("quad", 45, 1)
    made[2]["schemes"]["U"] = X.set_schemes(time=X.Euler, divergence=X.Upwind)
    made[2]["runtime"] = X.set_runtime(iterations=6, write_interval=-1, time_step=1e-3)
    got = {}
    for f in ("default", form):
        if f != "default":
            monkeypatch.setenv("XCAL_SYNC", "grid")
            monkeypatch.setenv("XCAL_CG", f)
        r = _Run(made, prec)
        try:
            got[f] = [r.run(6, piso=True)]
            assert r.s.last_form()["cg"] == ("cluster" if f == "default" else f)
            r.s.set_tolerance(5e-3)
            got[f].append(r.run(400))
        finally:
            r.s.close()
    assert 1 < got[form][1]["done"] < 400
    for a, b in zip(got["default"], got[form]):
        assert a["done"] == b["done"]
        for k in ("U", "p", "R_p", "krylov"):
            assert np.array_equal(a[k], b[k], equal_nan=True), k
