"""Runs that are cut at their pressure solves (a kernel of its own between
launches of the program) and end before their limit: by convergence, at every
place relative to the batches their launches are queued in, or at a non-finite
norm.  Same iterations and bits as the run in one launch, for the solve in one
cluster (quad 40^2) and on the whole GPU (hex 70^3, FP64), and a run that
stops at once costs about one iteration whatever its limit."""
import numpy as np
import pytest

import xcal as X
from xcal import _abi, cases

pytestmark = pytest.mark.gpu

FIELDS = (_abi.FIELD_UX, _abi.FIELD_UY, _abi.FIELD_UZ, _abi.FIELD_P)


def _solver(geom, n, flags=0):
    mesh, model, config, pref = cases.cavity3d(n) if geom == "hex" else cases.cavity2d(n)
    case, keep = X.make_case(model, config, pref)
    s = X.Solver(mesh, flags=flags)
    s.setup(case)
    return s, (mesh, model, keep)


def _start(s, mesh):
    c = mesh.cell_centres()
    c = (c - c.min(axis=0)) / np.ptp(c[:, 0])
    for f, v in zip(FIELDS, (np.sin(5.0 * c[:, 1]), 0.2 * np.cos(4.0 * c[:, 0]), 0.0 * c[:, 0], 0.1 * c[:, 0])):
        s.set_field(f, v)


def _run(s, mesh, iters, piso=False):
    _start(s, mesh)
    out = s.run(iters, piso=piso)
    return out, [s.get_field(f) for f in FIELDS]


def _residual(out, ns):
    return np.max([out[k] for k in ("R_ux", "R_uy", "R_p") + ("R_uz",) * (ns == 3)], axis=0)


@pytest.mark.parametrize("geom,n,limit", [("quad", 40, 40), ("hex", 70, 14)])
def test_stop_by_convergence(geom, n, limit, monkeypatch):
    s, (mesh, model, keep) = _solver(geom, n)
    ns = 3 if geom == "hex" else 2
    try:
        s.set_tolerance(0.0)
        full, _ = _run(s, mesh, limit)
        R = _residual(full, ns)
        low = np.flatnonzero(R <= np.minimum.accumulate(R))   # iterations that a tolerance of their own residual stops
        stops = [k for k in low if k + 1 in (1, 2, 3, 4, 5, 7, 8, 9, 13, 16, 17, 33)]
        assert len(stops) >= 2
        for k in stops:
            s.set_tolerance(float(R[k]))
            monkeypatch.delenv("XCAL_SYNC", raising=False)
            out, f = _run(s, mesh, limit)
            monkeypatch.setenv("XCAL_SYNC", "grid")   # one launch
            ref, g = _run(s, mesh, limit)
            assert out["done"] == ref["done"] == k + 1
            assert np.array_equal(out["krylov"], ref["krylov"])
            for a, b in zip(f, g):
                assert np.array_equal(a, b)
    finally:
        s.close()


@pytest.mark.parametrize("geom,n", [("quad", 40), ("hex", 70)])
@pytest.mark.parametrize("piso", [False, True])
def test_stop_at_a_non_finite_norm(geom, n, piso):
    s, (mesh, model, keep) = _solver(geom, n, _abi.FLAG_ABORT_ON_NAN)
    try:
        ref, f = _run(s, mesh, 6, piso)
        _start(s, mesh)
        bad = np.zeros(mesh.ncells)
        bad[mesh.ncells // 2] = np.nan
        s.set_field(_abi.FIELD_P, bad)
        with pytest.raises(_abi.XcalError, match="XCAL_ERR_NAN .*iteration 1;"):
            s.run(1000, piso=piso)
        again, g = _run(s, mesh, 6, piso)   # the context is as good as before
    finally:
        s.close()
    assert again["done"] == ref["done"] == 6
    for a, b in zip(f, g):
        assert np.array_equal(a, b)


def test_restart_of_a_converged_run_costs_one_iteration():
    s, (mesh, model, keep) = _solver("quad", 40)
    try:
        s.set_tolerance(1e-3)
        _run(s, mesh, 2000)
        ms = {}
        for limit in (1, 1000, 20000):
            t = []
            for _ in range(5):
                assert s.run(limit)["done"] == 1
                t.append(s.last_ms())
            ms[limit] = min(t)
    finally:
        s.close()
    assert ms[1000] <= 2.0 * ms[1] and ms[20000] <= 2.0 * ms[1], ms
