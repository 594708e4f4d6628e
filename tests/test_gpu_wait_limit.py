"""A short limit on the device's waits (XCAL_BARRIER_TIMEOUT_US).  The limit
bounds the waits of the grid barrier and nothing else: where a run has no such
wait it changes nothing, and a run that reaches it ends with XCAL_ERR_TIMEOUT
and leaves the context usable.  The runs here solve the pressure with the
matrix rows in shared memory, whose columns become addresses: no limit may
let the solve go on without them."""
import numpy as np
import pytest

import xcal as X
from xcal import _abi, cases

pytestmark = pytest.mark.gpu

FIELDS = (_abi.FIELD_UX, _abi.FIELD_UY, _abi.FIELD_P)


def _start(s, model):
    U, p = cases.fields(model)
    for f, v in zip(FIELDS, (U[0], U[1], p)):
        s.set_field(f, v)


def _run(s, model, iters):
    _start(s, model)
    out = s.run(iters)
    return [out["krylov"]] + [s.get_field(f) for f in FIELDS]


@pytest.mark.parametrize("prec", [_abi.PREC_FP64, _abi.PREC_MIXED])
@pytest.mark.parametrize("sync,n", [("block", 20), ("cluster", 20), ("cluster", 61)])
def test_limit_does_not_reach_runs_without_a_grid_barrier(sync, n, prec, monkeypatch):
    monkeypatch.setenv("XCAL_SYNC", sync)
    mesh, model, config, pref = cases.cavity2d(n, iterations=3)
    case, keep = X.make_case(model, config, pref, prec)
    s = X.Solver(mesh)
    try:
        s.setup(case)
        ref = _run(s, model, 3)
        monkeypatch.setenv("XCAL_BARRIER_TIMEOUT_US", "1")
        got = _run(s, model, 3)
    finally:
        s.close()
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("limit_us", ["1", "4", "30", "500"])
def test_limit_of_the_grid_barrier_ends_the_run_cleanly(limit_us, monkeypatch):
    monkeypatch.setenv("XCAL_SYNC", "grid")
    mesh, model, config, pref = cases.bfs(14, iterations=3)
    case, keep = X.make_case(model, config, pref)
    s = X.Solver(mesh)
    try:
        s.setup(case)
        ref = _run(s, model, 3)
        monkeypatch.setenv("XCAL_BARRIER_TIMEOUT_US", limit_us)
        try:
            got = _run(s, model, 3)
        except _abi.XcalError as e:
            assert "XCAL_ERR_TIMEOUT" in str(e)
            got = ref
        monkeypatch.delenv("XCAL_BARRIER_TIMEOUT_US")
        again = _run(s, model, 3)
    finally:
        s.close()
    for a, b, c in zip(got, again, ref):
        assert np.array_equal(a, c) and np.array_equal(b, c)
