"""The build of the program for numberings with sweeps by one CTA, and the build
without them: the launch forms that can be asked for, mixed precision, and the
serving kernel of each, with numberings that the other build would take (a
two-colour numbering given as the caller's own, levels too wide for one CTA)."""
import numpy as np
import pytest

import xcal as X
from xcal import _abi, cases
from parity_util import assert_parity, compare, run_device, run_oracle

pytestmark = pytest.mark.gpu

FIELDS = (_abi.FIELD_UX, _abi.FIELD_UY, _abi.FIELD_UZ, _abi.FIELD_P)


@pytest.mark.parametrize("env", [{"XCAL_OCC": "4", "XCAL_SYNC": "grid"}, {"XCAL_SYNC": "block"},
                                 {"XCAL_SYNC": "cluster"}, {"XCAL_SYNC": "grid", "XCAL_NBLOCKS": "3"}])
@pytest.mark.parametrize("geom,n,renumber", [("quad", 33, _abi.RENUMBER_NONE), ("hex", 9, _abi.RENUMBER_RCM)])
def test_launch_forms_match_oracle(env, geom, n, renumber, monkeypatch):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    mesh, model, config, pref = cases.cavity3d(n, iterations=3) if geom == "hex" else cases.cavity2d(n, iterations=3)
    dev = run_device(mesh, model, config, pref, 3, renumber)
    orc = run_oracle(dev["dev_mesh"], model, config, pref, 3, dev["perm"])
    assert_parity(dev, orc, nU=3 if geom == "hex" else 2)


@pytest.mark.parametrize("renumber", [_abi.RENUMBER_NONE, _abi.RENUMBER_RCM])
def test_mixed_sweeps_converge_to_the_fp64_fields(renumber):
    """FP32 sweeps: the converged fields keep the bound of mixed precision, 1e-6."""
    mesh, model, config, pref = cases.cavity2d(33, iterations=1000)
    dev = run_device(mesh, model, config, pref, 1000, renumber, precision=_abi.PREC_MIXED)
    orc = run_oracle(dev["dev_mesh"], model, config, pref, 1000, dev["perm"])
    assert dev["done"] < 1000 and orc["done"] < 1000
    d = compare(dev, orc, 2, check_eqns=False)
    for k in ("U0", "U1", "p"):
        assert d[k] <= 1e-6, (k, d[k])


def _coloured(mesh):
    s = X.Solver(mesh, renumber=_abi.RENUMBER_COLOR)
    try:
        return s.exported_mesh()
    finally:
        s.close()


@pytest.mark.parametrize("precision", [_abi.PREC_FP64, _abi.PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("renumber", [_abi.RENUMBER_NONE, _abi.RENUMBER_RCM])
def test_serving_uncoloured_numberings(renumber, precision):
    iters = 5
    made = [cases.cavity2d(20), cases.cavity2d(33), cases.bfs(3), cases.cavity2d(125),
            cases.cavity2d(mesh=_coloured(cases.cavity2d(40)[0]))]
    srv = X.Server(slots=8, max_iterations=iters, tolerance=0.0, renumber=renumber, precision=precision,
                   device_bytes=4e8, host_bytes=2.5e8)
    try:
        tickets = [srv.submit(model, config, pref) for _, model, config, pref in made]
        got = [srv.poll(t, wait_ms=-1) for t in tickets]
    finally:
        srv.close()
    for (mesh, model, config, pref), r in zip(made, got):
        case, keep = X.make_case(model, config, pref, precision)
        s = X.Solver(mesh, renumber=renumber)
        try:
            s.setup(case)
            s.set_tolerance(0.0)
            U, p = cases.fields(model)
            for f, v in zip(FIELDS, (U[0], U[1], U[2], p)):
                s.set_field(f, v)
            out = s.run(iters)
            assert r["iterations"] == out["done"] == iters
            assert np.array_equal(r["p"], s.get_field(_abi.FIELD_P))
            for d in range(2):
                assert np.array_equal(r["U"][d], s.get_field(FIELDS[d]))
        finally:
            s.close()
