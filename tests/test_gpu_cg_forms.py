"""The pressure CG over a two-level numbering in its forms: one cluster with
the mesh in shared memory, inside the program with the matrix rows in shared
memory or streamed, and a kernel of its own on the whole GPU.  All compute the
same bits; the sizes sit at the edges of tiles (256 rows), of the split into
levels inside a tile, of the clusters' shares and of the row widths."""
import numpy as np
import pytest

from xcal import _abi, cases
from parity_util import assert_parity, run_device, run_oracle

pytestmark = pytest.mark.gpu

FORMS = {"own-kernel": {}, "resident": {"XCAL_SYNC": "grid"}, "streamed": {"XCAL_SYNC": "grid", "XCAL_NBLOCKS": "2"}}


def _env(monkeypatch, form):
    for k in ("XCAL_SYNC", "XCAL_NBLOCKS"):
        monkeypatch.delenv(k, raising=False)
    for k, v in FORMS[form].items():
        monkeypatch.setenv(k, v)


def _case(geom, n, iters):
    return cases.cavity3d(n, iterations=iters) if geom == "hex" else cases.cavity2d(n, iterations=iters)


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("geom,n", [("quad", 2), ("quad", 16), ("quad", 23), ("quad", 32), ("quad", 64), ("quad", 81),
                                    ("hex", 2), ("hex", 7), ("hex", 16), ("hex", 21)])
def test_cg_forms_match_oracle(form, geom, n, monkeypatch):
    _env(monkeypatch, form)
    mesh, model, config, pref = _case(geom, n, 4)
    dev = run_device(mesh, model, config, pref, 4, _abi.RENUMBER_COLOR)
    orc = run_oracle(dev["dev_mesh"], model, config, pref, 4, dev["perm"])
    assert_parity(dev, orc, nU=3 if geom == "hex" else 2)


@pytest.mark.parametrize("geom,n,prec", [("quad", 45, _abi.PREC_MIXED), ("quad", 155, _abi.PREC_MIXED),
                                         ("quad", 160, _abi.PREC_FP64), ("hex", 30, _abi.PREC_MIXED),
                                         ("hex", 70, _abi.PREC_FP64), ("hex", 77, _abi.PREC_MIXED)])
def test_cg_forms_agree(geom, n, prec, monkeypatch):
    """Larger meshes and mixed precision: every form gives the same bits."""
    mesh, model, config, pref = _case(geom, n, 3)
    got = {}
    for form in FORMS:
        _env(monkeypatch, form)
        got[form] = run_device(mesh, model, config, pref, 3, _abi.RENUMBER_COLOR, precision=prec)
    for form in ("resident", "streamed"):
        for k in ("U", "p", "R_p"):
            assert np.array_equal(got[form][k], got["own-kernel"][k], equal_nan=True), (form, k)
        assert np.array_equal(got[form]["krylov"], got["own-kernel"]["krylov"]), form
