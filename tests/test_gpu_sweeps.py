"""Preconditioner sweeps of numberings with many narrow levels (the caller's
order, RCM), done by one CTA: bitwise equal to the oracle at sizes around the
32 rows of an item, the shared memory the vector has to fit (12,288 values in
FP64), several items in a level, and the average width above which the grid
sweeps instead."""
import pytest

import xcal as X
from xcal import _abi, cases
from parity_util import assert_parity, run_device, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("geom,n,renumber,precon", [
    ("quad", 3, _abi.RENUMBER_NONE, X.DILU), ("quad", 32, _abi.RENUMBER_NONE, X.DILU),
    ("quad", 33, _abi.RENUMBER_RCM, X.DILU), ("quad", 33, _abi.RENUMBER_NONE, X.ILU0),
    ("quad", 80, _abi.RENUMBER_NONE, X.DILU), ("quad", 115, _abi.RENUMBER_RCM, X.DILU),
    ("bfs", 5, _abi.RENUMBER_NONE, X.DILU), ("bfs", 5, _abi.RENUMBER_RCM, X.ILU0),
    ("hex", 5, _abi.RENUMBER_NONE, X.DILU), ("hex", 16, _abi.RENUMBER_RCM, X.DILU),
    ("hex", 26, _abi.RENUMBER_NONE, X.DILU), ("hex", 40, _abi.RENUMBER_NONE, X.DILU)])
def test_sweeps_match_oracle(geom, n, renumber, precon):
    make = {"quad": cases.cavity2d, "bfs": cases.bfs, "hex": cases.cavity3d}[geom]
    iters = 2
    mesh, model, config, pref = make(n, iterations=iters, precon=precon)
    dev = run_device(mesh, model, config, pref, iters, renumber)
    orc = run_oracle(dev["dev_mesh"], model, config, pref, iters, dev["perm"])
    assert_parity(dev, orc, nU=3 if geom == "hex" else 2)
