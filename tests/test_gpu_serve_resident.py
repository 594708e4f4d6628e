"""Serving with the matrix rows of the pressure CG in shared memory: the rows are
those of the group a case gets, so cases of one tile, of a full group and of
several groups' size keep them where a CTA's tiles fit (mixed precision with the
default of 4 tiles per CTA, FP64 with 3), and give the bits of the case alone
either way."""
import numpy as np
import pytest

import xcal as X
from xcal import _abi, cases

pytestmark = pytest.mark.gpu

FIELDS = (_abi.FIELD_UX, _abi.FIELD_UY, _abi.FIELD_UZ, _abi.FIELD_P)


@pytest.mark.parametrize("dim,sizes,prec,tiles,resident", [
    (2, (16, 32, 101, 200), _abi.PREC_MIXED, 0, 4),    # 1, 4, 40 and 157 tiles
    (2, (16, 101, 200), _abi.PREC_FP64, 3, 3), (2, (16, 101, 200), _abi.PREC_FP64, 0, 0),
    (2, (16, 101), _abi.PREC_MIXED, 5, 0),
    (3, (6, 20), _abi.PREC_MIXED, 3, 2), (3, (6, 20), _abi.PREC_FP64, 2, 2), (3, (20,), _abi.PREC_FP64, 0, 0)])
def test_resident_rows_match_the_case_alone(dim, sizes, prec, tiles, resident):
    iters = 4
    make = cases.cavity3d if dim == 3 else cases.cavity2d
    made = [make(n) for n in sizes]
    srv = X.Server(slots=8, max_iterations=iters, tolerance=0.0, precision=prec, dim=dim, tiles_per_cta=tiles,
                   device_bytes=4e8, host_bytes=2.5e8)
    try:
        tickets = [srv.submit(model, config, pref) for _, model, config, pref in made]
        got = [srv.poll(t, wait_ms=-1) for t in tickets]
        assert srv.stats()["resident"] == resident
    finally:
        srv.close()
    for (mesh, model, config, pref), r in zip(made, got):
        case, keep = X.make_case(model, config, pref, prec)
        s = X.Solver(mesh)
        try:
            s.setup(case)
            s.set_tolerance(0.0)
            U, p = cases.fields(model)
            for f, v in zip(FIELDS, (U[0], U[1], U[2], p)):
                s.set_field(f, v)
            assert s.run(iters)["done"] == r["iterations"] == iters
            assert np.array_equal(r["p"], s.get_field(_abi.FIELD_P))
            for d in range(dim):
                assert np.array_equal(r["U"][d], s.get_field(FIELDS[d]))
        finally:
            s.close()
