"""Sweeps by one CTA over many levels.  The other CTAs wait at a barrier
meanwhile, and a wait is limited, so a wait must not span the whole sweep: on a
chain every row is a level of its own.  Sizes around the 1024 levels of one
wait (n rows are n forward and n - 1 backward levels at the set-up) and the
12,288 values of the vector in shared memory, bitwise against the oracle; and
a chain whose sweep pair takes many times the limit."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from xcal import _abi

pytestmark = pytest.mark.gpu


def _chain(n):
    rng = np.random.default_rng(n)
    lo = -1.0 + 0.1 * rng.random(n - 1)
    rp = np.concatenate([[0], np.cumsum(3 - (np.arange(n) == 0) - (np.arange(n) == n - 1))]).astype(np.int32)
    i = np.arange(n)
    ent = np.stack([i - 1, i, i + 1], axis=1)
    v = np.stack([np.r_[0.0, lo], np.full(n, 2.5), np.r_[lo, 0.0]], axis=1)
    keep = (ent >= 0) & (ent < n)
    return rp, ent[keep].astype(np.int32), v[keep], rng.standard_normal(n)


def _solve(solver, precon, rp, col, val, b, itmax):
    lib = _abi.load()
    h = C.c_void_p()
    _abi.check(lib.xcal_ctx_create(0, 0, C.byref(h)))
    try:
        x, it, rn = np.zeros(len(b)), np.zeros(1, dtype=np.int32), np.zeros(1)
        _abi.check(lib.xcal_linear_solve(h, solver, precon, len(b), _abi.i32ptr(rp), _abi.i32ptr(col), _abi.dptr(val),
                                         _abi.dptr(b), _abi.dptr(x), itmax, 0.0, 1e-10, _abi.i32ptr(it),
                                         _abi.dptr(rn)), h)
    finally:
        lib.xcal_ctx_destroy(h)
    return x, int(it[0])


@pytest.mark.parametrize("solver", [_abi.SOLVER_CG, _abi.SOLVER_BICGSTAB], ids=["cg", "bicgstab"])
@pytest.mark.parametrize("precon", [_abi.PRECON_DILU, _abi.PRECON_ILU0], ids=["dilu", "ilu0"])
@pytest.mark.parametrize("n", [3, 512, 513, 514, 1024, 1025, 3000, 12288, 12289])
def test_chain_matches_oracle(solver, precon, n):
    rp, col, val, b = _chain(n)
    x, it = _solve(solver, precon, rp, col, val, b, 12)
    xo, ito, _ = O.linear_solve(solver, precon, rp, col, val, b, np.zeros(n), itmax=12, atol=0.0, rtol=1e-10)
    assert it == ito
    assert np.array_equal(x, xo)


@pytest.mark.parametrize("precon", [_abi.PRECON_DILU, _abi.PRECON_ILU0], ids=["dilu", "ilu0"])
def test_sweep_longer_than_the_wait_limit(precon, monkeypatch):
    """A pair has 120,000 levels: at 0.7 us or more each over 80 ms, four times
    the limit of one wait here; 1024 levels at up to 5 us are 5 ms."""
    monkeypatch.setenv("XCAL_BARRIER_TIMEOUT_US", "20000")
    n = 60000
    rp, col, val, b = _chain(n)
    x, it = _solve(_abi.SOLVER_CG, precon, rp, col, val, b, 2)
    xo, ito, _ = O.linear_solve(_abi.SOLVER_CG, precon, rp, col, val, b, np.zeros(n), itmax=2, atol=0.0, rtol=1e-10)
    assert it == ito
    assert np.array_equal(x, xo)


def _band(n, h):
    """Symmetric band of half width h: every row a level, rows of 2h + 1 entries."""
    rng = np.random.default_rng(h)
    off = {d: -rng.random(n - d) for d in range(1, h + 1)}
    rows, cols, vals = [np.arange(n)], [np.arange(n)], [np.full(n, 2.0 * h + 1.0)]
    for d, v in off.items():
        i = np.arange(n - d)
        rows += [i, i + d]
        cols += [i + d, i]
        vals += [v, v]
    r, c, v = np.concatenate(rows), np.concatenate(cols), np.concatenate(vals)
    o = np.lexsort((c, r))
    return (np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32), c[o].astype(np.int32), v[o],
            rng.standard_normal(n))


@pytest.mark.parametrize("precon", [_abi.PRECON_DILU, _abi.PRECON_ILU0], ids=["dilu", "ilu0"])
@pytest.mark.parametrize("n,h", [(700, 3), (700, 4), (1500, 20), (300, 130)])
def test_wide_rows_match_oracle(precon, n, h):
    """Rows of 7 (unrolled), 9, 41 and 261 entries: a wait has 1024, 809, 38 and 1 of their levels."""
    rp, col, val, b = _band(n, h)
    x, it = _solve(_abi.SOLVER_CG, precon, rp, col, val, b, 4)
    xo, ito, _ = O.linear_solve(_abi.SOLVER_CG, precon, rp, col, val, b, np.zeros(n), itmax=4, atol=0.0, rtol=1e-10)
    assert it == ito
    assert np.array_equal(x, xo)


def test_wide_rows_within_the_wait_limit(monkeypatch):
    """The set-up of ILU(0) takes about 41^2/2 dependent steps of 0.25 us a level:
    200 ms for 1024 levels, twice the limit here, and 8 ms for the 38 of a wait."""
    monkeypatch.setenv("XCAL_BARRIER_TIMEOUT_US", "100000")
    test_wide_rows_match_oracle(_abi.PRECON_ILU0, 1500, 20)


@pytest.mark.parametrize("isolated", [16000, 16383, 16384])
def test_one_wide_level(isolated):
    """A chain and rows without neighbours: 1500 levels, the first of up to and above the 16,384 rows one CTA sweeps."""
    rp, col, val, b = _chain(1500)
    n = 1500 + isolated
    rp = np.concatenate([rp, rp[-1] + np.arange(1, isolated + 1)]).astype(np.int32)
    col = np.concatenate([col, np.arange(1500, n)]).astype(np.int32)
    val = np.concatenate([val, np.full(isolated, 3.0)])
    b = np.random.default_rng(1).standard_normal(n)
    x, it = _solve(_abi.SOLVER_CG, _abi.PRECON_DILU, rp, col, val, b, 6)
    xo, ito, _ = O.linear_solve(_abi.SOLVER_CG, _abi.PRECON_DILU, rp, col, val, b, np.zeros(n), itmax=6, atol=0.0,
                                rtol=1e-10)
    assert it == ito
    assert np.array_equal(x, xo)
