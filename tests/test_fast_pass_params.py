"""The parameters the column code's fast pass accepts (fast_pass_params_ok): with
each one at either end of its accepted range, alone, and the saturation
constants in pairs, the host builds find no operand outside the exact windows
in a column that was not reported, and the fast pass with its rerun gives the
plain column code's bits.  The ends are found by bisection on the accepting
function itself."""
import ctypes
import itertools
import math

import numpy as np
import pytest

from openifs_b200 import inputs
from tests import util

NPROMA, NBLK = 32, 2
SATURATION = ["r2es", "r3les", "r3ies", "r4les", "r4ies", "rtt", "retv"]


@pytest.fixture(scope="module")
def columns(built):
    """An ordinary block and a supersaturated one."""
    global _host
    _host = util.hostemu("lanes")
    p, _ = util.params()
    a = inputs.generate(NBLK, NPROMA, p, seed=71)
    b = util.apply_case(inputs.generate(NBLK, NPROMA, p, seed=72), "supersaturated")
    return {n: np.concatenate([a[n][:1], b[n][:1]]) for n in a}


def _accepted(p):
    return bool(_host.hostemu_params_ok(ctypes.byref(p)))


def _with(p, name, x):
    q = type(p).from_buffer_copy(p)
    setattr(q, name, x)
    return q


def _ends(p, name):
    """The largest, the smallest and the closest-to-zero accepted values (found
    from p's own value outward), or none for a parameter that is not checked."""
    d, out = getattr(p, name), []
    fwd = lambda x: math.copysign(math.log1p(abs(x) / 1e-16), x)
    back = lambda y: math.copysign(math.expm1(abs(y)) * 1e-16, y)
    for far in (-1e20, 1e20):
        if _accepted(_with(p, name, far)):
            continue
        lo, hi = fwd(d), fwd(far)
        for _ in range(80):
            m = 0.5 * (lo + hi)
            lo, hi = (m, hi) if _accepted(_with(p, name, back(m))) else (lo, m)
        out.append(back(lo))
    if d != 0.0 and not _accepted(_with(p, name, math.copysign(1e-30, d))):
        lo, hi = math.log(abs(d)), math.log(1e-30)
        for _ in range(80):
            m = 0.5 * (lo + hi)
            lo, hi = (m, hi) if _accepted(_with(p, name, math.copysign(math.exp(m), d))) else (lo, m)
        out.append(math.copysign(math.exp(lo), d))
    return sorted(set(out))


def _check(p, columns, what, build):
    before = util.hostemu_violations(util.hostemu(build))
    ref, nw = util.run_hostemu(p, columns, NPROMA, NBLK, NPROMA * NBLK)
    emu, nwe, violations = util.run_hostemu(p, columns, NPROMA, NBLK, NPROMA * NBLK, precision=0x200, libm=build)
    assert violations == before, what
    assert nw == nwe, what
    for n in util.COMPARED:
        assert np.array_equal(util.defined(n, emu[n]), util.defined(n, ref[n]), equal_nan=True), (what, n)


@pytest.mark.parametrize("build", ["lanes", "lanes_wide"])
def test_each_parameter_at_its_ends(columns, build):
    p, _ = util.params()
    assert _accepted(p)
    checked = 0
    for name in [n for n, t in p._fields_ if t is ctypes.c_double]:
        for x in _ends(p, name):
            _check(_with(p, name, x), columns, (name, x), build)
            checked += 1
    assert checked > 120


@pytest.mark.parametrize("pair", list(itertools.combinations(SATURATION, 2)), ids="-".join)
def test_saturation_constants_in_pairs(columns, pair):
    p, _ = util.params()
    for x in _ends(p, pair[0]):
        q = _with(p, pair[0], x)
        for y in _ends(q, pair[1]):
            _check(_with(q, pair[1], y), columns, (pair, x, y), "lanes")
