"""The column code's fast pass on the host: the level's input checks must place
every operand of its divisions, exps, logs and pows inside the windows where
the branch-free forms are exact, or report the column.  The window build
counts the operands that break that promise (none may), and the outputs equal
the plain column code's bit for bit whatever the inputs."""
import numpy as np
import pytest

from openifs_b200 import inputs
from tests import util


def _hostile(arrs, rng):
    """Values outside the checked ranges scattered over the fields: tiny,
    subnormal, huge, zero, negative, infinite and NaN."""
    bad = np.array([0.0, 1e-300, 5e-324, 1e-310, -1e-290, 1e-80, 1e30, 1e80, 1e300, -1e300, np.inf, -np.inf, np.nan])
    for n in ("pt", "pq", "pap", "pa", "pclv", "plude", "plu", "pmfu", "pmfd", "pludeli", "psnde", "tendency_cml_t",
              "tendency_cml_q", "tendency_cml_a", "tendency_cml_cld"):
        x = arrs[n].reshape(-1)
        i = rng.choice(x.size, max(1, x.size // 4000), replace=False)
        x[i] = rng.choice(bad, i.size)
    return arrs


def _cold(arrs, rng):
    """Temperatures of 60 .. 160 K and 300 .. 1200 K, pressures over 12 decades."""
    arrs["pt"][:2] = rng.uniform(60.0, 160.0, arrs["pt"][:2].shape)
    arrs["pt"][2:4] = rng.uniform(300.0, 1200.0, arrs["pt"][2:4].shape)
    arrs["pap"][4:] = 10.0 ** rng.uniform(-4.0, 8.0, arrs["pap"][4:].shape)
    return arrs


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("case", ["plain", "hostile", "ranges", "L60"] + util.EDGE_CASES)
def test_operands_stay_in_the_window(built, case, form):
    klev = 60 if case == "L60" else util.KLEV
    p, _ = util.params(inputs.ncldtop_for(klev))
    nproma, nblk = 32, 8
    arrs = inputs.generate(nblk, nproma, p, klev=klev, seed=71)
    rng = np.random.default_rng(72)
    if case == "hostile":
        arrs = _hostile(arrs, rng)
    elif case == "ranges":
        arrs = _cold(arrs, rng)
    elif case in util.EDGE_CASES:
        arrs = util.apply_case(arrs, case)
    ngptot = nproma * nblk - 5
    ref, nw = util.run_hostemu(p, arrs, nproma, nblk, ngptot, precision=form | 0x100, klev=klev)
    emu, nwe, violations = util.run_hostemu(p, arrs, nproma, nblk, ngptot, precision=form | 0x300, libm="window", klev=klev)
    assert violations == 0
    assert nw == nwe
    for n in util.COMPARED:
        a = util.defined(n, util._valid_cols(emu[n], ngptot, nproma))
        b = util.defined(n, util._valid_cols(ref[n], ngptot, nproma))
        assert np.array_equal(a, b, equal_nan=True), n
