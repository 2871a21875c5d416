"""The column code's fast pass as a lane of a warp runs it: every vote won by a
neighbour, so that the lane computes (and selects away) what it does not need,
with the GPU's own division and square-root sequences.  It must end for any
input, leave no operand outside the exact windows unreported, and give the
plain column code's bits, in the kernels' narrow and 256-thread forms."""
import numpy as np
import pytest

from openifs_b200 import fields, inputs
from tests import util
from tests.test_fast_pass_window import _hostile

NPROMA, NBLK = 32, 8
NGPTOT = NPROMA * NBLK - 5


def _non_finite(arrs, rng):
    """Infinite and NaN amounts, one value per point: each species of PCLV and
    of its tendency, the vapour, the convective inputs.  (A row whose amount or
    sink sum is infinite has a NaN ratio in the sink truncation.)"""
    for n in ("pclv", "tendency_cml_cld", "pludeli", "psnde"):
        for m in range(min(4, arrs[n].shape[1])):
            for v in (np.inf, -np.inf, np.nan):
                b, k, jl = rng.integers(0, NBLK), rng.integers(20, arrs["pt"].shape[1], 4), rng.integers(0, NPROMA)
                arrs[n][b, m, k, jl] = v
    for n in ("pq", "pa", "plu", "plude", "pmfu", "pmfd", "tendency_cml_q", "tendency_cml_a"):
        for v in (np.inf, -np.inf, np.nan):
            arrs[n][rng.integers(0, NBLK), rng.integers(20, arrs["pt"].shape[1]), rng.integers(0, NPROMA)] = v
    return arrs


def _inputs(case, p, seed):
    arrs = inputs.generate(NBLK, NPROMA, p, seed=seed)
    rng = np.random.default_rng(seed + 1)
    if case == "hostile":
        return _hostile(arrs, rng)
    if case == "non_finite":
        return _non_finite(arrs, rng)
    return arrs if case == "plain" else util.apply_case(arrs, case)


CASES = ["plain", "hostile", "non_finite", "supersaturated", "negative_condensate", "tiny_cloud_fraction"]


@pytest.mark.parametrize("build", ["lanes", "lanes_wide"])
@pytest.mark.parametrize("case", CASES)
def test_column(built, case, build):
    p, _ = util.params()
    arrs = _inputs(case, p, 81)
    for form in (0, 1):
        ref, nw = util.run_hostemu(p, arrs, NPROMA, NBLK, NGPTOT, precision=form | 0x100)
        emu, nwe, violations = util.run_hostemu(p, arrs, NPROMA, NBLK, NGPTOT, precision=form | 0x300, libm=build)
        assert violations == 0
        assert nw == nwe
        for n in util.COMPARED:
            a, b = (util.defined(n, util._valid_cols(x[n], NGPTOT, NPROMA)) for x in (emu, ref))
            assert np.array_equal(a, b, equal_nan=True), (form, n)


@pytest.mark.parametrize("build", ["lanes", "lanes_wide"])
@pytest.mark.parametrize("opt", ["budgets", "spp", "all+budgets"])
@pytest.mark.parametrize("case", ["plain", "hostile", "non_finite"])
def test_optional_forms(built, case, opt, build):
    p, _ = util.params()
    p = util.with_flags(p, util.BUDGET_CASES[-1]) if opt == "budgets" else util.opt_params(p, opt)
    arrs = _inputs(case, p, 83)
    diag = inputs.generate_diag(arrs, NPROMA, fields.budget_fields_needed(p) + 1, seed=84)
    ref, dref, nw = util.run_hostemu_diag(p, arrs, diag, NPROMA, NBLK, NGPTOT, flags=0x100)
    emu, demu, nwe, violations = util.run_hostemu_diag(p, arrs, diag, NPROMA, NBLK, NGPTOT, flags=0x300, libm=build)
    assert violations == 0
    assert nw == nwe
    for n in util.COMPARED:
        a, b = (util.defined(n, util._valid_cols(x[n], NGPTOT, NPROMA)) for x in (emu, ref))
        assert np.array_equal(a, b, equal_nan=True), n
    for n in ("pfsd", "pextra"):
        a, b = (util._valid_cols(x[n], NGPTOT, NPROMA) for x in (demu, dref))
        assert np.array_equal(a, b, equal_nan=True), n
