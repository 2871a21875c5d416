"""The column kernels on inputs no column should have -- tiny, huge, infinite and
NaN values scattered over the fields: the fast pass ends and reports those
columns, their rerun gives the plain column code's bits (host build), and the
other columns of the warp are untouched by them (GPU tests)."""
import numpy as np
import pytest

from openifs_b200 import cloudsc, fields, inputs
from tests import util
from tests.test_fast_pass_votes import NBLK, NGPTOT, NPROMA, _inputs

pytestmark = pytest.mark.gpu

# by size (the 256-thread build at this size), and the narrow builds
SCHEDULES = [None, (1, 448, 0), (2, 384, 0)]


def _nan_columns(ref):
    """Columns whose outputs hold a NaN.  Which of them a MIN or MAX passes on, and
    the sign of a new one, differ between the host's compiler and the GPU's, so
    their other values may too; they are run, and have to end."""
    return np.any([np.isnan(util.defined(n, ref[n])).reshape(NBLK, -1, NPROMA).any(axis=1) for n in util.COMPARED],
                  axis=0)


def _same(got, ref, names=util.COMPARED, skip=None):
    skip = _nan_columns(ref) if skip is None else skip
    assert skip.sum() < 64
    for n in names:
        a, b = (util.defined(n, util._valid_cols(x[n], NGPTOT, NPROMA)).reshape(NBLK, -1, NPROMA) for x in (got, ref))
        keep = ~skip[:, None, :] & np.ones(a.shape, bool)
        assert np.array_equal(a[keep], b[keep]), n


def _with_schedule(sched, run, precision=cloudsc.FP64):
    before = cloudsc.get_schedule(precision)
    if sched is None:
        return run()
    try:
        cloudsc.set_schedule(precision, *sched)
        return run()
    finally:
        cloudsc.set_schedule(precision, *before)


@pytest.mark.parametrize("sched", SCHEDULES)
@pytest.mark.parametrize("case", ["hostile", "non_finite"])
def test_fp64(cuda, case, sched):
    p, _ = util.params()
    arrs = _inputs(case, p, 81)
    ref, nw = util.run_hostemu(p, arrs, NPROMA, NBLK, NGPTOT, precision=0x100)
    gpu, nwg = _with_schedule(sched, lambda: util.run_gpu(p, arrs, NPROMA, NBLK, NGPTOT))
    _same(gpu, ref)
    assert nwg == nw


@pytest.mark.parametrize("precision", [cloudsc.MIXED, cloudsc.PHYS32])
def test_other_columns_untouched(cuda, precision):
    """The FP32 forms (their powf and expf are the GPU's): the columns without a
    foreign value equal those of a run without any."""
    p, _ = util.params()
    clean = _inputs("plain", p, 81)
    arrs = _inputs("non_finite", p, 81)
    foreign = np.zeros((NBLK, NPROMA), bool)
    for n in clean:
        if clean[n].ndim >= 3:
            d = ~((arrs[n] == clean[n]) | (np.isnan(arrs[n]) & np.isnan(clean[n])))
            foreign |= d.reshape(NBLK, -1, NPROMA).any(axis=1)
    assert 0 < foreign.sum() < foreign.size // 2
    a, _ = util.run_gpu(p, arrs, NPROMA, NBLK, NGPTOT, precision=precision)
    b, _ = util.run_gpu(p, clean, NPROMA, NBLK, NGPTOT, precision=precision)
    for n in util.COMPARED:
        x, y = (util.defined(n, util._valid_cols(v[n], NGPTOT, NPROMA)).reshape(NBLK, -1, NPROMA) for v in (a, b))
        keep = ~foreign[:, None, :] & np.ones(x.shape, bool)
        assert np.array_equal(x[keep], y[keep]), n


@pytest.mark.parametrize("case", ["hostile", "non_finite"])
def test_single_precision_interface(cuda, case):
    import torch
    p, _ = util.params()
    with np.errstate(over="ignore"):
        sp = fields.to_single(_inputs(case, p, 81))
    wide = {k: (v.astype(np.float64) if v.dtype == np.float32 else v.copy()) for k, v in sp.items()}
    ref, nw = util.run_hostemu(p, wide, NPROMA, NBLK, NGPTOT, precision=0x100)
    cloudsc.setup(p)
    d = {k: torch.from_numpy(v).cuda() for k, v in sp.items()}
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    cloudsc.cloudsc_batched_sp(p, d, NPROMA, util.KLEV, NBLK, NGPTOT, util.PTSPHY, counter=cnt)
    torch.cuda.synchronize()
    with np.errstate(over="ignore"):
        _same({n: d[n].cpu().numpy() for n in util.COMPARED}, {n: ref[n].astype(np.float32) for n in util.COMPARED})
    assert int(cnt.item()) == nw


@pytest.mark.parametrize("opt", ["budgets", "spp", "all+budgets"])
def test_optional_forms(cuda, opt):
    import torch
    p0, _ = util.params()
    p = util.with_flags(p0, util.BUDGET_CASES[-1]) if opt == "budgets" else util.opt_params(p0, opt)
    arrs = _inputs("non_finite", p, 83)
    diag = inputs.generate_diag(arrs, NPROMA, fields.budget_fields_needed(p) + 1, seed=84)
    ref, dref, nw = util.run_hostemu_diag(p, arrs, diag, NPROMA, NBLK, NGPTOT, flags=0x100)
    try:
        cloudsc.setup(p)
        d = {k: torch.from_numpy(v).cuda() for k, v in arrs.items()}
        g = {k: torch.from_numpy(v).cuda() for k, v in diag.items()}
        cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
        cloudsc.cloudsc_batched_diag(p, d, g, NPROMA, util.KLEV, NBLK, NGPTOT, util.PTSPHY, counter=cnt)
        torch.cuda.synchronize()
    finally:
        cloudsc.setup(p0)
    _same({n: d[n].cpu().numpy() for n in util.COMPARED}, ref)
    extra = ("pfsd", "pextra")
    _same({n: g[n].cpu().numpy() for n in extra}, dref, extra, _nan_columns(ref))
    assert int(cnt.item()) == nw
