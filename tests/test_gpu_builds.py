"""Every build of the optional forms and of the single-precision interface that a
call can be given, set or by size, against the oracle bit for bit (GPU tests).
The forms have fewer builds than the plain ones: a schedule names one of six
variants, and the call runs the form's own build of it or the one it maps to."""
import numpy as np
import pytest

from openifs_b200 import cloudsc, fields, inputs
from tests import util

pytestmark = pytest.mark.gpu

NPROMA, NBLK = 64, 9
NGPTOT = NPROMA * NBLK - 9
# by size (256-thread build), then every variant at its largest CTA and a small one
SCHEDULES = [None, (0, 640, 0), (1, 448, 0), (1, 128, 0), (2, 384, 0), (2, 96, 2), (3, 256, 0), (4, 256, 0), (5, 128, 3)]


@pytest.fixture(params=SCHEDULES, ids=lambda s: "by_size" if s is None else "v%d_t%d_c%d" % s)
def schedule(request):
    before = {pr: cloudsc.get_schedule(pr) for pr in (cloudsc.FP64, cloudsc.MIXED, cloudsc.PHYS32)}
    assert all(t == 0 for _, t, _ in before.values()), "an earlier test left a schedule set"
    try:
        for pr in before:
            if request.param:
                cloudsc.set_schedule(pr, *request.param)
        yield request.param
    finally:
        for pr, s in before.items():
            cloudsc.set_schedule(pr, *s)


@pytest.fixture(scope="module")
def oracle_of():
    done = {}

    def get(opt):
        if opt not in done:
            p0, po0 = util.params()
            if opt == "budgets":
                p, po = (util.with_flags(x, util.BUDGET_CASES[-1]) for x in (p0, po0))
            else:
                p, po = (util.opt_params(x, opt) for x in (p0, po0))
            arrs = inputs.generate(NBLK, NPROMA, p, seed=67)
            diag = inputs.generate_diag(arrs, NPROMA, fields.budget_fields_needed(p) + 1, seed=67)
            done[opt] = (p, arrs, diag) + util.run_oracle_diag(po, arrs, diag, NPROMA, NBLK, NGPTOT)
        return done[opt]
    return get


@pytest.mark.parametrize("opt", ["budgets", "spp", "all+budgets"])
def test_optional_forms(cuda, oracle_of, schedule, opt):
    import torch
    p, arrs, diag, ref, dref, nw = oracle_of(opt)
    try:
        cloudsc.setup(p)
        d = {k: torch.from_numpy(v).cuda() for k, v in arrs.items()}
        g = {k: torch.from_numpy(v).cuda() for k, v in diag.items()}
        cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
        cloudsc.cloudsc_batched_diag(p, d, g, NPROMA, util.KLEV, NBLK, NGPTOT, util.PTSPHY, counter=cnt)
        torch.cuda.synchronize()
    finally:
        cloudsc.setup(util.params()[0])
    for n in util.COMPARED:
        a, b = (util.defined(n, util._valid_cols(x, NGPTOT, NPROMA)) for x in (d[n].cpu().numpy(), ref[n]))
        assert np.array_equal(a, b), n
    for n in ("pfsd", "pextra"):
        assert np.array_equal(g[n].cpu().numpy(), dref[n]), n
    assert int(cnt.item()) == nw


@pytest.fixture(scope="module")
def single_oracle():
    p, po = util.params()
    sp = fields.to_single(inputs.generate(NBLK, NPROMA, p, seed=68))
    wide = {k: (v.astype(np.float64) if v.dtype == np.float32 else v.copy()) for k, v in sp.items()}
    return (p, sp) + util.run_oracle(po, wide, NPROMA, NBLK, NGPTOT)


def _single(p, sp, precision):
    import torch
    cloudsc.setup(p)
    d = {k: torch.from_numpy(v).cuda() for k, v in sp.items()}
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    cloudsc.cloudsc_batched_sp(p, d, NPROMA, util.KLEV, NBLK, NGPTOT, util.PTSPHY, precision=precision, counter=cnt)
    torch.cuda.synchronize()
    out = {n: util.defined(n, util._valid_cols(d[n].cpu().numpy(), NGPTOT, NPROMA)) for n in util.COMPARED}
    return out, int(cnt.item())


def test_single_precision_fp64(cuda, single_oracle, schedule):
    p, sp, ref, nw = single_oracle
    got, nwg = _single(p, sp, cloudsc.FP64)
    for n in util.COMPARED:
        b = util.defined(n, util._valid_cols(ref[n].astype(np.float32), NGPTOT, NPROMA))
        assert np.array_equal(got[n], b), n
    assert nwg == nw


@pytest.mark.parametrize("precision", [cloudsc.MIXED, cloudsc.PHYS32])
def test_single_precision_fp32_forms(cuda, single_oracle, schedule, precision):
    """The FP32 forms take the GPU's powf and expf: every build gives the bits of
    the call by size."""
    p, sp, _, _ = single_oracle
    got, nw = _single(p, sp, precision)
    with cloudsc.schedule_by_size():
        ref, nwr = _single(p, sp, precision)
    for n in util.COMPARED:
        assert np.array_equal(got[n], ref[n]), n
    assert nw == nwr
