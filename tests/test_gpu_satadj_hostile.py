"""CLOUD_SATADJ's fast pass on inputs outside its checked ranges: the points it
reports are computed again with IEEE division, so the kernel equals the host
build of the plain point code on every point (GPU test)."""
import numpy as np
import pytest

from openifs_b200 import cloudsc, fields, inputs
from tests import util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nproma,nblk,cut", [(1, 40, 0), (33, 7, 5)])
def test_points_outside_the_ranges(cuda, nproma, nblk, cut):
    import torch
    p, _ = util.params()
    arrs = inputs.generate_satadj(nblk, nproma, p, seed=91)
    rng = np.random.default_rng(92)
    bad = np.array([0.0, 1e-300, 5e-324, -1e-290, 1e-80, 1e30, 1e80, -1e300, np.inf, np.nan])
    for n in fields.SATADJ_INPUTS:
        if n != "paph":
            x = arrs[n].reshape(-1)
            i = rng.choice(x.size, max(1, x.size // 100), replace=False)
            x[i] = rng.choice(bad, i.size)
    arrs["pt"][0] = rng.uniform(60.0, 160.0, arrs["pt"][0].shape)
    arrs["pap"][1] = 10.0 ** rng.uniform(-4.0, 8.0, arrs["pap"][1].shape)
    ngptot = nproma * nblk - cut
    ref, nw = util.run_hostemu_satadj(p, arrs, nproma, nblk, ngptot)
    cloudsc.setup(p)
    d = {k: torch.from_numpy(v.copy()).cuda() for k, v in arrs.items()}
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    cloudsc.satadj_batched(p, d, nproma, util.KLEV, nblk, ngptot, util.PTSPHY, counter=cnt)
    torch.cuda.synchronize()
    for n in fields.SATADJ_OUTPUTS:
        assert np.array_equal(d[n].cpu().numpy(), ref[n], equal_nan=True), n
    assert int(cnt.item()) == nw
