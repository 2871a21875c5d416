"""The column kernels' branch-free square root (csqrt in cloudsc_column.cuh)
against IEEE square root on the host: bit for bit wherever it does not report,
and it reports only what its rounding check cannot confirm."""
import numpy as np
import pytest

from openifs_b200 import cloudsc

pytestmark = pytest.mark.gpu


def _bits(x):
    return np.ascontiguousarray(x, dtype=np.float64).view(np.int64)


def test_square_root(cuda):
    import torch
    rng = np.random.default_rng(31)
    n = 2_000_000
    e = rng.integers(-190, 191, n)
    u = rng.uniform(1, 2, n)
    near = lambda x: (_bits(x) + rng.integers(-4, 5, x.size)).view(np.float64)
    r = rng.uniform(1, 2, n)
    # squares of 27-bit roots and of midpoints between doubles, and their neighbours
    short = np.round(r * 2 ** 26) / 2 ** 26
    mid = (r.astype(np.longdouble) + np.longdouble(2.0) ** -53) ** 2
    x = np.concatenate([u * np.ldexp(1.0, e), np.exp(rng.normal(0, 12, n)), near(np.ldexp(1.0, e)),
                        near(np.nextafter(2.0, 0.0) * np.ldexp(1.0, e)), near(short * short), near(mid.astype(np.float64)),
                        mid.astype(np.float64) * np.ldexp(1.0, 2 * (e // 2))])
    y, bad = cloudsc.sqrt_check(torch.from_numpy(x).cuda())
    torch.cuda.synchronize()
    y, bad = y.cpu().numpy(), bad.cpu().numpy() != 0
    same = _bits(y) == _bits(np.sqrt(x))
    assert same[~bad].all(), x[~bad & ~same][:4]
    ones = (_bits(x) & ((1 << 52) - 1)) == (1 << 52) - 1
    # reports: every all-ones significand, and otherwise only roots within
    # 2^-52 ulp of a rounding midpoint (those constructed in the later sets)
    assert bad[ones].all()
    assert not (bad & ~ones)[:2 * n].any()
    y, bad = cloudsc.sqrt_check(torch.tensor([-1.0, float("nan"), float("inf"), -1e-30], dtype=torch.float64, device="cuda"))
    assert bad.cpu().numpy().all()
    with pytest.raises(cloudsc.CloudscError):
        cloudsc.sqrt_check(torch.ones(3, device="cuda"))
