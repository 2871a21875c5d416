"""The surrogate's GPU kernels: gradients of the whole network (tcgen05
forward, backward-data and weight-gradient GEMMs, loss kernel)
against the float64 CPU reference (tests/surrogate_ref.py, itself checked
against finite differences) on identical bf16-rounded weights and inputs;
a short training run that must lower the loss; and the guarded inference
path: exact water/enthalpy closure of every surrogate column and FP64
results on every flagged column."""
import numpy as np
import pytest

from openifs_b200 import cloudsc, fields, inputs, surrogate as S
from tests import surrogate_ref as R
from tests import util

pytestmark = pytest.mark.gpu


def _bf(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x)).float().bfloat16().double().numpy()


@pytest.mark.parametrize("width", [64, 128])
def test_gradients_match_cpu_reference(cuda, width):
    import torch
    rng = np.random.default_rng(11)
    P = R.random_params(width, rng)
    for k in list(P):
        if k.startswith("w"):
            P[k] = _bf(P[k])
    x0, tgt = R.random_batch(2, rng)
    x0 = _bf(x0)
    loss_ref, G = R.loss_and_grad(P, x0, tgt)

    net = S.Net(width)
    for i in range(1, 6):
        net.p[i] = torch.from_numpy(P[f"w{i}"]).float().cuda()
        net.b[i] = torch.from_numpy(P[f"b{i}"]).float().cuda()
        net.g[i].zero_()
        net.gb[i] = torch.zeros_like(net.b[i])
    net.sync_bf16()
    rows = x0.shape[0]
    B = net.buffers(rows)
    B["x0"].copy_(torch.from_numpy(x0).bfloat16())
    B["tb"].copy_(torch.from_numpy(tgt).float())
    net.forward(B, rows)
    w = np.ones(16, np.float32)
    L = S._lib()
    S._ok(L.cs_loss(B["y"].data_ptr(), B["tb"].data_ptr(), rows, S.LP, S.KLEV, w.ctypes.data, 2,
                    B["dy"].data_ptr(), B["loss"].data_ptr(), S._stream()), "cs_loss")
    net.backward(B, rows)
    torch.cuda.synchronize()
    loss = float(B["loss"].item())
    assert abs(loss - loss_ref) < 2e-2 * loss_ref, (loss, loss_ref)
    for i in range(1, 6):
        g = net.g[i].double().cpu().numpy()
        r = G[f"w{i}"]
        rel = np.linalg.norm(g - r) / np.linalg.norm(r)
        assert rel < 5e-2, (i, rel)
        gb = net.gb[i].double().cpu().numpy()
        relb = np.linalg.norm(gb - G[f"b{i}"]) / np.linalg.norm(G[f"b{i}"])
        assert relb < 5e-2, (i, relb)


@pytest.mark.parametrize("n,k,taps,rows", [(128, 128, 5, 20_000), (128, 128, 1, 7_777), (64, 128, 1, 9_000),
                                           (64, 64, 5, 12_345), (128, 64, 5, 3_001), (64, 64, 1, 100)])
def test_weight_gradient_gemm(cuda, n, k, taps, rows):
    """The tensor-core weight gradient dW[t][n][k] += sum_r dZ[r][n] X[r+t-taps/2][k]
    (MN-major operands, split over row chunks, f32 reductions into dW)
    against float64 sums of the same bf16 values: rows shifted past either
    end count as zero, dW accumulates onto what it holds, the error flag
    stays clear."""
    import torch
    rng = np.random.default_rng(rows + n + k + taps)
    dz = torch.from_numpy(rng.standard_normal((rows, n)).astype(np.float32)).bfloat16().cuda()
    x = torch.from_numpy(rng.standard_normal((rows, k)).astype(np.float32)).bfloat16().cuda()
    init = rng.standard_normal((taps, n, k)).astype(np.float32)
    dw = torch.from_numpy(init).cuda()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    L = S._lib()
    rc = L.cs_wgrad_tc(dz.data_ptr(), x.data_ptr(), rows, n, k, taps, dw.data_ptr(), err.data_ptr(), S._stream())
    assert rc == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    D = dz.double().cpu().numpy()
    X = x.double().cpu().numpy()
    ref = init.astype(np.float64)
    for t in range(taps):
        s = t - taps // 2
        xs = np.zeros_like(X)
        if s >= 0:
            xs[:rows - s] = X[s:]
        else:
            xs[-s:] = X[:rows + s]
        ref[t] += D.T @ xs
    got = dw.double().cpu().numpy()
    scale = np.sqrt(rows)
    assert np.abs(got - ref).max() <= 1e-4 * scale, np.abs(got - ref).max()


def _wgrad(dz, x, taps, dw, db):
    L = S._lib()
    S._ok(L.cs_wgrad(dz.data_ptr(), x.data_ptr(), dz.shape[0], dz.shape[1], x.shape[1], taps, dw.data_ptr(),
                     db.data_ptr(), S._stream()), "cs_wgrad")


@pytest.mark.parametrize("n,k,taps,rows", [(128, 128, 5, 20_000), (128, 128, 1, 7_777), (64, 128, 1, 9_000),
                                           (64, 64, 5, 12_345), (128, 64, 5, 3_001), (64, 64, 1, 100), (64, 64, 5, 100),
                                           (128, 128, 5, 1), (128, 128, 5, 513), (64, 128, 1, 64)])
def test_bias_gradient(cuda, n, k, taps, rows):
    """cs_wgrad's db, the column sums of dZ shared by the taps' CTAs (down to
    fewer row blocks than taps), against float64 sums of the same bf16 values;
    it accumulates onto what db holds, and dW is that of cs_wgrad_tc.  The sums
    are about sqrt(rows); f32 sums of up to a few thousand of them are off by
    less than 1e-6 of that."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(rows + n)
    dz = torch.randn(rows, n, generator=g, device="cuda").bfloat16()
    x = torch.randn(rows, k, generator=g, device="cuda").bfloat16()
    init = torch.randn(n, generator=g, device="cuda")
    db, dw, dw2 = init.clone(), torch.zeros(taps, n, k, device="cuda"), torch.zeros(taps, n, k, device="cuda")
    _wgrad(dz, x, taps, dw, db)
    assert S._lib().cs_wgrad_tc(dz.data_ptr(), x.data_ptr(), rows, n, k, taps, dw2.data_ptr(), None, S._stream()) == 0
    ref = init.double() + dz.double().sum(0)
    assert (db.double() - ref).abs().max().item() <= 4e-6 * np.sqrt(rows)
    assert (dw - dw2).abs().max().item() <= 1e-5 * np.sqrt(rows)


@pytest.mark.parametrize("n,k,taps,cols", [(128, 128, 5, 333), (128, 128, 5, 512), (128, 128, 1, 1000), (64, 64, 5, 1000)])
def test_weight_gradient_precision(cuda, n, k, taps, cols):
    """Over the batches training uses: the relative error of dW (2-norm) against
    64-bit sums grows with the rows a CTA accumulates, ceil(rows / CTAs per tap)
    of them: 1.05e-9 a row measured, 5e-7 for the f32 rounding of the rest; a
    third more allowed.  db, summed by all taps' CTAs, stays below 6e-7."""
    import torch
    rows = cols * S.LP
    g = torch.Generator(device="cuda").manual_seed(cols)
    dz = torch.randn(rows, n, generator=g, device="cuda").bfloat16()
    x = torch.randn(rows, k, generator=g, device="cuda").bfloat16()
    dw, db = torch.zeros(taps, n, k, device="cuda"), torch.zeros(n, device="cuda")
    _wgrad(dz, x, taps, dw, db)
    D, X = dz.double(), x.double()
    ref = torch.zeros(taps, n, k, dtype=torch.float64, device="cuda")
    for t in range(taps):
        s = t - taps // 2
        lo, hi = max(0, -s), min(rows, rows - s)
        ref[t] = D[lo:hi].T @ X[lo + s:hi + s]
    rel = ((dw.double() - ref).norm() / ref.norm()).item()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    chunk = max(512, rows / (2 * sms / taps))
    assert rel <= (5e-7 + 1.05e-9 * chunk) * 4 / 3, rel
    assert ((db.double() - D.sum(0)).norm() / D.sum(0).norm()).item() <= 6e-7


def test_weight_gradient_rejects_bad_shapes(cuda):
    import torch
    L = S._lib()
    a = torch.zeros(256, 128, dtype=torch.bfloat16, device="cuda")
    dw = torch.zeros(128, 128, device="cuda")
    assert L.cs_wgrad_tc(a.data_ptr(), a.data_ptr(), 256, 96, 128, 1, dw.data_ptr(), None, None) != 0
    assert L.cs_wgrad_tc(a.data_ptr(), a.data_ptr(), 256, 128, 128, 3, dw.data_ptr(), None, None) != 0
    assert L.cs_wgrad_tc(a.data_ptr() + 2, a.data_ptr(), 256, 128, 128, 1, dw.data_ptr(), None, None) != 0


@pytest.mark.parametrize("width,rows", [(128, 5 * 144 + 37), (64, 3 * 144), (128, 64)])
def test_fused_mlp_head_equals_two_kernels(cuda, width, rows):
    """cs_mlp_head (the MLP layer's SiLU output kept in shared memory and fed
    to the output head's MMAs) gives the two-kernel result bit for bit:
    cs_conv_gemm with the SiLU epilogue, then with the linear f32 one; the
    padding rows of the column layout zero in both; the error word clear."""
    import torch
    from openifs_b200 import tcgemm as E
    rng = np.random.default_rng(width + rows)
    a = torch.from_numpy(rng.standard_normal((rows, width)).astype(np.float32)).bfloat16().cuda()
    w1 = torch.from_numpy(0.1 * rng.standard_normal((1, width, width)).astype(np.float32)).bfloat16().cuda()
    w2 = torch.from_numpy(0.1 * rng.standard_normal((1, 64, width)).astype(np.float32)).bfloat16().cuda()
    b1 = torch.from_numpy(rng.standard_normal(width).astype(np.float32)).cuda()
    b2 = torch.from_numpy(rng.standard_normal(64).astype(np.float32)).cuda()
    h = torch.empty(rows, width, dtype=torch.bfloat16, device="cuda")
    y_ref = torch.full((rows, 64), 7.0, device="cuda")
    E.conv_gemm(a, w1, E.EPI_SILU, width, 1, S.LP, S.KLEV, b1, h)
    E.conv_gemm(h, w2, E.EPI_LINEAR_F32, 64, 1, S.LP, S.KLEV, b2, outf=y_ref)
    y = torch.full((rows, 64), 7.0, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    E.mlp_head(a, w1, b1, w2, b2, y, S.LP, S.KLEV, err=err)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert torch.equal(y, y_ref)
    pos = torch.arange(rows, device="cuda") % S.LP
    pad = (pos < 2) | (pos >= 2 + S.KLEV)
    assert bool((y[pad] == 0).all()) and float(y[~pad].abs().max()) > 0


@pytest.fixture(scope="module")
def small_data(cuda):
    p, _ = util.params()
    data = S.Dataset(p, nchunks=1, nblk=48, nproma=128, seed0=77, log=None)
    norm, scale = data.normalisation()
    data.apply_scale(scale)
    return p, data, norm, scale


def test_training_lowers_loss(small_data):
    p, data, norm, scale = small_data
    net = S.Net(128, seed=1)
    net.norm, net.out_scale = norm, scale
    hist = S.train(net, data, steps=400, nb=64, lr=2e-3, warmup=50, log=None, log_every=100)
    first, last = hist[0][1], hist[-1][1]
    # targets are normalised to unit RMS: predicting zero tendencies scores 1.0
    assert last < 0.5 * first and last < 0.5, hist


def test_guarded_inference_closes_budgets(small_data):
    import torch
    p, data, norm, scale = small_data
    net = S.Net(128, seed=1)
    net.norm, net.out_scale = norm, scale
    S.train(net, data, steps=300, nb=64, lr=2e-3, warmup=50, log=None, log_every=100)
    nproma, nblk = 128, 8
    host = inputs.generate(nblk, nproma, p, seed=91)
    cloudsc.setup(p)
    ref = {k: torch.from_numpy(v).cuda() for k, v in host.items()}
    cloudsc.cloudsc_batched(p, ref, nproma, S.KLEV, nblk, nproma * nblk, util.PTSPHY)
    dev = {k: torch.from_numpy(v).cuda() for k, v in host.items()}
    run = S.Runner(net, p, nproma, nblk, capacity=256, neg_tol=0.05, closure_tol=0.5, spread_tol=0.25)
    b = run.prepare(dev)
    run.run(b)
    run.run(b)  # a second run on the same batch sees the same input
    torch.cuda.synchronize()
    nflag = int(b.nflag.item())
    flagged = set(b.flagged[:min(nflag, run.cap)].cpu().tolist())
    out = {k: v.cpu().numpy() for k, v in dev.items()}
    r = {k: v.cpu().numpy() for k, v in ref.items()}
    ncol = nproma * nblk
    cols = np.arange(ncol)
    ib, jl = cols // nproma, cols % nproma
    # flagged columns carry the FP64 results bit for bit
    for n in ["tendency_loc_t", "tendency_loc_q", "pfplsl", "pfsqlf"]:
        for c in list(flagged)[:64]:
            assert np.array_equal(out[n][c // nproma, ..., c % nproma], r[n][c // nproma, ..., c % nproma]), n
    # water and enthalpy budgets of every column (those of cs_post)
    dp = np.diff(host["paph"], axis=1)
    g = p.rg
    L = out["tendency_loc_cld"]
    lev = np.arange(S.KLEV)
    loop = ((lev >= p.ncldtop - 1) & (lev < S.KLEV - 1))[None, :, None]
    active = loop & (out["plude"] != 0.0)
    sl = (host["pludeli"][:, 0] * active).sum(1)
    si = (host["pludeli"][:, 1] * active).sum(1)
    sr = (host["psnde"][:, 0] * loop).sum(1)
    ss = (host["psnde"][:, 1] * loop).sum(1)
    w_l = (dp / g * (out["tendency_loc_q"] + L[:, :4].sum(1))).sum(1)
    w_r = sl + si + sr + ss - out["pfplsl"][:, -1] - out["pfplsn"][:, -1]
    w_s = (np.abs(dp / g * out["tendency_loc_q"])).sum(1) + np.abs(w_r) + 1e-30
    e_l = (dp / g * (out["tendency_loc_t"] - p.ralvdcp * (L[:, 0] + L[:, 2]) - p.ralsdcp * (L[:, 1] + L[:, 3]))).sum(1)
    e_r = p.ralvdcp * (out["pfplsl"][:, -1] - sl - sr) + p.ralsdcp * (out["pfplsn"][:, -1] - si - ss)
    e_s = (np.abs(dp / g * out["tendency_loc_t"])).sum(1) + np.abs(e_r) + 1e-30
    wr = (np.abs(w_l - w_r) / w_s).reshape(-1)
    er = (np.abs(e_l - e_r) / e_s).reshape(-1)
    net_cols = np.ones(ncol, bool)
    net_cols[list(flagged)] = False
    # the network's columns close exactly (cs_post's shifts)
    assert wr[net_cols].max() < 1e-10, wr[net_cols].max()
    assert er[net_cols].max() < 1e-10, er[net_cols].max()
    # flagged columns carry CLOUDSC's own closure: its detrainment enters the
    # condensates with the scheme's phase split while this budget counts
    # PLUDELI, about 1e-9 relative at worst by this measure
    if flagged:
        assert wr[~net_cols].max() < 1e-8, wr[~net_cols].max()
        assert er[~net_cols].max() < 1e-10, er[~net_cols].max()
    # PLUDE as CLOUDSC writes it, on every column
    assert np.array_equal(out["plude"], r["plude"])


def test_inference_inputs_match_training_inputs(cuda):
    """The inference input x0 (cs_prep_inputs: normalised features, then the
    5-level window) is bit-identical to the training input built from the raw
    features of the same columns (cs_raw_features + cs_prep_batch), and every
    window slot holds the feature of the level it names."""
    import ctypes
    import torch
    p, _ = util.params()
    nproma, nblk = 64, 3
    ncol, rows = nproma * nblk, nproma * nblk * S.LP
    host = inputs.generate(nblk, nproma, p, seed=5)
    dev = {k: torch.from_numpy(v).cuda() for k, v in host.items()}
    colsum = torch.empty(ncol, S.KLEV, 2, device="cuda")
    c = S.columns(dev, nproma, nblk, colsum, p)
    L, s = S._lib(), S._stream()
    net = S.Net.load(S.WEIGHTS)
    S._ok(L.cs_column_sums(ctypes.byref(c), S._p(colsum), s), "cs_column_sums")
    fbuf = torch.empty(rows, 32, dtype=torch.bfloat16, device="cuda")
    x0 = torch.full((rows, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    S._ok(L.cs_prep_inputs(ctypes.byref(c), ctypes.byref(net.norm), S._p(fbuf), S._p(x0), s), "cs_prep_inputs")
    feat = torch.empty(rows, S.FSTRIDE, device="cuda")
    S._ok(L.cs_raw_features(ctypes.byref(c), S._p(feat), s), "cs_raw_features")
    tgt = torch.zeros(rows, 16, device="cuda")
    order = torch.arange(ncol, dtype=torch.int32, device="cuda")
    x0t = torch.full_like(x0, float("nan"))
    tb = torch.empty(rows, 16, device="cuda")
    S._ok(L.cs_prep_batch(S._p(feat), S._p(tgt), S._p(order), ncol, S.LP, S.KLEV, ctypes.byref(net.norm),
                          S._p(x0t), S._p(tb), s), "cs_prep_batch")
    torch.cuda.synchronize()
    assert torch.equal(x0.view(torch.int16), x0t.view(torch.int16))
    fb = fbuf.view(ncol, S.LP, 32)[..., :25]
    want = torch.zeros(ncol, S.LP, 128, dtype=torch.bfloat16, device="cuda")
    for tap in range(5):
        lo, hi = max(0, 2 - tap), min(S.KLEV, S.KLEV + 2 - tap)  # levels k whose k + tap - 2 exists
        want[:, 2 + lo:2 + hi, 25 * tap:25 * tap + 25] = fb[:, lo + tap:hi + tap]
    assert torch.equal(x0.view(ncol, S.LP, 128).view(torch.int16), want.view(torch.int16))


def test_trained_network_beats_the_methods_without_it(cuda):
    """What training buys, on 1,024 columns of a seed no training chunk used:
    the committed width-128 network (no column flagged, so every output is the
    network's, after the guard's closure shifts) against the same network
    untrained and against each level's mean FP64 tendency over these very
    columns (a climatology that has seen the answers).  Relative RMS errors
    against the FP64 kernel; the climatology scores about 0.94-0.99 here."""
    import torch
    p, _ = util.params()
    nproma, nblk = 128, 8
    host = inputs.generate(nblk, nproma, p, seed=4242)
    cloudsc.setup(p)
    ref = {k: torch.from_numpy(v).cuda() for k, v in host.items()}
    cloudsc.cloudsc_batched(p, ref, nproma, S.KLEV, nblk, nproma * nblk, util.PTSPHY)
    trained = S.Net.load(S.WEIGHTS)
    untrained = S.Net(trained.width, seed=3)
    untrained.norm, untrained.out_scale = trained.norm, trained.out_scale

    def predict(net):
        dev = {k: torch.from_numpy(v).cuda() for k, v in host.items()}
        run = S.Runner(net, p, nproma, nblk, capacity=nproma, neg_tol=1e30, closure_tol=1e30, spread_tol=1e30)
        b = run.prepare(dev)
        run.run(b)
        torch.cuda.synchronize()
        assert int(b.nflag.item()) == 0
        return dev

    def rel(g, r):
        return float((g - r).pow(2).mean().sqrt() / r.pow(2).mean().sqrt())

    out_t, out_u = predict(trained), predict(untrained)
    for n, m in [("tendency_loc_t", None), ("tendency_loc_q", None), ("tendency_loc_a", None),
                 ("tendency_loc_cld", 0), ("tendency_loc_cld", 1), ("tendency_loc_cld", 2), ("tendency_loc_cld", 3)]:
        pick = (lambda a: a) if m is None else (lambda a, m=m: a[:, m])
        r = pick(ref[n])
        clim = r.mean(dim=(0, 2), keepdim=True).expand_as(r)
        e_t, e_u, e_c = rel(pick(out_t[n]), r), rel(pick(out_u[n]), r), rel(clim, r)
        assert e_t < 0.5 * e_c and e_t < 0.5 * e_u, (n, m, e_t, e_u, e_c)
