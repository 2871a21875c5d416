"""Performance cases: the calls an IFS-style physics driver makes of this framework, over the range of sizes it is used at.

Every case is a call (or a training loop) through the package's public entry points on inputs drawn on the GPU from the
distributions documented in openifs_b200/inputs.py.  `exact` restates each scheme in plain torch, in double precision and
vectorised over the columns, for the outputs of one pass.

Sizes: the 3,200-column CPU-scale call (100 blocks of 32) and the 262,144-column call (2,048 blocks of 128) are the
repository's own two CLOUDSC workloads; 60, 91 and 137 levels and the ragged last blocks are its tests' grids; the
surrogate's width 128, 512-column training batch and 1/16 fallback capacity are its defaults.
"""
import math
import os
import types

import numpy as np
import torch

from openifs_b200 import cloudsc, fields, inputs, surrogate

PTSPHY = 3600.0
F64 = torch.float64


# ------------------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one NPROMA block through CLOUDSC's own argument list on host arrays: what the OpenMP block loop of the physics
        # driver calls, where copies, launches and the walk down one column decide
        dict(name="block 32", kind="block", nproma=32, ncol=32, klev=137),
        # the CPU-scale call on device arrays: a few columns per SM
        dict(name="fp64 3200", kind="cloudsc", nproma=32, ncol=3200, klev=137, precision=0),
        # a limited-area or coarse global task: ragged blocks, another vertical grid, less than one full wave of columns
        dict(name="fp64 20701 L91", kind="cloudsc", nproma=24, ncol=20701, klev=91, precision=0),
        # the headline workload
        dict(name="fp64 262144", kind="cloudsc", nproma=128, ncol=262144, klev=137, precision=0),
        # the mixed-precision form, between one and two waves of columns
        dict(name="mixed 90005", kind="cloudsc", nproma=64, ncol=90005, klev=137, precision=1),
        # the single-precision build's arrays (JPRB = REAL(4))
        dict(name="single 65536", kind="single", nproma=64, ncol=65536, klev=137, precision=0),
        # an ensemble member: SPP perturbations and the cloud-inhomogeneity paths on
        dict(name="spp 24576", kind="spp", nproma=96, ncol=24576, klev=137),
        # all blocks from pinned host memory, copies pipelined with the kernel
        dict(name="host 8192", kind="host", nproma=128, ncol=8192, klev=137, precision=0),
        # the saturation adjustment that runs before CLOUDSC
        dict(name="satadj 100000", kind="satadj", nproma=100, ncol=100000, klev=137),
        # STATE_INCREMENT after CLOUDSC: T, q, a and the four condensates
        dict(name="increment 65536", kind="increment", nproma=128, ncol=65536, klev=137),
        # guarded surrogate inference with the FP64 fallback on the flagged columns
        dict(name="surrogate 49152", kind="surrogate", nproma=128, ncol=49152, klev=137, width=128),
        # surrogate training: forward, loss, backward and AdamW on batches of 512 columns
        dict(name="train 512", kind="train", ncol=512, width=128, steps=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block", "cloudsc", "cloudsc", "mixed", "single", "spp", "host", "satadj", "increment", "surrogate", "train"])
    nproma = rng.choice([16, 24, 32, 37, 48, 64, 75, 96, 128, 160])
    klev = rng.choice([60, 91, 137, 137, 137])
    if kind == "block":
        nproma = _log(rng, 8, 256)
        return dict(kind=kind, nproma=nproma, ncol=nproma, klev=klev)
    if kind == "cloudsc":
        return dict(kind=kind, nproma=nproma, ncol=_log(rng, 500, 240000), klev=klev, precision=0)
    if kind == "mixed":
        return dict(kind="cloudsc", nproma=nproma, ncol=_log(rng, 2000, 240000), klev=klev, precision=rng.choice([1, 1, 2]))
    if kind == "single":
        return dict(kind=kind, nproma=nproma, ncol=_log(rng, 2000, 240000), klev=klev, precision=rng.choice([0, 0, 1, 2]))
    if kind == "spp":
        return dict(kind=kind, nproma=nproma, ncol=_log(rng, 1000, 60000), klev=klev)
    if kind == "host":
        return dict(kind=kind, nproma=nproma, ncol=_log(rng, 500, 10000), klev=klev, precision=0)
    if kind in ("satadj", "increment"):
        return dict(kind=kind, nproma=nproma, ncol=_log(rng, 1000, 200000), klev=klev)
    if kind == "surrogate":
        nproma = rng.choice([32, 64, 128])
        return dict(kind=kind, nproma=nproma, ncol=nproma * max(1, _log(rng, 1500, 50000) // nproma), klev=137,
                    width=rng.choice([64, 128, 128]))
    return dict(kind="train", ncol=_log(rng, 100, 1000), width=rng.choice([64, 128, 128]), steps=4)


def _nblk(case):
    return -(-case["ncol"] // case["nproma"])


def _params(case):
    p = cloudsc.default_params(PTSPHY, inputs.ncldtop_for(case.get("klev", 137)))
    if case["kind"] == "spp":  # all eight perturbations (field pointers 1..9) and both inhomogeneity paths
        p.lspp = p.lcloud_inhomog = p.lrad_cloud_inhomog = 1
        p.spp_nrftotal = 9
        for n in range(8):
            p.spp_on[n], p.spp_mp[n] = 1, n + 1
            sigma = 0.25 + 0.05 * n
            p.spp_mu[2 * n] = p.spp_mu[2 * n + 1] = -0.5 * sigma * sigma
            p.spp_xmag[2 * n] = p.spp_xmag[2 * n + 1] = sigma
    return p


# ---------------------------------------------------------------------------------------------------------------- inputs
def _state(case, seed, p):
    """The generator of openifs_b200/inputs.py on the GPU: batched arrays (NGPBLKS, ..., NPROMA), outputs zero."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    nb, np_, kl = _nblk(case), case["nproma"], case["klev"]
    one, lev = (nb, 1, np_), (nb, kl, np_)

    def uni(lo, hi, shape=lev):
        return torch.rand(shape, generator=g, device="cuda", dtype=F64) * (hi - lo) + lo

    def normal(sd, shape=lev):
        return torch.randn(shape, generator=g, device="cuda", dtype=F64) * sd

    def some(prob, shape=lev):
        return torch.rand(shape, generator=g, device="cuda") < prob

    out = fields.alloc(nb, np_, kl, alloc_fn=lambda s, dt: torch.zeros(
        s, dtype=F64 if np.dtype(dt) == np.float64 else torch.int32, device="cuda"))
    ha, hb = (torch.from_numpy(x.copy()).cuda().view(1, -1, 1) for x in inputs.hybrid_ab(kl))
    ps = uni(98000.0, 103000.0, one)
    paph = ha + hb * ps
    pap = 0.5 * (paph[:, :-1] + paph[:, 1:])
    t = torch.clamp(uni(280.0, 300.0, one) * (pap / ps) ** (p.rd * 0.0065 / p.rg), min=216.65) + normal(1.5)
    x = (t.clamp(p.rtice, p.rtwat) - p.rtice) * p.rtwat_rtice_r
    alfa = torch.clamp(x * x, max=1.0)
    ew = p.r2es * (alfa * torch.exp(p.r3les * (t - p.rtt) / (t - p.r4les)) +
                   (1 - alfa) * torch.exp(p.r3ies * (t - p.rtt) / (t - p.r4ies)))
    qsat = torch.clamp(ew / pap, max=0.5)
    q = uni(0.2, 1.05) * (qsat / (1 - p.retv * qsat))
    q = torch.where(pap < 10000.0, torch.minimum(q, 3e-6 * uni(0.8, 1.2)), q)
    top = (torch.arange(kl, device="cuda") < p.ncldtop - 1).view(1, -1, 1)
    warm = t > 273.0
    species = []
    for prob, none in ((0.5, t < 235.0), (0.5, warm), (0.35, None), (0.35, warm)):
        v = torch.clamp(torch.exp(math.log(1e-5) + normal(1.5)), max=5e-3)
        off = ~some(prob) | top if none is None else ~some(prob) | top | none
        species.append(v.masked_fill_(off, 0.0))
    out["pa"][:] = uni(0.0, 1.0).masked_fill_((species[0] <= 0) & (species[1] <= 0), 0.0)
    out["pt"][:], out["pq"][:], out["pap"][:], out["paph"][:] = t, q, pap, paph
    out["tendency_cml_t"][:], out["tendency_cml_a"][:] = normal(1e-4), normal(1e-5)
    out["tendency_cml_q"][:] = q * normal(1e-5)
    for m, v in enumerate(species):
        out["pclv"][:, m] = v
        out["tendency_cml_cld"][:, m] = v * normal(1e-5)
    out["pvfl"][:], out["pvfi"][:] = species[0] * normal(1e-5), species[1] * normal(1e-5)
    out["plsm"][:] = some(0.5, (nb, np_)).double()
    out["peis"][:] = uni(0.0, 15.0, (nb, np_))
    # convection on 30 % of the columns
    ldcum = some(0.3, one)
    r = uni(0.0, 1.0, one)
    ktype = torch.where(ldcum, torch.where(r < 0.5, 1, torch.where(r < 0.8, 2, 3)), 0)
    base = ps - uni(5000.0, 15000.0, one)
    ctop = torch.where(ktype == 1, uni(15000.0, 30000.0, one),
                       torch.where(ktype == 2, base - uni(10000.0, 25000.0, one), uni(40000.0, 60000.0, one)))
    m0 = uni(0.01, 0.1, one)
    inside = (pap > ctop) & (pap < base) & ldcum
    frac = (pap - ctop) / (base - ctop)
    pmfu = torch.where(inside, m0 * torch.sin(math.pi * frac), 0.0)
    mid = 0.5 * (ctop + base)
    down = (pap > mid) & (pap < ps) & ldcum
    out["pmfu"][:] = pmfu
    out["pmfd"][:] = torch.where(down, -0.3 * m0 * torch.sin(math.pi * (pap - mid) / (ps - mid)), 0.0)
    out["plu"][:] = torch.where(inside, uni(1e-4, 2e-3), 0.0)
    plude = torch.where(inside, torch.where(frac < 0.3, 0.2, 0.05) * pmfu * out["plu"], 0.0)
    out["plude"][:] = plude
    out["pludeli"][:, 0], out["pludeli"][:, 1] = plude * alfa, plude * (1 - alfa)
    out["psnde"][:, 0], out["psnde"][:, 1] = 0.1 * plude * alfa, 0.1 * plude * (1 - alfa)
    out["ldcum"][:], out["ktype"][:] = ldcum[:, 0].int(), ktype[:, 0].int()
    return out, uni, normal


def _satadj_state(case, seed, p):
    """CLOUD_SATADJ's arrays from the same state, with the fields only that scheme reads."""
    s, uni, normal = _state(case, seed, p)
    lev = s["pt"].shape
    a = {n: s[n] for n in ("pap", "paph", "pt", "pq", "pa", "tendency_cml_t", "tendency_cml_q", "tendency_cml_a")}
    for m, n in enumerate("li"):
        a["p" + n] = s["pclv"][:, m].contiguous()
        a["tendency_cml_" + n] = s["tendency_cml_cld"][:, m].contiguous()
    a["phrsw"], a["phrlw"] = uni(0.0, 2e-5), normal(1e-5) - 2e-5
    a["tendency_vdf_t"], a["tendency_vdf_q"] = normal(1e-4), s["pq"] * normal(1e-5)
    a["pludeli"] = s["pludeli"]
    a["pludeli"][:, 2], a["pludeli"][:, 3] = uni(0.0, 1.0) * s["plude"], 2500.0 * s["plude"] * normal(1.0)
    a["pvervel"] = normal(0.3)
    for n in fields.SATADJ_OUTPUTS:
        a[n] = torch.zeros(lev, dtype=F64, device="cuda")
    return a


def prepare(case, seed):
    kind, st = case["kind"], types.SimpleNamespace(case=case)
    st.p = p = _params(case)
    cloudsc.setup(p)
    if kind == "train":
        # 2,048 columns of training data: raw features and the FP64 scheme's tendencies
        st.net = surrogate.Net(case["width"], seed=seed)
        st.data = surrogate.Dataset(p, 1, nblk=16, nproma=128, seed0=seed % 100003, log=None)
        st.net.norm, st.net.out_scale = st.data.normalisation()
        st.data.apply_scale(st.net.out_scale)
        return st
    st.dims = (case["nproma"], case["klev"], _nblk(case), case["ncol"])
    if kind == "satadj":
        st.a = _satadj_state(case, seed, p)
        return st
    st.a, uni, normal = _state(case, seed, p)
    if kind == "increment":
        st.state = {"t": st.a["pt"], "q": st.a["pq"], "a": st.a["pa"], "cld": st.a["pclv"]}
        st.inc = {"t": st.a["tendency_cml_t"], "q": st.a["tendency_cml_q"], "a": st.a["tendency_cml_a"],
                  "cld": st.a["tendency_cml_cld"]}
        return st
    if kind == "surrogate":
        here = os.path.dirname(surrogate.__file__)
        st.net = surrogate.Net.load(os.path.join(here, "data", "surrogate_w%d.npz" % case["width"]))
        st.runner = surrogate.Runner(st.net, p, st.dims[0], st.dims[2], capacity=case["ncol"] / 16)
        st.batch = st.runner.prepare(st.a)
        return st
    if kind == "single":
        st.a = fields.to_single(st.a)
    if kind == "spp":
        nb, np_ = st.dims[2], st.dims[0]
        st.diag = {"pgaw": uni(1e-7, 3e-6, (nb, np_)), "pgp2dspp": normal(1.0, (nb, 9, np_)),
                   "pfsd": torch.zeros_like(st.a["pt"])}
    if kind == "host":
        st.a = {k: v.cpu().pin_memory() for k, v in st.a.items()}
    if kind == "block":
        st.a = {k: np.ascontiguousarray(v[0].cpu().numpy()) for k, v in st.a.items()}
    # PLUDE is read and written in place; each step of the model has new values there
    st.plude = st.a["plude"].copy() if kind == "block" else st.a["plude"].clone()
    return st


def run(st):
    kind, case = st.case["kind"], st.case
    if kind == "train":
        hist = surrogate.train(st.net, st.data, case["steps"], nb=case["ncol"], log=None, log_every=1)
        n = st.net
        return {"loss": torch.tensor([h[1] for h in hist], dtype=F64), "w": n.p, "b": n.b, "m": n.m, "v": n.v, "mb": n.mb, "vb": n.vb}
    if kind == "satadj":
        cloudsc.satadj_batched(st.p, st.a, *st.dims, PTSPHY)
        return {n: st.a[n] for n in fields.SATADJ_OUTPUTS}
    if kind == "increment":
        cloudsc.state_increment_batched(st.state, st.inc, *st.dims)
        return st.state
    if kind == "surrogate":
        st.runner.run(st.batch)
        out = {n: st.a[n] for n in SURROGATE_OUTPUTS}
        out["y"] = st.runner.B["y"]
        return out
    if kind == "block":
        np.copyto(st.a["plude"], st.plude)
        cloudsc.cloudsc_block(st.p, 1, st.dims[0], st.dims[0], st.dims[1], PTSPHY, st.a)
        return {n: st.a[n] for n in fields.OUTPUT_NAMES}
    st.a["plude"].copy_(st.plude)
    if kind == "cloudsc":
        cloudsc.cloudsc_batched(st.p, st.a, *st.dims, PTSPHY, precision=case["precision"],
                                stream=torch.cuda.current_stream())
    elif kind == "single":
        cloudsc.cloudsc_batched_sp(st.p, st.a, *st.dims, PTSPHY, precision=case["precision"],
                                   stream=torch.cuda.current_stream())
    elif kind == "spp":
        cloudsc.cloudsc_batched_diag(st.p, st.a, st.diag, *st.dims, PTSPHY, stream=torch.cuda.current_stream())
    else:
        cloudsc.cloudsc_batched_host(st.p, st.a, *st.dims, PTSPHY, precision=case["precision"])
    out = {n: st.a[n] for n in fields.OUTPUT_NAMES}
    if kind == "spp":
        out["pfsd"] = st.diag["pfsd"]
    return out


SURROGATE_OUTPUTS = ["tendency_loc_t", "tendency_loc_q", "tendency_loc_a", "tendency_loc_cld", "plude", "pfplsl", "pfplsn",
                     "pfhpsl", "pfhpsn"]


# ------------------------------------------------------------------------------------------------------ work and tolerance
def work(case):
    """Each input element the path reads once and each output element once; flops of the tensor-core contractions, and for
    the pointwise schemes a count of their arithmetic (an exp, log or pow as one operation)."""
    kind, n, kl = case["kind"], case["ncol"], case.get("klev", 137)
    if kind == "train":
        w = case["width"]
        macs = 128 * w + 10 * w * w + w * w + 64 * w
        rows = n * 144
        params = macs
        # per step: the batch's features and targets read, the weights and the two moments read and written
        return {"bytes": case["steps"] * (n * 137 * (28 + 16) * 4 + params * 6 * 4), "flops": case["steps"] * 6 * rows * macs}
    if kind == "satadj":
        r, w = fields.satadj_bytes_per_column(kl, inputs.ncldtop_for(kl))
        return {"bytes": n * (r + w), "flops": n * kl * 250}
    if kind == "increment":
        return {"bytes": n * kl * 7 * 3 * 8, "flops": n * kl * 7}
    if kind == "surrogate":
        w = case["width"]
        r = (22 * kl + 1) * 8 + 12   # level fields the features and the guard read
        wr = (8 * kl + 4 * (kl + 1)) * 8 + kl * 18 * 4
        return {"bytes": n * (r + wr), "flops": 2 * n * 144 * (128 * w + 10 * w * w + w * w + 64 * w)}
    r, w = fields.bytes_per_column(kl, 4 if kind == "single" else 8)
    if kind == "spp":
        r, w = r + 10 * 8, w + kl * 8
    return {"bytes": n * (r + w), "flops": n * kl * 700}


def tolerance(case):
    """About four times the distance from `exact` measured over the listed and drawn cases."""
    kind = case["kind"]
    if kind == "increment":  # one addition per value
        return {"rel": 1e-15, "max": 1e-14}
    if kind == "satadj":
        return {"rel": 1e-13, "max": 1e-11}
    if kind in ("train", "surrogate"):  # bf16 activations and gradients; AdamW's first steps follow a gradient's sign
        return {"rel": 2e-2, "max": 0.8}
    # the scheme is discontinuous in the last bit of its exponentials and powers: a limiter flips here and there
    form = case.get("precision", 0)
    if form == 0:
        return {"rel": 2e-7, "max": 1e-5} if kind == "single" else {"rel": 1e-11, "max": 1e-8}
    return {"rel": 1e-5, "max": 2e-2} if form == 1 else {"rel": 2e-2, "max": 0.9}


# ------------------------------------------------------------------------------------------------- the schemes in 64 bits
def _mn(a, b):
    return torch.minimum(torch.as_tensor(a, dtype=F64, device="cuda"), torch.as_tensor(b, dtype=F64, device="cuda"))


def _mx(a, b):
    return torch.maximum(torch.as_tensor(a, dtype=F64, device="cuda"), torch.as_tensor(b, dtype=F64, device="cuda"))


_W = torch.where


def _sat(p, t):
    """The liquid and ice saturation exponentials, the mixed-phase fraction and its weights at temperature t (FCTTRE)."""
    el = torch.exp(p.r3les * (t - p.rtt) / (t - p.r4les))
    ei = torch.exp(p.r3ies * (t - p.rtt) / (t - p.r4ies))
    x = (t.clamp(p.rtice, p.rtwat) - p.rtice) * p.rtwat_rtice_r
    alfa = torch.clamp(x * x, max=1.0)
    dem = (alfa * p.r5alvcp / (t - p.r4les) ** 2 + (1 - alfa) * p.r5alscp / (t - p.r4ies) ** 2)
    ldcpm = alfa * p.ralvdcp + (1 - alfa) * p.ralsdcp
    return el, ei, alfa, dem, ldcpm


def _supersat(p, t, q, a, pap):
    """CLOUD_SUPERSATCHECK: the condensate, the cloud increase, and the pieces its callers split it with."""
    zt, za = t.clamp(min=160.0), a.clamp(0.0, 1.0)
    el, ei, alfa, dem, ldcpm = _sat(p, zt)
    liq = torch.clamp(p.r2es * el / pap, max=0.5)
    ice = torch.clamp(p.r2es * _W(zt >= p.rtt, el, ei) / pap, max=0.5)
    koop = _mn(ice * (p.rkoop1 - p.rkoop2 * zt), liq)
    qk = koop / (1 - p.retv * koop)
    mix = torch.clamp(p.r2es * (alfa * el + (1 - alfa) * ei) / pap, max=0.5)
    cor = 1 / (1 - p.retv * mix)
    qs = mix * cor
    corqs = 1 + qs * cor * dem
    qk = 0.5 * (qk + qs)
    cond = torch.clamp(q - (za * qs + (1 - za) * qk), min=0.0)
    on = cond > 1e-14
    da = _W(on, (1 - za) * (alfa + (1 - alfa) * p.rssicefactor), 0.0)
    up = za + da
    cond = _W(on, (q - (up * qs + (1 - up) * qk)) / corqs, cond)
    return cond, da, alfa, ldcpm


def _exact_satadj(p, a, ncol):
    nb, kl, np_ = a["pt"].shape
    out = {n: torch.zeros_like(a["pt"]) for n in fields.SATADJ_OUTPUTS}
    dt, z = PTSPHY, 1 / PTSPHY
    k0 = p.ncldtop - 1
    f = {n: v[:, k0:] for n, v in a.items() if v.dim() == 3 and n != "paph"}
    ph = a["paph"]
    pap, t0, q0, a0 = f["pap"], f["pt"], f["pq"], f["pa"]
    zt, zq = t0 + dt * f["tendency_cml_t"], q0 + dt * f["tendency_cml_q"]
    za = (a0 + dt * f["tendency_cml_a"]).clamp(0.0, 1.0)
    zl, zi = f["pl"] + dt * f["tendency_cml_l"], f["pi"] + dt * f["tendency_cml_i"]
    dp = ph[:, k0 + 1:] - ph[:, k0:-1]
    dtg = dt * p.rg / dp
    dtdp = p.rd / p.rcpd * t0 / pap
    mxdt = dp * z
    wtot = _mn(mxdt, _mx(-mxdt, f["pvervel"]))
    diab = _mn(mxdt * dtdp, _mx(-mxdt * dtdp, f["phrsw"] + f["phrlw"])) * dt
    tf = dtdp * wtot * dt + diab + a["pludeli"][:, 3, k0:] * dtg + f["tendency_vdf_t"] * dt
    qf = a["pludeli"][:, 2, k0:] * dtg + f["tendency_vdf_q"] * dt
    li = zl + zi
    lf = _W(li > p.rlmin, zl / li, 0.0)
    icf = _W(li > p.rlmin, 1 - lf, 0.0)
    sig = pap / ph[:, -1:]
    rhc = p.ramid + (1 - p.ramid) * (((sig - 0.8) / 0.2).clamp(min=0.0)) ** 2
    el, ei, alfa, dem, _ = _sat(p, t0)
    liq = torch.clamp(p.r2es * el / pap, max=0.5)
    ice = torch.clamp(p.r2es * _W(t0 >= p.rtt, el, ei) / pap, max=0.5)
    koop = _mn(ice * (p.rkoop1 - p.rkoop2 * t0), liq)
    mix = torch.clamp(p.r2es * (alfa * el + (1 - alfa) * ei) / pap, max=0.5)
    qs = mix / (1 - p.retv * mix)
    qk = 0.5 * (koop / (1 - p.retv * koop) + qs)

    def qsmix(t):
        el, ei, alfa, dem, ldcpm = _sat(p, t)
        e = torch.clamp(p.r2es * (alfa * el + (1 - alfa) * ei) / pap, max=0.5)
        cor = 1 / (1 - p.retv * e)
        return e * cor, 1 + e * cor * cor * dem, ldcpm

    qs_up, cor_up, _ = qsmix(zt)
    nt, nq = (t0 + tf).clamp(min=160.0), qs + qf
    first = nq
    for _ in range(2):
        s, c, ld = qsmix(nt)
        cond = (nq - s) / c
        nt, nq = nt + ld * cond, nq - cond
    dqs = nq - first
    eps = 1e-14
    # clear-air condensation
    qe = _mx(0.0, (q0 - a0 * qs) / (1 - a0).clamp(min=eps))
    on = (dqs <= -p.rlmin) & (a0 < 1 - eps) & (qe >= rhc * qk) & (qe < qk)
    ac = _mn(-(1 - a0) * dqs / _mx(2 * (qk - qe), eps), 1 - a0)
    env = -dqs * 0.5 * ac
    env = _W(dqs < -2 * (qk - qe) / (1 - a0).clamp(min=eps), _mn(env, (a0 - 1) * dqs - qk + q0), env).clamp(min=0.0)
    on = on & ~((env < p.rlmin) | (1 - a0 < eps))
    ac, env = _W(on, ac, 0.0), _W(on, env, 0.0)
    # condensation and evaporation in the cloud
    cld = a0 * _mn((-dqs).clamp(min=0.0), ((zq - qs_up) / cor_up).clamp(min=0.0))
    cld = _W((a0 > eps) & (dqs <= -p.rlmin) & (cld >= p.rlmin), cld, 0.0)
    ev = _W((dqs > 0) & (li > 0), _mn(a0 * dqs, li), 0.0)
    warm = t0 > p.rthomo
    gl, gi = _W(warm, cld + env, 0.0) - lf * ev, _W(warm, 0.0, cld + env) - icf * ev
    tu, qu = zt + p.ralvdcp * gl + p.ralsdcp * gi, zq - gl - gi
    new = (za + ac).clamp(max=1.0)
    new = _W(new < p.ramin, 0.0, new)
    cond, da, _, _ = _supersat(p, tu, qu, new, pap)
    gl, gi = gl + _W(tu > p.rthomo, cond, 0.0), gi + _W(tu > p.rthomo, 0.0, cond)
    new = (za + ac + da).clamp(max=1.0)
    new = _W(new < p.ramin, 0.0, new)
    r = {"t": (p.ralvdcp * gl + p.ralsdcp * gi) * z, "q": -(gl + gi) * z, "a": (new - za) * z, "l": gl * z, "i": gi * z}
    for n, amount, heat in (("l", zl, p.ralvdcp), ("i", zi, p.ralsdcp)):
        neg = torch.clamp(amount + r[n] * dt, max=0.0)
        r[n], r["q"], r["t"] = r[n] - neg, r["q"] + neg, r["t"] - heat * neg
    for n in "tqali":
        out["tendency_loc_" + n][:, k0:] = r[n]
    _untouched(out, out, ncol, np_, zero=True)
    return out


def _untouched(out, start, ncol, np_, zero=False):
    """The columns past the last one keep what the arrays held."""
    last = ncol - (out["tendency_loc_t"].shape[0] - 1) * np_
    if last < np_:
        for n, v in out.items():
            v[-1, ..., last:] = 0.0 if zero else start[n][-1, ..., last:]


def _exact_cloudsc(p, a, ncol, diag=None):
    """CLOUDSC in its default configuration (IWARMRAIN = 3, IDEPICE = IDEPSNOW = ISUBLSNOW = 1) on batched double arrays, one
    level of every column at a time; with `diag` the SPP perturbations and the cloud-inhomogeneity paths."""
    nb, kl, np_ = a["pt"].shape
    out = {n: torch.zeros_like(a[n]) for n in fields.OUTPUT_NAMES}
    out["plude"] = a["plude"].clone()
    dt, z, eps = PTSPHY, 1 / PTSPHY, 1e-14
    zero = torch.zeros(nb, np_, dtype=F64, device="cuda")
    one = zero + 1
    surf, ktype, peis = a["paph"][:, -1], a["ktype"], a["peis"]
    cum = a["ldcum"] != 0
    adv = _W((ktype == 1) & (p.rmfadvw > 0), 1 - p.rmfadvw, one)
    advd = _W((ktype == 1) & (p.rmfadvw > 0), 1 - p.rmfadvw * p.rmfadvwdd, one)
    cpow = _W(a["plsm"] > 0.5, p.rcl_kk_cloud_num_land ** p.rcl_kkbaun * one, p.rcl_kk_cloud_num_sea ** p.rcl_kkbaun * one)
    spp = [one] * 9
    if diag is not None:
        g = diag["pgp2dspp"]
        spp = [torch.exp(p.spp_mu[2 * n] + p.spp_xmag[2 * n] * g[:, p.spp_mp[n] - 1]) for n in range(8)]
        n = SPP.index("cloudinhom")
        spp.append(torch.exp(p.spp_mu[2 * n + 1] + p.spp_xmag[2 * n + 1] * g[:, p.spp_mp[n]]))
        glen = 2 * p.ra * torch.sqrt(p.rpi * diag["pgaw"]) * 0.001
        out["pfsd"] = torch.zeros_like(a["pt"])
    by = dict(zip(SPP, spp))
    pa_, qr_, qs_, t_, pp_ = zero, zero, zero, zero, zero          # level above: a, rain, snow, T, pressure
    xl, xi, xr, anew = zero, zero, zero, zero                      # level above: solved liquid, ice, rain; cloud cover
    cov, covmax, ctd, frac = zero, zero, zero, zero
    rainliq = zero == 0
    fi, fr, fs = zero, zero, zero                                  # precipitation flux through the level's top
    acc = {n: zero for n in ("sql", "sqi", "cql", "cqi", "tl", "ti")}
    for k in range(kl):
        pap, ph0, ph1 = a["pap"][:, k], a["paph"][:, k], a["paph"][:, k + 1]
        t = a["pt"][:, k] + dt * a["tendency_cml_t"][:, k]
        qv = a["pq"][:, k] + dt * a["tendency_cml_q"][:, k]
        aorig = a["pa"][:, k] + dt * a["tendency_cml_a"][:, k]
        s0 = [a["pclv"][:, m, k] + dt * a["tendency_cml_cld"][:, m, k] for m in range(4)]
        vfl, vfi, dl, di = a["pvfl"][:, k], a["pvfi"][:, k], a["pludeli"][:, 0, k], a["pludeli"][:, 1, k]
        last = k == kl - 1
        # tidy up
        lt, lq = zero, zero
        neg = [zero, zero, zero, zero]
        s = list(s0)
        heat = (p.ralvdcp, p.ralsdcp, p.ralvdcp, p.ralsdcp)

        def remove(m, on):
            nonlocal lt, lq, qv
            d = _W(on, s[m], 0.0)
            neg[m] = neg[m] + d
            lq, lt, qv, s[m] = lq + d * z, lt - heat[m] * d * z, qv + d, s[m] - d

        none = (s[0] + s[1] < p.rlmin) | (aorig < p.ramin)
        remove(0, none)
        remove(1, none)
        ca = _W(none, 0.0, aorig)
        for m in range(4):
            remove(m, s[m] < p.rlmin)
        ca = ca.clamp(0.0, 1.0)
        ql, qi, qr, qs = s
        li = ql + qi
        lf = _W(li > p.rlmin, ql / li, 0.0)
        icf = _W(li > p.rlmin, 1 - lf, 0.0)
        la, lc = zero, [zero, zero, zero, zero]
        x = [zero, zero, zero, zero]
        fi1, fr1, fs1, covout = zero, zero, zero, zero
        lfsd, anewp, ratfsd, icef, liqf = one * p.rcloud_frac_std, zero, zero, zero, zero
        if k >= p.ncldtop - 1:
            # saturation
            el, ei, alfa, _, ldcpm = _sat(p, t)
            def qsat(e):
                e = torch.clamp(e, max=0.5)
                cor = 1 / (1 - p.retv * e)
                return e * cor, cor
            qsm, cm = qsat(p.r2es * (alfa * el + (1 - alfa) * ei) / pap)
            qsi, ci = qsat(p.r2es * _W(t >= p.rtt, el, ei) / pap)
            qsl, cl = qsat(p.r2es * el / pap)
            dp = ph1 - ph0
            gdp = p.rg / dp
            rho = pap / (p.rd * t)
            dtg, rdtg = dt * gdp, dp / (dt * p.rg)
            facw, faci = p.r5les / (t - p.r4les) ** 2, p.r5ies / (t - p.r4ies) ** 2
            corl, cori = 1 + p.ralvdcp * facw * cl * qsl, 1 + p.ralsdcp * faci * ci * qsi
            dqm = (alfa * facw + (1 - alfa) * faci) * cm * qsm
            corm = 1 + ldcpm * dqm
            evlim = ((qsm - qv) / corm).clamp(min=0.0)
            ra = 1 / ca.clamp(min=0.01)
            lcl, icl = ql * ra, qi * ra
            d1 = (1 - ca).clamp(min=eps)
            g = [ql, qi, qr, qs]
            # explicit rates: S[i][j] is the gain of species i from j (l, i, r, s, v)
            S = [[zero] * 5 for _ in range(5)]

            def move(i, j, r):
                S[i][j] = S[i][j] + r
                if i != j:
                    S[j][i] = S[j][i] - r

            move(4, 0, _W(ql < p.rlmin, ql, 0.0))
            move(4, 1, _W(qi < p.rlmin, qi, 0.0))
            ac, ab = zero, zero
            src, sink = [zero] * 4, [zero] * 2
            mf = a["pmfu"][:, k] * adv + a["pmfd"][:, k] * advd
            # detrainment
            pl = a["plude"][:, k]
            if not last:
                pl = pl * dtg
                on = cum & (pl > eps) & (a["plu"][:, k + 1] > eps)
                ac = ac + _W(on, pl / a["plu"][:, k + 1], 0.0)
                src[0], src[1] = _W(on, dl * dtg, 0.0), _W(on, di * dtg, 0.0)
                pl = _W(on, pl, 0.0)
                if p.lmfdsnow:
                    src[2], src[3] = a["psnde"][:, 0, k] * dtg, a["psnde"][:, 1, k] * dtg
                for m in range(4):
                    move(m, m, src[m])
                out["plude"][:, k] = pl
            # subsidence
            if k > p.ncldtop - 1:
                zmf = (mf * dtg).clamp(min=0.0)
                cust = (zmf * xl, zmf * xi)
                dtdp = p.rd / p.rcpd * 0.5 * (t_ + t) / ph0
                dqs = anew * dtdp * dt * _mn(p.rg * mf, (pap - pp_) / dt) * dqm
                fin = zero
                for m in (0, 1):
                    src[m] = src[m] + cust[m]
                    ev = _mn(cust[m] - (cust[m] - dqs).clamp(min=0.0), evlim)
                    fin = fin + cust[m] - ev
                    move(m, m, cust[m])
                    move(4, m, ev)
                ac = ac + _W(fin < eps, 0.0, zmf * anew)
            if not last:
                down = ((a["pmfu"][:, k + 1] * adv + a["pmfd"][:, k + 1] * advd) * dtg).clamp(min=0.0)
                ab = ab + down
                sink = [down, down]
            # erosion
            dif = p.rcldiff * dt * by["rcldiff"]
            dif = _W((ktype >= 2) & (pl > eps) & (peis < 10), 20 * p.rcldiff_convi * dif,
                     _W((ktype == 1) & (pl > eps), 2 * p.rcldiff_convi * dif, dif))
            ero = 0.333 * ca * (1 - ca) * dif * (qsm - (qv - ca * qsm) / d1).clamp(min=0.0)
            ero = _W(li > eps, _mn(_mn(ero, evlim), li), 0.0)
            ac = ac - _W(li > eps, 0.5 * ero / (lcl + icl), 0.0)
            move(4, 0, lf * ero)
            move(4, 1, icf * ero)
            # fall speeds and sedimentation
            vi, vs = p.rvice * by["fallspeed"], p.rvsnow * one
            dens = p.rdensref / rho
            tmp = 0.5 * (qr + xr)
            lam = (rho * tmp / p.rcl_lam1r) ** p.rcl_lam2r
            vr = _W(tmp != 0, p.rxfallspeedrain * dens ** 0.4 * p.rcl_const7r * lam ** p.rcl_dr, 0.0)
            pre, fall = zero, [zero] * 4
            if k > p.ncldtop - 1:
                fall = [zero, fi * dtg, fr * dtg, fs * dtg]
                for m in (1, 2, 3):
                    move(m, m, fall[m])
                    g[m] = g[m] + fall[m]
                    pre = pre + g[m]
            drop = [zero, dtg * rho * vi, dtg * rho * vr, dtg * rho * vs]
            # precipitation fraction
            on = pre > eps
            cov = _W(on, (1 - (1 - cov) * (1 - _mx(ca, pa_)) / (1 - _mn(pa_, 1 - 1e-6))).clamp(min=p.rcovpmin), 0.0)
            clr = _W(on, (cov - ca).clamp(min=0.0), 0.0)
            rc, rc1, sc = (_W(on, 0.5 * v / cov, 0.0) for v in (qr + qr_, qr + xr, qs + qs_))
            covmax = _W(on, _mx(cov, covmax), 0.0)
            # warm rain
            aut, accr = p.rcl_inhomogaut * one, p.rcl_inhomogacc * one
            wet = lcl > eps
            if diag is not None:
                qt = ((qv + ql) * 1000).clamp(max=30.0)
                c1 = 0.2 + 0.01 * qt + 0.0027 * qt ** 2 - 0.00008 * qt ** 3
                c3 = 0.123 * torch.exp(-c1 * 0.55)
                a2 = ca.clamp(min=0.1)
                phic = (glen * a2) ** (1 / 3) * ((c3 * glen * a2) ** 1.5 + 3 * c3) ** -0.17
                lfsd = _W(wet, 1.3 * _W(ca > 0.95, 0.17 * phic, (c1 - (c1 - 0.2) * a2) * phic), lfsd)
                phir = (glen * ca) ** (1 / 3) * ((0.11 * glen * ca) ** 1.14 + 1) ** -0.22
                fr2 = _W(ca > 0.95, 0.3 * phir, (1.1 - 0.8 * ca) * phir) ** 2
                fc2, kb = lfsd ** 2, p.rcl_kkbac
                aut = (1 + fc2) ** ((p.rcl_kkbauq - 1) * p.rcl_kkbauq / 2)
                accr = ((1 + fc2) * (1 + fr2)) ** ((kb - 1) * kb / 2) * torch.exp(
                    (1 - 0.8 * ca) * kb * kb * torch.sqrt(torch.log(1 + fc2) * torch.log(1 + fr2)))
                aut, accr = aut * by["cloudinhom"], accr * spp[8]
            q_rl = _W(wet, aut * dt * p.rcl_kkaau * lcl ** (p.rcl_kkbauq - 1) * cpow, 0.0)
            q_rl = q_rl + _W(wet & (rc > eps), accr * dt * p.rcl_kkaac * lcl ** (p.rcl_kkbac - 1) * rc ** p.rcl_kkbac, 0.0)
            # rain evaporation
            rhmax = (p.rprecrhmax + (1 - p.rprecrhmax) * covmax / d1).clamp(p.rprecrhmax, 1.0)
            mid = (p.ramid * by["ramid"])
            if diag is not None and p.spp_lramidlimit1:
                mid = mid.clamp(max=1.0)
            sig = pap / surf
            rhc = _W(sig > 0.8, mid + (1 - mid) * ((sig - 0.8) / 0.2) ** 2, mid)
            rh = _mn(rhc, rhmax).clamp(max=0.9)
            qe = _mn(qv, qsl).clamp(min=0.0)
            on = (clr > eps) & (rc1 > eps) & (qe < rh * qsl)
            el_, d4 = p.rv / p.rd * p.r2es * el, dens ** float(np.float32(0.4))
            lam = (p.rcl_lam1r / (rho * rc1)) ** p.rcl_lam2r
            den = p.rcl_cdenom1 * el_ - p.rcl_cdenom2 * t * el_ + p.rcl_cdenom3 * t ** 3 * pap
            c2 = (t / 273) ** 1.5 * 393 / (t + 120)
            beta = 0.15 / qsl * t ** 2 * el_ * p.rcl_const1r * (c2 / den) * (
                0.78 / lam ** p.rcl_const4r + p.rcl_const2r * (rho * d4) ** 0.5 / (c2 ** 0.5 * lam ** p.rcl_const3r))
            ev = clr * beta * dt * (rh * qsl - qe).clamp(min=0.0) / (1 + beta * dt * corl) * by["rainevap"]
            ev = _W(on, _mn(ev, g[2]), 0.0)
            move(4, 2, ev)
            g[2] = g[2] - ev
            # ice deposition
            ctd = _W((pa_ < p.rcldtopcf) & (ca >= p.rcldtopcf), 0.0, ctd + dp / (rho * p.rg))
            on = (t < p.rtt - 5) & (g[0] > p.rlmin)
            sup, vp = (qsl - qsi) / qsi, p.r2es * ei * p.rv / p.rd
            nuc = 1000 * torch.exp(12.96 * sup - 0.639)
            add = p.rlstt * (p.rlstt / (p.rv * t) - 1) / (2.4e-2 * t)
            bdd = p.rv * t * pap / (2.21 * vp)
            cvd = 7.8 * (nuc / rho) ** 0.666 * sup / (8.87 * (add + bdd))
            ice0 = _mx(icl, nuc * p.riceinit / rho)
            dep = p.rcl_overlapliqice * ca * ((0.666 * cvd * dt + ice0 ** 0.666) ** 1.5 - ice0)
            inf = (nuc / 15000).clamp(max=1.0)
            dep = _mn(dep.clamp(min=0.0), g[0]) * (inf + (1 - inf) * (p.rdepliqrefrate + ctd / p.rdepliqrefdepth)).clamp(max=1.0)
            dep = _W(on, dep, 0.0)
            move(1, 0, dep)
            g[0], g[1] = g[0] - dep, g[1] + dep
            # snow deposition
            sup = ((qv - qsm) / qsm).clamp(min=0.0)
            on = (t < p.rtt) & (sc > eps) & (sup > 0)
            apb = p.rcl_apb1 * vp - p.rcl_apb2 * vp * t + pap * p.rcl_apb3 * t ** 3
            cf = (1 / rho) ** 0.5
            pr2 = rho * sc * p.rcl_const1s
            t1 = sup * t ** 2 * vp * c2 * p.rcl_const2s / (rho * apb)
            t2 = 0.65 * p.rcl_const6s * pr2 ** p.rcl_const4s + p.rcl_const3s * cf ** 0.5 * rho ** 0.5 * pr2 ** p.rcl_const5s / c2 ** 0.5
            dep = _mn((cov * t1 * t2 * dt).clamp(min=0.0), qv - qsm) / corm
            move(3, 4, _W(on, dep, 0.0))
            lcl, icl = g[0] * ra, g[1] * ra
            # ice to snow
            co = dt * p.rsnowlin1 * torch.exp(p.rsnowlin2 * (t - p.rtt))
            q_si = _W((t <= p.rtt) & (icl > eps), co * -torch.expm1(-(icl / (p.rlcritsnow * by["rlcritsnow"])) ** 2), 0.0)
            # melting
            tot = g[1] + g[3]
            tw = t - p.rtt - (qsi - qv).clamp(min=0.0) * (1329.31 + 0.0074615 * (pap - 0.85e5) - 40.637 * (t - 275))
            most = (tw * (dt * (1 + 0.5 * tw) / p.rtaumel).abs() / p.ralfdcp).clamp(min=0.0)
            on = (tot > eps) & (t > p.rtt) & (most > eps)
            for m in (1, 3):
                melt = _W(on, _mn(g[m], g[m] / tot * most), 0.0)
                g[m], g[2] = g[m] - melt, g[2] + melt
                move(2, m, melt)
            # rain freezing
            rain = qr > eps
            new = rain & (t <= p.rtt) & (t_ > p.rtt)
            frac = _W(new, qr / (qs + qr).clamp(min=eps), frac)
            rainliq = _W(new, frac > float(np.float32(0.8)), rainliq)
            lam = (p.rcl_lam1r / (rho * qr)) ** p.rcl_lam2r
            f1 = dt * p.rcl_const5r / rho * torch.expm1((p.rcl_fzrab * (t - p.rtt)).clamp(max=50.0)) * lam ** p.rcl_const6r
            f2 = (p.rtt - t) * (dt * (1 + 0.5 * (p.rtt - t)) / p.rtaumel).abs() / p.ralfdcp
            most = _W(rainliq, f1, f2).clamp(min=0.0)
            move(3, 2, _W(rain & (t < p.rtt) & (most > eps), _mn(qr, most), 0.0))
            # homogeneous freezing
            most = ((p.rthomo - t) / p.ralfdcp).clamp(min=0.0)
            move(1, 0, _W((most > eps) & (g[0] > eps), _mn(g[0], most), 0.0))
            # riming and collection
            cold = t <= p.rtt
            rim = p.rcl_effrime * cov * dt * p.rcl_const7s * d4 * (rho * sc * p.rcl_const1s) ** p.rcl_const8s
            q_sl = _W(cold & (lcl > eps) & (sc > eps) & (cov > 0.01), rim.clamp(max=1.0), 0.0)
            on = cold & (frac < eps) & (rc > eps)
            lamr = (p.rcl_lam1r / (rho * rc)) ** p.rcl_lam2r
            n0r = p.rcl_x1r * lamr ** p.rcl_x2r
            for m, amount, v, fac in ((3, sc, vs, 1.0), (1, icl, vi, 0.1)):
                lam = (p.rcl_lam1s / (rho * amount)) ** p.rcl_lam2s
                rat = lamr / lam
                col = cov * dt * (p.rpi ** 2 * p.rdenswat * fac * rho * n0r * p.rcl_x1s / (lam * lamr ** 3)) * _mx(
                    (vr - v).abs(), (vr + v) / 8) * ((0.5 * rat + 2) * rat + 5) / lamr ** 3
                move(m, 2, _W(on & (amount > eps), col, 0.0))
            # snow sublimation
            qe = _mn((qv - ca * qsi) / d1, qsi).clamp(min=0.0)
            on = (clr > eps) & (g[3] > eps) & (qe < rhmax * qsi)
            aa = cov * dtg
            b1 = torch.sqrt(sig) / p.rvrfactor * (g[3] * clr / aa.abs().clamp(min=100 * 2.0 ** -52)) / clr.clamp(min=eps)
            beta = p.rg * p.rpecons * b1 ** 0.5777
            ev = clr * beta * (qsi - qe) / (1 + beta * dt * cori) * dp / p.rg * dtg * by["snowsublim"]
            ev = _W(on, _mn(ev, g[3]), 0.0)
            move(4, 3, ev)
            cov = _W(on, (cov - ((cov - ca) * ev / g[3]).clamp(min=0.0)).clamp(min=p.rcovpmin), cov)
            g[3] = g[3] - ev
            for m in (1, 2, 3):
                move(4, m, _W(g[m] < p.rlmin, g[m], 0.0))
            # cloud cover
            anew = ((ca + ac) / (1 + ab)).clamp(max=1.0)
            anew = _W(anew < p.ramin, 0.0, anew)
            da = anew - aorig
            # sink truncation, the species in the order of their ratios (stable)
            amount = [ql, qi, qr, qs, qv]
            amt = torch.stack(amount)
            A = torch.stack([torch.stack(r) for r in S])
            room = amt.clamp(min=eps)
            order = torch.argsort(room / _mx(-A.sum(1), room), dim=0, stable=True)
            for rank in range(5):
                i = order[rank].view(1, 1, nb, np_)
                row = A.gather(0, i.expand(1, 5, nb, np_))[0]
                mm = amt.gather(0, i[0])[0].clamp(min=eps)
                ratio = mm / _mx(-row.sum(0), mm)
                scale = _W(row < 0, ratio, one)
                A = A.scatter(0, i.expand(1, 5, nb, np_), (row * scale).unsqueeze(0))
                colm = A.gather(1, i.expand(5, 1, nb, np_))[:, 0]
                A = A.scatter(1, i.expand(5, 1, nb, np_), (colm * scale).unsqueeze(1))
            ex = [amount[m] + A[m].sum(0) for m in range(5)]
            # implicit solve
            dl_, di_ = 1 + sink[0] + q_rl + q_sl, 1 + drop[1] + sink[1] + q_si
            x[0], x[1] = ex[0] / dl_, ex[1] / di_
            x[2] = (ex[2] + q_rl * x[0]) / (1 + drop[2])
            x[3] = (ex[3] + q_sl * x[0] + q_si * x[1]) / (1 + drop[3])
            xv = ex[4]
            for m in range(4):
                xv, x[m] = xv + _W(x[m] < eps, x[m], 0.0), _W(x[m] < eps, 0.0, x[m])
            xl, xi, xr = x[0], x[1], x[2]
            fi1, fr1, fs1 = (drop[m] * x[m] * rdtg for m in (1, 2, 3))
            cov = _W(fs1 + fr1 < eps, 0.0, cov)
            # tendencies
            for m in range(4):
                fq = src[m] + fall[m] - (drop[m] + (sink[m] if m < 2 else 0.0)) * x[m]
                lt = lt + heat[m] * (x[m] - amount[m] - fq) * z
                lc[m] = (x[m] - s0[m]) * z
            lq, la = lq + (xv - qv) * z, da * z
            cond, up, alfa, ldcpm = _supersat(p, a["pt"][:, k] + dt * (lt + a["tendency_cml_t"][:, k]),
                                              a["pq"][:, k] + dt * (lq + a["tendency_cml_q"][:, k]),
                                              a["pa"][:, k] + dt * (la + a["tendency_cml_a"][:, k]), pap)
            lq, lt, la = lq - cond * z, lt + ldcpm * cond * z, la + up * z
            lc[0], lc[1] = lc[0] + cond * alfa * z, lc[1] + cond * (1 - alfa) * z
            for m in (0, 1):
                under = (s0[m] + lc[m] * dt).clamp(max=0.0) * z
                lc[m], lq, lt = lc[m] - under, lq + under, lt - heat[m] * under
            covout = cov
            if diag is not None:
                pda = a["pa"][:, k] + da
                anewp = _W(pda > 0.001, _mx(pda, cov).clamp(min=0.1), 0.0)
                tot = s0[0] + s0[1] + pl
                ratfsd = _W(tot > p.rlmin, (pl / tot).clamp(0.0, 1.0), 0.0)
                icef, liqf = x[1], x[0]
        if diag is not None:
            back = 0.446585 * glen ** (1 / 3) * ((0.308061 * glen) ** 0.395736 + 1) ** -0.744527
            qt = ((qv + qi) * 1000).clamp(max=30.0).clamp(min=float(np.float32(1e-5)))
            dz = ((ph1 - ph0) / (p.rg * pap / (p.rd * t)) * 0.001).clamp(float(np.float32(0.001)), 0.5)
            phi = (dz / float(np.float32(0.24))) ** float(np.float32(0.11)) * (qt / 10) ** float(np.float32(0.03))
            f = _W(anewp > 0.95, 1.3 * (back * phi + ratfsd * 1.5), 1.3 * (back * phi * 1.5 + ratfsd * 1.5))
            f = _W(anewp > 0.001, f, p.rcloud_frac_std * one)
            f = _W(icef > eps, f, _W(liqf > 0, lfsd, p.rcloud_frac_std * one))
            out["pfsd"][:, k] = f.clamp(0.1, 3.575)
        for n, v in (("t", lt), ("q", lq), ("a", la)):
            out["tendency_loc_" + n][:, k] = v
        for m in range(4):
            out["tendency_loc_cld"][:, m, k] = lc[m]
        out["pcovptot"][:, k] = covout
        # fluxes
        out["pfplsl"][:, k], out["pfplsn"][:, k] = fr, fs + fi
        w = -(ph1 - ph0) / p.rg * z
        out["pfsqrf"][:, k + 1] = acc["sql"] + (x[2] - s0[2]) * w
        out["pfcqrng"][:, k + 1] = acc["cql"] + neg[2] * w
        out["pfsqsf"][:, k + 1] = acc["sqi"] + (x[3] - s0[3]) * w
        out["pfcqsng"][:, k + 1] = acc["cqi"] + neg[3] * w
        acc["sql"] = acc["sql"] + (x[0] - s0[0] + vfl * dt) * w + dl
        acc["sqi"] = acc["sqi"] + (x[1] - s0[1] + vfi * dt) * w + di
        acc["cql"], acc["cqi"] = acc["cql"] + neg[0] * w, acc["cqi"] + neg[1] * w
        acc["tl"], acc["ti"] = acc["tl"] + vfl * dt * w, acc["ti"] + vfi * dt * w
        for n, v in (("pfsqlf", "sql"), ("pfsqif", "sqi"), ("pfcqlng", "cql"), ("pfcqnng", "cqi"), ("pfsqltur", "tl"), ("pfsqitur", "ti")):
            out[n][:, k + 1] = acc[v]
        pa_, qr_, qs_, t_, pp_ = ca, qr, qs, t, pap
        fi, fr, fs = fi1, fr1, fs1
    out["pfplsl"][:, kl], out["pfplsn"][:, kl] = fr, fs + fi
    out["pfhpsl"][:], out["pfhpsn"][:] = -p.rlvtt * out["pfplsl"], -p.rlstt * out["pfplsn"]
    out["prainfrac_toprfz"][:] = frac
    _untouched(out, {n: (a[n] if n == "plude" else torch.zeros_like(v)) for n, v in out.items()}, ncol, np_)
    return out


# the perturbations in the order of the parameter arrays
SPP = ["ramid", "rcldiff", "rclcrit", "rlcritsnow", "rainevap", "snowsublim", "fallspeed", "cloudinhom"]


def _conv(h, w):
    """The network's convolution over levels: h [columns, levels, k], w [taps, n, k]."""
    return torch.nn.functional.conv1d(h.transpose(1, 2), w.permute(1, 2, 0), padding=w.shape[0] // 2).transpose(1, 2)


def _network(w, b, feat):
    """[columns, levels, 25] normalised features to [columns, levels, 64]."""
    win = torch.nn.functional.pad(feat, (0, 0, 2, 2)).unfold(1, 5, 1).transpose(2, 3).reshape(*feat.shape[:2], 125)
    silu = torch.nn.functional.silu
    h = silu(_conv(torch.nn.functional.pad(win, (0, 3)), w[1]) + b[1])
    h = h + silu(_conv(h, w[2]) + b[2])
    h = h + silu(_conv(h, w[3]) + b[3])
    return _conv(silu(_conv(h, w[4]) + b[4]), w[5]) + b[5]


def _normalise(norm, f):
    for ch in range(surrogate.NIN):
        v = f[..., ch]
        if norm.use_log[ch]:
            v = torch.log(v.clamp(min=0.0) + norm.eps[ch])
        f[..., ch] = (v - norm.mean[ch]) * norm.inv_std[ch]
    return f


def _features(p, a):
    """The surrogate's 25 raw input fields of every column and level."""
    nb, kl, np_ = a["pt"].shape
    dpg = (a["paph"][:, 1:] - a["paph"][:, :-1]) / 9.80665
    t, q = a["pt"] + PTSPHY * a["tendency_cml_t"], a["pq"] + PTSPHY * a["tendency_cml_q"]
    el, ei, alfa, _, _ = _sat(p, t)
    mix = torch.clamp(p.r2es * (alfa * el + (1 - alfa) * ei) / a["pap"], max=0.5)
    ice = torch.clamp(p.r2es * ei / a["pap"], max=0.5)
    c = a["pclv"]
    mass = torch.stack([dpg * c[:, :4].clamp(min=0.0).sum(1), dpg * c[:, 2:4].clamp(min=0.0).sum(1)])
    above = torch.cumsum(mass, 2) - mass
    f = [a["pt"], a["pq"], a["pap"], c[:, 0], c[:, 1], c[:, 2], c[:, 3], a["plude"], a["pa"], a["pmfu"] + a["pmfd"],
         a["tendency_cml_t"], a["tendency_cml_q"], a["tendency_cml_a"], a["tendency_cml_cld"][:, 0] + a["tendency_cml_cld"][:, 1],
         a["pmfu"], a["pmfd"], a["plu"], a["pludeli"][:, 0] + a["pludeli"][:, 1], a["psnde"].sum(1), dpg * 9.80665,
         q * (1 - p.retv * mix) / mix, a["plsm"][:, None].expand(nb, kl, np_), above[0], above[1], q * (1 - p.retv * ice) / ice]
    return torch.stack(f, -1).transpose(1, 2).reshape(nb * np_, kl, len(f))


def _exact_train(st):
    """The training loop of one pass on double weights, by autograd."""
    case, net, data = st.case, st.net, st.data
    w = {i: v.double().clone().requires_grad_() for i, v in net.p.items()}
    b = {i: v.double().clone().requires_grad_() for i, v in net.b.items()}
    every = [*w.values(), *b.values()]
    m, v = [torch.zeros_like(x) for x in every], [torch.zeros_like(x) for x in every]
    gen = torch.Generator(device="cuda").manual_seed(0)
    lp, kl, no, losses = surrogate.LP, surrogate.KLEV, surrogate.NOUT, []
    feat = data.feat.view(data.ncol, lp, -1)[:, 2:2 + kl, :surrogate.NIN].double()
    feat = _normalise(net.norm, feat)
    tgt = data.tgt.view(data.ncol, lp, -1)[:, 2:2 + kl, :no].double()
    for it in range(case["steps"]):
        cols = torch.randint(0, data.ncol, (case["ncol"],), device="cuda", generator=gen, dtype=torch.int32).long()
        y, goal = _network(w, b, feat[cols]), tgt[cols]
        loss = sum((y[..., h:h + no] - goal).square().mean() for h in (0, 32))
        losses.append(loss.detach() / 2)
        grads = torch.autograd.grad(loss, every)
        lr, n = 2e-3 * (it + 1) / 200, it + 1
        with torch.no_grad():
            for j, (x, gr) in enumerate(zip(every, grads)):
                m[j] = 0.9 * m[j] + 0.1 * gr
                v[j] = 0.999 * v[j] + 0.001 * gr * gr
                wd = 1e-4 if j < len(w) else 0.0
                x -= lr * ((m[j] / (1 - 0.9 ** n)) / (torch.sqrt(v[j] / (1 - 0.999 ** n)) + 1e-8) + wd * x)
    keys = list(w)
    pick = lambda s, o: dict(zip(keys, s[o:o + len(keys)]))  # noqa: E731
    return {"loss": torch.stack(losses), "w": {i: x.detach() for i, x in w.items()}, "b": {i: x.detach() for i, x in b.items()},
            "m": pick(m, 0), "v": pick(v, 0), "mb": pick(m, len(keys)), "vb": pick(v, len(keys))}


def exact(case, seed):
    kind = case["kind"]
    st = prepare(case, seed)
    p = st.p
    if kind == "train":
        return _exact_train(st)
    if kind == "satadj":
        return _exact_satadj(p, st.a, case["ncol"])
    if kind == "increment":
        out = {n: st.state[n].clone() for n in ("t", "q", "a", "cld")}
        last = case["ncol"] - (_nblk(case) - 1) * case["nproma"]
        for n, v in out.items():
            d = st.inc[n].clone()
            d[-1, ..., last:] = 0.0
            if n == "cld":
                d[:, 4] = 0.0
            v += d
        return out
    if kind == "surrogate":
        # the network alone: the guard sends a column to the FP64 scheme by thresholds, which has no such value
        f = _normalise(st.net.norm, _features(p, st.a))
        y = torch.zeros(f.shape[0], surrogate.LP, 64, dtype=F64, device="cuda")
        w, b = ({i: v.double() for i, v in x.items()} for x in (st.net.wbf, st.net.b))
        for c in range(0, f.shape[0], 4096):
            y[c:c + 4096, 2:2 + case["klev"]] = _network(w, b, f[c:c + 4096])
        return {**{n: None for n in SURROGATE_OUTPUTS}, "y": y.view(-1, 64)}
    if kind == "block":
        out = _exact_cloudsc(p, {n: torch.from_numpy(v).cuda()[None] for n, v in st.a.items()}, case["ncol"])
        return {n: v[0] for n, v in out.items()}
    a = {n: v.cuda().double() if v.is_floating_point() else v.cuda() for n, v in st.a.items()}
    return _exact_cloudsc(p, a, case["ncol"], st.diag if kind == "spp" else None)
