"""Workloads of the solver and of its warm-start network, for timing and for
comparing results between two builds.

Each case is one call (or one short sequence of calls) that a program using
the library makes, through the public Python entry points:

  pass    one crystal pass of one instance (Plan.crystal_pass)
  cavity  a block of round trips of one instance (Plan.round_trips)
  sweep   a batch of instances for some round trips (Batch)
  fft     the stand-alone batched transform (fft_c2c)
  train   one optimiser step of the warm-start network (MLP.train_step)
  infer   its forward pass (MLP.forward)
  bands   fields synthesised from its predictions (WarmStartModel.fields)

exact() restates the same mathematics in FP64 with plain torch and numpy.
"""
import math

import numpy as np
import torch

import cuopo_b200 as cu
from cuopo_b200 import warmstart as ws

# MgO:PPLN 532 -> 1064 nm, 5 mm at 4x threshold, and MgO:sPPLT 532 -> 1550 nm, 20 mm
# at 3x threshold: what the parameter set-up gives for the repository's own configurations.
PPLN2 = dict(vp=122.810791015625, vs=136.0599365234375, vi=0.0, b2p=7.161680173339846e-07,
             b2s=2.3455552877749142e-07, b2i=0.0, kp=8.515240187989548e-05, ks=4.408850509207696e-05, ki=0.0,
             t_rt=352.72381591796875, ap0=0.09526284039020538, length=5000.0)
SPPLT3 = dict(vp=125.78053283691406, vs=138.75430297851562, vi=134.7908477783203, b2p=6.033708359609591e-07,
              b2s=6.692553000675616e-08, b2i=2.9862749784115294e-07, kp=3.760041363420896e-05,
              ks=1.3409882740234025e-05, ki=2.526531352486927e-05, t_rt=408.0742492675781,
              ap0=0.0564594566822052, length=20000.0)
ALPHA = (2.499999936844688e-06, 2.0000000233721948e-07, 2.0000000233721948e-07)
MIXED = (4096, 8192, 16384, 32768)   # grid sizes of the benchmark's sweep


def listed():
    return [
        # the plugin boundary: one EvolutionInCrystal call of the smallest kind, launch latency and serial slices
        dict(name="pass_2eq_1024", kind="pass", n_eqs=2, n_t=1024, n_z=50, f64=False, dk=4e-4),
        # the single CW OPO configuration (2^13, 100 slices): one process, one instance, a block of its round trips
        dict(name="cavity_cw_8192", kind="cavity", n_eqs=2, n_t=8192, n_z=100, rts=2, f64=False, ns=False,
             gdd=False, eom=False, dk=8.4e-7),
        # the nanosecond 3-wave configuration (2^16, 200 slices)
        dict(name="cavity_ns_65536", kind="cavity", n_eqs=3, n_t=65536, n_z=200, rts=1, f64=False, ns=True,
             gdd=False, eom=False, dk=1e-6),
        # the FP64 plan a caller validates with, every cavity element on
        dict(name="cavity_f64_8192", kind="cavity", n_eqs=2, n_t=8192, n_z=100, rts=1, f64=True, ns=False,
             gdd=True, eom=True, dk=4e-4),
        # the headline sweep: grids 2^12..2^15 mixed, GDD drawn per instance, fields near saturation
        dict(name="sweep_mixed_256", kind="sweep", n_eqs=2, n_t=0, n_z=100, rts=2, count=256, f64=False,
             noise=False, dk=8.4e-7),
        # training data of the warm start: 2^13 instances from seeded noise, a count that fills no whole wave
        dict(name="sweep_8192_333", kind="sweep", n_eqs=2, n_t=8192, n_z=100, rts=2, count=333, f64=False,
             noise=True, dk=8.4e-7),
        # the script's sweep over a 3-wave crystal
        dict(name="sweep_3wave_4096", kind="sweep", n_eqs=3, n_t=4096, n_z=100, rts=2, count=150, f64=False,
             noise=True, dk=1e-6),
        # the FP64 solver on a batch
        dict(name="sweep_f64_16384", kind="sweep", n_eqs=2, n_t=16384, n_z=50, rts=1, count=45, f64=True,
             noise=False, dk=4e-4),
        # spectra of a batch of fields (the warm start's targets)
        dict(name="fft_f32_8192", kind="fft", n=8192, batch=3001, sign=-1, f64=False),
        # one step of training at the configuration's batch
        dict(name="train_4096", kind="train", rows=4096),
        # predictions for a ragged number of parameter sets
        dict(name="infer_1500", kind="infer", rows=1500),
        # initial fields from the predictions for the bench's held-out set
        dict(name="bands_296", kind="bands", count=296, n_t=8192),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pass", "cavity", "cavity", "cavity", "sweep", "sweep", "sweep", "sweep", "fft", "train",
                       "infer", "bands"])
    f64 = rng.random() < 0.25
    n_eqs = rng.choice([2, 2, 3])
    dk = rng.uniform(-1e-3, 1e-3)
    if kind == "pass":
        return dict(kind=kind, n_eqs=n_eqs, n_t=2 ** rng.randint(9, 13), n_z=_log(rng, 10, 200), f64=f64, dk=dk)
    if kind == "cavity":
        n_t = 2 ** rng.randint(9, 16)
        n_z = _log(rng, 20, 200)
        rts = max(1, min(8, 200 // n_z, int(4e6 / (n_t * n_z) * rng.random())))
        return dict(kind=kind, n_eqs=n_eqs, n_t=n_t, n_z=n_z, rts=rts, f64=f64, ns=rng.random() < 0.3,
                    gdd=rng.random() < 0.5, eom=rng.random() < 0.3, dk=dk)
    if kind == "sweep":
        n_t = 0 if rng.random() < 0.3 and n_eqs == 2 else 2 ** rng.randint(10, 14 if f64 or n_eqs == 3 else 15)
        pts = n_t or 15360
        n_z = _log(rng, 20, 100)
        most = 7e8 / (3 if f64 else 1) / (2 if n_eqs == 3 else 1)
        rts = rng.randint(1, max(1, min(3, 200 // n_z)))
        count = max(2, min(600, _log(rng, 3, max(4, int(most / (pts * n_z * rts))))))
        return dict(kind=kind, n_eqs=n_eqs, n_t=n_t, n_z=n_z, rts=rts, count=count, f64=f64,
                    noise=n_eqs == 3 or (not f64 and rng.random() < 0.4), dk=dk) if not (f64 and n_eqs == 3) else \
            dict(kind=kind, n_eqs=2, n_t=n_t, n_z=n_z, rts=rts, count=count, f64=True, noise=False, dk=dk)
    if kind == "fft":
        n = 2 ** rng.randint(9, 12 if f64 else 13)
        return dict(kind=kind, n=n, batch=_log(rng, 1, 2.4e7 / n / (2 if f64 else 1)), sign=rng.choice([-1, 1]),
                    f64=f64)
    if kind in ("train", "infer"):
        return dict(kind=kind, rows=_log(rng, 64, 4096))
    n_t = 2 ** rng.randint(12, 15)
    return dict(kind=kind, count=_log(rng, 8, 4e6 / n_t), n_t=n_t)


# ------------------------------------------------------------------ parameters

def _params(c, n_t):
    m = PPLN2 if c["n_eqs"] == 2 else SPPLT3
    return dict(n_eqs=c["n_eqs"], n_t=n_t, n_z=c["n_z"], regime=1 if c.get("ns") else 0,
                vp=m["vp"], vs=m["vs"], vi=m["vi"], b2p=m["b2p"], b2s=m["b2s"], b2i=m["b2i"], dk=c["dk"],
                kp=m["kp"], ks=m["ks"], ki=m["ki"], dz=m["length"] / c["n_z"], alpha_crp=ALPHA[0],
                alpha_crs=ALPHA[1], alpha_cri=ALPHA[2], Rs=0.98, Ri=0.98, delta=0.05,
                gdd=-2.5e-4 if c.get("gdd") else 0.0, use_eom=1 if c.get("eom") else 0, eom_idler=1,
                mod_depth=1.884955644607544 if c.get("eom") else 0.0, fpm=0.0028, t_rt=m["t_rt"],
                ap0=float(np.float32(m["ap0"])))


def _instances(c, seed):
    """Per instance (n_t, ap0, Rs, delta, gdd, noise seed), drawn as the benchmark's sweep draws them."""
    rng = np.random.default_rng(seed)
    m = PPLN2 if c["n_eqs"] == 2 else SPPLT3
    k = c["count"]
    # the grids of a mixed sweep are the case's, the other parameters the seed's
    nt = np.random.default_rng(k).choice(MIXED, k) if c["n_t"] == 0 else np.full(k, c["n_t"])
    ap0 = (m["ap0"] * np.sqrt(rng.uniform(0.3, 1.5, k))).astype(np.float32).astype(np.float64)
    return [dict(n_t=int(nt[i]), ap0=float(ap0[i]), Rs=float(r), delta=float(d), gdd=float(g), seed=int(seed) * 1000 + i)
            for i, (r, d, g) in enumerate(zip(rng.uniform(0.90, 0.99, k), rng.uniform(-1, 1, k),
                                              rng.uniform(-5e-4, 5e-4, k)))]


def _field(n, scale, seed, f64):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    x = torch.randn(n, 2, generator=g, device="cuda", dtype=torch.float64) * scale
    return torch.view_as_complex(x.contiguous()).to(torch.complex128 if f64 else torch.complex64)


def _start(c, seed):
    n, f64 = c["n_t"], c["f64"]
    return [_field(n, s, 10 * seed + f, f64) for f, s in enumerate((0.08, 0.3, 0.3)[:c["n_eqs"]])]


def _window(c, p, seed):
    """Nanosecond pump window, one round trip longer than the block: a Gaussian pulse, its peak where the seed puts it."""
    n = p["n_t"] * (c["rts"] + 1)
    x = torch.linspace(-1, 1, n, device="cuda", dtype=torch.float64)
    a = p["ap0"] * torch.exp(-(x - 0.1 * math.sin(seed)) ** 2 / 0.5)
    return torch.complex(a, torch.zeros_like(a)).to(torch.complex128 if c["f64"] else torch.complex64)


def _weights(seed):
    """Parameters of the 4 -> 512 x 4 -> 512 network (per layer W [N][K] then b [N]), trained-like magnitudes."""
    rng = np.random.default_rng(seed)
    parts = []
    for n, k in _dims():
        parts += [rng.uniform(-1, 1, n * k) * math.sqrt(6.0 / k), 0.1 * rng.standard_normal(n)]
    return np.concatenate(parts).astype(np.float32)


def _dims():
    return [(ws.WIDTH, ws.N_FEATURES)] + [(ws.WIDTH, ws.WIDTH)] * (ws.DEPTH - 1) + [(512, ws.WIDTH)]


def _rows(c, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    x = torch.rand(c["rows"], ws.N_FEATURES, generator=g, device="cuda") * 2 - 1
    t = torch.randn(c["rows"], 512, generator=g, device="cuda") * 0.5
    return x, t


def _prediction(c, seed):
    """Rows of the band representation: two bands of magnitudes, pair phase, centre, log10 power."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    k, n_t = c["count"], c["n_t"]
    y = torch.empty(k, 512, device="cuda")
    d = torch.arange(256, device="cuda") % 128 - 64
    y[:, :256] = torch.exp(-(d / 25.0) ** 2) * (0.5 + torch.rand(k, 256, generator=g, device="cuda"))
    phi = (torch.rand(k, 1, generator=g, device="cuda") * 2 - 1) * math.pi
    q0 = torch.randint(64, n_t // 2 - 64, (k, 1), generator=g, device="cuda").float()
    y[:, 256:320] = torch.cos(phi)
    y[:, 320:384] = torch.sin(phi)
    y[:, 384:448] = ws.centre_code(q0, n_t)
    y[:, 448:512] = torch.rand(k, 1, generator=g, device="cuda") - 1
    return y


# ---------------------------------------------------------------- prepare, run

def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind in ("pass", "cavity"):
        p = _params(c, c["n_t"])
        plan = cu.Plan(cu.Params(**p), precision=cu.F64 if c["f64"] else cu.F32)
        fields = _start(c, seed)
        s = dict(case=c, plan=plan, start=fields, fields=[f.clone() for f in fields])
        if kind == "cavity":
            s["ps"] = torch.zeros(c["rts"], dtype=torch.float64, device="cuda")
            s["pump"] = _window(c, p, seed) if c["ns"] else None
        return s
    if kind == "sweep":
        inst = _instances(c, seed)
        prec = cu.F64 if c["f64"] else cu.F32
        b = cu.Batch(cu.Params(**_params(c, inst[0]["n_t"])), inst, precision=prec)
        s = dict(case=c, batch=b, out=torch.empty(b.total, dtype=torch.complex128 if c["f64"] else torch.complex64,
                                                  device="cuda"))
        if not c["noise"]:
            s["start"] = _field(b.total, 0.3, seed, c["f64"])
        return s
    if kind == "fft":
        x = _field(c["batch"] * c["n"], 1.0, seed, c["f64"]).reshape(c["batch"], c["n"])
        return dict(case=c, x=x, out=torch.empty_like(x))
    if kind in ("train", "infer"):
        m = ws.MLP(max_batch=c["rows"])
        m.set_params(_weights(seed))
        x, t = _rows(c, seed)
        s = dict(case=c, mlp=m, x=x, t=t, loss=torch.zeros(1, device="cuda"))
        if kind == "train":
            s["view"] = m.grad_tensor()
            s["grad"] = torch.empty_like(s["view"])
        return s
    return dict(case=c, model=ws.WarmStartModel(None, 1.0, {"kind": "band"}), pred=_prediction(c, seed))


def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind == "pass":
        # the caller's fields of this pass, then the pass in place
        for f, x in zip(state["fields"], state["start"]):
            f.copy_(x)
        state["plan"].crystal_pass(*state["fields"])
        return state["fields"]
    if kind == "cavity":
        # the run's initial fields, then its first block of round trips
        f = state["fields"]
        for y, x in zip(f, state["start"]):
            y.copy_(x)
        state["plan"].round_trips(f[0], f[1], f[2] if c["n_eqs"] == 3 else None, state["pump"],
                                  c["rts"] + 1 if c["ns"] else 0, 0, c["rts"], ps_hist=state["ps"])
        return dict(fields=f, ps=state["ps"] if c["f64"] else state["ps"].float())
    if kind == "sweep":
        b = state["batch"]
        if c["noise"]:
            b.seed_noise(NOISE)
        else:
            b.set_signal(state["start"])
        b.run(c["rts"], 0.0)
        b.get_signal(state["out"])
        ps, rts, flags = b.results()
        return dict(signal=state["out"], ps=ps if c["f64"] else ps.astype(np.float32), rts=rts, flags=flags)
    if kind == "fft":
        return cu.fft_c2c(state["x"], c["sign"], out=state["out"])
    if kind == "train":
        # the late, small learning rate of a fine-tuning run
        m = state["mlp"]
        m.train_step(state["x"], state["t"], LR, loss=state["loss"])
        # (a copy: the gradient buffer is the network's own and goes with it)
        return dict(loss=state["loss"], grad=state["grad"].copy_(state["view"]))
    if kind == "infer":
        return state["mlp"].forward(state["x"])
    fields, power = state["model"].fields(state["pred"], c["n_t"])
    return dict(fields=fields, power=power.astype(np.float32))


NOISE = 1e-3   # noise amplitude of the noise-seeded sweeps
LR = 1e-5


# ---------------------------------------------------------------------- work

def _slice_flops(n_eqs, n_t):
    """Per point and slice: 2 transforms per field (5 log2 N each), both RK4 half steps, the dispersion factor."""
    return 10 * n_eqs * math.log2(n_t) + ((328 + 12) if n_eqs == 2 else (492 + 18))


def work(case):
    c, kind = case, case["kind"]
    e = 16 if c.get("f64") else 8
    if kind in ("pass", "cavity"):
        rts = c.get("rts", 1)
        flops = c["n_t"] * c["n_z"] * rts * _slice_flops(c["n_eqs"], c["n_t"])
        moved = (2 * c["n_eqs"] + (rts if c.get("ns") else 0)) * e * c["n_t"]   # fields in and out, the pump window
        return dict(bytes=moved, flops=flops)
    if kind == "sweep":
        nt = [i["n_t"] for i in _instances(c, 0)]
        return dict(bytes=2 * e * sum(nt),
                    flops=c["n_z"] * c["rts"] * sum(n * _slice_flops(c["n_eqs"], n) for n in nt))
    if kind == "fft":
        n = c["n"] * c["batch"]
        return dict(bytes=2 * e * n, flops=5 * n * math.log2(c["n"]))
    if kind in ("train", "infer"):
        p = sum(n * k for n, k in _dims())
        f = 2 * c["rows"] * p
        if kind == "infer":
            return dict(bytes=4 * p + 4 * c["rows"] * 516, flops=f)
        return dict(bytes=4 * 7 * p + 4 * c["rows"] * 516, flops=3 * f - 2 * c["rows"] * 4 * ws.WIDTH)
    return dict(bytes=c["count"] * (4 * 512 + 8 * c["n_t"]), flops=8.0 * 256 * c["count"] * c["n_t"])


# --------------------------------------------------------------------- exact

def _grids(n_t, t_rt):
    """Time and angular-frequency grids in float, as the solver's are (index times float step)."""
    f = np.float32

    def lin(lo, hi):
        lo, hi = f(lo), f(hi)
        return lo + np.arange(n_t).astype(f) * f(hi - lo) / f(n_t - 1)

    t = f(t_rt)
    df = f(1) / t
    F = np.fft.fftshift(lin(-0.5 * n_t * float(df), 0.5 * n_t * float(df)))
    w = f(2 * f(np.pi)) * F
    return lin(-0.5 * float(t), 0.5 * float(t)).astype(np.float64), w.astype(np.float64)


def _solve(p, A, per, rts, pump, f64, cavity):
    """FP64 restatement of the crystal pass and the cavity loop for a stack of
    instances A = [pump, signal(, idler)], each [instances][n_t]."""
    dev = A[0].device
    n, F, z = p["n_t"], p["n_eqs"], p["dz"]
    T, w = (torch.from_numpy(x).to(dev) for x in _grids(n, p["t_rt"]))
    gv = [1 / p["vp"] - 1 / p["vs"], 0.0] if F == 2 else [1 / p["vp"] - 1 / p["vi"], 0.0, 1 / p["vi"] - 1 / p["vs"]]
    b2, al = (p["b2p"], p["b2s"], p["b2i"]), ALPHA
    D = [math.exp(-0.5 * al[f] * z) * torch.exp(1j * z * w * (gv[f] + 0.5 * w * b2[f])) for f in range(F)]
    r = np.float64 if f64 else np.float32
    h = float(r(r(z) / r(2)))
    zs, zz = [], r(0)
    for _ in range(p["n_z"]):
        zs.append((float(zz), float(r(zz + r(z) / r(4))), float(r(zz + r(z) / r(2)))))
        zz = r(zz + r(z))
    kp, ks, ki, dk = 1j * p["kp"], 1j * p["ks"], 1j * p["ki"], p["dk"]

    def half(A, s):
        e = [complex(math.cos(dk * x), math.sin(dk * x)) for x in zs[s]]
        if F == 2:
            k = []
            P, S = A
            for j, c in ((0, 0.0), (1, 0.5), (1, 0.5), (2, 1.0)):
                a, b = (P + c * k[-1][0], S + c * k[-1][1]) if k else (P, S)
                k.append((kp * e[j] * b * b, ks * e[j].conjugate() * a * b.conj()))
            return [x + (h / 6) * (k[0][f] + 2 * (k[1][f] + k[2][f]) + k[3][f]) for f, x in enumerate(A)]
        g = e[0] + 4 * e[1] + e[2]
        P, S, I = A
        return [P + h / 6 * kp * g.conjugate() * S * I, S + h / 6 * ks * g * P * I.conj(),
                I + h / 6 * ki * g * P * S.conj()]

    def inv(x):
        return torch.fft.ifft(x, dim=-1, norm="forward")

    hist = []
    for rt in range(rts):
        if cavity:
            o = rt * n
            A[0] = (pump[o:o + n].to(torch.complex128).expand_as(A[1]).clone() if pump is not None
                    else per["ap0"].to(torch.complex128).expand_as(A[1]).clone())
        for s in range(p["n_z"]):
            A = half(A, s)
            A = [torch.fft.fft(inv(x) * D[f], dim=-1) / n for f, x in enumerate(A)]
            A = half(A, s)
        if not cavity:
            return A, None
        if p["use_eom"]:
            ef = torch.exp(1j * p["mod_depth"] * torch.sin(2 * math.pi * p["fpm"] * T))
            A[1:] = [x * ef for x in A[1:]]
        if bool((per["gdd"] != 0).any()):
            G = torch.exp(0.5j * w * w * per["gdd"])
            A[1:] = [torch.fft.fft(inv(x) * G, dim=-1) / n for x in A[1:]]
        A[1] = A[1] * (torch.sqrt(per["Rs"]) * torch.exp(1j * math.pi * per["delta"]))
        if F == 3:
            A[2] = A[2] * (math.sqrt(p["Ri"]) * torch.exp(1j * math.pi * per["delta"]))
        hist.append((A[1].abs() ** 2).mean(dim=-1))
    return A, torch.stack(hist)


def _noise(n, seed, stream):
    """Value i of stream (seed, stream): Philox4x32-10 on the counter (i, stream) and Box-Muller, as float."""
    i = np.arange(n, dtype=np.uint64)
    m32 = np.uint64(0xFFFFFFFF)
    s32 = np.uint64(32)
    c = [i & m32, i >> s32, np.full(n, stream, np.uint64), np.zeros(n, np.uint64)]
    k = [seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF]
    for _ in range(10):
        a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> s32) ^ c[1] ^ np.uint64(k[0]), b & m32, (a >> s32) ^ c[3] ^ np.uint64(k[1]), a & m32]
        k = [(k[0] + 0x9E3779B9) & 0xFFFFFFFF, (k[1] + 0xBB67AE85) & 0xFFFFFFFF]
    u1 = (((c[0] << np.uint64(21)) ^ c[1]).astype(np.float64) + 1.0) / 9007199254740992.0
    u2 = (((c[2] << np.uint64(21)) ^ c[3]).astype(np.float64) + 1.0) / 9007199254740992.0
    r = NOISE * np.sqrt(-2.0 * np.log(u1))
    return ((r * np.cos(2 * np.pi * u2)).astype(np.float32) + 1j * (r * np.sin(2 * np.pi * u2)).astype(np.float32))


def _exact_sweep(c, seed):
    inst = _instances(c, seed)
    offs = np.concatenate([[0], np.cumsum([i["n_t"] for i in inst])])
    total = int(offs[-1])
    if c["noise"]:
        sig = torch.from_numpy(np.concatenate([_noise(i["n_t"], i["seed"], 0) for i in inst])).cuda().to(torch.complex128)
        idl = torch.from_numpy(np.concatenate([_noise(i["n_t"], i["seed"], 1) for i in inst])).cuda().to(torch.complex128)
    else:
        sig, idl = _field(total, 0.3, seed, c["f64"]).to(torch.complex128), None
    ps = torch.zeros(len(inst), dtype=torch.float64, device="cuda")
    for n in sorted({i["n_t"] for i in inst}):
        ids = [k for k, i in enumerate(inst) if i["n_t"] == n]
        at = torch.cat([torch.arange(offs[k], offs[k + 1], device="cuda") for k in ids])
        per = {f: torch.tensor([inst[k][f] for k in ids], dtype=torch.float64, device="cuda")[:, None]
               for f in ("ap0", "Rs", "delta", "gdd")}
        S = sig[at].reshape(len(ids), n)
        A = [torch.zeros_like(S), S] + ([idl[at].reshape(len(ids), n)] if c["n_eqs"] == 3 else [])
        A, hist = _solve(_params(c, n), A, per, c["rts"], None, c["f64"], True)
        sig[at] = A[1].reshape(-1)
        ps[torch.tensor(ids, device="cuda")] = hist[-1]
    return dict(signal=sig, ps=ps, rts=None, flags=None)


def _gelu(z):
    phi = 0.5 * (1 + torch.erf(z / math.sqrt(2)))
    return z * phi, phi + z * torch.exp(-0.5 * z * z) / math.sqrt(2 * math.pi)


def _exact_net(c, seed):
    flat = torch.from_numpy(_weights(seed)).cuda().double()
    x, t = _rows(c, seed)
    W, B, o = [], [], 0
    for n, k in _dims():
        W.append(flat[o:o + n * k].reshape(n, k))
        B.append(flat[o + n * k:o + n * k + n])
        o += n * k + n
    a, acts, gps = x.double(), [], []
    for l in range(len(W)):
        acts.append(a)
        z = a @ W[l].T + B[l]
        if l + 1 < len(W):
            a, gp = _gelu(z)
            gps.append(gp)
        else:
            a = z
    if c["kind"] == "infer":
        return a
    d = a - t.double()
    g = 2 * d / d.numel()
    grads = []
    for l in range(len(W) - 1, -1, -1):
        gw = g.T @ acts[l]
        if l == 0:   # the gradient buffer keeps layer 0's inputs padded to 64
            gw = torch.cat([gw, torch.zeros(gw.shape[0], 64 - gw.shape[1], dtype=gw.dtype, device="cuda")], dim=1)
        grads = [gw.reshape(-1), g.sum(dim=0)] + grads
        if l:
            g = (g @ W[l]) * gps[l - 1]
    return dict(loss=(d * d).mean().reshape(1), grad=torch.cat(grads))


def _exact_bands(c, seed):
    y = _prediction(c, seed).double()
    n_t = c["n_t"]
    mag = y[:, :256].clamp_min(0)
    phi = torch.atan2(y[:, 320:384].mean(1), y[:, 256:320].mean(1))
    q0 = torch.round(torch.sqrt((0.5 * (y[:, 384:448].mean(1) + 1)).clamp_min(0)) * (n_t / 2))
    q0 = q0.clamp(64, n_t // 2 - 64).long()
    power = 10 ** y[:, 448:512].mean(1)
    amp = torch.sqrt(power / (mag ** 2).sum(1))
    coef = mag * (amp * torch.exp(0.5j * phi))[:, None]
    k = torch.arange(128, device="cuda") - 64
    q = torch.cat([(q0[:, None] + k) % n_t, (-q0[:, None] + k) % n_t], dim=1)
    spec = torch.zeros(c["count"], n_t, dtype=torch.complex128, device="cuda").scatter_add_(1, q, coef)
    return dict(fields=torch.fft.ifft(spec, dim=-1, norm="forward"), power=power)


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("pass", "cavity"):
        p = _params(c, c["n_t"])
        A = [f.to(torch.complex128)[None, :] for f in _start(c, seed)]
        per = {k: torch.tensor([[p[k]]], dtype=torch.float64, device="cuda") for k in ("ap0", "Rs", "delta", "gdd")}
        pump = _window(c, p, seed) if c.get("ns") else None
        A, hist = _solve(p, A, per, c.get("rts", 1), pump, c["f64"], kind == "cavity")
        A = [a[0] for a in A]
        return A if kind == "pass" else dict(fields=A, ps=hist[:, 0])
    if kind == "sweep":
        return _exact_sweep(c, seed)
    if kind == "fft":
        x = _field(c["batch"] * c["n"], 1.0, seed, c["f64"]).reshape(c["batch"], c["n"]).to(torch.complex128)
        return torch.fft.fft(x, dim=-1) if c["sign"] < 0 else torch.fft.ifft(x, dim=-1, norm="forward")
    if kind in ("train", "infer"):
        return _exact_net(c, seed)
    return _exact_bands(c, seed)
