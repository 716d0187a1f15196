"""Performance cases of the package: what its users have it do, through its public calls.

A case is a dict of plain values.  ``prepare`` makes what a program holds
before the call, ``run`` makes one call, ``work`` counts the bytes and
operations the call cannot do without and ``exact`` computes the same outputs
in 64 bits with plain numpy and torch.

Kinds of case:

``single``    one run of the drop-in class with its TL grid, host arrays in,
              host arrays out: the smallest calls, where latency counts
``shared``    environments x frequencies on one grid, with TL grids: a
              broadband run of the drop-in class
``munk``      a batch prepared by a worker process and marched by the main
              one (``Engine(batch).run()``): deep water, equal depths
``wedge``     the same with uneven rays: every slope, frequency, range and
              Pade order of the wedge workload
``predict``   ensemble inference on requests, mean and spread of the fields
``train``     one training step of one ensemble member
``gemm``      one contraction with the surrogate's epilogues
"""
import math

import numpy as np
import torch

from cupyram_b200 import CuPyRAM
from cupyram_b200 import surrogate as S
from cupyram_b200 import workloads as W
from cupyram_b200.engine import Engine


def listed():
    return [
        # RAM's own test size: a sloping bottom, 500 m steps, grid output.  The call a notebook makes.
        dict(name="ram_single", kind="single", freq=50.0, depth=200.0, depth2=400.0, rmax=50000.0, dr=500.0, dz=2.0,
             np=8, ndr=1, ndz=1, precision="plain"),
        # the Pekeris benchmark ray: 2401 depths, 5000 steps; one long march
        dict(name="pekeris_single", kind="single", freq=50.0, depth=100.0, depth2=100.0, rmax=10000.0, dr=2.0,
             dz=0.25, np=8, ndr=1, ndz=4, precision="plain"),
        # the same guide in the complex64 form that a user picks for speed
        dict(name="pekeris_chosen", kind="single", freq=50.0, depth=100.0, depth2=100.0, rmax=4000.0, dr=2.0,
             dz=0.25, np=8, ndr=1, ndz=4, precision="chosen"),
        # a broadband run: 4 environments x 16 frequencies, every ray with its grid
        dict(name="broadband", kind="shared", envs=4, freqs=16, fmin=50.0, fmax=200.0, depth=300.0, rmax=5000.0,
             np=6, ndr=2, ndz=4),
        # the headline batch (4096 rays, 5000 m, 25 m steps, np 6) over a shorter track
        dict(name="munk_4096", kind="munk", rays=4096, depth=5000.0, rmax=5000.0, update=2500.0, np=6,
             precision="plain"),
        # a batch that does not fill the GPU, with the remainder of a tile
        dict(name="munk_301", kind="munk", rays=301, depth=5000.0, rmax=10000.0, update=5000.0, np=6,
             precision="plain"),
        # the FP32 form of the headline batch
        dict(name="munk_fast", kind="munk", rays=4096, depth=5000.0, rmax=2500.0, update=2500.0, np=6,
             precision="fast"),
        # the form that recovers complex128 from complex64 sweeps, on part of a batch
        dict(name="munk_refined", kind="munk", rays=900, depth=2500.0, rmax=2500.0, update=2500.0, np=6,
             precision="refined"),
        # uneven rays: depth, range, steps and Pade order all differ
        dict(name="wedge_256", kind="wedge", rays=256, layout=7, track=0.25),
        # an ensemble of four answers a chunk of requests
        dict(name="predict_4000", kind="predict", requests=4000, members=4, width=512),
        # one step of training on the batch size the pipeline uses
        dict(name="train_512", kind="train", batch=512, width=512),
        # the output layer's contraction, 8192 requests
        dict(name="gemm_out", kind="gemm", m=8192, n=8192, k=512, epi="f32"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["single", "single", "shared", "munk", "munk", "wedge", "predict", "train", "gemm"])
    if kind == "single":
        depth = _log(rng, 80.0, 1000.0)
        dz = round(depth / _log(rng, 60.0, 400.0), 3)
        dr = round(_log(rng, 4.0, 200.0), 2)
        return dict(kind=kind, freq=round(_log(rng, 25.0, 150.0), 2), depth=round(depth, 1),
                    depth2=round(depth * rng.choice([1.0, rng.uniform(0.7, 1.4)]), 1),
                    rmax=round(dr * _log(rng, 60.0, 3000.0), 1), dr=dr, dz=dz, np=rng.randint(3, 8),
                    ndr=rng.randint(1, 4), ndz=rng.randint(1, 5), precision="plain")
    if kind == "shared":
        return dict(kind=kind, envs=rng.randint(1, 5), freqs=rng.randint(2, 14), fmin=round(rng.uniform(30.0, 60.0), 1),
                    fmax=round(rng.uniform(90.0, 200.0), 1), depth=round(rng.uniform(80.0, 300.0), 1),
                    rmax=round(rng.uniform(1000.0, 4000.0), 1), np=rng.randint(4, 8), ndr=rng.randint(1, 3),
                    ndz=rng.randint(2, 6))
    if kind == "munk":
        rays = int(_log(rng, 24.0, 800.0))
        return dict(kind=kind, rays=rays, depth=10.0 * rng.randint(150, 500),
                    rmax=round(min(10000.0, 400000.0 / rays + 1000.0), 1), update=5000.0, np=rng.randint(4, 8),
                    precision=rng.choice(["plain", "plain", "refined"]))
    if kind == "wedge":
        return dict(kind=kind, rays=int(_log(rng, 4.0, 200.0)), layout=rng.randint(0, 1 << 20),
                    track=round(_log(rng, 0.03, 0.25), 3))
    if kind == "predict":
        return dict(kind=kind, requests=int(_log(rng, 100.0, 4000.0)), members=rng.randint(2, 4),
                    width=rng.choice([256, 512]))
    if kind == "train":
        return dict(kind=kind, batch=128 * rng.randint(1, 8), width=rng.choice([256, 512]))
    return dict(kind=kind, m=128 * int(_log(rng, 1.0, 64.0)), n=256 * int(_log(rng, 1.0, 32.0)),
                k=64 * int(_log(rng, 1.0, 16.0)), epi=rng.choice(["f32", "bias_f32", "bias_relu", "mask"]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _single_args(c, seed):
    """A shallow-water run: a measured-looking profile over a sediment half-space."""
    rng = np.random.Generator(np.random.PCG64(seed))
    deepest = max(c["depth"], c["depth2"])
    z = np.array([0.0, 0.25, 0.5, 1.0]) * deepest
    cw = 1500.0 + rng.uniform(-15.0, 15.0, 4)[:, None]
    zs = max(1.1 * c["dz"], rng.uniform(0.2, 0.5) * min(c["depth"], c["depth2"]))
    zr = rng.uniform(0.2, 0.8) * min(c["depth"], c["depth2"])
    cb = rng.uniform(1600.0, 1800.0)
    args = [c["freq"], zs, zr, z, np.array([0.0]), cw, np.array([0.0, 200.0]), np.array([0.0]),
            np.full((2, 1), cb), np.full((2, 1), rng.uniform(1.4, 1.9)), np.full((2, 1), rng.uniform(0.3, 0.8)),
            np.array([[0.0, c["depth"]], [c["rmax"], c["depth2"]]])]
    kw = dict(rmax=c["rmax"], dr=c["dr"], dz=c["dz"], np=c["np"], ns=1, lyrw=10, ndr=c["ndr"], ndz=c["ndz"],
              c0=1500.0, precision=c["precision"])
    return args, kw


def _shared_args(c, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    n, rmax = c["envs"], c["rmax"]
    depth = c["depth"] * rng.uniform(0.85, 1.0, (n, 2))
    z = [np.array([0.0, 0.3, 0.6, 1.0]) * c["depth"]] * n
    rp = [np.array([0.0, 0.4, 0.8]) * rmax] * n
    cw = [1500.0 + rng.uniform(-12.0, 12.0, (4, 3)) for _ in range(n)]
    freq = list(np.linspace(c["fmin"], c["fmax"], c["freqs"]))
    args = [freq, 0.3 * c["depth"], 0.5 * c["depth"], z, rp, cw,
            [np.array([0.0, 100.0])] * n, [np.array([0.0])] * n,
            [np.full((2, 1), v) for v in rng.uniform(1600.0, 1800.0, n)],
            [np.full((2, 1), v) for v in rng.uniform(1.4, 1.9, n)],
            [np.full((2, 1), v) for v in rng.uniform(0.3, 0.8, n)],
            [np.array([[0.0, d[0]], [rmax, d[1]]]) for d in depth]]
    lam = 1500.0 / c["fmax"]
    kw = dict(batch_size=n, rmax=rmax, dr=round(2.0 * lam, 2), dz=round(0.1 * lam, 3), np=c["np"], ndr=c["ndr"],
              ndz=c["ndz"], c0=1500.0, zmplt=0.8 * c["depth"])
    return args, kw


def _batch_args(c, seed):
    if c["kind"] == "munk":
        return W.munk_batch(n_rays=c["rays"], seed=seed, depth=c["depth"], rmax=c["rmax"], update=c["update"],
                            np_pade=c["np"])
    # the layout's rays (depths, slopes, frequencies, ranges, Pade orders) over part of their tracks, other bottoms
    args, kw = W.wedge_batch(n_rays=c["rays"], seed=c["layout"])
    rng = np.random.Generator(np.random.PCG64(seed))
    kw["rmax"] = c["track"] * kw["rmax"]
    for k, lo, hi in ((8, 1550.0, 1800.0), (9, 1.3, 2.0), (10, 0.2, 1.0)):
        args[k] = [np.full((2, 1), v) for v in rng.uniform(lo, hi, c["rays"])]
    args[11] = [b * [[1.0, 1.0], [c["track"], 1.0]] for b in args[11]]
    return args, kw


_EPI = {"f32": S.EPI_F32, "bias_f32": S.EPI_BIAS_F32, "bias_relu": S.EPI_BIAS_RELU_BF16, "mask": S.EPI_RELU_MASK_BF16}


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "single":
        args, kw = _single_args(c, seed)
        return {"kind": kind, "ram": CuPyRAM(*args, **kw)}
    if kind == "shared":
        args, kw = _shared_args(c, seed)
        return {"kind": kind, "ram": CuPyRAM(*args, **kw)}
    if kind in ("munk", "wedge"):
        args, kw = _batch_args(c, seed)
        return {"kind": kind, "batch": W.build(args, kw), "precision": c.get("precision", "plain")}
    g = torch.Generator(device="cuda").manual_seed(seed)
    if kind == "predict":
        ens = S.Ensemble(c["members"], S.default_dims(c["width"]), seed=seed)
        return {"kind": kind, "ens": ens, "X": S.to_device_inputs(S.features(S.requests(c["requests"], seed)))}
    if kind == "train":
        B = c["batch"]
        m = S.MLP(S.default_dims(c["width"]), seed=seed)
        X = S.to_device_inputs(S.features(S.requests(4 * B, seed)))
        Y = (0.5 * torch.randn(4 * B, S.NZ_OUT * S.NR_OUT, generator=g, device="cuda")).to(torch.bfloat16)
        idx = torch.randperm(4 * B, generator=g, device="cuda")[:B]
        valid = torch.ones(B * Y.shape[1], dtype=torch.uint8, device="cuda")
        return {"kind": kind, "m": m, "X": X, "Y": Y, "idx": idx, "valid": valid,
                "sse": torch.zeros(1, dtype=torch.float64, device="cuda")}
    M, N, K = c["m"], c["n"], c["k"]
    A = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    B = (torch.randn(N, K, generator=g, device="cuda") / math.sqrt(K)).to(torch.bfloat16)
    half = c["epi"] in ("bias_relu", "mask")
    out = torch.empty(M, N, dtype=torch.bfloat16 if half else torch.float32, device="cuda")
    bias = torch.randn(N, generator=g, device="cuda") if c["epi"].startswith("bias") else None
    mask = torch.relu(torch.randn(M, N, generator=g, device="cuda")).to(torch.bfloat16) if c["epi"] == "mask" else None
    return {"kind": kind, "epi": _EPI[c["epi"]], "A": A, "B": B, "out": out, "bias": bias, "mask": mask}


def run(s):
    kind = s["kind"]
    if kind in ("single", "shared"):
        r = s["ram"].run()
        return [r["TL Line"], r["CP Line"], r["TL Grid"], r["CP Grid"]]
    if kind in ("munk", "wedge"):
        with Engine(s["batch"], precision=s["precision"]) as eng:
            out = eng.run()
        return [out["tll"], out["cpl"]]
    if kind == "predict":
        return list(s["ens"].predict(s["X"]))
    if kind == "train":
        m, B = s["m"], s["idx"].numel()
        s["sse"].zero_()
        xb = s["X"].index_select(0, s["idx"])
        yb = s["Y"].index_select(0, s["idx"])
        S.mse_grad(m.forward(xb), yb, s["valid"], s["valid"].numel(), m.grad_buffer(B), s["sse"])
        m.backward(m.grad_buffer(B))
        m.step(1e-3)
        return [s["sse"], m.gW, m.gb, m.W, m.b]
    S.gemm(s["epi"], s["A"], s["B"], s["out"], bias=s["bias"], mask=s["mask"])
    return s["out"]


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _rays(c, seed=0):
    """(per-ray grids, environments) of a march case, in plain numpy."""
    kind = c["kind"]
    if kind == "single":
        args, kw = _single_args(c, seed)
    elif kind == "shared":
        args, kw = _shared_args(c, seed)
    else:
        args, kw = _batch_args(c, seed)
    n = kw.get("batch_size", 1)

    def per_env(x):
        return [np.asarray(v, np.float64) for v in x] if isinstance(x, list) else [np.asarray(x, np.float64)] * n

    names = ["z_ss", "rp_ss", "cw", "z_sb", "rp_sb", "cb", "rhob", "attn", "rbzb"]
    envs = [dict(zip(names, v)) for v in zip(*(per_env(a) for a in args[3:]))]
    for e in envs:
        e["z_sb"] = e["z_sb"] + e["z_ss"][-1]
    freqs = np.atleast_1d(np.asarray(args[0], np.float64))
    paired = bool(kw.get("per_ray"))
    pick = (lambda key, i, dflt: np.broadcast_to(np.asarray(kw.get(key, dflt)), (n,))[i])
    c0 = [float(pick("c0", i, np.nan)) for i in range(n)]
    c0 = [float(np.mean(e["cw"][:, 0])) if np.isnan(v) else v for v, e in zip(c0, envs)]
    rays = []
    for i in range(n):
        for f in ([freqs[i]] if paired else freqs):
            lam = (c0[i] / f) if paired else np.mean(c0) / freqs.max()
            lyr = kw.get("lyrw", 20) * lam
            zmax = (envs[i]["z_sb"].max() if paired else max(e["z_sb"].max() for e in envs)) + lyr
            dr, dz, rmax = float(pick("dr", i, 0.0)), float(pick("dz", i, 0.0)), float(pick("rmax", i, 0.0))
            ndr, ndz = int(pick("ndr", i, 1)), int(pick("ndz", i, 1))
            zplt = envs[i]["rbzb"][:, 1].max() if paired else max(e["rbzb"][:, 1].max() for e in envs)
            zplt = float(pick("zmplt", i, zplt))
            nvr = int(np.floor(rmax / (dr * ndr)))
            rays.append(dict(env=i, freq=float(f), c0=c0[i], zmax=zmax, lyr=lyr, dr=dr, dz=dz, ndr=ndr, ndz=ndz,
                             nz=int(np.floor(zmax / dz) - 1), nvr=nvr, nvz=int(np.floor(zplt / dz)) // ndz,
                             nr=int(np.round(nvr * dr * ndr / dr) - 1), np=int(pick("np", i, 8)),
                             ns=int(kw.get("ns", 1)), rs=rmax + dr, rmax=rmax,
                             zs=float(np.broadcast_to(np.asarray(args[1]), (n,))[i]),
                             zr=float(np.broadcast_to(np.asarray(args[2]), (n,))[i])))
    return rays, envs


def work(case):
    c, kind = case, case["kind"]
    if kind in ("single", "shared", "munk", "wedge"):
        rays, envs = _rays(c)
        # per point and Pade term a tridiagonal solve (18 multiply-adds) and its share of the sum (4)
        flops = 2.0 * sum(r["nz"] * r["nr"] * r["np"] * 22 for r in rays)
        outs = sum(24.0 * r["nvr"] * (1 + (r["nvz"] if kind in ("single", "shared") else 0)) for r in rays)
        ins = sum(8.0 * sum(v.size for v in e.values()) for e in envs)
        # the field of a ray and its factors fit the chip: only inputs and outputs have to cross memory
        return {"bytes": ins + outs, "flops": flops}
    if kind == "gemm":
        M, N, K = c["m"], c["n"], c["k"]
        ob = 2 if c["epi"] in ("bias_relu", "mask") else 4
        more = 4 * N if c["epi"].startswith("bias") else (2 * M * N if c["epi"] == "mask" else 0)
        return {"bytes": 2.0 * K * (M + N) + ob * M * N + more, "flops": 2.0 * M * N * K}
    d = S.default_dims(c["width"])
    weights = sum(a * b for a, b in zip(d[:-1], d[1:]))
    if kind == "predict":
        n = -(-c["requests"] // 128) * 128
        return {"bytes": c["members"] * 2.0 * weights + 2.0 * n * d[0] + 8.0 * n * d[-1],
                "flops": 2.0 * c["members"] * n * weights}
    B = c["batch"]
    return {"bytes": weights * (4.0 * 3 * 2 + 4 + 2 * 2) + B * (2.0 * d[0] + 2.0 * d[-1]), "flops": 6.0 * B * weights}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------
def _pade(freq, c0, n, ns, dr, ip):
    """Coefficients of prod (1 + a_j X) / (1 + b_j X) ~ exp(i k0 dr (sqrt(1 + X) - 1)) [(1 + X)^-1/4 (1 - X)^2]
    matched at X = 0 to order 2n, less ns stability constraints (Collins)."""
    ld, cl = np.longdouble, np.clongdouble
    sig = ld(2.0) * ld(np.pi) * ld(freq) / ld(c0) * ld(dr)
    nu, alp = (0.0, 0.0) if ip == 1 else (1.0, -0.25)
    m = 2 * n
    # Taylor series of the operator from its logarithmic derivative, (log F)' = sum of three simple terms
    t = np.zeros(m + 1, cl)
    ser = np.zeros(m + 1, cl)
    root = ld(0.5)  # coefficients of (1 + X)^(-1/2) / 2
    geo, inv = ld(1.0), ld(1.0)
    for k in range(m + 1):
        ser[k] = cl(1j) * sig * root + ld(alp) * geo - ld(2.0 * nu) * inv
        root = root * (ld(-0.5) - k) / (k + 1)
        geo = -geo
    t[0] = 1.0
    for k in range(m):
        t[k + 1] = sum(ser[j] * t[k - j] for j in range(k + 1)) / (k + 1)
    A = np.zeros((m, m), cl)  # unknowns: numerator 1..n, denominator 1..n
    b = np.zeros(m, cl)
    for i in range(1, m + 1):
        if i <= n:
            A[i - 1, i - 1] = 1.0
        for j in range(1, min(i, n) + 1):
            A[i - 1, n + j - 1] = -t[i - j]
        b[i - 1] = t[i]
    for k in range(min(ns, 2)):
        A[m - 1 - k] = 0.0
        A[m - 1 - k, :n] = np.cumprod(np.full(n, ld((-3.0, -1.5)[k])))
        b[m - 1 - k] = -1.0
    for i in range(m):  # elimination with partial pivoting, extended precision
        p = i + int(np.argmax(np.abs(A[i:, i])))
        A[[i, p]], b[[i, p]] = A[[p, i]], b[[p, i]]
        for k in range(i + 1, m):
            f = A[k, i] / A[i, i]
            A[k, i:] -= f * A[i, i:]
            b[k] -= f * b[i]
    x = np.zeros(m, cl)
    for i in range(m - 1, -1, -1):
        x[i] = (b[i] - A[i, i + 1:] @ x[i + 1:]) / A[i, i]
    out = []
    for co in (x[:n], x[n:]):
        # 1 + sum co_k X^k = prod (1 + a_j X): the a_j are the negated roots of the reversed polynomial
        poly = np.concatenate([np.ones(1, cl), co])
        r = np.roots(poly.astype(np.complex128)).astype(cl)
        der = poly[:-1] * np.arange(n, 0, -1)
        for _ in range(6):
            r = r - np.polyval(poly, r) / np.polyval(der, r)
        out.append(-r)
    return out


def _fractions(num, den):
    """c_inf and the residues c_k of prod (1 + num_j X) / (1 + den_j X)."""
    ck = np.zeros(len(den), np.clongdouble)
    for k in range(len(den)):
        ck[k] = 1 - num[k] / den[k]
        for j in range(len(den)):
            if j != k:
                ck[k] *= (1 - num[j] / den[k]) / (1 - den[j] / den[k])
    return np.prod(num / den), ck


def _table(z, x, y):
    """Piecewise-linear y(x) at z, constant outside; at a repeated x the later value holds."""
    if x.size == 1:
        return np.full(z.size, y[0])
    k = np.clip(np.searchsorted(x, z, side="right") - 1, 0, x.size - 2)
    w = x[k + 1] - x[k]
    v = y[k] + (y[k + 1] - y[k]) * ((z - x[k]) / np.where(w == 0, 1.0, w))
    return np.where(z <= x[0], y[0], np.where(z >= x[-1], y[-1], v))


def _rows(r, e, ss, sb, iz, n):
    """f1, f2, f3 and ksq of rows 0..n-1 (stored to 32 bits, as the method's definition has them)."""
    nz = r["nz"]
    z = np.arange(nz + 2) * (r["zmax"] / (nz + 1))
    z[-1] = r["zmax"]
    k0, om = 2 * np.pi * r["freq"] / r["c0"], 2 * np.pi * r["freq"]
    cw = _table(z, e["z_ss"], e["cw"][:, ss]).astype(np.float32).astype(np.float64)
    cb = _table(z, e["z_sb"], e["cb"][:, sb]).astype(np.float32)
    rho = _table(z, e["z_sb"], e["rhob"][:, sb]).astype(np.float32)
    at, zl = _table(z, e["z_sb"], e["attn"][:, sb]), e["z_sb"][-1]
    last = e["attn"][-1, sb]
    ramp = np.clip((z - (zl + 0.75 * r["lyr"])) / (0.25 * r["lyr"]), 0.0, 1.0)
    at = np.where(z <= zl, at, last + (10.0 - last) * ramp).astype(np.float32).astype(np.float64)
    water = np.arange(nz + 2) <= iz
    alpw = np.sqrt(cw / r["c0"])
    alpb = np.sqrt((rho * cb).astype(np.float64) / r["c0"])
    cbd, rhod = cb.astype(np.float64), rho.astype(np.float64)
    wave = om / cbd * (1 + 1j * at / (40 * np.pi * 0.43429448190325176))
    f = [np.where(water, 1 / alpw, rhod / alpb), np.where(water, 1.0, 1 / rhod), np.where(water, alpw, alpb)]
    f = [v.astype(np.float32).astype(np.float64) for v in f]
    k = np.where(water, (om / cw) ** 2 - k0 ** 2, wave ** 2 - k0 ** 2).astype(np.complex64).astype(np.complex128)
    pad = n - (nz + 2)
    return [np.pad(v, (0, pad)) for v in f] + [np.pad(k, (0, pad))]


class _Rotor:
    """Solves batches of tridiagonal systems by parallel cyclic reduction, in complex128, with stored factors."""

    def __init__(self, lo, di, up):
        self.levels, s, n = [], 1, di.shape[-1]
        while s < n:
            # row i less its neighbours at distance s
            ka, kc = torch.zeros_like(di), torch.zeros_like(di)
            ka[..., s:] = -lo[..., s:] / di[..., :-s]
            kc[..., :-s] = -up[..., :-s] / di[..., s:]
            self.levels.append((s, ka, kc))
            nlo, nup, ndi = torch.zeros_like(di), torch.zeros_like(di), di.clone()
            ndi[..., s:] += ka[..., s:] * up[..., :-s]
            ndi[..., :-s] += kc[..., :-s] * lo[..., s:]
            nlo[..., s:] = ka[..., s:] * lo[..., :-s]
            nup[..., :-s] = kc[..., :-s] * up[..., s:]
            lo, di, up, s = nlo, ndi, nup, 2 * s
        self.inv = 1 / di

    def solve(self, b):
        for s, ka, kc in self.levels:
            d = b.clone()
            d[..., s:] += ka[..., s:] * b[..., :-s]
            d[..., :-s] += kc[..., :-s] * b[..., s:]
            b = d
        return b * self.inv


def _march(rays, envs, grids):
    """TL and complex pressure of every ray (lists), all rays in step."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    B, n, T = len(rays), max(r["nz"] for r in rays) + 2, max(r["np"] for r in rays)
    to = (lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev))
    col = (lambda v: to(np.asarray(v, np.float64))[:, None])
    rows = np.arange(n)[None, :]
    inside = to((rows >= 1) & (rows <= np.asarray([r["nz"] for r in rays])[:, None]))
    k0 = np.asarray([2 * np.pi * r["freq"] / r["c0"] for r in rays])
    a1, a2, cf = col(k0 ** 2 / 6), col(2 * k0 ** 2 / 3), col([0.5 / r["dz"] ** 2 for r in rays])

    # operator sets: two self-starter factors, the march; (poles, residues, c_inf) per ray
    def operator(which):
        p, ck, ci = np.zeros((B, T), complex), np.zeros((B, T), complex), np.zeros(B, complex)
        known = {}
        for i, r in enumerate(rays):
            if which == "smooth":
                num, den = np.zeros(1, np.clongdouble), np.full(1, -1, np.clongdouble)
                p[i, 0], ck[i, 0] = -1, 1
                continue
            key = (r["freq"], r["c0"], r["np"], r["ns"], r["dr"])
            if key not in known:
                known[key] = _pade(*key[:4], key[4], 2 if which == "start" else 1)
            num, den = known[key]
            ci[i], c = _fractions(num, den)
            p[i, :len(den)], ck[i, :len(den)] = den, c
        return to(p), to(ck)[:, :, None], to(ci)[:, None]

    state = [dict(ss=0, sb=0, bt=0, iz=0) for _ in rays]
    bath = []
    for r, s in zip(rays, state):
        b = envs[r["env"]]["rbzb"]
        if b[-1, 0] < r["rmax"]:
            b = np.vstack([b, [r["rmax"], b[-1, 1]]])
        bath.append(b)
        s["iz"] = max(1, min(r["nz"] - 1, int(np.floor(b[0, 1] / r["dz"]))))
    F = [np.zeros((B, n)) for _ in range(3)] + [np.zeros((B, n), complex)]

    def assemble(i):
        for dst, v in zip(F, _rows(rays[i], envs[rays[i]["env"]], state[i]["ss"], state[i]["sb"], state[i]["iz"], n)):
            dst[i] = v

    for i in range(B):
        assemble(i)

    def system(op):
        f1, f2, f3, k = (to(v) for v in F)
        c = torch.zeros((3, B, n), dtype=torch.complex128, device=dev)
        m, q = slice(1, -1), f2[:, :-1] + f2[:, 1:]
        c[0][:, m] = cf * f1[:, m] * q[:, :-1] * f3[:, :-2] + (k[:, :-2] + k[:, m]) / 12
        c[1][:, m] = -cf * f1[:, m] * (q[:, :-1] + q[:, 1:]) * f3[:, m] + (k[:, :-2] + 6 * k[:, m] + k[:, 2:]) / 12
        c[2][:, m] = cf * f1[:, m] * q[:, 1:] * f3[:, 2:] + (k[:, m] + k[:, 2:]) / 12
        p = op[0][:, :, None]
        lo, di, up = (torch.where(inside[:, None], a[:, None] + p * d[:, None], torch.full_like(p, fill))
                      for a, d, fill in ((a1, c[0], 0.0), (a2, c[1], 1.0), (a1, c[2], 0.0)))
        lo[..., 1] = 0
        return _Rotor(lo, di, torch.where(inside[:, None].roll(-1, -1), up, torch.zeros_like(up)))

    def step(u, op, sol):
        b = a2 * u
        b[:, 1:] += a1 * u[:, :-1]
        b[:, :-1] += a1 * u[:, 1:]
        x = sol.solve((b * inside)[:, None].expand(B, T, n))
        return (op[2] * u + (op[1] * x).sum(1)) * inside

    u0 = np.zeros((B, n), complex)
    for i, r in enumerate(rays):
        e, si = envs[r["env"]], r["zs"] / r["dz"]
        js = int(np.floor(si))
        for j, w in ((js, 1 - (si - js)), (js + 1, si - js)):
            z = np.asarray([r["zmax"] if j == r["nz"] + 1 else j * (r["zmax"] / (r["nz"] + 1))])
            alp = np.sqrt(np.float64(np.float32(_table(z, e["z_ss"], e["cw"][:, 0])[0])) / r["c0"])
            if 1 <= j <= r["nz"]:
                u0[i, j] += w * np.sqrt(2 * np.pi / k0[i]) / (r["dz"] * alp)
    u = to(u0)
    op = operator("smooth")
    sol = system(op)
    u = step(step(u, op, sol), op, sol)
    op = operator("start")
    u = step(u, op, system(op))
    op = operator("march")
    sol = system(op)

    ir = np.asarray([int(np.floor(r["zr"] / r["dz"])) for r in rays])
    dir_ = np.asarray([r["zr"] / r["dz"] for r in rays]) - ir
    at, wa, wb, every = to(ir)[:, None], col(1 - dir_)[:, 0], col(dir_)[:, 0], torch.arange(B, device=dev)
    f3 = to(F[2])
    line, grid = [[] for _ in rays], [[] for _ in rays]
    depth = [to((np.arange(r["nvz"]) + 1) * r["ndz"]) for r in rays] if grids else None

    def emit(k):  # the field after range k + 1
        v = u * f3
        p = wa * v[every, at[:, 0]] + wb * v[every, at[:, 0] + 1]
        for i, r in enumerate(rays):
            if (k + 1) % r["ndr"] == 0 and (k + 1) // r["ndr"] <= r["nvr"] and k <= r["nr"]:
                line[i].append(p[i])
                if grids:
                    grid[i].append(v[i][depth[i]])

    emit(0)
    for k in range(max(r["nr"] for r in rays)):
        changed = False
        for i, (r, s) in enumerate(zip(rays, state)):
            if k >= r["nr"]:
                continue
            e, b, x = envs[r["env"]], bath[i], (r["dr"] if k == 0 else (k + 1) * r["dr"])
            old = (s["ss"], s["sb"], s["iz"])
            while s["bt"] < len(b) - 1 and x >= b[s["bt"] + 1, 0]:
                s["bt"] += 1
            j = min(s["bt"] + 1, len(b) - 1)
            zc = b[s["bt"], 1]
            if j != s["bt"]:
                zc = zc + (x + 0.5 * r["dr"] - b[s["bt"], 0]) * (b[j, 1] - zc) / (b[j, 0] - b[s["bt"], 0])
            s["iz"] = max(1, min(r["nz"] - 1, int(np.floor(zc / r["dz"]))))
            while s["ss"] < e["rp_ss"].size - 1 and x >= e["rp_ss"][s["ss"] + 1]:
                s["ss"] += 1
            while s["sb"] < e["rp_sb"].size - 1 and x >= e["rp_sb"][s["sb"] + 1]:
                s["sb"] += 1
            if old != (s["ss"], s["sb"], s["iz"]):
                assemble(i)
                changed = True
        if changed:
            sol, f3 = system(op), to(F[2])
        u = step(u, op, sol)
        emit(k + 1)
    tl, cp = [], []
    for i, r in enumerate(rays):
        x = 10 * np.log10((np.arange(len(line[i])) + 1) * r["ndr"] * r["dr"] + 1e-20)
        p = torch.stack(line[i]).cpu().numpy()
        q = torch.stack(grid[i], 1).cpu().numpy() if grids else None
        loss = [None if v is None else x - 20 * np.log10(np.abs(v) + 1e-20) for v in (p, q)]
        tl.append(loss)
        cp.append([p, q])
    return tl, cp


def _march_seconds(rays):
    """Rough time of _march on a GPU, for the caller to decide."""
    steps = max(r["nr"] for r in rays) + 4
    size = len(rays) * max(r["nz"] for r in rays) * max(r["np"] for r in rays)
    levels = math.ceil(math.log2(max(r["nz"] for r in rays)))
    slopes = 3.0 if any(r["sloping"] for r in rays) else 1.0
    return steps * (levels * (1e-4 + size * 16 * 14 / 4e12)) * slopes + steps * len(rays) * 3e-5


def _step64(W_, b_, X, Y, lr):
    """Loss, gradients and updated weights of one Adam step in float64."""
    Wd = [w.double().requires_grad_(True) for w in W_]
    bd = [v.double().requires_grad_(True) for v in b_]
    h = X.double()
    for i, (w, v) in enumerate(zip(Wd, bd)):
        h = h @ w.T + v
        h = torch.relu(h) if i < len(Wd) - 1 else h
    sse = ((h - Y.double()) ** 2).sum()
    (sse / Y.numel()).backward()
    gW, gb = [w.grad for w in Wd], [v.grad for v in bd]
    with torch.no_grad():  # the first step: m / (1 - beta1) = g, sqrt(v / (1 - beta2)) = |g|
        new = [w - lr * w.grad / (w.grad.abs() + 1e-8) for w in Wd]
    # the biases start at zero: their first step is the gradient's sign, which says nothing about rounding
    return [sse.detach().reshape(1), gW, gb, new, [None] * len(bd)]


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("single", "shared", "munk", "wedge"):
        rays, envs = _rays(c, seed)
        for r in rays:
            b = envs[r["env"]]["rbzb"]
            r["sloping"] = bool(np.any(b[:, 1] != b[0, 1]))
        if not torch.cuda.is_available() or _march_seconds(rays) > 15.0:
            return None
        tl, cp = _march(rays, envs, kind not in ("munk", "wedge"))
        if kind in ("munk", "wedge"):
            return [np.concatenate([t[0] for t in tl]), np.concatenate([p[0] for p in cp])]
        lines = [[t[0] for t in tl], [p[0] for p in cp], [t[1] for t in tl], [p[1] for p in cp]]
        if kind == "single":
            return [v[0] for v in lines]
        shape = (c["envs"], c["freqs"]) if c["envs"] > 1 else (c["freqs"],)
        return [np.stack(v).reshape(shape + v[0].shape) for v in lines]
    s = prepare(c, seed)
    if kind == "train":
        m = s["m"]
        return _step64(m.W, m.b, s["X"].index_select(0, s["idx"]), s["Y"].index_select(0, s["idx"]), 1e-3)
    if kind == "predict":
        tl = []
        for m in s["ens"].models:
            h = s["X"].double()
            for i, (w, v) in enumerate(zip(m.W, m.b)):
                h = h @ w.double().T + v.double()
                h = torch.relu(h) if i < len(m.W) - 1 else h
            tl.append((h * S.TL_SCALE + S.TL_MID).clamp_(S.TL_LO, S.TL_HI))
        mean = sum(tl) / len(tl)
        std = torch.sqrt(sum((t - mean) ** 2 for t in tl) / len(tl))
        return [v.view(-1, S.NZ_OUT, S.NR_OUT) for v in (mean, std)]
    x = s["A"].double() @ s["B"].double().T
    if s["bias"] is not None:
        x += s["bias"].double()
    if c["epi"] == "bias_relu":
        x = torch.relu(x)
    return x * (s["mask"] > 0) if s["mask"] is not None else x
