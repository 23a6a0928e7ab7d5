"""The framework's performance cases: what a program that simulates sea
surfaces calls, through the package's public entry points.

Kinds of case (one dict of plain values each):

generate  white noise + AR filter + variance renormalisation of one surface or
          of a batch (``Context.batch_generate``), in the reference's own FP64
          summation order or in compensated FP32, optionally with the
          nonlinear transform applied on the way (``batch_generate_nit``) or
          into page-locked host buffers
velocity  velocity potentials of every slice of a surface
          (``Context.velocity_linear``; linear or high-amplitude solver)
nit       the reference's per-point bisection of the nonlinear transform
          (``Context.nit_apply``)
ma        white noise + moving-average filter + renormalisation
          (``Context.ma_generate``)
autocov   circular auto-covariance of a realisation
          (``Context.auto_covariance``)
serve     chunks of several surface streams through the continuous-batching
          server, delivered into page-locked host memory (``Server``)

Sizes come from the configurations of ``bench.py`` and of the tests: the plain
standing wave 200 x 40 x 40 of order 7^3, the propagating wave 400 x 128 x 128
of order 10^3, its 512 x 256 x 256 form with the nonlinear transform, the
batch of 256 mixed surfaces, the serving chunks of 64 slices, the MA order
20 x 10 x 10.
"""
import functools
import math
import os

import numpy as np
import torch

import arma_b200 as A
from arma_b200 import capi

MT_FILE = os.path.join(os.path.dirname(os.path.abspath(A.__file__)), "data", "mt.dat")
MT_SETS = 16
SKEW_NORMAL = (0.0, 1.0, 1.499)  # mean, stdev, alpha: skewness 0.3
GRAM_CHARLIER = (0.1, 3.2)       # skewness, kurtosis


# ------------------------------------------------------------------ the cases
def _one(name, precision, shape, order, acf, b, **more):
    return {"name": name, "kind": "generate", "precision": precision, "surfaces": 1,
            "nt": shape[0], "nx": shape[1], "ny": shape[2],
            "pt": order[0], "px": order[1], "py": order[2], "acf": acf, "b": b,
            "nit": "none", "out": "device", **more}


def _batch(name, precision, surfaces, mix, **more):
    return {"name": name, "kind": "generate", "precision": precision, "surfaces": surfaces,
            "mix": mix, "nit": "none", "out": "device", **more}


def listed():
    return [
        # one small surface, as an interactive program asks for: latency and
        # the number of launches count
        _one("fp32-small", "fp32", (64, 32, 32), (4, 6, 4), "standing", 0.05),
        # the plain configuration: the reference's order of summation, as a
        # program run from a configuration file gets it by default
        _one("fp64-plain", "fp64", (200, 40, 40), (7, 7, 7), "standing", 0.05),
        # one long propagating wave in the reference's order of summation
        _one("fp64-propagating", "fp64", (400, 128, 128), (10, 10, 10), "propagating", 0.04),
        # some realisations of mixed size at once in FP64
        _batch("fp64-batch", "fp64", 16, 1),
        # the batch of independent realisations: 256 mixed surfaces
        _batch("fp32-batch", "fp32", 256, 0),
        # one large surface with the skew-normal transform in the same pass
        _one("fp32-nit-large", "fp32", (512, 256, 256), (10, 10, 10), "propagating", 0.04,
             nit="skew"),
        # velocity potentials of the propagating wave at four depths
        {"name": "velocity-fp32", "kind": "velocity", "precision": "fp32", "mode": "linear",
         "nt": 400, "nx": 128, "ny": 128, "nz": 4, "depth": 0.0},
        # FP64 potentials on a ragged grid over a finite depth (0: infinite)
        {"name": "velocity-fp64", "kind": "velocity", "precision": "fp64", "mode": "linear",
         "nt": 48, "nx": 200, "ny": 100, "nz": 3, "depth": 40.0},
        # the reference's nonlinear transform of the plain surface, point by point
        {"name": "nit-bisection", "kind": "nit", "precision": "fp64", "dist": "skew",
         "nt": 200, "nx": 40, "ny": 40, "eps": 1e-6},
        # a moving-average model of the reference's order
        {"name": "ma-fp64", "kind": "ma", "precision": "fp64", "nt": 256, "nx": 128, "ny": 128,
         "pt": 20, "px": 10, "py": 10},
        # the covariance of a realisation, against which a model is checked
        {"name": "autocov", "kind": "autocov", "precision": "fp64", "nt": 256, "nx": 128,
         "ny": 128},
        # two chunks of each of twelve new streams, with potentials at z = 0
        {"name": "serve", "kind": "serve", "streams": 12, "chunks": 2, "sides": "64,128,256",
         "slices": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(n):
    for p in range(2, 65):
        while n % p == 0:
            n //= p
    return n == 1


def _side(rng, lo, hi):
    while True:
        n = _log_int(rng, lo, hi)
        if _smooth(n):
            return n


def draw(rng):
    kind = rng.choice(["fp32", "fp32", "fp32", "fp64", "fp64", "fp64", "velocity", "velocity",
                       "velocity", "nit", "ma", "autocov", "serve"])
    if kind in ("fp32", "fp64"):
        out = "host" if kind == "fp32" and rng.random() < 0.25 else "device"
        if rng.random() < 0.35:
            count = _log_int(rng, 2, 128 if kind == "fp32" else 16)
            if out == "host":
                count = min(count, 24)
            return {"kind": "generate", "precision": kind, "surfaces": count,
                    "mix": rng.randrange(2, 10 ** 6), "nit": "none", "out": out}
        return {"kind": "generate", "precision": kind, "surfaces": 1,
                "nt": _log_int(rng, 24, 512), "nx": _log_int(rng, 16, 256),
                "ny": _log_int(rng, 16, 256), "pt": rng.randint(3, 10),
                "px": rng.randint(3, 10), "py": rng.randint(3, 10),
                "acf": rng.choice(["standing", "propagating"]),
                "b": round(rng.uniform(0.03, 0.1), 4),
                "nit": rng.choice(["none", "none", "skew", "gram"]) if out == "device" else "none",
                "out": out}
    if kind == "velocity":
        nx, ny, nz = _side(rng, 16, 256), _side(rng, 16, 256), rng.randint(1, 4)
        most = 26_000_000 // (nx * ny * nz)
        return {"kind": "velocity", "precision": rng.choice(["fp32", "fp64"]),
                "mode": rng.choice(["linear", "linear", "high"]),
                "nt": min(most, _log_int(rng, 8, 400)), "nx": nx, "ny": ny, "nz": nz,
                "depth": rng.choice([0.0, 0.0, 25.0, 80.0])}
    if kind == "nit":
        return {"kind": "nit", "precision": rng.choice(["fp64", "fp32"]),
                "dist": rng.choice(["skew", "gram"]), "nt": _log_int(rng, 24, 256),
                "nx": _log_int(rng, 16, 96), "ny": _log_int(rng, 16, 96),
                "eps": rng.choice([1e-4, 1e-6, 1e-8])}
    if kind == "ma":
        return {"kind": "ma", "precision": rng.choice(["fp64", "fp32"]),
                "nt": _log_int(rng, 24, 256), "nx": _log_int(rng, 16, 128),
                "ny": _log_int(rng, 16, 128), "pt": rng.randint(2, 32),
                "px": rng.randint(1, 10), "py": rng.randint(1, 10)}
    if kind == "autocov":
        return {"kind": "autocov", "precision": rng.choice(["fp64", "fp32"]),
                "nt": _log_int(rng, 16, 400), "nx": _log_int(rng, 16, 160),
                "ny": _log_int(rng, 16, 160)}
    return {"kind": "serve", "streams": rng.randint(1, 12), "chunks": rng.randint(1, 2),
            "sides": rng.choice(["64", "128", "64,128,256", "100,72"]), "slices": 64}


# ------------------------------------------------------------------ the inputs
def _gamma(acf, b, i, j, k):
    """The analytic auto-covariance at signed lags (arrays)."""
    e = np.exp(-b * (np.abs(i) + np.abs(j) + np.abs(k)))
    if acf == "propagating":
        return e * np.cos(0.6 * i + 0.3 * j + 0.2 * k)
    return 1.5 * e * np.cos(0.8 * i) * np.cos(0.5 * j) * np.cos(0.5 * k)


@functools.lru_cache(maxsize=None)
def _model(acf, b, order):
    """AR coefficients, white-noise variance and variance of the surface."""
    P = int(np.prod(order))
    i, j, k = (v.ravel().astype(np.float64) for v in np.indices(order))
    full = _gamma(acf, b, i[:, None] - i, j[:, None] - j, k[:, None] - k)
    phi = np.zeros(P)
    phi[1:] = np.linalg.solve(full[1:, 1:], full[1:, 0])
    phi.setflags(write=False)
    return phi.reshape(order), float(full[0, 0] - phi @ full[0]), float(full[0, 0])


def _members(case):
    """(shape, order, acf, b) of every surface of a generate case."""
    if "mix" not in case:
        return [((case["nt"], case["nx"], case["ny"]), (case["pt"], case["px"], case["py"]),
                 case["acf"], case["b"])]
    rng = np.random.default_rng(42 + case["mix"])
    got = []
    for _ in range(case["surfaces"]):
        nt = int(rng.integers(64, 513))
        nx, ny = (int((32, 64, 128, 256)[rng.integers(0, 4)]) for _ in range(2))
        order = tuple(int((4, 6, 8, 10)[rng.integers(0, 4)]) for _ in range(3))
        acf = "propagating" if rng.random() < 0.5 else "standing"
        got.append(((nt, nx, ny), order, acf, float(rng.choice([0.03, 0.05, 0.07, 0.1]))))
    return got


def _seed(seed, k):
    return (seed * 1009 + 42 + k) & 0xffffffff


def _waves(shape, seed):
    """A rough random sea (FP64, on the GPU): white noise filtered by the
    square root of the spectrum of a decaying standing wave's covariance."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1000 + seed)
    z = torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)
    acf = torch.ones((), dtype=torch.float64, device="cuda")
    for axis, (n, w) in enumerate(zip(shape, (0.8, 0.5, 0.5))):
        lag = torch.arange(n, dtype=torch.float64, device="cuda")
        lag = torch.minimum(lag, n - lag)
        c = torch.exp(-0.05 * lag) * torch.cos(w * lag)
        acf = acf * c.reshape([n if a == axis else 1 for a in range(3)])
    root = torch.fft.rfftn(acf).real.clamp_min(0.0).sqrt()
    return torch.fft.irfftn(torch.fft.rfftn(z) * root, s=shape).contiguous()


def _levels(case):
    return [0.0, -1.0, -2.0, -4.0][:case["nz"]]


def _theta(case, seed):
    order = (case["pt"], case["px"], case["py"])
    rng = np.random.default_rng(77 + seed)
    return rng.normal(0.0, 0.2 / math.sqrt(np.prod(order)), order)


def _context():
    ctx = A.Context(0)
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    return ctx


def _kind(case):
    fp64 = case["precision"] == "fp64"
    return (A.FP64, torch.float64) if fp64 else (A.FP32C, torch.float32)


def _prepare_generate(case, seed):
    prec, dtype = _kind(case)
    sets = [A.mt_file_read(MT_FILE, k) for k in range(MT_SETS)]
    members = _members(case)
    # every surface starts on a 256-byte boundary of one buffer
    starts, total = [], 0
    for shape, _, _, _ in members:
        starts.append(total)
        total += -(-int(np.prod(shape)) // 64) * 64
    if case["out"] == "host":
        flat = torch.zeros(total, dtype=dtype, pin_memory=True)
    else:
        flat = torch.zeros(total, dtype=dtype, device="cuda")
    surfs, tables = [], []
    for k, ((shape, order, acf, b), at) in enumerate(zip(members, starts)):
        phi, var, acf0 = _model(acf, b, order)
        surfs.append(capi.make_surface(shape, phi, var, acf0, sets[k % MT_SETS], _seed(seed, k),
                                       flat[at:].data_ptr()))
        if case["nit"] == "skew":
            tables.append(A.nit_table(A.NIT_SKEW_NORMAL, SKEW_NORMAL, math.sqrt(acf0)))
        elif case["nit"] == "gram":
            tables.append(A.nit_table(A.NIT_GRAM_CHARLIER, GRAM_CHARLIER, math.sqrt(acf0)))
    return {"ctx": _context(), "prec": prec, "flat": flat, "surfs": surfs, "tables": tables}


def _stream_seed(seed, k):
    return _seed(seed, 500 + k)


def _streams(case):
    sides = [int(s) for s in case["sides"].split(",")]
    return [(sides[k % len(sides)], ("standing", "propagating")[k % 2])
            for k in range(case["streams"])]


def _prepare_serve(case, seed):
    T = case["slices"]
    sets = [A.mt_file_read(MT_FILE, k) for k in range(MT_SETS)]
    server = A.Server(chunk_slices=T, velocity=1, z_levels=[0.0], max_inflight=3,
                      hbm_budget=8 << 30)
    specs, bufs = [], []
    for k, (side, acf) in enumerate(_streams(case)):
        phi, var, acf0 = _model(acf, 0.05, (8, 8, 8))
        specs.append((side, side, phi, var, acf0, sets[k % MT_SETS], _stream_seed(seed, k)))
        bufs.append([tuple(torch.zeros(s, dtype=torch.float32, pin_memory=True)
                           for s in ((T, side, side), (T, 1, side, side)))
                     for _ in range(case["chunks"])])
    return {"server": server, "specs": specs, "bufs": bufs}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "generate":
        return {"case": case, **_prepare_generate(case, seed)}
    if kind == "serve":
        return {"case": case, **_prepare_serve(case, seed)}
    prec, dtype = _kind(case)
    shape = (case["nt"], case["nx"], case["ny"])
    s = {"case": case, "ctx": _context(), "prec": prec, "shape": shape}
    if kind == "velocity":
        s["zeta"] = _waves(shape, seed).to(dtype)
        s["out"] = torch.zeros((shape[0], case["nz"]) + shape[1:], dtype=dtype, device="cuda")
        s["slices"] = list(range(shape[0]))
    elif kind == "nit":
        s["zeta"] = _waves(shape, seed).to(dtype)
        s["out"] = torch.empty_like(s["zeta"])
    elif kind == "autocov":
        s["zeta"] = _waves(shape, seed).to(dtype)
        s["out"] = torch.zeros(shape, dtype=torch.float64, device="cuda")
    elif kind == "ma":
        s["out"] = torch.zeros(shape, dtype=dtype, device="cuda")
        s["surf"] = capi.make_surface(shape, _theta(case, seed), 0.8, 1.2,
                                      A.mt_file_read(MT_FILE, 3), _seed(seed, 0),
                                      s["out"].data_ptr())
    return s


# ------------------------------------------------------------------ one pass
def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "generate":
        ctx = state["ctx"]
        if state["tables"]:
            scales = ctx.batch_generate_nit(state["surfs"], state["prec"], state["tables"])
        else:
            scales = ctx.batch_generate(state["surfs"], state["prec"],
                                        host=case["out"] == "host")
        return [state["flat"], np.array(scales)]
    if kind == "velocity":
        depth = case["depth"] or math.inf
        state["ctx"].velocity_linear(state["zeta"].data_ptr(), state["shape"], state["prec"],
                                     (1.0, 1.0, 1.0), depth, _levels(case), state["slices"],
                                     state["out"].data_ptr(), case["mode"] == "high")
        return state["out"]
    if kind == "nit":
        out = state["out"].copy_(state["zeta"])  # the transform works in place
        skew = case["dist"] == "skew"
        state["ctx"].nit_apply(A.NIT_SKEW_NORMAL if skew else A.NIT_GRAM_CHARLIER,
                               SKEW_NORMAL if skew else GRAM_CHARLIER, 1.0, A.NIT_BISECTION,
                               out.numel(), state["prec"], out.data_ptr(),
                               interval=(-10.0, 10.0), eps=case["eps"], max_iter=100)
        return out
    if kind == "autocov":
        state["ctx"].auto_covariance(state["zeta"].data_ptr(), state["shape"], state["prec"],
                                     state["out"].data_ptr())
        return state["out"]
    if kind == "ma":
        scales = state["ctx"].ma_generate([state["surf"]], state["prec"])
        return [state["out"], np.array(scales)]
    server = state["server"]
    ids = [server.open_stream(*spec) for spec in state["specs"]]
    for c in range(case["chunks"]):
        for sid, bufs in zip(ids, state["bufs"]):
            zeta, velocity = bufs[c]
            server.submit(sid, zeta.data_ptr(), velocity.data_ptr())
    done = server.wait(len(ids) * case["chunks"])
    if any(d["status"] for d in done):
        raise RuntimeError(server.last_failure())
    for sid in ids:
        server.close_stream(sid)
    return state["bufs"]


# ------------------------------------------------------------------ its work
def _fft_flops(n):
    return 5.0 * n * math.log2(n)


def work(case):
    kind = case["kind"]
    if kind == "generate":
        es = 8 if case["precision"] == "fp64" else 4
        pts = [(int(np.prod(m[0])), int(np.prod(m[1]))) for m in _members(case)]
        return {"bytes": float(sum(n * es for n, _ in pts)),
                "flops": float(sum(n * 2 * (P - 1) for n, P in pts))}
    if kind == "serve":
        n = sum(case["slices"] * case["chunks"] * side * side for side, _ in _streams(case))
        f = sum(case["slices"] * case["chunks"] * 2 * _fft_flops(side * side)
                for side, _ in _streams(case))
        return {"bytes": 8.0 * n, "flops": 2.0 * 511 * n + f}
    es = 8 if case["precision"] == "fp64" else 4
    n = case["nt"] * case["nx"] * case["ny"]
    if kind == "velocity":
        n2, nz = case["nx"] * case["ny"], case["nz"]
        return {"bytes": float(n * es * (1 + nz)),
                "flops": case["nt"] * (_fft_flops(n2) * (1 + nz) + 6.0 * n2 * nz)}
    if kind == "nit":
        return {"bytes": 2.0 * n * es, "flops": 50.0 * n}
    if kind == "ma":
        return {"bytes": float(n * es),
                "flops": 2.0 * n * case["pt"] * case["px"] * case["py"]}
    return {"bytes": float(n * (es + 8)), "flops": 2 * _fft_flops(n)}


# ------------------------------------------------------------------ in 64 bits
@functools.lru_cache(maxsize=None)
def _mt_fields(index):
    raw, at = open(MT_FILE, "rb").read(), 0
    for k in range(index + 1):
        f = np.frombuffer(raw, np.uint32, 15, at)
        at += 72 + 4 * int(f[2])
    return [int(v) for v in f]


def _noise(index, seed, n, stddev):
    """n normal values of one dcmt stream by Marsaglia's polar method."""
    (a, mm, nn, _, _, _, upper, lower, s0, s1, sb, sc, mb, mc, _) = _mt_fields(index)
    count = 4 * int(n / 2 * 4 / math.pi + 12 * math.sqrt(n) + 400)
    x = np.zeros(nn + count + nn, np.uint32)
    v = seed & 0xffffffff
    for k in range(nn):
        x[k] = v
        v = (1812433253 * (v ^ (v >> 30)) + k + 1) & 0xffffffff
    step = nn - mm
    u32 = np.uint32
    for j in range(nn, nn + count, step):
        y = (x[j - nn:j - mm] & u32(upper)) | (x[j - nn + 1:j - mm + 1] & u32(lower))
        x[j:j + step] = x[j - nn + mm:j] ^ (y >> u32(1)) ^ ((y & u32(1)) * u32(a))
    w = x[nn:nn + count]
    w = w ^ (w >> u32(s0))
    w = w ^ ((w << u32(sb)) & u32(mb))
    w = w ^ ((w << u32(sc)) & u32(mc))
    w = (w ^ (w >> u32(s1))).astype(np.float64).reshape(-1, 4)
    u = 2.0 * ((w[:, 0::2] + w[:, 1::2] * 2.0 ** 32) * 2.0 ** -64) - 1.0
    r2 = u[:, 0] ** 2 + u[:, 1] ** 2
    u = u[(r2 <= 1.0) & (r2 > 0.0)][:(n + 1) // 2]
    r2 = u[:, 0] ** 2 + u[:, 1] ** 2
    u = u * np.sqrt(-2.0 * np.log(r2) / r2)[:, None]
    return u[:, ::-1].ravel()[:n] * stddev


def _ar(eps, phi):
    """The causal AR filter: per slice, the earlier slices' terms and the
    quarter-plane recursion, both as products of padded transforms."""
    nt, nx, ny = eps.shape
    pt, px, py = phi.shape
    # impulse response of 1 / (1 - A0) on the slice, row by row
    taps = np.zeros((px, ny))
    taps[:, :min(py, ny)] = phi[0][:, :ny]
    lag = np.arange(ny)[:, None] - np.arange(ny)
    toeplitz = [np.where(lag >= 0, t[np.abs(lag)], 0.0) for t in taps]
    inverse = np.linalg.inv(np.eye(ny) - toeplitz[0])
    h = np.zeros((nx, ny))
    h[0] = inverse[:, 0]
    for x in range(1, nx):
        h[x] = inverse @ sum(toeplitz[i] @ h[x - i] for i in range(1, min(px, x + 1)))
    size, fft = (2 * nx, 2 * ny), torch.fft
    device = "cuda" if torch.cuda.is_available() else "cpu"
    H = fft.rfft2(torch.from_numpy(h).to(device), size)
    F = [fft.rfft2(torch.from_numpy(p[:nx, :ny].copy()).to(device), size) for p in phi]
    eps, hist = torch.from_numpy(eps).to(device), []
    zeta = torch.empty_like(eps)
    for t in range(nt):
        S = eps[t]
        if hist:
            past = sum(F[k + 1] * z for k, z in enumerate(hist))
            S = S + fft.irfft2(past, size)[:nx, :ny]
        zeta[t] = fft.irfft2(H * fft.rfft2(S, size), size)[:nx, :ny]
        hist = [fft.rfft2(zeta[t], size)] + hist[:pt - 2] if pt > 1 else []
    return zeta.cpu().numpy()


def _scale(zeta, acf0):
    nt, nx, ny = zeta.shape
    at = ((nt // 2) * nx + nx // 2) * ny + ny // 2
    n = (nt - nt // 2) * (nx - nx // 2) * (ny - ny // 2)
    return math.sqrt(acf0 / zeta.ravel()[at:at + n].var(ddof=1))


def _exact_generate(case, seed):
    members = _members(case)
    if case["nit"] != "none" or sum(np.prod(m[0]) for m in members) > 8_000_000:
        return None
    flat, scales = [], []
    for k, (shape, order, acf, b) in enumerate(members):
        phi, var, acf0 = _model(acf, b, order)
        n = int(np.prod(shape))
        zeta = _ar(_noise(k % MT_SETS, _seed(seed, k), n, math.sqrt(var)).reshape(shape), phi)
        scales.append(_scale(zeta, acf0))
        flat += [zeta.ravel() * scales[-1], np.zeros(-n % 64)]
    return [np.concatenate(flat), np.array(scales)]


def _exact_serve(case, seed):
    T = case["slices"]
    out = []
    for k, (side, acf) in enumerate(_streams(case)):
        phi, var, acf0 = _model(acf, 0.05, (8, 8, 8))
        shape = (T * case["chunks"], side, side)
        zeta = _ar(_noise(k % MT_SETS, _stream_seed(seed, k), int(np.prod(shape)),
                          math.sqrt(var)).reshape(shape), phi)
        zeta *= _scale(zeta[:T], acf0)
        out.append([(zeta[c * T:(c + 1) * T], None) for c in range(case["chunks"])])
    return out


def _exact_ma(case, seed):
    shape = (case["nt"], case["nx"], case["ny"])
    n = int(np.prod(shape))
    eps = _noise(3, _seed(seed, 0), n, math.sqrt(0.8)).reshape(shape)
    kernel = -_theta(case, seed)
    kernel[0, 0, 0] = 1.0
    size = [a + b for a, b in zip(shape, kernel.shape)]
    zeta = np.fft.irfftn(np.fft.rfftn(eps, size) * np.fft.rfftn(kernel, size), size)
    zeta = np.ascontiguousarray(zeta[:shape[0], :shape[1], :shape[2]])
    s = _scale(zeta, 1.2)
    return [zeta * s, np.array([s])]


def _target_cdf(dist, x):
    if dist == "skew":
        mean, sd, alpha = SKEW_NORMAL
        h = (x - mean) / sd
        # Owen's T by the 20-point Gauss-Legendre rule (even integrand)
        nodes, weights = np.polynomial.legendre.leggauss(20)
        t = torch.zeros_like(x)
        for v, w in zip(nodes[10:], weights[10:]):
            term = 1.0 + (alpha * v) ** 2
            t += w * torch.exp(-0.5 * h * h * term) / term
        return 0.5 * torch.special.erfc(-h / math.sqrt(2.0)) - t * alpha / math.pi
    s, k = GRAM_CHARLIER
    return (torch.exp(-0.5 * x * x) *
            (k * (3.0 * x - x ** 3) + s * (4.0 - 4.0 * x * x) + 3.0 * x ** 3 - 9.0 * x) /
            (24.0 * 2.506628274631) + 0.5 * torch.special.erf(x / 1.4142135623731) + 0.5)


def _exact_nit(case, seed):
    shape = (case["nt"], case["nx"], case["ny"])
    z = _waves(shape, seed).to(_kind(case)[1]).double().ravel()
    goal = 0.5 * torch.special.erfc(-z / math.sqrt(2.0))
    a, b = torch.full_like(z, -10.0), torch.full_like(z, 10.0)
    root, live = torch.zeros_like(z), torch.ones_like(z, dtype=torch.bool)
    for _ in range(100):
        c = 0.5 * (a + b)
        fc = _target_cdf(case["dist"], c) - goal
        root = torch.where(live, c, root)
        na = (_target_cdf(case["dist"], a) - goal) * fc < 0.0
        nb = torch.where(na, c, b)
        move = (_target_cdf(case["dist"], nb) - goal) * fc < 0.0
        a, b = torch.where(live & move, c, a), torch.where(live, nb, b)
        live = live & (b - a > case["eps"]) & (fc.abs() > case["eps"])
        if not bool(live.any()):
            break
    return root.reshape(shape).cpu().numpy()


def _exact_autocov(case, seed):
    shape = (case["nt"], case["nx"], case["ny"])
    w = _waves(shape, seed).to(_kind(case)[1]).double().cpu().numpy()
    f = np.fft.rfftn(w)
    return np.fft.irfftn(f.real ** 2 + f.imag ** 2, shape) / w.size


def _min_wave_number(z, t):
    """Smallest wave number of the same-sign runs of extrema of z, walked down
    its columns, one after another."""
    zc = z.T
    z0 = zc[:, 1:-1]
    d1, d2 = z0 - zc[:, :-2], z0 - zc[:, 2:]
    at = (d1 > 0.0) == (d2 > 0.0)
    z0, d1, d2 = z0[at], d1[at], d2[at]
    a = -0.5 * (d1 + d2)
    b = d1 - a * (2.0 * t - 1.0)
    c = z0 - t * (a * t + b)
    period = -0.5 * b / a
    e = c + period * (b + a * period)
    if not e.size:
        return np.finfo(np.float64).max
    first = np.flatnonzero(np.r_[True, (e[1:] > 0.0) != (e[:-1] > 0.0)])
    top = np.maximum.reduceat(np.abs(e), first)
    run = np.repeat(np.arange(first.size), np.diff(np.r_[first, e.size]))
    hits = np.flatnonzero(np.abs(e) == top[run])
    lead = hits[np.unique(run[hits], return_index=True)[1]]
    gaps = np.abs(np.diff(period[lead]))[:-1]  # the last run never closes
    if not gaps.size:
        return np.finfo(np.float64).max
    return float((2.0 * math.pi / (2.0 * gaps.max())) ** 2 / 9.82)


def _plane(f1, f2, f3, p1, p2, p3, p):
    (a1, b1), (a2, b2), (a3, b3), (pa, pb) = p1, p2, p3, p
    den = a2 * b1 - a3 * b1 - a1 * b2 + a3 * b2 + a1 * b3 - a2 * b3
    c0 = (f2 * b1 - f3 * b1 - f1 * b2 + f3 * b2 + f1 * b3 - f2 * b3) / den
    c1 = (f3 * (a2 - a1) + f2 * (a1 - a3) + f1 * (a3 - a2)) / \
        (a3 * (b1 - b2) + a1 * (b2 - b3) + a2 * (b3 - b1))
    c2 = (f3 * a2 * b1 - f2 * a3 * b1 - f3 * a1 * b2 + f1 * a3 * b2 + f2 * a1 * b3 -
          f1 * a2 * b3) / den
    return c0 * pa + c1 * pb + c2


def _window(nx, ny, wx, wy, z, depth):
    u = (wx / (nx - 1) * np.arange(nx))[:, None]
    v = wy / (ny - 1) * np.arange(ny)
    l = 2.0 * math.pi * np.sqrt(u * u + v * v)
    ez, eh = np.exp(-l * z), np.exp(-2.0 * l * depth)
    r = 4.0 * math.pi * (1.0 + ez * ez * eh) / (ez * (1.0 + eh))
    r[0, 0] = r[1, 1] if np.isfinite(r[1, 1]) else np.nan
    for i in range(1, nx):
        if not np.isfinite(r[i, 0]):
            r[i, 0] = _plane(r[i - 1, 1], r[i, 1], r[i - 1, 2], (i - 1, 1), (i, 1), (i - 1, 2),
                             (i, 0))
    for j in range(1, ny):
        if not np.isfinite(r[0, j]):
            r[0, j] = _plane(r[1, j - 1], r[1, j], r[2, j - 1], (1, j - 1), (1, j), (2, j - 1),
                             (0, j))
    r[~np.isfinite(r)] = 0.0
    for axis, n in enumerate((nx, ny)):  # rotation by swaps, element after element
        at = list(range(n))
        for k in range(n // 2):
            q = (k + n // 2) % n
            at[k], at[q] = at[q], at[k]
        r = np.take(r, at, axis)
    return r


def _slope(z, axis):
    z = np.moveaxis(z, axis, 0)
    d = np.empty_like(z)
    d[1:-1] = 0.5 * (z[2:] - z[:-2])
    d[0] = 0.5 * (-z[2] + 4.0 * z[1] - 3.0 * z[0])
    d[-1] = 0.5 * (3.0 * z[-1] - 4.0 * z[-2] + z[-3])
    return np.moveaxis(d, 0, axis)


def _exact_velocity(case, seed):
    nt, nx, ny = shape = (case["nt"], case["nx"], case["ny"])
    if nt * nx * ny > 8_000_000 or min(shape) < 3:
        return None
    z = _waves(shape, seed).to(_kind(case)[1]).double().cpu().numpy()
    zt = _slope(z, 0)
    out = np.empty((nt, case["nz"], nx, ny))
    depth = case["depth"] or math.inf
    flat = {}
    with np.errstate(all="ignore"):
        for t in range(nt):
            if case["mode"] == "high":
                zx, zy = _slope(z[t], 0), _slope(z[t], 1)
                s = np.sqrt(1.0 + zx * zx + zy * zy)
                f = np.fft.fft2(zt[t] / (-1.0 / s + 1j * ((zx + zy) / s - zx - zy)))
            else:
                f = np.fft.fft2(-zt[t])
            wx, wy = (1.0 / _min_wave_number(m, t) for m in (z[t], z[t].T))
            for j, level in enumerate(_levels(case)):
                r = np.fft.ifft2(f * _window(nx, ny, wx, wy, level, depth)).real
                r[0, 0] = _plane(r[1, 1], r[1, 2], r[2, 1], (1, 1), (1, 2), (2, 1), (0, 0))
                for k in range(1, nx):
                    r[k, 0] = _plane(r[k - 1, 1], r[k, 1], r[k - 1, 2], (k - 1, 1), (k, 1),
                                     (k - 1, 2), (k, 0))
                for k in range(1, ny):
                    r[0, k] = _plane(r[1, k - 1], r[1, k], r[2, k - 1], (1, k - 1), (1, k),
                                     (2, k - 1), (0, k))
                out[t, j] = r
    return out


def exact(case, seed):
    return {"generate": _exact_generate, "serve": _exact_serve, "ma": _exact_ma,
            "nit": _exact_nit, "autocov": _exact_autocov,
            "velocity": _exact_velocity}[case["kind"]](case, seed)
