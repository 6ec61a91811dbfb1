"""The workloads whose speed is watched, through the public entry points of hteno.

A pass is what a host program does with a solver that it keeps: hand over a state, advance it by a
number of SSP-RK3 steps, read the state back (or, for the classifier, train and predict).  Sizes and
options follow the tests, the benchmark and the configurations of this repository: 1D tubes of a few
hundred cells, 2D grids from 64^2 to 4096^2, batches of grids with sides 64..512, Hermite grids up to
2048^2, and a classifier trained on up to millions of recorded stencils.

The module also holds a plain torch restatement of the schemes in 64 bits (`exact`), written from the
formulas and sharing no code with the library.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "hermite-teno_gb300"))
import hteno  # noqa: E402

F64 = torch.float64
GAMMA = 1.4
RECON = {"teno5": 0, "teno5i": 1, "linear": 2, "weno5z": 4}


# ---- the cases ---------------------------------------------------------------------------------

def _fv1d(nx, steps, recon="teno5", flux="hllc", bc="zerograd", precision="fp64"):
    return dict(kind="fv1d", nx=nx, steps=steps, recon=recon, flux=flux, bc=bc, precision=precision)


def _fv2d(nx, ny, steps, precision, recon="teno5", flux="hllc", bc="zerograd", data="quadrants", routed=False):
    return dict(kind="fv2d", nx=nx, ny=ny, steps=steps, precision=precision, recon=recon, flux=flux, bc=bc,
                data=data, routed=routed)


def _hermite2d(nx, ny, steps, precision):
    return dict(kind="hermite2d", nx=nx, ny=ny, steps=steps, precision=precision)


def listed():
    return [
        # the 1D shock-tube configuration: 400 cells, host arrays in and out, all latency
        dict(_fv1d(400, 96), name="tube_400"),
        # the LMPE-routed Hermite scheme in 1D, periodic, as small and as serial
        dict(kind="hermite1d", nx=320, steps=12, precision="fp64", name="hermite1d_320"),
        # a small plain FP64 grid: a first look at a problem, a convergence study
        dict(_fv2d(64, 48, 24, "fp64"), name="fp64_64x48"),
        # the plain FP64 headline grid, part-developed flow
        dict(_fv2d(1024, 1024, 2, "fp64"), name="fp64_1024"),
        # plain FP64, smooth and periodic, ragged sides, the shipped teno5i + Rusanov choice
        dict(_fv2d(333, 257, 4, "fp64", recon="teno5i", flux="rusanov", bc="periodic", data="waves"),
             name="fp64_333x257_waves"),
        # small mixed-precision grid
        dict(_fv2d(96, 80, 24, "mixed"), name="mixed_96x80"),
        # ordinary mixed-precision grid
        dict(_fv2d(1024, 1024, 10, "mixed"), name="mixed_1024"),
        # the largest grid, mixed precision with the learned router
        dict(_fv2d(4096, 4096, 3, "mixed", routed=True), name="mixed_4096_routed"),
        # independent grids of uneven sides advanced together
        dict(kind="batch", count=64, lo=64, hi=512, steps=4, name="batch_64"),
        # the Hermite scheme in 2D, plain FP64, ragged sides
        dict(_hermite2d(300, 211, 2, "fp64"), name="hermite_fp64_300x211"),
        # the Hermite configuration: 2048^2, mixed precision
        dict(_hermite2d(2048, 2048, 2, "mixed"), name="hermite_mixed_2048"),
        # the classifier: two epochs of training on recorded rows, then their probabilities
        dict(kind="mlp", rows=1_000_000, batch=16384, epochs=2, name="classifier_1m"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fv1d", "hermite1d", "fv2d_fp64", "fv2d_fp64", "fv2d_mixed", "fv2d_mixed", "fv2d_mixed",
                       "batch", "hermite2d_fp64", "hermite2d_mixed", "hermite2d_mixed", "mlp"])
    recon = rng.choice(["teno5", "teno5", "teno5", "teno5i", "linear", "weno5z"])
    flux, bc = rng.choice(["hllc", "hllc", "rusanov"]), rng.choice(["zerograd", "zerograd", "periodic"])
    if kind == "fv1d":
        return _fv1d(_log(rng, 50, 5000), _log(rng, 8, 100), recon, flux, bc, rng.choice(["fp64", "fp64", "mixed"]))
    if kind == "hermite1d":
        return dict(kind=kind, nx=_log(rng, 40, 500), steps=_log(rng, 2, 12), precision=rng.choice(["fp64", "fp64", "mixed"]))
    if kind == "batch":
        return dict(kind=kind, count=_log(rng, 2, 64), lo=64, hi=rng.choice([128, 256, 512]), steps=_log(rng, 2, 6))
    if kind == "mlp":
        return dict(kind=kind, rows=_log(rng, 2000, 4_000_000), batch=rng.choice([4096, 8192, 16384]), epochs=1)
    if kind.startswith("hermite2d"):
        precision = kind.split("_")[1]
        hi = 320 if precision == "fp64" else 2048
        nx, ny = _log(rng, 40, hi), _log(rng, 40, hi)
        return _hermite2d(nx, ny, 1 if nx * ny > hi * hi / 4 else 2, precision)
    precision = kind.split("_")[1]
    hi = 1024 if precision == "fp64" else 4096
    nx, ny = _log(rng, 32, hi), _log(rng, 32, hi)
    most = 2_000_000 if precision == "fp64" else 30_000_000
    steps = max(1, min(rng.choice([2, 6, 20]), most // (nx * ny)))
    return _fv2d(nx, ny, steps, precision, recon, flux, bc, rng.choice(["quadrants", "quadrants", "waves"]),
                 routed=precision == "mixed" and recon in ("teno5", "teno5i") and rng.random() < 0.25)


# ---- inputs ------------------------------------------------------------------------------------

def _conservative(rho, u, v, p):
    return torch.stack([rho, rho * u, rho * v, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)])


def _centres(nx, ny):
    x = (torch.arange(nx, dtype=F64, device="cuda") + 0.5) / nx
    y = (torch.arange(ny, dtype=F64, device="cuda") + 0.5) / ny
    return x[None, :], y[:, None]


def _quadrants(nx, ny, seed):
    """A four-quadrant Riemann problem some way into its run: constant far states, bit for bit, and
    waves around the four interfaces that fade into the constants through the rounding level."""
    r = np.random.default_rng(seed)
    X, Y = _centres(nx, ny)
    bend = 0.02 * torch.sin(2 * math.pi * (Y + r.uniform()))
    sx = 0.5 + 0.5 * torch.tanh((X - 0.5 - bend) * nx / r.uniform(1.0, 3.0))
    sy = 0.5 + 0.5 * torch.tanh((Y - 0.5) * ny / r.uniform(1.0, 3.0))
    band = torch.exp(-((X - 0.5) / 0.03) ** 2) + torch.exp(-((Y - 0.5) / 0.03) ** 2)
    w = []
    for lo, hi in ((0.3, 1.5), (-0.75, 0.75), (-0.75, 0.75), (0.2, 1.5)):
        a, b, c, d = r.uniform(lo, hi, 4)
        s = a * (1 - sx) * (1 - sy) + b * sx * (1 - sy) + c * (1 - sx) * sy + d * sx * sy
        kx, ky = r.uniform(20, 60, 2)
        w.append(s + 0.04 * band * torch.sin(kx * X + ky * Y + r.uniform(0, 6.28)))
    return _conservative(*w)


def _waves(nx, ny, seed):
    """A smooth periodic flow without a discontinuity."""
    r = np.random.default_rng(seed)
    X, Y = _centres(nx, ny)
    ph = r.uniform(0, 2 * math.pi, 6)
    tp = 2 * math.pi
    rho = 1 + 0.2 * torch.sin(tp * X + ph[0]) * torch.sin(tp * Y + ph[1])
    u = 0.5 + 0.1 * torch.sin(tp * Y + ph[2]) + 0 * X
    v = -0.3 + 0.1 * torch.cos(tp * X + ph[3]) + 0 * Y
    p = 1 + 0.1 * torch.cos(tp * (X + Y) + ph[4])
    return _conservative(rho, u, v, p)


def _tube(nx, seed):
    """Sod-like data with other states and a short wave packet about the jump, [3][nx]."""
    r = np.random.default_rng(seed)
    x = (np.arange(nx) + 0.5) / nx
    left = x < 0.5
    pkt = 0.05 * np.exp(-((x - 0.5) / 0.05) ** 2) * np.sin(80 * x + r.uniform(0, 6.28))
    rho = np.where(left, r.uniform(0.8, 1.2), r.uniform(0.1, 0.2)) * (1 + pkt)
    u = np.where(left, r.uniform(-0.2, 0.2), r.uniform(-0.2, 0.2)) + pkt
    p = np.where(left, r.uniform(0.8, 1.2), r.uniform(0.08, 0.15)) * (1 - pkt)
    return np.ascontiguousarray(np.stack([rho, rho * u, p / (GAMMA - 1.0) + 0.5 * rho * u * u]))


def _blobs(nx, ny, seed):
    """32 Gaussian density blobs and a Mach-2 shock entering at x = 0: state and its face-difference
    moments, as the Hermite configuration starts."""
    r = np.random.default_rng(seed)
    blobs = [(r.uniform(0.2, 1.0), r.uniform(0.01, 0.05), r.uniform(), r.uniform()) for _ in range(32)]
    M, g = 2.0, GAMMA
    rho1 = (g + 1) * M * M / ((g - 1) * M * M + 2)
    p1 = (2 * g * M * M - (g - 1)) / (g + 1)
    u1 = M * math.sqrt(g) * (1 - 1 / rho1)

    def q(X, Y):
        rho = 1 + 0 * X + 0 * Y
        for a, s, cx, cy in blobs:
            rho = rho + a * torch.exp(-((X - cx) ** 2 + (Y - cy) ** 2) / s ** 2)
        post = (X < 0.02) & (Y > -1)
        return _conservative(torch.where(post, rho1, rho), torch.where(post, u1, 0.0 * rho), 0.0 * rho,
                             torch.where(post, p1, 1.0 + 0.0 * rho))

    X, Y = _centres(nx, ny)
    v = (q(X + 0.5 / nx, Y) - q(X - 0.5 / nx, Y)) * nx
    w = (q(X, Y + 0.5 / ny) - q(X, Y - 0.5 / ny)) * ny
    return q(X, Y).contiguous(), v.contiguous(), w.contiguous()


def _line(nx, seed):
    """Periodic 1D data on [-1, 1]: an entropy wave and a density block, state and moments [3][nx]."""
    r = np.random.default_rng(seed)
    a, b, ph = r.uniform(0.2, 0.5), r.uniform(0.2, 0.6), r.uniform(0, 6.28)

    def q(x):
        x = (x + 1) % 2 - 1
        rho = 1.5 + a * np.sin(math.pi * x + ph) + np.where(np.abs(x) < 0.4, b, 0.0)
        return np.stack([rho, rho, 1 / (GAMMA - 1.0) + 0.5 * rho])

    dx = 2.0 / nx
    x = -1 + (np.arange(nx) + 0.5) * dx
    return np.ascontiguousarray(q(x)), np.ascontiguousarray((q(x + dx / 2) - q(x - dx / 2)) / dx)


def _stencils(n, seed):
    """n normalised 6-cell stencils as the classifier sees them (smooth, kinked and jumping data), BF16
    values in float [n][6], and their three TENO cut-off bits [n]."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def rnd(*s):
        return torch.rand(*s, generator=g, device="cuda", dtype=F64)

    t = torch.arange(6, device="cuda", dtype=F64)[None, :] - 2.5
    u = torch.sin(rnd(n, 1) * 6.28 + t * rnd(n, 1) * 1.5) + (rnd(n, 1) - 0.5) * t * t * 0.2
    u = u + (rnd(n, 1) < 0.4) * (rnd(n, 1) - 0.5) * 4 * (t > torch.floor(rnd(n, 1) * 5) - 2.0)
    lo, hi = u.min(1, keepdim=True).values, u.max(1, keepdim=True).values
    x = ((u - u.mean(1, keepdim=True)) / (hi - lo + 1e-30)).clamp(-1, 1)
    keep = _teno_keep("teno5", [u[:, k] for k in range(5)])
    y = sum((k.to(torch.uint8) << i) for i, k in enumerate(keep))
    return x.to(torch.bfloat16), y


def _params(seed):
    """Start weights of the classifier, public parameter layout."""
    r = np.random.default_rng(seed)
    p = np.zeros(1379, dtype=np.float32)
    for a, n, fan in ((0, 192, 6), (224, 1024, 32), (1280, 96, 32)):
        p[a:a + n] = r.uniform(-1, 1, n) * math.sqrt(6 / fan)
    return p


def _split(p):
    return (p[:192].view(32, 6), p[192:224], p[224:1248].view(32, 32), p[1248:1280], p[1280:1376].view(3, 32), p[1376:])


def _logits(p, x):
    W1, b1, W2, b2, W3, b3 = _split(p)
    return torch.relu(torch.relu(x @ W1.T + b1) @ W2.T + b2) @ W3.T + b3


def _trained(seed):
    """Weights of a classifier trained (in torch) on synthetic stencils: what a program that routes has."""
    x, y = _stencils(32768, 7)
    x = x.double()
    bits = torch.stack([(y >> k) & 1 for k in range(3)], 1).double()
    p = torch.from_numpy(_params(seed)).cuda().double().requires_grad_()
    opt = torch.optim.Adam([p], lr=1e-2)
    for _ in range(120):
        opt.zero_grad()
        torch.nn.functional.binary_cross_entropy_with_logits(_logits(p, x), bits).backward()
        opt.step()
    return p.detach().float().cpu().numpy()


def _state2d(case, seed):
    return (_waves if case["data"] == "waves" else _quadrants)(case["nx"], case["ny"], seed).contiguous()


def _sides(case, seed):
    """Sides of the grids of a batch.  They come from the case alone, so that states made from
    different seeds are the same amount of work."""
    r = np.random.default_rng([case["count"], case["lo"], case["hi"]])
    return [tuple(int(s) for s in r.integers(case["lo"], case["hi"] + 1, 2)) for _ in range(case["count"])]


# ---- preparing and running ---------------------------------------------------------------------

def _config(case, **kw):
    return hteno.config(recon=RECON[case.get("recon", "teno5")],
                        flux=hteno.FLUX_HLLC if case.get("flux", "hllc") == "hllc" else hteno.FLUX_RUSANOV,
                        bc=hteno.BC_PERIODIC if case.get("bc") == "periodic" else hteno.BC_ZEROGRAD,
                        precision=hteno.PREC_MIXED if case.get("precision") == "mixed" else hteno.PREC_FP64, **kw)


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "steps": case.get("steps", 0)}
    if kind == "fv1d":
        st["q"] = _tube(case["nx"], seed)
        st["out"] = np.empty_like(st["q"])
        st["solver"] = hteno.Solver(_config(case, dims=1, nx=case["nx"], cfl=0.5))
    elif kind == "hermite1d":
        st["q"], st["v"] = _line(case["nx"], seed)
        st["solver"] = hteno.Solver(_config(case, dims=1, scheme=hteno.SCHEME_HERMITE, nx=case["nx"], xl=-1.0, xr=1.0, cfl=0.5))
    elif kind == "fv2d":
        st["q"] = _state2d(case, seed)
        st["out"] = torch.empty_like(st["q"])
        st["solver"] = hteno.Solver(_config(case, dims=2, nx=case["nx"], ny=case["ny"], cfl=0.4))
        if case["routed"]:
            st["mlp"] = hteno.Mlp(0)
            st["mlp"].set_params(_trained(seed))
            st["solver"].set_router(st["mlp"], 0.9)
            st["solver"].set_router_schedule(4, 2)
    elif kind == "hermite2d":
        st["q"], st["v"], st["w"] = _blobs(case["nx"], case["ny"], seed)
        st["out"] = [torch.empty_like(st["q"]) for _ in range(3)]
        st["solver"] = hteno.Solver(_config(case, dims=2, scheme=hteno.SCHEME_HERMITE, nx=case["nx"], ny=case["ny"], cfl=0.4))
    elif kind == "batch":
        sides = _sides(case, seed)
        st["q"] = [_quadrants(nx, ny, 1000 * seed + k).contiguous() for k, (nx, ny) in enumerate(sides)]
        st["out"] = torch.empty(sum(q.numel() for q in st["q"]), dtype=F64, device="cuda")
        st["batch"] = hteno.Batch([_config(dict(case, precision="mixed"), dims=2, nx=nx, ny=ny, cfl=0.4) for nx, ny in sides])
    else:
        x, y = _stencils(case["rows"], seed)
        rows = torch.zeros(case["rows"], 8, dtype=torch.bfloat16, device="cuda")
        rows[:, :6] = x
        st.update(x=rows.view(torch.int16).contiguous(), y=y.contiguous(), start=_params(seed), mlp=hteno.Mlp(0),
                  p=torch.empty(case["rows"], 3, device="cuda"), batch=case["batch"], epochs=case["epochs"])
    torch.cuda.synchronize()  # the solvers work on streams of their own
    if kind in ("fv1d", "fv2d"):
        st["solver"].set_state(st["q"])
    elif kind == "batch":
        for k, q in enumerate(st["q"]):
            st["batch"].set_state(k, q)
        st["batch"].tile()
    return st


def run(st):
    kind = st["kind"]
    if kind == "mlp":
        m = st["mlp"]
        m.set_params(st["start"])
        loss = m.train(st["x"], st["y"], st["epochs"], st["batch"], 1e-3)
        return {"loss": loss, "p": m.predict(st["x"], st["p"]), "weights": m.params()}
    if kind == "batch":
        b = st["batch"]
        for k, q in enumerate(st["q"]):
            b.set_state(k, q)
        b.step(st["steps"])
        at = 0
        for k, q in enumerate(st["q"]):
            b.get_state(k, st["out"][at:at + q.numel()])
            at += q.numel()
        return st["out"]
    s = st["solver"]
    s.set_state(st["q"])
    if kind == "hermite1d":
        s.set_moments(st["v"])
        s.step(st["steps"])
        return {"q": s.get_state(), "v": s.get_moments()}
    if kind == "hermite2d":
        q, v, w = st["out"]
        s.set_moments(st["v"], st["w"])
        s.step(st["steps"])
        s.get_state(q)
        rc = hteno.lib().hteno_get_moments(s.h, v.data_ptr(), w.data_ptr(), hteno.DEVICE)
        if rc:
            raise hteno.HtenoError(rc, "moments")
        return {"q": q, "v": v, "w": w}
    s.step(st["steps"])
    return s.get_state(st["out"])


def work(case):
    """Bytes: the inputs once and the outputs once.  Flops: the reference's operations per cell and stage
    (5520 in FV 2D: 2734 per face and direction, 52 in the update), or the network's products."""
    kind = case["kind"]
    if kind == "mlp":
        n = case["rows"]
        return {"bytes": n * (16 + 1 + 12), "flops": n * 2624.0 * (1 + 3 * case["epochs"])}
    if kind == "batch":
        cells = sum(nx * ny for nx, ny in _sides(case, 0))
    else:
        cells = case["nx"] * case.get("ny", 1)
    per_state, per_stage = {"fv1d": (48, 1000), "hermite1d": (96, 1300), "fv2d": (64, 5520), "batch": (64, 5520),
                            "hermite2d": (192, 16500)}[kind]
    return {"bytes": cells * per_state, "flops": float(cells) * per_stage * 3 * case["steps"]}


# ---- the same in 64 bits, plain torch ------------------------------------------------------------
# Arrays are [field, line, along the sweep]; a y sweep is an x sweep of the transposed grid with the
# two momenta exchanged.

SQ15 = math.sqrt(15.0)
DK = ((0.3, 0.6, 0.1), (0.1, 0.6, 0.3))


def _pad(a, n, bc):
    size = a.shape[-1]
    i = torch.arange(-n, size + n, device=a.device)
    return a[..., i % size if bc == "periodic" else i.clamp(0, size - 1)]


def _indicators(v):
    c = (v[2] - 2 * v[3] + v[4], v[1] - 2 * v[2] + v[3], v[0] - 2 * v[1] + v[2])
    b = (3 * v[2] - 4 * v[3] + v[4], v[1] - v[3], v[0] - 4 * v[1] + 3 * v[2])
    return [0.25 * b[k] * b[k] + 13 / 12 * c[k] * c[k] for k in range(3)]


def _keep(SI, tau, ct):
    r = [1 + tau / (s + 1e-40) for s in SI]
    m = torch.maximum(torch.maximum(r[0], r[1]), r[2])
    a = [(x / m) ** 2 for x in r]
    a = [x * x * x for x in a]
    lim = ct * (a[0] + a[1] + a[2])
    return [~(x < lim) for x in a]


def _teno_keep(recon, v):
    SI = _indicators(v)
    if recon == "teno5i":
        tau = torch.maximum(torch.maximum(SI[0], SI[1]), SI[2])
    else:
        b35 = (v[4] * (6908 * v[4] - 51001 * v[3] + 67923 * v[2] - 38947 * v[1] + 8209 * v[0])
               + v[3] * (104963 * v[3] - 299076 * v[2] + 179098 * v[1] - 38947 * v[0])
               + v[2] * (231153 * v[2] - 299076 * v[1] + 67923 * v[0])
               + v[1] * (104963 * v[1] - 51001 * v[0]) + 6908 * v[0] * v[0]) / 5040
        tau = (b35 - (SI[0] + SI[2] + 4 * SI[1]) / 6).abs()
    return _keep(SI, tau, 5e-4)


def _blend(p, w):
    return (p[0] * w[0] + p[1] * w[1] + p[2] * w[2]) / (w[0] + w[1] + w[2])


def _lagrange(recon, u):
    out = []
    for side in range(2):
        v = u[side:side + 5]
        if side == 0:
            p = [1 / 3 * v[2] + 5 / 6 * v[3] - 1 / 6 * v[4], -1 / 6 * v[1] + 5 / 6 * v[2] + 1 / 3 * v[3],
                 1 / 3 * v[0] - 7 / 6 * v[1] + 11 / 6 * v[2]]
        else:
            p = [11 / 6 * v[2] - 7 / 6 * v[3] + 1 / 3 * v[4], 1 / 3 * v[1] + 5 / 6 * v[2] - 1 / 6 * v[3],
                 -1 / 6 * v[0] + 5 / 6 * v[1] + 1 / 3 * v[2]]
        if recon == "linear":
            w = DK[side]
        elif recon == "weno5z":
            SI = _indicators(v)
            tau = (SI[2] - SI[0]).abs()
            w = [d * (1 + tau / (s + 1e-40)) for d, s in zip(DK[side], SI)]
        else:
            w = [d * k for d, k in zip(DK[side], _teno_keep(recon, v))]
        out.append(_blend(p, w))
    return out


_den_p, _den_m = 15720 * SQ15 + 10480, 15720 * SQ15 - 10480
LIN_P = [(2882 * SQ15 - 1179) / _den_p, (9672 * SQ15 + 6448) / _den_p, (3166 * SQ15 + 5211) / _den_p]
LIN_M = [(2882 * SQ15 + 1179) / _den_m, (9672 * SQ15 - 6448) / _den_m, (3166 * SQ15 - 5211) / _den_m]
_lin0 = (-9 / 80, 49 / 40, -9 / 80)
ZERO_P = [0.5 * (x + 3 * abs(x)) for x in _lin0]
ZERO_M = [p - x for p, x in zip(ZERO_P, _lin0)]


def _points(u):
    """Values at the three Gauss-Legendre points of the middle of five cells."""
    b = (u[0] - 4 * u[1] + 3 * u[2], u[1] - u[3], 3 * u[2] - 4 * u[3] + u[4])
    c = (u[0] - 2 * u[1] + u[2], u[1] - 2 * u[2] + u[3], u[2] - 2 * u[3] + u[4])
    al = [1 / (1e-6 + 0.25 * b[k] * b[k] + 13 / 12 * c[k] * c[k]) ** 2 for k in range(3)]
    a, h, e = SQ15 / 20, 1 / 30, 31 / 30
    gp = ((h + a, -1 / 15 - 4 * a, e + 3 * a), (h - a, 14 / 15, h + a), (e - 3 * a, -1 / 15 + 4 * a, h - a))
    gm = ((h - a, -1 / 15 + 4 * a, e - 3 * a), (h + a, 14 / 15, h - a), (e + 3 * a, -1 / 15 - 4 * a, h + a))

    def mix(p, lin):
        return _blend(p, [l * x for l, x in zip(lin, al)])

    def cand(g):
        return [sum(g[k][j] * u[k + j] for j in range(3)) for k in range(3)]

    mid = [(-u[0] + 2 * u[1] + 23 * u[2]) / 24, (-u[1] + 26 * u[2] - u[3]) / 24, (23 * u[2] + 2 * u[3] - u[4]) / 24]
    return [mix(cand(gp), LIN_P), sum(ZERO_P) * mix(mid, ZERO_P) - sum(ZERO_M) * mix(mid, ZERO_M), mix(cand(gm), LIN_M)]


def _prim(q):
    u, v = q[1] / q[0], q[2] / q[0]
    return u, v, (q[3] - 0.5 * (q[1] * u + q[2] * v)) * (GAMMA - 1)


class _Roe:
    def __init__(self, q):
        """Face states of the line-padded state q (one ghost cell each side)."""
        u, v, p = _prim(q)
        h, s = (q[3] + p) / q[0], q[0].abs().sqrt()
        l, r = (..., slice(None, -1)), (..., slice(1, None))
        t = s[l] / (s[l] + s[r])
        self.u, self.v, self.h = (t * x[l] + (1 - t) * x[r] for x in (u, v, h))
        self.k = 0.5 * (self.u ** 2 + self.v ** 2)
        self.c = ((GAMMA - 1) * (self.h - self.k)).abs().sqrt()
        self.b = (GAMMA - 1) / self.c ** 2

    def left(self, q):
        u, v, c, b = self.u, self.v, self.c, self.b
        k, m = b * self.k, u / c
        return torch.stack([0.5 * ((k + m) * q[0] - (b * u + 1 / c) * q[1] - b * v * q[2] + b * q[3]),
                            q[2] - v * q[0], (1 - k) * q[0] + b * u * q[1] + b * v * q[2] - b * q[3],
                            0.5 * ((k - m) * q[0] - (b * u - 1 / c) * q[1] - b * v * q[2] + b * q[3])])

    def right(self, w):
        u, v, c = self.u, self.v, self.c
        return torch.stack([w[0] + w[2] + w[3], (u - c) * w[0] + u * w[2] + (u + c) * w[3],
                            v * (w[0] + w[2] + w[3]) + w[1],
                            (self.h - u * c) * w[0] + v * w[1] + self.k * w[2] + (self.h + u * c) * w[3]])


def _flux(q, w):
    return torch.stack([q[1], q[1] * w[0] + w[2], q[1] * w[1], w[0] * (q[3] + w[2])])


def _hllc(a, b):
    wa, wb = _prim(a), _prim(b)
    ha, hb = (a[3] + wa[2]) / a[0], (b[3] + wb[2]) / b[0]
    r = (b[0] / a[0]).abs().sqrt()
    u, v, h = ((x + y * r) / (1 + r) for x, y in ((wa[0], wb[0]), (wa[1], wb[1]), (ha, hb)))
    c = ((GAMMA - 1) * (h - 0.5 * (u * u + v * v))).abs().sqrt()
    sl = torch.minimum(wa[0] - (wa[2] / a[0]).abs().sqrt(), u - c)
    sr = torch.maximum(wb[0] + (wb[2] / b[0]).abs().sqrt(), u + c)
    sm = (b[1] * (sr - wb[0]) - a[1] * (sl - wa[0]) + wa[2] - wb[2]) / (b[0] * (sr - wb[0]) - a[0] * (sl - wa[0]))
    ps = wa[2] + a[0] * (wa[0] - sl) * (wa[0] - sm)

    def star(q, w, s):
        n, d = s - w[0], s - sm
        qs = torch.stack([q[0] * n, n * q[1] + ps - w[2], n * q[2], n * q[3] - wa[2] * w[0] + ps * sm]) / d
        return _flux(q, w) + s * (qs - q)

    return torch.where(sl > 0, _flux(a, wa), torch.where(sm > 0, star(a, wa, sl), torch.where(sr >= 0, star(b, wb, sr), _flux(b, wb))))


def _speeds(a, b):
    (ua, _, pa), (ub, _, pb) = _prim(a), _prim(b)
    ca, cb = (GAMMA * pa / a[0]).abs().sqrt(), (GAMMA * pb / b[0]).abs().sqrt()
    m = torch.maximum(ua.abs(), ub.abs())
    return torch.stack([torch.maximum((ua - ca).abs(), (ub - cb).abs()), m, m, torch.maximum((ua + ca).abs(), (ub + cb).abs())])


def _rusanov(roe, a, b):
    return 0.5 * (_flux(a, _prim(a)) + _flux(b, _prim(b)) - roe.right(_speeds(a, b) * roe.left(b - a)))


def _jacobian(q, x):
    u, v, p = _prim(q)
    g, g1 = GAMMA, GAMMA - 1
    k, h = 0.5 * g1 * (u * u + v * v), (q[3] + p) / q[0]
    return torch.stack([x[1], (k - u * u) * x[0] + (3 - g) * u * x[1] - g1 * v * x[2] + g1 * x[3],
                        -u * v * x[0] + v * x[1] + u * x[2],
                        (k - h) * u * x[0] + (h - g1 * u * u) * x[1] - g1 * u * v * x[2] + g * u * x[3]])


def _drusanov(roe, a, b, da, db):
    return 0.5 * (_jacobian(a, da) + _jacobian(b, db) - roe.right(_speeds(a, b) * roe.left(db - da)))


def _faces(roe, q, n):
    """The n cells around every face in the face's characteristic basis; q padded by n/2 cells."""
    nf = q.shape[-1] - n + 1
    return [roe.left(q[..., m:m + nf]) for m in range(n)]


def _at_points(f, bc):
    """Face values [field, line, face] at the faces' three Gauss points."""
    p = _pad(f.transpose(-1, -2), 2, bc).transpose(-1, -2)
    n = f.shape[-2]
    return _points([p[..., m:m + n, :] for m in range(5)])


GAUSS = (5 / 18, 4 / 9, 5 / 18)


def _sweep(q, recon, flux, bc):
    roe = _Roe(_pad(q, 1, bc))
    minus, plus = _lagrange(recon, _faces(roe, _pad(q, 3, bc), 6))
    F = 0
    for wt, a, b in zip(GAUSS, _at_points(minus, bc), _at_points(plus, bc)):
        a, b = roe.right(a), roe.right(b)
        F = F + wt * (_hllc(a, b) if flux == "hllc" else _rusanov(roe, a, b))
    return F


def _swap(a):
    return a[[0, 2, 1, 3]].transpose(-1, -2)


def _drop(F):
    return F[..., :-1] - F[..., 1:]


def _rk(s, base, cur, rhs, dt):
    if s == 0:
        return base + dt * rhs
    if s == 1:
        return 0.75 * base + 0.25 * (cur + dt * rhs)
    return (base + 2 * (cur + dt * rhs)) / 3


def _speed2d(q):
    u, v, p = _prim(q)
    c = (GAMMA * p / q[0]).abs().sqrt()
    return max(float(x.max()) for x in (u - c, (u + c).abs(), v - c, (v + c).abs()))


def _fv2d_exact(q, steps, recon, flux, bc, cfl=0.4):
    ny, nx = q.shape[1:]
    dx, dy = 1.0 / nx, 1.0 / ny
    for _ in range(steps):
        dt, base = cfl * min(dx, dy) / _speed2d(q), q
        for s in range(3):
            rhs = _drop(_sweep(q, recon, flux, bc)) / dx + _swap(_drop(_sweep(_swap(q), recon, flux, bc))) / dy
            q = _rk(s, base, q, rhs, dt)
    return q


def _fv1d_exact(q, steps, recon, flux, bc):
    q = torch.stack([q[0], q[1], 0 * q[0], q[2]])[:, None, :]
    dx = 1.0 / q.shape[-1]
    for _ in range(steps):
        u, _, p = _prim(q)
        c = (GAMMA * p / q[0]).abs().sqrt()
        dt, base = 0.5 * dx / float(torch.maximum((u - c).abs(), (u + c).abs()).max()), q
        for s in range(3):
            roe = _Roe(_pad(q, 1, bc))
            a, b = (roe.right(x) for x in _lagrange(recon, _faces(roe, _pad(q, 3, bc), 6)))
            q = _rk(s, base, q, _drop(_hllc(a, b) if flux == "hllc" else _rusanov(roe, a, b)) / dx, dt)
    return q[[0, 1, 3], 0]


# Hermite reconstruction: value and derivative on the left of the face between u[1] and u[2], from
# three cells; the right side is the mirror image (moments change sign).
HD = (9 / 80, 42 / 80, 29 / 80)
HDD = (1 / 18, 5 / 6, 1 / 9)


def _brk(u, d):
    return ((1029270 * u[2] - 2129184 * u[1] + 1099914 * u[0] + 281121 * d[0] - 494958 * d[2]) * d[0]
            + (-1029270 * u[0] + 2129184 * u[1] - 1099914 * u[2] + 281121 * d[2]) * d[2]
            + (1099445 * u[2] - 4317056 * u[1] + 2118166 * u[0]) * u[2] + 4317056 * (u[1] - u[0]) * u[1]
            + 1099445 * u[0] * u[0]).abs() / 6720


def _brkd(u, d):
    return ((3156862 * d[2] + 13189240 * d[1] + 1710479 * d[0] - 9617754 * u[2] - 531552 * u[1] + 10149306 * u[0]) * d[0]
            + (13189240 * d[2] + 26511200 * d[1] - 39700440 * u[2] + 39700440 * u[0]) * d[1]
            + (1710479 * d[2] - 10149306 * u[2] + 531552 * u[1] + 9617754 * u[0]) * d[2]
            + (15136011 * u[2] - 1076544 * u[1] - 29195478 * u[0]) * u[2] + 1076544 * (u[1] - u[0]) * u[1]
            + 15136011 * u[0] * u[0]).abs() / 1680


def _hsi(u, d):
    b = (-2 * (u[0] - u[1]) - d[0], -2 * (u[1] - u[2]) - d[2], 0.5 * (u[2] - u[0]))
    c = (-2 * (u[0] - u[1] + d[0]), 2 * (u[1] - u[2]) + 2 * d[2], u[0] - 2 * u[1] + u[2])
    return [13 / 12 * y * y + x * x for x, y in zip(b, c)]


def _hsid(u, d):
    b = (6 * (u[0] - u[1]) + 2 * d[0] + 4 * d[1], 6 * (u[2] - u[1]) - 4 * d[1] - 2 * d[2], u[0] - 2 * u[1] + u[2])
    c = (12 * (u[0] - u[1]) + 6 * (d[0] + d[1]), 12 * (u[1] - u[2]) + 6 * (d[1] + d[2]), 3 * (u[2] - u[0]) - 6 * d[1])
    return [13 / 12 * y * y + x * x for x, y in zip(b, c)]


def _hermite_faces(u, d, h, linear=None):
    """(value, derivative) on both sides of each face from four cells' averages u and moments d; where
    `linear` is given (1D), linear weights where it is set and the max-indicator tau elsewhere."""
    def weigh(p, SI, tau, dk):
        return _blend(p, [a * k for a, k in zip(dk, _keep(SI, tau, 1e-3))])

    def taus(full, SI):
        if linear is not None:
            return torch.maximum(torch.maximum(SI[0], SI[1]), SI[2])
        return (full - 0.25 * (SI[0] + SI[1] + 2 * SI[2])).abs()

    # u^- and d^-
    U, D = u[:3], d[:3]
    S = [h * x for x in D]
    p = [-7 / 6 * U[0] + 13 / 6 * U[1] - 2 / 3 * S[0], U[1] / 6 + 5 / 6 * U[2] - S[2] / 3, -U[0] / 6 + 5 / 6 * U[1] + U[2] / 3]
    SI = _hsi(U, S)
    um = weigh(p, SI, taus(_brk(U, S), SI), HD)
    p = [4 * (U[0] - U[1]) / h + 1.5 * D[0] + 3.5 * D[1], 2 * (U[2] - U[1]) / h - 0.5 * (D[1] + D[2]),
         (0.25 * U[0] - U[1] + 0.75 * U[2]) / h + 0.5 * D[1]]
    SI = _hsid(U, S)
    dm = weigh(p, SI, taus(_brkd(U, S), SI), HDD)
    # u^+ and d^+
    U, D = u[1:], d[1:]
    S = [h * x for x in D]
    p = [5 / 6 * U[0] + U[1] / 6 + S[0] / 3, 13 / 6 * U[1] - 7 / 6 * U[2] + 2 / 3 * S[2], U[0] / 3 + 5 / 6 * U[1] - U[2] / 6]
    SI = _hsi(U, S)
    up = weigh(p, SI, taus(_brk(U, S), SI), (HD[1], HD[0], HD[2]))
    p = [2 * (U[1] - U[0]) / h - 0.5 * (D[0] + D[1]), 4 * (U[1] - U[2]) / h + 3.5 * D[1] + 1.5 * D[2],
         -(0.75 * U[0] - U[1] + 0.25 * U[2]) / h + 0.5 * D[1]]
    SI = _hsid(U, S)
    dp = weigh(p, SI, taus(_brkd(U, S), SI), (HDD[1], HDD[0], HDD[2]))
    if linear is not None:
        lm = -23 / 120 * u[0] + 19 / 30 * u[1] + 67 / 120 * u[2] - h * (3 / 40 * d[0] + 7 / 40 * d[2])
        lp = 67 / 120 * u[1] + 19 / 30 * u[2] - 23 / 120 * u[3] + h * (7 / 40 * d[1] + 3 / 40 * d[3])
        ldm = (0.25 * u[0] - 2 * u[1] + 1.75 * u[2]) / h + d[0] / 12 - d[1] / 6 - 5 / 12 * d[2]
        ldp = (-1.75 * u[1] + 2 * u[2] - 0.25 * u[3]) / h - 5 / 12 * d[1] - d[2] / 6 + d[3] / 12
        um, up, dm, dp = (torch.where(linear, a, b) for a, b in ((lm, um), (lp, up), (ldm, dm), (ldp, dp)))
    return um, up, dm, dp


def _limit_cell(u, d, h):
    p1, p2 = (u[1] - u[0]) / h, (u[2] - u[1]) / h
    p0 = 0.75 * (u[2] - u[0]) / h - 0.25 * (d[0] + d[2])
    s = [_brk(u, [h * x for x in d]), (u[0] - u[1]) ** 2, (u[1] - u[2]) ** 2]
    tau = ((s[0] - s[1]).abs() + (s[0] - s[2]).abs()) ** 2 / 4
    lw = (1 - 2e-5, 1e-5, 1e-5)
    w = [a * (1 + tau / (x + 1e-6)) for a, x in zip(lw, s)]
    t = w[0] + w[1] + w[2]
    return w[0] / t * (p0 / lw[0] - (lw[1] * p1 + lw[2] * p2) / lw[0]) + (w[1] * p1 + w[2] * p2) / t


def _limited(q, d, h):
    """The in-place limiter sweep along the last axis; ghost moments keep their old values."""
    u = _pad(q, 1, "zerograd").movedim(-1, 0).contiguous()
    m = _pad(d, 1, "zerograd").movedim(-1, 0).contiguous()
    for i in range(1, m.shape[0] - 1):
        m[i] = _limit_cell(u[i - 1:i + 2], m[i - 1:i + 2], h)
    return m[1:-1].movedim(0, -1).contiguous()


def _hermite_sweep(q, along, across, h):
    bc = "zerograd"
    roe = _Roe(_pad(q, 1, bc))
    values = list(_hermite_faces(_faces(roe, _pad(q, 2, bc), 4), _faces(roe, _pad(along, 2, bc), 4), h))
    values += _lagrange("teno5", _faces(roe, _pad(across, 3, bc), 6))
    F = [0, 0, 0]
    for wt, *x in zip(GAUSS, *(_at_points(v, bc) for v in values)):
        a, b, da, db, ta, tb = (roe.right(y) for y in x)
        F[0] = F[0] + wt * _rusanov(roe, a, b)
        F[1] = F[1] + wt * _drusanov(roe, a, b, da, db)
        F[2] = F[2] + wt * _drusanov(roe, a, b, ta, tb)
    return [_drop(f) for f in F]


def _hermite2d_exact(q, v, w, steps):
    ny, nx = q.shape[1:]
    dx, dy, h = 1.0 / nx, 1.0 / ny, 1.0 / nx
    for _ in range(steps):
        dt = 0.4 * min(dx, dy) / _speed2d(q)
        for s in range(3):
            raw = (q, v, w)
            lv, lw = _limited(q, v, h), _swap(_limited(_swap(q), _swap(w), h))
            if s == 0:
                raw = base = (q, lv, lw)
            x = _hermite_sweep(q, lv, lw, h)
            y = [_swap(f) for f in _hermite_sweep(_swap(q), _swap(lw), _swap(lv), h)]
            rhs = (x[0] / dx + y[0] / dy, x[1] / dx + y[2] / dy, x[2] / dx + y[1] / dy)
            q, v, w = (_rk(s, b, c, r, dt) for b, c, r in zip(base, raw, rhs))
    return {"q": q, "v": v, "w": w}


def _hermite1d_exact(q, v, steps):
    n, k = q.shape[1], 4
    h = 2.0 / n
    wrap = (np.arange(n + 2 * k) - k) % n
    flag = np.zeros((3, n + 2 * k), dtype=bool)

    def lift(a):
        t = torch.from_numpy(np.ascontiguousarray(a))
        return torch.stack([t[0], t[1], 0 * t[0], t[2]])[:, None, :]

    for _ in range(steps):
        u, p = q[1] / q[0], (q[2] - 0.5 * q[1] * q[1] / q[0]) * (GAMMA - 1)
        c = np.sqrt(np.abs(GAMMA * p / q[0]))
        dt = 0.5 * h ** (5 / 3) / max(np.abs(u - c).max(), np.abs(u + c).max())
        for s in range(3):
            U, V = q[:, wrap], v[:, wrap]
            for e in range(3):
                for i in range(2, n + 2 * k - 2):
                    if flag[e, i]:
                        continue
                    a, b, d = U[e, i - 1], U[e, i], U[e, i + 1]
                    curve = -a + 2 * b - d
                    if abs(curve) / 2 > 0.5 * h and 0 <= (-2 * a + 3 * b - d) / curve * h <= 3 * h:
                        flag[e, i - 1:i + 2] = True
            if flag[:, 2:-2].any():
                Ut, Vt = torch.from_numpy(np.ascontiguousarray(U.T)), torch.from_numpy(np.ascontiguousarray(V.T))
                for i in range(k - 1, n + k + 1):
                    Vt[i] = _limit_cell(Ut[i - 1:i + 2], Vt[i - 1:i + 2], h)
                V = Vt.numpy().T
            lv = V[:, k:n + k]
            Q, L = lift(q), lift(lv)
            roe = _Roe(_pad(Q, 1, "periodic"))
            f = torch.from_numpy(flag[:, k - 1:n + k].copy())  # the flag of the cell left of each face
            linear = ~torch.stack([f[0], f[1], f[1], f[2]])[:, None, :]
            um, up, dm, dp = _hermite_faces(_faces(roe, _pad(Q, 2, "periodic"), 4), _faces(roe, _pad(L, 2, "periodic"), 4), h, linear)
            a, b, da, db = (roe.right(x) for x in (um, up, dm, dp))
            ru, rv = ((_drop(F) / h)[[0, 1, 3], 0].numpy() for F in (_rusanov(roe, a, b), _drusanov(roe, a, b, da, db)))
            raw = (q, v)
            if s == 0:
                raw = base = (q, lv)
            q, v = _rk(s, base[0], raw[0], ru, dt), _rk(s, base[1], raw[1], rv, dt)
    return {"q": q, "v": v}


def _mlp_exact(case, seed):
    x, y = _stencils(case["rows"], seed)
    x, p = x.double(), torch.from_numpy(_params(seed)).cuda().double().requires_grad_()
    bits = torch.stack([(y >> k) & 1 for k in range(3)], 1).double()
    opt = torch.optim.Adam([p], lr=1e-3)
    n, b = case["rows"], case["batch"]
    for _ in range(case["epochs"]):
        total = 0.0
        for a in range(0, n, b):
            opt.zero_grad()
            m = min(b, n - a)
            loss = torch.nn.functional.binary_cross_entropy_with_logits(_logits(p, x[a:a + m]), bits[a:a + m], reduction="sum")
            (loss / m).backward()
            opt.step()
            total += float(loss.detach())
    with torch.no_grad():
        return {"loss": total / n, "p": torch.sigmoid(_logits(p, x)), "weights": p.detach().cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        return _mlp_exact(case, seed)
    if kind == "fv1d":
        q = torch.from_numpy(_tube(case["nx"], seed))
        return _fv1d_exact(q, case["steps"], case["recon"], case["flux"], case["bc"]).numpy()
    if kind == "hermite1d":
        return _hermite1d_exact(*_line(case["nx"], seed), case["steps"])
    if kind == "hermite2d":
        return _hermite2d_exact(*_blobs(case["nx"], case["ny"], seed), case["steps"])
    if kind == "batch":
        return torch.cat([_fv2d_exact(_quadrants(nx, ny, 1000 * seed + k), case["steps"], "teno5", "hllc", "zerograd").reshape(-1)
                          for k, (nx, ny) in enumerate(_sides(case, seed))])
    return _fv2d_exact(_state2d(case, seed), case["steps"], case["recon"], case["flux"], case["bc"])
