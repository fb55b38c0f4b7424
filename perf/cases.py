"""Workloads of the reconstruction engine for performance measurement.

Every case is a dict of plain values.  `listed()` names the fixed ones,
`draw(rng)` gives another of the same ranges, `prepare(case, seed)` builds
what a program holds before the call (inputs on the GPU made from the seed
alone, a plan or a network), `run(state)` is one pass through the public
entry points, `work(case)` the bytes and operations it cannot do without and
`exact(case, seed)` the same outputs in 64-bit arithmetic by plain torch.

Acquisitions are linear sweeps (geometry.linear_sweep).  Input data never
come from the engine's own projectors: volumes are rasterised ellipsoids,
projections their analytic line integrals with Poisson counting noise.
"""
import ctypes
import math
import os

import numpy as np
import torch

from kevernals_gb300 import _lib, engine
from kevernals_gb300 import geometry as geo

HERE = os.path.dirname(os.path.abspath(__file__))
WEIGHTS = os.path.join(os.path.dirname(HERE), "kevernals_gb300", "weights", "unet_chest_dt.npz")

# the U-Net's 3x3x3 convolutions after the first: (c1, c2, cout), and the level each runs at
CONVS = [(16, 0, 16), (16, 0, 32), (32, 0, 32), (32, 0, 64), (64, 0, 64), (64, 0, 128), (128, 0, 128),
         (128, 64, 64), (64, 0, 64), (64, 32, 32), (32, 0, 32), (32, 16, 16), (16, 0, 16)]
LEVELS = [0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0]


def _acq(nx, ny, nz, dx, dz, views, nu, nv, du, angle):
    return {"nx": nx, "ny": ny, "nz": nz, "dx": dx, "dz": dz, "views": views, "nu": nu, "nv": nv, "du": du,
            "angle": angle}


SMALL = _acq(256, 256, 64, 0.5, 1.0, 15, 512, 512, 0.4, 15.0)         # geometry.config_small()
CHEST = _acq(1024, 1024, 128, 0.4, 2.5, 60, 2048, 2048, 0.2, 17.5)    # geometry.config_chest()
MEDIUM = _acq(512, 512, 96, 0.5, 1.0, 25, 1024, 1024, 0.4, 20.0)      # the largest of geometry.uneven_cases
TINY = _acq(48, 40, 12, 0.5, 1.0, 7, 64, 56, 0.4, 15.0)               # the smoke test's size
RAGGED = _acq(213, 187, 41, 0.5, 1.0, 21, 333, 287, 0.45, 17.0)       # odd rows: no whole 16-byte units


def listed():
    return [
        # the smallest call: a whole solve of a test-sized problem, latency and launches
        {"name": "mlem_tiny", "kind": "mlem", "family": "exact", "storage": "f32", "iterations": 5, **TINY},
        # both operators once, as gradient-type solvers written on top of them call them
        {"name": "project_small", "kind": "project", **SMALL},
        # a solve with the 16-bit storage option
        {"name": "mlem_small_bf16", "kind": "mlem", "family": "exact", "storage": "bf16", "iterations": 5, **SMALL},
        # SART on a cropped detector and volume: odd sizes in every direction
        {"name": "sart_ragged", "kind": "sart", "iterations": 5, **RAGGED},
        # the headline: MLEM at the chest tomosynthesis size
        {"name": "mlem_chest", "kind": "mlem", "family": "exact", "storage": "f32", "iterations": 2, **CHEST},
        # the reference-compatible operators, what the C++ drop-in classes run by default
        {"name": "mlem_small_rc", "kind": "mlem", "family": "rc", "storage": "f32", "iterations": 2, **SMALL},
        # shift-and-add of a whole chest acquisition
        {"name": "saa_chest", "kind": "saa", **CHEST},
        # filtered backprojection of the largest of the uneven problems
        {"name": "fbp_medium", "kind": "fbp", "half_taps": 128, **MEDIUM},
        # many small uneven problems solved together
        {"name": "batch_uneven", "kind": "batch", "count": 32, "scale": 4, "iterations": 5, "set": 3000},
        # one layer of the warm-start network: the full-resolution decoder's concatenated input
        {"name": "conv_decoder", "kind": "conv", "c1": 32, "c2": 16, "cout": 16, "D": 128, "H": 256, "W": 128},
        # the warm-start network on half the chest volume's sampling
        {"name": "unet_forward", "kind": "unet_forward", "D": 128, "H": 512, "W": 512},
        # its training: loss and all gradients on one training crop
        {"name": "unet_gradients", "kind": "unet_gradients", "D": 128, "H": 256, "W": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_acq(rng, rays):
    """An acquisition with at most `rays` rays in all."""
    while True:
        dx = rng.choice([0.4, 0.5, 0.8])
        nx, ny, nz = _log(rng, 40, 700), _log(rng, 40, 700), _log(rng, 8, 128)
        if rng.random() < 0.5:
            nx, ny = (nx + 31) // 32 * 32, (ny + 31) // 32 * 32
        views, du = rng.randint(7, 60), round(dx * rng.uniform(0.5, 0.95), 2)
        nu = int(nx * dx * rng.uniform(1.05, 1.3) / du)
        nv = int(ny * dx * rng.uniform(1.05, 1.3) / du)
        if rng.random() < 0.5:
            nu, nv = (nu + 15) // 16 * 16, (nv + 15) // 16 * 16
        if views * nu * nv <= rays:
            return _acq(nx, ny, nz, dx, rng.choice([1.0, 2.5]), views, nu, nv, du, round(rng.uniform(8.0, 22.0), 1))


def draw(rng):
    kind = rng.choice(["mlem", "mlem", "project", "sart", "rc", "saa", "fbp", "batch", "conv", "unet_forward",
                       "unet_gradients"])
    if kind == "mlem":
        return {"kind": "mlem", "family": "exact", "storage": rng.choice(["f32", "f32", "bf16", "f16"]),
                "iterations": rng.randint(1, 6), **_draw_acq(rng, 3.0e7)}
    if kind == "rc":
        return {"kind": "mlem", "family": "rc", "storage": "f32", "iterations": rng.randint(1, 3),
                **_draw_acq(rng, 6.0e6)}
    if kind == "sart":
        return {"kind": "sart", "iterations": rng.randint(1, 6), **_draw_acq(rng, 3.0e7)}
    if kind == "fbp":
        return {"kind": "fbp", "half_taps": rng.choice([16, 64, 128, 256]), **_draw_acq(rng, 3.0e7)}
    if kind in ("project", "saa"):
        return {"kind": kind, **_draw_acq(rng, 6.0e7)}
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(4, 48), "scale": rng.choice([2, 4, 8]),
                "iterations": rng.randint(2, 8), "set": rng.randint(1, 1 << 20)}
    if kind == "conv":
        n = rng.randrange(len(CONVS))
        c1, c2, cout = CONVS[n]
        l = LEVELS[n]
        d, h, w = 8 * rng.randint(1, 16), 8 * rng.randint(2, 32), 128 * rng.randint(1, 3)
        return {"kind": "conv", "c1": c1, "c2": c2, "cout": cout, "D": d >> l, "H": h >> l, "W": w >> l}
    if kind == "unet_forward":
        return {"kind": kind, "D": 8 * _log(rng, 1, 16), "H": 8 * _log(rng, 2, 64), "W": 128 * rng.randint(1, 4)}
    return {"kind": kind, "D": 8 * _log(rng, 1, 16), "H": 8 * _log(rng, 2, 32), "W": 128 * rng.randint(1, 2)}


# ---------------------------------------------------------------- inputs

_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = engine.Context(0)
    return _ctx


def _geometry(c):
    return geo.linear_sweep(c["nx"], c["ny"], c["nz"], c["dx"], c["dx"], c["dz"], c["views"], c["nu"], c["nv"],
                            c["du"], c["du"], c["angle"])


def _ellipsoids(g, seed, n=10):
    """[(centre, 1 / semi-axes, density)]: a body and n smaller parts."""
    r = np.random.default_rng(seed)
    ext = np.array([g.nx * g.dx, g.ny * g.dy, g.nz * g.dz])
    out = [(np.zeros(3), 1.0 / (0.45 * ext), 0.02)]
    for _ in range(n):
        out.append((r.uniform(-0.33, 0.33, 3) * ext, 1.0 / (r.uniform(0.03, 0.15, 3) * ext), r.uniform(0.0, 0.05)))
    return out


def _volume(g, seed, dev="cuda"):
    ax = [(torch.arange(n, device=dev, dtype=torch.float32) + 0.5 - 0.5 * n) * d
          for n, d in ((g.nz, g.dz), (g.ny, g.dy), (g.nx, g.dx))]
    v = torch.zeros(g.volume_shape, device=dev)
    for c, ia, mu in _ellipsoids(g, seed):
        z, y, x = (((a - float(c[i])) * float(ia[i])) ** 2 for a, i in zip(ax, (2, 1, 0)))
        v += float(mu) * ((z[:, None] + y)[:, :, None] + x <= 1.0)
    return v


def _projections(g, seed, i0=5.0e4, dev="cuda"):
    """ln(I0 / counts) of the ellipsoids' analytic line integrals."""
    gen = torch.Generator(device=dev).manual_seed(int(seed) + 7)
    parts = _ellipsoids(g, seed)
    out = torch.empty(g.proj_shape, device=dev)
    for p in range(g.n_views):
        s, o = g.src[p].astype(np.float64), g.det_origin[p].astype(np.float64)
        d = [torch.arange(g.nu, device=dev, dtype=torch.float32).add_(0.5).mul_(g.du).add_(float(o[0] - s[0])),
             torch.arange(g.nv, device=dev, dtype=torch.float32).add_(0.5).mul_(g.du).add_(float(o[1] - s[1])),
             torch.tensor(float(o[2] - s[2]), device=dev)]
        length = torch.sqrt((d[1] ** 2)[:, None] + d[0] ** 2 + d[2] ** 2)
        line = torch.zeros_like(length)
        for c, ia, mu in parts:
            e = [float((s[i] - c[i]) * ia[i]) for i in range(3)]
            q = [d[i] * float(ia[i]) for i in range(3)]
            a = (q[1] ** 2 + q[2] ** 2)[:, None] + q[0] ** 2
            b = (q[1] * e[1] + q[2] * e[2])[:, None] + q[0] * e[0]
            disc = b * b - a * (e[0] ** 2 + e[1] ** 2 + e[2] ** 2 - 1.0)
            line += (2.0 * float(mu)) * disc.clamp_min_(0.0).sqrt_() / a
        counts = torch.poisson(i0 * torch.exp(-line * length), generator=gen)
        out[p] = torch.log(i0 / counts.clamp_min(1.0)).clamp_min(0.0)
    return out


def _unet_pair(D, H, W, seed):
    """A blurred, noisy volume (the network's input) and the one it stands for, NaN where no ray sees it."""
    g = geo.linear_sweep(W, H, D, 0.4, 0.4, 2.5, 2, 8, 8, 0.4, 0.4, 10.0)
    t = _volume(g, seed)
    gen = torch.Generator(device="cuda").manual_seed(int(seed) + 11)
    x = torch.nn.functional.avg_pool3d(t[None], (5, 3, 3), 1, (2, 1, 1), count_include_pad=False)[0]
    x = (x + 0.001 * torch.randn(t.shape, device="cuda", generator=gen)).contiguous()
    t[:, :, : max(1, W // 32)] = float("nan")
    return x, t


def _batch_geometries(c):
    return geo.uneven_cases(c["count"], c["set"], scale=c["scale"])


def _conv_inputs(c, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))

    def rnd(*shape):
        return torch.randn(shape, device="cuda", generator=gen)
    D, H, W, c1, c2, n = (c[k] for k in ("D", "H", "W", "c1", "c2", "cout"))
    a = torch.relu(rnd(D, H, W, c1)).to(torch.bfloat16)
    b = torch.relu(rnd(D, H, W, c2)).to(torch.bfloat16) if c2 else None
    w = (rnd(n, 27, c1 + c2) * math.sqrt(2.0 / (27 * (c1 + c2)))).to(torch.bfloat16)
    return a, b, w, 0.1 * rnd(n)


def prepare(case, seed):
    c, kind, ctx = case, case["kind"], _context()
    st = {"case": c, "kind": kind}
    if kind == "conv":
        st["a"], st["b"], st["w"], st["bias"] = _conv_inputs(c, seed)
        st["out"] = torch.empty((c["D"], c["H"], c["W"], c["cout"]), dtype=torch.bfloat16, device="cuda")
    elif kind in ("unet_forward", "unet_gradients"):
        st["net"] = engine.UNet(ctx, seed=1)
        st["net"].load(WEIGHTS)
        st["x"], st["t"] = _unet_pair(c["D"], c["H"], c["W"], seed)
    elif kind == "batch":
        gs = _batch_geometries(c)
        st["plans"] = [engine.Plan(ctx, g) for g in gs]
        st["p"] = [_projections(g, seed + 13 * i) for i, g in enumerate(gs)]
        st["x"] = [torch.empty(g.volume_shape, device="cuda") for g in gs]
        for plan in st["plans"]:
            plan.sensitivity(device=True)
    else:
        g = _geometry(c)
        st["plan"] = engine.Plan(ctx, g, c.get("family", "exact"), c.get("storage", "f32"))
        if kind == "project":
            st["v"], st["p"] = _volume(g, seed), _projections(g, seed)
        else:
            st["p"] = _projections(g, seed)
        if kind in ("mlem", "sart"):
            st["x"] = torch.empty(g.volume_shape, device="cuda")
        if kind in ("mlem", "sart", "fbp") and c.get("family", "exact") == "exact":
            st["plan"].sensitivity(device=True)
    return st


def run(state):
    c, kind = state["case"], state["kind"]
    if kind == "project":
        return {"projections": state["plan"].forward(state["v"]), "volume": state["plan"].back(state["p"])}
    if kind == "mlem":
        state["plan"].mlem(state["p"], state["x"].fill_(1.0), c["iterations"])
        return state["x"]
    if kind == "sart":
        state["plan"].sart(state["p"], state["x"].fill_(0.0), c["iterations"], 0.5)
        return state["x"]
    if kind == "saa":
        return state["plan"].shift_and_add(state["p"])
    if kind == "fbp":
        return state["plan"].fbp(state["p"], c["half_taps"])
    if kind == "batch":
        for x in state["x"]:
            x.fill_(1.0)
        engine.batch_mlem(_context(), state["plans"], state["p"], state["x"], c["iterations"])
        return torch.cat([x.reshape(-1) for x in state["x"]])
    if kind == "conv":
        ctx, b, out = _context(), state["b"], state["out"]
        ctx.use_torch_stream()
        ctx.check(_lib.lib().kv_conv3_bf16(
            ctx.handle, ctypes.c_void_p(state["a"].data_ptr()), c["c1"],
            ctypes.c_void_p(b.data_ptr() if b is not None else 0), c["c2"], ctypes.c_void_p(state["w"].data_ptr()),
            ctypes.c_void_p(state["bias"].data_ptr()), 1, ctypes.c_void_p(out.data_ptr()), c["cout"], c["D"], c["H"],
            c["W"], 0))
        return out
    if kind == "unet_forward":
        return state["net"].forward(state["x"])
    loss, grads = state["net"].gradients(state["x"], state["t"])
    return {"loss": loss, "gradients": grads}


# ---------------------------------------------------------------- work

def _unet_macs(D, H, W):
    n0 = D * H * W
    return n0 * (27 * 16 + 16) + sum((n0 >> (3 * l)) * 27 * (a + b) * n for (a, b, n), l in zip(CONVS, LEVELS))


def work(case):
    c, kind = case, case["kind"]
    if kind == "conv":
        n, k = c["D"] * c["H"] * c["W"], c["c1"] + c["c2"]
        return {"bytes": 2 * (n * (k + c["cout"]) + 27 * k * c["cout"]), "flops": 54 * n * k * c["cout"]}
    if kind.startswith("unet"):
        n, macs = c["D"] * c["H"] * c["W"], _unet_macs(c["D"], c["H"], c["W"])
        if kind == "unet_forward":
            return {"bytes": 8 * n + 4 * 1459592, "flops": 2 * macs}
        return {"bytes": 8 * n + 8 * 1459592, "flops": 6 * macs}
    if kind == "batch":
        seg = [geo.siddon_segments(g, 8) for g in _batch_geometries(c)]
        byt = [8 * g.n_rays + 16 * g.n_voxels for g in _batch_geometries(c)]
        return {"bytes": sum(byt) * c["iterations"], "flops": 4 * sum(seg) * c["iterations"]}
    g = _geometry(c)
    V, R = g.n_voxels, g.n_rays
    if kind == "saa":
        return {"bytes": 4 * R + 4 * g.nz * g.nu * g.nv, "flops": g.nz * R}
    seg = geo.siddon_segments(g, 16)
    if kind == "project":
        return {"bytes": 8 * (V + R), "flops": 4 * seg}
    if kind == "fbp":
        return {"bytes": 4 * R + 12 * V, "flops": 2 * seg + R * (4 * c["half_taps"] + 1)}
    es = 4 if c.get("storage", "f32") == "f32" else 2
    it = c["iterations"]
    return {"bytes": it * (es * (2 * R + 3 * V) + 8 * V + es * R), "flops": 4 * seg * it}


# ---------------------------------------------------------------- 64-bit values

class _Projector:
    """Line integrals through a voxel grid and their transpose, in 64 bits: slice by slice, the part of the slice
    a ray spends in a voxel is the overlap of its column's and its row's intervals."""

    def __init__(self, g):
        self.g = g
        self.src = torch.from_numpy(g.src.astype(np.float64)).cuda()
        self.det = torch.from_numpy(g.det_origin.astype(np.float64)).cuda()
        self.H = self.src[:, 2] - self.det[:, 2]
        self.pu = self.det[:, 0:1] + (torch.arange(g.nu, device="cuda", dtype=torch.float64) + 0.5) * g.du
        self.pv = self.det[:, 1:2] + (torch.arange(g.nv, device="cuda", dtype=torch.float64) + 0.5) * g.dv
        self.step = max(1, int(3.0e7 // (g.nu * g.nv)))

    def lengths(self, a, b):
        ax = self.src[a:b, 0:1] - self.pu[a:b]
        ay = self.src[a:b, 1:2] - self.pv[a:b]
        H = self.H[a:b]
        return torch.sqrt(ax[:, None, :] ** 2 + ay[:, :, None] ** 2 + (H * H)[:, None, None]) * (self.g.dz / H)[:, None, None]

    def cells(self, a, b, k, axis):
        """[(index, in-range lo, hi)] over the candidate columns (axis 0) or rows (1) of slice k."""
        g = self.g
        pix, s = (self.pu, self.src[a:b, 0:1]) if axis == 0 else (self.pv, self.src[a:b, 1:2])
        n, sp = (g.nx, g.dx) if axis == 0 else (g.ny, g.dy)
        pos = []
        for kk in (k + 1, k):   # top plane (t = 0), bottom plane (t = 1)
            z = (kk - 0.5 * g.nz) * g.dz
            h = ((z - self.det[a:b, 2]) / self.H[a:b])[:, None]
            pos.append((pix[a:b] + (s - pix[a:b]) * h) / sp + 0.5 * n)
        top, bot = pos
        first = torch.floor(torch.minimum(top, bot))
        count = int((torch.floor(torch.maximum(top, bot)) - first).max().item()) + 1
        slope = bot - top
        flat = slope.abs() < 1e-12
        slope = torch.where(flat, torch.ones_like(slope), slope)
        out = []
        for m in range(count):
            c = first + m
            t0, t1 = (c - top) / slope, (c + 1 - top) / slope
            lo = torch.where(flat, torch.zeros_like(t0), torch.minimum(t0, t1).clamp_min(0.0))
            hi = torch.where(flat, torch.full_like(t0, 1.0 if m == 0 else 0.0), torch.maximum(t0, t1).clamp_max(1.0))
            inside = (c >= 0) & (c < n)
            out.append((torch.where(inside, c, torch.zeros_like(c)).long(), torch.where(inside, lo, torch.ones_like(lo)),
                        torch.where(inside, hi, torch.zeros_like(hi))))
        return out

    def weights(self, a, b, k):
        cols, rows = self.cells(a, b, k, 0), self.cells(a, b, k, 1)
        for i, xl, xh in cols:
            for j, yl, yh in rows:
                w = torch.minimum(xh[:, None, :], yh[:, :, None])
                w -= torch.maximum(xl[:, None, :], yl[:, :, None])
                yield w.clamp_min_(0.0), j[:, :, None] * self.g.nx + i[:, None, :]

    def forward(self, x):
        out = torch.empty(self.g.proj_shape, device="cuda", dtype=torch.float64)
        for a in range(0, self.g.n_views, self.step):
            b = min(a + self.step, self.g.n_views)
            acc = torch.zeros((b - a, self.g.nv, self.g.nu), device="cuda", dtype=torch.float64)
            for k in range(self.g.nz):
                flat = x[k].reshape(-1)
                for w, idx in self.weights(a, b, k):
                    acc.addcmul_(w, flat[idx])
            out[a:b] = acc * self.lengths(a, b)
        return out

    def back(self, y):
        out = torch.zeros((self.g.nz, self.g.ny * self.g.nx), device="cuda", dtype=torch.float64)
        for a in range(0, self.g.n_views, self.step):
            b = min(a + self.step, self.g.n_views)
            ys = y[a:b] * self.lengths(a, b)
            for k in range(self.g.nz):
                for w, idx in self.weights(a, b, k):
                    out[k].index_add_(0, idx.reshape(-1), w.mul_(ys).reshape(-1))
        return out.reshape(self.g.volume_shape)


def _safe_div(a, b):
    return torch.where(b > 0, a / torch.where(b > 0, b, torch.ones_like(b)), torch.zeros_like(a))


def _exact_solve(g, p, iterations, sart):
    A = _Projector(g)
    p = p.double()
    one = torch.ones_like(p)
    sens = A.back(one)
    x = torch.zeros(g.volume_shape, device="cuda", dtype=torch.float64) if sart else \
        torch.ones(g.volume_shape, device="cuda", dtype=torch.float64)
    rows = A.forward(torch.ones_like(x)) if sart else None
    for _ in range(iterations):
        q = A.forward(x)
        if sart:
            x = x + _safe_div(0.5 * A.back(_safe_div(p - q, rows)), sens)
        else:
            x = torch.where(sens > 0, x * _safe_div(A.back(_safe_div(p, q)), sens), x)
    return x


def _shifts(g):
    sid = float(np.mean(g.src[:, 2].astype(np.float32))) - float(np.float32(np.mean(g.det_origin[:, 2].astype(np.float64))))
    det = float(np.float32(np.mean(g.det_origin[:, 2].astype(np.float64))))
    mf = sid / (sid - (g.fulcrum_z - det))
    hz = -0.5 * g.nz * g.dz + (np.arange(g.nz) + 0.5) * g.dz - det
    q = g.src[None, :, 1].astype(np.float64) * ((sid / (sid - hz)) - mf)[:, None] / g.dv
    return (np.sign(q) * np.floor(np.abs(q) + 0.5)).astype(np.int64)


def _exact_saa(g, p):
    sh = _shifts(g)
    out = torch.zeros((g.nz, g.nv, g.nu), device="cuda", dtype=torch.float64)
    for k in range(g.nz):
        for i in range(g.n_views):
            t = int(sh[k, i])
            a, b = max(0, -t), min(g.nv, g.nv - t)
            if a < b:
                out[k, a:b] += p[i, a + t:b + t]
    return out / g.n_views


def _exact_fbp(g, p, K):
    p = p.double()
    f = torch.zeros_like(p)
    for n in range(-K, K + 1):
        h = -2.0 / (math.pi ** 2 * (4.0 * n * n - 1.0))
        a, b = max(0, n), min(g.nv, g.nv + n)
        if a < b:
            f[:, a:b] += h * p[:, a - n:b - n]
    A = _Projector(g)
    return _safe_div(A.back(f), A.back(torch.ones_like(p)))


class _Conv64(torch.autograd.Function):
    """3x3x3 convolution with zero padding on [D][H][W][C], weights [N][27][C]."""

    @staticmethod
    def taps(x):
        D, H, W, C = x.shape
        xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
        for t in range(27):
            z, y, w = t // 9, t // 3 % 3, t % 3
            yield t, xp[z:z + D, y:y + H, w:w + W].reshape(-1, C)

    @staticmethod
    def apply_(x, w):
        out = x.new_zeros((x.shape[0] * x.shape[1] * x.shape[2], w.shape[0]))
        for t, a in _Conv64.taps(x):
            out.addmm_(a, w[:, t].t())
        return out.reshape(*x.shape[:3], w.shape[0])

    @staticmethod
    def forward(ctx, x, w):
        ctx.save_for_backward(x, w)
        return _Conv64.apply_(x, w)

    @staticmethod
    def backward(ctx, g):
        x, w = ctx.saved_tensors
        gf = g.reshape(-1, g.shape[-1])
        dw = torch.stack([gf.t() @ a for _, a in _Conv64.taps(x)], 1)
        dx = _Conv64.apply_(g.contiguous(), w.flip(1).permute(2, 1, 0).contiguous()) if ctx.needs_input_grad[0] else None
        return dx, dw


def _unet64(x, flat):
    off = [0]

    def take(n, shape):
        v = flat[off[0]:off[0] + n].reshape(shape)
        off[0] += n
        return v

    def conv(v, w, b):
        return torch.relu(_Conv64.apply(v, w) + b)

    def pool(v):
        return torch.nn.functional.avg_pool3d(v.permute(3, 0, 1, 2)[None], 2)[0].permute(1, 2, 3, 0)

    def up(v):
        return v.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)
    w0, b0 = take(432, (16, 27, 1)), take(16, (16,))
    lay = []
    for a, b, n in CONVS:
        lay.append((take(n * 27 * (a + b), (n, 27, a + b)), take(n, (n,))))
        off[0] = (off[0] + 7) & ~7
    wo, bo = take(16, (16,)), take(1, (1,))
    e1 = conv(conv(x[..., None], w0, b0), *lay[0])
    e2 = conv(conv(pool(e1), *lay[1]), *lay[2])
    e3 = conv(conv(pool(e2), *lay[3]), *lay[4])
    m = conv(conv(pool(e3), *lay[5]), *lay[6])
    d3 = conv(conv(torch.cat([up(m), e3], 3), *lay[7]), *lay[8])
    d2 = conv(conv(torch.cat([up(d3), e2], 3), *lay[9]), *lay[10])
    d1 = conv(conv(torch.cat([up(d2), e1], 3), *lay[11]), *lay[12])
    return x + d1 @ wo + bo


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "conv":
        a, b, w, bias = _conv_inputs(c, seed)
        x = (a if b is None else torch.cat([a, b], 3)).double()
        return torch.relu(_Conv64.apply_(x, w.double()) + bias.double())
    if kind.startswith("unet"):
        n = c["D"] * c["H"] * c["W"]
        flat = torch.from_numpy(np.asarray(np.load(WEIGHTS)["params"], np.float64)).cuda()
        x, t = _unet_pair(c["D"], c["H"], c["W"], seed)
        if kind == "unet_forward":
            return None if n > 4.0e7 else _unet64(x.double(), flat)
        if n > 5.0e6:
            return None
        flat.requires_grad_(True)
        y = _unet64(x.double(), flat)
        seen = ~torch.isnan(t)
        loss = ((y - torch.where(seen, t, torch.zeros_like(t)).double()) ** 2)[seen].sum() / n
        loss.backward()
        return {"loss": float(loss), "gradients": flat.grad.cpu().numpy()}
    if kind == "batch":
        gs = _batch_geometries(c)
        if sum(g.n_rays * g.nz for g in gs) * c["iterations"] > 1.0e10:
            return None
        return torch.cat([_exact_solve(g, _projections(g, seed + 13 * i), c["iterations"], False).reshape(-1)
                          for i, g in enumerate(gs)])
    g = _geometry(c)
    cost = g.n_rays * g.nz
    if kind == "saa":
        return _exact_saa(g, _projections(g, seed).double())
    if c.get("family") == "rc":
        return None   # the reference's own float arithmetic, roundings included, is the definition
    passes = 2 if kind in ("project", "fbp") else 2 * c["iterations"] + 2
    if cost * passes > 8.0e9:
        return None
    if kind == "project":
        A = _Projector(g)
        return {"projections": A.forward(_volume(g, seed).double()), "volume": A.back(_projections(g, seed).double())}
    if kind == "fbp":
        return _exact_fbp(g, _projections(g, seed), c["half_taps"])
    return _exact_solve(g, _projections(g, seed), c["iterations"], kind == "sart")
