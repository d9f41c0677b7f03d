"""Performance cases of the distance-field solver: what its users run.

Every case goes through the package's public entry points (pdfs_gb300.api) on
seeded synthetic inputs of the kinds the solver is used for: unions of spheres
and Gaussian-bump heightmaps whose nodes near the interface are frozen at their
exact distance, and the reference program's own pipeline input (a field of
known and unknown nodes without a mask).  Inputs are made on the GPU from the
seed alone.

The kinds:
  sweep   one ordering of a host field (api.sweep)
  run_fsm rounds of the 8 orderings of a host field, no convergence test
          (api.run_fsm, the reference program's call)
  solve   a whole call on a host field: create, load, run, store, destroy
          (api.solve)
  context a resident context given new inputs: load, run, store (api.Context),
          on device tensors or, with "host", on pinned host arrays
  batch   many grids of uneven sizes in one call (api.solve_batch)
  train   a training step of the block scheduler's network: gradient of a
          mini-batch and the Adam update (api.mlp_grad, api.mlp_adam)
"""
import math

import numpy as np
import torch

from pdfs_gb300 import _lib as L
from pdfs_gb300 import api

FAR = 1.0e10      # unknown nodes of a solve
UNKNOWN = 90000.0  # unknown nodes of the reference program's pipeline

PRECISION = {"fp64": L.PREC_FP64, "fp32": L.PREC_FP32, "polish": L.PREC_FP32_POLISH64}
ARITH = {"reference": L.ARITH_REFERENCE, "fast": L.ARITH_FAST, "mixed": L.ARITH_MIXED, "pair": L.ARITH_PAIR}
SCHED = {"none": L.SCHED_NONE, "change": L.SCHED_CHANGE, "learned": L.SCHED_LEARNED, "octant": L.SCHED_OCTANT}

# the largest drawn grid of each kind (nodes): no drawn case costs more than the largest listed one
MOST_CONTEXT = 768 ** 3


def _context(name, nx, ny, nz, dz, shape, precision, arith, scheduler, tol, host=False, dx=1.0):
    return {"name": name, "kind": "context", "nx": nx, "ny": ny, "nz": nz, "dx": dx, "dz": dz, "shape": shape,
            "precision": precision, "arith": arith, "scheduler": scheduler, "tol": tol, "host": host}


def listed():
    return [
        # the smallest call: one ordering of a small ragged host grid, as a caller that keeps the reference
        # program's loop makes it; launches and set-up are all it costs
        {"name": "sweep_37x22x19", "kind": "sweep", "nx": 37, "ny": 22, "nz": 19, "dx": 1.0, "dz": 1.0, "sn": 3},
        # the unit sphere at 64^3 in the reference's arithmetic to 1e-12: the small whole solve on host data
        {"name": "solve_sphere_64_reference", "kind": "solve", "nx": 64, "ny": 64, "nz": 64, "dx": 1.0 / 63,
         "dz": 1.0 / 63, "shape": "sphere", "precision": "fp64", "arith": "reference", "scheduler": "none",
         "tol": 1e-12},
        # the reference program's call on its pipeline's input: one round, anisotropic spacing, odd sizes
        {"name": "run_fsm_151x127x110", "kind": "run_fsm", "nx": 151, "ny": 127, "nz": 110, "dx": 1.0, "dz": 0.8,
         "rounds": 1},
        # the plain FP64 solve in the library's own FP64 arithmetic, a resident grid of ordinary size
        _context("spheres_192x176x160_fp64_fast", 192, 176, 160, 1.0, "spheres", "fp64", "fast", "none", 1e-12),
        # FP32 alone, for callers who need 1e-5 relative: a mid-size grid of odd sizes
        _context("spheres_251x233x241_fp32", 251, 233, 241, 1.0, "spheres", "fp32", "fast", "none", 0.0),
        # terrain: distance above a heightmap, flat grid with half spacing in z, the default (unscheduled) polish
        _context("heightmap_512x512x128_pair", 512, 512, 128, 0.5, "heightmap", "polish", "pair", "none", 5e-6),
        # the learned block scheduler (inference inside the solve), FP32 bulk + pair polish
        _context("spheres_384_learned_pair", 384, 384, 384, 1.0, "spheres", "polish", "pair", "learned", 1e-5),
        # the octant scheduler on a large anisotropic grid that is no multiple of the tiles
        _context("spheres_530x475x500_octant_pair", 530, 475, 500, 0.5, "spheres", "polish", "pair", "octant",
                 5e-6),
        # the benchmark's grid: 768^3, 150 spheres, octant scheduler, FP32 bulk + pair polish
        _context("spheres_768_octant_pair", 768, 768, 768, 1.0, "spheres", "polish", "pair", "octant", 1e-5),
        # the same solve end to end from pinned host arrays, a grid of ordinary size
        _context("host_320x300x280_octant_pair", 320, 300, 280, 1.0, "spheres", "polish", "pair", "octant", 1e-5,
                 host=True),
        # a batch of independent grids of uneven sizes, device tensors in place
        {"name": "batch_32_grids_32_160", "kind": "batch", "count": 32, "lo": 32, "hi": 160, "precision": "polish",
         "arith": "pair", "tol": 1e-5},
        # a training step of the scheduler's network at the trainer's mini-batch size
        {"name": "train_step_8192", "kind": "train", "n": 8192},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["sweep", "run_fsm", "solve", "context", "context", "context", "context", "context", "batch",
                       "train"])
    if kind == "sweep":
        return {"kind": kind, "nx": log(7, 64), "ny": log(7, 64), "nz": log(7, 64), "dx": 1.0,
                "dz": rng.choice([1.0, 0.6]), "sn": rng.randint(1, 8)}
    if kind == "run_fsm":
        return {"kind": kind, "nx": log(40, 220), "ny": log(40, 220), "nz": log(40, 220), "dx": 1.0,
                "dz": rng.choice([1.0, 0.8]), "rounds": rng.randint(1, 2)}
    if kind == "solve":
        return {"kind": kind, "nx": log(24, 128), "ny": log(24, 128), "nz": log(24, 128), "dx": 1.0, "dz": 1.0,
                "shape": "spheres", "precision": rng.choice(["fp64", "polish"]),
                "arith": "reference", "scheduler": rng.choice(["none", "change"]), "tol": 1e-12}
    if kind == "batch":
        return {"kind": kind, "count": log(6, 40), "lo": 24, "hi": log(64, 176),
                "precision": rng.choice(["polish", "polish", "fp32"]), "arith": "pair", "tol": 1e-5}
    if kind == "train":
        return {"kind": kind, "n": log(1000, 20000)}
    precision = rng.choice(["fp32", "polish", "polish", "polish", "fp64"])
    arith = {"fp32": "fast", "polish": rng.choice(["pair", "pair", "mixed"]),
             "fp64": rng.choice(["reference", "fast"])}[precision]
    scheduler = rng.choice(["none", "change", "learned", "octant"])
    dz = rng.choice([1.0, 1.0, 0.5])
    hi = 208 if precision == "fp64" else 600
    nx, ny, nz = log(48, hi), log(48, hi), log(48, hi)
    while nx * ny * nz > MOST_CONTEXT // 3:
        nx, ny, nz = nx * 9 // 10, ny * 9 // 10, nz * 9 // 10
    tol = {"fp32": 0.0, "polish": 1e-5 * min(1.0, dz), "fp64": 1e-12}[precision]
    c = _context("", nx, ny, nz, dz, rng.choice(["spheres", "spheres", "heightmap"]), precision, arith, scheduler,
                 tol, host=rng.random() < 0.2)
    del c["name"]
    return c


# ---- inputs ------------------------------------------------------------------------
def _spacing(case):
    return (case["dx"], case["dx"], case["dz"])


def _blank(nx, ny, nz, far, dev):
    f = torch.full((nz + 2, ny + 2, nx + 2), far, dtype=torch.float64, device=dev)
    for d in range(3):
        f.select(d, 0).fill_(math.inf)
        f.select(d, -1).fill_(math.inf)
    return f


def _spheres(nx, ny, nz, sp, centres, radii, dev):
    """A union-of-spheres interface: nodes within one spacing of a sphere are frozen at their exact distance."""
    f = _blank(nx, ny, nz, FAR, dev)
    m = torch.zeros(f.shape, dtype=torch.uint8, device=dev)
    thr, n = max(sp), (nx, ny, nz)
    for c, r in zip(centres, radii):
        lo = [max(1, int(math.floor((c[a] - r - thr) / sp[a])) + 1) for a in range(3)]
        hi = [min(n[a], int(math.ceil((c[a] + r + thr) / sp[a])) + 1) for a in range(3)]
        if any(h < l for l, h in zip(lo, hi)):
            continue
        ax = [(torch.arange(lo[a], hi[a] + 1, dtype=torch.float64, device=dev) - 1) * sp[a] - float(c[a])
              for a in range(3)]
        d = (torch.sqrt(ax[2][:, None, None] ** 2 + ax[1][None, :, None] ** 2 + ax[0][None, None, :] ** 2)
             - float(r)).abs_()
        s = tuple(slice(lo[a], hi[a] + 1) for a in (2, 1, 0))
        near = d <= thr
        f[s] = torch.minimum(f[s], torch.where(near, d, FAR))
        m[s] |= near.to(torch.uint8)
    return f, m


def _random_spheres(nx, ny, nz, sp, seed, dev, count=None, rmin=4.0, rmax=50.0, log_radii=True):
    """Seeded spheres at the density of the 768^3, 150-sphere benchmark grid, radii log-uniform."""
    rng = np.random.default_rng(seed)
    ext = np.array([(nx - 1) * sp[0], (ny - 1) * sp[1], (nz - 1) * sp[2]])
    if count is None:
        count = max(4, int(150 * nx * ny * nz / 768.0 ** 3))
    rmax = max(rmin + 1.0, min(rmax, float(ext.min()) / 4))
    centres = rng.uniform(0.0, 1.0, size=(count, 3)) * ext
    radii = (np.exp(rng.uniform(math.log(rmin), math.log(rmax), size=count)) if log_radii
             else rng.uniform(rmin, rmax, size=count))
    return _spheres(nx, ny, nz, sp, centres, radii, dev)


def _heightmap(nx, ny, nz, sp, seed, dev):
    """z = h(x, y), a flat base and 8 seeded Gaussian bumps; nodes within one z-cell of it are frozen at the
    vertical distance corrected by the local slope.  The surface stays within 0.8 of the grid's height."""
    rng = np.random.default_rng(seed)
    ext = ((nx - 1) * sp[0], (ny - 1) * sp[1], (nz - 1) * sp[2])
    cx, cy = rng.uniform(0.0, ext[0], 8), rng.uniform(0.0, ext[1], 8)
    amp = rng.uniform(5.0, 40.0, 8)
    wid = rng.uniform(20.0, 120.0, 8)
    x = (torch.arange(nx, dtype=torch.float64, device=dev) * sp[0])[None, :]
    y = (torch.arange(ny, dtype=torch.float64, device=dev) * sp[1])[:, None]
    h = torch.full((ny, nx), 10.0, dtype=torch.float64, device=dev)
    hx, hy = torch.zeros_like(h), torch.zeros_like(h)
    for i in range(8):
        g = amp[i] * torch.exp(-((x - cx[i]) ** 2 + (y - cy[i]) ** 2) / (2.0 * wid[i] ** 2))
        h += g
        hx -= g * (x - cx[i]) / wid[i] ** 2
        hy -= g * (y - cy[i]) / wid[i] ** 2
    fit = min(1.0, 0.8 * ext[2] / float(h.max()))
    h, hx, hy = h * fit, hx * fit, hy * fit
    corr = torch.rsqrt(1.0 + hx ** 2 + hy ** 2)
    f = _blank(nx, ny, nz, FAR, dev)
    m = torch.zeros(f.shape, dtype=torch.uint8, device=dev)
    z = (torch.arange(nz, dtype=torch.float64, device=dev) * sp[2])[:, None, None]
    d = (z - h).abs()
    near = d <= sp[2]
    f[1:-1, 1:-1, 1:-1] = torch.where(near, d * corr, FAR)
    m[1:-1, 1:-1, 1:-1] = near.to(torch.uint8)
    return f, m


def _pipeline_field(nx, ny, nz, sp, seed, dev):
    """The field the reference program's pipeline hands to run_fsm: distances next to a few surfaces,
    the "unknown" value elsewhere, no mask."""
    f, m = _random_spheres(nx, ny, nz, sp, seed, dev, count=6, rmin=2.0, rmax=max(4.0, 0.2 * min(nx, ny, nz)))
    f[f == FAR] = UNKNOWN
    return f


def _inputs(case, seed, dev):
    nx, ny, nz, sp = case["nx"], case["ny"], case["nz"], _spacing(case)
    if case["kind"] in ("sweep", "run_fsm"):
        return _pipeline_field(nx, ny, nz, sp, seed, dev), None
    if case["shape"] == "heightmap":
        return _heightmap(nx, ny, nz, sp, seed, dev)
    if case["shape"] == "sphere":  # the unit cube's sphere, a little off centre by the seed
        rng = np.random.default_rng(seed)
        c = 0.5 + rng.uniform(-0.02, 0.02, 3)
        return _spheres(nx, ny, nz, sp, [c], [0.25], dev)
    return _random_spheres(nx, ny, nz, sp, seed, dev)


def _batch_sizes(case):
    """The grids of a batch: per-axis sizes log-uniform in lo .. hi, the same ones for every seed."""
    rng = np.random.default_rng(5)
    s = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), size=(case["count"], 3))).astype(int)
    return [tuple(int(v) for v in n) for n in s]


def _batch_inputs(case, seed, dev):
    rng = np.random.default_rng(seed)
    out = []
    for nx, ny, nz in _batch_sizes(case):
        k, s = int(rng.integers(1, 21)), int(rng.integers(0, 2 ** 31 - 1))
        out.append(_random_spheres(nx, ny, nz, (1.0, 1.0, 1.0), s, dev, count=k, rmin=3.0, rmax=30.0,
                                   log_radii=False))
    return out


def _bf16_bits(a):
    u = np.ascontiguousarray(a, dtype=np.float32).view(np.uint32).astype(np.uint64)
    return ((u + 0x7FFF + ((u >> 16) & 1)) >> 16).astype(np.uint16)


def _bf16_values(bits):
    return (bits.astype(np.uint32) << 16).view(np.float32)


def _train_inputs(case, seed):
    rng = np.random.default_rng(seed)
    p = _bf16_values(_bf16_bits(rng.normal(0.0, 0.2, L.MLP_PARAMS)))
    x = _bf16_bits(rng.uniform(-2.0, 2.0, (case["n"], L.MLP_IN)))
    y = (rng.random(case["n"]) < 0.3).astype(np.uint8)
    m = (rng.normal(0.0, 1e-3, L.MLP_PARAMS)).astype(np.float32)
    v = (rng.uniform(1e-7, 1e-5, L.MLP_PARAMS)).astype(np.float32)
    return p, x, y, m, v


def _options(case):
    return dict(freeze=L.FREEZE_MASK, precision=PRECISION[case["precision"]], arith=ARITH[case["arith"]],
                scheduler=SCHED[case["scheduler"]], tol=case["tol"])


def _pinned(t):
    return t.cpu().pin_memory().numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        return {"case": case, "in": _train_inputs(case, seed)}
    if kind == "batch":
        grids = _batch_inputs(case, seed, "cuda")
        return {"case": case, "fields": [g[0] for g in grids], "masks": [g[1] for g in grids],
                "work": [torch.empty_like(g[0]) for g in grids]}
    f, m = _inputs(case, seed, "cuda")
    if kind == "context":
        ctx = api.Context(case["nx"], case["ny"], case["nz"], _spacing(case), **_options(case))
        if case["host"]:
            f, m, out = _pinned(f), _pinned(m), _pinned(torch.empty_like(f))
            return {"case": case, "ctx": ctx, "field": f, "mask": m, "out": out}
        return {"case": case, "ctx": ctx, "field": f, "mask": m, "out": torch.empty_like(f)}
    f = f.cpu().numpy()
    m = None if m is None else m.cpu().numpy()
    return {"case": case, "field": f, "mask": m, "out": np.empty_like(f)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        p, x, y, m, v = state["in"]
        g, loss = api.mlp_grad(p, x, y, pos_weight=4.0)
        p2, m2, v2, _ = api.mlp_adam(p, m, v, g, 5, 2e-3)
        return {"grad": g, "loss": np.float32(loss), "params": p2, "m": m2, "v": v2}
    if kind == "batch":
        for a, b in zip(state["work"], state["fields"]):
            a.copy_(b)
        torch.cuda.synchronize()  # the solver works on streams of its own
        api.solve_batch(state["work"], [(1.0, 1.0, 1.0)] * case["count"], frozen=state["masks"], freeze=L.FREEZE_MASK,
                        precision=PRECISION[case["precision"]], arith=ARITH[case["arith"]], tol=case["tol"])
        return state["work"]
    if kind == "context":
        ctx = state["ctx"]
        if case["host"]:
            ctx.load(state["field"], state["mask"])
            ctx.run()
            ctx.store(state["out"])
        else:
            ctx.load(state["field"].data_ptr(), state["mask"].data_ptr())
            ctx.run()
            ctx.store(state["out"].data_ptr())
        return state["out"]
    a = state["out"]
    np.copyto(a, state["field"])
    if kind == "sweep":
        change = api.sweep(a, _spacing(case), case["sn"])
        return {"field": a, "change": np.float64(change)}
    if kind == "run_fsm":
        api.run_fsm(a, _spacing(case), rounds=case["rounds"])
        return a
    api.solve(a, _spacing(case), frozen=state["mask"], **_options(case))
    return a


def work(case):
    """One pass: every input read once and every output written once; operations: one local update (about 25
    operations) of each node, per ordering where their number is given (a network step: three products of each layer)."""
    kind = case["kind"]
    if kind == "train":
        layers = L.MLP_IN * L.MLP_HIDDEN + L.MLP_HIDDEN * L.MLP_HIDDEN + L.MLP_HIDDEN
        return {"bytes": case["n"] * (2 * L.MLP_IN + 1) + 7 * 4 * L.MLP_PARAMS, "flops": 6 * case["n"] * layers}
    if kind == "batch":
        nodes = sum(nx * ny * nz for nx, ny, nz in _batch_sizes(case))
        halo = sum((nx + 2) * (ny + 2) * (nz + 2) for nx, ny, nz in _batch_sizes(case))
        return {"bytes": 17 * halo, "flops": 25 * nodes}
    halo = (case["nx"] + 2) * (case["ny"] + 2) * (case["nz"] + 2)
    nodes = case["nx"] * case["ny"] * case["nz"]
    sweeps = {"sweep": 1, "run_fsm": 8 * case.get("rounds", 1)}.get(kind, 1)
    mask = 0 if kind in ("sweep", "run_fsm") else 1
    return {"bytes": (16 + mask) * halo, "flops": 25 * nodes * sweeps}


# ---- exact values: plain torch / numpy in 64 bits ------------------------------------
def _godunov(a, b, c, h):
    """The largest root u of sum_k max(u - m_k, 0)^2 / h_k^2 = 1, for the axis minima a, b, c."""
    m = torch.stack((a, b, c))
    m, order = torch.sort(m, dim=0)
    hs = torch.tensor(h, dtype=torch.float64, device=m.device)[order]
    q0, q1, q2 = (1.0 / hs[i] ** 2 for i in range(3))
    base = m[0]
    d1, d2 = m[1] - base, m[2] - base
    u1 = base + hs[0]
    s2 = q0 + q1
    u2 = base + (d1 * q1 + torch.sqrt((s2 - d1 * d1 * q0 * q1).clamp_min(0.0))) / s2
    s3 = s2 + q2
    B = d1 * q1 + d2 * q2
    u3 = base + (B + torch.sqrt((B * B - s3 * (d1 * d1 * q1 + d2 * d2 * q2 - 1.0)).clamp_min(0.0))) / s3
    u = torch.where(u1 <= m[1], u1, torch.where(u2 <= m[2], u2, u3))
    return torch.where(torch.isfinite(base), u, base)


def _signs(sn):
    desc = -1 if sn in (2, 5, 7, 8) else 1
    return ((-1 if sn in (4, 8) else 1) * desc, (-1 if sn in (2, 6) else 1) * desc, (-1 if sn in (3, 7) else 1) * desc)


def _orderings(f, sp, sweeps):
    """Gauss-Seidel orderings of a field in place, one hyperplane at a time; the last one's largest change."""
    nz, ny, nx = (s - 2 for s in f.shape)
    dev = f.device
    z, y, x = torch.meshgrid(*(torch.arange(n, device=dev) for n in (nz, ny, nx)), indexing="ij")
    level = (x + y + z).reshape(-1)
    order = torch.argsort(level, stable=True)
    x, y, z = (t.reshape(-1)[order] for t in (x, y, z))
    ends = torch.cumsum(torch.bincount(level), 0).tolist()
    u = f.view(-1)
    sy, sz = nx + 2, (nx + 2) * (ny + 2)
    change = 0.0
    for sn in sweeps:
        gx, gy, gz = _signs(sn)
        ix = 1 + (x if gx > 0 else nx - 1 - x)
        iy = 1 + (y if gy > 0 else ny - 1 - y)
        iz = 1 + (z if gz > 0 else nz - 1 - z)
        idx = iz * sz + iy * sy + ix
        old = u.clone()
        lo = 0
        for hi in ends:
            i = idx[lo:hi]
            v = _godunov(torch.minimum(u[i - 1], u[i + 1]), torch.minimum(u[i - sy], u[i + sy]),
                         torch.minimum(u[i - sz], u[i + sz]), sp)
            u[i] = torch.minimum(u[i], v)
            lo = hi
        d = (old - u)[idx]
        change = float(d.max())
    return change


def _fixed_point(f, m, sp):
    """The fixed point u = min(u, G(u)) on the nodes that are not frozen, by simultaneous updates."""
    c = f[1:-1, 1:-1, 1:-1]
    free = m[1:-1, 1:-1, 1:-1] == 0
    slabs = max(1, c.numel() // 30_000_000)
    h = float(min(sp))
    for it in range(1, 20000):
        bounds = [c.shape[0] * k // slabs for k in range(slabs + 1)]
        test = it % 25 == 0
        change = 0.0
        for a, b in zip(bounds, bounds[1:]):  # slab by slab: bounds the memory of the intermediate values
            v = f[a:b + 2]
            g = _godunov(torch.minimum(v[1:-1, 1:-1, :-2], v[1:-1, 1:-1, 2:]),
                         torch.minimum(v[1:-1, :-2, 1:-1], v[1:-1, 2:, 1:-1]),
                         torch.minimum(v[:-2, 1:-1, 1:-1], v[2:, 1:-1, 1:-1]), sp)
            w = v[1:-1, 1:-1, 1:-1]
            g = torch.where(free[a:b], torch.minimum(w, g), w)
            if test:
                change = max(change, float((w - g).max()))
            w.copy_(g)
        if test and change <= 1e-13 * h:
            break
    return f


def _train_exact(case, seed):
    p, x, y, m, v = _train_inputs(case, seed)

    def r(a):  # the network's bf16 activations
        return _bf16_values(_bf16_bits(a)).astype(np.float64)

    ni, nh, o = L.MLP_IN, L.MLP_HIDDEN, 0
    parts = []
    for n in (nh * ni, nh, nh * nh, nh, nh, 1):
        parts.append(p[o:o + n].astype(np.float64))
        o += n
    W1, b1, W2, b2, w3, b3 = parts
    W1, W2 = W1.reshape(nh, ni), W2.reshape(nh, nh)
    xv = _bf16_values(x).astype(np.float64)
    h1 = r(np.maximum(xv @ W1.T + b1, 0.0))
    h2 = r(np.maximum(h1 @ W2.T + b2, 0.0))
    s = h2 @ w3 + b3
    wy = np.where(y > 0, 4.0, 1.0)
    n = len(y)
    loss = float(np.sum(wy * (np.maximum(s, 0) - s * y + np.log1p(np.exp(-np.abs(s))))) / n)
    ds = wy * (1.0 / (1.0 + np.exp(-s)) - y) / n
    d2 = (h2 > 0) * ds[:, None] * w3[None, :]
    d1 = (h1 > 0) * (d2 @ W2)
    g = np.concatenate([(d1.T @ xv).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), h2.T @ ds, [ds.sum()]])
    m2 = 0.9 * m + 0.1 * g
    v2 = 0.999 * v + 0.001 * g * g
    p2 = p - 2e-3 * (m2 / (1 - 0.9 ** 5)) / (np.sqrt(v2 / (1 - 0.999 ** 5)) + 1e-8)
    return {"grad": g, "loss": np.float64(loss), "params": p2, "m": m2, "v": v2}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _train_exact(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "batch":
        return [_fixed_point(f, m, (1.0, 1.0, 1.0)) for f, m in _batch_inputs(case, seed, dev)]
    if case["nx"] * case["ny"] * case["nz"] > 60_000_000:
        return None  # too long in plain torch
    sp = _spacing(case)
    f, m = _inputs(case, seed, dev)
    if kind == "sweep":
        return {"field": f, "change": np.float64(_orderings(f, sp, [case["sn"]]))}
    if kind == "run_fsm":
        _orderings(f, sp, [s for _ in range(case["rounds"]) for s in range(1, 9)])
        return f
    return _fixed_point(f, m, sp)
