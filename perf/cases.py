"""The work that users of this package have it do, as cases to time.

Every case goes through the package's public Python entry points.  The sizes are those of the
repository's own benchmark workloads and tests, with odd and ragged ones between them.  Models are
seeded layered velocity models with smooth random perturbations; sources are seeded and uniform in
the domain (or on its surface).  `exact` restates the solver in plain numpy, and the network in
plain torch, in 64 bits, where that takes seconds.
"""
import math

import numpy as np
import torch

import eikonalxx_gb300 as ex
from eikonalxx_gb300.warmstart import WarmNet

DEV = "cuda"


def _solve3(name, nx, ny, nz, h, n_src, hz=None, precision="f32", near=False, slots=0, n_sweeps=10, tol=1e-5,
            surface=False, set_model=False):
    return {"name": name, "kind": "solve3d", "nx": nx, "ny": ny, "nz": nz, "h": float(h), "hz": float(hz or h),
            "n_src": n_src, "precision": precision, "near": near, "slots": slots, "n_sweeps": n_sweeps, "tol": tol,
            "surface": surface, "set_model": set_model}


def listed():
    return [
        # the first solve of a small survey, or one shot of an inversion on a coarse grid: the
        # package's default options, one source; launches and the wavefront's latency count
        _solve3("small_one_source", 64, 64, 32, 100.0, 1, n_sweeps=5),
        # the reference's own form of use: one source on the plain 3D configuration
        _solve3("plain_one_source", 256, 256, 128, 50.0, 1, near=True),
        # a shot gather: many sources on the plain 3D configuration, one batch
        _solve3("plain_64_sources", 256, 256, 128, 50.0, 64, near=True),
        # more sources than are kept in flight: a stream through slots
        _solve3("plain_stream", 256, 256, 128, 50.0, 128, near=True, slots=48),
        # station travel-time tables by reciprocity: a new model, then one field per surface station
        _solve3("station_tables", 200, 200, 100, 100.0, 64, near=True, surface=True, set_model=True),
        # a few sources in double precision, the precision of the reference's Solver3D
        _solve3("double_few_sources", 200, 200, 100, 100.0, 4, precision="f64", n_sweeps=5),
        # a vertical spacing finer than the horizontal one, odd extents
        _solve3("flat_cells", 151, 131, 87, 50.0, 8, hz=25.0, n_sweeps=5),
        # independent models of uneven size in one call (an ensemble), one source each
        {"name": "uneven_models", "kind": "models3d", "n_models": 32, "nxy_lo": 64, "nxy_hi": 256, "nz_lo": 32,
         "nz_hi": 128, "extents": 1, "h": 100.0, "near": True, "n_sweeps": 10, "tol": 1e-5},
        # the plain 2D configuration in double precision: one field and its gradient (ray tracing's input)
        {"name": "plain_2d", "kind": "solve2d", "nx": 501, "nz": 251, "h": 10.0, "hz": 10.0, "n_src": 1, "n_sweeps": 2,
         "tol": 1e-8, "gradient": True},
        # the same section for a line of sources
        {"name": "plain_2d_64_sources", "kind": "solve2d", "nx": 501, "nz": 251, "h": 10.0, "hz": 10.0, "n_src": 64,
         "n_sweeps": 2, "tol": 1e-8, "gradient": False},
        # the learned warm start's training: the gradient of one minibatch at its own grid
        {"name": "net_gradients", "kind": "net", "nx": 128, "ny": 128, "nz": 64, "h": 50.0, "batch": 8, "train": True},
        # and its use: predicted start fields for the sources of one shot gather
        {"name": "net_predict", "kind": "net", "nx": 128, "ny": 128, "nz": 64, "h": 50.0, "batch": 4, "train": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["one", "batch", "stream", "double", "flat", "models", "2d", "2d", "net"])
    nx, ny, nz = rng.randint(48, 256), rng.randint(48, 256), rng.randint(24, 128)
    h = rng.choice([25.0, 50.0, 100.0])
    if kind == "one":
        return _drop_name(_solve3("", nx, ny, nz, h, 1, near=rng.random() < 0.5, n_sweeps=rng.choice([5, 10])))
    if kind == "batch":
        return _drop_name(_solve3("", nx, ny, nz, h, _log(rng, 2, 64), near=rng.random() < 0.7,
                                  surface=rng.random() < 0.4, set_model=rng.random() < 0.4))
    if kind == "stream":
        n = _log(rng, 12, 128)
        return _drop_name(_solve3("", nx, ny, nz, h, n, near=rng.random() < 0.7, slots=max(2, n * 3 // 8)))
    if kind == "double":
        return _drop_name(_solve3("", min(nx, 200), min(ny, 200), min(nz, 100), h, rng.randint(1, 4),
                                  precision="f64", n_sweeps=5))
    if kind == "flat":
        return _drop_name(_solve3("", min(nx, 160), min(ny, 160), min(nz, 96), h, rng.randint(1, 8),
                                  hz=h * rng.choice([0.4, 0.5, 0.8]), n_sweeps=5))
    if kind == "models":
        return {"kind": "models3d", "n_models": rng.randint(2, 32), "nxy_lo": 48, "nxy_hi": rng.randint(96, 256),
                "nz_lo": 24, "nz_hi": rng.randint(48, 128), "extents": rng.randint(1, 1 << 20), "h": h,
                "near": rng.random() < 0.7, "n_sweeps": 10, "tol": 1e-5}
    if kind == "2d":
        one = rng.random() < 0.5
        return {"kind": "solve2d", "nx": _log(rng, 60, 600), "nz": _log(rng, 40, 300), "h": 10.0,
                "hz": rng.choice([10.0, 10.0, 12.5]), "n_src": 1 if one else _log(rng, 2, 64),
                "n_sweeps": rng.choice([2, 4]), "tol": 1e-8, "gradient": one}
    return {"kind": "net", "nx": rng.choice([32, 64, 96, 128]), "ny": 8 * rng.randint(4, 16), "nz": 8 * rng.randint(3, 8),
            "h": 50.0, "batch": rng.randint(1, 8), "train": rng.random() < 0.5}


def _drop_name(case):
    del case["name"]
    return case


# ---- inputs --------------------------------------------------------------------------------


def _smooth(shape, h, corr, gen):
    """A zero-mean random field of unit maximum with a Gaussian correlation length (metres)."""
    f = torch.fft.rfftn(torch.randn(shape, generator=gen, device=DEV, dtype=torch.float32))
    k2 = 0.0
    for axis, n in enumerate(shape):
        last = axis == len(shape) - 1
        k = (torch.fft.rfftfreq if last else torch.fft.fftfreq)(n, d=h, device=DEV) ** 2
        k2 = k2 + k.reshape([-1 if a == axis else 1 for a in range(len(shape))])
    p = torch.fft.irfftn(f * torch.exp(-(math.pi * corr) ** 2 * k2), s=shape)
    p = p - p.mean()
    return p / p.abs().max()


def _velocity(shape, h, seed):
    """Nodal velocities (m/s): 8 layers between 3000 and 7000 m/s increasing with depth, +-5 %."""
    rng = np.random.default_rng([seed, *shape])
    gen = torch.Generator(DEV).manual_seed(int(rng.integers(1 << 31)))
    layers = torch.tensor(np.sort(rng.uniform(3000.0, 7000.0, 8)), dtype=torch.float32, device=DEV)
    depth = torch.clamp(torch.arange(shape[0], device=DEV) * 8 // shape[0], max=7)
    v = layers[depth].reshape([-1] + [1] * (len(shape) - 1))
    return (v * (1.0 + 0.05 * _smooth(shape, h, 1000.0, gen))).contiguous()


def _sources(n, extents, seed, surface=False):
    rng = np.random.default_rng([seed, 77, n])
    p = rng.uniform(0.0, 1.0, (n, len(extents))) * np.asarray(extents)
    if surface:
        p[:, -1] = 0.0
    return p


def _extents(case):
    rng = np.random.default_rng(case["extents"])
    return [(*(int(q) for q in rng.integers(case["nxy_lo"], case["nxy_hi"] + 1, 2)),
             int(rng.integers(case["nz_lo"], case["nz_hi"] + 1))) for _ in range(case["n_models"])]


def _models(case, seed):
    rng = np.random.default_rng([seed, 5])
    out = []
    h = case["h"]
    for nx, ny, nz in _extents(case):
        s = int(rng.integers(1 << 30))
        out.append({"grid": (nx, ny, nz, h, h, h), "model": _velocity((nz, ny, nx), h, s), "nodal": True,
                    "sources": _sources(1, [(n - 1) * h for n in (nx, ny, nz)], s),
                    "out": torch.empty((1, nz, ny, nx), dtype=torch.float32, device=DEV)})
    return out


def _net_inputs(case, seed):
    """Samples of smooth models with travel times near those of straight rays, and trained-scale weights."""
    nx, ny, nz, h = case["nx"], case["ny"], case["nz"], case["h"]
    rng = np.random.default_rng([seed, 9])
    gen = torch.Generator(DEV).manual_seed(int(rng.integers(1 << 31)))
    z, y, x = torch.meshgrid(*[torch.arange(n, device=DEV, dtype=torch.float64) * h for n in (nz, ny, nx)],
                             indexing="ij")
    samples = []
    for src in _sources(case["batch"], [(n - 1) * h for n in (nx, ny, nz)], seed):
        mean, amp = rng.uniform(2500.0, 6000.0), rng.uniform(0.1, 0.5)
        v = (mean * (1.0 + amp * _smooth((nz, ny, nx), h, rng.uniform(500.0, 3000.0), gen))).clamp(1500.0, 8000.0)
        dist = torch.sqrt((x - src[0]) ** 2 + (y - src[1]) ** 2 + (z - src[2]) ** 2)
        at_src = v[tuple(int(round(float(c) / h)) for c in src[::-1])]
        t = (dist * 0.5 * (1.0 / v.double() + 1.0 / at_src.double())).float()
        samples.append((v.reshape(-1).contiguous(), t.reshape(-1).contiguous(), tuple(float(c) for c in src)))
    p = []
    for cin, cout, _ in _LAYERS:
        fan = 27 * (6 if not p else cin)
        p += [rng.standard_normal(27 * cin * cout) * math.sqrt(2.0 / fan), 0.05 * rng.standard_normal(cout)]
    p.append(0.1 * rng.standard_normal(17))
    return samples, np.concatenate(p).astype(np.float32)


def _options(case):
    return ex.Options(n_sweeps=case["n_sweeps"], tolerance=case["tol"], factored_radius=3,
                      near_fp64=case.get("near", False), max_in_flight=case.get("slots", 0))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "net":
        samples, params = _net_inputs(case, seed)
        nx, ny, nz, h = case["nx"], case["ny"], case["nz"], case["h"]
        net = WarmNet((nx, ny, nz, h, h, h), case["batch"])
        net.set_params(params)
        out = torch.empty((case["batch"], nz, ny, nx), dtype=torch.float32, device=DEV)
        torch.cuda.synchronize()
        return {"case": case, "net": net, "samples": samples, "out": out}
    ctx = ex.Context(0)
    state = {"case": case, "ctx": ctx, "opt": _options(case)}
    if kind == "models3d":
        state["models"] = _models(case, seed)
        torch.cuda.synchronize()
        return state
    nx, nz, h, hz = case["nx"], case["nz"], case["h"], case["hz"]
    if kind == "solve3d":
        ny = case["ny"]
        state["v"] = _velocity((nz, ny, nx), h, seed)
        state["src"] = _sources(case["n_src"], [(nx - 1) * h, (ny - 1) * h, (nz - 1) * hz], seed, case["surface"])
        state["precision"] = ex.F64 if case["precision"] == "f64" else ex.F32
        dt = torch.float64 if case["precision"] == "f64" else torch.float32
        state["out"] = torch.empty((case["n_src"], nz, ny, nx), dtype=dt, device=DEV)
        torch.cuda.synchronize()
        ctx.set_grid3d(nx, ny, nz, h, h, hz)
        ctx.set_nodal_velocity3d(state["v"])
    else:
        state["v"] = _velocity((nz, nx), h, seed).double()
        state["src"] = _sources(case["n_src"], [(nx - 1) * h, (nz - 1) * hz], seed)
        state["out"] = torch.empty((case["n_src"], nz, nx), dtype=torch.float64, device=DEV)
        state["grad"] = torch.empty((nz, nx, 2), dtype=torch.float64, device=DEV)
        torch.cuda.synchronize()
        ctx.set_grid2d(nx, nz, h, hz)
        ctx.set_nodal_velocity2d(state["v"])
    return state


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "net":
        if case["train"]:
            grad, loss = state["net"].gradients(state["samples"])
            return {"grad": grad, "loss": loss}
        t, loss = state["net"].predict(state["samples"], inflate=1.02, out=state["out"])
        return {"t": t, "loss": loss}
    ctx = state["ctx"]
    if kind == "models3d":
        return ctx.solve3d_batch(state["models"], state["opt"], ex.F32)
    if kind == "solve3d":
        if case["set_model"]:
            ctx.set_nodal_velocity3d(state["v"])
        return ctx.solve3d(state["src"], state["opt"], state["precision"], out=state["out"])
    t = ctx.solve2d(state["src"], state["opt"], ex.F64, out=state["out"])
    return [t, ctx.gradient2d(0, ex.F64, out=state["grad"])] if case["gradient"] else [t]


def work(case):
    """A solve: the model read and the fields written; each node is visited once by the
    initialisation pass and once by each ordering of at least one iteration, about 60 operations
    a visit in 3D and 25 in 2D.  The network: velocities in, travel times in or out, the parameters
    (and their gradient); the convolutions' multiplications and additions."""
    kind = case["kind"]
    if kind == "net":
        nodes = case["nx"] * case["ny"] * case["nz"] * case["batch"]
        flops = sum(2 * 27 * ci * co * nodes / 8 ** lv for ci, co, lv in _LAYERS)
        params = sum(27 * ci * co + co for ci, co, _ in _LAYERS) + 17
        return {"bytes": 8 * nodes + (8 if case["train"] else 4) * params,
                "flops": int(flops) * (3 if case["train"] else 1)}
    if kind == "models3d":
        nodes = sum(nx * ny * nz for nx, ny, nz in _extents(case))
        return {"bytes": 8 * nodes, "flops": 9 * 60 * nodes}
    if kind == "solve2d":
        nodes = case["nx"] * case["nz"]
        out = nodes * case["n_src"]
        return {"bytes": 8 * (nodes + out + (2 * nodes if case["gradient"] else 0)), "flops": 5 * 25 * out}
    nodes = case["nx"] * case["ny"] * case["nz"]
    size = 8 if case["precision"] == "f64" else 4
    return {"bytes": size * nodes * (1 + case["n_src"]), "flops": 9 * 60 * nodes * case["n_src"]}


# ---- plain 64-bit values -------------------------------------------------------------------


def _levels(shape, low):
    """Flat indices of the nodes at or beyond `low` along every axis, one array per wavefront."""
    ax = [np.arange(lo, n) for lo, n in zip(low, shape)]
    if any(len(a) == 0 for a in ax):
        return []
    flat, level = 0, 0
    for a, n, k in zip(ax, shape, range(len(shape))):
        dims = [1] * len(shape)
        dims[k] = -1
        flat = flat * n + a.reshape(dims)
        level = level + a.reshape(dims)
    flat, level = np.broadcast_arrays(flat, level)
    order = np.argsort(level, axis=None, kind="stable")
    edges = np.searchsorted(level.ravel()[order], np.arange(level.min(), level.max() + 2))
    flat = flat.ravel()[order]
    return [flat[a:b] for a, b in zip(edges[:-1], edges[1:])]


def _sweeps(shape, spacing, cells, src, n_sweeps, tol, update):
    """Fast sweeping of one source: the source cell's corners, one pass limited to each octant
    (quadrant) of the source, then refinement iterations until a whole round of orderings
    lowers no node by tol.  Axes are (z, y, x) or (z, x); ordering bit 0 reverses x."""
    dim = len(shape)
    kinds = 1 << dim
    off = np.asarray(src, np.float64)[::-1]
    cell = [min(n - 2, int(o / d)) for o, d, n in zip(off, spacing, shape)]
    t = np.full(shape, 1e10)
    s_src = cells[tuple(cell)]
    for c in np.ndindex(*[2] * dim):
        node = [a + b for a, b in zip(cell, c)]
        t[tuple(node)] = s_src * math.sqrt(sum((k * d - o) ** 2 for k, d, o in zip(node, spacing, off)))
    strides = [int(np.prod(shape[k + 1:])) for k in range(dim)]
    full = _levels(shape, [1] * dim)
    quiet = 0
    for k in range(kinds * (1 + n_sweeps)):
        init, e = k < kinds, k % kinds
        rev = [(e >> (dim - 1 - a)) & 1 for a in range(dim)]
        flip = tuple(slice(None, None, -1 if r else 1) for r in rev)
        w = np.ascontiguousarray(t[flip])
        tw = w.reshape(-1)
        pad = np.pad(cells[flip], 1, mode="edge")
        lists = full
        if init:
            low = [n - 1 - min(c + 1, n - 2) if r else max(1, c) for c, r, n in zip(cell, rev, shape)]
            lists = _levels(shape, low)
        most = 0.0
        for idx in lists:
            at = np.unravel_index(idx, shape)
            real = [n - 1 - a if r else a for a, r, n in zip(at, rev, shape)]
            near = np.all([np.abs(a - c) <= 3 for a, c in zip(real, cell)], axis=0)
            new = update(tw, idx, strides, pad, at, real, rev, off, s_src, near)
            old = tw[idx]
            lower = new < old
            if lower.any():
                most = max(most, float((old - new)[lower].max()))
                tw[idx] = np.where(lower, new, old)
        t = np.ascontiguousarray(w[flip])
        if not init:
            quiet = quiet + 1 if most < tol else 0
            if quiet >= kinds:
                break
    return t


def _root(a):
    return np.sqrt(np.maximum(a, 0.0))


def _factor(real, rev, spacing, off, slow, ups):
    """T0 = slow * distance at the node and at the given upwind neighbours, and its gradient
    along the walk."""
    step = [1 if r else -1 for r in rev]

    def dist(up):
        d = [(r + u * s) * h - o for r, u, s, h, o in zip(real, up, step, spacing, off)]
        return d, np.sqrt(sum(q * q for q in d))

    d, r0 = dist([0] * len(real))
    grad = [-s * slow * np.divide(q, r0, out=np.zeros_like(r0), where=r0 > 0) for q, s in zip(d, step)]
    return slow * r0, grad, [slow * dist(u)[1] for u in ups]


def _quadratic(a, b, c, t0, ok, floors):
    det = b * b - 4 * a * c
    t = t0 + (-b + _root(det)) / (2 * a)
    for f in floors:
        ok = ok & ~(t < f)
    return np.where(ok & (det >= 0), t, 1e10)


def _update3(spacing):
    hz, hy, hx = spacing
    inv = {"x": 1 / hx, "y": 1 / hy, "z": 1 / hz}
    inv2 = {k: v * v for k, v in inv.items()}
    same = hx == hy == hz

    def inside(ta, tb, a, b):
        return (ta <= tb + b) & (tb <= ta + a) if same else (ta < tb + b) & (tb < ta + a)

    def update(tw, idx, strides, pad, at, real, rev, off, s_src, near):
        sz, sy, sx = strides
        t1, t2, t3, t4 = tw[idx - sx], tw[idx - sx - sy], tw[idx - sy], tw[idx - sz]
        t5, t6, t7 = tw[idx - sx - sz], tw[idx - sx - sy - sz], tw[idx - sy - sz]
        z, y, x = at
        s0, s1, s2, s3 = pad[z, y, x], pad[z, y, x + 1], pad[z, y + 1, x + 1], pad[z, y + 1, x]
        s4, s5, s7 = pad[z + 1, y, x], pad[z + 1, y, x + 1], pad[z + 1, y + 1, x]
        m03, m01, m04 = np.minimum(s0, s3), np.minimum(s0, s1), np.minimum(s0, s4)
        t1d = np.minimum(np.minimum(t1 + hx * np.minimum(m03, np.minimum(s4, s7)),
                                    t3 + hy * np.minimum(m04, np.minimum(s1, s5))),
                         t4 + hz * np.minimum(m01, np.minimum(s2, s3)))
        t2d = np.full_like(t1d, 1e10)
        planes = [("x", "z", hx, hz, t1, t4, t5, m03), ("y", "z", hy, hz, t3, t4, t7, m01),
                  ("x", "y", hx, hy, t1, t3, t2, m04)]
        for _, _, ha, hb, ta, tb, td, m in planes:
            det = (ha * ha + hb * hb) * m * m - (ta - tb) ** 2
            v = ((ta - tb + td) * hb / ha + (tb - ta + td) * ha / hb + 2 * _root(det)) * ha * hb / (ha * ha + hb * hb)
            t2d = np.minimum(t2d, np.where((det > 0) & inside(ta, tb, ha * m, hb * m), v, 1e10))
        half = 0.5
        vx = t1 + half * (-t4 + t5 - t3 + t2) - t7 + t6
        vy = t3 + half * (-t4 + t7 - t1 + t2) - t5 + t6
        vz = t4 + half * (-t1 + t5 - t3 + t7) - t2 + t6
        ix, iy, iz = inv2["x"], inv2["y"], inv2["z"]
        det = 9 * s0 * s0 * (ix + iy + iz) - (vx - vz) ** 2 * ix * iz - (vy - vz) ** 2 * iy * iz - \
            (vx - vy) ** 2 * ix * iy
        open3 = np.minimum(t1d, t2d) > np.maximum(np.maximum(t1, t4), t3)
        v = (vx * ix + vy * iy + vz * iz + _root(det)) / (ix + iy + iz)
        out = np.minimum(t1d, np.minimum(t2d, np.where(open3 & (det >= 0), v, 1e10)))
        if not near.any():
            return out
        n = np.nonzero(near)[0]
        ups = [(0, 0, 1), (0, 1, 1), (0, 1, 0), (1, 0, 0), (1, 0, 1), (1, 1, 1), (1, 1, 0)]
        sl = s0[n]
        t0, grad, t0s = _factor([r[n] for r in real], rev, spacing, off, sl, ups)
        gz, gy, gx = grad
        ta = [t[n] - a for t, a in zip((t1, t2, t3, t4, t5, t6, t7), t0s)]
        u1, u2, u3, u4, u5, u6, u7 = ta
        excess = s_src * s_src - sl * sl
        t1n, t3n, t4n, d1 = t1[n], t3[n], t4[n], t1d[n]
        best = np.full_like(d1, 1e10)
        for a, b, ha, hb, ua, ub, ud, ga, gb, gc, m, fa, fb in (
                ("x", "z", hx, hz, u1, u4, u5, gx, gz, gy, m03[n], t1n, t4n),
                ("y", "z", hy, hz, u3, u4, u7, gy, gz, gx, m01[n], t3n, t4n),
                ("x", "y", hx, hy, u1, u3, u2, gx, gy, gz, m04[n], t1n, t3n)):
            p, q = ua - ub + ud, ub - ua + ud
            qa = inv2[a] + inv2[b]
            qb = 4 * (inv[a] * ga + inv[b] * gb) - 2 * (p * inv2[a] + q * inv2[b])
            qc = p * p * inv2[a] + q * q * inv2[b] - 4 * (ga * p * inv[a] + gb * q * inv[b]) + 4 * (excess + gc * gc)
            best = np.minimum(best, _quadratic(qa, qb, qc, t0, inside(fa, fb, ha * m, hb * m), (fa, fb)))
        wx = u1 + half * (-u4 + u5 - u3 + u2) - u7 + u6
        wy = u3 + half * (-u4 + u7 - u1 + u2) - u5 + u6
        wz = u4 + half * (-u1 + u5 - u3 + u7) - u2 + u6
        qb = -2 * (wx * ix + wy * iy + wz * iz) + 6 * (inv["x"] * gx + inv["y"] * gy + inv["z"] * gz)
        qc = wx * wx * ix + wy * wy * iy + wz * wz * iz - \
            6 * (gx * wx * inv["x"] + gy * wy * inv["y"] + gz * wz * inv["z"]) + 9 * excess
        ok = np.minimum(d1, best) > np.maximum(np.maximum(t1n, t4n), t3n)
        t3d = _quadratic(ix + iy + iz, qb, qc, t0, ok, (t1n, t3n, t4n))
        out[n] = np.minimum(d1, np.minimum(best, t3d))
        return out

    return update


def _update2(spacing):
    hz, hx = spacing
    same = hx == hz
    diag = math.hypot(hx, hz)

    def update(tw, idx, strides, pad, at, real, rev, off, s_src, near):
        sz, sx = strides
        t1, t2, t3 = tw[idx - sx], tw[idx - sx - sz], tw[idx - sz]
        z, x = at
        s0, s1, s3 = pad[z, x], pad[z, x + 1], pad[z + 1, x]
        one = np.minimum(t1 + hx * np.minimum(s0, s3), t3 + hz * np.minimum(s0, s1))
        dx, dz = t3 - t2, t1 - t2
        a, b = (hz * s0) ** 2 - dz * dz, (hx * s0) ** 2 - dx * dx
        ta = np.where((dz >= 0) & (a >= 0) & (dz <= hz * hz / diag * s0), t1 + hx / hz * _root(a), 1e10)
        tb = np.where((dx >= 0) & (b >= 0) & (dx <= hx * hx / diag * s0), t3 + hz / hx * _root(b), 1e10)
        det = (hx * hx + hz * hz) * s0 * s0 - (t1 - t3) ** 2
        wave = (dx >= 0) & (dz >= 0)
        wave &= ((t3 <= t1 + hx * s0) & (t1 <= t3 + hz * s0)) if same else ((t1 < t3 + hz * s0) & (t3 < t1 + hx * s0))
        v = ((t1 - t3 + t2) * hz / hx + (t3 - t1 + t2) * hx / hz + 2 * _root(det)) * hx * hz / (diag * diag)
        out = np.minimum(np.minimum(one, np.minimum(ta, tb)), np.where(wave & (det > 0) & ~(v < 0), v, 1e10))
        if not near.any():
            return out
        n = np.nonzero(near)[0]
        t0, (gz, gx), t0s = _factor([r[n] for r in real], rev, spacing, off, s_src, [(0, 1), (1, 1), (1, 0)])
        u1, u2, u3 = (t[n] - q for t, q in zip((t1, t2, t3), t0s))
        p, q = u1 - u3 + u2, u3 - u1 + u2
        ix, iz = 1 / (hx * hx), 1 / (hz * hz)
        qb = 4 * (gx / hx + gz / hz) - 2 * (p * ix + q * iz)
        qc = p * p * ix + q * q * iz - 4 * (gx * p / hx + gz * q / hz) + 4 * (s_src * s_src - s0[n] ** 2)
        ok = ((dx >= 0) & (dz >= 0) & (t1 < t3 + hz * s0) & (t3 < t1 + hx * s0))[n]
        out[n] = np.minimum(one[n], _quadratic(ix + iz, qb, qc, t0, ok, (t1[n], t3[n])))
        return out

    return update


def _gradient2(t, cells, spacing, src):
    hz, hx = spacing
    g = np.empty(t.shape + (2,))
    for k, (axis, h) in enumerate(((1, hx), (0, hz))):
        u = np.moveaxis(t, axis, 0)
        d = np.moveaxis(g[..., k], axis, 0)
        d[1:-1] = (u[2:] - u[:-2]) / (2 * h)
        d[0] = (-3 * u[0] + 4 * u[1] - u[2]) / (2 * h)
        d[-1] = (u[-3] - 4 * u[-2] + 3 * u[-1]) / (2 * h)
    nz, nx = t.shape
    cx, cz = min(nx - 2, int(src[0] / hx)), min(nz - 2, int(src[1] / hz))
    for j in (0, 1):
        for i in (0, 1):
            a, b = (cx + i) * hx - src[0], (cz + j) * hz - src[1]
            r = math.hypot(a, b)
            if abs(cx * hx - src[0]) > 1e-7:
                g[cz + j, cx + i, 0] = a / r * cells[cz, cx]
            if abs(cz * hz - src[1]) > 1e-7:
                g[cz + j, cx + i, 1] = b / r * cells[cz, cx]
    return g


def _cells(v):
    v = v.double().cpu().numpy()
    for axis in range(v.ndim):
        lo, hi = [slice(None)] * v.ndim, [slice(None)] * v.ndim
        lo[axis], hi[axis] = slice(None, -1), slice(1, None)
        v = 0.5 * (v[tuple(lo)] + v[tuple(hi)])
    return 1.0 / v


# (input channels, output channels, level) of the network's convolutions, in order
_LAYERS = [(16, 16, 0), (16, 16, 0), (16, 32, 1), (32, 32, 1), (32, 64, 2), (64, 64, 2), (64, 128, 3), (128, 128, 3),
           (192, 64, 2), (64, 64, 2), (96, 32, 1), (32, 32, 1), (48, 16, 0), (16, 16, 0)]


def _net_exact(case, seed):
    """The network in float64 torch: features, a U-Net of ReLU convolutions with average pooling
    and nearest upsampling, a linear head, the mean squared error of tau - 1."""
    F = torch.nn.functional
    samples, params = _net_inputs(case, seed)
    nx, ny, nz, h = case["nx"], case["ny"], case["nz"], case["h"]
    p = torch.tensor(params, dtype=torch.float64, device=DEV, requires_grad=case["train"])
    dims = torch.tensor([nx, ny, nz], device=DEV, dtype=torch.float64)
    z, y, x = torch.meshgrid(*[torch.arange(n, device=DEV, dtype=torch.float64) for n in (nz, ny, nx)], indexing="ij")
    node = torch.stack([x, y, z], -1)
    length = float(torch.sqrt((((dims - 1) * h) ** 2).sum()))
    total = None
    count = 0
    preds, losses = [], 0.0
    t0s, tgts = [], []
    for v, t, src in samples:
        s = 1.0 / v.double().reshape(nz, ny, nx)
        pos = torch.tensor(src, device=DEV, dtype=torch.float64) / h
        i = [int(min(n - 1, max(0, round(float(c))))) for c, n in zip(pos, (nx, ny, nz))]
        s_src = s[i[2], i[1], i[0]]
        d = (node - pos) * h
        dist = torch.sqrt((d * d).sum(-1))
        ray = 0.0
        for k in range(32):
            q = pos + (k + 0.5) / 32 * (node - pos)
            g = (2.0 * q / (dims - 1) - 1.0)[None]
            ray = ray + F.grid_sample(s[None, None], g, mode="bilinear", padding_mode="border", align_corners=True)[0, 0]
        feat = torch.zeros((16, nz, ny, nx), dtype=torch.float64, device=DEV)
        feat[0] = s / s_src - 1
        feat[1] = dist / length
        feat[2:5] = d.permute(3, 0, 1, 2) / length
        feat[5] = ray / 32 / s_src - 1
        t0s.append(s_src * dist)
        tgts.append(t.double().reshape(nz, ny, nx))
        count += int((t0s[-1] > 0).sum())
        preds.append(feat)
    grads = None
    outs = []
    for feat, t0, tgt in zip(preds, t0s, tgts):
        off = 0
        ws = []
        for cin, cout, _ in _LAYERS:
            w = p[off:off + 27 * cin * cout].reshape(3, 3, 3, cout, cin).permute(3, 4, 0, 1, 2)
            off += 27 * cin * cout
            ws.append((w, p[off:off + cout]))
            off += cout

        def conv(k, a):
            return torch.relu(F.conv3d(a, ws[k][0], ws[k][1], padding=1))

        def up(a):
            return F.interpolate(a, scale_factor=2, mode="nearest")

        e0 = conv(1, conv(0, feat[None]))
        e1 = conv(3, conv(2, F.avg_pool3d(e0, 2)))
        e2 = conv(5, conv(4, F.avg_pool3d(e1, 2)))
        b = conv(7, conv(6, F.avg_pool3d(e2, 2)))
        d2 = conv(9, conv(8, torch.cat([up(b), e2], 1)))
        d1 = conv(11, conv(10, torch.cat([up(d2), e1], 1)))
        d0 = conv(13, conv(12, torch.cat([up(d1), e0], 1)))
        o = (d0[0] * p[off:off + 16].reshape(16, 1, 1, 1)).sum(0) + p[off + 16]
        ok = t0 > 0
        diff = torch.where(ok, o - (tgt / torch.where(ok, t0, torch.ones_like(t0)) - 1), torch.zeros_like(o))
        loss = (diff * diff).sum() / count
        if case["train"]:
            g = torch.autograd.grad(loss, p)[0]
            grads = g if grads is None else grads + g
        losses += float(loss.detach())
        outs.append((t0 * (1 + o) * 1.02).detach())
    if case["train"]:
        return {"grad": grads.cpu().numpy(), "loss": losses}
    return {"t": torch.stack(outs), "loss": losses}


def exact(case, seed):
    kind = case["kind"]
    if kind == "models3d":
        return None
    if kind == "net":
        return _net_exact(case, seed)
    nx, nz, h, hz = case["nx"], case["nz"], case["h"], case["hz"]
    shape = (nz, case["ny"], nx) if kind == "solve3d" else (nz, nx)
    ops = 140 if kind == "solve3d" else 60
    rounds = (1 + case["n_sweeps"]) * (8 if kind == "solve3d" else 4)
    cost = case["n_src"] * rounds * ops * (2e-6 * sum(shape) + 2.5e-9 * math.prod(shape))
    if cost > 15.0:
        return None
    spacing = (hz, h, h) if kind == "solve3d" else (hz, h)
    extents = [(n - 1) * d for n, d in zip(shape[::-1], spacing[::-1])]
    src = _sources(case["n_src"], extents, seed, case.get("surface", False))
    v = _velocity(shape, h, seed)
    cells = _cells(v if kind == "solve3d" else v.double())
    update = (_update3 if kind == "solve3d" else _update2)(spacing)
    t = np.stack([_sweeps(shape, spacing, cells, p, case["n_sweeps"], case["tol"], update) for p in src])
    if kind == "solve3d":
        return t
    return [t, _gradient2(t[0], cells, spacing, src[0])] if case["gradient"] else [t]
