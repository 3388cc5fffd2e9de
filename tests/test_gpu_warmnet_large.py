"""The network against plain torch convolutions in FP64 on the device, at sizes where its kernels
run in their steady state (each block of the row-ring convolution walks several segments and reuses
its accumulators; each block of the weight gradient loops over several tiles, unevenly) and at
extents beyond 65535, which a launch grid's y and z do not hold.

The bounds are those of the small-grid tests: as close to FP64 as twice the distance of BF16
storage, which the reference repeats by rounding where the library stores BF16."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from eikonalxx_gb300 import warmstart as ws  # noqa: E402
from oracle import warmnet_oracle as wo  # noqa: E402

H = 50.0


class _Round(torch.autograd.Function):
    """BF16 storage of a value and of its gradient."""

    @staticmethod
    def forward(ctx, x):
        return x.float().bfloat16().double()

    @staticmethod
    def backward(ctx, g):
        return g.float().bfloat16().double()


def _features(v, src, grid):
    nx, ny, nz = grid
    s = 1.0 / v.double().reshape(nz, ny, nx)
    dims = torch.tensor([nx, ny, nz], device="cuda", dtype=torch.float64)
    pos = torch.tensor(src, device="cuda", dtype=torch.float64) / H
    z, y, x = torch.meshgrid(*[torch.arange(n, device="cuda", dtype=torch.float64) for n in (nz, ny, nx)], indexing="ij")
    node = torch.stack([x, y, z], -1)
    i = [int(min(n - 1, max(0, round(float(c))))) for c, n in zip(pos, grid)]
    s_src = s[i[2], i[1], i[0]]
    d = (node - pos) * H
    dist = torch.sqrt((d * d).sum(-1))
    ray = torch.zeros_like(s)
    for k in range(32):
        q = pos + (k + 0.5) / 32 * (node - pos)
        cell = torch.minimum(q.floor(), dims - 2).clamp_(min=0)
        f = q - cell
        c = cell.long()
        at = (c[..., 2] * ny + c[..., 1]) * nx + c[..., 0]
        flat = s.reshape(-1)
        g = [flat[at + (o & 1) + ((o >> 1) & 1) * nx + (o >> 2) * nx * ny] for o in range(8)]
        g = [g[o] + f[..., 0] * (g[o + 1] - g[o]) for o in (0, 2, 4, 6)]
        g = [g[o] + f[..., 1] * (g[o + 1] - g[o]) for o in (0, 2)]
        ray += g[0] + f[..., 2] * (g[1] - g[0])
    length = float(torch.sqrt((((dims - 1) * H) ** 2).sum()))
    feat = torch.zeros((16, nz, ny, nx), dtype=torch.float64, device="cuda")
    feat[0] = s / s_src - 1
    feat[1] = dist / length
    feat[2:5] = d.permute(3, 0, 1, 2) / length
    feat[5] = ray / 32 / s_src - 1
    return feat, s_src * dist


def _reference(params, samples, grid, emulate, centre_only):
    """(predicted times, T0, parameter gradient of the mean loss) in FP64."""
    F = torch.nn.functional
    rnd = _Round.apply if emulate else (lambda a: a)
    nx, ny, nz = grid
    p = torch.tensor(params, dtype=torch.float64, device="cuda", requires_grad=True)
    layers, head, _ = wo.layout()
    count = len(samples) * nx * ny * nz
    grad = torch.zeros_like(p)
    times, t0s = [], []
    for v, t, src in samples:
        feat, t0 = _features(v, src, grid)
        pr = p + (p.detach().float().bfloat16().double() - p.detach()) if emulate else p   # the weights as stored

        def conv(k, a):
            (cin, cout, _), (w, b) = wo.SPEC[k], layers[k]
            wt = pr[w:w + 27 * cin * cout].reshape(3, 3, 3, cout, cin).permute(3, 4, 0, 1, 2)
            if centre_only:
                a = F.conv3d(a, wt[:, :, 1:2, 1:2, 1:2], p[b:b + cout])
            else:
                a = F.conv3d(a, wt, p[b:b + cout], padding=1)
            return rnd(torch.relu(a))

        def up(a):
            return F.interpolate(a, scale_factor=2, mode="nearest")

        def pool(a):
            return rnd(F.avg_pool3d(a, 2))

        e0 = conv(1, conv(0, rnd(feat[None])))
        e1 = conv(3, conv(2, pool(e0)))
        e2 = conv(5, conv(4, pool(e1)))
        b = conv(7, conv(6, pool(e2)))
        d2 = conv(9, conv(8, torch.cat([up(b), e2], 1)))
        d1 = conv(11, conv(10, torch.cat([up(d2), e1], 1)))
        d0 = conv(13, conv(12, torch.cat([up(d1), e0], 1)))
        o = (d0[0] * p[head:head + 16].reshape(16, 1, 1, 1)).sum(0) + p[head + 16]
        ok = t0 > 0
        diff = torch.where(ok, o - (t.double().reshape(nz, ny, nx) / torch.where(ok, t0, torch.ones_like(t0)) - 1),
                           torch.zeros_like(o))
        grad += torch.autograd.grad((diff * diff).sum() / count, p)[0]
        times.append((t0 * (1 + o)).detach())
        t0s.append(t0)
    return torch.stack(times).cpu().numpy(), torch.stack(t0s).cpu().numpy(), grad.cpu().numpy()


def _case(grid, n, centre_only, seed):
    nx, ny, nz = grid
    rng = np.random.default_rng(seed)
    gen = torch.Generator("cuda").manual_seed(seed)
    samples = []
    for _ in range(n):
        v = 3000 + 300 * torch.randn((nz, ny, nx), generator=gen, device="cuda", dtype=torch.float32).clamp(-3, 3)
        # off the nodes by at least 0.2 cells: no node has T0 = 0
        src = tuple((rng.integers(0, m - 1) + rng.uniform(0.2, 0.8)) * H for m in grid)
        z, y, x = torch.meshgrid(*[torch.arange(m, device="cuda") * H for m in (nz, ny, nx)], indexing="ij")
        r = torch.sqrt((x - src[0]) ** 2 + (y - src[1]) ** 2 + (z - src[2]) ** 2)
        t = (r / 3000 * (1 + 0.2 * torch.sin(0.25 * x / H + 0.1 * z / H))).float()
        samples.append((v.reshape(-1).contiguous(), t.reshape(-1).contiguous(), src))
    p = np.zeros(wo.layout()[2], np.float32)
    layers, head, _ = wo.layout()
    for (cin, cout, _), (w, b) in zip(wo.SPEC, layers):
        wt = np.zeros((27, cout, cin), np.float32)
        taps = [13] if centre_only else list(range(27))
        wt[taps] = rng.standard_normal((len(taps), cout, cin)) * np.sqrt(2.0 / (len(taps) * cin))
        p[w:w + wt.size] = wt.ravel()
        p[b:b + cout] = rng.normal(0, 0.05, cout)
    p[head:head + 17] = rng.normal(0, 0.3, 17)
    return samples, p


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


# 294 segments of 12 tiles (the last of 8) for the blocks of 152 SMs; 65544 planes; 131088 rows
CASES = [((128, 56, 80), 3, False), ((8, 8, 65544), 1, True), ((8, 131088, 8), 1, True)]


@pytest.mark.parametrize("grid,n,centre_only", CASES)
def test_network_matches_torch_in_fp64(grid, n, centre_only):
    samples, p = _case(grid, n, centre_only, 33)
    with ws.WarmNet(grid + (H, H, H, 0.0, 0.0, 0.0), batch=n, seed=0) as net:
        net.set_params(p)
        g, _ = net.gradients(samples)
        t, _ = net.predict(samples, inflate=1.0)
    te, t0, ge = _reference(p, samples, grid, False, centre_only)
    tb, _, gb = _reference(p, samples, grid, True, centre_only)
    assert _rel(t, te) <= 2 * _rel(tb, te)
    # a wrong tile (four x-rows) is off by the order of the output itself; rounding alone leaves the
    # worst of them within a small multiple of the emulation's worst
    tiles = lambda a: np.sqrt((((a - te) / t0) ** 2).reshape(n, grid[2], grid[1] // 4, -1).mean(axis=3))
    assert tiles(t).max() <= 4 * tiles(tb).max()
    layers, head, _ = wo.layout()
    bad = []
    for L, ((cin, cout, _), (w, b)) in enumerate(zip(wo.SPEC, layers)):
        for name, sl in ((wo.NAMES[L], slice(w, w + 27 * cin * cout)), (wo.NAMES[L] + ".b", slice(b, b + cout))):
            a, e, m = g[sl], ge[sl], gb[sl]
            if centre_only and not name.endswith(".b"):
                a, e, m = (q.reshape(27, cout, cin)[13] for q in (a, e, m))
            if not _rel(a, e) < max(2e-2, 2 * _rel(m, e)):
                bad.append((name, _rel(a, e), _rel(m, e)))
    assert not bad, bad
    assert _rel(g[head:], ge[head:]) < max(2e-2, 2 * _rel(gb[head:], ge[head:]))
