"""Performance cases: the calls a user of the package makes, from the smallest particle sets to the largest.

Kinds of case:

* ``hot``      Meshoid(pos, m, des_ngb) and D(f): the neighbour search, smoothing lengths, densities and first
               derivatives of one snapshot, with a column density map or the neighbour lists where a case asks for them.
* ``grad``     D(f) of many fields on a Meshoid that the program keeps.
* ``order2``   D2(f) and D(f, order=2) after reset_dweights(): the second-derivative fit of a kept neighbour set.
* ``map``      SurfaceDensity on a snapshot that carries its own smoothing lengths.
* ``deposit``  DepositToGrid on such a snapshot.
* ``slice``    two Slice calls at different heights on a kept Meshoid: nearest particles, a masked search, derivatives.
* ``batch``    SnapshotBatch.run(): many uneven snapshots, one call.

Positions, masses and fields are FP64 tensors on the GPU, made from the seed.
"""
import math

import numpy as np
import torch

import meshoid_gb300
from meshoid_gb300.batch import SnapshotBatch

VOLNORM = {1: 2.0, 2: math.pi, 3: 4.0 * math.pi / 3.0}
HNORM = {1: 8.0 / 3.0, 2: 40.0 / 7.0, 3: 32.0 / 3.0}
BRUTE = 1.1e11  # query-particle pairs that exact() may visit


def listed():
    return [
        # the smallest: a test-sized set, called in a loop or by hand; launches and host work count
        _hot("hot_plummer_1536", 1536, "plummer", fields=1, ngb=True),
        # the reference's own CPU-sized workload: uniform points, one field, a 256^2 map
        _hot("hot_uniform_65536", 65536, "uniform", fields=1, res=256),
        # an ordinary snapshot of no round size, with the trained first guess of h
        _hot("hot_plummer_1000003_learned", 1000003, "plummer", fields=4, guess="learned"),
        # the headline: a Plummer sphere of 2^22, five components
        _hot("hot_plummer_2e22", 1 << 22, "plummer", fields=5),
        # the largest: 2^24 particles of a clump mixture, 16 scalar fields and a vector
        _hot("hot_clumps_2e24", 1 << 24, "clumps", fields=19),
        # a clumpy periodic box with 64 neighbours and the neighbour lists read back
        _hot("box_262147_k64", 262147, "boxclumps", fields=3, k=64, box=1.0, ngb=True),
        # sixteen fields differentiated on a kept neighbour set
        {"name": "grad_1000003_f16", "kind": "grad", "n": 1000003, "dist": "plummer", "k": 32, "fields": 16},
        # second derivatives of a field, with the fit's matrices
        {"name": "order2_131071_k64", "kind": "order2", "n": 131071, "dist": "plummer", "k": 64, "fields": 2},
        # a 1024^2 column density map
        {"name": "map_2e20_r1024", "kind": "map", "n": 1 << 20, "res": 1024, "size": 8.0},
        # a 128^3 density grid
        {"name": "deposit_2097143_r128", "kind": "deposit", "n": 2097143, "res": 128, "size": 8.0},
        # two planes through a snapshot
        {"name": "slice_1000003_r256", "kind": "slice", "n": 1000003, "dist": "plummer", "k": 32, "fields": 1,
         "res": 256, "size": 4.0},
        # sixteen uneven snapshots in one call
        {"name": "batch_16", "kind": "batch", "count": 16, "low": 1 << 14, "high": 1 << 20, "fields": 4, "res": 1024,
         "shape": 5},
    ]


def _hot(name, n, dist, fields, k=32, dim=3, box=0.0, res=0, ngb=False, guess="plain", mask=1.0):
    return {"name": name, "kind": "hot", "n": n, "dist": dist, "fields": fields, "k": k, "dim": dim, "box": box,
            "res": res, "ngb": ngb, "guess": guess, "mask": mask}


def draw(rng):
    def size(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    kind = rng.choice(["hot", "hot", "hot", "hot", "box", "grad", "order2", "map", "deposit", "slice", "batch"])
    dist = rng.choice(["plummer", "clumps", "uniform"])
    if kind == "hot":
        dim = 2 if dist == "uniform" and rng.random() < 0.3 else 3
        k = 20 if dim == 2 else rng.choice([32, 32, 32, 16, 48, 64])
        n = size(1000, 1 << (22 if k <= 32 else 19))
        guess = "learned" if dim == 3 and k == 32 and rng.random() < 0.2 else "plain"
        c = _hot("", n, dist, rng.choice([1, 3, 4, 5, 8, 16, 19]), k, dim, 0.0,
                 rng.choice([0, 0, 256]) if dim == 3 else 0, rng.random() < 0.2, guess,
                 rng.choice([1.0, 1.0, 1.0, 0.1]))
        if c["mask"] < 1.0:
            c["res"] = 0  # a map needs the smoothing lengths of all particles
    elif kind == "box":
        c = _hot("", size(2000, 1 << 18), rng.choice(["boxclumps", "uniform"]), rng.choice([1, 3, 5]),
                 rng.choice([32, 64, 100]), 3, 1.0, 0, rng.random() < 0.5)
    elif kind == "grad":
        c = {"kind": kind, "n": size(10000, 1 << 21), "dist": dist, "k": rng.choice([32, 32, 48]),
             "fields": rng.randint(1, 24)}
    elif kind == "order2":
        c = {"kind": kind, "n": size(2000, 1 << 19), "dist": dist, "k": rng.choice([64, 80, 100]),
             "fields": rng.randint(1, 6)}
    elif kind == "map":
        c = {"kind": kind, "n": size(20000, 1 << 22), "res": rng.choice([200, 256, 500, 512, 1000, 1024]),
             "size": rng.uniform(1.0, 16.0)}
    elif kind == "deposit":
        c = {"kind": kind, "n": size(20000, 1 << 22), "res": rng.choice([48, 64, 100, 128, 150]),
             "size": rng.uniform(4.0, 16.0)}
    elif kind == "slice":
        c = {"kind": kind, "n": size(10000, 1 << 21), "dist": dist, "k": 32, "fields": rng.choice([1, 3]),
             "res": rng.choice([64, 128, 200, 256, 512]), "size": rng.uniform(0.5, 4.0)}
    else:
        c = {"kind": kind, "count": rng.randint(4, 20), "low": 1 << 14, "high": 1 << rng.randint(16, 20),
             "fields": rng.randint(1, 5), "res": rng.choice([256, 512, 1024]), "shape": rng.randint(0, 1 << 20)}
    c.pop("name", None)
    return c


# ---- inputs ---------------------------------------------------------------------------

def _positions(dist, n, dim, g):
    """(n, dim) FP64 positions, in no particular order."""
    def rand(*s):
        return torch.rand(*s, generator=g, device="cuda", dtype=torch.float64)

    def randn(*s):
        return torch.randn(*s, generator=g, device="cuda", dtype=torch.float64)

    if dist == "uniform":
        return rand(n, dim)
    if dist == "plummer":  # scale 1, radii truncated at 20, isotropic
        top = (1.0 + 20.0 ** -2) ** -1.5
        r = 1.0 / torch.sqrt((rand(n) * top).clamp_(min=1e-15) ** (-2.0 / 3.0) - 1.0)
        v = randn(n, 3)
        return r[:, None] * v / v.norm(dim=1, keepdim=True)
    # 64 Gaussian clumps with uneven weights over a 20% uniform background; the narrowest are as well resolved in a
    # small set as the 1e-3 of 2^24 particles
    wrap = dist == "boxclumps"
    centre = rand(64, 3) * 2.0 - 1.0
    least = 1e-3 * ((1 << 24) / n) ** (1.0 / 3.0)
    width = torch.exp(math.log(least) + rand(64) * (math.log(1e-1) - math.log(least)))
    weight = -torch.log(rand(64).clamp_(min=1e-12))
    which = torch.searchsorted(torch.cumsum(weight / weight.sum(), 0), rand(n)).clamp_(max=63)
    pos = centre[which] + width[which, None] * randn(n, 3)
    back = rand(n) < 0.2
    pos[back] = rand(int(back.sum()), 3) * 2.0 - 1.0
    if wrap:
        pos = torch.remainder(pos * 0.5 + 0.5, 1.0)
        pos[pos >= 1.0] = 0.0
    return pos


def _fields(pos, dist, count, g, rng, box=0.0):
    """(n, count) FP64: log density, a product of coordinates and a noisy rotation on a Plummer sphere; else sums
    of eight Fourier modes with integer wave vectors up to |k| = 32."""
    n, dim = pos.shape
    out = torch.empty((n, count), dtype=torch.float64, device="cuda")
    if dist == "plummer":
        noise = 0.1 * torch.randn((n, count), generator=g, device="cuda", dtype=torch.float64)
        r2 = (pos * pos).sum(1)
        for c in range(count):
            if c == 0:
                out[:, c] = -2.5 * torch.log1p(r2)
            elif c == 1:
                out[:, c] = pos[:, 0] * pos[:, 1] * pos[:, 2]
            elif c == 2:
                out[:, c] = -pos[:, 1] + noise[:, c]
            elif c == 3:
                out[:, c] = pos[:, 0] + noise[:, c]
            elif c == 4:
                out[:, c] = noise[:, c]
            else:
                out[:, c] = torch.sin(pos @ torch.as_tensor(rng.normal(size=3), device="cuda") + c)
        return out
    out.zero_()
    turn = 2.0 * math.pi if dist in ("uniform", "boxclumps") else math.pi
    for c in range(count):
        for _ in range(8):
            while True:
                k = rng.integers(-32, 33, size=dim)
                if 1.0 <= np.linalg.norm(k) <= 32.0:
                    break
            amp = rng.normal() / np.linalg.norm(k)
            arg = pos @ torch.as_tensor(turn * k.astype(np.float64), device="cuda")
            out[:, c] += amp * torch.sin(arg + rng.uniform(0, 2 * np.pi))
    return out


def _plummer_radius(pos, n, g):
    """Smoothing lengths that a snapshot of n particles brings along: 32 neighbours at the local density, with scatter."""
    rho = n * 3.0 / (4.0 * math.pi) * (1.0 + (pos * pos).sum(1)) ** -2.5
    h = (32.0 / (VOLNORM[3] * rho)) ** (1.0 / 3.0)
    return h * torch.exp(0.1 * torch.randn(pos.shape[0], generator=g, device="cuda", dtype=torch.float64))


def _inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 13)
    rng = np.random.default_rng(int(seed) + 101)
    kind = case["kind"]
    if kind == "batch":
        shape = np.random.default_rng(case["shape"])
        sizes = np.exp(shape.uniform(math.log(case["low"]), math.log(case["high"]), case["count"])).astype(int)
        snaps = []
        for n in sizes:
            dist = "plummer" if shape.random() < 0.5 else "clumps"
            pos = _positions(dist, int(n), 3, g)
            m = (0.5 + torch.rand(int(n), generator=g, device="cuda", dtype=torch.float64)) / int(n)
            snaps.append((pos, m, _fields(pos, dist, case["fields"], g, rng)))
        return {"snaps": snaps}
    n = case["n"]
    dim = case.get("dim", 3)
    pos = _positions(case.get("dist", "plummer"), n, dim, g)
    m = (0.5 + torch.rand(n, generator=g, device="cuda", dtype=torch.float64)) / n
    got = {"pos": pos, "m": m}
    if kind in ("map", "deposit"):
        got["h"] = _plummer_radius(pos, n, g)
        return got
    got["f"] = _fields(pos, case["dist"], case["fields"], g, rng)
    if case["fields"] == 1:
        got["f"] = got["f"].reshape(-1)
    if case.get("mask", 1.0) < 1.0:
        count = max(case["k"], int(n * case["mask"]))
        got["mask"] = torch.zeros(n, dtype=torch.bool, device="cuda")
        got["mask"][torch.randperm(n, generator=g, device="cuda")[:count]] = True
    if kind == "slice":
        c = 0.5 if case["dist"] == "uniform" else 0.0
        got["centers"] = [[c, c, c + z] for z in rng.uniform(-0.2, 0.2, 2).tolist()]
        got["size"] = min(case["size"], 1.0) if case["dist"] == "uniform" else case["size"]
    return got


def prepare(case, seed):
    s = {"case": dict(case), **_inputs(case, seed)}
    kind = case["kind"]
    if kind in ("grad", "order2", "slice"):
        s["M"] = meshoid_gb300.Meshoid(s["pos"], s["m"], des_ngb=case["k"])
    elif kind in ("map", "deposit"):
        s["M"] = meshoid_gb300.Meshoid(s["pos"], s["m"], kernel_radius=s["h"], des_ngb=32)
    elif kind == "batch":
        s["B"] = SnapshotBatch(s["snaps"], des_ngb=32, map_res=case["res"])
    return s


def run(state):
    s, case = state, state["case"]
    kind = case["kind"]
    if kind == "hot":
        M = meshoid_gb300.Meshoid(s["pos"], s["m"], des_ngb=case["k"], boxsize=case["box"] or None,
                                  particle_mask=s.get("mask"), seed=case["guess"])
        out = {"h": M.SmoothingLength(), "density": M.Density(), "grad": M.D(s["f"])}
        if case["res"]:
            size = 1.0 if case["dist"] == "uniform" else 4.0
            c = 0.5 if case["dist"] == "uniform" else 0.0
            out["map"] = M.SurfaceDensity(M.m, center=[c, c, c], size=size, res=case["res"])
        if case["ngb"]:
            out["ngb"], out["dist"] = M.NearestNeighbors(), M.NeighborDistance()
        return out
    if kind == "grad":
        return s["M"].D(s["f"])
    if kind == "order2":
        s["M"].reset_dweights()
        return {"d2": s["M"].D2(s["f"]), "d1": s["M"].D(s["f"], order=2)}
    if kind == "map":
        return s["M"].SurfaceDensity(s["m"], center=[0.0, 0.0, 0.0], size=case["size"], res=case["res"])
    if kind == "deposit":
        return s["M"].DepositToGrid(s["m"], center=[0.0, 0.0, 0.0], size=case["size"], res=case["res"])
    if kind == "slice":
        return [s["M"].Slice(s["f"], center=c, size=s["size"], res=case["res"]) for c in s["centers"]]
    B = s["B"].run()
    return {"h": list(B.hsml), "grad": list(B.grad), "map": list(B.maps)}


def _sizes(case):
    shape = np.random.default_rng(case["shape"])
    return np.exp(shape.uniform(math.log(case["low"]), math.log(case["high"]), case["count"])).astype(int)


def work(case):
    """Bytes: each input once, each output once. Operations: per query and neighbour the distance, kernel weight,
    moments and right-hand sides; per pixel of a footprint the distance, kernel and sum."""
    kind, f = case["kind"], case.get("fields", 0)
    if kind == "hot":
        n, k, d = case["n"], case["k"], case["dim"]
        q = int(n * case["mask"])
        b = n * (8 * d + 8 + 8 * f) + q * (16 + 4 * d * f) + (16 * q * k if case["ngb"] else 0) + 8 * case["res"] ** 2
        return {"bytes": b, "flops": q * k * (60.0 + 8 * f)}
    if kind == "grad":
        n, k = case["n"], case["k"]
        return {"bytes": n * (24 + 8 + 4 * k + 20 * f), "flops": n * k * (40.0 + 8 * f)}
    if kind == "order2":
        n, k = case["n"], case["k"]
        return {"bytes": n * (24 + 8 + 4 * k + 8 * f + 36 * f), "flops": n * (k * (150.0 + 20 * f) + 300 + 162 * f)}
    if kind == "map":
        return {"bytes": case["n"] * 40 + 8 * case["res"] ** 2, "flops": case["n"] * 20.0 * 100}
    if kind == "deposit":
        return {"bytes": case["n"] * 40 + 8 * case["res"] ** 3, "flops": case["n"] * 20.0 * 30}
    if kind == "slice":
        p = 2 * case["res"] ** 2
        return {"bytes": p * (24 + 8 * f) + min(p, case["n"]) * 32 * 4, "flops": p * 32 * (60.0 + 8 * f)}
    n = int(_sizes(case).sum())
    return {"bytes": n * (32 + 8 * f + 8 + 12 * f) + 8 * case["count"] * case["res"] ** 2,
            "flops": n * 32 * (60.0 + 8 * f)}


# ---- the same in 64 bits, in plain torch ------------------------------------------------

def _spline(q):
    return torch.where(q <= 0.5, 1 - 6 * q ** 2 + 6 * q ** 3, 2 * (1 - q).clamp(min=0.0) ** 3)


def _wrap(d, box):
    return d - box * torch.round(d / box) if box else d


def _nearest(query, pos, k, box=0.0):
    """The k nearest of pos to each query point, nearest first, by all pairs: (indices, distances)."""
    step = max(1, int(2e8) // pos.shape[0])
    idx, dist = [], []
    for a in range(0, query.shape[0], step):
        d2 = torch.zeros((min(step, query.shape[0] - a), pos.shape[0]), dtype=torch.float64, device=pos.device)
        for c in range(pos.shape[1]):
            d2 += _wrap(query[a:a + step, c, None] - pos[None, :, c], box) ** 2
        v, i = torch.topk(d2, k, dim=1, largest=False, sorted=True) if k > 1 else d2.min(1, keepdim=True)
        idx.append(i)
        dist.append(torch.sqrt(v))
    return torch.cat(idx), torch.cat(dist)


def _radius(dist, dim):
    """The h at which the kernel-weighted neighbour count equals k, by bisection."""
    k = dist.shape[1]
    low, high = dist[:, 1].clone(), dist[:, -1] / (1.0 - (2.0 * HNORM[dim]) ** (-1.0 / 3.0))
    for _ in range(70):
        h = 0.5 * (low + high)
        over = HNORM[dim] * _spline(dist / h[:, None]).sum(1) > k
        high, low = torch.where(over, h, high), torch.where(over, low, h)
    return 0.5 * (low + high)


def _derivatives(pos, f, rows, idx, h, order=1, box=0.0):
    """Weighted least-squares derivatives of f (n, c) at the particles `rows` with neighbours idx: (rows, c, terms)."""
    out = []
    for a in range(0, rows.shape[0], 1 << 15):
        i, r = idx[a:a + (1 << 15)], rows[a:a + (1 << 15)]
        dx = _wrap(pos[i] - pos[r][:, None, :], box)
        w = _spline(dx.norm(dim=2) / h[a:a + (1 << 15), None])
        scale = h[a:a + (1 << 15), None, None]
        dx = dx / scale
        basis = [dx[..., c] for c in range(pos.shape[1])]
        unit = [scale[:, 0, 0]] * len(basis)
        if order == 2:
            basis += [0.5 * dx[..., c] ** 2 for c in range(3)] + [dx[..., c] * dx[..., (c + 1) % 3] for c in range(3)]
            unit += [scale[:, 0, 0] ** 2] * 6
        basis = torch.stack(basis, 2)
        lhs = basis.transpose(1, 2) @ (w[..., None] * basis)
        rhs = basis.transpose(1, 2) @ (w[..., None] * (f[i] - f[r][:, None, :]))
        got = torch.linalg.solve_ex(lhs, rhs)[0] / torch.stack(unit, 1)[..., None]
        out.append(got.transpose(1, 2))
    return torch.cat(out)


def _column_map(f, pos, h, center, size, res):
    """sum_i f_i K2(|x - x_i| / h_i) / h_i^2 at the nodes g size / (res - 1)."""
    dx = size / (res - 1)
    x = [pos[:, c] - center[c] + 0.5 * size for c in range(2)]
    grid = torch.zeros(res * res, dtype=torch.float64, device=pos.device)
    near = (x[0] + h > 0) & (x[1] + h > 0) & (x[0] - h < size) & (x[1] - h < size)
    width = torch.ceil(torch.log2(2 * h / dx + 1)).clamp(min=1).long()
    for w in torch.unique(width[near]).tolist():
        part = torch.nonzero(near & (width == w)).flatten()
        span = min(1 << w, res)
        for p in torch.split(part, max(1, (1 << 25) // span ** 2)):
            node, r2 = [], []
            for c in range(2):
                first = torch.ceil((x[c][p] - h[p]) / dx).clamp(min=0).long()
                g = first[:, None] + torch.arange(span, device=pos.device)
                node.append(g)
                r2.append((x[c][p][:, None] - g * dx) ** 2)
            ok = (node[0] < res)[:, :, None] & (node[1] < res)[:, None, :]
            q = torch.sqrt(r2[0][:, :, None] + r2[1][:, None, :]) / h[p][:, None, None]
            v = torch.where(ok, _spline(q) * (1.8189136353359467 * f[p] / h[p] ** 2)[:, None, None], 0.0)
            at = node[0].clamp(max=res - 1)[:, :, None] * res + node[1].clamp(max=res - 1)[:, None, :]
            grid.index_add_(0, at.reshape(-1), v.reshape(-1))
    return grid.reshape(res, res)


def _density_grid(f, pos, h, center, size, res):
    """Each particle's f spread over the grid's nodes by its kernel, normalised to 1 over them, per node volume."""
    dx = size / (res - 1)
    x = [pos[:, c] - center[c] + 0.5 * size - 0.5 * dx for c in range(3)]
    grid = torch.zeros(res ** 3, dtype=torch.float64, device=pos.device)
    width = torch.ceil(torch.log2(2 * h / dx + 1)).clamp(min=1).long()
    for w in torch.unique(width).tolist():
        part = torch.nonzero(width == w).flatten()
        span = min(1 << w, res)
        for p in torch.split(part, max(1, (1 << 25) // span ** 3)):
            node, r2, ok = [], 0.0, True
            for c in range(3):
                first = torch.ceil((x[c][p] - h[p]) / dx).clamp(min=0).long()
                g = first[:, None] + torch.arange(span, device=pos.device)
                shape = [-1] + [span if a == c else 1 for a in range(3)]
                node.append(g.reshape(shape))
                r2 = r2 + ((x[c][p][:, None] - g * dx) ** 2).reshape(shape)
                ok = (g < res).reshape(shape) & ok
            v = torch.where(ok, _spline(torch.sqrt(r2) / h[p][:, None, None, None]), 0.0)
            total = v.sum((1, 2, 3))
            v = v * torch.where(total > 0, f[p] / total, 0.0)[:, None, None, None]
            at = (node[0].clamp(max=res - 1) * res + node[1].clamp(max=res - 1)) * res + node[2].clamp(max=res - 1)
            grid.index_add_(0, at.expand_as(v).reshape(-1), v.reshape(-1))
    return grid.reshape(res, res, res) / dx ** 3


def _solve(pos, k, rows, box=0.0):
    idx, dist = _nearest(pos[rows], pos, k, box)
    return idx, dist, _radius(dist, pos.shape[1])


def _fits(queries, n):
    return float(queries) * n <= BRUTE


def exact(case, seed):
    kind = case["kind"]
    s = _inputs(case, seed)
    if kind == "batch":
        out = {"h": [], "grad": [], "map": []}
        spent = 0.0
        for pos, m, f in s["snaps"]:
            n = pos.shape[0]
            spent += float(n) * n
            if spent > BRUTE:
                for v in out.values():
                    v.append(None)
                continue
            rows = torch.arange(n, device="cuda")
            idx, _, h = _solve(pos, 32, rows)
            out["h"].append(h)
            out["grad"].append(_derivatives(pos, f, rows, idx, h))
            c = pos.quantile(0.5, dim=0)
            r2 = ((pos - c) ** 2).sum(1)
            size = float(2.0 * r2.quantile(0.9).sqrt())
            out["map"].append(_column_map(m, pos, h.clamp(min=2 * size / case["res"]), c, size, case["res"]))
        return out if any(v is not None for v in out["h"]) else None
    pos, m = s["pos"], s["m"]
    n = pos.shape[0]
    if kind == "map":
        if n * (case["res"] / case["size"]) ** 2 > 4e10:
            return None
        return _column_map(m, pos, s["h"].clamp(min=2 * case["size"] / case["res"]), [0.0] * 3, case["size"],
                           case["res"])
    if kind == "deposit":
        if n * (case["res"] / case["size"]) ** 3 > 4e10:
            return None
        return _density_grid(m, pos, s["h"].clamp(min=case["size"] / (case["res"] - 1)), [0.0] * 3, case["size"],
                             case["res"])
    f = s["f"].reshape(n, -1)
    if kind == "slice":
        if not _fits(4 * case["res"] ** 2, n):
            return None
        out = []
        lin = torch.linspace(-s["size"] / 2, s["size"] / 2, case["res"], dtype=torch.float64, device="cuda")
        x, y = torch.meshgrid(lin, lin, indexing="ij")
        for c in s["centers"]:
            at = torch.stack([x.flatten(), y.flatten(), torch.zeros_like(x).flatten()], 1) + \
                torch.tensor(c, dtype=torch.float64, device="cuda")
            nn = _nearest(at, pos, 1)[0].flatten()
            rows, inverse = torch.unique(nn, return_inverse=True)
            idx, _, h = _solve(pos, case["k"], rows)
            d = _derivatives(pos, f, rows, idx, h)[inverse]
            got = f[nn] + torch.einsum("ij,icj->ic", at - pos[nn], d)
            out.append(got.reshape((case["res"], case["res"]) + tuple(s["f"].shape[1:])))
        return out
    mask = s.get("mask")
    rows = torch.arange(n, device="cuda") if mask is None else torch.nonzero(mask).flatten()
    if not _fits(rows.shape[0], n):
        return None
    box = case.get("box", 0.0)
    idx, dist, h = _solve(pos, case["k"], rows, box)
    tail = tuple(s["f"].shape[1:])
    if kind == "order2":
        d = _derivatives(pos, f, rows, idx, h, 2)
        return {"d2": d[..., 3:].reshape((n,) + tail + (6,)), "d1": d[..., :3].reshape((n,) + tail + (3,))}
    d = _derivatives(pos, f, rows, idx, h, 1, box).reshape((rows.shape[0],) + tail + (pos.shape[1],))
    if kind == "grad":
        return d
    dim = pos.shape[1]
    out = {"h": h, "density": m[rows] * case["k"] / (VOLNORM[dim] * h ** dim), "grad": d}
    if case["res"]:
        size = 1.0 if case["dist"] == "uniform" else 4.0
        c = 0.5 if case["dist"] == "uniform" else 0.0
        out["map"] = _column_map(m, pos, h.clamp(min=2 * size / case["res"]), [c] * 3, size, case["res"])
    if case["ngb"]:
        out["ngb"], out["dist"] = None, dist
    return out
