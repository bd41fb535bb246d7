"""The workloads whose speed is tracked, each one pass through the public entry points.

Particles follow the recipe of cm_halofinder_b200/synth.py, drawn on the GPU:
a fraction of 0.6 sits in Plummer clumps (counts dN/dM ~ M^-1.9 on [10, 5000],
rescaled to hold that fraction), the rest is a uniform background, the array
order is random, velocities are Gaussian.  Sizes are those of the benchmark's
five workloads, of the tests, and odd ones between them.

A case's fields: ``kind`` (the entry point, see ``run``), ``n`` particles (of
the largest box for a batch), ``boxes``, ``sep`` (mean separation in Mpc/h),
``clumps`` per million particles, ``linkb`` (linking length over mean
separation), ``min_members``,
``boundary`` (ghost shell), ``pos64`` (double positions), ``precision`` (pair
tests), ``members`` (membership wanted), ``properties`` (bits: 1 inertia,
2 dispersion).
"""
import ctypes
import math

import numpy as np
import torch

from cm_halofinder_b200 import FofConfig, Plan, _abi, fof, fof_sampled, halosize

DEV = "cuda"
BASE = {"kind": "box", "n": 0, "boxes": 1, "sep": 1000.0 / 256, "clumps": 596.0, "linkb": 0.2,
        "min_members": 10, "boundary": 10.0, "pos64": False, "precision": "fp32",
        "members": False, "properties": 0}
MAX_EXACT = 1_600_000   # particles above which exact() gives None
PAIRS = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))


def listed():
    def case(name, **kw):
        return {**BASE, "name": name, **kw}

    return [
        # the smallest boxes of a batched run, alone: launches and latency
        case("box_10k", n=10_007, boundary=8.0),
        # the 64^3 box: double positions, double pair tests, many small halos
        case("box_64cubed_f64", n=64 ** 3, clumps=5722.0, boundary=8.0, pos64=True,
             precision="fp64"),
        # an odd mid-size box with everything the catalog can carry
        case("box_1500k_members", n=1_500_013, members=True, properties=3),
        # the headline box
        case("box_256cubed", n=256 ** 3),
        # the 1024^3 box's parameters over 1/8 of its volume
        case("box_512cubed", n=512 ** 3, sep=2000.0 / 1024, clumps=466.0, min_members=20),
        # lightcones with a variable linking length, isolated: a shell of a
        # survey, and the full benchmark one
        case("lightcone_700k", kind="lightcone", n=700_001, boundary=5.0, members=True),
        case("lightcone_50m", kind="lightcone", n=50_000_000, boundary=5.0),
        # 64 uneven boxes in one run
        case("batch_64", kind="batch", n=4_000_000, boxes=64, boundary=8.0),
        # the drop-in call: host arrays in, catalog and membership out, one shot
        case("oneshot_1m", kind="oneshot", n=1_000_003, members=True),
        # the one-shot call that also draws the subsample
        case("sampled_200k", kind="sampled", n=200_003, boundary=8.0, pos64=True),
        # a stream of boxes in pinned host memory: copies and compute
        case("host_4m", kind="host", n=4_000_037),
        # group labels without allocations, near its largest size
        case("labels_50k", kind="labels", n=50_021, boundary=0.0, precision="fp64"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "box", "box", "lightcone", "batch", "oneshot", "sampled", "host",
                       "labels"])
    lo, hi = {"box": (1e4, 512 ** 3), "lightcone": (1e5, 5e7), "batch": (1e5, 4e6),
              "oneshot": (1e4, 4e6), "sampled": (1e4, 2e6), "host": (1e5, 256 ** 3),
              "labels": (2e3, 65536)}[kind]
    n = _log_uniform(rng, lo, hi)
    c = {**BASE, "kind": kind, "n": n, "sep": rng.choice([1000.0 / 256, 2000.0 / 1024]),
         "clumps": rng.choice([466.0, 596.0, 5722.0]),
         "boundary": 5.0 if kind == "lightcone" else 8.0, "pos64": rng.random() < 0.25,
         "precision": rng.choice(["fp32", "fp32", "fp64"]), "min_members": rng.choice([10, 20])}
    if c["pos64"]:
        c["n"] = max(int(lo), n // 2)
    if kind != "lightcone":
        c["linkb"] = round(rng.uniform(0.15, 0.25), 4)
    if kind == "batch":
        c["boxes"] = rng.randint(2, 64)
    if kind in ("box", "host", "oneshot") and n < 4e6:
        c["members"] = rng.random() < 0.5
        c["properties"] = rng.choice([0, 0, 1, 2, 3])
    if kind == "labels":
        c["boundary"] = 0.0
    return c


# ---------------------------------------------------------------- inputs


def _clumps(rng, n, per_million):
    """Particle counts of the clumps and their Plummer radii."""
    target = int(round(0.6 * n))
    u = rng.random(max(int(round(per_million * n / 1e6)), 1))
    m = (10.0 ** -0.9 + u * (5000.0 ** -0.9 - 10.0 ** -0.9)) ** (-1.0 / 0.9)
    cuts = np.rint(np.cumsum(m) * (target / m.sum())).astype(np.int64)
    cuts[-1] = target
    counts = np.diff(cuts, prepend=0)
    return counts, 0.05 * np.cbrt(np.maximum(counts, 1) / 10.0)


def _offsets(gen, counts, rs, lo, hi):
    """Clump index and Plummer offset of clump particles lo .. hi."""
    cum = torch.from_numpy(np.cumsum(counts)).to(DEV)
    cl = torch.searchsorted(cum, torch.arange(lo, hi, device=DEV), right=True)
    u = 0.999 * (1.0 - torch.rand(hi - lo, generator=gen, device=DEV, dtype=torch.float64))
    r = torch.from_numpy(rs).to(DEV)[cl] / torch.sqrt(u ** (-2.0 / 3.0) - 1.0)
    d = torch.randn((hi - lo, 3), generator=gen, device=DEV, dtype=torch.float64)
    return cl, d * (r / torch.linalg.norm(d, dim=1))[:, None]


def _finish(gen, pos):
    """Random array order, and velocities."""
    n = pos.shape[0]
    pos = pos[torch.randperm(n, generator=gen, device=DEV)]
    return pos, torch.randn((n, 3), generator=gen, device=DEV, dtype=torch.float32) * 300.0


def _box(case, n, seed, linkb):
    """A periodic box: positions, velocities and its configuration."""
    L = case["sep"] * n ** (1.0 / 3.0)
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    dt = torch.float64 if case["pos64"] else torch.float32
    counts, rs = _clumps(rng, n, case["clumps"])
    centres = torch.from_numpy(rng.random((len(counts), 3)) * L).to(DEV)
    target, step = int(counts.sum()), 1 << 25
    pos = torch.empty((n, 3), dtype=dt, device=DEV)
    for lo in range(0, target, step):
        hi = min(lo + step, target)
        cl, off = _offsets(gen, counts, rs, lo, hi)
        pos[lo:hi] = torch.remainder(centres[cl] + off, L).to(dt)
    for lo in range(target, n, step):
        hi = min(lo + step, n)
        pos[lo:hi] = (torch.rand((hi - lo, 3), generator=gen, device=DEV,
                                 dtype=torch.float64) * L).to(dt)
    pos[pos >= torch.tensor(L, dtype=dt).item()] = 0.0
    pos, vel = _finish(gen, pos)
    cfg = FofConfig(lo=(0.0,) * 3, hi=(L,) * 3, boundary=case["boundary"],
                    linklength=linkb * case["sep"], nphalomin=case["min_members"],
                    periodic=case["kind"] != "labels", precision=case["precision"],
                    properties=case["properties"])
    return pos, vel, cfg


def _lightcone(case, seed):
    """A sphere around the observer whose mean density falls threefold
    outwards, with the linking length 0.2 nbar(r)^(-1/3)."""
    n = case["n"]
    R = 1400.0 * (n / 50_000_000) ** (1.0 / 3.0)
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    slope = (2.0 / 3.0) / R
    n0 = n / (4.0 * math.pi * (R ** 3 / 3.0 - slope * R ** 4 / 4.0))
    table = 0.2 * (n0 * (1.0 - slope * np.linspace(0.0, R, 4097))) ** (-1.0 / 3.0)
    grid = torch.linspace(0.0, R, 1 << 16, device=DEV, dtype=torch.float64)
    cdf = grid ** 3 / 3.0 - slope * grid ** 4 / 4.0
    cdf /= cdf[-1].clone()

    def points(k):
        u = torch.rand(k, generator=gen, device=DEV, dtype=torch.float64)
        i = torch.searchsorted(cdf, u).clamp(1, grid.numel() - 1)
        f = (u - cdf[i - 1]) / (cdf[i] - cdf[i - 1])
        r = grid[i - 1] + f * (grid[i] - grid[i - 1])
        d = torch.randn((k, 3), generator=gen, device=DEV, dtype=torch.float64)
        return d * (r / torch.linalg.norm(d, dim=1))[:, None]

    counts, rs = _clumps(rng, n, case["clumps"])
    centres = points(len(counts))
    target, step = int(counts.sum()), 1 << 25
    dt = torch.float64 if case["pos64"] else torch.float32
    pos = torch.empty((n, 3), dtype=dt, device=DEV)
    for lo in range(0, n, step):
        hi = min(lo + step, n)
        mid = min(max(target, lo), hi)
        p = points(hi - mid)
        if mid > lo:
            cl, off = _offsets(gen, counts, rs, lo, mid)
            p = torch.cat([centres[cl] + off, p])
        rr = torch.linalg.norm(p, dim=1)     # members thrown out stay on the shell
        pos[lo:hi] = torch.where((rr > R)[:, None], p * (R / rr * (1.0 - 1e-7))[:, None], p).to(dt)
    pos, vel = _finish(gen, pos)
    lmax, b = float(table.max()), case["boundary"]
    cells = max(int((2 * R + 2 * b) / (4.0 * lmax)), 1)
    cfg = FofConfig(lo=(-R,) * 3, hi=(R,) * 3, boundary=b, linklength=lmax,
                    nphalomin=case["min_members"], periodic=False, precision=case["precision"],
                    properties=case["properties"],
                    varlink={"origin": (0.0,) * 3, "rmax": R, "table": table,
                             "ref_cells": cells})
    return pos, vel, cfg


def _batch_sizes(case):
    """Box sizes (log-uniform up to n) and linking lengths of a batch."""
    rng = np.random.default_rng(case["boxes"])
    ns = np.exp(rng.uniform(math.log(1e4), math.log(case["n"]), case["boxes"]))
    return ns.astype(np.int64), rng.uniform(0.15, 0.25, case["boxes"])


def _rows(case):
    """Halos that a catalog has room for: twice the clumps and some background."""
    n = int(_batch_sizes(case)[0].sum()) if case["kind"] == "batch" else case["n"]
    return int(2 * case["clumps"] * n / 1e6 + n / 2000) + 64


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        ns, bs = _batch_sizes(case)
        sets = [_box(case, int(ns[i]), 1000 * seed + i, float(bs[i])) for i in range(len(ns))]
        pos, vel, cfg = [list(v) for v in zip(*sets)]
    elif kind == "lightcone":
        pos, vel, cfg = _lightcone(case, seed)
    else:
        pos, vel, cfg = _box(case, case["n"], seed, case["linkb"])
    s = {"case": case, "pos": pos, "vel": vel, "cfg": cfg}
    if kind != "labels":    # the program's own catalog, with room for any box of this size
        rows = _rows(case)
        s["props"] = np.zeros((rows, halosize(case["properties"])), np.float32)
        s["head"] = np.zeros(rows, np.uint32)
    if kind in ("box", "lightcone", "batch", "host"):
        s["plan"] = Plan(cfg[0] if kind == "batch" else cfg,
                         pos_dtype=np.float64 if case["pos64"] else np.float32)
    if kind == "host":
        s["pos"], s["vel"] = (torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t).numpy()
                              for t in (pos, vel))
    elif kind in ("oneshot", "sampled"):
        s["pos"], s["vel"] = pos.cpu().numpy(), vel.cpu().numpy()
        if kind == "sampled":
            s["ids"] = np.arange(case["n"], dtype=np.uint64)
            s["inside"], s["outside"] = np.zeros((2, case["n"]), np.int64)
    elif kind == "labels":
        s["label"] = torch.empty(case["n"], dtype=torch.int32, device=DEV)
    torch.cuda.empty_cache()
    return s


# ---------------------------------------------------------------- one pass


def _keep(to, rows, at=0):
    """Puts `rows` into the program's own array; what it held beyond goes."""
    to[at:at + len(rows)] = rows
    return at + len(rows)


def _catalog(s, *cats):
    at = 0
    for cat in cats:
        _keep(s["head"], cat.head, at)
        at = _keep(s["props"], cat.props, at)
    s["head"][at:] = 0
    s["props"][at:] = 0.0
    out = {"halos": np.array([c.nhalos for c in cats]), "props": s["props"], "head": s["head"]}
    if cats[0].member is not None:
        out["member"] = cats[0].member
    return out


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    pos, vel, cfg = s["pos"], s["vel"], s["cfg"]
    if kind == "batch":
        return _catalog(s, *s["plan"].run_batch(cfg, pos, vel))
    if kind == "oneshot":
        return _catalog(s, fof(pos, vel, cfg, members=case["members"]))
    if kind == "sampled":
        cat, inside, outside = fof_sampled(pos, vel, cfg, 0.3, 0.05, seed=1234, ids=s["ids"])
        s["inside"][_keep(s["inside"], inside):] = -1
        s["outside"][_keep(s["outside"], outside):] = -1
        return {**_catalog(s, cat), "inside": s["inside"], "outside": s["outside"]}
    if kind == "labels":
        p = cfg.to_c()
        _abi.check(_abi.lib().cmh_fof_labels_noalloc(
            ctypes.byref(p), ctypes.c_void_p(pos.data_ptr()),
            _abi.CMH_FLOAT64 if case["pos64"] else _abi.CMH_FLOAT32, case["n"],
            ctypes.c_void_p(s["label"].data_ptr()), ctypes.c_void_p(0)))
        return s["label"]
    return _catalog(s, s["plan"].run(pos, vel, members=case["members"]))  # box, lightcone, host


def work(case):
    """Positions and velocities read once, membership or labels written once
    (the catalog itself is small)."""
    n = int(_batch_sizes(case)[0].sum()) if case["kind"] == "batch" else case["n"]
    if case["kind"] == "labels":
        return {"bytes": n * (3 * (8 if case["pos64"] else 4) + 4), "flops": 0}
    out = 8 if case["members"] else 0
    return {"bytes": n * (3 * (8 if case["pos64"] else 4) + 12 + out), "flops": 0}


# ---------------------------------------------------------------- the values in 64 bits


def _components(label, a, b):
    """Merges the components of `label` (each value a member's index) that the
    edges (a, b) join: hook to the lower label, then pointer jumping."""
    while True:
        la, lb = label[a], label[b]
        apart = la != lb
        if not bool(apart.any()):
            return label
        a, b, la, lb = a[apart], b[apart], la[apart], lb[apart]
        label.scatter_reduce_(0, torch.maximum(la, lb), torch.minimum(la, lb), "amin")
        while True:
            up = label[label]
            if torch.equal(up, label):
                break
            label = up


def _processed(pos, cfg):
    """Stored coordinates of the originals and of the periodic images, in
    processing order, and their source particles."""
    n, dev = pos.shape[0], pos.device
    src = torch.arange(n, device=dev)
    if not cfg.periodic:
        return pos, src
    L, b = cfg.hi[0] - cfg.lo[0], cfg.boundary
    near = ((pos < cfg.lo[0] + 1.01 * b) | (pos > cfg.hi[0] - 1.01 * b)).any(dim=1)
    edge, esrc = pos[near], src[near]
    got, gsrc, order = [], [], []
    for code in range(27):
        sh = [code % 3 - 1, code // 3 % 3 - 1, code // 9 - 1]
        if sh == [0, 0, 0]:
            continue
        x, ok = edge.clone(), torch.ones(edge.shape[0], dtype=torch.bool, device=dev)
        for a in range(3):
            if sh[a]:
                x[:, a] = (edge[:, a].double() + sh[a] * L).to(pos.dtype)
                xa = x[:, a].double()
                ok &= (xa >= cfg.lo[a] - b) & (xa <= cfg.hi[a] + b)
        got.append(x[ok])
        gsrc.append(esrc[ok])
        order.append(esrc[ok] * 27 + code)
    o = torch.argsort(torch.cat(order))
    return torch.cat([pos, torch.cat(got)[o]]), torch.cat([src, torch.cat(gsrc)[o]])


def _link_rule(x, cfg):
    """Per particle the grid cell and l^2 of the variable linking length."""
    v = cfg.varlink
    lo = torch.tensor(cfg.lo, dtype=torch.float64, device=x.device) - cfg.boundary
    side = (cfg.hi[0] - cfg.lo[0] + 2 * cfg.boundary) / v["ref_cells"]
    cell = torch.floor((x.double() - lo) / side).long()
    r = torch.sqrt((((lo + (cell + 0.5) * side) ** 2)).sum(dim=1))
    tab = torch.from_numpy(np.asarray(v["table"])).to(x.device)
    t = r / (v["rmax"] / (len(tab) - 1))
    i = t.long().clamp(max=len(tab) - 2)
    f = t - i
    ln = torch.where(t >= len(tab) - 1, tab[-1], tab[i] * (1.0 - f) + tab[i + 1] * f)
    return cell, ln * ln


def _groups(x, cfg):
    """Group of every processed particle (a label per group).  Particles in
    one cell of side l / sqrt(3) are linked; cells within reach are joined by
    the first linked pair found, all pairs being tried where need be."""
    dev = x.device
    var = cfg.varlink is not None
    lmin = float(np.min(cfg.varlink["table"])) if var else cfg.linklength
    h = lmin * (1.0 - 1e-6) / math.sqrt(3.0)
    W = int(cfg.linklength / h * (1.0 + 1e-6)) + 1
    lo = torch.tensor(cfg.lo, dtype=torch.float64, device=dev) - cfg.boundary
    g = torch.floor((x.double() - lo) / h).long() + W
    key = (g[:, 2] << 40) | (g[:, 1] << 20) | g[:, 0]
    cells, inv, num = torch.unique(key, return_inverse=True, return_counts=True)
    order = torch.argsort(inv)
    first = torch.cumsum(num, 0) - num
    rule = _link_rule(x, cfg) if var else None
    A, B = [], []
    for dz in range(0, W + 1):
        for dy in range(-W, W + 1):
            for dx in range(-W, W + 1):
                if (dz, dy, dx) <= (0, 0, 0):
                    continue
                want = cells + (dz << 40) + (dy << 20) + dx
                at = torch.searchsorted(cells, want).clamp(max=len(cells) - 1)
                hit = torch.nonzero(cells[at] == want).flatten()
                A.append(hit)
                B.append(at[hit])
    A, B = torch.cat(A), torch.cat(B)
    label = torch.arange(len(cells), device=dev)

    def test(a, b, cap):
        """Which pairs (a, b) hold a linked pair among their first `cap` particles."""
        na, nb = num[a].clamp(max=cap), num[b].clamp(max=cap)
        tests = na * nb
        pair = torch.repeat_interleave(torch.arange(len(a), device=dev), tests)
        k = torch.arange(len(pair), device=dev) - (torch.cumsum(tests, 0) - tests)[pair]
        i = order[first[a][pair] + k // nb[pair]]
        j = order[first[b][pair] + k % nb[pair]]
        d = (x[i] - x[j]).double()
        d2 = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
        if var:
            ci, cj = rule[0][i], rule[0][j]
            ki, kj = (c[:, 2] << 42 | c[:, 1] << 21 | c[:, 0] for c in (ci, cj))
            lsq = torch.where(ki <= kj, rule[1][i], rule[1][j])     # the lower cell's
            ok = (d2 <= lsq) & ((ci - cj).abs() <= 1).all(dim=1)
        else:
            ok = d2 <= cfg.linklength * cfg.linklength
        return torch.unique(pair[ok])

    for cap in (2, 8, 1 << 40):
        apart = label[A] != label[B]
        A, B = A[apart], B[apart]
        o = torch.argsort(num[A].clamp(max=cap) * num[B].clamp(max=cap))
        A, B = A[o], B[o]
        at = 0
        while at < len(A):
            cost = torch.cumsum(num[A[at:]].clamp(max=cap) * num[B[at:]].clamp(max=cap), 0)
            end = at + max(int(torch.searchsorted(cost, 60_000_000)), 1)
            a, b = A[at:end], B[at:end]
            apart = label[a] != label[b]
            a, b = a[apart], b[apart]
            if len(a):
                hit = test(a, b, cap)
                label = _components(label, a[hit], b[hit])
            at = end
    return label[inv]


def exact(case, seed):
    if case["kind"] in ("batch", "labels") or case["n"] > MAX_EXACT:
        return None
    s = prepare(case, seed)
    cfg = s["cfg"]
    pos, vel = (torch.as_tensor(s[k]).to(DEV) for k in ("pos", "vel"))
    x, src = _processed(pos, cfg)
    group = _groups(x, cfg)
    _, gid, num = torch.unique(group, return_inverse=True, return_counts=True)
    head = torch.full_like(num, x.shape[0]).scatter_reduce_(
        0, gid, torch.arange(x.shape[0], device=DEV), "amin")
    X, V = x.double(), vel[src].double()

    def total(v):
        return torch.zeros(len(num), dtype=torch.float64, device=DEV).index_add_(0, gid, v)

    n = num.double()
    SX, SV = [total(X[:, a]) for a in range(3)], [total(V[:, a]) for a in range(3)]
    own = num >= case["min_members"]
    for a in range(3):
        com = SX[a] / n
        own &= (com >= cfg.lo[a]) & (com < cfg.hi[a])
    rec = [n] + [t / n for t in SX + SV]
    if case["properties"] & 1:      # about the centre, so that nothing cancels
        D = [X[:, a] - (SX[a] / n)[gid] for a in range(3)]
        xx, yy, zz, xy, xz, yz = (total(D[a] * D[b]) for a, b in PAIRS)
        rec += [yy + zz, xx + zz, xx + yy, -xy, -xz, -yz]
    if case["properties"] & 2:
        D = [V[:, a] - (SV[a] / n)[gid] for a in range(3)]
        rec += [total(D[a] * D[b]) / n for a, b in PAIRS]
    pick = torch.nonzero(own).flatten()
    pick = pick[torch.argsort(head[pick])]
    props = torch.zeros(s["props"].shape, dtype=torch.float64, device=DEV)
    props[:len(pick)] = torch.stack(rec, dim=1)[pick]
    return {"props": props}
