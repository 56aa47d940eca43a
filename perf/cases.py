"""The calls that a user of this library makes, as measured cases: all-active walks over windows,
the engine's leaf-group walk from host arrays, sparse active sets, rebuild-and-walk steps, forests
in a captured plan, the tidal tensor and jerk, gas rules, the density solve, neighbour lists and the
direct sum.

A case is a dict of plain values; ``kind`` picks the call, ``ics`` the particle distribution (the
seeded workloads of ``gizmo_shared_memory_b200/ics.py``, drawn here on the GPU so that they are
quick to make), the rest its sizes and options.  ``exact`` repeats each call in 64 bits with plain
torch: an octree with the same cells, the same opening decisions, and sums in double.
"""
import math

import numpy as np
import torch

import gizmo_shared_memory_b200 as gt

F64 = torch.float64
_CTX = {}


def _ctx():
    """One context per process, on torch's stream, as a torch program keeps it."""
    if "c" not in _CTX:
        _CTX["c"] = gt.Context(0, torch_stream=True)
    return _CTX["c"]


# ---- the cases -------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest whole problem of the configurations: accelerations and potentials
        dict(name="walk_plummer_65k_phi", kind="walk", ics="plummer", n=65536, alpha=0.005, batch=32, phi=True),
        # the isolated galaxy, every particle active: the ordinary full step
        dict(name="walk_galaxy_4m", kind="walk", ics="galaxy", n=4194304, alpha=0.0025, batch=32, phi=False),
        # the clustered box the headline metric is quoted on: the largest
        dict(name="walk_box_16m", kind="walk", ics="box", n=16777216, alpha=0.0025, batch=32, phi=False),
        # the engine's own call: leaf groups (batch 0), Morton order, host arrays in and out, ragged n
        dict(name="engine_leaf_1m", kind="engine", ics="galaxy", n=1000003, alpha=0.0025, batch=0),
        # a deep time bin: a scattered 0.1 % of the galaxy, where latency and launches count
        dict(name="active_galaxy_4k", kind="active", ics="galaxy", n=4194304, alpha=0.0025, targets=4194),
        # a step that rebuilds: new positions, build, walk; ragged n
        dict(name="step_box_2m", kind="step", ics="box", n=2000003, alpha=0.0025, batch=32),
        # many independent clusters of uneven size in one captured launch
        dict(name="forest_256", kind="forest", systems=256, n=4000000, alpha=0.0025, batch=32),
        # the tidal timestep / Hermite engine: accelerations, tidal tensor and jerk
        dict(name="tidal_jerk_galaxy_1m", kind="ext", ics="galaxy", n=1048576, alpha=0.0025, batch=32, jerk=True),
        # adaptive softening with gas, stars and sinks: types and zeta handed over, then the walk
        dict(name="gas_galaxy_1m", kind="gas", ics="galaxy", n=1048577, alpha=0.0025, batch=32, sink_radius=0.02),
        # the hydro half: the density solve warm-started from the last step's smoothing lengths
        dict(name="density_galaxy_1m", kind="density", ics="galaxy", n=1048576),
        # the neighbour lists at those lengths, host arrays in and out as the engine's cache has them
        dict(name="lists_box_250k", kind="lists", ics="box", n=250001),
        # the FP64 direct sum over a seeded sample: the error oracle of every force table
        dict(name="direct_262k", kind="direct", ics="plummer", n=262144, targets=4096, fp32=False),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["walk", "walk", "walk", "engine", "active", "step", "forest", "ext", "gas", "density", "lists",
                       "direct"])
    ics = rng.choice(["plummer", "galaxy", "box"])
    alpha = 0.005 if ics == "plummer" else 0.0025
    c = dict(kind=kind, ics=ics, alpha=alpha)
    if kind == "walk":
        # windows of 32 are the recommended grouping; 8 is bench_treeforce's, 64 the autotuner's next
        c["batch"] = rng.choice([32, 32, 32, 24, 8, 64])
        c["n"] = _logint(rng, 8192, 16000000 if c["batch"] in (32, 24) else 4000000)
        c["phi"] = rng.random() < 0.3
    elif kind == "engine":
        c["n"], c["batch"] = _logint(rng, 8192, 4000000), rng.choice([0, 0, 8, 32])
    elif kind == "active":
        c["n"] = _logint(rng, 65536, 8000000)
        c["targets"] = max(32, int(c["n"] * math.exp(rng.uniform(math.log(1e-4), math.log(0.1)))))
    elif kind == "step":
        c["n"], c["batch"] = _logint(rng, 8192, 8000000), 32
    elif kind == "forest":
        del c["ics"]
        c["alpha"], c["batch"], c["systems"] = 0.0025, 32, _logint(rng, 2, 256)
        c["n"] = min(8000000, c["systems"] * _logint(rng, 2048, 65536))
    elif kind == "ext":
        c["n"], c["batch"], c["jerk"] = _logint(rng, 8192, 4000000), 32, rng.random() < 0.5
    elif kind == "gas":
        c["n"], c["batch"] = _logint(rng, 8192, 4000000), 32
        c["sink_radius"] = rng.choice([0.0, 0.02])
    elif kind == "density":
        c["n"] = _logint(rng, 16384, 4000000)
    elif kind == "lists":
        c["n"] = _logint(rng, 8192, 500000)
    else:
        c["targets"], c["fp32"] = _logint(rng, 64, 8192), rng.random() < 0.3
        c["n"] = _logint(rng, 8192, 1000000)
    if kind in ("density", "lists", "direct"):
        c.pop("alpha")
    return c


# ---- inputs ----------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _u(g, n, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(n, generator=g, dtype=F64, device="cuda")


def _dirs(g, n):
    ct = _u(g, n, -1.0, 1.0)
    st = torch.sqrt(torch.clamp(1.0 - ct * ct, min=0.0))
    ph = _u(g, n, 0.0, 2.0 * math.pi)
    return st * torch.cos(ph), st * torch.sin(ph), ct


def _plummer(g, n, a=1.0, soft=0.01):
    q = 20.0
    X = torch.clamp(_u(g, n, 0.0, q ** 3 / (1.0 + q * q) ** 1.5), min=1e-300)
    r = a / torch.sqrt(X ** (-2.0 / 3.0) - 1.0)
    ux, uy, uz = _dirs(g, n)
    one = torch.ones(n, dtype=F64, device="cuda")
    return dict(x=r * ux, y=r * uy, z=r * uz, m=one / n, soft=one * soft)


def _galaxy(g, n):
    nd = n // 4
    nh = n - nd
    q = 30.0
    s = torch.sqrt(_u(g, nh, 0.0, q * q / (1.0 + q) ** 2))
    r = s / (1.0 - s)
    ux, uy, uz = _dirs(g, nh)
    # 1 - (1 + x) e^-x is the distribution of the sum of two exponential deviates
    R = -0.1 * torch.log(torch.clamp(_u(g, nd) * _u(g, nd), min=1e-300))
    ph = _u(g, nd, 0.0, 2.0 * math.pi)
    dz = 0.01 * torch.atanh(_u(g, nd, -1.0 + 1e-15, 1.0 - 1e-15))
    one = torch.ones(n, dtype=F64, device="cuda")
    m, soft = one / nh, one * 0.005
    m[nh:] = 0.05 / max(nd, 1)
    soft[nh:] = 0.002
    return dict(x=torch.cat([r * ux, R * torch.cos(ph)]), y=torch.cat([r * uy, R * torch.sin(ph)]),
                z=torch.cat([r * uz, dz]), m=m, soft=soft)


def _box(g, n):
    c = [torch.full((1,), 0.5, dtype=F64, device="cuda") for _ in range(3)]
    R = 0.5
    while c[0].numel() < n:
        k = 4 * c[0].numel()
        rr = R * _u(g, k) ** (1.0 / 3.0)
        c = [torch.repeat_interleave(q, 4) + rr * d for q, d in zip(c, _dirs(g, k))]
        R /= 1.9
    k = c[0].numel()
    if k > n:
        keep = torch.randperm(k, generator=g, device="cuda")[:n]
        c = [q[keep] for q in c]
    uni = _u(g, n) < 0.1
    c = [torch.remainder(torch.where(uni, _u(g, n), q), 1.0).contiguous() for q in c]
    one = torch.ones(n, dtype=F64, device="cuda")
    return dict(x=c[0], y=c[1], z=c[2], m=one / n, soft=one * 1e-4)


def _particles(case, seed):
    return {"plummer": _plummer, "galaxy": _galaxy, "box": _box}[case["ics"]](_gen(seed), int(case["n"]))


def _forest(case, seed):
    """Independent Plummer spheres, sizes and scale radii log-uniform, side by side on a line."""
    S, n = int(case["systems"]), int(case["n"])
    rng = np.random.default_rng(S * 1000003 + n)  # sizes belong to the case, positions to the seed
    raw = np.exp(rng.uniform(math.log(1024), math.log(262144), S))
    ns = np.maximum(16, np.floor(raw * (n / raw.sum()))).astype(np.int64)
    off = np.concatenate([[0], np.cumsum(ns)])
    N = int(off[-1])
    a = torch.as_tensor(np.exp(rng.uniform(math.log(0.5), math.log(2.0), S)), device="cuda")
    sysid = torch.repeat_interleave(torch.arange(S, device="cuda"), torch.as_tensor(ns, device="cuda"))
    P = _plummer(_gen(seed), N)
    ai = a[sysid]
    P["x"] = P["x"] * ai + 400.0 * sysid.to(F64)
    P["y"], P["z"], P["soft"] = P["y"] * ai, P["z"] * ai, 0.01 * ai
    P["m"] = (1.0 / torch.as_tensor(ns, device="cuda").to(F64))[sysid]
    return P, off


def _coarse(a):
    """Rounded to seven leading bits: an earlier step's value, the same whichever build made it."""
    m, e = torch.frexp(a)
    return torch.ldexp(torch.round(m * 128.0) / 128.0, e)


def _bootstrap(ctx, T, alpha):
    """aold in tree order from a Barnes-Hut walk, as the first step of a run forms it."""
    a = ctx.accel_grouped(T, None, theta=0.7, batch=32, group_mode=gt.GT_GROUP_BATCH, device_out=True)
    return _coarse(ctx.form_aold(*a, alpha))


def _velocities(seed, n):
    g = _gen(seed + 1)
    return [0.3 * torch.randn(n, generator=g, dtype=F64, device="cuda") for _ in range(3)]


def _gas(case, seed, P):
    n = P["m"].numel()
    g = _gen(seed + 2)
    ty = torch.where(_u(g, n) < 0.7, 0, 4).to(torch.uint8)
    ty[torch.randperm(n, generator=g, device="cuda")[: n // 100]] = 5
    z = 0.1 * P["m"] ** 2 * P["soft"] ** 2 * torch.randn(n, generator=g, dtype=F64, device="cuda")
    return ty, torch.where(ty == 0, z, torch.zeros_like(z))


def _window_opts(batch):
    return dict(batch=batch, group_mode=gt.GT_GROUP_BATCH if batch else gt.GT_GROUP_LEAF, group_max=max(batch, 32))


def _hydro(case, seed):
    """Tree, all targets in tree order and a warm start: converged lengths, off by a few per cent."""
    ctx = _ctx()
    P = _particles(case, seed)
    T = ctx.build(P, key_mode=gt.GT_KEY_MORTON)
    d = T.download()
    ob, leaf = d["orderbuf"], d["leaf_of"][d["orderbuf"]]
    h0 = 0.8 * d["size"][leaf] * np.cbrt(16.0 / np.maximum((d["phi"] - d["plo"])[leaf], 1))
    tg = torch.as_tensor(ob.view(np.int32), device="cuda")
    h = ctx.density(T, tg, h_start=torch.as_tensor(h0, device="cuda"))["h"]
    drift = torch.exp(0.05 * torch.randn(h.numel(), generator=_gen(seed + 3), dtype=F64, device="cuda"))
    return P, T, tg, ob, _coarse(h * drift)


def _list_radii(ctx, P, T, ob, h):
    """Centres in tree order, each with a radius halfway between its 32nd and 33rd neighbour."""
    idx = ob.astype(np.int64)
    c = [P[k].cpu().numpy()[idx] for k in "xyz"]
    n, r = len(idx), (1.3 * h).cpu().numpy()
    while True:
        start, found = ctx.ngb_search(T, *c, r)
        few = np.diff(start) < 33
        if not few.any():
            break
        r = np.where(few, 1.25 * r, r)
    st, fd = torch.as_tensor(start, device="cuda"), torch.as_tensor(found.astype(np.int64), device="cuda")
    X = torch.stack([P[k] for k in "xyz"], 1)
    who = torch.repeat_interleave(torch.arange(n, device="cuda"), st[1:] - st[:-1])
    d = ((X[fd] - X[torch.as_tensor(idx, device="cuda")][who]) ** 2).sum(1).sqrt()
    d, o = torch.sort(d)
    who, o2 = torch.sort(who[o], stable=True)
    d = d[o2]
    return dict(c=c, r=(0.5 * (d[st[:-1] + 31] + d[st[:-1] + 32])).cpu().numpy())


def prepare(case, seed):
    ctx, kind = _ctx(), case["kind"]
    s = dict(case=case, kind=kind)
    if kind in ("density", "lists"):
        P, T, tg, ob, h = _hydro(case, seed)
        s.update(P=P, T=T, targets=tg, h=h)
        if kind == "lists":
            s.update(_list_radii(ctx, P, T, ob, h))
        return s
    if kind == "direct":
        P = _particles(case, seed)
        t = torch.randperm(P["m"].numel(), generator=_gen(seed + 4), device="cuda")[: int(case["targets"])]
        return dict(s, P=P, targets=t.to(torch.int32).contiguous())
    off = None
    if kind == "forest":
        P, off = _forest(case, seed)
    else:
        P = _particles(case, seed)
    s["P"] = P
    T = ctx.build(P, offsets=off, key_mode=gt.GT_KEY_MORTON if kind == "engine" else gt.GT_KEY_PEANO)
    s["aold"] = _bootstrap(ctx, T, case["alpha"])
    if kind != "step":
        s["T"] = T
    if kind == "engine":
        s["aold"] = s["aold"].cpu().numpy()
    elif kind == "active":
        nl = T.n_live
        pos = torch.randperm(nl, generator=_gen(seed + 5), device="cuda")[: int(case["targets"])].sort()[0]
        order = torch.as_tensor(T.download(nodes=False)["orderbuf"].view(np.int32), device="cuda")
        s["targets"], s["aold"] = order[pos].contiguous(), s["aold"][pos].contiguous()
    elif kind == "forest":
        s["outs"] = tuple(torch.empty(T.n_live, dtype=F64, device="cuda") for _ in range(3))
        s["plan"] = ctx.plan(T, s["aold"], s["outs"], **_window_opts(case["batch"]))
    elif kind == "ext":
        ctx.tree_velocities(T, *_velocities(seed, P["m"].numel()))
    elif kind == "gas":
        s["type"], s["zeta"] = _gas(case, seed, P)
    return s


def run(s):
    ctx, case, kind = _ctx(), s["case"], s["kind"]
    if kind == "walk":
        return ctx.accel_grouped(s["T"], None, aold=s["aold"], want_phi=case["phi"], **_window_opts(case["batch"]))
    if kind == "engine":
        return ctx.accel_grouped(s["T"], None, aold=s["aold"], **_window_opts(case["batch"]))
    if kind == "active":
        return ctx.accel_grouped(s["T"], s["targets"], aold=s["aold"], **_window_opts(0))
    if kind == "step":
        T = ctx.build(s["P"])
        return ctx.accel_grouped(T, None, aold=s["aold"], **_window_opts(case["batch"]))
    if kind == "forest":
        s["plan"].launch()
        return s["outs"]
    if kind == "ext":
        n = s["aold"].numel()
        mk = lambda *q: torch.empty(*q, dtype=F64, device="cuda")  # noqa: E731
        outs = (mk(n), mk(n), mk(n), None, mk(n, 6), mk(n, 3) if case["jerk"] else None)
        r = ctx.accel_grouped_ext(s["T"], None, aold=s["aold"], outs=outs, **_window_opts(case["batch"]))
        return [q for q in r if q is not None]
    if kind == "gas":
        ctx.tree_gas(s["T"], s["type"], s["zeta"])
        return ctx.accel_grouped(s["T"], None, aold=s["aold"], sink_direct_radius=case["sink_radius"],
                                 **_window_opts(case["batch"]))
    if kind == "density":
        return ctx.density(s["T"], s["targets"], h_start=s["h"])
    if kind == "lists":
        return ctx.ngb_search(s["T"], *s["c"], s["r"])
    return ctx.direct(s["P"], s["targets"], precision=gt.GT_DIRECT_FP32 if case["fp32"] else gt.GT_DIRECT_FP64)


# ---- the work a call cannot do without ---------------------------------------------------------------
def _interactions(case):
    """Interactions per particle of the relative criterion, as the walk counts them on the seeded
    workloads; they grow slowly with n."""
    if case["kind"] == "forest":
        return 1300.0
    base, ref = {"plummer": (890.0, 65536), "galaxy": (1650.0, 4194304), "box": (2525.0, 16777216)}[case["ics"]]
    b = int(case.get("batch", 0))
    return base * (1.0 + 0.06 * math.log(case["n"] / ref)) * {0: 0.65, 8: 0.65, 24: 0.93, 64: 1.25}.get(b, 1.0)


def work(case):
    kind, n = case["kind"], float(case["n"])
    nt = float(case.get("targets", n))
    tree = n * 40.0 + 0.24 * n * 64.0  # particles and packed nodes, each read once
    if kind == "direct":
        return {"bytes": n * 40.0 + nt * 36.0, "flops": 20.0 * n * nt}
    if kind == "density":
        return {"bytes": tree + n * (12.0 + 24.0), "flops": n * 2.0 * 45.0 * 30.0}
    if kind == "lists":
        return {"bytes": tree + n * (32.0 + 8.0 + 30.0 * 4.0), "flops": n * 45.0 * 8.0}
    out = 24.0 + (8.0 if case.get("phi") else 0.0)
    flops = 20.0 * nt * _interactions(case)
    if kind == "ext":
        out += 48.0 + (24.0 if case["jerk"] else 0.0)
        flops *= 2.1 if case["jerk"] else 1.6
    if kind == "active":
        # one leaf's targets touch a few thousand nodes and particles; never more than the tree
        return {"bytes": min(tree, nt * 1000.0 * 64.0) + nt * 36.0, "flops": flops}
    byt = tree + nt * (8.0 + out)
    if kind == "step":
        byt += n * (40.0 + 32.0 + 16.0) + 0.24 * n * 64.0
    if kind == "gas":
        byt += n * 9.0 * 2.0
    return {"bytes": byt, "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind == "density":
        # Sums in double, but the face-closure correction switches on and off with h: some targets near
        # its threshold do not settle (up to 100 iterations), and the last bit of a sum then decides
        # where one of them stops.  Against the same solve in another order: h 9e-5, rho 4e-4 apart in
        # the norm, from one target in some tens of thousands; four times that.
        return {"rel": 1.6e-3, "max": 1.0 - 1e-9, "differ": 1e-3}
    if kind == "lists":
        return "exact"
    if kind == "direct":
        return {"rel": 4e-6, "max": 1e-4} if case["fp32"] else {"rel": 1e-12, "max": 1e-10}
    # FP32 interactions on offsets from a group's centre, against the same sums in 64 bits: up to 1.6e-6
    # on the smooth systems and 9e-6 (potential 4e-5) where clumps a few softenings across dominate the
    # norm (the box, clusters far from the origin); four times that
    clumped = kind == "forest" or case["ics"] == "box"
    return {"rel": 1.6e-4 if clumped and case.get("phi") else 4e-5 if clumped else 6e-6}


# ---- the same calls in 64 bits -----------------------------------------------------------------------
# The Peano-Hilbert curve as a state machine, (next state << 3) | digit per (state, octant): it defines
# the order of the particles and so the windows; one three-digit hexadecimal number per entry.
_PH = """
1200e70c90de0530540ca0dd0ef05c0c60c512805b0d10d20440430cd0da0f71300ce0d904b1380c20c104c0ff0d50d6
1410c01661071420331650340c803b10f03c14914a16e16d0231520241750d015111717615a15917d17e02b0d802c11f
10e1191270e010d11a0140131011020e801b11611512f01c10a11d00300410911e0f013710510600c13f11211100b0f8
0c715610017107415507317215e15d17917a0cf07c10807b1450641620631460d716111006c0df06b11814d14e16a169
0e614f0e50b41311581320b31571400bc0bb0ee1390ed13a1481210a312215f0f60a40f51290fe12a0fd1501470ab0ac
0e20930e116813509413617f09b09c1701670ea13d0e913e08412516f1260830f21780f112d0fa12e0f908c08b177160
06702000e01911411300d01a02811b00100206f11c01601510310400a01d03007700901e10c07f00500610b038012011
0860070a10400850f40a20f300f0fc0480fb08e08d0a90aa0e40950e30b20170960500b109d09e0ba0b90ec01f0eb058
04905e06002704a05d0d30d404604502f0dc0510520680db04d05a0c40c304e0590370700420410cb0780550560cc03f
0000910470b61330921340b509909a0be0bd00813b04f13c0821230a51240810100a605712b01812c05f08a0890ad0ae
02108802217307609f07517409008717b17c02907e02a07d08f06616406509803116303206e03906d03a09708016c16b
0251540260af0721530710b815c15b0b70a002d07a02e0791430620a80611440350bf03606a03d06903e14b14c0b00a7
"""
_PH_TAB = [int("".join(_PH.split())[3 * i:3 * i + 3], 16) for i in range(384)]
_LEVELS, _LEAF = 20, 16


def _keys(P, peano):
    lo = [P[k].min() for k in "xyz"]
    hi = [P[k].max() for k in "xyz"]
    ext = torch.stack([h - q for h, q in zip(hi, lo)]).max()
    side = ext * 1.0000001 if float(ext) > 0 else torch.ones_like(ext)
    q = []
    for k, (a, b) in zip("xyz", zip(lo, hi)):
        corner = 0.5 * (a + b) - 0.5 * side
        q.append(((P[k] - corner) * (float(2 ** _LEVELS - 1) / side)).to(torch.int64))
    key = torch.zeros_like(q[0])
    tab = torch.tensor(_PH_TAB, device="cuda", dtype=torch.int64)
    state = torch.zeros_like(key)
    for lev in range(_LEVELS - 1, -1, -1):
        a, b, c = ((v >> lev) & 1 for v in q)
        if peano:
            step = tab[state * 8 + (a << 2 | b << 1 | c)]
            key, state = (key << 3) | (step & 7), step >> 3
        else:
            key = (key << 3) | (c << 2 | b << 1 | a)
    return key, side


def _cut(starts, values, reduce):
    """Sums or maxima of values over consecutive ranges that begin at starts."""
    seg = torch.zeros(values.shape[0], dtype=torch.int64, device="cuda")
    seg[starts[1:]] = 1
    seg = seg.cumsum(0)
    out = torch.zeros((starts.numel(),) + values.shape[1:], dtype=values.dtype, device="cuda")
    if reduce == "sum":
        return out.index_add_(0, seg, values)
    return out.scatter_reduce_(0, seg, values, reduce, include_self=False)


def _octree(P, peano, off=None, vel=None, sink=None):
    """The library's octree, level by level: cells of the key's digits, leaves of at most 16."""
    n = P["m"].numel()
    off = [0, n] if off is None else [int(v) for v in off]
    key, order, sides = [], [], []
    for a, b in zip(off[:-1], off[1:]):
        k, side = _keys({c: P[c][a:b] for c in "xyz"}, peano)
        k, o = torch.sort(k, stable=True)
        key.append(k)
        order.append(o + a)
        sides.append(side.reshape(1))
    key, order = torch.cat(key), torch.cat(order)
    X = torch.stack([P[c][order] for c in "xyz"], 1)
    plo = torch.tensor(off[:-1], device="cuda")
    phi = torch.tensor(off[1:], device="cuda")
    side = torch.cat(sides)
    lev, base = [], 0
    for L in range(_LEVELS + 1):
        split = (phi - plo > _LEAF) & (L < _LEVELS)
        d = dict(plo=plo, phi=phi, side=side, first=torch.full_like(plo, -1), nch=torch.zeros_like(plo), base=base)
        lev.append(d)
        base += plo.numel()
        if not bool(split.any()):
            break
        pre = key >> (3 * (_LEVELS - L - 1))
        new = torch.ones_like(pre, dtype=torch.bool)
        new[1:] = pre[1:] != pre[:-1]
        new[plo] = True
        st = torch.nonzero(new).flatten()
        del pre, new
        pa = torch.searchsorted(plo, st, right=True) - 1
        ok = (pa >= 0) & split[pa] & (st < phi[pa])
        st, pa = st[ok], pa[ok]
        en = phi[pa].clone()
        same = pa[1:] == pa[:-1]
        en[:-1] = torch.where(same, st[1:], en[:-1])
        nch = torch.bincount(pa, minlength=plo.numel())
        d["nch"] = nch
        d["first"] = torch.where(nch > 0, base + nch.cumsum(0) - nch, -torch.ones_like(nch))
        d["kid_parent"] = pa
        plo, phi, side = st, en, 0.5 * side[pa]
    m = P["m"][order]
    val = [m[:, None], m[:, None] * X]
    if vel is not None:
        V = torch.stack([v[order] for v in vel], 1)
        val.append(m[:, None] * V)
    val = torch.cat(val, 1)
    soft = P["soft"][order]
    cols, mx, cnt = [None] * len(lev), [None] * len(lev), [None] * len(lev)
    allp = torch.cat([d["plo"][d["first"] < 0] for d in lev])
    leaf_start, perm = torch.sort(allp)
    leaf_val, leaf_mx = _cut(leaf_start, val, "sum"), _cut(leaf_start, soft, "amax")
    leaf_cnt = _cut(leaf_start, sink[order].to(F64), "sum") if sink is not None else None
    inv = torch.empty_like(perm)
    inv[perm] = torch.arange(perm.numel(), device="cuda")
    at = perm.numel()
    for L in range(len(lev) - 1, -1, -1):
        d = lev[L]
        isl = d["first"] < 0
        k = int(isl.sum())
        rows = inv[at - k:at]
        at -= k
        v = torch.zeros((isl.numel(), val.shape[1]), dtype=F64, device="cuda")
        s = torch.zeros(isl.numel(), dtype=F64, device="cuda")
        c = torch.zeros(isl.numel(), dtype=F64, device="cuda")
        v[isl], s[isl] = leaf_val[rows], leaf_mx[rows]
        if leaf_cnt is not None:
            c[isl] = leaf_cnt[rows]
        if "kid_parent" in d:
            v.index_add_(0, d["kid_parent"], cols[L + 1])
            s.scatter_reduce_(0, d["kid_parent"], mx[L + 1], "amax")
            c.index_add_(0, d["kid_parent"], cnt[L + 1])
        cols[L], mx[L], cnt[L] = v, s, c
    cols = torch.cat(cols)
    M = cols[:, 0]
    t = dict(order=order, X=X, m=m, soft=soft, plo=torch.cat([d["plo"] for d in lev]),
             phi=torch.cat([d["phi"] for d in lev]), first=torch.cat([d["first"] for d in lev]),
             nch=torch.cat([d["nch"] for d in lev]), len=torch.cat([d["side"] for d in lev]).float().to(F64),
             M=M, C=cols[:, 1:4] / M[:, None], nsoft=torch.cat(mx).float().to(F64), nsink=torch.cat(cnt),
             roots=len(off) - 1, off=off)
    if vel is not None:
        t.update(V=V, VC=cols[:, 4:7] / M[:, None])
    return t


def _spread(first, count):
    """The ranges [first, first + count) one after another, and which range each value is of."""
    who = torch.repeat_interleave(torch.arange(count.numel(), device="cuda"), count)
    return first[who] + torch.arange(who.numel(), device="cuda") - (count.cumsum(0) - count)[who], who


def _wk(u):
    """Force, potential and second-derivative factors of the cubic-spline kernel, u = r / h < 1."""
    u2, u3 = u * u, u * u * u
    lo = u < 0.5
    us = torch.clamp(u, min=1e-30)
    f = torch.where(lo, 32.0 / 3.0 + u2 * (32.0 * u - 38.4),
                    64.0 / 3.0 - 48.0 * u + 38.4 * u2 - 32.0 / 3.0 * u3 - 1.0 / (15.0 * us ** 3))
    p = torch.where(lo, -2.8 + u2 * (16.0 / 3.0 + u2 * (6.4 * u - 9.6)),
                    -3.2 + 1.0 / (15.0 * us) + u2 * (32.0 / 3.0 + u * (-16.0 + u * (9.6 - 32.0 / 15.0 * u))))
    g = torch.where(lo, 76.8 - 96.0 * u, -0.2 / us ** 5 + 48.0 / us - 76.8 + 32.0 * u)
    return f, p, g


def _dw(r, h):
    """dW/dr / r of the 3-D cubic spline of support h; 0 outside."""
    q = r / h
    g = torch.where(q < 0.5, 18.0 * q - 12.0, -6.0 * (1.0 - q) ** 2 / torch.clamp(q, min=1e-30))
    return torch.where(q < 1.0, 8.0 / math.pi * g / h ** 5, torch.zeros_like(q))


def _walk64(t, tpos, gs, ge, groot, aold, phi=False, tidal=False, jerk=False, gas=None, sink_r=0.0):
    """The grouped walk with the relative criterion in double; outputs per target."""
    nt, out = tpos.numel(), []
    K = int((ge - gs).max())
    names = 3 + int(phi) + (6 if tidal else 0) + (3 if jerk else 0)
    res = torch.zeros((nt, names), dtype=F64, device="cuda")
    step = max(1, (1 << 19) // K)
    for c0 in range(0, gs.numel(), step):
        s, e = gs[c0:c0 + step], ge[c0:c0 + step]
        G = s.numel()
        idx = s[:, None] + torch.arange(K, device="cuda")[None]
        ok = idx < e[:, None]
        idx = torch.where(ok, idx, s[:, None])  # a short group repeats its first target
        tp = tpos[idx]
        TX, TH = t["X"][tp], t["soft"][tp]
        lo, hi = TX.amin(1), TX.amax(1)
        mid, hw = 0.5 * (lo + hi), 0.5 * (hi - lo)
        emax, amin = TH.amax(1), aold[idx].amin(1)
        has_sink = (gas[0][tp] == 5).any(1) if gas is not None else None
        acc = torch.zeros((names, G, K), dtype=F64, device="cuda")
        gi = torch.arange(G, device="cuda")
        node = groot[c0:c0 + step].clone()
        while gi.numel():
            d = torch.clamp((t["C"][node] - mid[gi]).abs() - hw[gi], min=0.0)
            r2 = (d * d).sum(1)
            ln = t["len"][node]
            op = (r2 < (emax[gi] + 0.6 * ln) ** 2) | (r2 < (t["nsoft"][node] + 0.6 * ln) ** 2)
            op |= t["M"][node] * ln * ln > r2 * r2 * amin[gi]
            op |= (d < (0.6 * ln)[:, None]).all(1)
            if has_sink is not None and sink_r > 0:
                op |= has_sink[gi] & (t["nsink"][node] > 0) & (r2 < (sink_r + 0.6 * ln) ** 2)
            leaf = t["first"][node] < 0
            for part in (False, True):
                sel = (op & leaf) if part else ~op
                if not bool(sel.any()):
                    continue
                eg, en = gi[sel], node[sel]
                if part:
                    en, who = _spread(t["plo"][en], t["phi"][en] - t["plo"][en])
                    eg = eg[who]
                _add_entries(t, acc, eg, en, part, TX, TH, tp, phi, tidal, jerk, gas)
            go = op & ~leaf
            kids, who = _spread(t["first"][node[go]], t["nch"][node[go]])
            gi, node = gi[go][who], kids
        res[idx[ok]] = acc.permute(1, 2, 0)[ok]
    return res


def _add_entries(t, acc, eg, en, part, TX, TH, tp, phi, tidal, jerk, gas):
    K = TX.shape[1]
    cut = max(1, (1 << 24) // K)
    for a in range(0, eg.numel(), cut):
        g, e = eg[a:a + cut], en[a:a + cut]
        pos, mass = (t["X"][e], t["m"][e]) if part else (t["C"][e], t["M"][e])
        T = TX[g]
        d = [pos[:, None, k] - T[:, :, k] for k in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        z = r2 == 0
        ri = torch.where(z, torch.zeros_like(r2), 1.0 / torch.sqrt(torch.where(z, torch.ones_like(r2), r2)))
        mass = mass[:, None]
        mr = mass * ri
        g1, p, g2 = mr * ri * ri, -mr, None
        if tidal or jerk:
            g2 = 3.0 * g1 * ri * ri
        fa = g1
        if part:
            r = torch.sqrt(r2)
            h = torch.maximum(TH[g], t["soft"][e][:, None])
            ins = (r < h) & ~z
            if bool(ins.any()):
                f, q, w = _wk(torch.where(ins, r / h, torch.full_like(r, 0.5)))
                g1 = torch.where(ins, mass * f / h ** 3, g1)
                p = torch.where(ins, mass * q / h, p)
                if g2 is not None:
                    g2 = torch.where(ins, mass * w / h ** 5, g2)
            fa = g1
            if gas is not None:
                ty, ze = gas
                mt = t["m"][tp[g]]
                both = (ty[tp[g]] == 0) & (ty[e] == 0)[:, None] & ~z
                hs = t["soft"][e][:, None]
                corr = ze[tp[g]] / mt * _dw(r, h) + (ze[e][:, None] / mt) * _dw(r, hs)
                fa = g1 - torch.where(both, corr, torch.zeros_like(corr))
        q = [fa * d[0], fa * d[1], fa * d[2]]
        if phi:
            q.append(p)
        if tidal:
            q += [g2 * d[0] * d[0] - g1, g2 * d[1] * d[1] - g1, g2 * d[2] * d[2] - g1, g2 * d[0] * d[1],
                  g2 * d[1] * d[2], g2 * d[0] * d[2]]
        if jerk:
            ev = (t["V"] if part else t["VC"])[e]
            dv = [ev[:, None, k] - t["V"][tp[g]][:, :, k] for k in range(3)]
            vg = (dv[0] * d[0] + dv[1] * d[1] + dv[2] * d[2]) * g2
            q += [g1 * dv[k] - vg * d[k] for k in range(3)]
        for k, v in enumerate(q):
            acc[k].index_add_(0, g, v)


def _direct64(P, tg, fp=F64):
    out = [[], [], [], []]
    n = P["m"].numel()
    cut = max(1, (1 << 26) // n)
    for a in range(0, tg.numel(), cut):
        i = tg[a:a + cut].long()
        d = [P[k][None, :] - P[k][i][:, None] for k in "xyz"]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        z = r2 == 0
        r = torch.sqrt(torch.where(z, torch.ones_like(r2), r2))
        h = torch.maximum(P["soft"][None, :], P["soft"][i][:, None])
        ins = r < h
        f, p, _ = _wk(torch.where(ins, r / h, torch.full_like(r, 0.5)))
        f = torch.where(ins, f / h ** 3, 1.0 / r ** 3) * P["m"][None, :]
        p = torch.where(ins, p / h, -1.0 / r) * P["m"][None, :]
        f, p = torch.where(z, torch.zeros_like(f), f), torch.where(z, torch.zeros_like(p), p)
        for k in range(3):
            out[k].append((f * d[k]).sum(1))
        out[3].append(p.sum(1))
    return [torch.cat(o) for o in out]


def _density64(P, order, h0):
    """The density solve's Newton iteration over candidate pairs, all targets at once."""
    t = _octree(P, False)
    X, n = t["X"], order.numel()
    lo = torch.full((t["plo"].numel(), 3), 1e300, dtype=F64, device="cuda")
    hi = -lo
    leaves = torch.nonzero(t["first"] < 0).flatten()
    leaves = leaves[torch.sort(t["plo"][leaves])[1]]
    st = t["plo"][leaves]
    lo[leaves], hi[leaves] = torch.stack([_cut(st, X[:, k], "amin") for k in range(3)], 1), \
        torch.stack([_cut(st, X[:, k], "amax") for k in range(3)], 1)
    inner = torch.nonzero(t["first"] >= 0).flatten()
    for _ in range(_LEVELS):  # boxes grow from the leaves towards the root
        kid, who = _spread(t["first"][inner], t["nch"][inner])
        w = inner[who][:, None].expand(-1, 3)
        lo.scatter_reduce_(0, w, lo[kid], "amin")
        hi.scatter_reduce_(0, w, hi[kid], "amax")
    H, RHO = torch.empty(n, dtype=F64, device="cuda"), torch.empty(n, dtype=F64, device="cuda")
    todo, grow = torch.arange(n, device="cuda"), 1.35
    while todo.numel():
        again = []
        for a in range(0, todo.numel(), 1 << 17):
            i = todo[a:a + (1 << 17)]
            again.append(i[~_newton64(P, t, X, lo, hi, i, h0, grow, H, RHO)])
        todo, grow = torch.cat(again), grow * 1.5
        if grow > 50:
            return None
    return H, RHO


def _newton64(P, t, X, lo, hi, i, h0, grow, H, RHO):
    C, R = X[i], h0[i] * grow
    who, node = torch.arange(i.numel(), device="cuda"), torch.zeros_like(i)
    pw, pj = [], []
    while who.numel():
        d = torch.clamp(torch.maximum(lo[node] - C[who], C[who] - hi[node]), min=0.0)
        near = (d * d).sum(1) < R[who] ** 2
        who, node = who[near], node[near]
        leaf = t["first"][node] < 0
        j, w = _spread(t["plo"][node[leaf]], (t["phi"] - t["plo"])[node[leaf]])
        w = who[leaf][w]
        near = ((X[j] - C[w]) ** 2).sum(1) < R[w] ** 2
        pw.append(w[near])
        pj.append(j[near])
        kid, w = _spread(t["first"][node[~leaf]], t["nch"][node[~leaf]])
        who, node = who[~leaf][w], kid
    pw, pj = torch.cat(pw), torch.cat(pj)
    d = X[pj] - C[pw]
    r = torch.sqrt((d * d).sum(1))
    mj = t["m"][pj]
    n = i.numel()
    h, h_lo, h_hi = h0[i].clone(), torch.zeros(n, dtype=F64, device="cuda"), torch.zeros(n, dtype=F64, device="cuda")
    done = torch.zeros(n, dtype=torch.bool, device="cuda")
    fine = torch.ones(n, dtype=torch.bool, device="cuda")
    rho = torch.zeros(n, dtype=F64, device="cuda")
    for it in range(101):  # a target that has not converged in 100 gets one more evaluation, at its last h
        hp = h[pw]
        use = (r < hp) & ~done[pw]
        w_, r_, d_, m_, hp = pw[use], r[use], d[use], mj[use], hp[use]
        q = r_ / hp
        norm = 8.0 / (math.pi * hp ** 3)
        f = torch.where(q < 0.5, 1.0 - 6.0 * q * q + 6.0 * q ** 3, 2.0 * (1.0 - q) ** 3)
        fp = torch.where(q < 0.5, -12.0 * q + 18.0 * q * q, -6.0 * (1.0 - q) ** 2)
        w = norm * f
        cols = torch.stack([w, -3.0 / hp * w - q / hp * norm * fp, m_ * w, d_[:, 0] ** 2 * w, d_[:, 1] ** 2 * w,
                            d_[:, 2] ** 2 * w, d_[:, 0] * d_[:, 1] * w, d_[:, 1] * d_[:, 2] * w, d_[:, 0] * d_[:, 2] * w,
                            d_[:, 0] * w, d_[:, 1] * w, d_[:, 2] * w], 1)
        s = torch.zeros((n, 12), dtype=F64, device="cuda").index_add_(0, w_, cols)
        ws, dh, xx, yy, zz, xy, yz, xz = (s[:, k] for k in (0, 1, 3, 4, 5, 6, 7, 8))
        B = torch.stack([yy * zz - yz * yz, xz * yz - xy * zz, xy * yz - xz * yy, xz * yz - xy * zz, xx * zz - xz * xz,
                         xy * xz - xx * yz, xy * yz - xz * yy, xy * xz - xx * yz, xx * yy - xy * xy], 1)
        det = xx * B[:, 0] - xy * (xy * zz - yz * xz) + xz * (xy * yz - yy * xz)
        good = (ws > 0) & (det != 0)
        vol = 1.0 / torch.where(ws > 0, ws, torch.ones_like(ws))
        leak = (B.view(n, 3, 3) @ s[:, 9:12, None]).squeeze(2) * (2.0 * vol / torch.where(good, det, torch.ones_like(det)))[:, None]
        fce = leak.abs().sum(1) / 3.0 / (6.0 * vol * (xx + yy + zz))
        nc = torch.where(good & (fce > 0.35), torch.clamp(fce / 0.35, 1.0, 2.0), torch.ones_like(ws))
        des, tol = 32.0 * nc, 0.05 * nc
        if it > 1:
            tol = torch.minimum(0.25 * des, tol * torch.exp(0.1 * torch.log(des / (16.0 * tol)) * it))
        ball = 4.0 * math.pi / 3.0 * h ** 3
        res = ball * ws - des
        conv = ~done & (res.abs() < tol)
        rho = torch.where(done, rho, s[:, 2])
        done |= conv
        if it == 100 or bool(done.all()):
            break
        h_hi = torch.where(~done & (res > 0), h, h_hi)
        h_lo = torch.where(~done & ~(res > 0), h, h_lo)
        dn = ball * (3.0 / h * ws + dh)
        hn = torch.where(dn > 0, h - res / dn, torch.zeros_like(h))
        out = (hn <= h_lo) | ((h_hi > 0) & (hn >= h_hi)) | (hn <= 0)
        half = torch.where(h_lo > 0, torch.sqrt(h_lo * h_hi), 0.5 * h_hi)
        alt = torch.where(h_hi > 0, half, h * torch.where(res > 0, 0.7, 1.6))
        h = torch.where(done, h, torch.where(out, alt, hn))
        over = ~done & (h > R)  # outgrew its candidates: again, with more
        fine &= ~over
        done |= over
    H[i[fine]], RHO[i[fine]] = h[fine], rho[fine]
    return fine


def exact(case, seed):
    s = prepare(case, seed)
    kind, P = s["kind"], s["P"]
    if kind == "lists":
        return None  # whole numbers
    if kind == "direct":
        return tuple(_direct64(P, s["targets"]))
    if kind == "density":
        got = _density64(P, s["targets"].long(), s["h"])
        return None if got is None else {"h": got[0], "rho": got[1], "nngb": None, "iters": None}
    nt = float(case.get("targets", case["n"]))
    if nt * _interactions(case) * (3.0 if kind == "ext" else 1.0) > 1.2e10:
        return None  # the sums in double take too long
    off = _forest(case, seed)[1] if kind == "forest" else None
    vel = _velocities(seed, P["m"].numel()) if kind == "ext" else None
    sink = s["type"] == 5 if kind == "gas" else None
    t = _octree(P, kind != "engine", off=off, vel=vel, sink=sink)
    n = t["order"].numel()
    aold = torch.as_tensor(s["aold"], device="cuda")
    leaf_start = torch.sort(t["plo"][t["first"] < 0])[0]
    if kind == "active":
        rank = torch.empty_like(t["order"])
        rank[t["order"]] = torch.arange(n, device="cuda")
        tpos = rank[s["targets"].long()]
        leaf = torch.searchsorted(leaf_start, tpos, right=True)
        new = torch.ones_like(leaf, dtype=torch.bool)
        new[1:] = leaf[1:] != leaf[:-1]
        gs = torch.nonzero(new).flatten()
    else:
        tpos = torch.arange(n, device="cuda")
        b = int(case["batch"])
        gs = leaf_start if b == 0 else torch.cat([torch.arange(a, e, b, device="cuda")
                                                  for a, e in zip(t["off"][:-1], t["off"][1:])])
    ge = torch.cat([gs[1:], torch.tensor([tpos.numel()], device="cuda")])
    if kind != "active" and int(case["batch"]) == 0:  # coinciding particles: longer leaves go in runs of 32
        k = (ge - gs + 31) // 32
        _, who = _spread(torch.zeros_like(gs), k)
        run_ = torch.arange(who.numel(), device="cuda") - (k.cumsum(0) - k)[who]
        gs, ge = gs[who] + 32 * run_, torch.minimum(gs[who] + 32 * run_ + 32, ge[who])
    groot = torch.searchsorted(torch.tensor(t["off"], device="cuda"), tpos[gs], right=True) - 1
    gas = None
    if kind == "gas":
        gas = (s["type"][t["order"]], s["zeta"][t["order"]])
    ext = kind == "ext"
    r = _walk64(t, tpos, gs, ge, groot, aold, phi=bool(case.get("phi")), tidal=ext, jerk=ext and case["jerk"], gas=gas,
                sink_r=float(case.get("sink_radius", 0.0)))
    out = [r[:, 0], r[:, 1], r[:, 2]]
    if case.get("phi"):
        out.append(r[:, 3])
    if ext:
        out.append(r[:, 3:9])
        if case["jerk"]:
            out.append(r[:, 9:12])
    return [v.contiguous() for v in out]
