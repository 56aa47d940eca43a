"""Neighbour search and the density solve on the GPU tree (shmem::ngb_search, ngb_search_reverse,
density: shmem/hydro.cc:37-327; Tree::init_hmax / raise_hmax: tree.cc:287-338), against the
reference's own results (golden fixtures ``ngb_*``) and the oracle restatement.

Bars: neighbour lists are integer results and must be bit-identical, in the same order (tree
order).  The density solve is FP64 in the reference's accumulation order; the reference's compiler
may contract multiply-adds where the device does not, so per target h and rho agree to 1e-10
relative and the iteration and neighbour counts are identical wherever the iteration took the same
path -- which must be at least 99.5 % of the targets (a last-ulp difference can move a residual
across the tolerance).
"""
import numpy as np
import pytest

import gizmo_shared_memory_b200 as g

pytestmark = pytest.mark.gpu


def particles(golden, prefix="ngb"):
    P = {k: golden[f"{prefix}_{k}"] for k in ("x", "y", "z", "m")}
    P["soft"] = np.full_like(P["m"], 0.01)
    return P


@pytest.fixture(scope="module")
def ngb_tree(gpu_ctx, golden):
    T = gpu_ctx.build(particles(golden), key_mode=g.GT_KEY_MORTON)
    gpu_ctx.tree_gas(T, golden["ngb_type"], None)
    n_gas = int(golden["ngb_n_gas"][0])
    gpu_ctx.tree_hmax(T, golden["ngb_h_part"][:n_gas], n_gas)
    return T


@pytest.mark.parametrize("mode,name", [(g.GT_NGB_GATHER, "gather"), (g.GT_NGB_REVERSE, "reverse"),
                                       (g.GT_NGB_PAIRS, "pairs")])
def test_search_matches_reference(gpu_ctx, golden, ngb_tree, mode, name):
    cen = [golden[f"ngb_c{k}"] for k in "xyz"]
    n_gas = int(golden["ngb_n_gas"][0])
    st, f = gpu_ctx.ngb_search(ngb_tree, *cen, golden["ngb_radius"], mode=mode, h=golden["ngb_h_part"][:n_gas],
                               n_gas=n_gas)
    assert np.array_equal(st, golden[f"ngb_{name}_start"])
    assert np.array_equal(f, golden[f"ngb_{name}_found"])


def test_periodic_search_matches_reference(gpu_ctx, golden):
    T = gpu_ctx.build(particles(golden, "ngb_box"), key_mode=g.GT_KEY_MORTON)
    cen = [golden[f"ngb_c{k}"] for k in "xyz"]
    st, f = gpu_ctx.ngb_search(T, *cen, 0.5 * golden["ngb_radius"], box=2.0)
    assert np.array_equal(st, golden["ngb_box_gather_start"])
    assert np.array_equal(f, golden["ngb_box_gather_found"])


def check_density(d, golden, case):
    same = d["iters"] == golden[f"ngb_{case}_iters"]
    assert same.mean() >= 0.995, same.mean()
    assert np.array_equal(d["nngb"][same], golden[f"ngb_{case}_nngb"][same])
    for k in ("h", "rho"):
        ref = golden[f"ngb_{case}_{k}"]
        e = np.abs(d[k] - ref) / np.abs(ref)
        assert e[same].max() <= 1e-10, (k, e[same].max())
        assert np.median(e) <= 1e-12


@pytest.mark.parametrize("case", ["cold", "warm", "cond"])
def test_density_matches_reference(gpu_ctx, golden, ngb_tree, case):
    kw = {}
    if case == "warm":
        kw["h_start"] = 1.1 * golden["ngb_cold_h"]
    if case == "cond":
        kw["cond_prev"] = golden["ngb_cond"]
    d = gpu_ctx.density(ngb_tree, golden["ngb_targets"], 32.0, 0.05, **kw)
    check_density(d, golden, case)


@pytest.mark.parametrize("case,dim", [("d2", 2), ("d1", 1)])
def test_low_dimension_density_matches_reference(gpu_ctx, golden, case, dim):
    """A sheet and a line with the 2-D and 1-D kernels (hydro.h:28-37, hydro.cc:172-177)."""
    T = gpu_ctx.build(particles(golden, f"ngb_{case}"), key_mode=g.GT_KEY_MORTON)
    d = gpu_ctx.density(T, golden[f"ngb_{case}_targets"], 12.0 if dim == 2 else 5.0, 0.05, n_dims=dim)
    check_density(d, golden, case)


def test_periodic_density_matches_reference(gpu_ctx, golden):
    T = gpu_ctx.build(particles(golden, "ngb_box"), key_mode=g.GT_KEY_MORTON)
    d = gpu_ctx.density(T, golden["ngb_box_targets"], 32.0, 0.05, box=2.0)
    check_density(d, golden, "box")


def test_search_matches_oracle_at_scale(gpu_ctx, oracle):
    """200k clustered particles, 20k centres with radii over two decades: the GPU lists equal the
    oracle restatement's, entry for entry, in all three modes; the raised hmax of a later
    GT_EVENT_HMAX is honoured."""
    from gizmo_shared_memory_b200 import ics

    P = ics.plummer(n=200000, seed=8, soft=0.01)
    P["m"][::101] = 0.0
    T = gpu_ctx.build(P, key_mode=g.GT_KEY_MORTON)
    OT = oracle.build(P)
    rng = np.random.default_rng(4)
    n_gas = 150000
    h = rng.uniform(0.01, 0.2, 200000)
    gpu_ctx.tree_hmax(T, h[:n_gas], n_gas)
    idx = rng.choice(200000, 20000, replace=False)
    cen = [P[k][idx] + rng.normal(0, 0.01, 20000) for k in "xyz"]
    rad = 10 ** rng.uniform(-2.5, -0.5, 20000)
    for mode in (g.GT_NGB_GATHER, g.GT_NGB_REVERSE, g.GT_NGB_PAIRS):
        a = gpu_ctx.ngb_search(T, *cen, rad, mode=mode, h=h[:n_gas], n_gas=n_gas)
        b = OT.ngb_search(*cen, rad, mode=mode, h=h[:n_gas], n_gas=n_gas)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]), mode
    # raise the support radius of a few gas particles (Tree::raise_hmax), then search again
    up = rng.choice(n_gas, 500, replace=False)
    up = up[P["m"][up] > 0]
    h2 = h.copy()
    h2[up] *= 3.0
    leaf = T.download()["leaf_of"][up]
    gpu_ctx.tree_events(T, g._gt.GT_EVENT_HMAX, leaf, a=h2[up])
    a = gpu_ctx.ngb_search(T, *cen, rad, mode=g.GT_NGB_REVERSE, h=h2[:n_gas], n_gas=n_gas)
    b = OT.ngb_search(*cen, rad, mode=g.GT_NGB_REVERSE, h=h2[:n_gas], n_gas=n_gas)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


def test_density_matches_oracle_at_scale(gpu_ctx, oracle):
    """A 100k Plummer sphere, every particle gas, cold start: the GPU solve agrees with the oracle
    restatement to the same bars as against the reference."""
    from gizmo_shared_memory_b200 import ics

    P = ics.plummer(n=100000, seed=9, soft=0.01)
    T = gpu_ctx.build(P, key_mode=g.GT_KEY_MORTON)
    OT = oracle.build(P)
    tg = OT.order()[0]
    d = gpu_ctx.density(T, tg)
    o = OT.density(tg)
    same = d["iters"] == o["iters"]
    assert same.mean() >= 0.995
    assert np.array_equal(d["nngb"][same], o["nngb"][same])
    for k in ("h", "rho"):
        e = np.abs(d[k] - o[k]) / np.abs(o[k])
        assert e[same].max() <= 1e-10 and np.median(e) <= 1e-12, k


def test_errors(gpu_ctx, golden):
    T = gpu_ctx.build(particles(golden), key_mode=g.GT_KEY_MORTON)
    one = np.zeros(1)
    with pytest.raises(g.GTError):  # the reverse search needs hmax
        gpu_ctx.ngb_search(T, one, one, one, one + 0.1, mode=g.GT_NGB_REVERSE, h=np.ones(10), n_gas=10)
    st, f = gpu_ctx.ngb_search(T, one[:0], one[:0], one[:0], one[:0])
    assert st.tolist() == [0] and f.size == 0
    with pytest.raises(g.GTError):
        gpu_ctx.density(T, np.array([0], np.uint32), n_dims=4)


@pytest.fixture(scope="module")
def ngb_counts():
    import os

    here = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "ngb_counts.npz")
    return dict(np.load(here))


def test_counters_match_reference(gpu_ctx, golden, ngb_tree, ngb_counts):
    """SHMEM_NGB_COUNT (hydro.cc:7-35): the totals of the reference's own search and solve on the
    same inputs (tests/golden/ngb_counts.npz).  The counts are integers over the same traversal in
    the same node order: nodes visited, particles examined, neighbours kept and pad-only nodes are
    identical, and so is the density's iteration histogram wherever every target took the
    reference's number of iterations (else within the targets that did not)."""
    cen = [golden[f"ngb_c{k}"] for k in "xyz"]
    rad = golden["ngb_radius"]
    n_gas = int(golden["ngb_n_gas"][0])
    gpu_ctx.ngb_count(True)
    try:
        gpu_ctx.ngb_counters(reset=True)
        gpu_ctx.ngb_search(ngb_tree, *cen, rad)
        c = gpu_ctx.ngb_counters(reset=True)
        ref = ngb_counts["gather"]
        assert [c["calls"], c["nodes"], c["examined"], c["kept"], c["pad_nodes"]] == ref[:5].tolist()
        assert not c["hiter"].any()
        # the reverse search is not counted; a pair search counts its gather half
        gpu_ctx.ngb_search(ngb_tree, *cen, rad, mode=g.GT_NGB_PAIRS, h=golden["ngb_h_part"][:n_gas], n_gas=n_gas)
        c = gpu_ctx.ngb_counters(reset=True)
        assert [c["calls"], c["nodes"], c["examined"], c["kept"], c["pad_nodes"]] == ref[:5].tolist()
        # a stale tree: the vmax * elapsed pad admits nodes that only it admits
        T = gpu_ctx.build(particles(golden), key_mode=g.GT_KEY_MORTON)
        gpu_ctx.tree_velocities(T, ngb_counts["vx"], ngb_counts["vy"], ngb_counts["vz"])
        el = float(ngb_counts["stale_elapsed"][0])
        st, f = gpu_ctx.ngb_search(T, *cen, rad, elapsed=el)
        assert np.array_equal(st, ngb_counts["stale_start"]) and np.array_equal(f, ngb_counts["stale_found"])
        c = gpu_ctx.ngb_counters(reset=True)
        ref = ngb_counts["stale"]
        assert ref[4] > 0
        assert [c["calls"], c["nodes"], c["examined"], c["kept"], c["pad_nodes"]] == ref[:5].tolist()
        # the density solve: one gather search per evaluation, and the iteration histogram
        d = gpu_ctx.density(ngb_tree, golden["ngb_targets"], 32.0, 0.05)
        c = gpu_ctx.ngb_counters(reset=False)
        ref = ngb_counts["density"]
        it = d["iters"]
        assert c["calls"] == int((it + 1).sum())
        used = np.where(it < 100, it + 1, 100)
        assert np.array_equal(c["hiter"], np.bincount(np.minimum(used, 8) - 1, minlength=8))
        if np.array_equal(it, golden["ngb_cold_iters"]):
            assert [c["calls"], c["nodes"], c["examined"], c["kept"], c["pad_nodes"]] == ref[:5].tolist()
            assert np.array_equal(c["hiter"], ref[5:])
        else:
            for k, i in (("calls", 0), ("nodes", 1), ("examined", 2), ("kept", 3)):
                assert abs(c[k] - ref[i]) <= 0.01 * ref[i], k
        # reading without reset keeps the totals; counting off adds nothing
        assert gpu_ctx.ngb_counters(reset=True)["calls"] == c["calls"]
        gpu_ctx.ngb_count(False)
        gpu_ctx.ngb_search(ngb_tree, *cen, rad)
        assert gpu_ctx.ngb_counters()["calls"] == 0
    finally:
        gpu_ctx.ngb_count(False)


@pytest.mark.parametrize("case", ["cold", "warm", "cond", "box"])
def test_candidate_cache_is_bit_identical(gpu_ctx, golden, ngb_tree, case):
    """The density solve scans a per-thread cache of one search's gas candidates when a Newton step
    shrinks h below the cached radius.  It keeps the particles, the order and the r^2 test of a
    search at h, so h, rho, the neighbour counts and the iterations are bit-identical to the
    solve that searches at every evaluation (the counting variant, SHMEM_NGB_COUNT on)."""
    kw = {}
    T = ngb_tree
    tg = golden["ngb_targets"]
    if case == "warm":
        kw["h_start"] = 1.1 * golden["ngb_cold_h"]
    if case == "cond":
        kw["cond_prev"] = golden["ngb_cond"]
    if case == "box":
        T = gpu_ctx.build(particles(golden, "ngb_box"), key_mode=g.GT_KEY_MORTON)
        tg = golden["ngb_box_targets"]
        kw["box"] = 2.0
    cached = gpu_ctx.density(T, tg, 32.0, 0.05, **kw)
    gpu_ctx.ngb_count(True)
    try:
        direct = gpu_ctx.density(T, tg, 32.0, 0.05, **kw)
    finally:
        gpu_ctx.ngb_count(False)
    for k in ("h", "rho", "nngb", "iters"):
        assert np.array_equal(cached[k], direct[k]), k


@pytest.mark.parametrize("nt", [1, 15, 16, 17, 33, 300, 3000])
@pytest.mark.parametrize("guess", ["close", "wide", "whole", "nan"])
def test_density_lanes_and_warps_match_counting_solve(gpu_ctx, nt, guess):
    """The solve takes targets into its lanes sixteen or more at a time and hands those with more than
    160 candidates to a warp, whose own cache holds 2048: target counts around the lanes, and first
    guesses with tens, hundreds and all 6000 particles inside, on a clump in a sparse box.  h, rho, the
    neighbour counts and the iterations equal the counting solve's, a thread per target, bit for bit;
    an h that is not a number ends after 100 iterations there and here."""
    rng = np.random.default_rng(7)
    x = np.concatenate([0.02 * rng.normal(size=(3000, 3)), rng.uniform(-1, 1, (3000, 3))])
    P = {"x": x[:, 0].copy(), "y": x[:, 1].copy(), "z": x[:, 2].copy(), "m": rng.uniform(0.5, 1.5, 6000)}
    T = gpu_ctx.build(P, key_mode=g.GT_KEY_MORTON)
    tg = rng.choice(6000, nt, replace=False).astype(np.uint32)
    h = {"close": np.where(tg < 3000, 0.01, 0.3), "wide": np.full(nt, 0.1), "whole": np.full(nt, 5.0),
         "nan": np.full(nt, np.nan)}[guess]
    if guess == "nan":
        tg, h = tg[:33], h[:33]
    got = gpu_ctx.density(T, tg, h_start=h)
    gpu_ctx.ngb_count(True)
    try:
        want = gpu_ctx.density(T, tg, h_start=h)
    finally:
        gpu_ctx.ngb_count(False)
    for k in ("h", "rho", "nngb", "iters"):
        assert np.array_equal(got[k], want[k], equal_nan=k in ("h", "rho")), k


def search64(d, root, P, cen, rad):
    """The reference's gather search over downloaded nodes and the particles' present positions, its
    prune in FP64 on float boxes (hydro.cc:51-106): the lists of the centres."""
    f32 = np.float32
    box = np.stack([d[k].astype(f32) for k in ("gcx", "gcy", "gcz")], 1).astype(float)
    top = np.max(np.abs(np.stack([d[k] for k in ("gcx", "gcy", "gcz")], 1)), axis=1)
    half = (0.5 * d["size"] + 1e-6 * root + 4.0 * np.finfo(f32).eps * top).astype(f32).astype(float)
    X = np.stack([P[k] for k in "xyz"], 1)[d["orderbuf"]]
    lists = []
    for c, r in zip(np.stack(cen, 1), rad):
        node, found = 0, []
        while node >= 0:
            o, dist = np.abs(box[node] - c), r + half[node]
            if (o > dist).any() or (o * o).sum() > (dist + 0.7320508075688772 * half[node]) ** 2:
                node = d["next"][node]
            elif d["first"][node] < 0:
                s = np.arange(d["plo"][node], d["phi"][node])
                found.append(d["orderbuf"][s[((X[s] - c) ** 2).sum(1) < r * r]])
                node = d["next"][node]
            else:
                node = d["first"][node]
        lists.append(np.concatenate(found))
    return lists


def test_counted_lists_of_moved_particles(gpu_ctx):
    """Lists longer than the counting pass keeps are found again, by the same prune: on a tree whose
    particles moved out of their boxes with no pad for it, a leaf that the counted search's FP64 prune
    leaves out by four parts in 10^7 belongs to the wider FP32 prune of the plain search, and entries
    found by one pass and not by the other would end up in the next centre's list."""
    rng = np.random.default_rng(3)
    x = np.concatenate([0.02 * rng.normal(size=(1200, 3)), [0.7, 1e-3, 1e-3] + 1e-4 * rng.normal(size=(10, 3)),
                        rng.uniform(-1, 1, (800, 3))])
    P = {k: x[:, i].copy() for i, k in enumerate("xyz")}
    P["m"] = np.ones(len(x))
    T = gpu_ctx.build(P, key_mode=g.GT_KEY_MORTON)
    d = T.download()
    leaf = d["leaf_of"][1200]
    gone = np.nonzero(d["leaf_of"] == leaf)[0]
    for k in "xyz":
        P[k][gone] = 0.01 * rng.normal(size=len(gone))
    gpu_ctx.tree_particles(T, *(P[k] for k in "xyz"))
    cen = [np.linspace(-0.05, 0.05, 40), np.full(40, d["gcy"][leaf]), np.full(40, d["gcz"][leaf])]
    half = 0.5 * d["size"][leaf] + 1e-6 * d["size"][0] + 4.0 * np.finfo(np.float32).eps * d["gcx"][leaf]
    rad = (np.float64(np.float32(d["gcx"][leaf])) - cen[0] - half) * (1.0 - 4e-7)
    plain = np.diff(gpu_ctx.ngb_search(T, *cen, rad)[0])
    gpu_ctx.ngb_count(True)
    try:
        st, f = gpu_ctx.ngb_search(T, *cen, rad)
    finally:
        gpu_ctx.ngb_count(False)
    want = search64(d, d["size"][0], P, cen, rad)
    assert min(len(w) for w in want) > 64  # past what the counting pass keeps
    assert (plain > np.diff(st)).any()     # the two prunes differ here
    assert np.array_equal(np.diff(st), [len(w) for w in want]) and np.array_equal(f, np.concatenate(want))


@pytest.mark.parametrize("power", [-70, -40, 40, 70])
def test_search_and_density_scale_with_the_lengths(gpu_ctx, power):
    """Lengths times a power of two change no decision: the prune's squares leave the FP32 range at 2^-70
    (below 1e-45) and at 2^70, and may then admit nodes that hold nothing but must not drop any.  The lists,
    the iterations and the neighbour counts stay; h and the density, whose iteration takes roots and
    exponentials, scale to this file's 1e-10."""
    f = 2.0 ** power
    rng = np.random.default_rng(11)
    x = np.concatenate([0.05 * rng.normal(size=(3000, 3)), rng.uniform(-1, 1, (3000, 3))])
    m = rng.uniform(0.5, 1.5, 6000)
    rad = 10 ** rng.uniform(-2.5, -0.5, 6000)
    tg = np.arange(6000, dtype=np.uint32)
    r = []
    for s in (1.0, f):
        P = {k: x[:, i] * s for i, k in enumerate("xyz")}
        P["m"] = m
        T = gpu_ctx.build(P, key_mode=g.GT_KEY_MORTON)
        hs = rad * s
        gpu_ctx.tree_hmax(T, hs, 6000)
        r.append([gpu_ctx.ngb_search(T, *(P[k] for k in "xyz"), hs),
                  gpu_ctx.ngb_search(T, *(P[k] for k in "xyz"), 0.5 * hs, mode=g.GT_NGB_PAIRS, h=hs, n_gas=6000),
                  gpu_ctx.density(T, tg, h_start=0.1 * s * np.ones(6000))])
    for a, b in zip(r[0][:2], r[1][:2]):
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    a, b = r[0][2], r[1][2]
    assert np.array_equal(a["iters"], b["iters"]) and np.array_equal(a["nngb"], b["nngb"])
    assert np.abs(a["h"] * f / b["h"] - 1).max() <= 1e-10 and np.abs(b["rho"] * f ** 3 / a["rho"] - 1).max() <= 1e-10


@pytest.mark.parametrize("scale", [1e-9, 1.0, 1e9])
def test_density_weights_in_ulps(gpu_ctx, scale):
    """One particle outweighs all others by 1e30, so a target's density is that one's kernel weight at the h
    the solve ends with: 8 / (pi h^3) times the spline of q = r / h, against extended precision.  r by the
    root of the sum of squares, q by the reciprocal of h and the norm are each a few roundings (2^-53) off,
    which the spline passes on q f'/f times: 16 + 4 q f'/f roundings."""
    rng = np.random.default_rng(5)
    x = scale * rng.uniform(-1, 1, (2000, 3))
    heavy = int(np.argmin((x ** 2).sum(1)))
    P = {k: x[:, i].copy() for i, k in enumerate("xyz")}
    P["m"] = np.full(2000, 1e-30)
    P["m"][heavy] = 1.0
    T = gpu_ctx.build(P, key_mode=g.GT_KEY_MORTON)
    near = np.argsort(((x - x[heavy]) ** 2).sum(1))[1:40].astype(np.uint32)
    d = gpu_ctx.density(T, near, h_start=np.full(39, 0.5 * scale))
    X, h = x.astype(np.longdouble), d["h"].astype(np.longdouble)
    q = np.sqrt(((X[near] - X[heavy]) ** 2).sum(1)) / h
    q, rho, h = q[q < 0.98], d["rho"][q < 0.98], h[q < 0.98]
    assert len(q) >= 15 and (q < 0.5).any() and (q > 0.5).any()
    low = q < 0.5
    f = np.where(low, 1 - 6 * q * q + 6 * q ** 3, 2 * (1 - q) ** 3)
    slope = np.where(low, 12 * q - 18 * q * q, 6 * (1 - q) ** 2)
    pi = np.longdouble("3.14159265358979323846264338327950288")
    e = np.abs(rho / (8 / (pi * h ** 3) * f) - 1)
    assert (e <= (16 + 4 * q * slope / f) * 2.0 ** -53).all()
