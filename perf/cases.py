"""The work that users have this engine do, as timed cases.

Each case is one call (or one step) through the public entry points of
``kiddo_b200`` on inputs resident where a program holds them: device tensors
for the device-side API, pinned host arrays for the host-buffer API.  Data are
the distributions of the repository's benchmark (Gaussian mixtures, periodic
particles, catalogues on the sphere, noisy planes and spheres) and plain
uniform points, drawn on the GPU from the seed alone.  Trees are built on the
device, as a program with device points does, and kept like a program keeps
them.
"""
import math

import numpy as np
import torch

import kiddo_b200 as kb
from kiddo_b200 import chamfer

TORCH = {"f32": torch.float32, "f64": torch.float64}
SIZE = {"f32": 4, "f64": 8}
METRIC = {"sq": kb.SquaredEuclidean, "manhattan": kb.Manhattan}


def listed():
    return [
        # an interactive program asking for a handful of neighbours per call:
        # latency, launches and host work are all there is
        dict(name="knn8_small_call", kind="knn", dtype="f32", dims=3, data="uniform", n=10_000,
             nq=64, k=8, metric="sq"),
        # the reference's plain benchmark shape: a tree that sits in cache,
        # nearest_one in f64
        dict(name="nearest_one_f64", kind="one", dtype="f64", dims=3, data="uniform", n=100_000,
             nq=1_000_000, approx=False, metric="sq"),
        # the benchmark's default workload: 16 neighbours in a clustered f32 cloud
        dict(name="knn16_mixture", kind="knn", dtype="f32", dims=3, data="mixture",
             n=16_000_000, nq=16_000_000, k=16, metric="sq"),
        # the same tree asked for the approximate nearest point (one leaf per query)
        dict(name="approx_mixture", kind="one", dtype="f32", dims=3, data="mixture",
             n=16_000_000, nq=16_000_000, approx=True, metric="sq"),
        # planar data of odd sizes with the other common metric
        dict(name="knn10_planar_odd", kind="knn", dtype="f32", dims=2, data="uniform",
             n=1_000_003, nq=300_007, k=10, metric="manhattan"),
        # neighbour lists of a particle simulation: every particle of a
        # periodic f64 box, 32 nearest within a cutoff
        dict(name="periodic_lists_f64", kind="periodic", dtype="f64", n=16_000_000,
             nq=16_000_000, k=32, radius=0.01),
        # a cross-match of one catalogue at a fixed angular radius, hits sorted
        dict(name="catalogue_match", kind="within", dtype="f32", n=4_000_000, nq=1_000_003,
             chord=3e-4, sort=True),
        # many catalogues of uneven size in one batch, a radius per query
        dict(name="forest_radius", kind="forest", n=6_000_000, trees=32, nq=1_000_000,
             family="within"),
        # the same, keeping the five best-ranked entries within each radius
        dict(name="forest_best5", kind="forest", n=6_000_000, trees=32, nq=4_000_000,
             family="best"),
        # one training step's neighbour loss over a batch of cloud pairs:
        # forward, and both gradients
        dict(name="chamfer8_step", kind="chamfer", pairs=16, n_src=2_000_000, k=8),
        # queries and results in host memory, as a CPU program calls it
        dict(name="knn16_host_buffers", kind="host", dtype="f32", n=4_000_000, nq=2_000_000,
             k=16),
        # (re)building the benchmark's tree from points already on the device
        dict(name="build_mixture", kind="build", dtype="f32", dims=3, data="mixture",
             n=16_000_000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["knn", "knn", "one", "periodic", "within", "forest", "chamfer", "host",
                       "build"])
    if kind in ("knn", "one"):
        c = dict(kind=kind, dtype=rng.choice(["f32", "f32", "f64"]),
                 dims=rng.choice([2, 3, 3, 3]), data=rng.choice(["uniform", "mixture"]),
                 n=_log(rng, 1e4, 1.6e7), nq=_log(rng, 50, 1.2e7),
                 metric=rng.choice(["sq", "sq", "manhattan"]))
        if kind == "knn":
            c["k"] = rng.choice([2, 4, 5, 8, 10, 16])
        else:
            c["approx"] = rng.random() < 0.4
        return c
    if kind == "periodic":
        n = _log(rng, 1e5, 1.2e7)
        return dict(kind=kind, dtype=rng.choice(["f64", "f64", "f32"]), n=n,
                    nq=rng.choice([n, _log(rng, 1e3, n)]), k=rng.choice([12, 24, 32]),
                    radius=rng.choice([0.01, 0.001]))
    if kind == "within":
        n = _log(rng, 2e4, 4e6)
        # about the listed case's number of hits per query or fewer
        return dict(kind=kind, dtype=rng.choice(["f32", "f64"]), n=n, nq=_log(rng, 200, 1.5e6),
                    chord=3e-4 * math.sqrt(4e6 / n) * rng.uniform(0.3, 1.0),
                    sort=rng.random() < 0.6)
    if kind == "forest":
        trees = rng.randint(2, 48)
        return dict(kind=kind, n=max(20_000 * trees, _log(rng, 2e5, 6e6)), trees=trees,
                    nq=_log(rng, 1e4, 9e5), family=rng.choice(["within", "unsorted", "best"]))
    if kind == "chamfer":
        pairs = rng.randint(1, 16)
        return dict(kind=kind, pairs=pairs, n_src=_log(rng, 1e4 * pairs, 2e6),
                    k=rng.choice([1, 4, 8]))
    if kind == "host":
        return dict(kind=kind, dtype=rng.choice(["f32", "f64"]), n=_log(rng, 1e5, 4e6),
                    nq=_log(rng, 1e3, 3e6), k=rng.choice([4, 8, 16]))
    return dict(kind=kind, dtype=rng.choice(["f32", "f32", "f64"]), dims=rng.choice([2, 3, 3]),
                data=rng.choice(["uniform", "mixture"]), n=_log(rng, 5e4, 1.2e7))


# ---- inputs -----------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)


def _mixture(g, n, dims, centres, weights):
    """1,024 Gaussian clumps of sigma 0.005 and Dirichlet(1) weights, and a
    20% uniform background (the benchmark's default cloud)."""
    lab = torch.searchsorted(torch.cumsum(weights, 0), _rand(g, n)).clamp_(max=len(weights) - 1)
    p = centres[lab].add_(_randn(g, n, dims), alpha=0.005)
    return torch.where(_rand(g, n, 1) < 0.2, _rand(g, n, dims), p)


def _cloud(g, case, dims):
    """Points and queries of one distribution."""
    if case["data"] == "uniform":
        p, q = _rand(g, case["n"], dims), _rand(g, case.get("nq", 0), dims)
    else:
        centres = _rand(g, 1024, dims)
        w = -torch.log(1.0 - _rand(g, 1024))
        w /= w.sum()
        p = _mixture(g, case["n"], dims, centres, w)
        q = _mixture(g, case.get("nq", 0), dims, centres, w)
    dt = TORCH[case["dtype"]]
    return p.to(dt), q.to(dt)


def _particles(g, n, centres):
    """70% of the particles in 4,096 clumps of sigma 0.002 wrapped into the
    unit box, 30% uniform."""
    lab = torch.randint(0, len(centres), (n,), generator=g, device="cuda")
    p = torch.where(_rand(g, n, 1) < 0.7, centres[lab].add_(_randn(g, n, 3), alpha=0.002),
                    _rand(g, n, 3))
    p = torch.remainder(p, 1.0)
    return torch.where(p >= 1.0, torch.zeros_like(p), p)


def _periodic_points(g, case):
    """The particles, and the ones that query (all, or a sample of them)."""
    p = _particles(g, case["n"], _rand(g, 4096, 3)).to(TORCH[case["dtype"]])
    p = torch.where(p >= 1.0, torch.zeros_like(p), p)  # f64 to f32 can round up to the edge
    if case["nq"] == case["n"]:
        return p, p
    at = torch.randint(0, case["n"], (case["nq"],), generator=g, device="cuda")
    return p, p[at].contiguous()


def _catalogue(g, n, mu):
    """Unit vectors, 30% of them in clumps around `mu` (von Mises-Fisher,
    kappa = 1e5, as tangent-plane Gaussians)."""
    v = torch.nn.functional.normalize(_randn(g, n, 3), dim=1)
    lab = torch.randint(0, len(mu), (n,), generator=g, device="cuda")
    c = mu[lab].add_(_randn(g, n, 3), alpha=1e-5 ** 0.5)
    return torch.nn.functional.normalize(torch.where(_rand(g, n, 1) < 0.3, c, v), dim=1)


def _directions(g, m):
    return torch.nn.functional.normalize(_randn(g, m, 3), dim=1)


def _ranks(g, n):
    """One u32 rank per entry: the place of its weight, 0 the heaviest."""
    return torch.randperm(n, generator=g, device="cuda").to(torch.int32)


def _surface(g, n, plane, frame, centre):
    """Points on a randomly oriented unit square or sphere, N(0, 0.001) jitter."""
    if plane:
        uv = _rand(g, n, 2) - 0.5
        p = uv[:, :1] * frame[0] + uv[:, 1:] * frame[1]
    else:
        p = 0.5 * torch.nn.functional.normalize(_randn(g, n, 3), dim=1)
    return (p + centre + 0.001 * _randn(g, n, 3)).to(torch.float32)


def _split(total, parts, lowest, spread):
    """`parts` sizes adding up to `total`, spread geometrically over a factor
    of `spread`, none below `lowest`."""
    w = [spread ** (i / max(1, parts - 1)) for i in range(parts)]
    s = [max(lowest, int(total * x / sum(w))) for x in w]
    s[-1] += max(0, total - sum(s))
    return s


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind in ("knn", "one"):
        p, q = _cloud(g, case, case["dims"])
        return dict(case=case, tree=kb.GpuTree.build(p), q=q)
    if kind == "build":
        return dict(case=case, p=_cloud(g, case, case["dims"])[0])
    if kind == "host":
        p, q = _cloud(g, dict(case, data="mixture"), 3)
        return dict(case=case, tree=kb.GpuTree.build(p), q=q.cpu().pin_memory().numpy())
    if kind == "periodic":
        p, q = _periodic_points(g, case)
        return dict(case=case, tree=kb.GpuTree.build(p), q=q)
    if kind == "within":
        mu = _directions(g, 32)
        dt = TORCH[case["dtype"]]
        p = _catalogue(g, case["n"], mu).to(dt)
        return dict(case=case, tree=kb.GpuTree.build(p), q=_catalogue(g, case["nq"], mu).to(dt),
                    room=_room(case))
    if kind == "forest":
        sizes = _split(case["n"], case["trees"], 10_000, 100.0)
        per = torch.bincount(torch.randint(0, case["trees"], (case["nq"],), generator=g,
                                           device="cuda"), minlength=case["trees"]).tolist()
        trees, qs, of = [], [], []
        for t, n in enumerate(sizes):
            mu = _directions(g, 32)
            trees.append(kb.GpuTree.build(_catalogue(g, n, mu).to(torch.float32), _ranks(g, n)))
            qs.append(_catalogue(g, per[t], mu).to(torch.float32))
            of.append(torch.full((per[t],), t, dtype=torch.int32, device="cuda"))
        chord = torch.exp(math.log(1e-4) + _rand(g, case["nq"]) * math.log(100.0))
        return dict(case=case, forest=kb.Forest(trees), q=torch.cat(qs), of=torch.cat(of),
                    radii=(chord * chord).to(torch.float32), room=_room(case))
    # chamfer: source clouds spread over a factor of 20, targets 4x as many
    trees, src, tgt, of, base, at = [], [], [], [], [], 0
    for t, n in enumerate(_split(case["n_src"], case["pairs"], 1000, 20.0)):
        frame = torch.linalg.qr(_randn(g, 3, 3)).Q
        centre = _rand(g, 3)
        tp = _surface(g, 4 * n, t % 2 == 0, frame, centre)
        trees.append(kb.GpuTree.build(tp))
        tgt.append(tp)
        src.append(_surface(g, n, t % 2 == 0, frame, centre))
        of.append(torch.full((n,), t, dtype=torch.int32, device="cuda"))
        base.append(at)
        at += 4 * n
    return dict(case=case, forest=kb.Forest(trees), src=torch.cat(src), tgt=torch.cat(tgt),
                of=torch.cat(of), base=torch.tensor(base, dtype=torch.int64, device="cuda"))


# ---- one pass ---------------------------------------------------------------
def _fields(r):
    return {k: v for k, v in r.__dict__.items() if v is not None}


def _static(r, room):
    """A radius result in buffers of a fixed size, zeros after the hits: what a
    program with static shapes hands on."""
    pad = (0, max(0, room - r.distances.shape[0]))
    return {"offsets": r.offsets, "distances": torch.nn.functional.pad(r.distances, pad),
            "items": torch.nn.functional.pad(r.items, pad)}


def _room(case):
    """Hits to make room for: well above what such a batch finds."""
    return int(2.5 * case["nq"] * _mean_hits(case)) + 20_000


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "knn":
        r = s["tree"].query(s["q"]).nearest_n(METRIC[c["metric"]], c["k"]).execute_gpu()
    elif kind == "host":
        r = s["tree"].query(s["q"]).nearest_n(kb.SquaredEuclidean, c["k"]).execute_gpu()
    elif kind == "one":
        b = s["tree"].query(s["q"]).nearest_one(METRIC[c["metric"]])
        r = (b.approx() if c["approx"] else b).execute_gpu()
    elif kind == "periodic":
        r = (s["tree"].query(s["q"]).periodic_boundary_condition(np.ones(3))
             .nearest_n(kb.SquaredEuclidean, c["k"]).within(c["radius"]).execute_gpu())
    elif kind == "within":
        b = s["tree"].query(s["q"]).within(kb.SquaredEuclidean, c["chord"] ** 2)
        return _static((b if c["sort"] else b.unsorted()).execute_gpu(), s["room"])
    elif kind == "forest":
        b = s["forest"].query(s["q"], s["of"], s["radii"])
        if c["family"] == "best":
            r = b.best_n_within(kb.SquaredEuclidean, 0.0, 5).execute_gpu()
        else:
            b = b.within(kb.SquaredEuclidean, 0.0)
            return _static((b if c["family"] == "within" else b.unsorted()).execute_gpu(),
                           s["room"])
    elif kind == "chamfer":
        loss, ctx = chamfer.chamfer_forward(s["forest"], s["src"], s["tgt"], c["k"], 0.01,
                                            s["of"], s["base"])
        g_src, g_tgt = chamfer.chamfer_backward(ctx)
        return {"loss": loss, "grad_src": g_src, "grad_tgt": g_tgt}
    else:
        items, points = kb.GpuTree.build(s["p"]).iter()
        return {"items": items, "points": points}
    return _fields(r)


# ---- what a pass cannot do without --------------------------------------------
def _hits(n, chord):
    """Expected entries within a chord of a catalogue member."""
    return 0.7 * n * chord * chord / 4 + 0.3 * (0.3 * n / 32) * (1 - math.exp(-chord * chord / 4e-5))


def _mean_hits(case):
    if case["kind"] == "within":
        return _hits(case["n"], case["chord"])
    # log-uniform radii over trees of geometric sizes: a mean over both
    sizes = _split(case["n"], case["trees"], 10_000, 100.0)
    chords = [1e-4 * 100 ** ((i + 0.5) / 16) for i in range(16)]
    return sum(_hits(m, r) for m in sizes for r in chords) / (len(sizes) * len(chords))


def work(case):
    """Queries in, results out, and the entries the answers come from: one
    32-entry leaf per query at least, the whole tree at most."""
    kind = case["kind"]
    sa = SIZE[case.get("dtype", "f32")]
    d = case.get("dims", 3)
    if kind == "build":  # points in; items and points out, twice (tree, iteration)
        return {"bytes": case["n"] * (3 * d * sa + 8), "flops": 0}
    if kind == "chamfer":
        ns, nt, k = case["n_src"], 4 * case["n_src"], case["k"]
        entries = min(nt, 32 * ns)
        return {"bytes": 2 * 12 * ns + 12 * nt + 16 * entries, "flops": ns * (32 * 8 + 40 * k)}
    n, nq = case["n"], case["nq"]
    if kind == "forest":
        hits = _mean_hits(case)
        out = 44 if case["family"] == "best" else 8 + 8 * hits
        scanned = max(32, hits)
        io = 12 + 4 + 4
    elif kind == "within":
        hits = _mean_hits(case)
        out, scanned, io = 8 + (sa + 4) * hits, max(32, hits), 3 * sa
    elif kind == "one":
        out, scanned, io = sa + 4, 32, d * sa
    else:
        out, scanned, io = case["k"] * (sa + 4) + 4, max(32, case["k"]), d * sa
    entries = min(n, nq * scanned)
    return {"bytes": entries * (d * sa + 4) + nq * (io + out),
            "flops": nq * scanned * (3 * d - 1)}


# ---- the same in 64 bits, brute force -------------------------------------------
def _pair_distances(q, p, metric, box=None):
    acc = torch.zeros((q.shape[0], p.shape[0]), dtype=torch.float64, device=q.device)
    for a in range(q.shape[1]):
        t = (q[:, a, None] - p[None, :, a]).abs_()
        if box is not None:
            t = torch.minimum(t, box - t)
        acc += t if metric == "manhattan" else t.mul_(t)
    return acc


def _smallest(q, p, k, metric, box=None):
    """The k smallest distances of each query (ascending) and their rows."""
    q, p = q.double(), p.double()
    step = max(1, int(4e8) // max(1, p.shape[0]))
    ds, ix = [], []
    for a in range(0, q.shape[0], step):
        d = _pair_distances(q[a:a + step], p, metric, box)
        if k == 1:
            v, i = d.min(dim=1, keepdim=True)
        else:
            v, i = d.topk(k, dim=1, largest=False)
        ds.append(v)
        ix.append(i)
    return torch.cat(ds), torch.cat(ix)


def exact(case, seed):
    """Distances (and the loss and gradients) by brute force where that is
    quick; items, counts and offsets are whole numbers and have no such value."""
    kind = case["kind"]
    if kind == "knn" and case["n"] * case["nq"] <= 8e9 and case["n"] >= case["k"]:
        g = _gen(seed)
        p, q = _cloud(g, case, case["dims"])
        return {"distances": _smallest(q, p, case["k"], case["metric"])[0], "items": None,
                "counts": None}
    if kind == "one" and not case["approx"] and case["n"] * case["nq"] <= 1.2e11:
        g = _gen(seed)
        p, q = _cloud(g, case, case["dims"])
        return {"distances": _smallest(q, p, 1, case["metric"])[0][:, 0], "items": None}
    if kind == "host" and case["n"] * case["nq"] <= 8e9:
        g = _gen(seed)
        p, q = _cloud(g, dict(case, data="mixture"), 3)
        return {"distances": _smallest(q, p, case["k"], "sq")[0], "items": None, "counts": None}
    if kind == "periodic" and case["n"] * case["nq"] <= 8e9:
        p, q = _periodic_points(_gen(seed), case)
        d = _smallest(q, p, case["k"], "sq", 1.0)[0]
        d[d > case["radius"]] = math.inf
        return {"distances": d, "items": None, "counts": None}
    if kind == "build":
        return None  # a permutation of the input: no computed number
    if kind == "chamfer" and case["n_src"] ** 2 * 4 <= 8e9 * case["pairs"]:
        s = prepare(case, seed)
        src, tgt = s["src"].double(), s["tgt"].double()
        g_src, g_tgt, loss = torch.zeros_like(src), torch.zeros_like(tgt), 0.0
        inv = 1.0 / (2.0 * 0.01 * 0.01)
        base = s["base"].tolist() + [len(tgt)]
        for t in range(case["pairs"]):
            rows = (s["of"] == t).nonzero()[:, 0]
            q, p = src[rows], tgt[base[t]:base[t + 1]]
            d, ix = _smallest(q, p, case["k"], "sq")
            w = torch.exp(-d * inv)
            loss += float((d * w).sum())
            diff = 2.0 * (w * (1.0 - d * inv))[..., None] * (q[:, None, :] - p[ix])
            g_src[rows] = diff.sum(dim=1)
            g_tgt[base[t]:base[t + 1]].index_add_(0, ix.reshape(-1), -diff.reshape(-1, 3))
        return {"loss": torch.tensor(loss, dtype=torch.float64), "grad_src": g_src,
                "grad_tgt": g_tgt}
    return None
