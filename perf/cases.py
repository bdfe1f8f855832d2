"""The workloads this library's speed is judged by, as calls of its public entry
points on synthetic inputs made from a seed.

Families (the `call` of a case):

* ``host``    ``Delaunay().build(points)`` on host points with every output
              (finite cells, all cells, incident lists) - the reference's own call;
* ``plain``   ``build_device`` - one set per call, points and cells on the device;
* ``batch``   ``build_batch_device`` - many independent sets in one call;
* ``predicate`` ``d3g_predicates_device`` - batch predicates over a point table;
* ``sort``    ``d3g_spatial_sort_device`` - the reference's insertion order;
* ``serve``   ``Server`` - a burst of requests of mixed sizes from host memory.

Every output is an integer (cells, counts, signs, orders), so there is no 64-bit
value to compare with: ``exact`` is None for every case.
"""
import math

import numpy as np
import torch

import del3d_b200 as d3

DISTRIBUTIONS = ("uniform", "clusters", "lattice", "sphere")
MIXED = "mixed"                    # every set of one of the four, drawn per set
SPHERE_Q = 1024                    # quantised spheres: coordinates on a 2^-10 grid
CLUSTERS, SIGMA = 8, 0.02
PREDICATES = {"orient3d": (d3.ORIENT3D, 4), "in_sphere": (d3.IN_SPHERE, 5)}
# Per point of a build: 24 bytes in, about 6.75 finite tets of 16 bytes out, and
# about 45 conflict tests of 111 double operations each.
TETS_PER_POINT, TEST_FLOPS_PER_POINT = 6.75, 45 * 111


def listed():
    return [
        # The smallest call: an interactive program triangulates a few hundred points
        # and reads every output.
        {"name": "host_uniform_500", "call": "host", "dist": "uniform", "n": 500, "dups": False},
        # One set of the mixed workload's median size per call, points already on the device.
        {"name": "plain_clusters_1448", "call": "plain", "dist": "clusters", "n": 1448},
        # A scanned surface with repeated samples, from host memory, every output.
        {"name": "host_sphere_20k_dups", "call": "host", "dist": "sphere", "n": 20011, "dups": True},
        # The 100^3 integer lattice: every query is degenerate (voxel and grid data).
        {"name": "plain_lattice_1e6", "call": "plain", "dist": "lattice", "n": 1000000},
        # A million points in general position.
        {"name": "plain_uniform_1e6", "call": "plain", "dist": "uniform", "n": 1000000},
        # A quantised surface without repeats (points on a sphere: long walks, flat tets).
        {"name": "plain_sphere_1e6", "call": "plain", "dist": "sphere", "n": 999983},
        # The largest single set of the repository's own benchmarks.
        {"name": "plain_uniform_1e7", "call": "plain", "dist": "uniform", "n": 10000000},
        # A batch as a simulation step or a data loader makes it: 256 sets of every size.
        {"name": "batch_mixed_256", "call": "batch", "dist": MIXED, "sets": 256, "lo": 32, "hi": 65536,
         "sizes": 11},
        # The headline batched workload: 4096 sets, 35 million points.
        {"name": "batch_mixed_4096", "call": "batch", "dist": MIXED, "sets": 4096, "lo": 32, "hi": 65536,
         "sizes": 2024},
        # Batch predicates over a table larger than L2, a tenth exactly degenerate.
        {"name": "in_sphere_1e7", "call": "predicate", "kind": "in_sphere", "table": 10000000, "queries": 10000000},
        # The reference's spatial sort of a few million points.
        {"name": "sort_uniform_3e6", "call": "sort", "dist": "uniform", "n": 3000017},
        # A burst of requests to the server, sizes over four decades.
        {"name": "serve_mixed_32", "call": "serve", "dist": MIXED, "sets": 32, "lo": 100, "hi": 1000000,
         "sizes": 31},
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    call = rng.choice(["host", "plain", "plain", "batch", "batch", "predicate", "sort", "serve"])
    dist = rng.choice(DISTRIBUTIONS)
    most = 1000000 if dist == "lattice" else 10000000     # long runs of equal coordinates cost more per point
    if call in ("host", "plain"):
        case = {"call": call, "dist": dist, "n": _log_uniform(rng, 100, 100000 if call == "host" else min(most, 4000000))}
        if call == "host":
            case["dups"] = dist == "sphere" and rng.random() < 0.5
        if dist == "lattice" and rng.random() < 0.5:      # a grid cut out of a larger volume
            case.update(corner=512, n=min(case["n"], 300000))
        return case
    if call == "batch":
        hi = _log_uniform(rng, 256, 65536)
        dist = rng.choice(DISTRIBUTIONS + (MIXED, MIXED))
        return {"call": call, "dist": dist, "sets": _log_uniform(rng, 2, 256 if dist == "lattice" else 2048),
                "lo": _log_uniform(rng, 32, hi), "hi": hi, "sizes": rng.randrange(1 << 20)}
    if call == "predicate":
        return {"call": call, "kind": rng.choice(sorted(PREDICATES)), "table": _log_uniform(rng, 10000, 10000000),
                "queries": _log_uniform(rng, 1000, 20000000)}
    if call == "sort":
        return {"call": call, "dist": dist, "n": _log_uniform(rng, 1000, most)}
    dist = rng.choice(DISTRIBUTIONS + (MIXED, MIXED))
    return {"call": call, "dist": dist, "sets": _log_uniform(rng, 2, 32), "lo": 100,
            "hi": _log_uniform(rng, 1000, 300000 if dist == "lattice" else 1000000), "sizes": rng.randrange(1 << 20)}


def _sizes(case):
    """Sizes of a case's sets (log-uniform in [lo, hi]) and their distributions: part of the case, not of the seed."""
    if "n" in case:
        return np.array([case["n"]], dtype=np.int64), np.array([DISTRIBUTIONS.index(case["dist"])])
    rng = np.random.default_rng(case["sizes"])
    n = np.floor(np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"] + 1), case["sets"]))).astype(np.int64)
    n = np.clip(n, case["lo"], case["hi"])
    kinds = rng.integers(0, len(DISTRIBUTIONS), case["sets"])
    if case["dist"] != MIXED:
        kinds[:] = DISTRIBUTIONS.index(case["dist"])
    return n, kinds


def _point_sets(sizes, kinds, seed, corner=0, repeats=False):
    """The sets back to back, (n, 3) float64 on the GPU, and their set numbers.  Uniform cube, Gaussian clusters,
    integer lattices in random order (their first corner within +-corner), and unit spheres snapped to a grid
    (without equal points, or with them as they fall)."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    nsets = len(sizes)
    n = torch.from_numpy(np.asarray(sizes, dtype=np.int64)).to(dev)
    kind = torch.from_numpy(np.asarray(kinds, dtype=np.int64)).to(dev)
    sid = torch.repeat_interleave(torch.arange(nsets, device=dev), n)
    local = torch.arange(sid.numel(), device=dev) - (torch.cumsum(n, 0) - n)[sid]
    pts = torch.rand((sid.numel(), 3), dtype=torch.float64, device=dev, generator=g)
    pkind = kind[sid]

    at = (pkind == DISTRIBUTIONS.index("clusters")).nonzero()[:, 0]
    if at.numel():
        centre = torch.rand((nsets, CLUSTERS, 3), dtype=torch.float64, device=dev, generator=g) * 0.8 + 0.1
        noise = torch.randn((at.numel(), 3), dtype=torch.float64, device=dev, generator=g)
        pts[at] = centre[sid[at], local[at] % CLUSTERS] + SIGMA * noise

    at = (pkind == DISTRIBUTIONS.index("lattice")).nonzero()[:, 0]
    if at.numel():
        side = torch.from_numpy(np.ceil(np.cbrt(np.asarray(sizes, dtype=np.float64)) - 1e-9).astype(np.int64)).to(dev)
        first = torch.randint(-corner, corner + 1, (nsets, 3), device=dev, generator=g)
        i, m = local[at], side[sid[at]]
        ijk = torch.stack([i // (m * m), (i // m) % m, i % m], 1) + first[sid[at]]
        mixed = torch.argsort(sid[at] + torch.rand(at.numel(), dtype=torch.float64, device=dev, generator=g))
        pts[at] = ijk[mixed].double()

    at = (pkind == DISTRIBUTIONS.index("sphere")).nonzero()[:, 0]
    if at.numel():
        # Enough samples that the first n distinct grid points of each set can be kept.
        want = torch.where(kind == DISTRIBUTIONS.index("sphere"), n, 0)
        made = want if repeats else torch.where(want > 0, want + 64 + want * want // 8000000, 0)
        of = torch.repeat_interleave(torch.arange(nsets, device=dev), made)
        u = torch.rand((of.numel(), 2), dtype=torch.float64, device=dev, generator=g)
        z = u[:, 0] * 2.0 - 1.0
        r, t = torch.sqrt(1.0 - z * z), u[:, 1] * (2.0 * math.pi)
        q = torch.floor(torch.stack([r * torch.cos(t), r * torch.sin(t), z], 1) * SPHERE_Q + 0.5)
        if not repeats:
            k = q.long() + SPHERE_Q
            key = ((of * 4096 + k[:, 0]) * 4096 + k[:, 1]) * 4096 + k[:, 2]
            _, inverse = torch.unique(key, return_inverse=True)
            first = torch.full((int(inverse.max()) + 1,), of.numel(), dtype=torch.int64, device=dev)
            first.scatter_reduce_(0, inverse, torch.arange(of.numel(), device=dev), "amin")
            first = torch.sort(first).values
            had = torch.bincount(of[first], minlength=nsets)
            rank = torch.arange(first.numel(), device=dev) - (torch.cumsum(had, 0) - had)[of[first]]
            q = q[first[rank < want[of[first]]]]
        pts[at] = q / SPHERE_Q
    return pts, sid


def _reordered(pts, sid, kinds, seed):
    """The same sets with their points in another order and, off the grids, at another scale: cells of other points,
    but as many of them."""
    g = torch.Generator(device=pts.device)
    g.manual_seed(int(seed))
    order = torch.argsort(sid + torch.rand(sid.numel(), dtype=torch.float64, device=pts.device, generator=g))
    free = torch.from_numpy(np.asarray(kinds) < DISTRIBUTIONS.index("lattice")).to(pts.device)
    scale = torch.where(free, 0.5 + torch.rand(len(kinds), dtype=torch.float64, device=pts.device, generator=g), 1.0)
    return (pts * scale[sid].unsqueeze(1))[order]


def _predicate_inputs(case, seed):
    """A table of points uniform in [-1, 1]^3 whose last part holds exactly degenerate groups on a 2^-20 grid
    (4 points of a lattice plane, 5 of an integer sphere), and queries: nine in ten random, one in ten a group."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    _, k = PREDICATES[case["kind"]]
    n, nq = case["table"], case["queries"]
    groups = max(1, n // 50)
    pts = torch.rand((n, 3), dtype=torch.float64, device=dev, generator=g) * 2.0 - 1.0
    if k == 4:
        slope = torch.randint(-2, 3, (groups, 1, 2), device=dev, generator=g)
        level = torch.randint(-(1 << 17), 1 << 17, (groups, 1), device=dev, generator=g)
        ij = torch.randint(-(1 << 17), 1 << 17, (groups, 4, 2), device=dev, generator=g)
        grid = torch.cat([ij, (level - (ij * slope).sum(2)).unsqueeze(2)], 2)
    else:
        base = torch.tensor([300, 500, 940], device=dev)
        perms = torch.tensor([[0, 1, 2], [0, 2, 1], [1, 0, 2], [1, 2, 0], [2, 0, 1], [2, 1, 0]], device=dev)
        signs = torch.tensor([[a, b, c] for a in (-1, 1) for b in (-1, 1) for c in (-1, 1)], device=dev)
        vecs = (base[perms].unsqueeze(1) * signs.unsqueeze(0)).reshape(48, 3)      # one sphere about the origin
        pick = torch.rand((groups, 48), device=dev, generator=g).argsort(1)[:, :5]
        grid = torch.randint(-(1 << 19), 1 << 19, (groups, 1, 3), device=dev, generator=g) + vecs[pick]
    first = n - groups * k
    pts[first:] = grid.reshape(-1, 3).double() * 2.0 ** -20
    idx = torch.randint(0, n, (nq, k), dtype=torch.int32, device=dev, generator=g)
    rows = torch.randint(0, nq, (nq // 10,), device=dev, generator=g).unique()
    which = torch.randint(0, groups, (rows.numel(), 1), device=dev, generator=g)
    turn = torch.randint(0, k, (rows.numel(), 1), device=dev, generator=g)
    idx[rows] = (first + which * k + (torch.arange(k, device=dev) + turn) % k).to(torch.int32)
    return pts, idx.contiguous()


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def prepare(case, seed):
    call = case["call"]
    if call == "predicate":
        pts, idx = _predicate_inputs(case, seed)
        out = torch.empty(case["queries"], dtype=torch.int8, device=pts.device)
        return {"call": call, "kind": PREDICATES[case["kind"]][0], "pts": pts, "idx": idx, "out": out}
    sizes, kinds = _sizes(case)
    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    corner = case.get("corner", 0)
    if call in ("host", "serve"):
        # Results come back in arrays of their own size, so the geometry belongs to the case and the order to the seed.
        pts, sid = _point_sets(sizes, kinds, 97, corner, case.get("dups", False))
        pts = _reordered(pts, sid, kinds, seed)
        if call == "host":
            return {"call": call, "pts": pts.cpu().numpy()}
        requests = [_pinned(pts[a:b]) for a, b in zip(offsets[:-1], offsets[1:])]
        return {"call": call, "requests": requests, "server": d3.Server()}
    pts, _ = _point_sets(sizes, kinds, seed, corner)
    if call == "sort":
        return {"call": call, "pts": pts, "out": torch.empty(pts.shape[0], dtype=torch.int32, device=pts.device)}
    # The caller's output buffer, at the library's own default size; cells end where the count says.
    out = torch.zeros((8 * pts.shape[0] + 64, 4), dtype=torch.int32, device=pts.device)
    return {"call": call, "pts": pts, "offsets": offsets, "out": out}


def run(state):
    call = state["call"]
    if call == "host":
        d = d3.Delaunay()
        d.build(state["pts"])
        offsets, incident = d.incident_csr()
        return {"cells": d.finite_cells(), "all": d.all_cells(), "incident_offsets": offsets, "incident": incident,
                "vertices": d.number_of_vertices()}
    if call == "plain":
        cells, vertices = d3.build_device(state["pts"], out=state["out"])
        return {"cells": state["out"], "count": cells.shape[0], "vertices": vertices}
    if call == "batch":
        _, offsets, vertices = d3.build_batch_device(state["pts"], state["offsets"], out=state["out"])
        return {"cells": state["out"], "offsets": offsets, "vertices": vertices}
    lib = d3.library()
    stream = torch.cuda.current_stream().cuda_stream
    if call == "predicate":
        pts, idx, out = state["pts"], state["idx"], state["out"]
        status = lib.d3g_predicates_device(pts.data_ptr(), pts.shape[0], idx.data_ptr(), idx.shape[0], state["kind"],
                                           out.data_ptr(), stream, None)
        if status != d3.OK:
            raise d3.Del3dError(status, "predicates")
        return out
    if call == "sort":
        pts, out = state["pts"], state["out"]
        status = lib.d3g_spatial_sort_device(pts.data_ptr(), pts.shape[0], out.data_ptr(), stream)
        if status != d3.OK:
            raise d3.Del3dError(status, "spatial_sort")
        return out
    server = state["server"]
    done = [server.wait(t) for t in [server.submit(p) for p in state["requests"]]]
    return {"cells": [r.cells for r in done], "vertices": np.array([r.n_vertices for r in done])}


def work(case):
    if case["call"] == "predicate":
        k = PREDICATES[case["kind"]][1]
        flops = 32 if k == 4 else 111
        return {"bytes": float(24 * min(case["table"], case["queries"] * k) + (4 * k + 1) * case["queries"]),
                "flops": float(flops * case["queries"])}
    n = float(_sizes(case)[0].sum())
    if case["call"] == "sort":
        return {"bytes": 28.0 * n, "flops": 0.0}
    per_tet = 16 * (3 if case["call"] == "host" else 1)      # host: cells, all cells and incident lists
    return {"bytes": (24.0 + per_tet * TETS_PER_POINT) * n, "flops": float(TEST_FLOPS_PER_POINT) * n}


def exact(case, seed):
    return None
