"""What a user of this framework has it do, as cases that can be timed and compared.

A case is a dict of plain values; `prepare` makes what a program holds before
the call (a mesh, sites, an engine for them), `run` is one pass through the
public entry points, `work` is what the pass cannot do without and `exact`
gives its result in 64 bits where that can be had in seconds.

Sizes, meshes and site distributions are those of the framework's own
generators (Kuhn cubes, the voxelised torus, uniform, Gaussian-mixture and
graded sites) over the range of its tests and benchmark: 500 sites in 384 tets
up to 1,000,000 sites in 1,955,088 tets.  The 8,000,000-site cube is left out:
its mesh alone takes minutes to make.
"""
import ctypes
import functools
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]


def _package():
    """The framework, under the name its tests use (its folder's is no identifier)."""
    if "voronoi_gb300" not in sys.modules:
        d = ROOT / "3d-voronoi-gpu_gb300"
        spec = importlib.util.spec_from_file_location("voronoi_gb300", d / "__init__.py",
                                                      submodule_search_locations=[str(d)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["voronoi_gb300"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["voronoi_gb300"]


def _meshgen():
    _package()
    return importlib.import_module("voronoi_gb300.meshgen")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _lloyd(name, mesh, cells, sites, n, iters, k=64, form="exact", volumes=False):
    return {"name": name, "call": "lloyd", "mesh": mesh, "cells": cells, "sites": sites, "n": n, "iters": iters,
            "k": k, "form": form, "volumes": volumes}


def listed():
    return [
        # The smallest problem of the batched workload on its own: one shape of
        # an interactive tool, a call is launches and latency.
        _lloyd("cube4_500", "cube", 4, "uniform", 500, 5),
        # The small configuration of the benchmark, the cell volumes read too.
        _lloyd("cube20_20k", "cube", 20, "uniform", 20_000, 5, volumes=True),
        # A mid-size remeshing job, a ragged count.
        _lloyd("torus64_125k", "torus", 64, "uniform", 124_987, 5, volumes=True),
        # The headline workload: a large uniform remesh.
        _lloyd("torus128_1m", "torus", 128, "uniform", 1_000_000, 5),
        # The same with sites graded 100:1 in density (the precision
        # configuration), in the clip form that the autotuner takes for it.
        _lloyd("torus128_gauss_1m", "torus", 128, "gaussian", 1_000_000, 3, form="pieces"),
        # The large cube's proportions (12 tets per site, 4:1 density
        # gradient, K = 48, pieces), at a mesh that is made in a second.
        _lloyd("cube64_grad_125k", "cube", 64, "gradient", 131_071, 3, k=48, form="pieces"),
        # Sites from voxel data: many on one lattice, where only the robust
        # predicates give whole cells.
        _lloyd("lattice_robust_20k", "cube", 20, "lattice", 20_000, 2, form="robust"),
        # The reference's own sums (tet_k candidates of each tet), for users
        # who need its results: the engine's default form, and its K.
        _lloyd("torus64_reference_60k", "torus", 64, "uniform", 60_003, 2, k=90, form="reference"),
        # The reference's other method: each candidate pair clipped from the tet.
        _lloyd("cube20_tet_cell_20k", "cube", 20, "uniform", 20_000, 2, form="tet_cell"),
        # The drop-in call of a program written against the reference: host
        # arrays in, a few Lloyd iterations, host arrays out.
        {"name": "diagram_cube20_20k", "call": "diagram", "mesh": "cube", "cells": 20, "sites": "uniform",
         "n": 20_000, "iters": 5, "k": 90, "form": "reference"},
        # Many small independent problems at once.
        {"name": "batch32", "call": "batch", "problems": 32, "cells_lo": 4, "cells_hi": 24, "sites_lo": 500,
         "sites_hi": 50_000, "iters": 3, "k": 64, "form": "pieces"},
        # Neighbour search alone, on the caller's device buffers.
        {"name": "knn_60k", "call": "knn", "n": 60_013, "k": 64, "sites": "uniform"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["exact"] * 6 + ["pieces"] * 3 + ["robust", "reference", "tet_cell", "diagram", "batch", "knn",
                                                        "knn"])
    k = rng.choice([48, 64, 64, 96])
    if kind == "knn":
        return {"call": "knn", "n": _log(rng, 500, 65_536), "k": rng.choice([16, 32, 64, 90, 128]),
                "sites": rng.choice(["uniform", "gaussian"])}
    if kind == "batch":
        hi = rng.randint(6, 24)
        return {"call": "batch", "problems": rng.randint(2, 32), "cells_lo": 4, "cells_hi": hi, "sites_lo": 500,
                "sites_hi": _log(rng, 2_000, 50_000), "iters": rng.randint(1, 3), "k": k,
                "form": rng.choice(["exact", "pieces"])}
    if kind in ("exact", "pieces"):
        mesh = rng.choice(["cube", "torus"])
        n = _log(rng, 500, 1_000_000)
        # a third to twelve tets per site, at most the largest listed mesh
        tets = min(max(n * math.exp(rng.uniform(math.log(0.33), math.log(12))), 400), 1_900_000)
        cells = (tets / 6) ** (1 / 3) if mesh == "cube" else (tets / 6 / 0.155) ** (1 / 3)
        cells = min(max(int(round(cells)), 4 if mesh == "cube" else 16), 64 if mesh == "cube" else 128)
        sites = rng.choice(["uniform", "gradient"] if mesh == "cube" else ["uniform", "gaussian"])
        return _unnamed(_lloyd("", mesh, cells, sites, n, rng.randint(1, 3 if n > 500_000 else 5), k, kind,
                               n <= 200_000 and rng.random() < 0.4))
    if kind == "robust":
        return _unnamed(_lloyd("", "cube", rng.randint(6, 20), rng.choice(["lattice", "uniform"]),
                               _log(rng, 500, 20_000), rng.randint(1, 2), k, kind))
    n = _log(rng, 500, 60_000)
    mesh = rng.choice(["cube", "torus"])
    cells = rng.randint(6, 20) if mesh == "cube" else rng.randint(16, 56)
    c = _unnamed(_lloyd("", mesh, cells, "uniform", n, rng.randint(1, 3), rng.choice([64, 90]),
                        "reference" if kind == "diagram" else kind))
    if kind == "diagram":
        c["call"] = "diagram"
    return c


def _unnamed(c):
    return {k: v for k, v in c.items() if k != "name"}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=8)
def _mesh(mesh, cells):
    """Unit-box vertices and tets; the mesh is the case's, the sites the seed's."""
    mg = _meshgen()
    pos, tets = mg.kuhn_cube(cells) if mesh == "cube" else mg.torus_mesh(cells)
    return pos, np.ascontiguousarray(tets, np.int32)


def _sites(case, seed):
    """Sites in the unit box."""
    mg, n, rng = _meshgen(), case["n"], np.random.default_rng(seed)
    if case["sites"] == "gradient":
        return mg.gradient_sites(n, rng)
    if case["sites"] == "gaussian":
        return mg.torus_gaussian_sites(n, rng)
    if case.get("mesh") == "torus":
        return mg.torus_uniform_sites(n, rng)
    s = rng.uniform(0.0, 1.0, (n, 3))
    if case["sites"] == "lattice":
        # half of them on distinct points of a lattice with three quarters of
        # its points taken
        m = n // 2
        side = int(math.ceil((m / 0.75) ** (1 / 3)))
        at = rng.choice(side ** 3, m, replace=False)
        s[:m] = (np.stack([at % side, at // side % side, at // side ** 2], 1) + 0.5) / side
    return s


def _problem(case, seed):
    mg = _meshgen()
    pos, tets = _mesh(case["mesh"], case["cells"])
    verts, sites = mg.normalize(pos, _sites(case, seed))
    return verts, tets, sites


def _batch_sizes(case):
    """(cube side, sites) of each problem, the same whatever the seed."""
    rng = np.random.default_rng(4)
    return [(int(rng.integers(case["cells_lo"], case["cells_hi"] + 1)),
             int(np.exp(rng.uniform(np.log(case["sites_lo"]), np.log(case["sites_hi"])))))
            for _ in range(case["problems"])]


def _batch(case, seed):
    mg, rng = _meshgen(), np.random.default_rng(seed)
    return [mg.cube_problem(cells, n, seed=int(rng.integers(1 << 31)), jitter=0.1) for cells, n in _batch_sizes(case)]


_ENGINE = {
    "exact": dict(exact=True),
    "pieces": dict(exact=True, tet_pieces=True),
    "robust": dict(exact=True, robust_predicates=True),
    "reference": dict(),
    "tet_cell": dict(method="site_major"),
}


def prepare(case, seed):
    V = _package()
    if case["call"] == "knn":
        s = 1000.0 * _sites(case, seed)
        n, k = case["n"], case["k"]
        pts = torch.from_numpy(s.astype(np.float32)).cuda()
        f = V.lib().vgb_knn_noalloc
        f.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
        f.restype = ctypes.c_int
        return {"call": "knn", "f": f, "pts": pts, "n": n, "k": k,
                "knn": torch.empty((n, k), dtype=torch.int32, device="cuda"),
                "perm": torch.empty((n,), dtype=torch.int32, device="cuda")}
    if case["call"] == "batch":
        P = _batch(case, seed)
        b = V.Batch([(p.verts, p.tets, p.sites) for p in P], site_k=case["k"], tune_grid=False,
                    tet_pieces=case["form"] == "pieces")
        return {"call": "batch", "batch": b, "iters": case["iters"]}
    verts, tets, sites = _problem(case, seed)
    if case["call"] == "diagram":
        return {"call": "diagram", "verts": verts, "tets": tets, "sites": sites, "iters": case["iters"],
                "k": case["k"]}
    e = V.Engine(verts, tets, sites, site_k=min(case["k"], case["n"] - 1), **_ENGINE[case["form"]])
    return {"call": "lloyd", "engine": e, "sites": sites, "iters": case["iters"], "volumes": case["volumes"]}


def run(state):
    V = _package()
    if state["call"] == "knn":
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        rc = state["f"](state["pts"].data_ptr(), state["n"], state["k"], state["knn"].data_ptr(),
                        state["perm"].data_ptr(), stream)
        if rc:
            raise RuntimeError(V.lib().vgb_last_error().decode())
        return {"knn": state["knn"], "perm": state["perm"]}
    if state["call"] == "diagram":
        # the reference's SoA layout, which keeps the order of the sites
        return V.clipped_voro_diagram(state["verts"], state["tets"], np.ascontiguousarray(state["sites"].T),
                                      site_is_transposed=True, nb_lloyd_iter=state["iters"], site_k=state["k"])
    if state["call"] == "batch":
        b = state["batch"]
        b.iterate(state["iters"])
        return [b.result(p)[0] for p in range(b.n_prob)]
    e = state["engine"]
    e.set_sites(state["sites"])
    e.iterate(state["iters"])
    if not state["volumes"]:
        return e.sites_original()
    # the volumes by site, as the single-precision values that they are
    # computed as (the engine writes its float sums out as doubles)
    xyz, ids = e.sites()
    sites, volumes = np.empty_like(xyz), np.empty(len(ids), np.float32)
    sites[ids] = xyz
    volumes[ids] = e.moments()[0]
    return {"sites": sites, "volumes": volumes}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _tets(mesh, cells):
    return 6.0 * cells ** 3 * (1.0 if mesh == "cube" else 2 * math.pi ** 2 * 0.35 * 0.15 ** 2)


def work(case):
    """One pass: each site and tet read once, each site written once per
    iteration; operations of the cells themselves, whatever way they are
    found: a Voronoi cell has about 15.5 faces and 27 vertices, each vertex
    made once (45), tested against each face (6) and decomposed (220)."""
    if case["call"] == "knn":
        # sites read, rows and order written; 27 cells' worth of distances (8)
        # is what a grid of three sites a cell leaves for the nearest few
        n, k = case["n"], case["k"]
        return {"bytes": 12.0 * n + 4.0 * n * (k + 1), "flops": 8.0 * n * 1.5 * k}
    if case["call"] == "batch":
        sizes = _batch_sizes(case)
        n, m = sum(s for _, s in sizes), sum(_tets("cube", c) for c, _ in sizes)
    else:
        n, m = case["n"], _tets(case["mesh"], case["cells"])
    cell = 27 * (45.0 + 6.0 * 15.5 + 220.0)
    if case["form"] in ("reference", "tet_cell"):
        # every (tet, cell) pair that meets: about a cell's faces crossed by
        # the tets it shares, pieces of nine vertices and four more planes
        pairs = m + n + 4.0 * (m * m * n) ** (1 / 3)
        cell += pairs / n * 9 * (45.0 + 6.0 * 8 + 220.0)
    return {"bytes": case["iters"] * (24.0 * n + 32.0 * m), "flops": case["iters"] * n * cell}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _polytopes(nrm, off):
    """Volume, first moment and largest squared vertex distance (from the
    origin) of the polytopes nrm . x <= off; nrm (B, F, 3) of unit length or
    zero (no plane), off (B, F).  Every edge is the line of two faces cut by
    all others; with its line's two face feet it spans two signed tets."""
    B, F, _ = nrm.shape
    i, j = torch.triu_indices(F, F, 1, device=nrm.device)
    ni, nj, di, dj = nrm[:, i], nrm[:, j], off[:, i], off[:, j]
    ray = torch.linalg.cross(ni, nj)
    rr = (ray * ray).sum(-1)
    ok = rr > 1e-20
    rr = torch.where(ok, rr, 1.0)
    at = (di[..., None] * torch.linalg.cross(nj, ray) + dj[..., None] * torch.linalg.cross(ray, ni)) / rr[..., None]
    rate = ray @ nrm.transpose(1, 2)
    slack = off[:, None, :] - at @ nrm.transpose(1, 2)
    own = torch.zeros(len(i), F, dtype=torch.bool, device=nrm.device)
    own[torch.arange(len(i)), i] = True
    own[torch.arange(len(i)), j] = True
    rate = rate.masked_fill(own, 0.0)
    ok &= ~((rate == 0) & (slack < 0) & ~own).any(-1)
    t = slack / rate
    hi = torch.where(rate > 0, t, math.inf).amin(-1)
    lo = torch.where(rate < 0, t, -math.inf).amax(-1)
    ok &= (hi > lo) & torch.isfinite(hi) & torch.isfinite(lo)
    hi, lo = torch.where(ok, hi, 0.0), torch.where(ok, lo, 0.0)
    a, b = at + lo[..., None] * ray, at + hi[..., None] * ray
    c = (ni * nj).sum(-1)
    vi, vj = di * (dj - c * di) * (hi - lo) / 6, dj * (di - c * dj) * (hi - lo) / 6
    both = (vi + vj)[..., None] * (a + b) + (vi * di)[..., None] * ni + (vj * dj)[..., None] * nj
    far = torch.where(ok, torch.maximum((a * a).sum(-1), (b * b).sum(-1)), 0.0)
    return (vi + vj).sum(-1), both.sum(1) / 4, far.amax(-1)


def _in_chunks(nrm_off, count, planes):
    """_polytopes over count polytopes; nrm_off(at) gives the planes of `at`."""
    step = max(1, int(4e8 / (8 * planes ** 3 / 2)))
    got = [_polytopes(*nrm_off(torch.arange(b, min(count, b + step), device="cuda"))) for b in range(0, count, step)]
    return [torch.cat(x) for x in zip(*got)]


def _nearest(s, k):
    """The k nearest others of each site, ordered: indices and distances.
    Block by block of the box, among the sites one block width around; a
    block with a site whose k-th lies farther is searched among all."""
    n = len(s)
    lo, size = s.min(0).values, float((s.max(0).values - s.min(0).values).max()) * (1 + 1e-9)
    g = max(1, int((n / 600) ** (1 / 3)))
    w = size / g
    block = ((s - lo) / w).long()
    nb, d = torch.empty((n, k), dtype=torch.long, device=s.device), torch.empty((n, k), dtype=s.dtype, device=s.device)
    for key in torch.unique(block, dim=0):
        mine = (block == key).all(1).nonzero()[:, 0]
        near = ((block - key).abs() <= 1).all(1).nonzero()[:, 0]
        for pool in (near, torch.arange(n, device=s.device)):
            if len(pool) <= k:
                continue
            dist = (s[mine][:, None] - s[pool]).norm(dim=-1)
            dist[mine[:, None] == pool] = math.inf
            far, at = dist.topk(k, dim=1, largest=False)
            if len(pool) == n or bool((far[:, -1] <= w).all()):
                break
        nb[mine], d[mine] = pool[at], far
    return nb, d


def _cells(s, lo, hi, k):
    """Cells of the sites s cut by their k nearest and by the box [lo, hi]:
    volumes and site-relative moments."""
    n = len(s)
    nb, d = _nearest(s, k)
    eye = torch.eye(3, dtype=s.dtype, device=s.device)

    def cut(at, m):
        def planes(c):
            z = s[nb[at[c], :m]] - s[at[c]][:, None]
            return (torch.cat([z / d[at[c], :m, None], torch.cat([eye, -eye]).expand(len(c), 6, 3)], 1),
                    torch.cat([d[at[c], :m] / 2, hi - s[at[c]], s[at[c]] - lo], 1))
        return _in_chunks(planes, len(at), m + 6)

    # with m neighbours a cell is done when the next lies beyond twice its radius
    vol, mom = s.new_empty(n), torch.empty_like(s)
    left = torch.arange(n, device=s.device)
    for m in (24, 40, 64, 96, k):
        m = min(m, k)
        v, x, r2 = cut(left, m)
        done = torch.ones_like(v, dtype=torch.bool) if m == k else d[left, m] >= 2 * r2.sqrt()
        vol[left[done]], mom[left[done]] = v[done], x[done]
        left = left[~done]
        if not len(left):
            break
    return vol, mom


def _lloyd64(case, verts, sites):
    """Sites after the case's iterations in a box mesh, and the last volumes,
    in 64 bits."""
    v, s = (torch.from_numpy(x.astype(np.float64)).cuda() for x in (verts, sites))
    if case.get("sites") == "lattice":  # volumes are continuous: any general position near by
        s = s + 1e-7 * torch.rand(s.shape, dtype=s.dtype, device=s.device, generator=torch.Generator("cuda").manual_seed(1))
    # the truncated forms take the K nearest, the exact ones all that matter
    k = min(case["k"] if case["form"] in ("reference", "tet_cell") else 192, len(s) - 1)
    for _ in range(case["iters"]):
        vol, mom = _cells(s, v.min(0).values, v.max(0).values, k)
        s = s + mom / vol[:, None]
    return s, vol


def exact(case, seed):
    """What run gives for these inputs, from half-space intersections: where
    the mesh is a box, a clipped cell is the site's cell in that box.  None for
    whole numbers, for more than 300,000 sites and a batch's larger problems
    (half a minute) and for the torus (each pair of a tet and a cell near its
    surface would have to be intersected: minutes)."""
    if case["call"] == "knn":
        return None
    if case["call"] == "batch":
        return [_lloyd64(case, p.verts, p.sites)[0].cpu().numpy() if len(p.sites) <= 8_000 else None
                for p in _batch(case, seed)]
    if case["mesh"] == "torus" or case["n"] > 300_000:
        return None
    verts, _, sites = _problem(case, seed)
    s, vol = (x.cpu().numpy() for x in _lloyd64(case, verts, sites))
    if case["call"] == "diagram":
        return np.ascontiguousarray(s.T)
    return {"sites": s, "volumes": vol} if case["volumes"] else s
