"""The workloads whose speed is followed, run through the package's public entry points.

Every case is one tessellation (or one batch of them) built from new generator positions
on a context that the program keeps, as a moving-mesh code does each step.

  api "device"  Context.build_device: generators in device memory, results as zero-copy
                tensors of the context's arrays (the production path)
  api "host"    Voronoi.build / build_partial: numpy in, numpy out (the crate's drop-in)
  api "batch"   Context.build_batch_device: many uneven tessellations in one build
  api "cells"   VoronoiIntegrator.with_faces().cells_arrays(): the cells themselves
                (planes, vertices, decomposition, face-vertex lists) for custom integrals

  kind "poisson"    i.i.d. uniform points
  kind "jitter"     a lattice jittered by half a spacing per axis (relaxed meshes)
  kind "lattice"    an exact lattice: every vertex needs the exact predicate's decision
  kind "clustered"  half the points in Gaussian clumps over four orders of magnitude
                    in density (cosmological and zoom-in set-ups)
"""
import itertools
import math

import numpy as np
import torch

from meshless_voro_b200 import Voronoi, VoronoiIntegrator, default_context
from meshless_voro_b200.voronoi import batch_inputs, device_tensors

FACES = {"owned": 0, "all": 1}  # MV_FACES_OWNED, MV_FACES_ALL


def _case(name, api, kind, n, dim=3, periodic=True, precision="filtered", faces="owned",
          active=1.0, jobs=1):
    return dict(name=name, api=api, kind=kind, n=n, dim=dim, periodic=periodic, precision=precision,
                faces=faces, active=active, jobs=jobs)


def listed():
    return [
        # the smallest tessellations that programs build one by one: latency and launches
        _case("tiny_1k", "device", "poisson", 1000),
        # a small relaxed mesh in a closed box (the 32^3 jittered-lattice configuration)
        _case("jitter_32", "device", "jitter", 32 ** 3, periodic=False),
        # initial conditions on a lattice (the 64^3 exact-lattice configuration)
        _case("lattice_64", "device", "lattice", 64 ** 3),
        # an ordinary 3-D simulation volume
        _case("poisson_128", "device", "poisson", 128 ** 3),
        # the headline: the largest mesh of the benchmark
        _case("poisson_256", "device", "poisson", 256 ** 3),
        # strongly uneven density (the clustered configuration)
        _case("clustered_8m", "device", "clustered", 8388608),
        # a 2-D mesh in a closed box
        _case("plane_1m", "device", "poisson", 1 << 20, dim=2, periodic=False),
        # a rebuild of the active quarter-step cells: a masked build, every face of each
        _case("partial_64", "device", "poisson", 64 ** 3, faces="all", active=0.75),
        # the f64 predicates throughout, on the crate's perturbed-grid example
        _case("fp64_64", "device", "jitter", 64 ** 3, periodic=False, precision="fp64"),
        # the crate's own call: arrays in, arrays out
        _case("host_64", "host", "jitter", 64 ** 3, periodic=False),
        # many uneven tessellations at once (the batched configuration's job mix)
        _case("batch_64", "batch", "mixed", 200000, jobs=64),
        # custom integrals over the cells and their faces
        _case("cells_4k", "cells", "poisson", 4096),
    ]


def _nameless(*args, **kw):
    return {k: v for k, v in _case("", *args, **kw).items() if k != "name"}


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    api = rng.choice(["device"] * 6 + ["host", "batch", "cells"])
    if api == "batch":
        return _nameless(api, "mixed", _log_size(rng, 4000, 200000), jobs=_log_size(rng, 2, 96))
    dim = rng.choice([3, 3, 3, 2, 1])
    kind = rng.choice(["poisson", "poisson", "jitter", "lattice", "clustered"] if dim == 3 else
                      ["poisson", "jitter"] if dim == 2 else ["poisson"])
    if api == "cells":
        dim, kind, top = 3, "poisson", 12000
    elif api == "host":
        top = 400000
    else:
        top = {"lattice": 150 ** 3, "clustered": 1500000}.get(kind, 9000000 if dim > 1 else 1000000)
    return _nameless(api, kind, _log_size(rng, 800, top), dim=dim, periodic=rng.random() < 0.6,
                     precision=rng.choice(["filtered"] * 4 + ["fp64"]),
                     faces=rng.choice(["owned"] * 4 + ["all"]) if api == "device" else "owned",
                     active=rng.choice([1.0, 1.0, 1.0, 0.75, 0.2]) if api != "cells" else 1.0)


# ------------------------------------------------------------------ inputs --
def _side(n, dim):
    return max(2, int(round(n ** (1.0 / dim))))


def _count(case):
    """Generators of a case: lattices have a whole number of points per side."""
    if case["kind"] in ("jitter", "lattice"):
        return _side(case["n"], case["dim"]) ** case["dim"]
    return case["n"]


def _points(case, seed, device):
    """(generators [n, 3] float64, anchor, width).  The seed gives the axes' order and the
    generators' order (random sets) or the box's corner (lattices): every seed is another
    input, and all of a case have equally many faces."""
    kind, dim, n = case["kind"], case["dim"], _count(case)
    gen = torch.Generator(device=device).manual_seed(7 * n + dim)
    rng = np.random.default_rng(seed)

    def uniform(*shape):
        return torch.rand(*shape, generator=gen, device=device, dtype=torch.float64)

    anchor, width = np.zeros(3), np.ones(3)
    if kind == "poisson":
        g = uniform(n, 3)
    elif kind in ("jitter", "lattice"):
        k = _side(case["n"], dim)
        idx = torch.arange(n, device=device)
        g = torch.zeros(n, 3, device=device, dtype=torch.float64)
        for i in range(dim):
            g[:, i] = (idx // k ** (dim - 1 - i)) % k
        g[:, :dim] += 0.5
        if kind == "jitter":
            g[:, :dim] += 0.5 * (uniform(n, dim) - 0.5)
        anchor = rng.integers(-8, 9, 3) * (1.0 / k)
        g = g * (1.0 / k) + torch.from_numpy(anchor).to(device)
    else:
        clumps = max(4, n // 4096)
        half = n // 2
        r = np.random.default_rng(n)
        w = r.pareto(1.5, clumps) + 1.0
        counts = torch.from_numpy(r.multinomial(n - half, w / w.sum())).to(device)
        sigma = torch.exp(math.log(1e-4) + uniform(clumps) * math.log(1e2))
        of = torch.repeat_interleave(torch.arange(clumps, device=device), counts)
        normal = torch.randn(n - half, 3, generator=gen, device=device, dtype=torch.float64)
        clumped = uniform(clumps, 3)[of] + sigma[of, None] * normal
        g = torch.cat([uniform(half, 3), clumped - torch.floor(clumped)])
    if kind in ("poisson", "clustered"):
        g = g[_order(n, seed, device)]
        g[:, :dim] = g[:, torch.from_numpy(rng.permutation(dim)).to(device)]
    if dim < 3:
        g[:, dim:] = 0.0
    return g.contiguous(), anchor, width


def _order(n, seed, device):
    return torch.randperm(n, generator=torch.Generator(device=device).manual_seed(seed), device=device)


def _mask(case, seed, n):
    if case["active"] >= 1.0:
        return None
    mask = np.random.default_rng(n).random(n) < case["active"]
    return mask[_order(n, seed, "cuda").cpu().numpy()] if case["kind"] in ("poisson", "clustered") else mask


def _batch(case, seed):
    """The batched configuration's job mix: sizes log-uniform up to n, 3-D with probability
    0.8 else 2-D, Poisson or jittered lattice, uneven boxes, a tenth of them masked.  The
    seed gives the order of the tessellations and of each one's generators."""
    rng = np.random.default_rng(case["n"] + case["jobs"])
    jobs = []
    for _ in range(case["jobs"]):
        n = int(round(math.exp(rng.uniform(math.log(1000), math.log(case["n"])))))
        dim = 3 if rng.random() < 0.8 else 2
        width, anchor = rng.uniform(0.5, 2.0, 3), rng.uniform(-1.0, 1.0, 3)
        periodic, k = bool(rng.random() < 0.5), _side(n, dim)
        if rng.random() < 0.5:
            u = rng.random((n, 3))
        else:
            u = np.full((k ** dim, 3), 0.5)
            i = np.indices((k,) * dim).reshape(dim, -1).T
            u[:, :dim] = (i + 0.5 + rng.uniform(-0.25, 0.25, i.shape)) / k
        mask = rng.random(len(u)) >= 0.25 if rng.random() < 0.1 else None
        jobs.append(dict(generators=anchor + u * width, anchor=anchor, width=width,
                         dimensionality=dim, periodic=periodic, mask=mask))
    rng = np.random.default_rng(seed)
    for j in jobs:
        at = rng.permutation(len(j["generators"]))
        j["generators"] = j["generators"][at]
        j["mask"] = None if j["mask"] is None else j["mask"][at]
    return [jobs[i] for i in rng.permutation(len(jobs))]


def prepare(case, seed):
    context = default_context()  # one context for the program, as Voronoi.build keeps it
    if case["api"] == "batch":
        g, m, descs = batch_inputs(_batch(case, seed))
        return dict(case=case, context=context, descs=descs, g=torch.from_numpy(g).cuda(),
                    mask=None if m is None else torch.from_numpy(m).cuda())
    g, anchor, width = _points(case, seed, "cuda")
    mask = _mask(case, seed, len(g))
    state = dict(case=case, context=context, anchor=anchor, width=width)
    if case["api"] == "device":
        state["g"] = g
        state["mask"] = None if mask is None else torch.from_numpy(mask.view(np.uint8)).cuda()
    else:
        state["g"], state["mask"] = g.cpu().numpy(), mask
    return state


# -------------------------------------------------------------------- runs --
_ARRAYS = ("cell_volume", "cell_centroid", "cell_safety_radius", "cell_face_offset",
           "cell_face_count", "face_left", "face_right", "face_area", "face_centroid",
           "face_normal", "face_shift_code", "cell_face_connections")


def run(state):
    case, context, mask = state["case"], state["context"], state.get("mask")
    if case["api"] == "batch":
        out = context.build_batch_device(state["g"].data_ptr(), 0 if mask is None else mask.data_ptr(),
                                         state["descs"], precision=case["precision"])
        return device_tensors(out)
    if case["api"] == "device":
        out = context.build_device(
            state["g"].data_ptr(), 0 if mask is None else mask.data_ptr(), len(state["g"]),
            state["anchor"], state["width"], case["dim"], case["periodic"],
            precision=case["precision"], face_mode=FACES[case["faces"]])
        return device_tensors(out)
    if case["api"] == "host":
        if mask is None:
            v = Voronoi.build(state["g"], state["anchor"], state["width"], case["dim"],
                              case["periodic"], precision=case["precision"])
        else:
            v = Voronoi.build_partial(state["g"], mask, state["anchor"], state["width"], case["dim"],
                                      case["periodic"], precision=case["precision"])
        return {k: getattr(v.arrays, k) for k in _ARRAYS}
    cells = VoronoiIntegrator.build(state["g"], mask, state["anchor"], state["width"], case["dim"],
                                    case["periodic"], precision=case["precision"])
    return {k: v for k, v in vars(cells.with_faces().cells_arrays()).items() if k != "n_cells"}


# --------------------------------------------------------- what it is held to --
def work(case):
    """Bytes: generators in, cells, faces and connections out.  Operations: the clip test of
    the neighbours a Voronoi cell needs against its vertices, each final vertex from its
    three planes once, and the tets of the decomposition once."""
    n = _count(case)
    if case["api"] == "batch":  # the mean of log-uniform sizes in [1000, n]
        n = case["jobs"] * int((n - 1000) / math.log(n / 1000.0))
    faces, verts, tests = {3: (15.5, 27, 900), 2: (8.0, 12, 250), 1: (6.0, 8, 60)}[case["dim"]]
    per_cell = faces if case["faces"] == "all" else faces / 2
    active = n * case["active"]
    out = 44.0 * n + active * (per_cell * 65 + (0 if case["faces"] == "all" else 8 + 4 * faces))
    if case["api"] == "host":  # the arrays the call returns hold 64-bit indices
        out += active * (per_cell * 11 + 4 * faces)
    if case["api"] == "cells":
        out += active * ((faces + 6) * 53 + verts * 36 + 6 * verts * 76 + faces * 40)
    flops = active * (6.0 * tests + verts * 50 + 3 * verts * 50 + 6 * verts * 70)
    return {"bytes": 24.0 * n + out, "flops": flops}


def _neighbours(g, i, dim, periodic, width, k):
    """Stream of cell i: offsets to the nearest k images, their generators and shift codes."""
    off = [(0, 0, 0)] if not periodic else \
        list(itertools.product(*[(-1, 0, 1) if a < dim else (0,) for a in range(3)]))
    img = torch.tensor(off, dtype=torch.float64, device=g.device) * width
    d = (g[None] + img[:, None] - g[i]).reshape(-1, 3)
    d2 = (d * d).sum(1)
    d2[off.index((0, 0, 0)) * len(g) + i] = math.inf
    k = min(k, len(d2) - 1)
    val, at = torch.topk(d2, k, largest=False, sorted=True)
    code = torch.tensor([13 + a + 3 * b + 9 * c for a, b, c in off], device=g.device)
    return d[at], at % len(g), code[at // len(g)], math.sqrt(float(val[-1])) if k < len(d2) - 1 else math.inf


def _exact_cell(g, i, dim, periodic, anchor, width):
    """Cell i as the intersection of half-spaces m.y <= h around its generator: the vertices
    are the plane triples whose point no other plane cuts off; volume, centroid and faces
    come from the tets generator - foot on plane - foot on line - vertex."""
    x = g[i]
    lo = torch.as_tensor(anchor, device=g.device).clone()
    hi = lo + torch.as_tensor(width, device=g.device)
    lo[dim:], hi[dim:] = -0.5, 0.5
    m, h, right, code = [], [], [], []
    for a in range(3):  # the box, left out along periodic axes
        if not (periodic and a < dim):
            for s, bound in ((-1.0, lo[a]), (1.0, hi[a])):
                e = torch.zeros(3, dtype=torch.float64, device=g.device)
                e[a] = s
                m.append(e), h.append(s * (bound - x[a])), right.append(-1), code.append(13)
    nb = len(m)
    for k in (60, 110, 170):
        d, idx, cd, reach = _neighbours(g, i, dim, periodic, torch.as_tensor(width, device=g.device), k)
        dist = d.norm(dim=1)
        M = torch.cat([torch.stack(m), d / dist[:, None]]) if nb else d / dist[:, None]
        H = torch.cat([torch.stack(h), 0.5 * dist]) if nb else 0.5 * dist
        R = torch.cat([torch.tensor(right, device=g.device, dtype=torch.int64), idx])
        S = torch.cat([torch.tensor(code, device=g.device, dtype=torch.int64), cd])
        t = torch.combinations(torch.arange(len(M), device=g.device), 3)
        A, b = M[t], H[t]
        c12, c20, c01 = (torch.linalg.cross(A[:, p], A[:, q]) for p, q in ((1, 2), (2, 0), (0, 1)))
        det = (A[:, 0] * c12).sum(1)
        v = (b[:, :1] * c12 + b[:, 1:2] * c20 + b[:, 2:] * c01) / det[:, None]
        ok = (det.abs() > 1e-12) & ((v @ M.T) <= H + 1e-9 * H.abs().max()).all(1)
        t, v = t[ok], v[ok]
        sr = 2.0 * float(v[:, :dim].norm(dim=1).max()) if len(v) else math.inf
        if len(v) >= 4 and sr < reach:
            break
    foot = M * H[:, None]
    vol = torch.zeros((), dtype=torch.float64, device=g.device)
    first = torch.zeros(3, dtype=torch.float64, device=g.device)
    area = torch.zeros(len(M), dtype=torch.float64, device=g.device)
    moment = torch.zeros(len(M), 3, dtype=torch.float64, device=g.device)
    for p, q, r in itertools.permutations(range(3)):
        P, Q = t[:, p], t[:, q]
        along = torch.linalg.cross(M[P], M[Q])
        along = along / along.norm(dim=1, keepdim=True)
        line = v - along * (v * along).sum(1, keepdim=True)
        # oriented by the corner: positive where the feet lie on their own plane and edge
        side = torch.sign((along * M[t[:, r]]).sum(1))
        tri = 0.5 * (torch.linalg.cross(line - foot[P], v - foot[P]) * M[P]).sum(1) * side
        area.index_add_(0, P, tri)
        moment.index_add_(0, P, tri[:, None] * (foot[P] + line + v) / 3.0)
        w = tri * H[P] / 3.0
        vol = vol + w.sum()
        first = first + (w[:, None] * (foot[P] + line + v) / 4.0).sum(0)
    used = torch.zeros(len(M), dtype=torch.bool, device=g.device)
    used[t.reshape(-1)] = True
    keep = used & ~((M[:, dim:] != 0).any(1) if dim < 3 else torch.zeros_like(used))
    keep &= (R < 0) | (S != 13) | (R > i)
    f = torch.nonzero(keep)[:, 0]
    return (vol, x + first / vol, sr, area[f], x + moment[f] / area[f, None], -M[f])


def _exact_lattice(case, g, width):
    """An exact lattice's cells are its boxes; a cell's own faces are those to a neighbour of
    larger index or across the period, in the order (index, shift code)."""
    k, n = _side(case["n"], 3), len(g)
    idx = np.stack([np.arange(n) // k ** 2, np.arange(n) // k % k, np.arange(n) % k], 1)
    order, dirs = [], []
    for a in range(3):
        for s in (-1, 1):
            j = idx.copy()
            j[:, a] += s
            wrap = j[:, a] // k
            j[:, a] %= k
            order.append(((j[:, 0] * k + j[:, 1]) * k + j[:, 2]) * 27 + 13 + wrap * 3 ** a)
            dirs.append([s if i == a else 0 for i in range(3)])
    order, dirs = np.stack(order, 1), np.array(dirs, dtype=np.float64)
    by = np.argsort(order, 1)
    order = np.take_along_axis(order, by, 1)
    own = (order // 27 > np.arange(n)[:, None]) | (order % 27 != 13)
    cell, col = np.nonzero(own)
    e = dirs[by[cell, col]]
    side = width[0] / k
    return dict(cell_volume=np.full(n, side ** 3), cell_centroid=g,
                cell_safety_radius=np.full(n, math.sqrt(3.0) * side),
                face_area=np.full(len(cell), side ** 2), face_centroid=g[cell] + 0.5 * side * e,
                face_normal=-e)


def exact(case, seed):
    """The floating results in plain 64-bit arithmetic: lattices in closed form, small random
    sets cell by cell from all plane triples; larger sets would take minutes."""
    if case["api"] not in ("device", "host") or case["active"] < 1.0 or case["faces"] == "all":
        return None
    n = _count(case)
    if case["kind"] == "lattice" and case["periodic"] and case["dim"] == 3 and _side(case["n"], 3) > 3:
        g, _, width = _points(case, seed, "cuda")
        got = _exact_lattice(case, g.cpu().numpy(), width)
    elif case["kind"] in ("poisson", "jitter") and case["dim"] == 3 and n <= 1500:
        g, anchor, width = _points(case, seed, "cuda")
        cells = [_exact_cell(g, i, 3, case["periodic"], anchor, width) for i in range(n)]
        col = [[c[j] for c in cells] for j in range(6)]
        got = dict(cell_volume=torch.stack(col[0]), cell_centroid=torch.stack(col[1]),
                   cell_safety_radius=torch.tensor(col[2], dtype=torch.float64),
                   face_area=torch.cat(col[3]), face_centroid=torch.cat(col[4]),
                   face_normal=torch.cat(col[5]))
    else:
        return None
    return {k: got.get(k) for k in _ARRAYS}
