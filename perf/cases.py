"""The work that users of this framework have it do, as measurable cases.

A program segments a porous sample into a (SZ, SX, SY) volume and calls either single stages on
CUDA tensors (squared EDT, containing balls, pore propagation with empty-pore removal, watershed,
geodesics), the whole chain stage by stage, the whole chain on a host volume in one call, or the
whole chain on a batch of volumes. The volumes are this repository's own generators: sphere packs
and unions (small samples), thresholded Gaussian random fields (rocks with small pores) and
leveled-wave spinodals (monoliths with large pores), in the sizes of its benchmark and tests.

A case: {"name", "do", "kind", "sz", "sx", "sy", "d3q7", "fp64", "volumes"}; "do" is the call,
"kind" the volume, "volumes" the number of volumes of a batch.
"""
import ctypes
import math

import numpy as np
import torch

import porousmediaanalysis_gb300 as pma
from porousmediaanalysis_gb300 import capi, synth

INF = float("inf")
HISTOGRAM = 4096  # squared distances counted


def _case(name, do, kind, shape, d3q7=False, fp64=False, volumes=1):
    return {"name": name, "do": do, "kind": kind, "sz": shape[0], "sx": shape[1], "sy": shape[2],
            "d3q7": d3q7, "fp64": fp64, "volumes": volumes}


def listed():
    return [
        # one EDT of a hand-sized block: the smallest call, launches and the read-back alone
        _case("edt_small", "edt", "pack", (33, 40, 29)),
        # EDT of the largest volume of the benchmark (1024^3 monolith)
        _case("edt_1024", "edt", "spinodal", (1024, 1024, 1024)),
        # containing balls of a large monolith: large radii, long lists of overlapping balls
        _case("balls_spinodal", "balls", "spinodal", (704, 768, 811)),
        # pore propagation and empty-pore removal of the 512^3 rock: many small pores
        _case("pores_grf_512", "pores", "grf", (512, 512, 512)),
        # the same of a mid-sized monolith of odd sizes: deep radius levels, long seed sets
        _case("pores_spinodal", "pores", "spinodal", (300, 341, 277)),
        # watershed of a monolith: few pores, large floods
        _case("watershed_spinodal", "watershed", "spinodal", (640, 600, 672)),
        # geodesic distances of the largest volume, float64
        _case("geodesic_1024_f64", "geodesic", "spinodal", (1024, 1024, 1024), fp64=True),
        # geodesic distances in the reference's float32, six-neighbour stencil, odd sizes
        _case("geodesic_grf_f32_d3q7", "geodesic", "grf", (301, 257, 411), d3q7=True),
        # whole chain stage by stage on the smallest kind of sample: latency
        _case("chain_small", "chain", "union", (40, 48, 44)),
        # whole chain of the 128^3 union of spheres
        _case("chain_union_128", "chain", "union", (128, 128, 128)),
        # whole chain of the 512^3 rock from page-locked host memory and back in one call
        _case("host_grf_512", "host", "grf", (512, 512, 512), fp64=True),
        # a batch of small packs of uneven sizes (axes 32 to 192), whole chain
        _case("batch_packs", "batch", "pack", (192, 192, 192), volumes=28),
    ]


# the most voxels drawn of each call, at or below the largest listed case of that call
_MOST = {"edt": 1 << 29, "balls": 1 << 28, "pores": 1 << 26, "watershed": 1 << 27, "geodesic": 1 << 29,
         "chain": 1 << 24, "host": 1 << 26}
_KIND_MOST = {"union": 1 << 22, "pack": 1 << 22, "grf": 1 << 27, "spinodal": 1 << 29}


def _shape(rng, voxels):
    """Three uneven extents of about `voxels` voxels."""
    side = voxels ** (1.0 / 3.0)
    a, b = rng.uniform(-0.35, 0.35), rng.uniform(-0.35, 0.35)
    return tuple(max(12, min(1400, int(side * math.exp(e)))) for e in (a, b, -a - b))


def draw(rng):
    do = rng.choice(["edt", "balls", "pores", "watershed", "geodesic", "chain", "host", "batch"])
    d3q7 = do in ("pores", "watershed", "geodesic", "chain", "host") and rng.random() < 0.25
    fp64 = do in ("geodesic", "chain", "host") and rng.random() < 0.5
    if do == "batch":
        side = rng.randint(64, 192)
        return _draw(do, "pack", (side, side, side), False, rng.random() < 0.5, rng.randint(2, 28))
    voxels = math.exp(rng.uniform(math.log(1 << 15), math.log(_MOST[do])))
    kinds = [k for k in ("union", "pack", "grf", "spinodal") if voxels <= _KIND_MOST[k]]
    return _draw(do, rng.choice(kinds), _shape(rng, voxels), d3q7, fp64, 1)


def _draw(*a):
    c = _case("", *a)
    del c["name"]
    return c


def _volume(kind, shape, seed, device="cuda"):
    """(SZ, SX, SY) uint8, non-zero = solid: a CUDA tensor."""
    if kind == "spinodal":
        return synth.spinodal(shape, seed=seed, device=device)
    if kind == "grf":
        return synth.grf(shape, sigma=3.0, porosity=0.65, seed=seed, device=device)
    return torch.from_numpy(_small_volume(kind, shape, seed)).to(device)


def _small_volume(kind, shape, seed):
    """Sphere union (300 spheres of radius 5 to 10 per 128^3) or sphere pack, on the host."""
    if kind == "union":
        count = max(8, round(300.0 * shape[0] * shape[1] * shape[2] / 128 ** 3))
        return synth.sphere_union(shape, count=count, seed=seed)
    return synth.sphere_pack(shape, seed=seed)


# A program keeps one context for the volumes that it works through; another kind of work gets a
# context of its own, and the old one's device memory goes back.
_kept = {}


def _context(case):
    key = tuple(sorted(case.items()))
    if key not in _kept:
        for c in _kept.values():
            c.close()
        _kept.clear()
        _kept[key] = pma.Context(0)
    return _kept[key]


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def prepare(case, seed):
    ctx = _context(case)
    do, shape = case["do"], (case["sz"], case["sx"], case["sy"])
    stencil = pma.D3Q7 if case["d3q7"] else pma.D3Q27
    state = {"do": do, "ctx": ctx, "stencil": stencil, "fp64": case["fp64"],
             "voxels": shape[0] * shape[1] * shape[2]}
    if do == "batch":  # the sizes are the case's, the volumes the seed's
        shapes = synth.batch_shapes(case["volumes"], 32, case["sz"])
        state["volumes"] = [torch.from_numpy(_small_volume(case["kind"], s, 1000 * seed + i)).cuda() for i, s in enumerate(shapes)]
        return state
    solid = _volume(case["kind"], shape, seed)
    if do == "host":
        state["solid"] = _pinned(shape, torch.uint8)
        state["solid"][...] = solid.cpu().numpy()
        dist = ("dist_f64", torch.float64) if case["fp64"] else ("dist_f32", torch.float32)
        state["fields"] = ("watershed_labels", dist[0])
        state["out"] = {"watershed_labels": _pinned(shape, torch.int32).view(np.uint32), dist[0]: _pinned(shape, dist[1])}
        return state
    if do in ("edt", "geodesic", "chain"):
        state["solid"] = solid
        return state
    edt2, most, _ = pma.compute_euclidean_distances(ctx, solid)
    state["edt2"], state["max"] = edt2, most
    if do == "balls":
        return state
    del solid
    crad2, _, _, _, mask, _ = pma.set_containing_balls(ctx, edt2, most)
    state["crad2"], state["mask"] = crad2, mask
    if do == "pores":
        return state
    labels, table = pma.assign_pore_and_throat_ids(ctx, mask, edt2, crad2, stencil)
    pma.remove_empty_pores(ctx, table, labels)
    state["table"] = table
    del state["edt2"], state["mask"]
    return state


def _padded(values, dtype, room):
    """`values` and zeros: how many rows there are depends on the volume, the room for them does not."""
    values = np.asarray(values, dtype).reshape(-1)
    if values.size > room:
        raise ValueError("%d values, room for %d" % (values.size, room))
    out = np.zeros(room, dtype)
    out[:values.size] = values
    return out


def _words(address, count, item):
    """A library table as 32-bit words."""
    if count == 0:
        return np.zeros(0, np.int32)
    return np.frombuffer((ctypes.c_int32 * (count * item // 4)).from_address(address), np.int32)


def _table(t, voxels):
    """The rows of a table: pores, throats (id, number of pores, volume, offset) and the throats' pore
    lists, each as 32-bit words in an array with room for what a volume of this size may give."""
    lib, h = capi.lib(), t.handle
    at = lambda p: ctypes.cast(p, ctypes.c_void_p).value  # noqa: E731
    parts = [_words(at(lib.pma_table_pores(h)), lib.pma_table_npores(h), ctypes.sizeof(capi.Pore)),
             _words(at(lib.pma_table_throats(h)), lib.pma_table_nthroats(h), ctypes.sizeof(capi.Throat)),
             _words(at(lib.pma_table_pool(h)), lib.pma_table_pool_size(h), 4)]
    return [_padded(p, np.int32, voxels // part + (1 << 13)) for p, part in zip(parts, (8, 2, 1))]


def _cavities(rows):
    return [_padded([r[:4] + r[5:] for r in rows], np.int64, 7 * 2048), _padded([r[4] for r in rows], np.float64, 2048)]


def _histogram(hist):
    return _padded(hist, np.int64, HISTOGRAM)


def _chain(s):
    ctx, st, n = s["ctx"], s["stencil"], s["voxels"]
    edt2, most, hist = pma.compute_euclidean_distances(ctx, s["solid"], hist_cap=HISTOGRAM)
    crad2, cx, cy, cz, mask, count = pma.set_containing_balls(ctx, edt2, most)
    labels, table = pma.assign_pore_and_throat_ids(ctx, mask, edt2, crad2, st)
    pma.remove_empty_pores(ctx, table, labels)
    flood, flood_table = pma.assign_watershed_ids(ctx, table, crad2, most, st)
    dist, cavity, rows = pma.compute_shortest_path_distances(ctx, s["solid"], st, fp64=s["fp64"])
    return {"dist": dist, "edt2": edt2, "hist": _histogram(hist), "balls": [crad2, cx, cy, cz, mask, count],
            "pores": [labels] + _table(table, n), "watershed": [flood] + _table(flood_table, n), "cavity": [cavity] + _cavities(rows)}


def run(state):
    s, do, ctx = state, state["do"], state["ctx"]
    if do == "edt":
        edt2, most, hist = pma.compute_euclidean_distances(ctx, s["solid"], hist_cap=HISTOGRAM)
        return {"edt2": edt2, "max": most, "hist": _histogram(hist)}
    if do == "balls":
        return list(pma.set_containing_balls(ctx, s["edt2"], s["max"]))
    if do == "pores":
        labels, table = pma.assign_pore_and_throat_ids(ctx, s["mask"], s["edt2"], s["crad2"], s["stencil"])
        pma.remove_empty_pores(ctx, table, labels)
        return [labels] + _table(table, s["voxels"])
    if do == "watershed":
        labels, table = pma.assign_watershed_ids(ctx, s["table"], s["crad2"], s["max"], s["stencil"])
        return [labels] + _table(table, s["voxels"])
    if do == "geodesic":
        dist, cavity, rows = pma.compute_shortest_path_distances(ctx, s["solid"], s["stencil"], fp64=s["fp64"])
        return {"dist": dist, "cavity": [cavity] + _cavities(rows)}
    if do == "chain":
        return _chain(s)
    if do == "host":
        r = pma.pipeline_host(ctx, s["solid"], s["stencil"], fp64=s["fp64"], fields=s["fields"], out_arrays=s["out"])
        return {"dist": r[s["fields"][1]], "labels": r["watershed_labels"].view(np.int32), "pores": _table(r["pores"], s["voxels"]),
                "watershed": _table(r["watershed"], s["voxels"]), "cavity": _cavities(r["cavities"])}
    dist = "dist_f64" if s["fp64"] else "dist_f32"
    got = pma.pipeline_batch(ctx, s["volumes"], s["stencil"], fp64=s["fp64"], fields=("watershed_labels", dist),
                             resident=True, lanes=16)
    tables = [_table(r["watershed"], v.numel()) for r, v in zip(got, s["volumes"])]
    return {"dist": [r[dist] for r in got], "labels": [r["watershed_labels"] for r in got],
            "tables": [np.concatenate([t[k] for t in tables]) for k in range(3)]}


def work(case):
    """Bytes of the volumes read and written once each; the integer work has no flops to speak of."""
    n = case["sz"] * case["sx"] * case["sy"]
    d = 8 if case["fp64"] else 4
    per = {"edt": 1 + 4, "balls": 4 + 17, "pores": 9 + 4, "watershed": 4 + 4, "geodesic": 1 + d + 4,
           "chain": 1 + 4 + 17 + 4 + 4 + d + 4, "host": 1 + 4 + d, "batch": 1 + 4 + d}[case["do"]]
    if case["do"] == "batch":
        n = sum(a * b * c for a, b, c in synth.batch_shapes(case["volumes"], 32, case["sz"]))
    return {"bytes": float(per * n), "flops": 0.0}


# --- geodesic distances in 64 bits, by relaxing until nothing changes ----------------------------

def _relax(solid, dist, d3q7):
    """Shortest 6- or 26-neighbour paths through the void from the voxels where dist is set."""
    pad = torch.full([e + 2 for e in dist.shape], INF, dtype=torch.float64, device=dist.device)
    inner = pad[1:-1, 1:-1, 1:-1]
    inner.copy_(dist)
    sz, sx, sy = dist.shape
    steps = [(a, b, c) for a in range(3) for b in range(3) for c in range(3) if (a, b, c) != (1, 1, 1)]
    steps = [s for s in steps if not d3q7 or sum(e != 1 for e in s) == 1]
    while True:
        best = inner.clone()
        for a, b, c in steps:
            w = math.sqrt((a != 1) + (b != 1) + (c != 1))
            torch.minimum(best, pad[a:a + sz, b:b + sx, c:c + sy] + w, out=best)
        best[solid] = INF
        if torch.equal(best, inner):
            return best
        inner.copy_(best)


def _start(free, half, size, centre, most):
    """First free voxel on the box shells from `half` on, in the reference's order (axes x, y, z):
    (x, y, z) and its shell, or None. free is [z][x][y]."""
    if free[centre[2], centre[0], centre[1]]:
        return tuple(centre), half
    while half < most:
        lo = [max(c - half, 0) for c in centre]
        hi = [min(c + half, e - 1) for c, e in zip(centre, size)]
        for k in range(3):
            a, b = (1, 2) if k == 0 else (0, 2) if k == 1 else (0, 1)
            for face in dict.fromkeys((lo[k], hi[k])):
                ix = [slice(lo[i], hi[i] + 1) for i in range(3)]
                ix[k] = slice(face, face + 1)
                plane = np.moveaxis(free[ix[2], ix[0], ix[1]], 0, 2)  # x, y, z
                at = np.argmax(plane.reshape(-1))
                if plane.reshape(-1)[at]:
                    p = np.unravel_index(at, plane.shape)
                    return tuple(int(p[i]) + ix[i].start for i in range(3)), half
        half += 1
    return None


def _exact_geodesic(solid, d3q7, fp64):
    sz, sx, sy = solid.shape
    size = (sx, sy, sz)
    centre = [min(int(e * 0.5 + 0.5), e - 1) for e in size]
    most = max(max(e - 1 - c, c) for e, c in zip(size, centre))
    mask = solid != 0
    dist = torch.full(solid.shape, INF, dtype=torch.float64, device=solid.device)
    half = 0
    while True:
        half += 1
        found = _start((~mask & torch.isinf(dist)).cpu().numpy(), half, size, centre, most)
        if found is None:
            break
        (x, y, z), half = found
        before = torch.isfinite(dist)
        dist[z, x, y] = 0.0
        dist = _relax(mask, dist, d3q7)
        new = torch.isfinite(dist) & ~before
        if all(bool(new.select(k, i).any()) for k in range(3) for i in (0, -1)):
            break
    dist[torch.isinf(dist)] = float(np.finfo(np.float64 if fp64 else np.float32).max)
    dist[mask] = -1.0
    return dist


def exact(case, seed):
    """The geodesic distances in 64 bits; every other output is whole numbers."""
    shape = (case["sz"], case["sx"], case["sy"])
    if case["do"] not in ("geodesic", "chain", "host") or shape[0] * shape[1] * shape[2] > 1 << 25:
        return None
    dist = _exact_geodesic(_volume(case["kind"], shape, seed), case["d3q7"], case["fp64"])
    return {"dist": dist}
