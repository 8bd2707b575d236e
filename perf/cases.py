"""Timed cases of the LOD octree builder, through its public entry points.

A case is one user's build: a cloud (generator kind, record type and stride, point count), the octree settings, and
the form in which the program calls the library:

  call      a whole call on host buffers: ocpi_init_octree (upload), ocpi_generate_octree with the records and cloud
            indices filled into pinned arrays, the hierarchy read back.  The records of a node come in no fixed
            order, so the program brings them into the cloud's own order, level by level.
  resident  the cloud stays on the device between builds (ocpi_init_octree once): one ocpi_generate_octree, the
            hierarchy and the tree statistics read back.  The records stay on the device, as they do until a program
            exports them.  Large clouds are built this way; the host link, shared by a machine's GPUs, would
            otherwise be most of the time.
  served    a long-lived server (ocpi_server_*) takes a burst of requests and fills their pinned result arrays.

Clouds are the package's seeded synthetic ones (0 heightfield and boxes, 1 planes and cylinders, 2 terrain with
Zipf-distributed density), which stand in for scans.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "octree-cuda_gb300"))
import octree_api  # noqa: E402

# subsampling options in use: first point of a cell or a random one, its colour as it is, averaged over the cell,
# averaged over the 27 cells around it, or weighted by distance
MODES = {
    "first": dict(),
    "first_intra": dict(intra=True),
    "first_inter": dict(inter=True),
    "first_weighted": dict(inter=True, weighting=True),
    "random": dict(random=True),
    "random_intra": dict(random=True, intra=True),
    "random_inter": dict(random=True, inter=True),
    "random_weighted": dict(random=True, inter=True, weighting=True),
}
THRESHOLD = 10000
OUTPUT_FACTOR = 2.2
SERVED_LANES = 4


def _case(name, form, kind, cloud_type, n, chunk_grid, sub_grid, mode, stride=None, requests=0):
    c = dict(form=form, kind=kind, cloud_type=cloud_type, n=n, stride=stride or (15 if cloud_type == 0 else 27),
             chunk_grid=chunk_grid, sub_grid=sub_grid, mode=mode)
    if requests:
        c["requests"] = requests
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest cloud of a batch of scans: a few nodes, so launches and host round trips count
        _case("call_50k_f32_inter", "call", 0, 0, 50_003, 128, 64, "first_inter"),
        # a single scan position in metric double coordinates, colours averaged per cell
        _case("call_400k_f64_intra", "call", 2, 1, 400_009, 128, 64, "first_intra"),
        # an indoor scan at the default grids with the best colours
        _case("call_1M_f32_weighted", "call", 1, 0, 1_000_003, 512, 128, "random_weighted"),
        # an outdoor scan without averaging, records padded to 32 bytes by the program that wrote them
        _case("resident_2M_f64_first", "resident", 2, 1, 2_000_003, 512, 128, "first", stride=32),
        # a scanned object (5.1M points), the default options
        _case("resident_5M_f32_inter", "resident", 0, 0, 5_138_448, 512, 128, "first_inter"),
        # part of an aerial survey, random points with averaged colours on a smaller counting grid
        _case("resident_12M_f64_random_inter", "resident", 2, 1, 12_345_679, 256, 128, "random_inter"),
        # a building (25.8M points), random points, colours averaged per cell
        _case("resident_26M_f32_random_intra", "resident", 1, 0, 25_836_417, 512, 128, "random_intra"),
        # the same building with distance-weighted colours, the dearest option
        _case("resident_26M_f32_weighted", "resident", 1, 0, 25_836_417, 512, 128, "random_weighted"),
        # the whole survey (119.7M points), the benchmark's workload
        _case("resident_120M_f64_inter", "resident", 2, 1, 119_701_547, 512, 128, "first_inter"),
        # a burst of requests of mixed kinds, types, grids and options at a conversion service
        _case("served_16_mixed", "served", 0, 0, 300_007, 128, 64, "mixed", requests=16),
    ]


def draw(rng):
    form = rng.choice(["call", "resident", "resident", "resident", "served"])
    cloud_type = rng.randrange(2)
    kind = rng.randrange(3)
    mode = rng.choice(sorted(MODES))
    chunk_grid, sub_grid = rng.choice([(128, 64), (256, 64), (256, 128), (512, 128), (512, 128)])
    stride = rng.choice([15, 15, 16, 20]) if cloud_type == 0 else rng.choice([27, 27, 28, 32])
    if form == "served":
        n = int(50_000 * 6 ** rng.random())
        return _case(None, form, 0, 0, n, 128, 64, "mixed", requests=rng.randrange(4, 17))
    # whole calls up to 1.5M points; resident clouds up to what costs as much as the dearest listed ones
    if form == "call":
        top = 1.5e6
    elif mode.endswith("weighted"):
        top = 2e7
    else:
        top = 1.1e8 if kind == 2 and not mode.startswith("random") else 5e7
    n = int(50_000 * (top / 50_000) ** rng.random())
    return _case(None, form, kind, cloud_type, n, chunk_grid, sub_grid, mode, stride=stride)


def _scale(kind):
    # a float32 value widened to double, as the command line passes it
    return (float(np.float32(0.01 if kind == 2 else 0.001)),) * 3


def _room(n):
    """Records that a program keeps room for."""
    return int(n * 2.6) + 1024


def _nodes(n):
    """Hierarchy entries that a program keeps room for."""
    return 4096 + n // 2000


def _table(nodes):
    return np.zeros((nodes, 5), np.int64)


def _pinned(nbytes):
    return torch.empty(max(nbytes, 16), dtype=torch.uint8, pin_memory=True).numpy()


def _cloud(kind, cloud_type, n, stride, seed, pin):
    cloud = octree_api.synthetic_cloud(kind, cloud_type, n, seed, stride)
    bb = octree_api.cubic_bbox(cloud, n, stride, cloud_type)
    if pin:
        host = _pinned(n * stride)[: n * stride]
        host[:] = cloud
        cloud = host
    return cloud, tuple(bb[:3]), tuple(bb[3:])


def _requests(case):
    """The requests of a served burst: sizes within a factor of six around the case's, every option in turn."""
    out = []
    for i in range(case["requests"]):
        n = max(20_000, int(case["n"] * (0.4, 1.0, 2.4, 0.7, 1.6)[i % 5])) + i
        out.append(dict(kind=i % 3, cloud_type=(i // 2) % 2, n=n, grids=((128, 64), (512, 128), (256, 64))[i % 3],
                        mode=("first_inter", "random_weighted", "first", "random_intra", "first_inter")[i % 5]))
    return out


def prepare(case, seed):
    seed = 20240600 + 7919 * int(seed)
    if case["form"] == "served":
        jobs, keep, hiers = [], [], []
        for i, r in enumerate(_requests(case)):
            stride = 15 if r["cloud_type"] == 0 else 27
            cloud, lo, hi = _cloud(r["kind"], r["cloud_type"], r["n"], stride, seed + i, True)
            cap = _room(r["n"])
            rec, lut = _pinned(cap * 18), _pinned(cap * 4).view(np.uint32)[:cap]
            hier = np.zeros(_nodes(r["n"]) * octree_api.HIER_DTYPE.itemsize, np.uint8)
            m = MODES[r["mode"]]
            flags = ((octree_api.SUB_INTRA if m.get("intra") else 0) | (octree_api.SUB_INTER if m.get("inter") else 0) |
                     (octree_api.SUB_RANDOM if m.get("random") else 0) |
                     (octree_api.SUB_WEIGHTING if m.get("weighting") else 0))
            jobs.append(octree_api.make_job(cloud, n=r["n"], stride=stride, cloud_type=r["cloud_type"],
                                            scale=_scale(r["kind"]), bb_min=lo, bb_max=hi, chunk_grid=r["grids"][0],
                                            merge_threshold=THRESHOLD, output_factor=OUTPUT_FACTOR,
                                            sub_grid=r["grids"][1], flags=flags, records=rec, lut=lut, hierarchy=hier))
            keep.append((cloud, rec, lut))
            hiers.append(hier)
        server = octree_api.Server(0, lanes=SERVED_LANES, memory_budget=40 << 30)
        return dict(case=case, server=server, jobs=jobs, keep=keep, hiers=hiers,
                    columns=[_table(_nodes(r["n"])) for r in _requests(case)])
    call = case["form"] == "call"
    cloud, lo, hi = _cloud(case["kind"], case["cloud_type"], case["n"], case["stride"], seed, call)
    s = octree_api.OctreeSession(0)
    s.set_cloud(cloud, n=case["n"], stride=case["stride"], cloud_type=case["cloud_type"], scale=_scale(case["kind"]),
                bb_min=lo, bb_max=hi)
    s.configure(chunk_grid=case["chunk_grid"], merge_threshold=THRESHOLD, output_factor=OUTPUT_FACTOR,
                sub_grid=case["sub_grid"], seed=0x5EED, **MODES[case["mode"]])
    state = dict(case=case, session=s, columns=_table(_nodes(case["n"])))
    if call:
        cap = _room(case["n"])
        rec = torch.empty(cap * 18, dtype=torch.uint8, pin_memory=True)
        lut = torch.empty(cap, dtype=torch.int32, pin_memory=True)
        s.set_output_host(rec.numpy(), lut.numpy().view(np.uint32))
        state.update(rec=rec, lut=lut)
    else:
        s.init()
    return state


def _columns(hier, table):
    """Hierarchy entries (type, child mask, points, byte offset, byte size) as whole numbers in the first rows of
    the program's table."""
    for j, f in enumerate(("type", "mask", "points", "byte_offset", "byte_size")):
        table[: len(hier), j] = hier[f]
    table[len(hier):] = 0
    return table


def _levels(mask):
    """Level below the root of every node, from the breadth-first child masks."""
    kids = np.unpackbits(np.ascontiguousarray(mask)[:, None], axis=1).sum(axis=1, dtype=np.int64)
    level = np.zeros(len(mask), np.int64)
    begin, end, depth = 0, 1, 0
    while end < len(mask):
        below = int(kids[begin:end].sum())
        begin, end, depth = end, end + below, depth + 1
        level[begin:end] = depth
    return level


def _in_cloud_order(state, hier):
    """The records and cloud indices of every level in the cloud's own order, on the device: a level holds a point
    of the cloud at most once, so (level, index) is a record's place."""
    n = state["case"]["n"]
    order = np.argsort(hier["byte_offset"], kind="stable")
    levels = _levels(hier["mask"])
    level = torch.from_numpy(levels[order]).cuda()
    points = torch.from_numpy(hier["points"].astype(np.int64)[order]).cuda()
    total = int(hier["points"].sum(dtype=np.int64))
    rec = state["rec"][: total * 18].cuda(non_blocking=True).view(torch.int16).view(total, 9)
    lut = state["lut"][:total].cuda(non_blocking=True)
    level_of = torch.repeat_interleave(level, points, output_size=total)
    place = level_of * n + lut
    seen = torch.zeros(int(levels.max() + 1) * n, dtype=torch.int32, device="cuda")
    seen[place] = 1
    rank = (torch.cumsum(seen, 0, dtype=torch.int32) - 1)[place].long()
    room = len(state["lut"])
    out_rec = torch.zeros((room, 9), dtype=torch.int16, device="cuda")
    out_lut = torch.zeros(room, dtype=torch.int32, device="cuda")
    out_level = torch.zeros(room, dtype=torch.int64, device="cuda")
    # (places past the last record stay zero)
    out_rec[rank] = rec
    out_lut[rank] = lut
    out_level[rank] = level_of
    return out_rec, out_lut, out_level


def run(state):
    if state["case"]["form"] == "served":
        server = state["server"]
        tickets = [server.submit(j) for j in state["jobs"]]
        results = [server.wait(t) for t in tickets]
        for t in tickets:
            server.release(t)
        if any(r.status for r in results):
            raise RuntimeError("a request failed: %s" % [r.error for r in results if r.status][:1])
        return [_columns(h.view(octree_api.HIER_DTYPE)[: r.nodeCount], t)
                for h, r, t in zip(state["hiers"], results, state["columns"])]
    s = state["session"]
    if state["case"]["form"] == "call":
        s.init()
        s.generate()
        hier = s.hierarchy()
        rec, lut, level = _in_cloud_order(state, hier)
        return dict(hierarchy=_columns(hier, state["columns"]), records=rec, indices=lut, levels=level)
    s.generate()
    st = s.stats()
    # the mean and deviation of the leaves' point counts follow from the hierarchy
    return dict(hierarchy=_columns(s.hierarchy(), state["columns"]),
                stats=np.array([st[k] for k in ("points_total", "p_in", "p_out", "sparse_nodes", "min_leaf_points",
                                                "max_leaf_points", "max_leaf_depth")], np.int64))


# inner records per point of the cloud, about (a cloud of a few nodes has fewer)
INNER = {0: 0.55, 1: 0.75, 2: 0.95}


def work(case):
    """Bytes: the cloud read once; a record (18) and a cloud index (4) written for every point and every inner
    record.  Operations: per candidate (each point and inner record once) the cell of three coordinates and the sums
    of three colours, per inner record the sums over its 27 cells (and, weighted, a weight of 12 operations for each
    of the about nine points around it)."""
    if case["form"] == "served":
        parts = [(r["kind"], r["n"], 15 if r["cloud_type"] == 0 else 27, r["mode"]) for r in _requests(case)]
    else:
        parts = [(case["kind"], case["n"], case["stride"], case["mode"])]
    b = f = 0.0
    for kind, n, stride, mode in parts:
        inner = INNER[kind] * n
        b += n * stride + 22 * (n + inner)
        f += (n + inner) * (9 + 3)
        if mode.endswith("inter"):
            f += inner * 27 * 3
        if mode.endswith("weighted"):
            f += inner * 9 * (12 + 8)
    return {"bytes": b, "flops": f}
