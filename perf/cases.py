"""Performance cases: what a program has this framework do, through its public entry points.

Kinds of cases (`kind`), all over Zel'dovich-displaced particle lattices in a box of 100 units:

* ``call``     -- the reference boundary: particle patches in host memory, a mass grid in host memory
  (``DepositWrapper.deposit_tets``, float32 as in the reference, or ``deposit_tets_ex``), one call per
  periodic image of the grid box;
* ``device``   -- the same deposit between device buffers (``adeco_deposit_tets_device`` and the form
  that allocates nothing);
* ``octree``   -- ``Session.build_octree`` over a resident lattice;
* ``leaves``   -- ``Session.deposit_leaves`` of a built octree, the masses taken on the device;
* ``workflow`` -- a C host's single-rank run: a session from positions in host memory, octree, deposit, all
  leaf grids into its buffer in host memory;
* ``zoom``     -- a batch of zoom requests against a resident lattice, submitted, waited for, fetched.
"""
import ctypes
import math

import numpy as np
import torch

from adeco_gb300 import _lib, deposit

BOX = 100.0
PAD = 666.0  # a padding vertex of a patch
META = 7     # lattice cubes per meta-cell edge


def listed():
    return [
        # the smallest call a worker makes: one patch onto a leaf-sized grid; latency and launches count
        {"name": "call_smallest", "kind": "call", "cubes": 8, "m": 8, "dims": 16, "rms": 1.0, "images": 1,
         "out": "f32", "precision": 0, "order": 0, "margin": 0.0},
        # the plain configuration: a periodic 64^3 lattice onto a uniform 128^3 grid, 27 image boxes
        {"name": "call_periodic_64", "kind": "call", "cubes": 64, "m": 16, "dims": 128, "rms": 0.5, "images": 27,
         "out": "f32", "precision": 0, "order": 0, "margin": 0.0},
        # the FP64 option of the boundary, FP64 grid
        {"name": "call_fp64", "kind": "call", "cubes": 24, "m": 12, "dims": 40, "rms": 1.0, "images": 1,
         "out": "f64", "precision": 1, "order": 0, "margin": 5.0},
        # device buffers, an odd patch size with padded last patches, the conforming corner order, odd grid
        {"name": "device_ragged", "kind": "device", "cubes": 50, "m": 13, "dims": 75, "rms": 2.0, "alloc": True,
         "order": 1, "margin": 3.0},
        # the entry point that allocates nothing, 512 patches of 7^3 cubes onto its largest grid
        {"name": "device_noalloc_96", "kind": "device", "cubes": 56, "m": 7, "dims": 96, "rms": 1.5, "alloc": False,
         "order": 0, "margin": 0.0},
        # refinement alone, over the 256^3 lattice of the octree configuration
        {"name": "octree_256", "kind": "octree", "n": 256, "rms": 3.0, "infall": 0, "per_cell": 64, "leaf": 16,
         "max_level": 8},
        # a small snapshot, small leaf blocks
        {"name": "leaves_64", "kind": "leaves", "n": 64, "rms": 1.0, "infall": 0, "per_cell": 64, "leaf": 8,
         "max_level": 8},
        # the octree configuration: 256^3, rms displacement 3 spacings, 16^3-cell leaves, depth 8
        {"name": "leaves_256", "kind": "leaves", "n": 256, "rms": 3.0, "infall": 0, "per_cell": 64, "leaf": 16,
         "max_level": 8},
        # strong clustering, with the infall density of the 512^3 configuration (2000 regions there), depth 12
        {"name": "leaves_clustered_256", "kind": "leaves", "n": 256, "rms": 3.0, "infall": 250, "per_cell": 64,
         "leaf": 16, "max_level": 12},
        # a whole single-rank run: upload, octree, deposit, all leaf grids back
        {"name": "workflow_128", "kind": "workflow", "n": 128, "rms": 3.0, "infall": 0, "per_cell": 64, "leaf": 16,
         "max_level": 8},
        # one request as a serving loop sees it: 128^3 cells over a tenth of the box
        {"name": "zoom_one_128", "kind": "zoom", "n": 256, "rms": 3.0, "count": 1, "side_lo": 10.0, "side_hi": 10.0,
         "dims": "128"},
        # a batch of requests of uneven extent and resolution
        {"name": "zoom_batch_24", "kind": "zoom", "n": 256, "rms": 3.0, "count": 24, "side_lo": 1.0, "side_hi": 25.0,
         "dims": "32,64,128,256"},
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["call", "call", "device", "device", "octree", "leaves", "leaves", "workflow", "zoom", "zoom"])
    rms = round(rng.uniform(0.3, 3.0), 3)
    if kind == "call":
        if rng.random() < 0.2:  # FP64 arithmetic
            return {"kind": kind, "cubes": int(log(6, 28)), "m": rng.randint(5, 16), "dims": int(log(8, 48)), "rms": rms,
                    "images": 1, "out": "f64", "precision": 1, "order": rng.randint(0, 1), "margin": rng.uniform(0, 10)}
        cubes = int(log(7, 64))
        return {"kind": kind, "cubes": cubes, "m": rng.randint(5, 24), "dims": max(5, int(cubes * log(0.4, 2.0))),
                "rms": min(rms, 1.0), "images": rng.choice([1, 1, 27]), "out": rng.choice(["f32", "f32", "f64"]),
                "precision": 0, "order": rng.randint(0, 1), "margin": 0.0}
    if kind == "device":
        alloc = rng.random() < 0.5
        cubes = int(log(8, 64))
        dims = max(5, int(cubes * log(0.4, 2.0)))
        return {"kind": kind, "cubes": cubes, "m": rng.randint(7, 21), "dims": dims if alloc else min(dims, 96),
                "rms": rms, "alloc": alloc, "order": rng.randint(0, 1), "margin": rng.uniform(0.0, 8.0)}
    infall = rng.random() < 0.4
    if kind == "zoom":
        lo = log(1.0, 20.0)
        return {"kind": kind, "n": int(log(64, 256)), "rms": rms, "count": rng.randint(1, 6), "side_lo": round(lo, 3),
                "side_hi": round(min(25.0, lo * rng.uniform(1.0, 3.0)), 3),
                "dims": rng.choice(["32", "48,64", "100", "64,128", "128"])}
    n = int(log(40, 240))
    return {"kind": kind, "n": n, "rms": rms, "infall": max(1, int(250 * (n / 256) ** 3)) if infall else 0,
            "per_cell": rng.choice([32, 64, 96]), "leaf": rng.choice([8, 12, 16, 24]), "max_level": rng.randint(5, 12)}


# ------------------------------------------------------------------ inputs
def lattice(n, rms, seed, infall=0):
    """(n, n, n, 3) FP32 positions on the GPU, x fastest: a lattice displaced by the Zel'dovich field of a
    Gaussian random field, P(k) ~ k^-2 exp(-(k / k_c)^2), k_c = 8 2 pi / L, scaled to `rms` spacings;
    `infall` spherical regions with radially compressed particles."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    f64 = dict(dtype=torch.float64, device="cuda")
    dk = torch.fft.rfftn(torch.randn((n, n, n), generator=gen, **f64))
    kf = 2.0 * math.pi / BOX
    kr = torch.fft.rfftfreq(n, d=1.0 / n, **f64) * kf
    kc = torch.fft.fftfreq(n, d=1.0 / n, **f64) * kf
    kx, ky, kz = kr[None, None, :], kc[None, :, None], kc[:, None, None]
    k2 = kx * kx + ky * ky + kz * kz
    k2[0, 0, 0] = 1.0
    dk *= torch.exp(-0.5 * k2 / (8.0 * kf) ** 2) / (k2 * k2.sqrt())
    dk[0, 0, 0] = 0.0
    pos = torch.stack([torch.fft.irfftn(1j * k * dk, s=(n, n, n)) for k in (kx, ky, kz)], dim=-1)
    h = BOX / n
    pos *= rms * h / pos.square().sum(-1).mean().sqrt()
    q = (torch.arange(n, **f64) + 0.5) * h
    pos[..., 0] += q[None, None, :]
    pos[..., 1] += q[None, :, None]
    pos[..., 2] += q[:, None, None]
    if infall:
        draws = torch.rand((infall, 4), generator=gen, **f64).cpu()
        for u in draws.tolist():
            compress(pos, q, [BOX * x for x in u[:3]], 0.5 * 10.0 ** u[3] * h, rms)
    return pos.float()


def compress(pos, q, centre, radius, rms):
    """Pulls the particles within 3 radii of `centre` towards it (an NFW-like profile of concentration 10); a
    particle of another periodic image moves next to this one, so that long, flat tets occur."""
    n, h, reach = len(q), BOX / len(q), 3.0 * radius
    w = int((reach / h) + 4.0 * rms + 4.0)  # lattice sites that may have moved into reach
    at = [(torch.arange(int(c / h) - w, int(c / h) + w + 1, device="cuda") % n).unique() for c in centre]
    win = (at[2][:, None, None], at[1][None, :, None], at[0][None, None, :])
    sub = pos[win]
    c = torch.tensor(centre, dtype=torch.float64, device="cuda")
    d = sub - c
    d -= BOX * torch.round(d / BOX)
    x = d.square().sum(-1).sqrt() / reach
    s = 0.5 + 0.5 * torch.log1p(10.0 * x) / math.log1p(10.0)
    pos[win] = torch.where((x < 1.0)[..., None], c + d * s[..., None], sub)


def ghosted(pos):
    """The lattice with its first planes repeated at the far sides, shifted by the box: its cubes are the periodic ones."""
    for axis, comp in ((2, 0), (1, 1), (0, 2)):
        first = pos.narrow(axis, 0, 1).clone()
        first[..., comp] += BOX
        pos = torch.cat([pos, first], dim=axis)
    return pos


def patches_of(vertices, m):
    """Patches of (m + 1)^3 vertices that share their boundary planes, the last ones padded."""
    k = -(-(vertices.shape[0] - 1) // m)
    full = torch.full((k * m + 1,) * 3 + (3,), PAD, device=vertices.device)
    nv = vertices.shape[0]
    full[:nv, :nv, :nv] = vertices
    p = full.unfold(0, m + 1, m).unfold(1, m + 1, m).unfold(2, m + 1, m)  # (k, k, k, 3, m+1, m+1, m+1)
    return p.permute(0, 1, 2, 4, 5, 6, 3).contiguous().reshape(-1)


def image_boxes(box, images):
    shifts = (0.0,) if images == 1 else (-BOX, 0.0, BOX)
    return [np.array([box[0] + x, box[1] + x, box[2] + y, box[3] + y, box[4] + z, box[5] + z], np.float32)
            for z in shifts for y in shifts for x in shifts]


def boundary_inputs(case, seed):
    pos = lattice(case["cubes"], case["rms"], seed)
    lo, hi = case["margin"], BOX - case["margin"]
    return ghosted(pos), image_boxes([lo, hi, lo, hi, lo, hi], case.get("images", 1))


def requests_of(case, seed):
    rng = np.random.default_rng(seed)
    dims = [int(d) for d in case["dims"].split(",")]
    count = case["count"]
    sides = np.exp(rng.uniform(math.log(case["side_lo"]), math.log(case["side_hi"]), count))
    centres = rng.uniform(0.0, BOX, (count, 3))
    return [(tuple(map(float, c)), float(s), dims[i % len(dims)]) for i, (c, s) in enumerate(zip(centres, sides))]


def max_tets(case):
    return case["per_cell"] * case["leaf"] ** 3


def most_leaves(case):
    """Leaves that a program's buffers have room for."""
    return 64 + 24 * case["n"] ** 3 // max_tets(case)


class DeviceGrids:
    """The session's FP64 leaf grids on the device, for torch.as_tensor."""

    def __init__(self, pointer, count):
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f8", "data": (pointer, False), "version": 3}


# ------------------------------------------------------------------ the passes
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("call", "device"):
        vertices, boxes = boundary_inputs(case, seed)
        patches = patches_of(vertices, case["m"])
        state = {"case": case, "boxes": boxes, "per_patch": 3 * (case["m"] + 1) ** 3}
        if kind == "call":
            state["patches"] = patches.cpu().numpy()
            state["data"] = np.zeros(case["dims"] ** 3, np.float64 if case["out"] == "f64" else np.float32)
        else:
            state["patches"] = patches
            state["data"] = torch.zeros(case["dims"] ** 3, dtype=torch.float64, device="cuda")
            state["lib"] = _lib.load()
        return state
    pos = lattice(case["n"], case["rms"], seed, case.get("infall", 0)).cpu().numpy()
    room = most_leaves(case) * case["leaf"] ** 3 if "leaf" in case else 0
    if kind == "workflow":
        return {"case": case, "positions": pos, "lib": _lib.load(), "grids": np.zeros(room)}
    session = deposit.Session(pos)
    state = {"case": case, "session": session}
    if kind == "octree":
        nodes = 2 * most_leaves(case)
        state["nodes"] = np.zeros((nodes, 7), np.float32)
        state["leaves"] = np.zeros((nodes, 2), np.int64)
    if kind == "leaves":
        session.build_octree(max_tets(case), case["max_level"], case["leaf"])
        state["grids"] = torch.zeros(room, dtype=torch.float64, device="cuda")
    if kind == "zoom":
        state["requests"] = requests_of(case, seed)
    return state


def run(state):
    case = state["case"]
    return {"call": run_call, "device": run_device, "octree": run_octree, "leaves": run_leaves,
            "workflow": run_workflow, "zoom": run_zoom}[case["kind"]](state, case)


def run_call(state, case):
    pos, data = state["patches"], state["data"]
    count = pos.size // state["per_patch"]
    data[:] = 0
    for box in state["boxes"]:
        if case["out"] == "f32" and case["order"] == 0:
            deposit.DepositWrapper.deposit_tets(True, 0, 0, count, pos, pos.size, case["m"], box, case["dims"], data)
        else:
            deposit.deposit_tets_ex(pos, case["m"], box, case["dims"], data=data, precision=case["precision"],
                                    tet_order=case["order"])
    return data


def run_device(state, case):
    pos, out, lib = state["patches"], state["data"], state["lib"]
    box = state["boxes"][0]
    out.zero_()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    args = [ctypes.c_void_p(pos.data_ptr()), pos.numel(), 0, pos.numel() // state["per_patch"], case["m"],
            ctypes.c_void_p(box.ctypes.data), case["dims"], ctypes.c_void_p(out.data_ptr())]
    if case["alloc"]:
        _lib.check(lib.adeco_deposit_tets_device(*args, _lib.PREC_MIXED, case["order"], 1.0, stream))
    else:
        _lib.check(lib.adeco_deposit_tets_device_noalloc(*args, case["order"], 1.0, stream))
    return out


def run_octree(state, case):
    info = state["session"].build_octree(max_tets(case), case["max_level"], case["leaf"])
    nodes, leaves, n = state["nodes"], state["leaves"], len(info.nodes)
    nodes[:n, :3] = info.nodes["min"]
    for i, field in enumerate(("ext", "level", "first_child", "n_meta")):
        nodes[:n, 3 + i] = info.nodes[field]
    leaves[:n, 0] = info.nodes["estimate"]
    leaves[:len(info.leaves), 1] = info.leaves
    return [nodes, leaves]


def run_leaves(state, case):
    session, grids = state["session"], state["grids"]
    session.deposit_leaves(fetch=False)
    got = torch.as_tensor(DeviceGrids(*session.leaf_grids_device()), device="cuda")
    grids[:len(got)] = got
    return grids


def run_workflow(state, case):
    lib, grids, n = state["lib"], state["grids"], case["n"]
    config = _lib.SessionConfig(0, 0, 1.0, 0.75, 1)
    handle = ctypes.c_void_p()
    _lib.check(lib.adeco_session_create(ctypes.byref(config), ctypes.c_void_p(state["positions"].ctypes.data), n, n, n,
                                        ctypes.byref(handle)))
    _lib.check(lib.adeco_session_build_octree(handle, None, None, max_tets(case), case["max_level"], case["leaf"]))
    leaves = ctypes.c_int()
    _lib.check(lib.adeco_session_octree_size(handle, None, ctypes.byref(leaves), None))
    if leaves.value > most_leaves(case):
        raise RuntimeError("the octree has %d leaves, the buffer room for %d" % (leaves.value, most_leaves(case)))
    _lib.check(lib.adeco_session_deposit_leaves(handle, _lib.PREC_MIXED, ctypes.c_void_p(grids.ctypes.data), 0, None))
    _lib.check(lib.adeco_session_destroy(handle))
    return grids


def run_zoom(state, case):
    session, requests = state["session"], state["requests"]
    batch = session.submit(requests)
    session.wait(batch)
    grids = [session.result(batch, i, r[2]) for i, r in enumerate(requests)]
    session.release(batch)
    return grids


# ------------------------------------------------------------------ what a pass cannot do without
PAIR_FLOPS = 100  # of one (tet, cell) pair that overlaps: four plane tests and a volume, at least


def pairs(tets, spacing, cell):
    """Overlapping (tet, cell) pairs of `tets` lattice tets: the cells that the body of a tet of edge `spacing` meets."""
    r = spacing / cell
    return tets * (1.0 + 1.5 * r + 1.2 * r * r + r ** 3 / 6.0)


def work(case):
    kind = case["kind"]
    if kind in ("call", "device"):
        cells, tets = case["dims"] ** 3, 6 * case["cubes"] ** 3
        size = 4 if case.get("out") == "f32" else 8
        width = BOX - 2 * case["margin"]
        return {"bytes": 12.0 * (case["cubes"] + 1) ** 3 + size * cells,
                "flops": PAIR_FLOPS * pairs(tets * (width / BOX) ** 3, BOX / case["cubes"], width / case["dims"])}
    n = case["n"]
    if kind == "zoom":
        h, got = BOX / n, {"bytes": 0.0, "flops": 0.0}
        for _, side, d in requests_of(case, 0):
            inside = (side / h + 1.0) ** 3  # particles of the box
            got["bytes"] += 12.0 * inside + 8.0 * d ** 3
            got["flops"] += PAIR_FLOPS * pairs(6.0 * (side / h) ** 3, h, side / d)
        return got
    metas = (-(-(n - 1) // META)) ** 3
    if kind == "octree":  # every meta-cell's box once, and one estimate per level
        return {"bytes": 24.0 * metas, "flops": 30.0 * metas * 3}
    tets = 6.0 * (n - 1) ** 3
    cells = 4.0 * tets / case["per_cell"]  # a refined node's children hold an eighth of its tets at the most
    return {"bytes": 12.0 * n ** 3 + 8.0 * cells, "flops": PAIR_FLOPS * pairs(tets, 1.0, (tets / 6.0 / cells) ** (1 / 3))}


# ------------------------------------------------------------------ the same in 64 bits
CORNERS = {0: [(0, 0, 0), (1, 0, 0), (0, 1, 0), (1, 1, 0), (0, 1, 1), (1, 1, 1), (0, 0, 1), (1, 0, 1)],
           1: [(s >> 2 & 1, s >> 1 & 1, s & 1) for s in range(8)]}  # offsets (x, y, z) of a cube's 8 corners
TETS = [(1, 0, 2, 4), (4, 2, 1, 3), (3, 5, 1, 4), (4, 5, 6, 3), (3, 2, 6, 4), (3, 7, 5, 6)]
EDGES = [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]


def cut_table():
    """Per mask of a tet's vertices inside a plane: the tets of its inside part, over the 4 vertices and 6 edge points."""
    table = torch.zeros((16, 3, 4), dtype=torch.int64)
    count = torch.zeros(16, dtype=torch.int64)
    for mask in range(1, 16):
        ins = [v for v in range(4) if mask >> v & 1]
        out = [v for v in range(4) if not mask >> v & 1]

        def x(a, b):
            return 4 + EDGES.index((min(a, b), max(a, b)))

        if len(ins) == 4:
            parts = [(0, 1, 2, 3)]
        elif len(ins) == 1:
            parts = [(ins[0], *[x(ins[0], o) for o in out])]
        elif len(ins) == 2:
            (a, b), (c, d) = ins, out
            parts = [(a, b, x(b, c), x(b, d)), (a, x(b, c), x(a, c), x(b, d)), (a, x(a, c), x(a, d), x(b, d))]
        else:
            (a, b, c), (d,) = ins, out
            parts = [(a, b, c, x(c, d)), (a, b, x(c, d), x(b, d)), (a, x(b, d), x(c, d), x(a, d))]
        count[mask] = len(parts)
        for i, p in enumerate(parts):
            table[mask, i] = torch.tensor(p)
    return table.cuda(), count.cuda()


def volume6(p):
    a, b, c = (p[:, i] - p[:, 3] for i in range(3))
    return (a * torch.linalg.cross(b, c)).sum(-1).abs()


def clipped6(p, table, count):
    """6 x the volume inside the unit cube of each tet of p (N, 4, 3)."""
    own = torch.arange(len(p), device="cuda")
    n = len(p)
    first, second = (torch.tensor([e[i] for e in EDGES], device="cuda") for i in (0, 1))
    bit = torch.tensor([1, 2, 4, 8], device="cuda")
    for axis in range(3):
        for upper in (0.0, 1.0):
            x = p[:, :, axis]
            ins = x < 1.0 if upper else x > 0.0
            mask = (ins * bit).sum(1)
            todo = (mask != 0) & (mask != 15)
            rest, rest_own = p[mask == 15], own[mask == 15]
            p, own, mask = p[todo], own[todo], mask[todo]
            xa, xb = p[:, first, axis], p[:, second, axis]
            s = ((upper - xa) / torch.where(xa == xb, torch.ones_like(xa), xb - xa)).clamp(0.0, 1.0)
            e = p[:, first] + s[..., None] * (p[:, second] - p[:, first])
            e[:, :, axis] = upper
            pts = torch.cat([p, e], dim=1)
            parts = [rest]
            owners = [rest_own]
            for i in range(3):
                has = count[mask] > i
                idx = table[mask[has], i][..., None].expand(-1, -1, 3)
                parts.append(torch.gather(pts[has], 1, idx))
                owners.append(own[has])
            p, own = torch.cat(parts), torch.cat(owners)
    return torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, own, volume6(p))


def deposited(tets, box, dims, tables):
    """Masses (dims^3, x fastest) of FP32 tets (N, 4, 3), mass 1 each, on the grid over box (xmin, xmax, ...): a cell
    starts at its index times its axis' cell size and is a cube of the first axis' cell size."""
    grid = torch.zeros(dims ** 3, dtype=torch.float64, device="cuda")
    lo = torch.tensor(np.asarray(box[0::2], np.float64), device="cuda")
    hi = torch.tensor(np.asarray(box[1::2], np.float64), device="cuda")
    delta = (hi - lo) / dims
    scale = 1.0 / delta[0]
    step = delta * scale
    tets = tets[((tets.amin(1) < hi) & (lo < tets.amax(1))).all(1)]
    a, b, c = (tets[:, i] - tets[:, 3] for i in range(3))  # FP32: tets of no FP32 volume have no mass
    flat = (a[:, 0] * (b[:, 1] * c[:, 2] - b[:, 2] * c[:, 1]) + b[:, 0] * (c[:, 1] * a[:, 2] - c[:, 2] * a[:, 1])
            + c[:, 0] * (a[:, 1] * b[:, 2] - a[:, 2] * b[:, 1]))
    t = (tets[flat.abs() > 3 * 2.0 ** -149].double() - lo) * scale
    mn, mx = t.amin(1), t.amax(1)
    c0 = torch.floor((mn - 1.0) / step).long().clamp(min=0)
    c1 = torch.floor(mx / step).long().clamp(max=dims - 1)
    ext = (c1 - c0 + 1).clamp(min=0)
    cells = ext.prod(1)
    share = torch.cumsum(cells, 0)
    total = int(share[-1]) if len(share) else 0
    factor = (delta.prod() * scale ** 3) / volume6(t)
    normals, offsets = face_planes(t)
    start = 0
    while start < len(t):
        base = int(share[start - 1]) if start else 0
        end = max(start + 1, int(torch.searchsorted(share, torch.tensor(base + 6_000_000, device="cuda"))))
        owner = torch.repeat_interleave(torch.arange(start, end, device="cuda"), cells[start:end])
        local = torch.arange(len(owner), device="cuda") - (share[owner] - cells[owner] - base)
        cell = torch.stack([local % ext[owner, 0], local // ext[owner, 0] % ext[owner, 1],
                            local // (ext[owner, 0] * ext[owner, 1])], 1) + c0[owner]
        o = cell * step
        meets = ((mn[owner] < o + 1.0) & (o < mx[owner])).all(1)
        owner, cell, o = owner[meets], cell[meets], o[meets]
        at = torch.einsum("nfa,na->nf", normals[owner], o) - offsets[owner]
        up, down = normals[owner].clamp(min=0).sum(2), normals[owner].clamp(max=0).sum(2)
        keep = (at + up > 0).all(1)
        inside = (at + down > 0).all(1)[keep]
        owner, cell, o = owner[keep], cell[keep], o[keep]
        whole = ((mn[owner] >= o) & (mx[owner] <= o + 1.0)).all(1)
        mass = torch.where(whole, torch.ones_like(factor[owner]), 6.0 * factor[owner])
        part = ~(whole | inside)
        mass[part] = clipped6(t[owner[part]] - o[part][:, None, :], *tables) * factor[owner[part]]
        grid.index_add_(0, cell[:, 0] + dims * (cell[:, 1] + dims * cell[:, 2]), mass)
        start = end
    return grid, total


def face_planes(t):
    """Inward normals (N, 4, 3) and offsets (N, 4) of the tets' faces."""
    faces = [(1, 2, 3, 0), (0, 2, 3, 1), (0, 1, 3, 2), (0, 1, 2, 3)]
    n = torch.stack([torch.linalg.cross(t[:, b] - t[:, a], t[:, c] - t[:, a]) for a, b, c, _ in faces], 1)
    d = torch.stack([(n[:, i] * t[:, f[0]]).sum(-1) for i, f in enumerate(faces)], 1)
    far = torch.stack([(n[:, i] * t[:, f[3]]).sum(-1) for i, f in enumerate(faces)], 1)
    s = torch.where(far < d, -1.0, 1.0)
    return n * s[..., None], d * s


def tets_of(v, order=0):
    """(N, 4, 3) FP32 tets of the cubes of vertices v (nz, ny, nx, 3)."""
    nz, ny, nx = (k - 1 for k in v.shape[:3])
    c = torch.stack([v[z:z + nz, y:y + ny, x:x + nx] for x, y, z in CORNERS[order]], 3).reshape(-1, 8, 3)
    return c[:, torch.tensor(TETS, device="cuda")].reshape(-1, 4, 3)


def octree_leaves(pos, case):
    """The leaves' boxes in depth-first order: nodes refine while their tet estimate, summed over the meta-cells that
    meet them (FP32 terms), is over the limit."""
    n = pos.shape[0]
    k = -(-(n - 1) // META)
    f32 = np.float32
    boxes, cubes = [], []
    for z in range(k):
        slab = pos[z * META:z * META + META + 1]
        for y in range(k):
            row = slab[:, y * META:y * META + META + 1]
            w = [row[:, :, x * META:x * META + META + 1].reshape(-1, 3) for x in range(k)]
            boxes += [torch.cat([b.amin(0), b.amax(0)]) for b in w]
            cubes += [min(META, n - 1 - z * META) * min(META, n - 1 - y * META) * min(META, n - 1 - x * META)
                      for x in range(k)]
    boxes, six = torch.stack(boxes).cpu().numpy(), (6 * np.array(cubes)).astype(f32)
    whole = ((boxes[:, 3] - boxes[:, 0]) * (boxes[:, 4] - boxes[:, 1])) * (boxes[:, 5] - boxes[:, 2])
    mn, mx = boxes[:, :3].min(0), boxes[:, 3:].max(0)
    limit = min(6 * (n - 1) ** 3, max_tets(case))
    leaves, stack = [], [(mn, (mx - mn).max(), 0, np.arange(len(boxes)))]
    while stack:
        low, ext, level, ids = stack.pop()
        high = low + ext
        b = boxes[ids]
        e = np.minimum(high, b[:, 3:]) - np.maximum(low, b[:, :3])
        est = six[ids] * ((e[:, 0] * e[:, 1]) * e[:, 2]) / whole[ids]
        if int(np.maximum(est, 0).astype(np.int64).sum()) <= limit or level >= case["max_level"]:
            leaves.append((low, ext, ids))
            continue
        half = f32(ext / 2)
        for q in range(8):
            corner = low + np.array([q & 1, q >> 1 & 1, q >> 2], f32) * half
            top = corner + half
            stack.append((corner, half, level + 1, ids[((b[:, :3] < top) & (corner < b[:, 3:])).all(1)]))
    return leaves, k


def exact_leaves(case, seed, tables):
    pos = lattice(case["n"], case["rms"], seed, case["infall"])
    leaves, k = octree_leaves(pos, case)
    d, got = case["leaf"], []
    for low, ext, ids in leaves:
        top = low + ext
        box = [low[0], top[0], low[1], top[1], low[2], top[2]]
        tets = [tets_of(pos[z * META:z * META + META + 1, y * META:y * META + META + 1, x * META:x * META + META + 1])
                for x, y, z in ((i % k, i // k % k, i // (k * k)) for i in ids.tolist())]
        got.append(deposited(torch.cat(tets), box, d, tables)[0] if tets
                   else torch.zeros(d ** 3, dtype=torch.float64, device="cuda"))
    return torch.stack(got)


def exact(case, seed):
    kind = case["kind"]
    if kind == "octree" or work(case)["flops"] > 3e10:
        return None
    tables = cut_table()
    if kind in ("call", "device"):
        vertices, boxes = boundary_inputs(case, seed)
        tets = tets_of(vertices, case["order"])
        return sum(deposited(tets, box, case["dims"], tables)[0] for box in boxes)
    if kind in ("leaves", "workflow"):
        grids = exact_leaves(case, seed, tables)
        room = torch.zeros(most_leaves(case) * case["leaf"] ** 3, dtype=torch.float64, device="cuda")
        room[:grids.numel()] = grids.reshape(-1)
        return room
    pos = lattice(case["n"], case["rms"], seed)
    got = []
    for centre, side, d in requests_of(case, seed):
        half, c = np.float32(0.5) * np.float32(side), np.asarray(centre, np.float32)
        box = [c[0] - half, c[0] + half, c[1] - half, c[1] + half, c[2] - half, c[2] + half]
        grid = torch.zeros(d ** 3, dtype=torch.float64, device="cuda")
        for z in range(0, pos.shape[0] - 1, 32):  # slabs of the lattice
            grid += deposited(tets_of(pos[z:z + 33]), box, d, tables)[0]
        got.append(grid.reshape(d, d, d))
    return got
