"""Performance cases: what programs do with this framework, through its public entry points.

A case is one repeated unit of work of such a program: a stencil step, a time loop, an update of a
block map with staged points, a rebuild of the map, a re-tagging after a removal, a ghost exchange,
a quantum of a batch of grids.  Domains, point sets and parameters are those of this repository's
benchmark configurations (a shell in 128^3, unions of balls in 512^3, the reference's Conv3x3x3
grid in 1000^3, clustered inserts in 1024^3, ghost slabs of a 2x2x2 split, uneven batched grids) or
generic ragged ones.  The geometry follows from the case alone, so that results have one shape; values, the order and
place of inserted points and the points that are missing follow the seed.

All grids are 3-D with float32 stencil fields; the insert cases mix float32, float64, int32 and
uint8 properties.
"""
import math
import random

import numpy as np
import torch

import openfpm_data_b200 as sgb
from openfpm_data_b200 import workloads as W

DEV = "cuda" if torch.cuda.is_available() else "cpu"
HEAT_PRM = [W.HEAT_DT]
GS_PRM = [W.GS_PARAMS[k] for k in ("Du", "Dv", "F", "k", "dt")]
KIND = {"heat": sgb.HEAT7, "gs": sgb.GS7, "box27": sgb.BOX27, "box27_ns": sgb.BOX27_NS}
NF = {"heat": 1, "gs": 2, "box27": 1, "box27_ns": 1}
BCK = {"heat": [0.0], "gs": [1.0, 0.0], "box27": [0.0], "box27_ns": [0.0]}
TORCH = {"f32": torch.float32, "f64": torch.float64, "i32": torch.int32, "u8": torch.uint8}


def listed():
    def grid(nx, ny, nz, **kw):
        return dict(nx=nx, ny=ny, nz=nz, **kw)

    balls512 = grid(512, 512, 512, scene="balls", nballs=40, rmin=16.0, rmax=48.0)
    return [
        # one explicit step of the small heat problem (379 chunks): what a coupled program that looks
        # at the field after each step calls; launch and latency count
        dict(name="heat_step_128", op="step", kind="heat", edge=8, lin="smb", boxed=False,
             **grid(128, 128, 128, scene="shell", rmin=20.0, rmax=32.0)),
        # the whole 100-step solve of it
        dict(name="heat_solve_128", op="solve", kind="heat", edge=8, lin="smb", steps=100,
             **grid(128, 128, 128, scene="shell", rmin=20.0, rmax=32.0)),
        # a heat time loop on a ragged, elongated domain whose last chunks are cut
        dict(name="heat_ragged", op="solve", kind="heat", edge=8, lin="smb", steps=31,
             **grid(509, 301, 211, scene="balls", nballs=9, rmin=25.0, rmax=60.0)),
        # Gray-Scott on the 512^3 grid, the headline workload: the steps between two outputs
        dict(name="gs_512", op="solve", kind="gs", edge=8, lin="smb", steps=50, **balls512),
        # Gray-Scott on 4^3 chunks (thin structures), ragged domain
        dict(name="gs_chunk4", op="solve", kind="gs", edge=4, lin="smb", steps=20,
             **grid(250, 190, 131, scene="balls", nballs=10, rmin=20.0, rmax=45.0)),
        # heat on Morton chunk ids (SparseGridGpu_z)
        dict(name="heat_morton", op="solve", kind="heat", edge=8, lin="zmb", steps=20,
             **grid(256, 256, 256, scene="balls", nballs=12, rmin=20.0, rmax=48.0)),
        # Conv3x3x3 on the reference's benchmark grid
        dict(name="box27_1000", op="step", kind="box27", edge=8, lin="smb", boxed=False,
             **grid(1000, 1000, 1000, scene="shell", rmin=56.0, rmax=128.0)),
        # a small update of an existing map: a few thousand points, mixed types and reductions
        dict(name="update_5k", op="update", edge=8, types="f32,f64,i32", ops="smax_,sLeft_,sRight_", npts=5003,
             **grid(128, 128, 128, scene="balls", nballs=8, rmin=12.0, rmax=24.0)),
        # rebuild of a large map: clear, three rounds of 2M clustered inserts with duplicates and a flush
        # each (the later ones merge into the map), boundary tagging, one 27-point average
        dict(name="rebuild_1024", op="rebuild", edge=8, npts=2000000, rounds=3, nclusters=64, sigma=16.0,
             **grid(1024, 1024, 1024)),
        # re-tagging of the 512^3 grid after a block of points was removed
        dict(name="retag_512", op="retag", edge=8, lin="smb", nn="star", **balls512),
        # ghost exchange: pack six slabs, replace them in the neighbour
        dict(name="ghost_512", op="ghost", edge=8, width=1, **balls512),
        # a quantum of steps of a batch of heat grids of uneven sizes, and their states handed back
        dict(name="batch_heat", op="batch", kind="heat", edge=8, steps=20, ngrids=48, emin=32, emax=384, nx=0, ny=0, nz=0),
    ]


def draw(rng: random.Random):
    def logu(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    def dims(a, b):
        return dict(zip(("nx", "ny", "nz"), (int(round(logu(a, b))) for _ in range(3))))

    def balls(d, most):
        m = min(d["nx"], d["ny"], d["nz"])
        lo = rng.uniform(0.08, 0.15) * m
        return dict(scene="balls", nballs=int(round(logu(1, most))), rmin=round(lo, 1), rmax=round(lo * rng.uniform(1.2, 2.2), 1))

    def volume(c):
        r = 0.5 * (c["rmin"] + c["rmax"])
        return min(c["nballs"] * 4.2 * r ** 3, c["nx"] * c["ny"] * c["nz"]) + 1.0

    op = rng.choice(["step", "step", "solve", "solve", "solve", "update", "rebuild", "retag", "ghost", "batch"])
    if op in ("step", "solve"):
        kind = rng.choice(["heat", "gs", "box27", "box27_ns"] if op == "step" else ["heat", "gs"])
        d = dims(64, 512)
        c = dict(op=op, kind=kind, edge=rng.choice([8, 8, 8, 4]), lin=rng.choice(["smb", "smb", "smb", "zmb"]), **d, **balls(d, 40))
        if op == "step":
            c["boxed"] = rng.random() < 0.25
        else:
            slow = 8.0 if c["edge"] == 4 or c["lin"] == "zmb" else 1.0
            c["steps"] = max(1, min(int(round(logu(3, 120))), int(1.5e8 / slow / volume(c))))
        return c
    if op == "update":
        d = dims(64, 300)
        types, ops = rng.choice([("f32,f64,i32", "smax_,sLeft_,sRight_"), ("f32", "sRight_"), ("u8,f32", "sLeft_,smin_"),
                                 ("i32,f32", "sBitwiseOr_,sLeft_")])
        return dict(op=op, edge=rng.choice([8, 8, 4]), types=types, ops=ops, npts=int(logu(1000, 1e6)), **d, **balls(d, 20))
    if op == "rebuild":
        n = int(logu(3e4, 1.5e6))
        s = int(logu(200, 1000))
        return dict(op=op, edge=8, npts=n, rounds=rng.choice([1, 2, 3]), nclusters=rng.randint(4, 64), sigma=round(s * rng.uniform(0.01, 0.022), 2),
                    nx=s, ny=s - rng.randint(0, 60), nz=s - rng.randint(0, 60))
    if op == "retag":
        d = dims(100, 512)
        return dict(op=op, edge=rng.choice([8, 8, 4]), lin=rng.choice(["smb", "zmb"]), nn=rng.choice(["star", "star", "full"]), **d, **balls(d, 40))
    if op == "ghost":
        d = dims(100, 512)
        return dict(op=op, edge=8, width=rng.choice([1, 1, 2, 3]), **d, **balls(d, 40))
    lo = int(logu(24, 96))
    return dict(op="batch", kind=rng.choice(["heat", "gs"]), edge=8, steps=rng.randint(3, 20), ngrids=rng.randint(4, 48), emin=lo,
                emax=int(lo * logu(1.5, 3.0)), nx=0, ny=0, nz=0)


# ------------------------------------------------------------------ geometry
def _rng(seed, salt=0):
    return np.random.default_rng([int(seed), 77, salt])


def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1009 + salt)
    return g


def _size(case):
    return (case["nx"], case["ny"], case["nz"])


def _bsz(size, edge):
    return [-(-s // edge) for s in size]


def _spread3(v):
    out = torch.zeros_like(v)
    for i in range(12):
        out |= ((v >> i) & 1) << (3 * i)
    return out


def _chunk_keys(bc, bsz, lin):
    if lin == "zmb":
        return _spread3(bc[:, 0]) | _spread3(bc[:, 1]) << 1 | _spread3(bc[:, 2]) << 2
    return bc[:, 0] + bsz[0] * (bc[:, 1] + bsz[1] * bc[:, 2])


def _offsets(edge):
    p = torch.arange(edge ** 3, device=DEV)
    return torch.stack([p % edge, (p // edge) % edge, p // (edge * edge)], dim=1)


def _balls(case):
    """Centres [k, 3] and radii [k] (outer, inner) of a scene."""
    rng = _rng(case["nx"] * 1000003 + case["ny"] * 1009 + case["nz"], int(10 * case["rmax"]))
    size = np.array(_size(case), dtype=np.float64)
    if case["scene"] == "shell":
        c = np.floor(size / 2)[None, :] + rng.uniform(-0.5, 0.5, size=(1, 3))
        return c, np.array([case["rmax"]]), np.array([case["rmin"]])
    k = case["nballs"]
    r = np.linspace(case["rmin"], case["rmax"], k)
    if case.get("kind", "").startswith("box27"):
        # clear of the domain's faces (an NNFull neighbour of a chunk at a low face wraps around)
        lo = np.minimum(r[:, None] + 9, size[None, :] / 2)
        c = lo + rng.uniform(0, 1, size=(k, 3)) * np.maximum(size[None, :] - 2 * lo, 0)
    else:
        c = rng.uniform(0, 1, size=(k, 3)) * size[None, :]
    return c, r, np.full(k, -1.0)


def _occupancy(size, edge, lin, centres, outer, inner, margin=0):
    """Block map of a union of balls / shells: sorted keys [n], block coordinates [n, 3], existence [n, bs]."""
    bsz = _bsz(size, edge)
    half = (edge - 1) / 2.0
    diag = half * math.sqrt(3.0) + 1e-6
    bx, by, bz = (torch.arange(b, device=DEV) for b in bsz)
    near = torch.zeros(bsz[2], bsz[1], bsz[0], dtype=torch.bool, device=DEV)
    for c, r, q in zip(centres, outer, inner):
        d = [((b * edge + half).double() - float(c[i])) ** 2 for i, b in enumerate((bx, by, bz))]
        dist = (d[2][:, None, None] + d[1][None, :, None] + d[0][None, None, :]).sqrt_()
        near |= (dist <= r + diag) & (dist >= q - diag)
    zyx = near.nonzero()
    bc = zyx.flip(1)
    off = _offsets(edge)
    pt = bc[:, None, :] * edge + off[None, :, :]
    ok = torch.ones(pt.shape[:2], dtype=torch.bool, device=DEV)
    for d in range(3):
        ok &= (pt[:, :, d] < size[d] - margin) & (pt[:, :, d] >= margin)
    ex = torch.zeros_like(ok)
    ptd = [pt[:, :, d].double() for d in range(3)]
    for c, r, q in zip(centres, outer, inner):
        d2 = (ptd[0] - float(c[0])) ** 2 + (ptd[1] - float(c[1])) ** 2 + (ptd[2] - float(c[2])) ** 2
        ex |= (d2 <= float(r) ** 2) & (d2 >= float(q) * abs(float(q)))
    ex &= ok
    keep = ex.any(dim=1)
    bc, ex = bc[keep], ex[keep]
    keys = _chunk_keys(bc, bsz, lin)
    order = torch.argsort(keys)
    return keys[order].contiguous(), bc[order], ex[order].contiguous()


def _scene(case):
    margin = 9 if case.get("kind", "").startswith("box27") else 0
    return _occupancy(_size(case), case["edge"], case.get("lin", "smb"), *_balls(case), margin=margin)


def _fields(kind, bc, ex, edge, centres, seed):
    """Initial values in chunk layout [n, bs]: uniform noise (heat, box27), or Gray-Scott's u = 1, v = 0 with a
    perturbed cube at each centre."""
    gen = _gen(seed)
    if kind != "gs":
        f = torch.rand(ex.shape, generator=gen, device=DEV)
        return [torch.where(ex, f, torch.zeros_like(f))]
    pt = bc[:, None, :] * edge + _offsets(edge)[None, :, :]
    cube = torch.zeros_like(ex)
    for c in centres:
        inside = torch.ones_like(ex)
        for d in range(3):
            f = math.floor(float(c[d]))
            inside &= (pt[:, :, d] >= f - 3) & (pt[:, :, d] < f + 3)
        cube |= inside
    a = 2 * torch.rand(ex.shape, generator=gen, device=DEV) - 1
    b = 2 * torch.rand(ex.shape, generator=gen, device=DEV) - 1
    cube &= ex
    u = torch.where(cube, 0.5 * (1 + 0.01 * a), torch.ones_like(a))
    v = torch.where(cube, 0.25 * (1 + 0.01 * b), torch.zeros_like(b))
    return [u, v]


def _coeffs(case):
    """27 weights of a smoothing kernel, different along the axes."""
    w = [[0.2, 0.55, 0.25], [0.25, 0.5, 0.25], [0.3, 0.45, 0.25]]
    return [float(np.float32(w[0][a] * w[1][b] * w[2][c])) for a in range(3) for b in range(3) for c in range(3)]


def _params(case):
    return HEAT_PRM if case["kind"] == "heat" else GS_PRM if case["kind"] == "gs" else _coeffs(case)


def _box(case):
    s = _size(case)
    return ([s[0] // 5, s[1] // 7, s[2] // 4], [s[0] - s[0] // 6, s[1] - s[1] // 9, s[2] - s[2] // 5])


def _cut(case):
    """A block of points inside the domain, about a thirtieth of it."""
    s = _size(case)
    return ([(5 * v) // 9 for v in s], [(5 * v) // 9 + v // 3 for v in s])


def _holes(case, seed, bc, ex):
    """The scene without a hundredth of its points (as many for every seed), none of them in _cut()."""
    lo, hi = (torch.tensor(v, device=DEV) for v in _cut(case))
    pt = bc[:, None, :] * case["edge"] + _offsets(case["edge"])[None, :, :]
    pos = (ex & ~((pt >= lo) & (pt <= hi)).all(dim=2)).reshape(-1).nonzero().squeeze(1)
    gone = pos[torch.randperm(len(pos), generator=_gen(seed, 6), device=DEV)[: len(pos) // 100]]
    out = ex.clone().reshape(-1)
    out[gone] = False
    return out.reshape(ex.shape)


def _make_grid(size, kind, edge, lin, keys, ex, fields):
    nf = NF[kind]
    g = sgb.SparseGridGpu(size, ["f32"] * (2 * nf), edge=edge, linearizer=lin)
    for j in range(2 * nf):
        g.setBackgroundValue(j, BCK[kind][j % nf])
    data = [f.reshape(-1).contiguous() for f in fields]
    rest = [torch.full_like(d, BCK[kind][j]) for j, d in enumerate(data)]
    g.load_map_dev(keys, data + rest, ex.to(torch.uint8).reshape(-1))
    torch.cuda.synchronize()
    return g


# ------------------------------------------------------------------ staged points
def _cluster_round(case, seed, k):
    """Coordinates int32 [n, 3] and values of one round of clustered inserts with 30 % exact duplicates."""
    size = np.array(_size(case))
    rng = _rng(case["npts"] + case["nx"], 3)  # the clusters stay over the rounds
    margin = np.minimum(4.5 * case["sigma"] + 10, size / 2.5)
    cen = torch.from_numpy(margin + rng.uniform(0, 1, size=(case["nclusters"], 3)) * (size - 2 * margin)).to(DEV)
    n = case["npts"]
    gen = _gen(case["npts"] + case["nx"], k)
    fresh = n - int(round(0.3 * n))
    which = torch.randint(0, case["nclusters"], (fresh,), generator=gen, device=DEV)
    pts = torch.round(cen[which] + case["sigma"] * torch.randn((fresh, 3), generator=gen, device=DEV, dtype=torch.float64))
    hi = torch.tensor([s - 42 for s in size.tolist()], device=DEV, dtype=torch.float64)
    pts = torch.minimum(pts.clamp(min=9), hi).to(torch.int32)
    # the seed moves the whole set by up to three chunks, picks the repeated points and orders the inserts
    gen = _gen(seed, 50 + k)
    move = _rng(seed, 4).integers(0, 4, size=3) * case["edge"]
    pts = pts + torch.from_numpy(move.astype(np.int32)).to(DEV)
    dup = pts[torch.randint(0, fresh, (n - fresh,), generator=gen, device=DEV)]
    pts = torch.cat([pts, dup])[torch.randperm(n, generator=gen, device=DEV)].contiguous()
    f = torch.rand(n, generator=gen, device=DEV)
    i = torch.randint(-(2 ** 31), 2 ** 31 - 1, (n,), generator=gen, device=DEV).to(torch.int32)
    return pts, f, i


def _values(t, n, gen):
    if t in ("f32", "f64"):
        return torch.rand(n, generator=gen, device=DEV, dtype=TORCH[t])
    return torch.randint(0, 200, (n,), generator=gen, device=DEV).to(TORCH[t])


def _update_points(case, seed, bc):
    """Points inside the map's chunks (existing or not), some of them more than once."""
    gen = _gen(seed, 5)
    n = case["npts"]
    size = torch.tensor(_size(case), device=DEV)
    ch = torch.randint(0, bc.shape[0], (n,), generator=gen, device=DEV)
    o = torch.randint(0, case["edge"], (n, 3), generator=gen, device=DEV)
    pts = torch.minimum(bc[ch] * case["edge"] + o, size - 1)
    # a point past a cut chunk is moved onto the domain's last layer, which the chunk holds
    return pts.to(torch.int32).contiguous(), [_values(t, n, gen) for t in case["types"].split(",")]


def _slabs(case):
    """The ghost slabs on both sides of the three mid planes (inclusive boxes)."""
    s, w, out = _size(case), case["width"], []
    for a in range(3):
        m = s[a] // 2
        for lo_a, hi_a in ((m - w, m - 1), (m, m + w - 1)):
            lo, hi = [0, 0, 0], [v - 1 for v in s]
            lo[a], hi[a] = lo_a, hi_a
            out.append((lo, hi))
    return out


def _batch_members(case):
    rng = _rng(case["ngrids"] * 1000 + case["emax"], 9)
    edges = np.exp(np.linspace(math.log(case["emin"]), math.log(case["emax"]), case["ngrids"]))
    edges = (np.rint(edges / 8) * 8).astype(int).clip(16)
    radii = rng.uniform(0.25, 0.5, size=case["ngrids"]) * edges
    return [(int(e), float(r)) for e, r in zip(edges, radii)]


def _member(case, seed, k, e, r):
    c = np.array([[e / 2.0] * 3])
    keys, bc, ex = _occupancy((e, e, e), case["edge"], "smb", c, [r], [-1.0])
    return keys, bc, ex, _fields(case["kind"], bc, ex, case["edge"], c, seed + 7919 * k)


# ------------------------------------------------------------------ prepare / run
def _held(g, t):
    """A view of a buffer of grid g that keeps the grid (which owns the memory) alive."""
    t.owner = g
    return t


def prepare(case, seed):
    op, size, edge = case["op"], _size(case), case["edge"]
    if op in ("step", "solve"):
        kind, nf = case["kind"], NF[case["kind"]]
        keys, bc, ex = _scene(case)
        g = _make_grid(size, kind, edge, case["lin"], keys, ex, _fields(kind, bc, ex, edge, _balls(case)[0], seed))
        views = [_held(g, g.private_get_data_array(p)) for p in range(2 * nf)]
        return dict(op=op, g=g, kind=KIND[kind], src=list(range(nf)), dst=list(range(nf, 2 * nf)), prm=_params(case),
                    box=_box(case) if case.get("boxed") else None, steps=case.get("steps", 1), views=views, nf=nf)
    if op == "update":
        keys, bc, ex = _scene(case)
        types = case["types"].split(",")
        g = sgb.SparseGridGpu(size, types, edge=edge)
        gen = _gen(seed, 4)
        data = [(_values(t, ex.numel(), gen) * ex.reshape(-1)).to(TORCH[t]) for t in types]
        g.load_map_dev(keys, data, ex.to(torch.uint8).reshape(-1))
        pts, vals = _update_points(case, seed, bc)
        torch.cuda.synchronize()
        views = [_held(g, g.private_get_data_array(p)) for p in range(len(types))] + [_held(g, g.private_get_mask_array())]
        return dict(op=op, g=g, pts=pts, vals=vals, ops=case["ops"].split(","), views=views)
    if op == "rebuild":
        g = sgb.SparseGridGpu(size, ["f32", "i32", "f32"], edge=edge)
        rounds = [_cluster_round(case, seed, k) for k in range(case["rounds"])]
        none = [torch.empty(0, dtype=t, device=DEV) for t in (torch.int64, torch.float32, torch.int32, torch.float32, torch.uint8)]
        return dict(op=op, g=g, rounds=rounds, none=none, coeff=[float(np.float32(1.0 / 27.0))] * 27)
    if op == "retag":
        keys, bc, ex = _scene(case)
        ex = _holes(case, seed, bc, ex)
        g = _make_grid(size, "heat", edge, case["lin"], keys, ex, _fields("heat", bc, ex, edge, None, seed))
        return dict(op=op, g=g, nn=sgb.NN_STAR if case["nn"] == "star" else sgb.NN_FULL, box=_cut(case),
                    mask=_held(g, g.private_get_mask_array()))
    if op == "ghost":
        keys, bc, ex = _scene(case)
        cen = _balls(case)[0]
        a, b = (_make_grid(size, "gs", edge, "smb", keys, ex, _fields("gs", bc, ex, edge, cen, seed + k)) for k in (0, 500))
        return dict(op=op, a=a, b=b, slabs=_slabs(case),
                    views=[_held(b, b.private_get_data_array(p)) for p in (0, 1)] + [_held(b, b.private_get_mask_array())])
    nf = NF[case["kind"]]
    b = sgb.Batch()
    grids, slots, views = [], [], []
    for k, (e, r) in enumerate(_batch_members(case)):
        keys, bc, ex, f = _member(case, seed, k, e, r)
        g = _make_grid((e, e, e), case["kind"], edge, "smb", keys, ex, f)
        slots.append(b.add(g, KIND[case["kind"]], list(range(nf)), list(range(nf, 2 * nf)), _params(case), 10 ** 9))
        grids.append(g)
        views.append([_held(g, g.private_get_data_array(p)) for p in range(2 * nf)])
    return dict(op=op, b=b, grids=grids, slots=slots, views=views, steps=case["steps"], nf=nf)


def run(s):
    op = s["op"]
    if op == "step":
        s["g"].applyStencils(s["kind"], s["src"], s["dst"], s["prm"], box=s["box"])
        return s["views"][s["nf"]:]
    if op == "solve":
        fin = s["g"].run_steps(s["kind"], s["src"], s["dst"], s["prm"], s["steps"])
        return s["views"][s["nf"]:] if fin else s["views"][: s["nf"]]
    if op == "update":
        s["g"].insert(s["pts"], s["vals"])
        s["g"].flush(s["ops"])
        return s["views"]
    if op == "rebuild":
        g, none = s["g"], s["none"]
        g.load_map_dev(none[0], none[1:4], none[4])
        for pts, f, i in s["rounds"]:
            g.insert(pts, [f, i, None])
            g.flush(["sRight_", "sRight_"])
        g.tagBoundaries(sgb.NN_STAR)
        g.applyStencils(sgb.BOX27, [0], [2], s["coeff"])
        out = [g.private_get_index_array()] + [g.private_get_data_array(p) for p in range(3)] + [g.private_get_mask_array()]
        return [_held(g, t) for t in out]
    if op == "retag":
        g = s["g"]
        g.remove(s["box"])
        g.removePoints()
        g.findNeighbours(s["nn"])
        g.tagBoundaries(s["nn"], calculate_existing_points=True)
        return [s["mask"], g.existing_point_list()]
    if op == "ghost":
        a, b = s["a"], s["b"]
        a.packReset()
        for bx in s["slabs"]:
            a.packRequest(bx)
        buf = torch.empty(a.packCalculate([0, 1]), dtype=torch.uint8, device="cuda")
        a.packFinalize(buf, [0, 1])
        for bx in s["slabs"]:
            b.remove(bx)
        b.unpack_boxes(buf, [0, 1], [bx[0] for bx in s["slabs"]])
        b.removeAddUnpackFinalize([0, 1])
        return [buf] + s["views"]
    b, nf = s["b"], s["nf"]
    b.step(s["steps"])
    out = []
    for slot, g, v in zip(s["slots"], s["grids"], s["views"]):
        fin = b.extract(slot, g)
        out.append(v[nf] if fin else v[0])
    return out


# ------------------------------------------------------------------ work and tolerances
def _count(case):
    """(existing points, chunks) of the scene of one seed."""
    _, _, ex = _scene(case)
    return int(ex.sum()), ex.shape[0]


STEP_BYTES = {"heat": 9, "gs": 17, "box27": 9, "box27_ns": 9}  # fields read and written, a mask byte
STEP_FLOPS = {"heat": 9, "gs": 32, "box27": 54, "box27_ns": 54}


def work(case):
    """Each input read once and each output written once; a time loop does that in every step (a step's input is
    the step before it)."""
    op = case["op"]
    if op in ("step", "solve"):
        n = _count(case)[0] * case.get("steps", 1)
        return dict(bytes=n * STEP_BYTES[case["kind"]], flops=n * STEP_FLOPS[case["kind"]])
    if op == "update":
        es = sum({"f32": 4, "f64": 8, "i32": 4, "u8": 1}[t] for t in case["types"].split(","))
        return dict(bytes=case["npts"] * (12 + 3 * es + 2), flops=0)  # staged point in, old value in, new value out
    if op == "rebuild":
        pts = torch.cat([_cluster_round(case, 1, k)[0] for k in range(case["rounds"])])
        bs = _bsz(_size(case), case["edge"])
        b = (pts // case["edge"]).long()
        n = int(torch.unique(b[:, 0] + bs[0] * (b[:, 1] + bs[1] * b[:, 2])).numel())
        u = int(torch.unique(pts[:, 0].long() + 1024 * (pts[:, 1].long() + 1024 * pts[:, 2].long())).numel())
        return dict(bytes=pts.shape[0] * 20 + n * (8 + case["edge"] ** 3 * 13), flops=54 * u)
    if op == "retag":
        n = _count(case)
        return dict(bytes=n[1] * (2 * case["edge"] ** 3 + 8) + 8 * n[0], flops=0)  # masks in and out, the list (int64) out
    if op == "ghost":
        s, w = _size(case), case["width"]
        n, c = _count(case)
        share = 2 * w * sum(1.0 / v for v in s)
        return dict(bytes=max(1.0, n * share * (8 + 11 + 11 + 9)), flops=0)  # values in, packed out and in, values and masks out
    n = sum(4.19 * r ** 3 for _, r in _batch_members(case))
    return dict(bytes=n * (STEP_BYTES[case["kind"]] * case["steps"] + 8 * NF[case["kind"]]), flops=n * case["steps"] * STEP_FLOPS[case["kind"]])


def tolerance(case):
    op = case["op"]
    if op in ("step", "solve", "batch"):
        if case["kind"] == "gs":
            return dict(rel=5e-6, max=1e-3)   # the reaction amplifies float32 rounding over the steps
        return dict(rel=5e-7, max=2e-5)
    if op == "rebuild":
        return dict(rel=5e-7, max=1e-5)       # keys, masks and inserted values exactly, one 27-point sum
    return "exact"


# ------------------------------------------------------------------ the same results in 64 bits
class _Points:
    """The existing points of a block map as a flat list, with their neighbours' places in it."""

    def __init__(self, size, edge, bc, ex):
        self.size = size
        pt = (bc[:, None, :] * edge + _offsets(edge)[None, :, :]).reshape(-1, 3)
        self.pos = ex.reshape(-1).nonzero().squeeze(1)
        self.xyz = pt[self.pos]
        self.n = len(self.pos)
        self.total = (ex.shape[0] + 1) * edge ** 3
        self.dense = torch.full((size[0] * size[1] * size[2],), self.n, dtype=torch.int32, device=DEV)
        self.dense[self._lin(self.xyz)] = torch.arange(self.n, dtype=torch.int32, device=DEV)

    def _lin(self, p):
        return p[:, 0] + self.size[0] * (p[:, 1] + self.size[1] * p[:, 2])

    def at(self, dx, dy, dz):
        """Place of the neighbour at (dx, dy, dz) of every point; n where there is none."""
        q = self.xyz + torch.tensor([dx, dy, dz], device=DEV)
        ok = torch.ones(self.n, dtype=torch.bool, device=DEV)
        for d in range(3):
            ok &= (q[:, d] >= 0) & (q[:, d] < self.size[d])
        i = self.dense[torch.where(ok, self._lin(q), torch.zeros_like(ok, dtype=torch.int64))].long()
        return torch.where(ok, i, torch.full_like(i, self.n))

    def take(self, f, bck):
        """float64 values of the points from a chunk-layout array, the background behind them."""
        return torch.cat([f.reshape(-1)[self.pos].double(), torch.tensor([bck], dtype=torch.float64, device=DEV)])

    def chunks(self, v, bck):
        out = torch.full((self.total,), float(bck), dtype=torch.float64, device=DEV)
        out[self.pos] = v[: self.n]
        return out


STAR = [(-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1), (0, 0, 1)]


def _f32(v):
    return float(np.float32(v))


def _march(P, kind, fields, steps):
    bck = BCK[kind]
    nb = [P.at(*d) for d in STAR]
    x = [P.take(f, b) for f, b in zip(fields, bck)]

    def lap(f):
        s = -6.0 * f[: P.n]
        for i in nb:
            s = s + f[i]
        return s

    prm = [_f32(v) for v in (HEAT_PRM if kind == "heat" else GS_PRM)]
    for _ in range(steps):
        if kind == "heat":
            x[0] = torch.cat([x[0][: P.n] + prm[0] * lap(x[0]), x[0][P.n:]])
        else:
            u, v = x[0][: P.n], x[1][: P.n]
            uvv = u * v * v
            du = prm[0] * lap(x[0]) - uvv + prm[2] * (1.0 - u)
            dv = prm[1] * lap(x[1]) + uvv - (prm[2] + prm[3]) * v
            x = [torch.cat([u + prm[4] * du, x[0][P.n:]]), torch.cat([v + prm[4] * dv, x[1][P.n:]])]
    return x


def _box27(P, x, coeff, xouter):
    acc = torch.zeros(P.n, dtype=torch.float64, device=DEV)
    for a in range(3):
        for b in range(3):
            for c in range(3):
                d = (a - 1, b - 1, c - 1) if xouter else (c - 1, b - 1, a - 1)
                acc += _f32(coeff[a * 9 + b * 3 + c]) * x[P.at(*d)]
    return acc


def exact(case, seed):
    op, size, edge = case["op"], _size(case), case["edge"]
    if op in ("step", "solve"):
        kind = case["kind"]
        _, bc, ex = _scene(case)
        f = _fields(kind, bc, ex, edge, _balls(case)[0], seed)
        P = _Points(size, edge, bc, ex)
        if kind.startswith("box27"):
            new = [_box27(P, P.take(f[0], 0.0), _coeffs(case), kind == "box27")]
        else:
            new = _march(P, kind, f, case.get("steps", 1))
        if case.get("boxed"):  # outside the box heat copies its source, the others leave the destination
            lo, hi = (torch.tensor(v, device=DEV) for v in _box(case))
            inb = ((P.xyz >= lo) & (P.xyz <= hi)).all(dim=1)
            old = [P.take(f[0], 0.0)[: P.n]] if kind == "heat" else [torch.full((P.n,), b, dtype=torch.float64, device=DEV) for b in BCK[kind]]
            new = [torch.where(inb, v[: P.n], o) for v, o in zip(new, old)]
        return [P.chunks(v, b) for v, b in zip(new, BCK[kind])]
    if op == "rebuild":
        allp, allf = [], []
        for k in range(case["rounds"]):
            pts, f, _ = _cluster_round(case, seed, k)
            p = pts.long()
            lin = p[:, 0] + size[0] * (p[:, 1] + size[1] * p[:, 2])
            order = torch.argsort(lin, stable=True)
            s = lin[order]
            last = torch.ones_like(s, dtype=torch.bool)
            last[:-1] = s[1:] != s[:-1]           # the last insert of a point stands
            allp.append(s[last])
            allf.append(f[order][last].double())
        lin, f = allp[0], allf[0]
        for p2, f2 in zip(allp[1:], allf[1:]):    # a point that is there keeps its value
            fresh = ~torch.isin(p2, lin)
            lin, f = torch.cat([lin, p2[fresh]]), torch.cat([f, f2[fresh]])
        xyz = torch.stack([lin % size[0], (lin // size[0]) % size[1], lin // (size[0] * size[1])], dim=1)
        bsz = _bsz(size, edge)
        b = xyz // edge
        key = b[:, 0] + bsz[0] * (b[:, 1] + bsz[1] * b[:, 2])
        keys = torch.unique(key)
        bc = torch.stack([keys % bsz[0], (keys // bsz[0]) % bsz[1], keys // (bsz[0] * bsz[1])], dim=1)
        o = xyz % edge
        at = torch.searchsorted(keys, key) * edge ** 3 + o[:, 0] + edge * (o[:, 1] + edge * o[:, 2])
        ex = torch.zeros(len(keys) * edge ** 3, dtype=torch.bool, device=DEV)
        ex[at] = True
        val = torch.zeros(len(keys) * edge ** 3, dtype=torch.float64, device=DEV)
        val[at] = f
        P = _Points(size, edge, bc, ex.reshape(len(keys), -1))
        x = P.take(val, 0.0)
        inner = torch.ones(P.n, dtype=torch.bool, device=DEV)
        for d in STAR:
            inner &= P.at(*d) < P.n
        avg = torch.where(inner, _box27(P, x, [1.0 / 27.0] * 27, True), torch.zeros(P.n, dtype=torch.float64, device=DEV))
        return [None, P.chunks(x, 0.0), None, P.chunks(avg, 0.0), None]
    if op == "ghost":
        _, bc, ex = _scene(case)
        cen = _balls(case)[0]
        a, b = (_fields("gs", bc, ex, edge, cen, seed + k) for k in (0, 500))
        P = _Points(size, edge, bc, ex)
        m = torch.zeros(P.n, dtype=torch.bool, device=DEV)
        for lo, hi in _slabs(case):
            m |= ((P.xyz >= torch.tensor(lo, device=DEV)) & (P.xyz <= torch.tensor(hi, device=DEV))).all(dim=1)
        out = [P.chunks(torch.where(m, P.take(p, c)[: P.n], P.take(q, c)[: P.n]), c) for p, q, c in zip(a, b, BCK["gs"])]
        return [None] + out + [None]
    if op == "batch":
        out = []
        for k, (e, r) in enumerate(_batch_members(case)):
            _, bc, ex, f = _member(case, seed, k, e, r)
            P = _Points((e, e, e), edge, bc, ex)
            x = _march(P, case["kind"], f, case["steps"])
            out.append(P.chunks(x[0], BCK[case["kind"]][0]))
        return out
    return None  # an update moves and compares values, a re-tagging makes whole numbers only
