"""Values that a caller writes to points that do not exist, through a view it took before, reach no result.

The reference is a second grid that runs the tile kernel, which tests the mask of every value it reads; results are
equal bit for bit.  On 8^3 chunks with x-fastest ids the written property is a step's destination; on 4^3 chunks, on
Morton ids, and in solves of grids of at most 4 chunks per SM it may be its source as well."""
import numpy as np
import pytest
import torch

from tests.test_gpu_star7 import _grid

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sgb():
    import openfpm_data_b200 as m
    m.load()
    return m


PRM = {"HEAT7": [0.1], "GS7": [0.16, 0.08, 0.035, 0.065, 1.0]}
GRIDS = [(8, "smb", (75, 50, 61), 100), (8, "smb", (75, 50, 61), 200), (8, "smb", (100, 99, 75), 900), (8, "zmb", (64, 64, 64), 300),
         (4, "smb", (64, 60, 52), 700), (4, "zmb", (64, 64, 64), 30)]


def _pair(sgb, kind, e, lin, size, n):
    """The grid under test with the views a program keeps, and its twin."""
    g, h = (_grid(sgb, size, n, lin, 3, e=e) for _ in range(2))
    if kind == "GS7" and (e, lin) == (8, "smb"):  # there Gray-Scott leaves the x quads of padding points alone
        for x in (g, h):
            x.private_get_mask_array().bitwise_and_(1)
    views = [g.private_get_data_array(p) for p in range(4)]
    mask = g.private_get_mask_array()
    return g, h, views, mask


def _fields(kind):
    return ([0], [2]) if kind == "HEAT7" else ([0, 1], [2, 3])


def _same(g, h, props):
    ex = (h.private_get_mask_array() & 1).bool()
    for p in props:
        x, w = g.private_get_data_array(p)[ex], h.private_get_data_array(p)[ex]
        assert torch.equal(x.view(torch.int32), w.view(torch.int32)), f"property {p}"


def _twin_steps(sgb, h, kind, a, b, steps):
    for k in range(steps):
        h.applyStencils(getattr(sgb, kind), a if k % 2 == 0 else b, b if k % 2 == 0 else a, PRM[kind], tiled=True)


@pytest.mark.parametrize("kind", ["HEAT7", "GS7"])
@pytest.mark.parametrize("e,lin,size,n", GRIDS)
def test_single_steps(sgb, kind, e, lin, size, n):
    g, h, views, mask = _pair(sgb, kind, e, lin, size, n)
    a, b = _fields(kind)
    gone = (mask == 0)
    gone[g.nchunks * g.bs:] = False  # the background chunk is not a caller's to write
    g.applyStencils(getattr(sgb, kind), a, b, PRM[kind])
    _twin_steps(sgb, h, kind, a, b, 1)
    for p in b if (e, lin) == (8, "smb") else a + b:
        views[p].masked_fill_(gone, float("nan"))
    g.applyStencils(getattr(sgb, kind), a, b, PRM[kind])
    g.applyStencils(getattr(sgb, kind), b, a, PRM[kind])
    _twin_steps(sgb, h, kind, a, b, 2)
    _same(g, h, a + b)


@pytest.mark.parametrize("nsteps", [2, 3])
@pytest.mark.parametrize("kind", ["HEAT7", "GS7"])
@pytest.mark.parametrize("e,lin,size,n", GRIDS)
def test_run_steps(sgb, kind, e, lin, size, n, nsteps):
    g, h, views, mask = _pair(sgb, kind, e, lin, size, n)
    a, b = _fields(kind)
    gone = (mask == 0)
    gone[g.nchunks * g.bs:] = False
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert (n <= 4 * sms) == (n != 900 and n != 700)
    g.run_steps(getattr(sgb, kind), a, b, PRM[kind], 2)
    _twin_steps(sgb, h, kind, a, b, 2)
    for p in b if n == 900 else a + b:
        views[p].masked_fill_(gone, float("nan"))
    g.run_steps(getattr(sgb, kind), a, b, PRM[kind], nsteps)
    _twin_steps(sgb, h, kind, a, b, nsteps)
    _same(g, h, a + b)


@pytest.mark.parametrize("kind", ["HEAT7", "GS7"])
@pytest.mark.parametrize("e", [8, 4])
def test_batch_member(sgb, kind, e):
    g, h, views, mask = _pair(sgb, kind, e, "smb", (75, 50, 61), 200)
    a, b = _fields(kind)
    gone = (mask == 0)
    gone[g.nchunks * g.bs:] = False
    g.run_steps(getattr(sgb, kind), a, b, PRM[kind], 2)
    _twin_steps(sgb, h, kind, a, b, 2)
    for p in a + b:
        views[p].masked_fill_(gone, float("nan"))
    batch = sgb.Batch()
    slot = batch.add(g, getattr(sgb, kind), a, b, PRM[kind], 3)
    batch.step(3)
    batch.extract(slot, g)
    _twin_steps(sgb, h, kind, a, b, 3)
    _same(g, h, a + b)
    batch.close()


@pytest.mark.parametrize("kind", ["HEAT7", "GS7"])
@pytest.mark.parametrize("e,lin,size,n", [g for g in GRIDS if g[:2] != (8, "smb")])
def test_points_taken_out_through_a_kept_mask(sgb, kind, e, lin, size, n):
    g, h, views, mask = _pair(sgb, kind, e, lin, size, n)
    a, b = _fields(kind)
    g.applyStencils(getattr(sgb, kind), a, b, PRM[kind])
    _twin_steps(sgb, h, kind, a, b, 1)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    out = torch.rand(mask.shape, generator=gen, device="cuda") < 0.05
    for m in (mask, h.private_get_mask_array()):
        m.masked_fill_(out, 0)
    g.applyStencils(getattr(sgb, kind), b, a, PRM[kind])
    g.applyStencils(getattr(sgb, kind), a, b, PRM[kind])
    h.applyStencils(getattr(sgb, kind), b, a, PRM[kind], tiled=True)
    h.applyStencils(getattr(sgb, kind), a, b, PRM[kind], tiled=True)
    _same(g, h, a + b)


@pytest.mark.parametrize("kind", ["HEAT7", "GS7"])
@pytest.mark.parametrize("e,lin,size,n", GRIDS)
@pytest.mark.parametrize("how", ["steps", "run_steps"])
def test_captured_before_the_view_was_taken(sgb, how, kind, e, lin, size, n):
    """Two steps in a graph, captured while nobody has had a view of the grid, replayed after writes through one."""
    g, h = (_grid(sgb, size, n, lin, 3, e=e) for _ in range(2))
    a, b = _fields(kind)
    if kind == "GS7" and (e, lin) == (8, "smb"):  # the same, for a map whose views nobody has had
        keys, data, mask = h.deviceToHost()
        for x in (g, h):
            x.load_map(keys, [d[: n * x.bs] for d in data], mask[: n * x.bs] & 1)
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    g.findNeighbours(sgb.NN_STAR)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side):
        if how == "steps":
            g.applyStencils(getattr(sgb, kind), a, b, PRM[kind])
            g.applyStencils(getattr(sgb, kind), b, a, PRM[kind])
        else:
            g.run_steps(getattr(sgb, kind), a, b, PRM[kind], 2, use_graph=False)
    graph.replay()
    torch.cuda.synchronize()
    views = [g.private_get_data_array(p) for p in range(4)]
    gone = g.private_get_mask_array() == 0
    gone[g.nchunks * g.bs:] = False
    for p in b:
        views[p].masked_fill_(gone, float("nan"))
    graph.replay()
    torch.cuda.synchronize()
    _twin_steps(sgb, h, kind, a, b, 2)
    _twin_steps(sgb, h, kind, a, b, 2)
    _same(g, h, a + b)


@pytest.mark.parametrize("kind,e,lin,size,n", [("HEAT7", *g) for g in GRIDS] +
                         [("GS7", *g) for g in GRIDS if g[:2] != (8, "smb")])
def test_boxed_steps(sgb, kind, e, lin, size, n):
    g, h, views, mask = _pair(sgb, kind, e, lin, size, n)
    a, b = _fields(kind)
    box = ((3, 2, 5), (size[0] - 6, size[1] - 3, size[2] - 2))
    gone = (mask == 0)
    gone[g.nchunks * g.bs:] = False
    for k in range(4):
        x, y = (a, b) if k % 2 == 0 else (b, a)
        g.applyStencils(getattr(sgb, kind), x, y, PRM[kind], box=box)
        h.applyStencils(getattr(sgb, kind), x, y, PRM[kind], box=box, tiled=True)
        for p in a if k % 2 == 0 else b:  # the source of this step, the destination of the next one
            views[p].masked_fill_(gone, float("nan"))
    _same(g, h, a + b)


@pytest.mark.parametrize("kind", ["HEAT7", "GS7"])
@pytest.mark.parametrize("e,lin,size,n", GRIDS)
def test_writes_before_the_map_grows(sgb, kind, e, lin, size, n):
    """A flush with new chunks moves the map to other buffers, what the caller wrote included, and ends its views."""
    g, h, views, mask = _pair(sgb, kind, e, lin, size, n)
    a, b = _fields(kind)
    gone = (mask == 0)
    gone[g.nchunks * g.bs:] = False
    g.applyStencils(getattr(sgb, kind), a, b, PRM[kind])
    _twin_steps(sgb, h, kind, a, b, 1)
    for p in a + b:
        views[p].masked_fill_(gone, float("nan"))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    pts = torch.stack([torch.randint(0, s, (4000,), generator=gen, device="cuda") for s in size], 1).to(torch.int32)
    vals = [torch.rand(4000, generator=gen, device="cuda") for _ in range(4)]
    before = g.nchunks
    for x in (g, h):
        x.insert(pts, vals)
        x.flush(["sRight_"] * 4)
    assert g.nchunks > before
    for k in range(2):
        x, y = (a, b) if k == 0 else (b, a)
        g.applyStencils(getattr(sgb, kind), x, y, PRM[kind])
        h.applyStencils(getattr(sgb, kind), x, y, PRM[kind], tiled=True)
    _same(g, h, a + b)
