"""The 7-point kernels against the one-chunk-per-CTA kernel, bit for bit: both evaluate the same
float32 operations in the same order, so no tolerance is needed."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sgb():
    import openfpm_data_b200 as m
    m.load()
    return m


def _grid(sgb, size, nchunks, lin, seed, density=0.5, e=8):
    """A grid of about nchunks random chunks, a part of whose points exist, some of them padding."""
    rng = np.random.default_rng(seed)
    b = [-(-s // e) for s in size]
    pick = rng.permutation(b[0] * b[1] * b[2])[:nchunks]
    bc = np.stack([pick % b[0], pick // b[0] % b[1], pick // (b[0] * b[1])], axis=1)
    if lin == "zmb":
        spread = lambda v: sum(((v >> i) & 1) << (3 * i) for i in range(8))  # noqa: E731
        key = spread(bc[:, 0]) | spread(bc[:, 1]) << 1 | spread(bc[:, 2]) << 2
    else:
        key = pick
    order = np.argsort(key)
    key, bc = key[order].astype(np.int64), bc[order]
    p = np.arange(e ** 3)
    xyz = bc[:, None, :] * e + np.stack([p % e, p // e % e, p // e ** 2], axis=1)[None]
    rows = rng.random((len(key), e * e, 1)) < 0.8  # whole x rows are missing too
    ex = (rng.random((len(key), e * e, e)) < density) & rows
    ex = ex.reshape(len(key), e ** 3) & (xyz < np.array(size)).all(axis=2)
    pad = ex & (rng.random(ex.shape) < 0.1)
    mask = (ex | pad << 1).astype(np.uint8).reshape(-1)
    g = sgb.SparseGridGpu(size, ["f32"] * 4, edge=e, linearizer=lin)
    for q, v in enumerate([0.25, -1.5, 3.0, 0.5]):
        g.setBackgroundValue(q, v)
    g.load_map(key, [rng.standard_normal(len(mask)).astype(np.float32) for _ in range(4)], mask)
    return g


@pytest.mark.parametrize("e,stages", [(8, 3), (8, 4), (4, -1)])
@pytest.mark.parametrize("lin,size,nchunks", [
    ("smb", (8, 8, 8), 1), ("smb", (70, 20, 9), 7), ("smb", (130, 33, 30), 60), ("smb", (157, 61, 90), 1500),
    ("zmb", (64, 64, 64), 300), ("zmb", (75, 50, 41), 200)])
@pytest.mark.parametrize("kind", ["HEAT7", "GS7"])
def test_star7_equals_tiled(sgb, kind, lin, size, nchunks, e, stages):
    prm = [0.1] if kind == "HEAT7" else [0.16, 0.08, 0.035, 0.065, 1.0]
    src, dst = ([0], [2]) if kind == "HEAT7" else ([0, 1], [2, 3])
    for box in (None, ((3, 2, 1), (size[0] - 4, size[1] - 3, size[2] - 2))):
        out = []
        for tiled in (True, False):
            g = _grid(sgb, size, nchunks, lin, 7, e=e)
            g.setLaunchConfig(-1, stages)
            m = g.private_get_mask_array()  # also: no property counts as background-clean any more
            g.applyStencils(getattr(sgb, kind), src, dst, prm, box=box, tiled=tiled)
            g.check_device_errors()
            keep = torch.from_numpy(np.ones(m.numel(), bool)).cuda() if kind == "HEAT7" else (m & 1).bool()
            out.append([g.private_get_data_array(d)[keep].cpu() for d in dst])
        for a, b in zip(*out):
            assert torch.equal(a.view(torch.int32), b.view(torch.int32))


def test_star7_eight_slices_by_size(sgb):
    """Past two waves of blocks the automatic choice changes; the steps stay the same."""
    g = _grid(sgb, (240, 240, 240), 20000, "smb", 3)
    got = []
    for stages in (3, -1):
        g.setLaunchConfig(-1, stages)
        g.applyStencils(sgb.HEAT7, [0], [2], [0.1])
        got.append(g.private_get_data_array(2).clone())
    assert torch.equal(*got)
    g.check_device_errors()


@pytest.mark.parametrize("nchunks", [1, 2, 5, 17, 33, 144, 145, 160, 161, 256, 257])
@pytest.mark.parametrize("kind", ["HEAT7", "GS7"])
def test_solve_in_one_launch_equals_steps(sgb, kind, nchunks):
    """run_steps of a small grid (both sides of the size limit) against single steps of the tile kernel."""
    prm = [0.1] if kind == "HEAT7" else [0.16, 0.08, 0.035, 0.065, 1.0]
    a, b = ([0], [2]) if kind == "HEAT7" else ([0, 1], [2, 3])
    size = (75, 80, 70) if nchunks < 100 else (100, 99, 75)
    for nsteps in (2, 9):
        g, h = (_grid(sgb, size, nchunks, "smb", 11, density=0.9) for _ in range(2))
        fin = g.run_steps(getattr(sgb, kind), a, b, prm, nsteps)
        for k in range(nsteps):
            h.applyStencils(getattr(sgb, kind), a if k % 2 == 0 else b, b if k % 2 == 0 else a, prm, tiled=True)
        assert fin == (nsteps % 2 == 1)
        g.check_device_errors()
        ex = (g.private_get_mask_array() & 1).bool()
        for q in a + b:  # the last state and the one before it
            x, w = g.private_get_data_array(q)[ex], h.private_get_data_array(q)[ex]
            assert torch.equal(x.view(torch.int32), w.view(torch.int32))


@pytest.mark.parametrize("per_sm,more", [(0, 1), (0, 8), (0, 9), (1, 0), (1, 1), (3, 0), (3, 1)])
@pytest.mark.parametrize("kind,lin", [("HEAT7", "smb"), ("GS7", "smb"), ("GS7", "zmb")])
def test_solve_of_4_chunks_equals_steps(sgb, kind, lin, per_sm, more):
    """run_steps on 4^3 chunks, both sides of the limits in chunks and steps, against steps of the tile kernel."""
    prm = [0.1] if kind == "HEAT7" else [0.16, 0.08, 0.035, 0.065, 1.0]
    a, b = ([0], [2]) if kind == "HEAT7" else ([0, 1], [2, 3])
    nchunks = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    for nsteps in (2, 3, 4, 8, 9):
        g, h = (_grid(sgb, (40, 33, 38), nchunks, lin, 13, density=0.9, e=4) for _ in range(2))
        fin = g.run_steps(getattr(sgb, kind), a, b, prm, nsteps)
        for k in range(nsteps):
            h.applyStencils(getattr(sgb, kind), a if k % 2 == 0 else b, b if k % 2 == 0 else a, prm, tiled=True)
        assert fin == (nsteps % 2 == 1)
        g.check_device_errors()
        ex = (g.private_get_mask_array() & 1).bool()
        for q in a + b:
            x, w = g.private_get_data_array(q)[ex], h.private_get_data_array(q)[ex]
            assert torch.equal(x.view(torch.int32), w.view(torch.int32))


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("kind", ["HEAT7", "GS7"])
def test_batch_stepped_past_its_slots(sgb, kind, use_graph):
    """4^3 chunks: most launches of the call find no slot with a step left; what is read behind them is the last
    live step's result, of a step long enough for the idle launches to overtake it."""
    prm = [0.1] if kind == "HEAT7" else [0.16, 0.08, 0.035, 0.065, 1.0]
    a, b = ([0], [2]) if kind == "HEAT7" else ([0, 1], [2, 3])
    batch = sgb.Batch()
    slots, want = [], []
    for nchunks, nsteps in ((40000, 4), (500, 3)):
        size = (240, 240, 240) if nchunks > 1000 else (64, 60, 52)
        g, h = (_grid(sgb, size, nchunks, "smb", 5, density=0.9, e=4) for _ in range(2))
        slots.append((batch.add(g, getattr(sgb, kind), a, b, prm, nsteps), g))
        for k in range(nsteps):
            h.applyStencils(getattr(sgb, kind), a if k % 2 == 0 else b, b if k % 2 == 0 else a, prm, tiled=True)
        want.append(h)
    for _ in range(2):  # the second call has idle launches only
        batch.step(24, use_graph=use_graph)
        for (slot, g), h in zip(slots, want):
            batch.extract(slot, g)
            ex = (h.private_get_mask_array() & 1).bool()
            for q in a + b:
                x, w = g.private_get_data_array(q)[ex], h.private_get_data_array(q)[ex]
                assert torch.equal(x.view(torch.int32), w.view(torch.int32))
    batch.close()


@pytest.mark.parametrize("what", ["solve", "step"])
def test_threads_with_different_shared_memory(sgb, what):
    """Host threads, each with its own grid and stream, launch one kernel with different amounts of shared memory:
    none may lower another's limit between its setting and its launch."""
    import threading
    # chunks, CTAs per SM, steps a call: small grids run in one cluster launch, larger ones by a launch per step
    plans = [(256, -1, 2), (20, -1, 2), (120, -1, 2), (3, -1, 2)] if what == "solve" else [(400, 1, 50), (400, 3, 50)]
    calls = 2000 if what == "solve" else 100
    want, got, bad = {}, {}, []
    together = threading.Barrier(len(plans), timeout=120)

    def grid(n):
        return _grid(sgb, (75, 80, 70), n, "smb", n, density=0.9)

    for n, _, steps in plans:
        g = grid(n)
        for k in range(steps):
            g.applyStencils(sgb.HEAT7, [2 * (k % 2)], [2 - 2 * (k % 2)], [0.1], tiled=True)
        want[n] = g.deviceToHost()[1][0]

    def work(k):
        try:
            n, ctas, steps = plans[k]
            stream = torch.cuda.Stream()
            g = grid(n)
            g.setLaunchConfig(ctas, -1)
            first = g.deviceToHost()[1][0]
            together.wait()
            for _ in range(calls):
                g.run_steps(sgb.HEAT7, [0], [2], [0.1], steps, use_graph=False, stream=stream)
            stream.synchronize()
            g.private_get_data_array(0).copy_(torch.from_numpy(first))
            torch.cuda.synchronize()
            g.run_steps(sgb.HEAT7, [0], [2], [0.1], steps, use_graph=False, stream=stream)
            got[k] = g.deviceToHost(stream)[1][0]
        except Exception as e:  # noqa: BLE001
            bad.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(plans))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
    for k, (n, _, _) in enumerate(plans):
        assert np.array_equal(want[n].view(np.uint32), got[k].view(np.uint32))
