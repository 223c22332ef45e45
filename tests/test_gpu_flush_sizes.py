"""Flush at the sizes where its kernels change or their tiles end, against the CPU oracle; block maps, masks and values
are exact.  One launch takes up to 8192 points; above, the sort's tiles hold 1024 keys, 4096 past 4096 points per SM,
and the heads' and lookup's tiles 1024 points and chunks.  Ids above 32 bits have kernels of their own."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sgb():
    import openfpm_data_b200 as m
    m.load()
    return m


@pytest.mark.parametrize("edge", [8, 4])
@pytest.mark.parametrize("n", [1, 31, 1023, 1024, 1025, 2047, 2048, 2049, 4096, 4097, 8191, 8192, 8193, 9215, 9216, 9217, 12289, 70000])
@pytest.mark.parametrize("spread", [6, 120])
def test_flush_sizes(sgb, edge, n, spread):
    """n inserts with duplicates in a small or large part of the domain, then as many again (merge into the map).
    float32 maxima, float64 and uint8 last / first values, int32 bit sets: no sum whose order could matter."""
    rng = np.random.default_rng(n + spread + edge)
    size = (130, 121, 125)
    g = sgb.SparseGridGpu(size, ["f32", "f64", "i32", "u8"], edge=edge)
    o = O.OracleGrid(size, edge=edge, ptypes=[O.T_F32, O.T_F64, O.T_I32, O.T_U8])
    names = ["smax_", "sRight_", "sBitwiseOr_", "sLeft_"]
    ops = [O.OP_MAX, O.OP_RIGHT, O.OP_OR, O.OP_LEFT]
    for _ in range(2):
        pts = rng.integers(0, spread, size=(n, 3)).astype(np.int64)
        vals = [rng.standard_normal(n).astype(np.float32), rng.standard_normal(n),
                rng.integers(0, 2 ** 31 - 1, n).astype(np.int32), rng.integers(0, 255, n).astype(np.uint8)]
        g.insert(torch.from_numpy(pts.astype(np.int32)).cuda(), [torch.from_numpy(v).cuda() for v in vals])
        g.flush(names)
        o.insert_flush(pts, vals, ops)
    keys, data, mask = g.deviceToHost()
    okeys, odata, omask = o.export()
    assert np.array_equal(keys, okeys) and np.array_equal(mask, omask)
    ex = (mask & 1).astype(bool)
    for a, b in zip(data, odata):
        assert np.array_equal(a[ex], np.asarray(b)[ex])


def _one_property(sgb, size, edge, rounds, rng):
    g = sgb.SparseGridGpu(size, ["f32"], edge=edge)
    o = O.OracleGrid(size, edge=edge, ptypes=[O.T_F32])
    for pts in rounds:
        v = rng.standard_normal(len(pts)).astype(np.float32)
        g.insert(torch.from_numpy(pts.astype(np.int32)).cuda(), [torch.from_numpy(v).cuda()])
        g.flush(["sLeft_"])
        o.insert_flush(pts, [v], [O.OP_LEFT])
    keys, data, mask = g.deviceToHost()
    okeys, odata, omask = o.export()
    assert np.array_equal(keys, okeys) and np.array_equal(mask, omask)
    ex = (mask & 1).astype(bool)
    assert np.array_equal(data[0][ex], np.asarray(odata[0])[ex])


@pytest.mark.parametrize("n", [8191, 8192, 8193])
@pytest.mark.parametrize("spread", [20, 125])
def test_flush_at_the_limit_of_one_launch(sgb, n, spread):
    rng = np.random.default_rng(n + spread)
    _one_property(sgb, (130, 121, 125), 8, [rng.integers(0, [min(spread, s) for s in (130, 121, 125)], size=(n, 3)) for _ in range(3)], rng)


@pytest.mark.parametrize("more", [0, 1])
def test_flush_at_the_limit_of_small_sort_tiles(sgb, more):
    rng = np.random.default_rng(more)
    n = torch.cuda.get_device_properties(0).multi_processor_count * 4096 + more
    _one_property(sgb, (130, 121, 125), 8, [rng.integers(0, 121, size=(n, 3)), rng.integers(0, 121, size=(5000, 3))], rng)


@pytest.mark.parametrize("edge", [8, 4])
@pytest.mark.parametrize("n", [1, 3000, 8192, 8193, 700000])
def test_flush_with_ids_above_32_bits(sgb, edge, n):
    """A 2000^3 domain: points at both ends of it, so that ids below and above 2^32 are sorted together."""
    rng = np.random.default_rng(n + edge)
    size = np.array([2000, 1990, 2010])
    rounds = []
    for _ in range(2):
        p = rng.integers(0, 90, size=(n, 3))
        p[n // 2:] += size - 90
        rounds.append(p[rng.permutation(n)])
    _one_property(sgb, tuple(int(v) for v in size), edge, rounds, rng)


@pytest.mark.parametrize("n,distinct", [(5, 1), (8192, 1), (8192, 3), (8193, 1), (20001, 1), (33000, 6)])
def test_points_inserted_many_times(sgb, n, distinct):
    """Long runs of one point in the sorted list, in the one-launch flush and in the tiles of the other; the sums are
    taken in insertion order, so they are exact too."""
    rng = np.random.default_rng(n)
    size = (40, 40, 40)
    g = sgb.SparseGridGpu(size, ["f32", "f64", "i32", "u8"], edge=8)
    o = O.OracleGrid(size, edge=8, ptypes=[O.T_F32, O.T_F64, O.T_I32, O.T_U8])
    pool = np.array([[9, 9, 9], [1, 2, 3], [10, 9, 9], [39, 39, 39], [0, 0, 0], [16, 8, 8]], dtype=np.int64)[:distinct]
    for _ in range(2):
        pts = pool[rng.integers(0, distinct, n)]
        vals = [rng.standard_normal(n).astype(np.float32), rng.standard_normal(n),
                rng.integers(0, 2 ** 31 - 1, n).astype(np.int32), rng.integers(0, 255, n).astype(np.uint8)]
        g.insert(torch.from_numpy(pts.astype(np.int32)).cuda(), [torch.from_numpy(v).cuda() for v in vals])
        g.flush(["sadd_", "smin_", "sBitwiseOr_", "smax_"])
        o.insert_flush(pts, vals, [O.OP_ADD, O.OP_MIN, O.OP_OR, O.OP_MAX])
    keys, data, mask = g.deviceToHost()
    okeys, odata, omask = o.export()
    assert np.array_equal(keys, okeys) and np.array_equal(mask, omask)
    ex = (mask & 1).astype(bool)
    for a, b in zip(data, odata):
        assert np.array_equal(a[ex], np.asarray(b)[ex])


def test_flush_drops_out_of_domain(sgb):
    """The staged points are dropped and the map stays as it was when one of them lies outside."""
    g = sgb.SparseGridGpu((40, 40, 40), ["f32"], edge=8)
    p = torch.tensor([[1, 2, 3], [9, 9, 9]], dtype=torch.int32, device="cuda")
    g.insert(p, [torch.ones(2, device="cuda")])
    g.flush(["sRight_"])
    g.insert(torch.tensor([[20, 20, 20], [40, 0, 0]], dtype=torch.int32, device="cuda"), [torch.ones(2, device="cuda")])
    with pytest.raises(sgb.SgbError):
        g.flush(["sRight_"])
    g.flush(["sRight_"])
    assert g.countExistingElements() == 2 and g.nchunks == 2


def test_rejected_flush_keeps_what_was_made_from_the_map(sgb):
    """A mark in the existing-point list's memory is still there after a flush that was refused (the list stands),
    and gone after one that was taken (it is built again)."""
    import ctypes as C
    from openfpm_data_b200 import _lib as L
    from openfpm_data_b200.grid import _DevView
    g = sgb.SparseGridGpu((40, 40, 40), ["f32"], edge=8)
    g.insert(torch.tensor([[1, 2, 3], [9, 9, 9]], dtype=torch.int32, device="cuda"), [torch.ones(2, device="cuda")])
    g.flush(["sRight_"])

    def ids():
        p, n = C.c_void_p(), C.c_int64()
        L.check(g._lib.sgb_existing_point_list(g.handle, C.byref(p), C.byref(n), 0), "sgb_existing_point_list")
        torch.cuda.synchronize()
        return torch.as_tensor(_DevView(p.value, (n.value,), "<i4"), device="cuda")

    want = ids().clone()
    ids()[0] = -7
    g.insert(torch.tensor([[20, 20, 20], [40, 0, 0]], dtype=torch.int32, device="cuda"), [torch.ones(2, device="cuda")])
    with pytest.raises(sgb.SgbError):
        g.flush(["sRight_"])
    assert ids()[0].item() == -7
    g.insert(torch.tensor([[1, 2, 3]], dtype=torch.int32, device="cuda"), [torch.ones(1, device="cuda")])
    g.flush(["sRight_"])
    assert torch.equal(ids(), want)
