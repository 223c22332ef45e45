"""The existing-point list asked for on a stream that is not torch's current one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sgb():
    import openfpm_data_b200 as m
    m.load()
    return m


@pytest.mark.parametrize("other", ["side", "default"])
def test_point_list_on_another_stream(sgb, other):
    """The list is long enough for its last kernel to run well past the call that queues it; every round has
    another set of points, and the same buffers."""
    nb = 36
    n = nb ** 3 * 512
    g = sgb.SparseGridGpu((nb * 8,) * 3, ["u8"], edge=8)
    one = torch.ones(n, dtype=torch.uint8, device="cuda")
    g.load_map_dev(torch.arange(nb ** 3, device="cuda"), [one], one)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    side = torch.cuda.Stream()
    lists, want = [], []
    for k in range(3):
        m = (torch.rand(n, generator=gen, device="cuda") < 0.3 + 0.2 * k).to(torch.uint8)
        g.private_get_mask_array()[:n].copy_(m)
        torch.cuda.synchronize()
        if other == "side":
            got = g.existing_point_list(stream=side)
        else:
            with torch.cuda.stream(side):
                got = g.existing_point_list(stream=torch.cuda.default_stream())
        with torch.cuda.stream(torch.cuda.current_stream() if other == "side" else side):
            lists.append(got.clone())  # at once, on the stream that the call was made from
        del got
        want.append(m)
    torch.cuda.synchronize()
    for a, m in zip(lists, want):
        assert torch.equal(a, m.nonzero().squeeze(1))


@pytest.mark.parametrize("n", [1, 511, 512, 513, 16384, 16385, 49151, 49152, 49153])
def test_point_offsets_at_the_limits_of_the_prefix_sums(sgb, n):
    """First existing point of every chunk, and the list made from it, for chunk counts at which the prefix sum
    changes its kernel or takes another round."""
    g = sgb.SparseGridGpu((8 * n, 8, 8), ["u8"], edge=8)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    m = (torch.rand(n * 512, generator=gen, device="cuda") < 0.02).to(torch.uint8)
    g.load_map_dev(torch.arange(n, device="cuda"), [m], m)
    per = m.reshape(n, 512).sum(dim=1)
    want = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), per.cumsum(0)])
    assert torch.equal(g.existing_offsets(), want)
    assert torch.equal(g.existing_point_list(), m.nonzero().squeeze(1))
