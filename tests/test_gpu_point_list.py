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
