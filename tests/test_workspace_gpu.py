"""The library's own device buffers (one per device and stream): calls captured into a graph, streams and threads side by
side, buffers that grow, are evicted or released while graphs and other streams still use theirs."""
import pytest

from hipgpt_b200 import _capi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _st():
    return torch.cuda.current_stream().cuda_stream


def _rand(seed, *shape, scale=1.0):
    return torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda") * scale


@pytest.mark.parametrize("D", [16, 64])
def test_a_captured_backward_allocates_nothing_outside_its_graph(D):
    """A first call (larger than any other test's) inside a capture: at head_dim 16 the row sums need a buffer, at 64 they do not."""
    lib = _capi.lib()
    B, H, S = 32, 16, 300
    E = H * D
    qkv, g = _rand(1, 3, B * S, E), _rand(2, B * S, E)
    want, got = torch.empty_like(qkv), torch.full_like(qkv, float("nan"))
    nbytes = int(lib.hipgpt_mha_backward_scratch_bytes(B, H, S))
    scratch = torch.empty(nbytes // 4, device="cuda")
    _capi.check(lib.hipgpt_mha_backward(g.data_ptr(), qkv[0].data_ptr(), qkv[1].data_ptr(), qkv[2].data_ptr(), None, want[0].data_ptr(),
                                        want[1].data_ptr(), want[2].data_ptr(), scratch.data_ptr(), nbytes, B, S, E, H, 1, _st()))
    torch.cuda.synchronize()
    lib.hipgpt_release_workspace()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _capi.check(lib.hipgpt_mha_backward_planes(g.data_ptr(), qkv.data_ptr(), None, got.data_ptr(), B, S, E, H, 1, _st()))
    for _ in range(2):
        got.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)


def test_released_buffers_of_the_backward_are_given_back():
    lib = _capi.lib()
    B, H, S, D = 32, 64, 1024, 8                            # row sums: 16 MB
    E = H * D
    qkv, g, out = _rand(3, 3, B * S, E), _rand(4, B * S, E), torch.empty(3, B * S, E, device="cuda")
    free = []
    for _ in range(2):                                      # the first call also loads the kernels
        _capi.check(lib.hipgpt_mha_backward_planes(g.data_ptr(), qkv.data_ptr(), None, out.data_ptr(), B, S, E, H, 0, _st()))
        torch.cuda.synchronize()
        held = torch.cuda.mem_get_info()[0]
        lib.hipgpt_release_workspace()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[1] == free[0] and free[0] - held >= 16 << 20


def test_backwards_of_two_streams_have_their_own_row_sums():
    lib = _capi.lib()
    B, H, S, D = 8, 8, 256, 16
    E = H * D
    streams = [torch.cuda.Stream() for _ in range(2)]
    qkv, g = [_rand(5 + i, 3, B * S, E) for i in range(2)], [_rand(7 + i, B * S, E) for i in range(2)]
    want = []
    for i in range(2):
        out = torch.empty(3, B * S, E, device="cuda")
        _capi.check(lib.hipgpt_mha_backward_planes(g[i].data_ptr(), qkv[i].data_ptr(), None, out.data_ptr(), B, S, E, H, 0, _st()))
        torch.cuda.synchronize()
        want.append(out)
    got = [[torch.full_like(qkv[0], float("nan")) for _ in range(8)] for _ in range(2)]
    torch.cuda.synchronize()
    for r in range(8):
        for i, st in enumerate(streams):
            _capi.check(lib.hipgpt_mha_backward_planes(g[i].data_ptr(), qkv[i].data_ptr(), None, got[i][r].data_ptr(), B, S, E, H, 0, st.cuda_stream))
    torch.cuda.synchronize()
    for i in range(2):
        for r in range(8):
            assert torch.equal(got[i][r], want[i])
