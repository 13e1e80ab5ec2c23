"""The library's own device buffers (one per device and stream): calls captured into a graph, streams and threads side by
side, buffers that grow, are evicted or released while graphs and other streams still use theirs."""
import threading

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


class _Backward:
    """dQ, dK, dV with the probabilities formed again; head_dim 64: the tensor pipe's images, 16: row sums."""

    def __init__(self, seed, size, D):
        self.shape = B, H, S, D = size, 4, 192, D
        self.inputs = _rand(seed, B * S, H * D), _rand(seed + 1, 3, B * S, H * D)

    def empty(self):
        return torch.full_like(self.inputs[1], float("nan"))

    def run(self, out, stream):
        g, qkv = self.inputs
        B, H, S, D = self.shape
        _capi.check(_capi.lib().hipgpt_mha_backward_planes(g.data_ptr(), qkv.data_ptr(), None, out.data_ptr(), B, S, H * D, H, 1, stream))


class _Matmul:
    def __init__(self, seed, size):
        self.shape = M, N, K = 300 * size, 320, 256
        self.inputs = _rand(seed, M, N), _rand(seed + 1, N, K)

    def empty(self):
        return torch.full((self.shape[0], self.shape[2]), float("nan"), device="cuda")

    def run(self, out, stream):
        a, w = self.inputs
        _capi.check(_capi.lib().hipgpt_matmul_tc(a.data_ptr(), w.data_ptr(), None, out.data_ptr(), *self.shape, stream))


class _Attention:
    """The tiled kernel's packed K and V; `groups`: cut into groups of batches, packed on a second stream (unmasked)."""

    def __init__(self, seed, size, groups):
        self.shape, self.groups = (size, 16, 128, 64), groups       # 0.5 MB of images per batch
        B, H, S, D = self.shape
        self.inputs = _rand(seed, 3, B * S, H * D)

    def empty(self):
        B, H, S, D = self.shape
        return torch.full((B * S, H * D), float("nan"), device="cuda")

    def run(self, out, stream):
        B, H, S, D = self.shape
        _capi.check(_capi.lib().hipgpt_mha_forward_planes(self.inputs.data_ptr(), out.data_ptr(), None, B, S, H * D, H, int(not self.groups), stream))


KINDS = {"attention": lambda seed, size: _Attention(seed, size, False), "attention_groups": lambda seed, size: _Attention(seed, size, True),
         "backward": lambda seed, size: _Backward(seed, size, 64), "backward_rows": lambda seed, size: _Backward(seed, size, 16), "matmul": _Matmul}


@pytest.fixture(autouse=True)
def _groups(request, monkeypatch):
    if "attention_groups" in request.node.name:
        monkeypatch.setenv("HIPGPT_PACK_GROUP_MB", "1")             # two batches


def _expected(job):
    out = job.empty()
    job.run(out, _st())
    torch.cuda.synchronize()
    assert bool(torch.isfinite(out).all())
    return out


@pytest.mark.parametrize("kind", KINDS)
def test_a_graph_keeps_its_buffer_when_later_calls_grow_or_release_theirs(kind):
    lib = _capi.lib()
    small, big = KINDS[kind](10, 2), KINDS[kind](20, 24)
    want, want_big = _expected(small), _expected(big)
    stream = torch.cuda.Stream()
    lib.hipgpt_release_workspace()
    before, out, out_big = small.empty(), small.empty(), big.empty()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    small.run(before, stream.cuda_stream)                   # the stream's buffer, in the size of the captured call
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        small.run(out, torch.cuda.current_stream().cuda_stream)
    big.run(out_big, stream.cuda_stream)                    # grows it
    torch.cuda.synchronize()
    assert torch.equal(before, want) and torch.equal(out_big, want_big)
    for _ in range(2):
        lib.hipgpt_release_workspace()
        out.fill_(float("nan"))
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)


@pytest.mark.parametrize("kind", KINDS)
def test_threads_that_share_a_stream_and_grow_its_buffer(kind):
    jobs = [KINDS[kind](100 + 10 * i, size) for i, size in enumerate((1, 3, 7, 20))]
    want = [_expected(j) for j in jobs]
    _capi.lib().hipgpt_release_workspace()
    stream = torch.cuda.Stream()
    outs = [[j.empty() for _ in range(6)] for j in jobs]
    torch.cuda.synchronize()
    failed = []

    def work(i):
        try:
            for out in outs[i]:
                jobs[i].run(out, stream.cuda_stream)
        except Exception as e:                              # noqa: BLE001
            failed.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed
    for i, w in enumerate(want):
        assert all(torch.equal(out, w) for out in outs[i])


@pytest.mark.parametrize("kind", KINDS)
def test_more_streams_than_buffers(kind):
    """Twelve streams in turn, eight buffers: the ninth stream takes the buffer that was used longest ago."""
    jobs = [KINDS[kind](200 + 10 * i, 6 + 2 * (i % 3)) for i in range(3)]
    want = [_expected(j) for j in jobs]
    _capi.lib().hipgpt_release_workspace()
    streams = [torch.cuda.Stream() for _ in range(12)]
    outs = [[jobs[(i + r) % 3].empty() for i in range(12)] for r in range(3)]
    torch.cuda.synchronize()
    for r in range(3):
        for i, s in enumerate(streams):
            jobs[(i + r) % 3].run(outs[r][i], s.cuda_stream)
    torch.cuda.synchronize()
    for r in range(3):
        for i in range(12):
            assert torch.equal(outs[r][i], want[(i + r) % 3])


@pytest.mark.parametrize("kind", KINDS)
def test_a_buffer_grows_on_one_stream_while_another_is_captured(kind):
    """Capture in its strictest mode forbids cudaMalloc to every thread; a growing call on a stream outside the capture has to do
    it all the same, and must not end the capture."""
    job = KINDS[kind](300, 3)
    want = _expected(job)
    _capi.lib().hipgpt_release_workspace()
    other, x, out = torch.cuda.Stream(), torch.zeros(1000, device="cuda"), job.empty()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="global"):
        x += 1.0
        job.run(out, other.cuda_stream)
        x += 1.0
    graph.replay()
    torch.cuda.synchronize()
    assert bool((x == 2.0).all()) and torch.equal(out, want)
