"""GPU tests of the order of launches on one stream: kernels of this library that are launched programmatically (they may
start while the kernel in front still runs) behind kernels whose outputs they read."""
import pytest
import torch

from nanoserve_b200.ops import FLAG_DECODE_NARROW, FLAG_GEMM_NARROW, FLAG_NO_PDL, narrow_flags

pytestmark = pytest.mark.gpu


def rand_w4(N, K, G, gen):
    Wq = torch.randint(-2**31, 2**31 - 1, (N, K // 8), dtype=torch.int32, device="cuda", generator=gen)
    S = (0.005 + (torch.randn(N, K // G, device="cuda", generator=gen) * 0.01).abs()).to(torch.bfloat16)
    return Wq, S


def rand_x(M, K, gen):
    return torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)


@pytest.mark.parametrize("M,G,flags", [(3, 128, FLAG_DECODE_NARROW), (8, 128, FLAG_DECODE_NARROW), (13, 128, FLAG_DECODE_NARROW),
                                       (4, 64, FLAG_DECODE_NARROW), (48, 128, FLAG_GEMM_NARROW), (48, 32, FLAG_GEMM_NARROW), (300, 128, 0)])
def test_weights_written_by_the_kernel_in_front(kernels, M, G, flags):
    """The kernel in front lets its dependents start at once and stores at its end: a linear whose output is the next one's
    scales, or its packed words.  The result is that of the same launches with a synchronisation in between."""
    gen = torch.Generator(device="cuda").manual_seed(M)
    N, K = 1024, 1024
    x, (Wq, S) = rand_x(M, K, gen), rand_w4(N, K, G, gen)
    front_x, (front_q, front_s) = rand_x(64, 18944, gen), rand_w4(N * (K // G) // 64, 18944, 128, gen)
    words_x, (words_q, words_s) = rand_x(64, 8192, gen), rand_w4(N * K // 4 // 64, 8192, 128, gen)
    scales, words = torch.empty_like(S), torch.empty_like(Wq)

    def chain(sync):
        sync()
        kernels.w4_linear(front_x, front_q, front_s, 128, flags=narrow_flags(split=1), out=scales.view(64, -1))
        sync()
        a = kernels.w4_linear(x, Wq, scales, G, flags=flags)
        sync()
        kernels.w4_linear(words_x, words_q, words_s, 128, flags=narrow_flags(split=1),
                          out=words.view(torch.bfloat16).view(64, -1))
        sync()
        b = kernels.w4_linear(x, words, S, G, flags=flags)
        sync()
        return a, b

    want = chain(torch.cuda.synchronize)
    assert all(bool(w.isfinite().all()) and float(w.float().abs().max()) > 0 for w in want)
    for _ in range(20):
        scales.zero_()
        words.zero_()
        got = chain(lambda: None)
        assert all(torch.equal(g, w) for g, w in zip(got, want))
    assert kernels.device_status() == 0


@pytest.mark.parametrize("M", [3, 8, 13, 48])
def test_linear_behind_its_quantizer(kernels, M):
    gen = torch.Generator(device="cuda").manual_seed(M)
    W, x = rand_x(5000, 3584, gen), rand_x(M, 3584, gen)
    Wq, S = kernels.w4_quantize(W)
    torch.cuda.synchronize()
    want = kernels.w4_linear(x, Wq, S)
    for _ in range(10):
        Wq.zero_()
        S.zero_()
        torch.cuda.synchronize()
        rc = kernels.lib.ns_w4_quantize(W.data_ptr(), Wq.data_ptr(), S.data_ptr(), 5000, 3584, 128, kernels._stream())
        assert rc == 0 and torch.equal(kernels.w4_linear(x, Wq, S), want)
    assert kernels.device_status() == 0


@pytest.fixture(scope="module")
def long_launch(kernels):
    """A launch that lets its dependents start at once and then runs longer than any bounded wait of the library (10^9
    cycles, 0.51 s at 1.965 GHz): one CTA walks a long K, doubled until that is so however fast a step has become (2^28 are
    2^21 steps of some 560 cycles)."""
    for K in (2**28, 2**29, 2**30):
        go, ms = _walk(kernels, K, 64)
        if ms > 600:
            return go
    pytest.fail(f"a K of 2^30 takes {ms} ms: no launch here is longer than a bounded wait")


def _walk(kernels, K, G):
    x = torch.zeros(1, K, dtype=torch.bfloat16, device="cuda")
    Wq = torch.zeros(1, K // 8, dtype=torch.int32, device="cuda")
    S = torch.ones(1, K // G, dtype=torch.bfloat16, device="cuda")
    go = lambda: kernels.w4_linear(x, Wq, S, G, flags=FLAG_DECODE_NARROW | narrow_flags(split=1, tile=1))
    go()
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    start.record()
    y = go()
    end.record()
    end.synchronize()
    assert kernels.device_status() == 0 and float(y) == 0
    return go, start.elapsed_time(end)


@pytest.mark.parametrize("M,G,flags", [(3, 128, FLAG_DECODE_NARROW), (8, 128, FLAG_DECODE_NARROW), (13, 128, FLAG_DECODE_NARROW),
                                       (4, 64, FLAG_DECODE_NARROW), (48, 128, FLAG_GEMM_NARROW)])
def test_wait_for_a_long_launch_is_no_time_out(kernels, long_launch, M, G, flags):
    gen = torch.Generator(device="cuda").manual_seed(M)
    x, (Wq, S) = rand_x(M, 1024, gen), rand_w4(1024, 1024, G, gen)
    want = kernels.w4_linear(x, Wq, S, G, flags=flags)
    torch.cuda.synchronize()
    long_launch()
    got = kernels.w4_linear(x, Wq, S, G, flags=flags)
    assert kernels.device_status() == 0 and torch.equal(got, want)


@pytest.mark.parametrize("M,N,K,G", [(1, 3584, 3584, 128), (4, 1000, 2048, 64), (8, 3584, 18944, 128), (13, 3584, 3584, 128),
                                     (16, 3584, 18944, 32), (48, 4608, 3584, 128), (2, 1000, 2048, 32), (2, 512, 3584, 128), (3, 3584, 3584, 128)])
def test_a_plain_launch_runs_the_same_kernel(kernels, M, N, K, G):
    assert kernels.gemv_describe(M, N, K, G, FLAG_NO_PDL) == kernels.gemv_describe(M, N, K, G)
    gen = torch.Generator(device="cuda").manual_seed(N)
    x, (Wq, S) = rand_x(M, K, gen), rand_w4(N, K, G, gen)
    assert torch.equal(kernels.w4_linear(x, Wq, S, G, flags=FLAG_NO_PDL), kernels.w4_linear(x, Wq, S, G))
    assert kernels.device_status() == 0


@pytest.mark.parametrize("M,G", [(1, 128), (3, 128), (4, 128), (8, 128), (13, 128), (16, 128), (4, 64), (16, 32), (48, 128), (300, 64)])
def test_chain_of_dependent_launches(kernels, M, G):
    """Linears that read one another's outputs and write into buffers that are still being read, eager and captured: bit for
    bit the chain with a synchronisation after each launch."""
    gen = torch.Generator(device="cuda").manual_seed(M)
    dims = [1024, 2304, 512, 1024, 1024, 3584, 1024]
    weights = [rand_w4(n, k, G, gen) for k, n in zip(dims, dims[1:])]
    x = rand_x(M, dims[0], gen)
    buffers = [torch.zeros(M * max(dims), dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    kernels.w4_linear(x, *weights[0], G)  # kernels loaded before the capture

    def chain(sync):
        h = x
        for i, w in enumerate(weights):
            y = buffers[i % 2][:M * dims[i + 1]].view(M, dims[i + 1])
            h = kernels.w4_linear(h, *w, G, out=y)
            sync()
        return h

    want = chain(torch.cuda.synchronize).clone()
    assert bool(want.isfinite().all()) and float(want.float().abs().max()) > 0
    for _ in range(20):
        buffers[0].zero_()
        buffers[1].zero_()
        assert torch.equal(chain(lambda: None), want)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        got = chain(lambda: None)
    for _ in range(20):
        buffers[0].zero_()
        buffers[1].zero_()
        graph.replay()
        assert torch.equal(got, want)
    assert kernels.device_status() == 0
