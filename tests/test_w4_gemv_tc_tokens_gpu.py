"""GPU parity tests of the tcgen05 GEMV at one to eight tokens (up to four with X in 32 bits, above in 16) against the CPU
oracle, and of the rule that brings plain calls of two to sixteen tokens there."""
import numpy as np
import pytest
import torch

import oracle
from nanoserve_b200.ops import FLAG_DECODE_NARROW, FLAG_MID_KERNEL, FLAG_NO_PDL, FLAG_RING_KERNEL, narrow_flags
from tests.util import bits_to_torch, check_bf16_output, torch_to_bits, u32_to_torch

pytestmark = pytest.mark.gpu


def slack(M):
    # relative to the largest output: fp32 summation order for X in 32 bits; half a unit of 2^-15 per activation in 16
    return 3e-6 if M <= 4 else 2e-5


def run(k, X, Wq, S, flags):
    y = k.w4_linear(bits_to_torch(X), u32_to_torch(Wq), bits_to_torch(S), 128, flags=flags)
    torch.cuda.synchronize()
    assert k.device_status() == 0
    return torch_to_bits(y)


@pytest.mark.parametrize("tile", [1, 2])
@pytest.mark.parametrize("split", [1, 2, 3, 5, 8])
def test_tiles_and_splits(kernels, tile, split):
    # one row; a row tile less one, plus one; one pair of steps (a group of warps without work), odd numbers of them, rings
    # that wrap; scales by two (K / 128 = 2, 6) and by four
    for M, N, K in [(1, 1, 256), (2, 127, 512), (4, 129, 768), (3, 257, 2304), (5, 255, 1280), (8, 257, 4096), (7, 40, 9216)]:
        X, Wq, S = oracle.synth_inputs(M, N, K, 128, seed=M + N)
        flags = FLAG_DECODE_NARROW | narrow_flags(split, tile)
        y = run(kernels, X, Wq, S, flags)
        check_bf16_output(y, oracle.w4_linear_f32(X, Wq, S, 128), slack(M))
        assert np.array_equal(y, run(kernels, X, Wq, S, flags))
        assert np.array_equal(y, run(kernels, X, Wq, S, flags | FLAG_NO_PDL))


@pytest.mark.parametrize("M,K", [(2, 1024), (3, 1536), (8, 768)])  # scales by four, by four and by two
@pytest.mark.parametrize("y_off,s_off", [(0, 0), (1, 0), (2, 2), (3, 4), (0, 1), (1, 3)])
def test_alignments(kernels, M, K, y_off, s_off):
    """The outputs are stored one by one, wherever they start; scales are loaded in pairs or fours, and where S starts at an odd
    one another kernel runs, within the 16-bit form's bound."""
    N = 1000
    X, Wq, S = oracle.synth_inputs(M, N, K, 128, seed=6)
    out = torch.full((M * N + 8,), 7.0, dtype=torch.bfloat16, device="cuda")
    y = out[y_off:y_off + M * N].view(M, N)
    s = torch.empty(S.size + 8, dtype=torch.bfloat16, device="cuda")[s_off:s_off + S.size].view(*S.shape)
    s.copy_(bits_to_torch(S))
    kernels.w4_linear(bits_to_torch(X), u32_to_torch(Wq), s, 128, out=y)
    torch.cuda.synchronize()
    assert kernels.device_status() == 0
    check_bf16_output(torch_to_bits(y), oracle.w4_linear_f32(X, Wq, S, 128), slack(M) if s_off % 2 == 0 else 2e-5)
    assert bool((out[:y_off] == 7.0).all()) and bool((out[y_off + M * N:] == 7.0).all())
    if s_off % 2 == 0:
        assert np.array_equal(torch_to_bits(y), run(kernels, X, Wq, S, FLAG_DECODE_NARROW))


@pytest.mark.parametrize("M", [4, 8, 16])
def test_longest_k_of_a_cta(kernels, M):
    N, K = 130, 28672  # 112 pairs in one CTA
    X, Wq, S = oracle.synth_inputs(M, N, K, 128, seed=9)
    ref = oracle.w4_linear_f32(X, Wq, S, 128, threads=oracle.max_threads())
    for tile in (1, 2):
        check_bf16_output(run(kernels, X, Wq, S, FLAG_DECODE_NARROW | narrow_flags(1, tile)), ref, slack(M))


@pytest.mark.parametrize("M", [3, 4, 8])
def test_extreme_inputs(kernels, M):
    N, K = 200, 1024
    X, Wq, S = oracle.synth_inputs(M, N, K, 128, seed=5)
    f = oracle.bf16_bits_to_f32(X).copy()
    f[0] *= np.float32(2.0**110)
    f[1] *= np.float32(2.0**-60)
    f[1, 128:256] = 0
    X = oracle.f32_to_bf16_bits(f)
    ref = oracle.w4_linear_f32(X, Wq, S, 128)
    X[2, 300] = 0x7FC0 if M == 4 else 0xFF80
    y = run(kernels, X, Wq, S, FLAG_DECODE_NARROW | narrow_flags())
    assert np.isnan(oracle.bf16_bits_to_f32(y[2])).all()
    for m in (0, 1):
        check_bf16_output(y[m:m + 1], ref[m:m + 1], slack(M))


@pytest.mark.parametrize("M,N,K", [(2, 3584, 18944), (4, 37888, 3584), (6, 4608, 3584), (8, 10240, 8192), (16, 18944, 3584)])
def test_rule_on_layer_shapes(kernels, M, N, K):
    assert "tcgen05" in kernels.gemv_describe(M, N, K, 128) and kernels.gemv_scratch_bytes(M, N, K) == 0
    X, Wq, S = oracle.synth_inputs(M, N, K, 128, seed=4)
    y = run(kernels, X, Wq, S, 0)
    rows = np.unique(np.concatenate([[0, N - 1], np.random.default_rng(0).integers(0, N, 40)]))
    check_bf16_output(y[:, rows], oracle.w4_linear_f32(X, Wq[rows], S[rows], 128, threads=oracle.max_threads()), slack(M))


# the shorter kernel, us of the other and of this one
@pytest.mark.parametrize("M,N,K,here", [
    (2, 18944, 3584, False),  # 8.9 and 10.0
    (4, 22705, 1024, False),  # 4.8, 5.4
    (8, 512, 3584, True),     # 6.6, 3.9
    (2, 512, 3584, True),     # 6.7, 3.6
    (1, 37888, 3584, False),  # 13.7, 15.7
    (4, 3584, 3584, True),    # 7.5, 5.6
    (8, 700, 256, True),      # 3.1, 2.5
    (4, 8192, 28672, True),   # 40.7, 28
    (16, 57344, 8192, True),  # 91, 68
])
def test_rule_takes_the_shorter_kernel(kernels, M, N, K, here):
    assert ("tcgen05" in kernels.gemv_describe(M, N, K, 128)) == here


# us of the kernel that keeps the call and of this one
@pytest.mark.parametrize("M,N,K", [
    (10, 178, 26112),   # 9.4, 14.5
    (9, 440, 27648),    # 11.1, 15.5
    (16, 144, 19456),   # 9.0, 11.4
    (16, 290, 22784),   # 10.7, 12.0
    (12, 84, 13824),    # 7.6, 8.3
    (7, 54677, 256),    # 6.3, 7.6
    (2, 29616, 5632),   # 19.3, 21.7
    (2, 37888, 3584),   # 14.6, 15.5
    (2, 18928, 4096),   # 10.2, 11.9
])
def test_rule_leaves_calls_where_they_are_shorter(kernels, M, N, K):
    assert "tcgen05" not in kernels.gemv_describe(M, N, K, 128)


@pytest.mark.parametrize("M,N,K", [(5, 2300, 2048), (8, 700, 256), (16, 1500, 11008), (10, 178, 26112), (2, 900, 2560)])
def test_a_plain_call_runs_the_kernel_it_is_described_as(kernels, M, N, K):
    """The kernels differ in the order of their fp32 sums: the call's bits are those of the kernel with its name."""
    flags = {"tcgen05 GEMV": FLAG_DECODE_NARROW, "many-token kernel": FLAG_MID_KERNEL, "ring kernel": FLAG_RING_KERNEL}
    name = kernels.gemv_describe(M, N, K, 128).split(":")[0]
    assert kernels.gemv_describe(M, N, K, 128, flags[name]) == kernels.gemv_describe(M, N, K, 128)
    X, Wq, S = oracle.synth_inputs(M, N, K, 128, seed=8)
    assert np.array_equal(run(kernels, X, Wq, S, 0), run(kernels, X, Wq, S, flags[name]))


# us of the streaming kernel and of this one
@pytest.mark.parametrize("N,K,here", [
    (512, 3584, True),      # 4.5, 3.4
    (130, 1024, True),      # 3.5, 2.7
    (130, 768, False),
    (4096, 2048, True),     # 4.4, 4.1
    (4997, 1536, False),    # 4.2, 4.8
    (4980, 14080, True),    # 15.0, 12.8
    (8192, 28672, True),    # 29.2, 26.6
    (3584, 3584, False),    # 5.0, 5.1
    (8430, 1024, False),    # 4.1, 4.8
    (6308, 5632, False),    # 7.8, 8.4
])
def test_one_token_runs_the_shorter_kernel(kernels, N, K, here):
    assert ("tcgen05" in kernels.gemv_describe(1, N, K, 128)) == here
    X, Wq, S = oracle.synth_inputs(1, N, K, 128, seed=7)
    f = oracle.bf16_bits_to_f32(X).copy()
    f[0, ::97] *= np.float32(1000.0)  # X has 32 bits in either kernel: outliers cost the others nothing
    X = oracle.f32_to_bf16_bits(f)
    rows = np.unique(np.concatenate([[0, N - 1], np.random.default_rng(0).integers(0, N, 60)]))
    ref = oracle.w4_linear_f32(X, Wq[rows], S[rows], 128, threads=oracle.max_threads())
    check_bf16_output(run(kernels, X, Wq, S, 0)[:, rows], ref, slack(1))


# both sides of every line, us of the streaming kernel and of this one
@pytest.mark.parametrize("N,K,here", [
    (3500, 2048, False),    # 4.4, 5.3: tiles of 256 rows
    (4096, 1024, True),     # 4.1, 3.2
    (2861, 3584, False),    # 5.1, 5.6
    (1909, 4352, True),     # 5.5, 4.1
    (11771, 28160, False),  # 38.9, 54.3: 92 CTAs
    (10140, 26880, True),   # 31.4, 29.0: 120
    (8264, 25088, True),    # 24.1, 22.7: clusters of four in all their places
    (11343, 26624, True),   # 36.4, 34: clusters of three in all their places
    (13819, 25856, True),   # 53.8, 43.0: the other kernel's 216 CTAs take an SM each
    (14651, 27136, False),  # 48.1, 54.8: its 115 CTAs do
    (7300, 24064, False),   # outside the lines in N and K
    (4992, 12544, True),    # 13.5, 11.4
    (5100, 12544, False),
    (256, 896, False),      # K is no multiple of 256
])
def test_one_token_on_both_sides_of_the_lines(kernels, N, K, here):
    assert ("tcgen05" in kernels.gemv_describe(1, N, K, 128)) == here


# K / 256 odd and more than eight pairs per CTA: scales that are brought into L2 ahead; tiles cut off, one CTA, K cut
@pytest.mark.parametrize("M,N,K,form,split", [(1, 300, 2816, 2, 1), (4, 129, 4352, 1, 1), (8, 700, 12544, 2, 1), (13, 257, 5888, 2, 2),
                                              (16, 64, 8448, 1, 3), (5, 513, 2304, 2, 1)])
def test_scales_ahead(kernels, M, N, K, form, split):
    flags = FLAG_DECODE_NARROW | narrow_flags(split, form)
    X, Wq, S = oracle.synth_inputs(M, N, K, 128, seed=N)
    ref = oracle.w4_linear_f32(X, Wq, S, 128, threads=oracle.max_threads())
    check_bf16_output(run(kernels, X, Wq, S, flags), ref, slack(M))


# clusters of three in nearly all places of the device (44 and 45 of 45 on 148 SMs), one after the other: their CTAs leave together
@pytest.mark.parametrize("M,N,K", [(4, 11500, 5632), (13, 11300, 6144), (8, 11200, 5888), (4, 11500, 5120)])
def test_clusters_of_three_in_a_chain(kernels, M, N, K):
    flags = FLAG_DECODE_NARROW | narrow_flags(3, 2)
    X, Wq, S = oracle.synth_inputs(M, N, K, 128, seed=M)
    x, wq, s = bits_to_torch(X), u32_to_torch(Wq), bits_to_torch(S)
    outs = [kernels.w4_linear(x, wq, s, 128, flags=flags) for _ in range(8)]
    torch.cuda.synchronize()
    assert kernels.device_status() == 0 and all(torch.equal(o, outs[0]) for o in outs)
    rows = np.random.default_rng(M).integers(0, N, 40)
    check_bf16_output(torch_to_bits(outs[0])[:, rows], oracle.w4_linear_f32(X, Wq[rows], S[rows], 128, threads=oracle.max_threads()), slack(M))
