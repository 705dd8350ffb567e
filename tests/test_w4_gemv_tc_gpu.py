"""GPU parity tests of the tcgen05 decode GEMV (nine to sixteen tokens, groups of 128, exact weights) against the CPU
oracle: both tile forms, every cluster size class, ragged rows, odd and even numbers of steps."""
import numpy as np
import pytest
import torch

import oracle
from nanoserve_b200.ops import FLAG_DECODE_NARROW, FLAG_MID_KERNEL, narrow_flags
from tests.util import bits_to_torch, check_bf16_output, torch_to_bits, u32_to_torch

pytestmark = pytest.mark.gpu

SLACK = 2e-5  # 16-bit fixed point per (token, 128-chunk): half a unit of 2^-15 per activation, relative to the largest output


def run(k, X, Wq, S, flags):
    y = k.w4_linear(bits_to_torch(X), u32_to_torch(Wq), bits_to_torch(S), 128, flags=flags)
    torch.cuda.synchronize()
    assert k.device_status() == 0
    return torch_to_bits(y)


@pytest.mark.parametrize("tile", [1, 2])
@pytest.mark.parametrize("split", [0, 1, 2, 3, 7, 8])
def test_tiles_and_splits(kernels, tile, split):
    # one row; a row tile less one, full, plus one; 2, 4, 18, 28 steps; scales by two (K / 128 = 2, 6, 18) and by four
    for M, N, K in [(9, 1, 256), (16, 127, 512), (13, 128, 768), (10, 257, 2304), (16, 520, 1024), (11, 300, 2048)]:
        X, Wq, S = oracle.synth_inputs(M, N, K, 128, seed=M + N)
        y = run(kernels, X, Wq, S, FLAG_DECODE_NARROW | narrow_flags(split, tile))
        check_bf16_output(y, oracle.w4_linear_f32(X, Wq, S, 128), SLACK)
        assert np.array_equal(y, run(kernels, X, Wq, S, FLAG_DECODE_NARROW | narrow_flags(split, tile)))


@pytest.mark.parametrize("M", [9, 13, 16])
def test_rule_on_layer_shapes(kernels, M):
    """What the rule picks, against the oracle on sampled rows and against the mma.sync kernel: the same integers in
    another order of fp32 sums."""
    for N, K in [(3584, 3584), (512, 3584), (3584, 18944)]:
        assert kernels.gemv_describe(M, N, K, 128, 0).startswith("tcgen05 GEMV")
        X, Wq, S = oracle.synth_inputs(M, N, K, 128, seed=4)
        y = run(kernels, X, Wq, S, 0)
        rows = np.unique(np.concatenate([[0, N - 1], np.random.default_rng(0).integers(0, N, 40)]))
        check_bf16_output(y[:, rows], oracle.w4_linear_f32(X, Wq[rows], S[rows], 128, threads=oracle.max_threads()), SLACK)
        other = run(kernels, X, Wq, S, FLAG_MID_KERNEL)
        assert (y != other).mean() < 2e-3


def test_extreme_inputs(kernels):
    """A chunk with an infinite or nan x makes its token's outputs nan and touches no other token; x of any magnitude keeps
    its relative precision."""
    M, N, K = 16, 200, 1024
    X, Wq, S = oracle.synth_inputs(M, N, K, 128, seed=5)
    f = oracle.bf16_bits_to_f32(X).copy()
    f[3] *= np.float32(2.0**110)
    f[4] *= np.float32(2.0**-60)
    f[7, 128:256] = 0
    X = oracle.f32_to_bf16_bits(f)
    ref = oracle.w4_linear_f32(X, Wq, S, 128)
    X[0, 130], X[2, 300], X[5, 0] = 0x7F80, 0x7FC0, 0xFF80
    y = run(kernels, X, Wq, S, FLAG_DECODE_NARROW | narrow_flags())
    assert np.isnan(oracle.bf16_bits_to_f32(y[[0, 2, 5]])).all()
    for m in (1, 3, 4, 6, 7, 15):
        check_bf16_output(y[m:m + 1], ref[m:m + 1], SLACK)


@pytest.mark.parametrize("y_off,s_off", [(4, 0), (2, 0), (0, 2), (0, 1), (1, 1)])
def test_alignments(kernels, y_off, s_off):
    """S from 4 bytes and any Y run this kernel, anything less the kernel that serves it: within the same bounds."""
    M, N, K = 13, 1000, 1536
    X, Wq, S = oracle.synth_inputs(M, N, K, 128, seed=6)
    out = torch.zeros(M * N + 8, dtype=torch.bfloat16, device="cuda")
    y = out[y_off:y_off + M * N].view(M, N)
    s = torch.empty(S.size + 8, dtype=torch.bfloat16, device="cuda")[s_off:s_off + S.size].view(*S.shape)
    s.copy_(bits_to_torch(S))
    kernels.w4_linear(bits_to_torch(X), u32_to_torch(Wq), s, 128, out=y)
    torch.cuda.synchronize()
    assert kernels.device_status() == 0
    check_bf16_output(torch_to_bits(y), oracle.w4_linear_f32(X, Wq, S, 128), SLACK)
    assert not out[:y_off].any() and not out[y_off + M * N:].any()
    if s_off % 2 == 0:
        assert np.array_equal(torch_to_bits(y), run(kernels, X, Wq, S, FLAG_DECODE_NARROW))


# tokens, rows, columns, the shorter kernel, us of the many-token and of this kernel
@pytest.mark.parametrize("M,N,K,kernel", [
    (10, 1500, 11008, "tcgen05 GEMV"),  # 10.8, 10.2
    (11, 1444, 9472, "tcgen05 GEMV"),  # 10.4, 9.2
    (16, 57344, 8192, "tcgen05 GEMV"),  # 93, 74
    (16, 700, 256, "tcgen05 GEMV"),  # 3.3, 3.2
    (16, 144, 19456, "many-token kernel"),  # 9.0, 11.4
    (13, 512, 3584, "tcgen05 GEMV"),  # 7.3, 4.5
    (9, 545, 768, "tcgen05 GEMV"),  # 5.7, 3.5
    (13, 3584, 3584, "tcgen05 GEMV"),  # 9.5, 6.7
    (13, 10240, 8192, "tcgen05 GEMV"),  # 24.2, 15.8
    (13, 14336, 4096, "tcgen05 GEMV"),  # 17.3, 12.2
    (13, 37888, 3584, "tcgen05 GEMV"),  # 26.0, 18.1
    (16, 3584, 18944, "tcgen05 GEMV"),  # 20.6, 14.8
])
def test_rule_takes_the_shorter_kernel(kernels, M, N, K, kernel):
    assert kernels.gemv_describe(M, N, K, 128).startswith(kernel)
