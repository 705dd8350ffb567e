"""GPU parity tests of the quantizer through the C ABI: bit-exact against the CPU oracle."""
import ctypes
import os

import numpy as np
import pytest
import torch

import oracle
from tests.util import bits_to_torch, torch_to_bits, torch_to_u32

pytestmark = pytest.mark.gpu


def quant(k, W_bits, G):
    Wq, S = k.w4_quantize(bits_to_torch(W_bits), G)
    torch.cuda.synchronize()
    return torch_to_u32(Wq), torch_to_bits(S)


@pytest.mark.parametrize("N,K,G", [(256, 512, 128), (64, 256, 32), (33, 384, 64), (8, 1024, 256), (5, 96, 96),
                                   (3584, 3584, 128)])
def test_bit_exact_against_oracle(kernels, N, K, G):
    rng = np.random.default_rng([N, K, G])
    cases = {
        "reference fill (bench_w4a16.cu:32-40, seed 11)": oracle.fill_bf16(N * K, 11, 0.05).reshape(N, K),
        "normal": oracle.f32_to_bf16_bits(rng.standard_normal((N, K), dtype=np.float32) * 0.02),
        "wide dynamic range": oracle.f32_to_bf16_bits(
            (rng.standard_normal((N, K)) * np.exp(rng.uniform(-20, 20, size=(N, 1)))).astype(np.float32)),
    }
    z = cases["normal"].copy()
    z[0, :G] = 0          # an all-zero group: scale 1, q = 8
    z[-1, -G:] = 0x8000   # negative zeros
    cases["zero groups"] = z
    for name, W in cases.items():
        Wq, S = quant(kernels, W, G)
        Wq_o, S_o = oracle.w4_quantize(W, G)
        assert np.array_equal(S, S_o), name
        assert np.array_equal(Wq, Wq_o), name


def test_ties_round_to_even(kernels):
    G = 32
    vals = np.zeros((1, 32), dtype=np.float32)
    vals[0, :8] = [7.0, 0.5, 1.5, 2.5, -0.5, -1.5, -2.5, 3.5]
    Wq, S = quant(kernels, oracle.f32_to_bf16_bits(vals), G)
    q = oracle.w4_unpack(Wq)[0][:8]
    assert list(q) == [7, 0, 2, 2, 0, -2, -2, 4]


@pytest.mark.parametrize("G", [32, 64, 128, 256])
def test_every_significand_and_special_groups(kernels, G):
    """The division-free rounding against the oracle's division: every significand of a group's largest value, which sets s,
    with every significand of another member at every exponent where w / s can be halfway between two integers (|w| from
    1/32 of the largest value up), scales at both ends of the range, infinite and nan members, and a word count that fills
    no block."""
    rng = np.random.default_rng(G)
    rows = []
    for top in range(128, 256):
        w = (np.arange(128, 256, dtype=np.float64)[:, None] * 2.0 ** np.arange(-5, 1)).reshape(-1)
        w = w[w <= top] * rng.choice([-1, 1], (w <= top).sum())
        for i in range(0, len(w), G - 1):
            g = np.resize(w[i:i + G - 1], G)
            g[G - 1] = top  # (np.resize wraps round: the last member of a full part is a repeat of its first)
            rows.append(rng.permutation(g))
    W = oracle.f32_to_bf16_bits(np.array(rows, dtype=np.float32))
    halves = (np.array(rows) * 0 + rng.integers(-14, 15, (len(rows), G)) / 2)  # s = 1: every second one is a tie
    halves[:, 0] = 7.0
    special = oracle.f32_to_bf16_bits(rng.standard_normal((12, G), dtype=np.float32))
    for r, (lo, hi) in enumerate([(0x0001, 0x0040), (0x0080, 0x0100), (0x0300, 0x0D80), (0x7000, 0x7F7F)]):
        special[r] = rng.integers(lo, hi, G) | (rng.integers(0, 2, G) << 15)  # subnormal to largest magnitudes
    W = np.concatenate([W, oracle.f32_to_bf16_bits(halves.astype(np.float32)), special])
    Wq, S = quant(kernels, W, G)
    Wq_o, S_o = oracle.w4_quantize(W, G)
    assert np.array_equal(S, S_o) and np.array_equal(Wq, Wq_o)
    # an infinite or nan member changes its own group only
    bad = W.copy()
    bad[1, 3], bad[5, 0], bad[9, G - 1] = 0x7F80, 0x7FC0, 0xFF80
    Wq_b, S_b = quant(kernels, bad, G)
    keep = np.setdiff1d(np.arange(len(W)), [1, 5, 9])
    assert np.array_equal(Wq_b[keep], Wq_o[keep]) and np.array_equal(S_b[keep], S_o[keep])
    assert oracle.bf16_bits_to_f32(S_b[1])[0] == np.inf and oracle.bf16_bits_to_f32(S_b[9])[0] == np.inf
    assert (Wq_b[5, 0] & 15) == 8  # a nan is stored as the zero point, its group scaled by the other members


def test_error_codes(kernels):
    W = torch.zeros(4, 96, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(RuntimeError, match="ns_w4_quantize failed with code -1"):
        kernels.w4_quantize(W, 64)   # K % G  (csrc/nanoserve_ops.cu:67)
    with pytest.raises(RuntimeError, match="ns_w4_quantize failed with code -1"):
        kernels.w4_quantize(W, 48)   # G % 32


def test_round_trip_then_linear_matches_oracle(kernels):
    """quantize -> linear on the GPU equals quantize -> linear in the oracle (the reference's own check,
    bench/bench_w4a16.cu:142-180, on its own seeded inputs)."""
    from tests.util import check_bf16_output, u32_to_torch
    N, K, G = 256, 512, 128
    W = oracle.fill_bf16(N * K, 11, 0.05).reshape(N, K)
    Wq, S = kernels.w4_quantize(bits_to_torch(W), G)
    for M in (1, 8, 16):
        X = oracle.fill_bf16(M * K, 12, 1.0).reshape(M, K)
        y = kernels.w4_linear(bits_to_torch(X), Wq, S, G)
        torch.cuda.synchronize()
        ref = oracle.w4_linear_f32(X, torch_to_u32(Wq), torch_to_bits(S), G)
        check_bf16_output(torch_to_bits(y), ref, 3e-6)


def test_against_reference_quantizer(kernels):
    path = oracle.REF_LIB_PATH
    if not os.path.exists(path):
        pytest.skip("reference library not built (oracle/_ref/libnanoserve_ref.so)")
    ref = ctypes.CDLL(path)
    vp, i32 = ctypes.c_void_p, ctypes.c_int
    ref.ns_w4_quantize.argtypes = [vp, vp, vp, i32, i32, i32, vp]
    ref.ns_w4_quantize.restype = i32
    N, K, G = 1024, 3584, 128
    W = bits_to_torch(oracle.fill_bf16(N * K, 11, 0.05).reshape(N, K))
    Wq_r = torch.empty(N, K // 8, dtype=torch.int32, device="cuda")
    S_r = torch.empty(N, K // G, dtype=torch.bfloat16, device="cuda")
    assert ref.ns_w4_quantize(W.data_ptr(), Wq_r.data_ptr(), S_r.data_ptr(), N, K, G,
                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    Wq, S = kernels.w4_quantize(W, G)
    torch.cuda.synchronize()
    assert torch.equal(Wq, Wq_r) and torch.equal(S.view(torch.int16), S_r.view(torch.int16))
