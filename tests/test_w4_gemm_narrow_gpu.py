"""GPU parity tests of the few-token GEMM (weights as the M side of the MMA, converted into tensor memory) against the
CPU oracle: every tile form and cluster size, at the edges of the token, row and K tiles."""
import numpy as np
import pytest
import torch

import oracle
from nanoserve_b200.ops import FLAG_DECODE_NARROW, FLAG_GEMM_NO_PAIRS, FLAG_GEMM_WIDE, narrow_flags
from tests.test_w4_gemm_gpu import rounded_weight_reference
from tests.util import bits_to_torch, check_bf16_output, torch_to_bits, u32_to_torch

pytestmark = pytest.mark.gpu


def run(k, X, Wq, S, G, flags):
    y = k.w4_linear(bits_to_torch(X), u32_to_torch(Wq), bits_to_torch(S), G, flags=flags)
    torch.cuda.synchronize()
    assert k.device_status() == 0
    return torch_to_bits(y)


# token columns 32 to 128 and two token tiles; rows below, at and above a tile, N odd; K of a quarter block, of whole
# blocks, with a tail of 32, 64 and 96, shorter than the cluster; scales that load by four, by two and one by one
SHAPES = [(17, 300, 1024, 128), (33, 129, 384, 128), (48, 513, 1152, 128), (64, 256, 640, 64), (65, 131, 544, 32),
          (96, 256, 96, 96), (113, 77, 1120, 32), (128, 512, 2048, 128), (129, 260, 1024, 128), (200, 1, 160, 32),
          (31, 400, 32, 32), (40, 128, 4096, 256)]


@pytest.mark.parametrize("tile", [1, 2])
@pytest.mark.parametrize("split", [0, 1, 2, 5, 8])
def test_tiles_and_splits(kernels, tile, split):
    for M, N, K, G in SHAPES:
        X, Wq, S = oracle.synth_inputs(M, N, K, G, seed=M + N)
        y = run(kernels, X, Wq, S, G, narrow_flags(split, tile))
        # weights rounded to bf16 once, fp32 sums: half a bf16 step plus the sums' error (K <= 4096 terms)
        check_bf16_output(y, rounded_weight_reference(X, Wq, S, G), 3e-5)
        assert np.array_equal(y, run(kernels, X, Wq, S, G, narrow_flags(split, tile))), "two identical launches differ"


@pytest.mark.parametrize("M", [17, 48, 100, 128, 300, 512])
def test_rule_agrees_with_the_wide_kernel(kernels, M):
    """What the rule picks against the general kernel on layer shapes: the same products in another order of sums."""
    for N, K, G in [(4608, 3584, 128), (3584, 18944, 128), (1000, 4096, 64)]:
        X, Wq, S = oracle.synth_inputs(M, N, K, G, seed=3)
        a = oracle.bf16_bits_to_f32(run(kernels, X, Wq, S, G, 0))
        b = oracle.bf16_bits_to_f32(run(kernels, X, Wq, S, G, FLAG_GEMM_WIDE))
        assert np.abs(a - b).max() <= 2.0**-7 * np.abs(b).max()
        assert (a != b).mean() < 0.05  # sums that differ in the last fp32 bits round differently once in a while


@pytest.mark.parametrize("tile", [1, 2])
@pytest.mark.parametrize("split", [0, 1, 3, 8])
def test_decode_tokens(kernels, tile, split):
    """At most 16 tokens: row tiles cut off, one K block, odd and even numbers of blocks, every way to read scales."""
    for M, N, K, G in [(1, 300, 1024, 64), (2, 129, 256, 32), (16, 512, 3584, 64), (13, 260, 2304, 32), (7, 77, 640, 128),
                       (5, 256, 1088, 64), (16, 130, 640, 32), (9, 131, 352, 32), (3, 64, 192, 96)]:
        X, Wq, S = oracle.synth_inputs(M, N, K, G, seed=M + K)
        y = run(kernels, X, Wq, S, G, FLAG_DECODE_NARROW | narrow_flags(split, tile))
        check_bf16_output(y, rounded_weight_reference(X, Wq, S, G), 3e-5)


def test_decode_of_fine_groups_takes_any_alignment(kernels):
    """Fine groups at decode token counts run the few-token GEMM where pointers are 16-byte aligned, and the GEMV where they
    are not: the results agree to a rounding of the output and of the sums."""
    M, N, K, G = 4, 1000, 2048, 64
    assert kernels.gemv_describe(M, N, K, G, 0).startswith("few-token GEMM")
    X, Wq, S = oracle.synth_inputs(M, N, K, G, seed=8)
    x, wq, s = bits_to_torch(X), u32_to_torch(Wq), bits_to_torch(S)
    want = oracle.bf16_bits_to_f32(torch_to_bits(kernels.w4_linear(x, wq, s, G)))
    room = torch.empty(M * N + 8, dtype=torch.bfloat16, device="cuda")
    out = room[1:1 + M * N].view(M, N)
    s_off = torch.empty(S.size + 1, dtype=torch.bfloat16, device="cuda")[1:].view(*S.shape).copy_(s)
    kernels.w4_linear(x, wq, s_off, G, out=out)
    torch.cuda.synchronize()
    assert kernels.device_status() == 0
    got = oracle.bf16_bits_to_f32(torch_to_bits(out))
    assert np.abs(got - want).max() <= 2.0**-7 * np.abs(want).max()


# tokens, rows, K, group, the kernel that was the shorter one, us of the general and of this kernel timed in turn
@pytest.mark.parametrize("M,N,K,G,kernel", [
    (2048, 3584, 18944, 128, "prefill GEMM"),  # 221, 255
    (1536, 3584, 18944, 128, "prefill GEMM"),  # 178, 191
    (512, 3584, 18944, 128, "few-token GEMM"),  # 77, 64
    (2048, 4096, 13696, 128, "prefill GEMM"),  # 167, 235 (scales one by one)
    (768, 4096, 13696, 128, "prefill GEMM"),  # 87, 102
    (256, 4096, 13696, 128, "few-token GEMM"),  # 63, 36
    (2048, 8192, 28672, 128, "prefill GEMM"),  # 774, 843
    (256, 8192, 28672, 128, "few-token GEMM"),  # 135, 99
    (2048, 4096, 14336, 128, "prefill GEMM"),  # 184, 196
    (4096, 4096, 14336, 128, "prefill GEMM"),  # 363, 420
    (512, 4096, 14336, 128, "few-token GEMM"),  # 68, 52
    (1536, 5120, 13824, 128, "prefill GEMM"),  # 164, 178
    (2048, 8192, 8192, 128, "prefill GEMM"),  # 201, 234
    (768, 28672, 8192, 128, "few-token GEMM"),  # 344, 288
    (512, 37888, 3584, 128, "prefill GEMM"),  # 108, 118
    (512, 4608, 3584, 128, "few-token GEMM"),  # 41, 19
    (8192, 18944, 3584, 128, "prefill GEMM"),
    (1070, 6051, 1792, 128, "few-token GEMM"),  # 108, 32 (an odd number of rows: the general kernel stores value by value)
])
def test_rule_takes_the_shorter_kernel(kernels, M, N, K, G, kernel):
    assert kernels.gemv_describe(M, N, K, G).startswith(kernel)


# tokens, rows, K, group, the kernel that was the shorter one, us of the ring GEMV and of this kernel
@pytest.mark.parametrize("M,N,K,G,kernel", [
    (14, 313, 28224, 64, "ring kernel"),  # 13.7, 31.2 (441 groups a row: scales one by one)
    (6, 8436, 8032, 32, "ring kernel"),  # 24.4, 39.9
    (16, 449, 13920, 32, "ring kernel"),  # 14.4, 24.1
    (4, 18944, 3584, 64, "few-token GEMM"),
    (16, 3584, 18944, 64, "few-token GEMM"),  # 64.4, 18.4
    (16, 3584, 18944, 32, "few-token GEMM"),
])
def test_rule_at_decode_tokens(kernels, M, N, K, G, kernel):
    assert kernels.gemv_describe(M, N, K, G).startswith(kernel)


@pytest.mark.parametrize("M,flags", [(32, narrow_flags(1, 1)), (32, narrow_flags(2, 2)), (32, FLAG_GEMM_WIDE), (300, FLAG_GEMM_NO_PAIRS | FLAG_GEMM_WIDE),
                                     (300, FLAG_GEMM_WIDE)])
@pytest.mark.parametrize("G", [32, 64, 128])
def test_scales_of_any_size(kernels, M, flags, G):
    """Tokens that pick one k each give back single weights, which are RN_bf16((q - 8) * s) to the bit: scales on either side of
    the line below which a weight is one fused multiply-add, rows that cross it and rows beside them that do not."""
    N, K = 200, 512
    gen = torch.Generator(device="cuda").manual_seed(G)
    Wq = torch.randint(-2**31, 2**31 - 1, (N, K // 8), dtype=torch.int32, device="cuda", generator=gen)
    sizes = torch.tensor([1.0, 7.96875, 8.0, -7.96875, -8.0, 0.0133, 1e4, 3e37, 1e-30, 0.0], device="cuda")
    S = sizes[torch.randint(0, 10, (N, K // G), device="cuda", generator=gen)].to(torch.bfloat16)
    S[:N // 2, 1:] = 0.02  # warps whose rows leave the line for a group only
    ks = torch.randint(0, K, (M,), device="cuda", generator=gen)
    x = torch.zeros(M, K, dtype=torch.bfloat16, device="cuda")
    x[torch.arange(M, device="cuda"), ks] = 1.0
    shifts = torch.arange(0, 32, 4, device="cuda", dtype=torch.int32)
    w = (((Wq[:, :, None] >> shifts) & 15).flatten(1) - 8).float() * S.float().repeat_interleave(G, dim=1)
    y = kernels.w4_linear(x, Wq, S, G, flags=flags)
    assert kernels.device_status() == 0
    assert torch.equal(y.float(), w.to(torch.bfloat16)[:, ks].T.float())
    S[3, 0] = float("inf")
    y = kernels.w4_linear(x, Wq, S, G, flags=flags)
    assert bool(y[:, 3].isnan().any()) and bool(y[:, :3].isfinite().all()) and bool(y[:, 4:].isfinite().all())
    assert kernels.device_status() == 0


@pytest.mark.parametrize("M,flags", [(32, narrow_flags(1, 1)), (32, narrow_flags(2, 2)), (32, FLAG_GEMM_WIDE), (300, FLAG_GEMM_NO_PAIRS | FLAG_GEMM_WIDE),
                                     (300, FLAG_GEMM_WIDE)])
@pytest.mark.parametrize("G", [32, 64, 128])
@pytest.mark.parametrize("up", [2.0**100, 1.0])
def test_scales_at_the_ends_of_their_range(kernels, M, flags, G, up):
    """Weights down to the smallest bf16 and up to the largest, picked out one by one: RN_bf16((q - 8) * s) to the bit.  Small ones
    are picked with 2^100 and come out as normal numbers."""
    N, K = 200, 512
    gen = torch.Generator(device="cuda").manual_seed(G)
    Wq = torch.randint(-2**31, 2**31 - 1, (N, K // 8), dtype=torch.int32, device="cuda", generator=gen)
    below = [2.0**-133, 3 * 2.0**-133, 1.3e-39, 2.0**-126, 1.9e-38, 2.0**-122, 1.1e-37, 2.0**-121, 3.1e-36, 2.0**-118, 5e-36, 1e-33]
    above = [0.2490234375, 0.25, -0.25, 0.49, 0.5, 1.3, 2.0**100, 2.0**124, -1.1 * 2.0**124]
    sizes = torch.tensor(below if up > 1 else above, device="cuda", dtype=torch.float64).float().to(torch.bfloat16)
    S = sizes[torch.randint(0, len(sizes), (N, K // G), device="cuda", generator=gen)]
    S[:N // 2, 1:] = sizes[0]  # warps whose rows leave a range for a group only
    S[N // 2:N // 2 + 32] = below[4] if up > 1 else 2.0  # a warp of one size
    if up > 1:
        S[1] = 0.3  # small scales beside one above the line
    ks = torch.randint(0, K, (M,), device="cuda", generator=gen)
    x = torch.zeros(M, K, dtype=torch.bfloat16, device="cuda")
    x[torch.arange(M, device="cuda"), ks] = up
    shifts = torch.arange(0, 32, 4, device="cuda", dtype=torch.int32)
    w = (((Wq[:, :, None] >> shifts) & 15).flatten(1) - 8).double() * S.double().repeat_interleave(G, dim=1)
    q = torch.exp2(torch.clamp(torch.floor(torch.log2(w.abs())) - 7, min=-133.0))  # a bf16's last place
    want = torch.where(w == 0, w, torch.round(w / q) * q)[:, ks].T * up
    y = kernels.w4_linear(x, Wq, S, G, flags=flags).double()
    assert kernels.device_status() == 0
    assert bool(want.isfinite().all()) and torch.equal(y, want)


@pytest.mark.parametrize("G", [64, 32])
@pytest.mark.parametrize("M,N,K,split", [(3, 300, 6400, 1), (48, 257, 6400, 1), (64, 31, 6912, 1), (20, 513, 12544, 2), (20, 256, 6144, 1),
                                         (70, 256, 6400, 1)])
def test_scales_ahead(kernels, M, N, K, split, G):
    """Shares of K around the line from which scales are brought into L2 ahead: above it with rows cut off, parts that are sent, and on
    the other side (K a multiple of 512, more than 64 token columns)."""
    X, Wq, S = oracle.synth_inputs(M, N, K, G, seed=N)
    flags = narrow_flags(split, 2) | (FLAG_DECODE_NARROW if M <= 16 else 0)
    check_bf16_output(run(kernels, X, Wq, S, G, flags), rounded_weight_reference(X, Wq, S, G), 6e-5)
