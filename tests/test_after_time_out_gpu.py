"""GPU test of the tcgen05 kernels behind a launch that gave up: they end, store nothing and leave the status as it is; once it
is cleared they answer as before."""
import pytest
import torch

from nanoserve_b200.ops import FLAG_DECODE_NARROW, FLAG_GEMM_NARROW, FLAG_GEMM_NO_PAIRS, FLAG_GEMM_WIDE, narrow_flags

pytestmark = pytest.mark.gpu

CALLS = [(m, FLAG_DECODE_NARROW | narrow_flags(split, tile)) for m in (4, 8, 16) for split in (1, 3) for tile in (1, 2)]
CALLS += [(48, FLAG_GEMM_NARROW | narrow_flags(split, tile)) for split in (1, 3) for tile in (1, 2)]
CALLS += [(300, FLAG_GEMM_WIDE), (300, FLAG_GEMM_WIDE | FLAG_GEMM_NO_PAIRS)]


def test_kernels_behind_a_time_out(kernels):
    gen = torch.Generator(device="cuda").manual_seed(1)
    N, K = 1000, 2048
    Wq = torch.randint(-2**31, 2**31 - 1, (N, K // 8), dtype=torch.int32, device="cuda", generator=gen)
    S = torch.rand(N, K // 128, device="cuda", generator=gen).to(torch.bfloat16)
    xs = {m: torch.randn(m, K, device="cuda", generator=gen).to(torch.bfloat16) for m, _ in CALLS}
    want = [kernels.w4_linear(xs[m], Wq, S, flags=f) for m, f in CALLS]
    sig, epoch = (torch.zeros(1, dtype=torch.int32, device="cuda") for _ in range(2))
    kernels.tp_wait(sig.data_ptr(), epoch.data_ptr(), 1)  # a counter that nothing raises: gives up after its bound
    outs = [torch.full((m, N), 7.0, dtype=torch.bfloat16, device="cuda") for m, _ in CALLS]
    torch.cuda.synchronize()
    try:
        for (m, f), out in zip(CALLS, outs):
            kernels.w4_linear(xs[m], Wq, S, flags=f, out=out)
        assert kernels.device_status() != 0
        assert all(bool((out == 7.0).all()) for out in outs)
    finally:
        kernels.clear_status()
    assert kernels.device_status() == 0
    for (m, f), w in zip(CALLS, want):
        assert torch.equal(kernels.w4_linear(xs[m], Wq, S, flags=f), w)
