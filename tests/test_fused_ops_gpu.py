"""GPU tests of the element-wise neighbours of the linears (ns_rmsnorm, ns_rope, ns_swiglu) and of the decode
helpers, against plain PyTorch fp32 references of the same ops (the reference project's own *_ref functions follow the
same formulas, python/nanoserve/ops.py:101-142).  Bound: 3e-2 relative to |ref| + 1, the reference's fused-op gate
(bench/bench_fused.cu:70-77)."""
import ctypes
import os
import subprocess
import sys

import pytest
import torch
import torch.nn.functional as F

from nanoserve_b200.ops import FLAG_GEMM_NO_PAIRS, FLAG_GEMM_WIDE

pytestmark = pytest.mark.gpu


def close(a, ref, tol=3e-2):
    return bool(torch.all((a.float() - ref.float()).abs() <= tol * (ref.float().abs() + 1)))


@pytest.mark.parametrize("T,H", [(1, 3584), (8, 256), (5, 8192)])
def test_rmsnorm(kernels, T, H):
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(T, H, device="cuda", generator=g).to(torch.bfloat16)
    r = torch.randn(T, H, device="cuda", generator=g).to(torch.bfloat16)
    w = (1 + 0.1 * torch.randn(H, device="cuda", generator=g)).to(torch.bfloat16)
    for res in (None, r):
        xi = x.clone()
        y = kernels.rmsnorm(xi, res, w, 1e-6)
        xs = (x.float() + res.float()).to(torch.bfloat16) if res is not None else x
        h = xs.float()
        ref = h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-6) * w.float()
        assert close(y, ref)
        assert torch.equal(xi, xs)  # the residual stream is updated in place, rounded to bf16


def test_rope_and_swiglu(kernels):
    g = torch.Generator(device="cuda").manual_seed(2)
    T, Hq, Hk, D = 6, 4, 2, 128
    q = torch.randn(T, Hq * D, device="cuda", generator=g).to(torch.bfloat16)
    k = torch.randn(T, Hk * D, device="cuda", generator=g).to(torch.bfloat16)
    inv = 1.0 / (1e4 ** (torch.arange(0, D, 2, device="cuda").float() / D))
    q0, k0 = q.clone().float(), k.clone().float()
    kernels.rope(q, k, inv, Hq, Hk, D, 7)
    fr = torch.outer(torch.arange(7, 7 + T, device="cuda").float(), inv)
    cos, sin = torch.cat([fr, fr], -1).cos()[:, None], torch.cat([fr, fr], -1).sin()[:, None]
    for got, src, H in ((q, q0, Hq), (k, k0, Hk)):
        v = src.view(T, H, D)
        ref = v * cos + torch.cat([-v[..., D // 2:], v[..., :D // 2]], -1) * sin
        assert close(got.view(T, H, D), ref)
    a = torch.randn(3, 512, device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn(3, 512, device="cuda", generator=g).to(torch.bfloat16)
    assert close(kernels.swiglu(a, b), F.silu(a.float()) * b.float())
    with pytest.raises(RuntimeError, match="ns_swiglu failed with code -1"):
        kernels.swiglu(a[:1, :4].contiguous(), b[:1, :4].contiguous())  # T*I % 8 (csrc/nanoserve_ops.cu:39)


@pytest.mark.parametrize("T,Hq,Hk,D,with_bias", [(1, 4, 1, 128, True), (7, 3, 2, 64, True), (33, 28, 4, 128, False),
                                                 (5, 2, 1, 16, True)])
def test_qkv_prefill_equals_its_parts(kernels, T, Hq, Hk, D, with_bias):
    """Bias, rotation and cache stores in one kernel: bit for bit what the separate operators give; cache rows behind the
    prompt stay."""
    g = torch.Generator(device="cuda").manual_seed(T)
    W = (Hq + 2 * Hk) * D
    qkv = torch.randn(T, W, device="cuda", generator=g).to(torch.bfloat16)
    bias = torch.randn(W, device="cuda", generator=g).to(torch.bfloat16) if with_bias else None
    inv = 1.0 / (1e6 ** (torch.arange(0, D, 2, device="cuda").float() / D))
    ck = torch.full((Hk, T + 3, D), 5.0, dtype=torch.bfloat16, device="cuda")
    cv = ck.clone()
    ref = qkv + bias if with_bias else qkv.clone()
    q, k, v = ref[:, :Hq * D], ref[:, Hq * D:(Hq + Hk) * D], ref[:, (Hq + Hk) * D:]
    kernels.rope(q, k, inv, Hq, Hk, D, 0)
    kernels.qkv_prefill(qkv, bias, inv, ck, cv, Hq, Hk, D)
    assert torch.equal(qkv[:, :Hq * D], q)
    assert torch.equal(ck[:, :T], k.reshape(T, Hk, D).transpose(0, 1)) and bool((ck[:, T:] == 5).all())
    assert torch.equal(cv[:, :T], v.reshape(T, Hk, D).transpose(0, 1)) and bool((cv[:, T:] == 5).all())
    with pytest.raises(RuntimeError, match="b2_qkv_prefill failed with code -1"):
        kernels.qkv_prefill(qkv, bias, inv, ck[:, :T - 1].contiguous(), cv, Hq, Hk, D)  # a cache shorter than the prompt


def test_qkv_prefill_refuses_what_it_would_misread(kernels):
    """Everything the kernel takes on trust is checked on the host: it writes the caches by the layout of one of them."""
    T, Hq, Hk, D, L = 8, 4, 2, 64, 16
    W = (Hq + 2 * Hk) * D
    z = lambda *shape, dtype=torch.bfloat16: torch.zeros(*shape, dtype=dtype, device="cuda")
    good = dict(qkv=z(T, W), bias=z(W), inv_freq=z(D // 2, dtype=torch.float32), cache_k=z(Hk, L, D), cache_v=z(Hk, L, D))
    kernels.qkv_prefill(**good, n_heads=Hq, n_kv_heads=Hk, head_dim=D)
    bad = [dict(cache_v=z(Hk, L - 4, D)), dict(cache_v=z(Hk - 1, L, D)), dict(cache_k=z(Hk - 1, L, D), cache_v=z(Hk - 1, L, D)),
           dict(cache_k=z(Hk, L, D // 2), cache_v=z(Hk, L, D // 2)), dict(cache_k=z(Hk, L, D, dtype=torch.float32)),
           dict(cache_v=z(Hk, L, D, dtype=torch.float16)), dict(qkv=z(T, W, dtype=torch.float32)),
           dict(qkv=z(T, W, dtype=torch.float16)), dict(bias=z(W - D)), dict(bias=z(W, dtype=torch.float32)),
           dict(bias=z(2 * W)[::2]), dict(inv_freq=z(D // 4, dtype=torch.float32)), dict(inv_freq=z(D // 2)),
           dict(inv_freq=z(D, dtype=torch.float32)[::2]), dict(cache_v=z(Hk, D, L).transpose(1, 2)), dict(qkv=z(T * W))]
    for change in bad:
        with pytest.raises(AssertionError):
            kernels.qkv_prefill(**{**good, **change}, n_heads=Hq, n_kv_heads=Hk, head_dim=D)
    with pytest.raises(AssertionError):
        kernels.swiglu_blocks(z(2, 33), 8)


@pytest.mark.parametrize("T,I,block", [(1, 16, 16), (3, 48, 8), (129, 1024, 16), (2, 8, 8)])
def test_swiglu_blocks_equals_swiglu(kernels, T, I, block):
    gu = torch.randn(T, 2 * I, device="cuda").to(torch.bfloat16) * 3
    b = gu.view(T, I // block, 2, block)
    want = kernels.swiglu(b[:, :, 0].reshape(T, I).contiguous(), b[:, :, 1].reshape(T, I).contiguous())
    assert torch.equal(kernels.swiglu_blocks(gu, block), want)
    with pytest.raises(RuntimeError, match="b2_swiglu_blocks failed with code -1"):
        kernels.swiglu_blocks(gu, 12)


def _reference_kernels():
    """The reference's own library (its C-ABI source built unchanged for sm_100a by oracle/Makefile) behind this
    repository's binding class: the live checker for the three element-wise operators."""
    import os
    import oracle
    from nanoserve_b200.ops import Kernels
    if not os.path.exists(oracle.REF_LIB_PATH):
        pytest.skip("reference library not built (oracle/_ref/libnanoserve_ref.so)")
    return Kernels(oracle.REF_LIB_PATH)


@pytest.mark.parametrize("T,H", [(1, 3584), (7, 512), (3, 8192)])
def test_rmsnorm_rope_swiglu_against_the_reference_kernels(kernels, T, H):
    """Same inputs through the reference's ns_rmsnorm / ns_rope / ns_swiglu (kernels/fused/*.cuh behind
    csrc/nanoserve_ops.cu:21-45) and through this library's.  Both compute in fp32 and round once to bf16; the
    summation order of the norm's sum of squares differs, so the bound is one bf16 ulp of the value plus 1e-3 absolute;
    the residual stream (bf16(x + r), an exact operation) must be bit-identical."""
    ref = _reference_kernels()
    g = torch.Generator(device="cuda").manual_seed(11)
    x = torch.randn(T, H, device="cuda", generator=g).to(torch.bfloat16)
    r = torch.randn(T, H, device="cuda", generator=g).to(torch.bfloat16)
    w = (1 + 0.1 * torch.randn(H, device="cuda", generator=g)).to(torch.bfloat16)

    def near(a, b):
        a, b = a.float(), b.float()
        return bool(torch.all((a - b).abs() <= torch.maximum(a.abs(), b.abs()) * 2.0**-7 + 1e-3))

    for res in (None, r):
        xa, xb = x.clone(), x.clone()
        ya, yb = kernels.rmsnorm(xa, res, w, 1e-6), ref.rmsnorm(xb, res, w, 1e-6)
        assert near(ya, yb) and torch.equal(xa, xb)
    D, Hq, Hk = 128, H // 128, max(1, H // 512)
    if H % 128 == 0:
        q = torch.randn(T, Hq * D, device="cuda", generator=g).to(torch.bfloat16)
        k = torch.randn(T, Hk * D, device="cuda", generator=g).to(torch.bfloat16)
        inv = 1.0 / (1e6 ** (torch.arange(0, D, 2, device="cuda").float() / D))
        qa, ka, qb, kb = q.clone(), k.clone(), q.clone(), k.clone()
        kernels.rope(qa, ka, inv, Hq, Hk, D, 37)
        ref.rope(qb, kb, inv, Hq, Hk, D, 37)
        assert near(qa, qb) and near(ka, kb)
    a = (3 * torch.randn(T, H, device="cuda", generator=g)).to(torch.bfloat16)
    b = torch.randn(T, H, device="cuda", generator=g).to(torch.bfloat16)
    assert near(kernels.swiglu(a, b), ref.swiglu(a, b))
    torch.cuda.synchronize()


def test_misaligned_pointers_are_refused_not_faulted(kernels):
    """The element-wise kernels move 16 bytes at a time: a view that starts in the middle of a row is refused with -4
    on the host (nothing is launched) instead of faulting on the device."""
    lib = kernels.lib
    t = torch.zeros(4096, dtype=torch.bfloat16, device="cuda")
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    p = t.data_ptr()
    assert lib.ns_rmsnorm(p + 2, None, p, p, 1, 64, 1e-6, st) == -4
    assert lib.ns_rmsnorm(p, p + 4, p, p, 1, 64, 1e-6, st) == -4
    assert lib.ns_swiglu(p, p + 8, p, 1, 64, st) == -4
    assert lib.ns_rope(p + 2, p, p, 1, 1, 1, 64, 0, 64, 64, st) == -4
    assert lib.b2_decode_attention(p + 2, p, p, p, p, p, 4, 2, 128, 16, st) == -4
    torch.cuda.synchronize()
    assert kernels.device_status() == 0


def test_flash_fwd_is_reported_as_not_implemented(kernels):
    q = torch.zeros(64, 128, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(RuntimeError, match="ns_flash_fwd failed with code -3"):
        kernels.flash_attention(q, q, q, 1, 1, 128)


def test_decode_attention_and_rope_kv_store(kernels):
    lib = kernels.lib
    g = torch.Generator(device="cuda").manual_seed(3)
    Hq, Hk, D, L, pos = 8, 2, 128, 64, 37
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    ck = torch.randn(Hk, L, D, device="cuda", generator=g).to(torch.bfloat16)
    cv = torch.randn(Hk, L, D, device="cuda", generator=g).to(torch.bfloat16)
    qkv = torch.randn((Hq + 2 * Hk) * D, device="cuda", generator=g).to(torch.bfloat16)
    bias = (0.1 * torch.randn((Hq + 2 * Hk) * D, device="cuda", generator=g)).to(torch.bfloat16)
    inv = 1.0 / (1e4 ** (torch.arange(0, D, 2, device="cuda").float() / D))
    p = torch.tensor([pos], dtype=torch.int32, device="cuda")
    src = (qkv.float() + bias.float()).to(torch.bfloat16).float().view(Hq + 2 * Hk, D)
    assert lib.b2_rope_kv_store(qkv.data_ptr(), bias.data_ptr(), inv.data_ptr(), p.data_ptr(), ck.data_ptr(),
                                cv.data_ptr(), Hq, Hk, D, L, st) == 0
    fr = pos * inv
    cos, sin = torch.cat([fr, fr]).cos(), torch.cat([fr, fr]).sin()
    rot = src * cos + torch.cat([-src[:, D // 2:], src[:, :D // 2]], -1) * sin
    ref = torch.cat([rot[:Hq + Hk], src[Hq + Hk:]])
    got = qkv.view(Hq + 2 * Hk, D)
    assert close(got, ref)
    assert torch.equal(ck[:, pos], got[Hq:Hq + Hk]) and torch.equal(cv[:, pos], got[Hq + Hk:])
    out = torch.empty(Hq * D, dtype=torch.bfloat16, device="cuda")
    ws = torch.empty(int(lib.b2_decode_workspace_bytes(Hq, D)), dtype=torch.uint8, device="cuda")
    assert lib.b2_decode_attention(qkv.data_ptr(), ck.data_ptr(), cv.data_ptr(), p.data_ptr(), out.data_ptr(),
                                   ws.data_ptr(), Hq, Hk, D, L, st) == 0
    qh = got[:Hq].float()[None, :, None, :]
    ref_o = F.scaled_dot_product_attention(qh, ck[None, :, :pos + 1].float(), cv[None, :, :pos + 1].float(),
                                           enable_gqa=True)
    assert close(out.view(Hq, D), ref_o[0, :, 0])


@pytest.mark.parametrize("Hq,Hk,D,L,pos", [(8, 2, 128, 64, 37), (28, 4, 128, 1024, 0), (28, 4, 128, 1024, 599),
                                            (28, 4, 128, 1024, 1023), (16, 2, 64, 300, 131), (4, 4, 128, 96, 95),
                                            (8, 1, 128, 40, 40)])
def test_fused_attention_equals_the_two_calls(kernels, Hq, Hk, D, L, pos):
    """b2_decode_attention_fused against b2_rope_kv_store + b2_decode_attention on the same inputs: the attention
    output and the appended cache rows must be bit-identical, qkv must be left as it was, and the arrival counters
    must be back at zero (the launch is repeated).  pos == L: the cache is full, nothing is appended."""
    lib = kernels.lib
    g = torch.Generator(device="cuda").manual_seed(100 + pos)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    ck = torch.randn(Hk, L, D, device="cuda", generator=g).to(torch.bfloat16)
    cv = torch.randn(Hk, L, D, device="cuda", generator=g).to(torch.bfloat16)
    qkv = torch.randn((Hq + 2 * Hk) * D, device="cuda", generator=g).to(torch.bfloat16)
    bias = (0.1 * torch.randn((Hq + 2 * Hk) * D, device="cuda", generator=g)).to(torch.bfloat16)
    inv = 1.0 / (1e4 ** (torch.arange(0, D, 2, device="cuda").float() / D))
    p = torch.tensor([pos], dtype=torch.int32, device="cuda")
    # the two-call form on copies
    qkv2, ck2, cv2 = qkv.clone(), ck.clone(), cv.clone()
    out2 = torch.empty(Hq * D, dtype=torch.bfloat16, device="cuda")
    ws2 = torch.empty(int(lib.b2_decode_workspace_bytes(Hq, D)), dtype=torch.uint8, device="cuda")
    assert lib.b2_rope_kv_store(qkv2.data_ptr(), bias.data_ptr(), inv.data_ptr(), p.data_ptr(), ck2.data_ptr(),
                                cv2.data_ptr(), Hq, Hk, D, L, st) == 0
    assert lib.b2_decode_attention(qkv2.data_ptr(), ck2.data_ptr(), cv2.data_ptr(), p.data_ptr(), out2.data_ptr(),
                                   ws2.data_ptr(), Hq, Hk, D, L, st) == 0
    # the fused form, twice
    ws = torch.zeros(int(lib.b2_decode_attention_fused_workspace_bytes(Hq, Hk, D)), dtype=torch.uint8, device="cuda")
    keep = qkv.clone()
    for flags in (1, 1, 0, 2, 3, 4, 6):
        ck1, cv1 = ck.clone(), cv.clone()
        out = torch.full((Hq * D,), 7.0, dtype=torch.bfloat16, device="cuda")
        assert lib.b2_decode_attention_fused(qkv.data_ptr(), bias.data_ptr(), inv.data_ptr(), p.data_ptr(),
                                             ck1.data_ptr(), cv1.data_ptr(), out.data_ptr(), ws.data_ptr(), Hq, Hk, D,
                                             L, None, flags, st) == 0
        torch.cuda.synchronize()
        assert torch.equal(out, out2)
        assert torch.equal(ck1, ck2) and torch.equal(cv1, cv2)
        assert torch.equal(qkv, keep)
        assert int(ws[-4 * Hk:].view(torch.int32).abs().sum()) == 0
    assert kernels.device_status() == 0


# slices of more rows than are staged at a time, the new row in the first and in the last pass; one head to a KV head and eight
@pytest.mark.parametrize("Hq,Hk,D,L,pos", [(8, 2, 128, 2100, 2050), (28, 4, 128, 1100, 1055), (8, 1, 64, 3000, 2999),
                                            (3, 3, 128, 1300, 1024), (16, 2, 64, 1040, 1039), (28, 7, 128, 7000, 6600), (4, 4, 64, 9000, 8800)])
def test_fused_attention_in_several_passes(kernels, Hq, Hk, D, L, pos):
    test_fused_attention_equals_the_two_calls(kernels, Hq, Hk, D, L, pos)


@pytest.mark.parametrize("Hq,Hk,D,flags", [(28, 7, 128, 0), (28, 7, 128, 1), (28, 7, 128, 2), (16, 2, 64, 0), (16, 2, 64, 1)])
def test_fused_attention_appends_the_rows_of_rope_kv_store(kernels, Hq, Hk, D, flags):
    """Key pairs (a, b) whose products cancel in the rotation: which of them is rounded first then shows in one of some 250
    elements, where it shows in one of 2 * 10^5 of ordinary ones."""
    lib, L, half = kernels.lib, 1100, D // 2
    g = torch.Generator(device="cuda").manual_seed(D)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    inv = 1.0 / (1e6 ** (torch.arange(0, D, 2, device="cuda").float() / D))
    ck = torch.zeros(2, Hk, L, D, dtype=torch.bfloat16, device="cuda")
    cv = torch.zeros_like(ck)
    out = torch.empty(Hq * D, dtype=torch.bfloat16, device="cuda")
    ws = torch.zeros(int(lib.b2_decode_attention_fused_workspace_bytes(Hq, Hk, D)), dtype=torch.uint8, device="cuda")
    for pos in range(1, L, 5):
        p = torch.tensor([pos], dtype=torch.int32, device="cuda")
        sn, cs = (pos * inv).double().sin(), (pos * inv).double().cos()
        qkv = torch.randn(Hq + 2 * Hk, D, device="cuda", generator=g).to(torch.bfloat16)
        a = qkv[Hq:Hq + Hk, :half].double()
        first = torch.rand(Hk, half, device="cuda", generator=g) < 0.5  # a cos - b sin vanishes, or b cos + a sin
        qkv[Hq:Hq + Hk, half:] = torch.where(first, a * cs / sn, -a * sn / cs).clamp(-1e4, 1e4).to(torch.bfloat16)
        assert lib.b2_decode_attention_fused(qkv.data_ptr(), None, inv.data_ptr(), p.data_ptr(), ck[0].data_ptr(),
                                             cv[0].data_ptr(), out.data_ptr(), ws.data_ptr(), Hq, Hk, D, L, None, flags, st) == 0
        assert lib.b2_rope_kv_store(qkv.data_ptr(), None, inv.data_ptr(), p.data_ptr(), ck[1].data_ptr(), cv[1].data_ptr(),
                                    Hq, Hk, D, L, st) == 0
    assert torch.equal(ck[0], ck[1]) and torch.equal(cv[0], cv[1]) and bool(ck[0].any())
    assert kernels.device_status() == 0


@pytest.mark.parametrize("Hq,Hk,D,one", [(28, 4, 128, True), (7, 1, 64, True), (64, 32, 128, False), (40, 40, 64, False),
                                         (32, 8, 128, None), (28, 7, 128, None)])
def test_attention_in_one_launch_equals_two(kernels, Hq, Hk, D, one):
    """The form that plain flags take against the two launches, to the bit, over a thousand positions; it is the one in clusters,
    which leaves the workspace alone, only where all its clusters run at once (32 clusters of sixteen never do)."""
    lib, L = kernels.lib, 1000
    g = torch.Generator(device="cuda").manual_seed(Hq)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=g).to(torch.bfloat16)
    inv = 1.0 / (1e6 ** (torch.arange(0, D, 2, device="cuda").float() / D))
    caches = rand(2, Hk, L, D)[None].repeat(2, 1, 1, 1, 1)
    bias, outs = 0.1 * rand((Hq + 2 * Hk) * D), torch.empty(2, Hq * D, dtype=torch.bfloat16, device="cuda")
    ws = torch.zeros(int(lib.b2_decode_attention_fused_workspace_bytes(Hq, Hk, D)), dtype=torch.uint8, device="cuda")
    for pos in range(0, L, 7):
        p, qkv = torch.tensor([pos], dtype=torch.int32, device="cuda"), rand((Hq + 2 * Hk) * D)
        for i, flags in enumerate((2 * (pos & 1), 4 + 2 * (pos & 1))):
            ws[:-4 * Hk] = 0xA5
            assert lib.b2_decode_attention_fused(qkv.data_ptr(), bias.data_ptr(), inv.data_ptr(), p.data_ptr(),
                                                 caches[i, 0].data_ptr(), caches[i, 1].data_ptr(), outs[i].data_ptr(),
                                                 ws.data_ptr(), Hq, Hk, D, L, None, flags, st) == 0
            untouched = bool((ws[:-4 * Hk] == 0xA5).all())
            assert untouched == (one if i == 0 and one is not None else untouched and i == 0)
        assert torch.equal(outs[0], outs[1])
    assert torch.equal(caches[0], caches[1])
    assert kernels.device_status() == 0


FIRST_CALL = """
import sys, torch
from nanoserve_b200.ops import Kernels
lib = (k := Kernels(sys.argv[1])).lib
Hq, Hk, D, L = 28, 4, 128, 64
z = lambda *shape, t=torch.bfloat16: torch.zeros(*shape, dtype=t, device="cuda")
qkv, ck, cv, out, inv, p = z((Hq + 2 * Hk) * D), z(Hk, L, D), z(Hk, L, D), z(Hq * D), z(D // 2, t=torch.float32), z(1, t=torch.int32)
ws = z(lib.b2_decode_attention_fused_workspace_bytes(Hq, Hk, D), t=torch.uint8)
def run():
    assert lib.b2_decode_attention_fused(qkv.data_ptr(), None, inv.data_ptr(), p.data_ptr(), ck.data_ptr(), cv.data_ptr(),
                                         out.data_ptr(), ws.data_ptr(), Hq, Hk, D, L, None, 0, k._stream()) == 0
def untouched(go):
    ws[:-4 * Hk] = 0xA5
    go()
    return bool((ws[:-4 * Hk] == 0xA5).all())
graph = torch.cuda.CUDAGraph()
torch.cuda.synchronize()
with torch.cuda.graph(graph):
    run()
assert not untouched(graph.replay) and not untouched(run)
k.init()
assert untouched(run) and not untouched(graph.replay) and lib.b2_device_status() == 0
"""


def test_attention_as_the_first_call(lib_path):
    """The form whose waits may give up runs only where the status word that records it exists: a first call, captured or not,
    takes the two launches, which write to the workspace."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    res = subprocess.run([sys.executable, "-c", FIRST_CALL, lib_path], cwd=root, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr


def test_greedy_next(kernels):
    lib = kernels.lib
    V, H = 152064, 64
    g = torch.Generator(device="cuda").manual_seed(4)
    logits = torch.randn(V, device="cuda", generator=g).to(torch.bfloat16)
    logits[777] = 50.0
    logits[90000] = 50.0  # tie: the lower index wins, as torch.argmax on the first occurrence
    embed = torch.randn(V, H, device="cuda", generator=g).to(torch.bfloat16)
    pos = torch.tensor([11], dtype=torch.int32, device="cuda")
    step = torch.tensor([2], dtype=torch.int32, device="cuda")
    toks = torch.zeros(8, dtype=torch.int64, device="cuda")
    x = torch.zeros(H, dtype=torch.bfloat16, device="cuda")
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    ws = torch.empty(int(lib.b2_decode_workspace_bytes(28, 128)), dtype=torch.uint8, device="cuda")
    assert lib.b2_greedy_next(logits.data_ptr(), V, embed.data_ptr(), H, pos.data_ptr(), toks.data_ptr(),
                              step.data_ptr(), x.data_ptr(), ws.data_ptr(), st) == 0
    torch.cuda.synchronize()
    assert int(toks[2]) == 777 and int(pos) == 12 and int(step) == 3 and torch.equal(x, embed[777])


# one CTA per tile and pairs of them, tiles cut along K with ragged tokens, the few-token kernel, a GEMV; a tile of rows less a block
@pytest.mark.parametrize("M,N,K,flags", [(100, 512, 1024, FLAG_GEMM_WIDE), (300, 1504, 2048, FLAG_GEMM_WIDE),
                                         (300, 736, 8192, FLAG_GEMM_WIDE | FLAG_GEMM_NO_PAIRS), (513, 32, 512, FLAG_GEMM_WIDE),
                                         (700, 4096, 1024, 0), (48, 1024, 1024, 0), (5, 1024, 1024, 0)])
def test_linear_swiglu_equals_its_parts(kernels, M, N, K, flags):
    gen = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)
    Wq = torch.randint(-2**31, 2**31 - 1, (N, K // 8), dtype=torch.int32, device="cuda", generator=gen)
    S = (0.005 + (torch.randn(N, K // 128, device="cuda", generator=gen) * 0.01).abs()).to(torch.bfloat16)
    want = kernels.swiglu_blocks(kernels.w4_linear(x, Wq, S, flags=flags), 16)
    assert torch.equal(kernels.w4_linear_swiglu(x, Wq, S, flags=flags), want)
    with pytest.raises(RuntimeError, match="b2_w4_linear_swiglu failed with code -1"):
        kernels.w4_linear_swiglu(x, Wq[:N - 16].contiguous(), S[:N - 16].contiguous(), flags=flags)
    assert kernels.device_status() == 0
