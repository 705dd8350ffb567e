"""The native host side of w4_linear and w4_quantize hands everything that is not a plain call on CUDA tensors back to the
ctypes path, which answers as ever; on CUDA tensors both give the same bits, for outputs given or not, strided inputs and flags."""
import shutil

import pytest
import torch
import torch.autograd.forward_ad as fwAD
from torch._subclasses.fake_tensor import FakeTensorMode
from torch.overrides import TorchFunctionMode
from torch.utils._python_dispatch import TorchDispatchMode

from nanoserve_b200 import ops


@pytest.fixture
def call(lib_path):
    """The extension, built with the library on demand; missing only where there is no g++ to build it."""
    if not ops._find_call():
        if shutil.which("g++"):
            pytest.fail("nanoserve_call.so was not built or does not load")
        pytest.skip("no g++ to build the extension")


def test_hands_back_what_it_does_not_take(call):
    x = torch.zeros(2, 256, dtype=torch.bfloat16)
    for args in [(), (1,), (1, x, x, x, 128, 0, None), (1, None, x, x, 128, 0, None), (1, x, x, x, 128.0, 0, None),
                 (1, x, x, x, 1 << 40, 0, None), (1, x, x, x, 128, 0, 3)]:
        assert ops._call_linear(*args) is NotImplemented
    for args in [(), (1, x, 128), (1, x, 0), (1, None, 128), (1, x, 128.0)]:
        assert ops._call_quantize(*args) is NotImplemented


@pytest.mark.gpu
def test_same_answers_as_through_ctypes(kernels, call):
    g = torch.Generator(device="cuda").manual_seed(1)
    N, K = 300, 1024
    wq = torch.randint(-2**31, 2**31 - 1, (N, K // 8), dtype=torch.int32, device="cuda", generator=g)
    s = torch.rand(N, K // 128, device="cuda", generator=g).to(torch.bfloat16)
    slow = ops.Kernels()
    slow._linear = slow._quantize = None
    assert kernels._linear is not None and kernels._quantize is not None
    wide = torch.randn(5, 2 * K, device="cuda", generator=g).to(torch.bfloat16)
    for group in (128, 64):
        for W in (wide[:, :K], wide.contiguous()):
            for a, b in zip(kernels.w4_quantize(W, group), slow.w4_quantize(W, group)):
                assert torch.equal(a, b) and a.dtype == b.dtype and a.shape == b.shape
    for x in (wide[:, :K], wide[:1, :K].contiguous(), wide[:4, K:], torch.nn.Parameter(wide[:2, :K].clone())):
        for flags in (0, ops.FLAG_RING_KERNEL, ops.FLAG_DECODE_NARROW):
            want = slow.w4_linear(x, wq, s, 128, flags=flags)
            got = kernels.w4_linear(x, wq, s, 128, flags=flags)
            assert torch.equal(got, want) and got.dtype == torch.bfloat16 and not got.requires_grad
        out = torch.empty(x.shape[0], N, dtype=torch.bfloat16, device="cuda")
        assert kernels.w4_linear(x, wq, s, out=out) is out and torch.equal(out, slow.w4_linear(x, wq, s))
    pinned = torch.empty(1, N, dtype=torch.bfloat16, pin_memory=True)
    assert kernels.w4_linear(wide[:1, :K], wq, s, out=pinned) is pinned
    torch.cuda.synchronize()
    assert torch.equal(pinned.cuda(), slow.w4_linear(wide[:1, :K], wq, s))


@pytest.mark.gpu
def test_errors_and_streams(kernels, call):
    wq = torch.zeros(64, 32, dtype=torch.int32, device="cuda")
    s = torch.ones(64, 2, dtype=torch.bfloat16, device="cuda")
    x = torch.ones(1, 256, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(RuntimeError, match="ns_w4_linear failed with code -1"):
        kernels.w4_linear(x, wq, s, group=96)
    with pytest.raises(RuntimeError, match="ns_w4_quantize failed with code -1"):
        kernels.w4_quantize(x, 96)
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        kernels.w4_quantize(x.cpu())
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        kernels.w4_linear(x.cpu(), wq, s)
    with pytest.raises(ValueError):
        kernels.w4_linear(x[0], wq, s)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):  # captured on the stream that is current
        kernels.w4_linear(x, wq, s)
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            y = kernels.w4_linear(x, wq, s)
    x.fill_(2.0)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, kernels.w4_linear(x, wq, s))


@pytest.mark.gpu
def test_hands_back_cuda_calls_that_are_not_plain(kernels, call):
    """On CUDA tensors, so that nothing but the subclass, the mode or the transform is the reason; the call through ctypes then
    answers or refuses as it does without the extension."""
    g = torch.Generator(device="cuda").manual_seed(2)
    N, K = 96, 512
    wq = torch.randint(-2**31, 2**31 - 1, (N, K // 8), dtype=torch.int32, device="cuda", generator=g)
    s = torch.rand(N, K // 128, device="cuda", generator=g).to(torch.bfloat16)
    x = torch.randn(3, K, device="cuda", generator=g).to(torch.bfloat16)
    out = torch.empty(3, N, dtype=torch.bfloat16, device="cuda")
    linear = lambda *a: ops._call_linear(kernels._linear, *a[:3], 128, 0, a[3] if len(a) > 3 else None)
    quantize = lambda w: ops._call_quantize(kernels._quantize, w, 128)
    want, want_q = linear(x, wq, s), quantize(x)
    assert isinstance(want, torch.Tensor) and torch.equal(want_q[0], kernels.w4_quantize(x)[0])
    assert linear(x[0], wq, s) is NotImplemented and quantize(x[0]) is NotImplemented

    class Sub(torch.Tensor):
        pass

    for i in range(4):
        args = [x, wq, s, out]
        args[i] = args[i].as_subclass(Sub)
        assert linear(*args) is NotImplemented
        assert torch.equal(kernels.w4_linear(*args[:3], out=args[3]), want)
    assert quantize(x.as_subclass(Sub)) is NotImplemented

    seen = []

    class Dispatch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    class Function(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(getattr(func, "__name__", str(func)))
            return func(*args, **(kwargs or {}))

    for mode in (Dispatch(), Function(), torch.device("cpu")):
        seen.clear()
        with mode:
            assert linear(x, wq, s) is NotImplemented and quantize(x) is NotImplemented
            got = kernels.w4_linear(x, wq, s)
        assert got.is_cuda and torch.equal(got, want)
        assert isinstance(mode, torch.device) or any("empty" in name for name in seen)  # the mode sees the allocation
    with FakeTensorMode(allow_non_fake_inputs=True):
        assert linear(x, wq, s) is NotImplemented

    def mapped(v):
        assert linear(v, wq, s) is NotImplemented and linear(x, wq, s) is NotImplemented
        assert quantize(v) is NotImplemented
        with pytest.raises(RuntimeError):  # a batched tensor has no data pointer
            kernels.w4_linear(v, wq, s)
        return v

    torch.func.vmap(mapped)(torch.stack([x, x]))
    assert torch.equal(linear(x, wq, s), want)


@pytest.mark.gpu
def test_grad_modes(kernels, call):
    """Calls under inference mode or with a tangent are taken: the outputs are what the call through ctypes makes of them."""
    wq = torch.full((64, 32), 0x12345678, dtype=torch.int32, device="cuda")
    s = torch.ones(64, 2, dtype=torch.bfloat16, device="cuda")
    x = torch.ones(1, 256, dtype=torch.bfloat16, device="cuda", requires_grad=True)
    slow = ops.Kernels()
    slow._linear = slow._quantize = None
    assert ops._call_linear(kernels._linear, x, wq, s, 128, 0, None) is not NotImplemented
    with torch.inference_mode():
        a, b = kernels.w4_linear(x, wq, s), slow.w4_linear(x, wq, s)
        assert a.is_inference() and b.is_inference() and torch.equal(a, b)
    with fwAD.dual_level():
        dual = fwAD.make_dual(x.detach(), torch.ones_like(x))
        a, b = kernels.w4_linear(dual, wq, s), slow.w4_linear(dual, wq, s)
        assert fwAD.unpack_dual(a).tangent is None and fwAD.unpack_dual(b).tangent is None and torch.equal(a, b)
    assert not kernels.w4_linear(x, wq, s).requires_grad
