"""The native call path of bound layers: what it serves itself and what it hands to the Python callable."""

from __future__ import annotations

import copy
import gc
import weakref

import pytest
import torch

from conftest import seeded
from xqt_b200 import native, quantize
from xqt_b200.errors import CudaCallError, XQTBackendError
from xqt_b200.modules import AWQW4A16Linear
from xqt_b200.ops import w8a8
from xqt_b200.ops.mlp import W4A16SwiGLUMLP
from xqt_b200.ops.w4a16 import bind_w4a16_decode, bind_w4a16_linear, prepare_decode, w4a16_linear

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def _layer(n, k, seed):
    return quantize.quantize_w4_asymmetric((torch.randn((n, k), generator=seeded(seed)) * 0.02).to(DEV), group_size=128)


@pytest.mark.parametrize("m", [1, 16])
def test_decode_call_forms(m):
    n, k = 264, 256
    w = _layer(n, k, 1)
    run = bind_w4a16_decode(prepare_decode(w.qweight, w.scales, w.zero_points, group_size=128, nibble_signed=False), rows=m, dtype=torch.bfloat16)
    x = torch.randn((m, k), generator=seeded(2)).to(DEV, torch.bfloat16)
    residual = torch.randn((m, n), generator=seeded(3)).to(DEV, torch.bfloat16)
    plain = run(x)
    out = torch.empty_like(plain)
    assert run(x, out) is out and torch.equal(out, plain)
    assert torch.equal(run(x, out=out), plain) and torch.equal(run(x, None, residual), run.slow(x, None, residual))
    other = torch.cuda.Stream(DEV)
    other.wait_stream(torch.cuda.current_stream(DEV))
    with torch.cuda.stream(other):
        again = run(x)
    torch.cuda.current_stream(DEV).wait_stream(other)
    assert torch.equal(again, plain)
    for bad in (x.to(torch.float16), x[:, :128], x.cpu(), torch.empty((m + 1, k), device=DEV, dtype=torch.bfloat16),
                torch.empty((k, m), device=DEV, dtype=torch.bfloat16).t()[:, :k] if m > 1 else x.reshape(1, 1, k)):
        with pytest.raises(XQTBackendError):
            run(bad)
    for bad_out in (torch.empty((m, n + 8), device=DEV, dtype=torch.bfloat16), torch.empty((m, n), device=DEV)):
        with pytest.raises(XQTBackendError):
            run(x, bad_out)
    with pytest.raises(XQTBackendError):
        run(x, None, residual.to(torch.float16))


def test_leading_dimensions_and_lifetime():
    n, k, m = 256, 512, 6
    codes, scale = quantize.quantize_w8_per_channel(torch.randn((n, k), generator=seeded(4)).to(DEV))
    run = w8a8.bind_convrot_w8a8_linear(w8a8.pack_convrot_w8a8_linear(codes.t().contiguous(), scale), rows=m)
    x = torch.randn((2, 3, k), generator=seeded(5)).to(DEV, torch.bfloat16)
    assert tuple(run(x).shape) == (2, 3, n) and torch.equal(run(x).reshape(m, n), run(x.reshape(m, k)))
    # a block that has bound its calls is freed with its last reference, without the garbage collector's help
    block = W4A16SwiGLUMLP(_layer(256, 256, 6), _layer(256, 256, 7), _layer(256, 256, 8), device=DEV)
    y = torch.randn((40, 256), generator=seeded(9)).to(DEV, torch.bfloat16)
    for rows in (1, 17, 40):
        assert torch.equal(block(y[:rows]), block._forward(y[:rows]))
    gone = weakref.ref(block)
    gc.disable()
    try:
        del block
        assert gone() is None
    finally:
        gc.enable()


def test_errors_keep_their_types():
    n, k = 256, 512
    w = _layer(n, k, 10)
    run = bind_w4a16_decode(prepare_decode(w.qweight, w.scales, w.zero_points, group_size=128, nibble_signed=False), rows=2, dtype=torch.bfloat16)
    x = torch.randn((2, k), generator=seeded(11)).to(DEV, torch.bfloat16)
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode():
        fake = torch.empty((2, k), device=DEV, dtype=torch.bfloat16)
    with pytest.raises((RuntimeError, CudaCallError)):        # no data: torch or the library refuses the pointer
        run(fake)
    # an output of 8 TiB: the error is torch's own, as from torch.empty
    big = native.host().Bound(((2, 2, (), (), 0, 0),), run.slow, None, torch.bfloat16, torch.bfloat16, 0, 2, k, 1 << 41)
    with pytest.raises(torch.OutOfMemoryError):
        big(x)
    assert torch.equal(run(x), run.slow(x))


def _bound_gemm(rows, n, k, seed):
    w = _layer(n, k, seed)
    return bind_w4a16_linear(w.qweight, w.scales, w.zero_points, rows=rows, dtype=torch.bfloat16, group_size=128, nibble_signed=False, variant="tcgen05")


def test_workspace_is_the_pools_current_one():
    """Calls bound before the pool has grown report into the buffer that ``workspace_status`` reads, and the buffer before
    it is released."""
    k = 512
    stream = torch.cuda.Stream(DEV)
    with torch.cuda.stream(stream):
        small, x = _bound_gemm(40, 256, k, 20), torch.randn((40, k), generator=seeded(21)).to(DEV, torch.bfloat16)
        want = small(x)
        key = (0, native.stream_handle(DEV), "run")
        before = weakref.ref(native._workspaces[key])
        size = before().numel()
        large = _bound_gemm(64, 1024 + size // (2 * k), k, 22)
        large(torch.randn((64, k), generator=seeded(23)).to(DEV, torch.bfloat16))
        assert before() is None and native._workspaces[key].numel() > size
        assert torch.equal(small(x), want) and native.workspace_status(DEV) == 0
        small(x * 2.0 ** 20)                                   # beyond fp16's range: clamped and reported
        assert native.workspace_status(DEV) == 256
        native._workspaces[key][:4].zero_()
        stream.synchronize()


def test_workspace_of_a_captured_graph_outlives_its_replacement():
    k = 512
    stream = torch.cuda.Stream(DEV)
    with torch.cuda.stream(stream):
        run, x = _bound_gemm(40, 256, k, 24), torch.randn((40, k), generator=seeded(25)).to(DEV, torch.bfloat16)
        want = run(x)
        key = (0, native.stream_handle(DEV), "run")
        used = weakref.ref(native._workspaces[key])
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            got = run(x)
        size = used().numel()
        assert native.workspace(DEV, size + 1).numel() >= 2 * size and used() is not None
        filler = [torch.full((size // 4,), float("nan"), device=DEV) for _ in range(4)]      # would take its memory
        got.zero_()
        graph.replay()
        assert torch.equal(got, want) and len(filler) == 4
        assert native.workspace_status(DEV) == 0
        stream.synchronize()


def test_one_bound_layer_serves_every_row_count():
    """Row counts in any order through one bound call per layer; growing counts leave nothing behind but the pool's buffer."""
    n, k = 768, 512
    module = AWQW4A16Linear(_layer(n, k, 30), bias=torch.randn((n,), generator=seeded(31)).to(DEV)).eval()
    blocks = [W4A16SwiGLUMLP(_layer(640, k, 32), _layer(640, k, 33), _layer(k, 640, 34), device=DEV)]
    odd = [type(w)(qweight=w.qweight, scales=w.scales, zero_points=w.zero_points + 0.25, metadata=w.metadata) for w in (_layer(640, k, 32), _layer(640, k, 33), _layer(k, 640, 34))]
    blocks.append(W4A16SwiGLUMLP(*odd, device=DEV))                # zero points that are no integers: two passes
    x = torch.randn((700, k), generator=seeded(35)).to(DEV, torch.bfloat16)
    assert module(x[:0]).shape == (0, n)
    for m in (1, 17, 300, 16, 32, 33, 128, 129, 40, 600, 2, 18, 300, 700):
        for layer, general in ((module, module._forward_flat), *((block, block._forward) for block in blocks)):
            got, want = layer(x[:m]), general(x[:m])
            assert got.shape == want.shape
            # the general form of the integer blocks sums the down projection the same way, gating apart: two roundings may differ
            assert torch.equal(got, want) if layer is module or m <= 128 else (got - want).norm() <= 4e-3 * want.norm()
    assert len(module._gemm) == 1 and len(blocks[0]._decode) == 2
    kept = {id(module._gemm[torch.bfloat16][2]), *(id(run) for block in blocks for run in (*block._decode.values(), block._gemm[1]))}
    first = W4A16SwiGLUMLP(_layer(640, k, 32), _layer(640, k, 33), _layer(k, 640, 34), device=DEV)
    for m in (300, 64, 300, 33, 400):                              # the single library call first, then the separate launches
        assert torch.equal(first(x[:m]), blocks[0](x[:m]))
    with pytest.raises(XQTBackendError):
        first(x[:300, :128])
    baseline = None
    for m in range(17, 700, 3):
        module(x[:m]), blocks[0](x[:m])
        baseline = torch.cuda.memory_allocated() if m == 200 else baseline
    # one buffer of the pool: the activations' copies grow with the rows, sizes by an eighth at a time
    assert torch.cuda.memory_allocated() - baseline <= 1.25 * native._workspaces[(0, native.stream_handle(DEV), "run")].numel()
    assert kept == {id(module._gemm[torch.bfloat16][2]), *(id(run) for block in blocks for run in (*block._decode.values(), block._gemm[1]))}
    module.cpu()
    assert not module._gemm


def test_weights_first_seen_inside_a_graph_capture():
    """Whether the zero points are integers takes a device-to-host copy, which a capture cannot hold: such a call takes the two
    passes, which serve any zero point, and is captured."""
    n, k, m = 24576, 1024, 600
    w = _layer(n, k, 40)
    x = torch.randn((m, k), generator=seeded(41)).to(DEV, torch.bfloat16)
    want = w4a16_linear(x, w.qweight, w.scales, w.zero_points.clone(), group_size=128, nibble_signed=False, variant="tcgen05")
    module = AWQW4A16Linear(w).eval()
    stream, graph = torch.cuda.Stream(DEV), torch.cuda.CUDAGraph()
    stream.wait_stream(torch.cuda.current_stream(DEV))
    with torch.cuda.graph(graph, stream=stream):
        one = module(x)
        two = w4a16_linear(x, w.qweight, w.scales, w.zero_points.clone(), group_size=128, nibble_signed=False)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(one, want) and torch.equal(two, want)
    # and the small layer that never asks: above 512 rows two passes whatever its zero points are
    small = AWQW4A16Linear(_layer(256, k, 42)).eval()
    stream.wait_stream(torch.cuda.current_stream(DEV))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        one = small(x)
    graph.replay()
    torch.cuda.synchronize()
    assert small._gemm[torch.bfloat16][3] is None and torch.equal(small(x), one)
    want_small = w4a16_linear(x[:300], small.canonical_qweight, small.weight_scale, small.weight_zero_point, group_size=128, nibble_signed=False)
    assert torch.equal(small(x[:300]), want_small) and small._gemm[torch.bfloat16][3] is True
    assert torch.equal(module(x), w4a16_linear(x, w.qweight, w.scales, w.zero_points, group_size=128, nibble_signed=False, variant="tcgen05_fused"))


def test_copies_and_saved_layers(tmp_path):
    """A layer that has run can be copied and saved; what comes back is a layer of its own."""
    n, k = 256, 512
    module = AWQW4A16Linear(_layer(n, k, 50), bias=torch.randn((n,), generator=seeded(51)).to(DEV)).eval()
    frozen = AWQW4A16Linear(_layer(n, k, 52)).eval()
    frozen.freeze_native_inference(device=DEV, dtype=torch.bfloat16, rows=(1,))
    block = W4A16SwiGLUMLP(_layer(256, k, 53), _layer(256, k, 54), _layer(k, 256, 55), device=DEV)
    x = torch.randn((300, k), generator=seeded(56)).to(DEV, torch.bfloat16)
    sizes = (1, 16, 20, 40, 300)
    want, want_block, want_frozen = [module(x[:m]) for m in sizes], [block(x[:m]) for m in sizes], frozen(x[:1])
    block.gate_up.gated(x[:4])
    torch.save((module, frozen, block), tmp_path / "layers.pt")
    for other, other_frozen, other_block in (copy.deepcopy((module, frozen, block)), torch.load(tmp_path / "layers.pt", weights_only=False)):
        assert other._execution_weight is not module._execution_weight and not other._bound and not other_block._decode
        assert all(torch.equal(other(x[:m]), y) for m, y in zip(sizes, want))
        assert all(torch.equal(other_block(x[:m]), y) for m, y in zip(sizes, want_block))
        assert torch.equal(other_frozen(x[:1]), want_frozen)
        with pytest.raises(RuntimeError):
            other_frozen(x[:2])
        other.weight_scale.zero_()                          # its own scales
        other_block.down.scales.zero_()
        assert not other_block(x[:40]).any() and torch.equal(other(x[:40]), other.bias.to(torch.bfloat16).expand(40, n))
        assert torch.equal(module(x[:40]), want[3]) and torch.equal(block(x[:40]), want_block[3])
    # saved before the present fields existed
    old, old_block = module.__getstate__(), block.__getstate__()
    for name in ("_gemm", "_decode", "_can_bind", "_fuse_gating"):
        old.pop(name, None), old_block.pop(name, None)
    old["_last_execution"] = {"implementation": "not_run", "native": False}
    for kind, state, y in ((AWQW4A16Linear, old, want), (W4A16SwiGLUMLP, old_block, want_block)):
        back = kind.__new__(kind)
        back.__setstate__(state)
        assert torch.equal(back(x[:300]), y[4]) and torch.equal(back(x[:1]), y[0])
    run = module.bind(rows=1, dtype=torch.bfloat16)
    run.note = "attributes and weak references, as the closures took them"
    assert copy.deepcopy(run) is run and weakref.ref(run)() is run and run.note
    for wrong in ("delattr(run, 'slow')", "setattr(run, 'slow', 3)", "delattr(run, 'keep')"):
        with pytest.raises((TypeError, AttributeError)):
            eval(wrong)
