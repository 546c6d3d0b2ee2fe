"""SVDQuant W8A8 (int8 x int8 GEMM + low-rank branch) against its CPU oracle."""

from __future__ import annotations

import pytest
import torch

from conftest import seeded
from oracle import svdq_w8a8 as oracle
from oracle import w4a16 as o16

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def _layer(n, k, rank, seed, dtype):
    w = (torch.randn((n, k), generator=seeded(seed)) * 0.02).to(dtype)
    w[3] = 0                                                  # a zero row: scale 1, codes 0
    down = (torch.randn((rank, k), generator=seeded(seed + 1)) * 0.05).to(dtype) if rank else None
    up = (torch.randn((n, rank), generator=seeded(seed + 2)) * 0.05).to(dtype) if rank else None
    return w, down, up


@pytest.mark.parametrize("m,n,k,rank,dtype", [(1, 256, 512, 16, torch.bfloat16), (130, 264, 1024, 32, torch.bfloat16),
                                              (300, 512, 4096, 8, torch.float16), (64, 128, 256, 0, torch.bfloat16)])
def test_svdq_w8a8_forward(m, n, k, rank, dtype):
    from xqt_b200 import native
    from xqt_b200.ops.svdq_w8a8 import pack_svdq_w8a8_linear, svdq_w8a8_linear, w8a8_linear
    w, down, up = _layer(n, k, rank, 40 + n, dtype)
    bias = torch.randn((n,), generator=seeded(5))
    x = torch.randn((m, k), generator=seeded(m)).to(dtype)
    x[m // 2] = 0                                             # an all-zero token: scale 0, codes 0, output = bias
    packed = pack_svdq_w8a8_linear(w.to(DEV), None if down is None else down.to(DEV), None if up is None else up.to(DEV), bias.to(DEV))
    q_w, s_w = oracle.quantize_weight(w)
    assert torch.equal(packed.qweight.cpu(), q_w) and torch.equal(packed.weight_scales.cpu(), s_w)
    out, parts = svdq_w8a8_linear(x.to(DEV), packed, lora_scale=0.5, return_parts=True)
    ref, rparts = oracle.forward(x, q_w, s_w, down, up, bias, lora_scale=0.5, return_parts=True)
    assert torch.equal(parts["codes"].cpu(), rparts["q_a"])          # bit-exact codes and scales
    assert torch.equal(parts["scales"].cpu(), rparts["s_a"])
    assert o16.rel_l2(out.cpu(), ref) <= 1e-3
    plain = w8a8_linear(x.to(DEV), packed)
    assert o16.rel_l2(plain.cpu(), oracle.forward(x, q_w, s_w, None, None, bias)) <= 1e-3
    assert native.workspace_status(DEV) == 0


def test_bound_call_reuses_its_workspace():
    from xqt_b200.ops.svdq_w8a8 import allocate_svdq_w8a8_workspace, bind_svdq_w8a8_linear, pack_svdq_w8a8_linear, svdq_w8a8_linear
    m, n, k, rank = 96, 384, 768, 32
    w, down, up = _layer(n, k, rank, 9, torch.bfloat16)
    packed = pack_svdq_w8a8_linear(w.to(DEV), down.to(DEV), up.to(DEV))
    x = torch.randn((m, k), generator=seeded(2)).to(torch.bfloat16).to(DEV)
    ws = allocate_svdq_w8a8_workspace(m, packed)
    bound = bind_svdq_w8a8_linear(packed, ws, rows=m)
    assert torch.equal(bound(x), svdq_w8a8_linear(x, packed))
    with pytest.raises(Exception):
        bound(x[:10])


def test_workspace_fields_and_inputs_at_any_address():
    from xqt_b200.errors import XQTBackendError
    from xqt_b200.ops import svdq_w8a8 as op
    m, n, k = 20, 264, 512
    w, down, up = _layer(n, k, 16, 70, torch.bfloat16)
    packed, plain = op.pack_svdq_w8a8_linear(w.to(DEV), down.to(DEV), up.to(DEV)), op.pack_svdq_w8a8_linear(w.to(DEV), None, None)
    x = torch.randn((m, k), generator=seeded(71)).to(DEV, torch.bfloat16)
    odd = torch.empty(m * k + 1, device=DEV, dtype=torch.bfloat16)[1:].view(m, k).copy_(x)        # two bytes past a 16-byte boundary
    want, want_plain = op.svdq_w8a8_linear(x, packed), op.w8a8_linear(x, packed)
    assert torch.equal(op.w8a8_linear(odd, packed), want_plain) and torch.equal(op.svdq_w8a8_linear(odd, plain), op.svdq_w8a8_linear(x, plain))
    assert torch.equal(op.bind_svdq_w8a8_linear(plain, rows=m)(odd), op.svdq_w8a8_linear(x, plain))
    # the workspace by its fields, as callers build it
    ws = op.allocate_svdq_w8a8_workspace(m, packed)
    assert tuple(ws.lora_activation.shape) == (m, 32) and tuple(ws.low_rank_output.shape) == (m, n)
    assert ws.lora_activation.dtype == ws.low_rank_output.dtype == torch.float32 and ws.low_rank_output is ws.low_rank_output
    again = op.W8A8SVDQWorkspace(ws.quantized_activation, ws.activation_scales, ws.lora_activation, ws.lora_activation16, ws.low_rank_output)
    assert torch.equal(op.svdq_w8a8_linear(x, packed, workspace=again), want)
    other = op.allocate_svdq_w8a8_workspace(m, op.pack_svdq_w8a8_linear(w[:128].contiguous().to(DEV), down.to(DEV), up[:128].to(DEV)))
    with pytest.raises(ValueError):
        op.svdq_w8a8_linear(x, packed, workspace=other)                      # another layer's N
    for field, wrong in (("quantized_activation", ws.quantized_activation.float()), ("activation_scales", ws.activation_scales.half()),
                         ("activation_scales", ws.activation_scales[: m // 2]), ("quantized_activation", torch.empty((k, m), device=DEV, dtype=torch.int8).t())):
        bad = op.W8A8SVDQWorkspace(**{**ws.__dict__, field: wrong})
        with pytest.raises((XQTBackendError, ValueError)):
            op.svdq_w8a8_linear(x, packed, workspace=bad)
        with pytest.raises((XQTBackendError, ValueError)):
            op.bind_svdq_w8a8_linear(packed, bad, rows=m)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_up_projection_entry(dtype):
    """``xqt_b200_lowrank_up``, the fp32 product of a caller's own low-rank activations."""
    from xqt_b200 import native
    m, n = 130, 264
    la, up = (torch.randn(s, generator=seeded(sum(s))).to(DEV, dtype) for s in ((m, 64), (n, 64)))
    out, scratch = torch.empty((m, n), device=DEV), native.workspace(DEV, 256, "gemm")
    native.check(native.library().xqt_b200_lowrank_up(la.data_ptr(), up.data_ptr(), out.data_ptr(), m, n, 64, native.DTYPE_CODE[dtype], scratch.data_ptr(),
                                                      scratch.numel(), native.stream_handle(DEV)), "xqt_b200_lowrank_up")
    # exact products, 64 of them summed in fp32: 2^-24 of the partial sums for each addition
    assert ((out.double() - la.double() @ up.double().t()).abs() <= 64 * 2.0 ** -24 * (la.double().abs() @ up.double().abs().t())).all()
