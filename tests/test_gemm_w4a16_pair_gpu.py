"""The CTA-pair W4A16 GEMM at the edges of its tiles, chunks and K splits, against the two-pass form: both multiply the same
fp16 operands, so only the order of the fp32 sums differs."""

from __future__ import annotations

import pytest
import torch

from conftest import seeded
from xqt_b200 import native, quantize
from xqt_b200.ops.mlp import W4A16SwiGLUMLP
from xqt_b200.ops.w4a16 import w4a16_linear

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("m,n,k,group", [
    (129, 8, 64, 64), (256, 72, 1024, 64), (257, 264, 576, 64), (300, 4096, 4096, 128), (512, 1000, 14336, 128),
    (513, 4104, 640, 128), (1000, 12288, 2048, 64), (200, 28672, 256, 128)])
@pytest.mark.parametrize("dtype,params,symmetric,shrink", [
    (torch.bfloat16, torch.bfloat16, False, 1.0), (torch.float16, torch.float32, True, 1.0),
    (torch.float16, torch.bfloat16, False, 2.0 ** -14)])
def test_pair_form_equals_two_pass(m, n, k, group, dtype, params, symmetric, shrink):
    gen = seeded(m + n + k)
    w = torch.randn((n, k), generator=gen) * 0.02
    pw = quantize.quantize_w4_symmetric(w, group_size=group) if symmetric else quantize.quantize_w4_asymmetric(w, group_size=group, param_dtype=params)
    # shrink: scales below fp16's normal range take the fp32 conversion
    scales = (pw.scales.float() * shrink).to(DEV, params)
    zeros = None if pw.zero_points is None else pw.zero_points.to(DEV, params)
    x, bias = torch.randn((m, k), generator=gen).to(DEV, dtype), torch.randn(n, generator=gen).to(DEV)
    residual = torch.randn((m, n), generator=gen).to(DEV, dtype)

    def run(variant, **options):
        return w4a16_linear(x, pw.qweight.to(DEV), scales, zeros, group_size=group, nibble_signed=symmetric, variant=variant, **options)

    got, want = run("tcgen05_fused", bias=bias, residual=residual).double(), run("tcgen05", bias=bias, residual=residual).double()
    # fp32 sums in two orders (an error of 2^-24 per addition, a tensor-core step adds at least 16 products at once), one rounding
    values = (scales.float().abs().max() * 15 * x.float().abs().sum(1, keepdim=True) + bias.abs()[None] + residual.float().abs()).double()
    eps = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    assert ((got - want).abs() <= eps * want.abs() + 2.0 ** -23 * (k / 16) * values + 2.0 ** -24).all()
    assert (got - want).norm() <= 0.25 * eps * want.norm() + 1e-6
    assert torch.equal(run("tcgen05_fused", bias=bias, residual=residual).double(), got)      # the same bits every time
    assert native.workspace_status(DEV) == 0


@pytest.mark.parametrize("m,hidden,inter,group", [(129, 128, 128, 64), (300, 1024, 2944, 64), (512, 4096, 14336, 128), (513, 4096, 6144, 128), (256, 2048, 8192, 128)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_mlp_with_the_gating_in_the_epilogue(m, hidden, inter, group, dtype):
    gen = seeded(m + hidden + inter)

    def layer(rows, columns):
        return quantize.quantize_w4_asymmetric(torch.randn((rows, columns), generator=gen) * 0.02, group_size=group, param_dtype=dtype)

    block = W4A16SwiGLUMLP(layer(inter, hidden), layer(inter, hidden), layer(hidden, inter), device=DEV, dtype=dtype)
    assert block._one_entry(m)
    x = torch.randn((m, hidden), generator=gen).to(DEV, dtype)
    got, want = block(x).double(), block._forward(x).double()      # linear, SwiGLU kernel, linear
    # the same roundings in the same places; sums in another order flip some of them by a unit in the last place
    eps = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    assert (got - want).norm() <= 0.5 * eps * want.norm() + 1e-6
    assert native.workspace_status(DEV) == 0


# 160-column tiles of two token blocks (the narrowest that leave room for four stages only), in one wave, two waves and a
# partial last tile; K short enough for the rings never to wrap, and long; token counts past 1000
@pytest.mark.parametrize("m,n,k", [(300, 11008, 512), (512, 22016, 320), (512, 11000, 4096), (1024, 5120, 5120), (1024, 5112, 2304),
                                   (2600, 4096, 6144)])             # and 256 columns, eleven chunks of which the last is ragged
def test_wide_tiles_and_many_chunks(m, n, k):
    gen = seeded(m + n + k)
    pw = quantize.quantize_w4_asymmetric(torch.randn((n, k), generator=gen) * 0.02, group_size=64, param_dtype=torch.float16)
    weight = (pw.qweight.to(DEV), pw.scales.to(DEV), pw.zero_points.to(DEV))
    x = torch.randn((m, k), generator=gen).to(DEV, torch.float16)

    def run(variant):
        return w4a16_linear(x, *weight, group_size=64, nibble_signed=False, variant=variant, out_dtype=torch.float32)

    got, want = run("tcgen05_fused"), run("tcgen05")
    # the same exact products summed in fp32 in another order: 2^-24 of the partial sums for each of the K / 16 additions
    bound = 2.0 ** -23 * (k / 16) * weight[1].float().abs().max() * 15 * x.float().abs().sum(1, keepdim=True)
    assert ((got - want).abs() <= bound).all()
    for _ in range(5):
        assert torch.equal(run("tcgen05_fused"), got)
    assert native.workspace_status(DEV) == 0
