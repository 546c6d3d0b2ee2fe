"""The int8 GEMM over the sizes at which its launch forms change: few tokens (K split over a cluster), single tiles, CTA
pairs; ragged edges of every tile.  int32 sums are exact, and the scaling is the same fp32 expression in torch."""

from __future__ import annotations

import pytest
import torch

from conftest import seeded
from xqt_b200 import native

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n,k", [
    (1, 8, 16), (1, 4096, 4096), (9, 1032, 8192), (64, 264, 1040), (127, 512, 2048), (128, 520, 384), (129, 1000, 144),
    (300, 3000, 1024), (513, 4104, 528), (1000, 2568, 2064), (2048, 4096, 512), (2305, 4112, 656)])
def test_int8_gemm_is_exact(m, n, k, dtype):
    gen = seeded(m + n + k)
    a = torch.randint(-128, 128, (m, k), generator=gen, dtype=torch.int8).to(DEV)
    b = torch.randint(-128, 128, (n, k), generator=gen, dtype=torch.int8).to(DEV)
    rows, cols = (torch.rand(m, generator=gen) * 1e-3).to(DEV), (torch.rand(n, generator=gen) * 1e-3).to(DEV)
    bias, addend = torch.randn(n, generator=gen).to(DEV), torch.randn((m, n), generator=gen).to(DEV)
    la, up = torch.randn((m, 64), generator=gen).to(DEV, dtype), torch.randn((n, 64), generator=gen).to(DEV, dtype)
    lib, scratch, code, stream = native.library(), native.workspace(DEV, 256, "gemm"), native.DTYPE_CODE[dtype], native.stream_handle(DEV)
    acc = (a.double() @ b.double().t()).to(torch.float32)          # exact in fp64; |sum| < 2^28 is converted to fp32 by both
    plain = acc * (rows[:, None] * cols[None])
    head = (a.data_ptr(), b.data_ptr(), rows.data_ptr(), cols.data_ptr())
    tail = (m, n, k, code, scratch.data_ptr(), scratch.numel(), stream)

    def call(fn, *middle):
        out = torch.full((m, n), float("nan"), device=DEV, dtype=dtype)
        native.check(fn(*head, *middle, out.data_ptr(), *tail), "int8 GEMM")
        return out

    assert torch.equal(call(lib.xqt_b200_w8a8_gemm, 0), plain.to(dtype))
    assert torch.equal(call(lib.xqt_b200_w8a8_gemm, bias.data_ptr()), (plain + bias).to(dtype))
    assert torch.equal(call(lib.xqt_b200_w8a8_gemm_addend, bias.data_ptr(), addend.data_ptr()), (plain + bias + addend).to(dtype))
    low = la[:, :32].double() @ up[:, :32].double().t()
    want = (plain.double() + bias.double()) + low
    got = call(lib.xqt_b200_w8a8_gemm_lowrank, bias.data_ptr(), la.data_ptr(), up.data_ptr()).double()
    # one rounding to the output type plus fp32 sums of 32 products and three additions (2^-18 of the largest magnitude met)
    eps = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    magnitude = plain.double().abs() + bias.double().abs() + la[:, :32].double().abs() @ up[:, :32].double().abs().t()
    assert ((got - want).abs() <= eps * want.abs() + 2.0 ** -18 * magnitude + 2.0 ** -24).all()
    assert native.workspace_status(DEV) == 0


@pytest.mark.parametrize("m,n,k", [(5, 136, 256), (300, 4096, 512)])         # the single and the pair form
def test_scales_and_bias_at_any_address(m, n, k):
    gen = seeded(m + n)
    a, b = (torch.randint(-128, 128, s, generator=gen, dtype=torch.int8).to(DEV) for s in ((m, k), (n, k)))
    a_scale = (torch.rand(m, generator=gen) * 0.01).to(DEV)
    lib, scratch, stream = native.library(), native.workspace(DEV, 256, "gemm"), native.stream_handle(DEV)
    values = torch.rand(2 * n + 8, generator=gen).to(DEV)

    def run(scale, bias):
        out = torch.empty((m, n), device=DEV, dtype=torch.bfloat16)
        native.check(lib.xqt_b200_w8a8_gemm(a.data_ptr(), b.data_ptr(), a_scale.data_ptr(), scale.data_ptr(), native.ptr(bias), out.data_ptr(), m, n, k,
                                            native.BF16, scratch.data_ptr(), scratch.numel(), stream), "xqt_b200_w8a8_gemm")
        return out

    for at, bias_at in ((1, None), (2, 0), (0, 3), (3, 1)):
        scale, bias = values[at:at + n], None if bias_at is None else values[n + bias_at:2 * n + bias_at]
        assert torch.equal(run(scale, bias), run(scale.clone(), None if bias is None else bias.clone()))
