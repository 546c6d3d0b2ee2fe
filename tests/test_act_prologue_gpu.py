"""The fused activation prologue (rotation, quantisation, down projection) against the two-kernel form, whose codes and
scales other tests hold to the oracle: codes and scales bit for bit, the down projection against fp32 torch."""

from __future__ import annotations

import pytest
import torch

from conftest import seeded
from xqt_b200 import native, quantize
from xqt_b200.ops.activation import _KIND, _column_scale, rotate_quantize

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)
ROTATIONS = {"none": None, "r16": quantize.regular_rotation(16), "r64": quantize.randomized_rotation(64, 3), "r256": quantize.regular_rotation(256),
             "s32": quantize.randomized_rotation(32, 4), "s128": quantize.randomized_rotation(128, 5)}


# rows: one, the remainders of a 4-row unit, and (2400, 1100) the 16- and 8-row CTAs; K: below and across a 256-feature chunk
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,k,rotation,mode", [
    (1, 64, "r64", 6), (3, 320, "r64", 6), (5, 768, "s128", 6), (130, 3072, "r256", 6), (1100, 512, "s32", 6), (2400, 384, "s128", 6), (9, 192, "none", 6), (40, 8192, "s128", 6), (1400, 4096, "r64", 6),
    (1, 64, "r16", 8), (6, 288, "s32", 8), (7, 2304, "r256", 8), (1100, 512, "s128", 8), (33, 544, "none", 8), (1300, 4096, "r256", 8), (3, 20480, "s32", 8), (2, 16384, "r64", 8),
    (1, 32, "none", 9), (18, 4096, "none", 9), (1100, 1056, "none", 9), (2400, 640, "none", 9)])
def test_matches_the_separate_kernels(m, k, rotation, mode, dtype):
    rot = ROTATIONS[rotation]
    x = torch.randn((m, k), generator=seeded(m + k)) * 3
    x[:, ::37] *= 20
    x[m // 2] = 0                                          # an all-zero token
    x = x.to(DEV, dtype)
    down = (torch.randn((32, k), generator=seeded(k)) * 0.05).to(DEV, dtype)
    want_codes, want_scales, rotated = rotate_quantize(x, rot, bits=4 if mode == 6 else 8, sign_magnitude=mode == 6, tiled_scales=mode == 6,
                                                       scale_in_act_dtype=mode == 9, return_rotated=True)
    lib = native.library()
    kind, block = _KIND[None if rot is None else rot.kind], 0 if rot is None else rot.block
    assert lib.xqt_b200_act_prologue_supported(k, kind, block, mode)
    column_scale = None if rot is None else _column_scale(rot, DEV)
    want_la = 0.5 * rotated.float() @ down.float().t()
    # the MMA's fp32 sums of K exact products: the error of a sum of K terms in fp32 is below K * 2^-24 of the sum of magnitudes
    bound = 0.5 * k * 2.0 ** -24 * (rotated.float().abs() @ down.float().abs().t()) + 1e-30
    for form in (0, 1, 2, 3):
        codes = torch.full((m, k), 99, device=DEV, dtype=torch.int8)
        scales = torch.full_like(want_scales, -1.0)
        la = torch.zeros({0: (1,), 1: (m, 32), 2: (-(-m // 128) * 128, 32), 3: (m, 64)}[form], device=DEV, dtype=dtype if form == 3 else torch.float32)
        native.check(lib.xqt_b200_act_prologue(
            x.data_ptr(), native.ptr(column_scale), codes.data_ptr(), scales.data_ptr(), down.data_ptr() if form else 0, la.data_ptr() if form else 0,
            0.5, m, k, kind, block, mode, form, native.DTYPE_CODE[dtype], native.stream_handle(DEV)), "xqt_b200_act_prologue")
        assert torch.equal(codes, want_codes)
        if mode == 6:                                      # tile-major: only the rows below M are written
            order = lambda s: s.reshape(-1, k // 64, 128).permute(0, 2, 1).reshape(-1, k // 64)[:m]
            assert torch.equal(order(scales), order(want_scales))
        else:
            assert torch.equal(scales, want_scales)
        if form == 1:
            assert ((la - want_la).abs() <= bound).all()
            plain = la
        elif form == 2:                                    # [hi | lo] bf16 rows, chunks swizzled by row
            chunks = la.view(torch.bfloat16).reshape(-1, 8, 8)
            index = torch.arange(8, device=DEV)[None] ^ (torch.arange(chunks.shape[0], device=DEV)[:, None] & 7)
            straight = torch.gather(chunks, 1, index[:, :, None].expand_as(chunks)).reshape(-1, 64).float()[:m]
            hi = plain.to(torch.bfloat16).float()
            assert torch.equal(straight[:, :32], hi) and torch.equal(straight[:, 32:], (plain - hi).to(torch.bfloat16).float())
        elif form == 3:
            assert torch.equal(la[:, :32], plain.to(dtype)) and not la[:, 32:].any()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,k,rotation,mode", [
    (21, 768, "s128", 6), (21, 320, "r64", 6), (21, 3072, "none", 6), (1300, 512, "r256", 6), (2400, 512, "none", 6),
    (21, 2304, "r256", 8), (21, 544, "none", 8), (21, 20480, "s32", 8), (1300, 512, "s128", 8), (21, 1056, "none", 9), (2400, 640, "none", 9)])
def test_values_that_are_not_finite(m, k, rotation, mode, dtype):
    """Infinities, NaN and sums that overflow: the separate kernels' codes and scales, which leave a NaN out of a maximum, give
    it the lowest code and let an infinite maximum make an infinite scale."""

    rot, gen = ROTATIONS[rotation], seeded(m * k)
    x = torch.randn((m, k), generator=gen) * 3
    inf, nan, top = float("inf"), float("nan"), torch.finfo(dtype).max
    x[1, 5], x[2, k - 1], x[3, 7] = inf, -inf, nan
    x[4, :64], x[5, 64:] = nan, nan
    x[6], x[7] = nan, inf
    x[8, 3], x[8, 40], x[8, k - 2] = nan, inf, -inf
    x[9], x[10, ::5], x[11] = 0.0, -top, top
    x[12, k // 2:] = -nan
    x[13, 11], x[13, 12] = inf, -inf
    x[14, 0] = -nan
    x[m - 1, k - 1] = nan
    x = x.to(DEV, dtype)
    down = (torch.randn((32, k), generator=gen) * 0.05).to(DEV, dtype)
    want_codes, want_scales, _ = rotate_quantize(x, rot, bits=4 if mode == 6 else 8, sign_magnitude=mode == 6, tiled_scales=mode == 6,
                                                 scale_in_act_dtype=mode == 9, return_rotated=True)
    kind, block = _KIND[None if rot is None else rot.kind], 0 if rot is None else rot.block
    column_scale = None if rot is None else _column_scale(rot, DEV)
    for form in (0, 1):
        codes, scales = torch.full((m, k), 99, device=DEV, dtype=torch.int8), torch.full_like(want_scales, -1.0)
        la = torch.zeros((m, 32), device=DEV)
        native.check(native.library().xqt_b200_act_prologue(
            x.data_ptr(), native.ptr(column_scale), codes.data_ptr(), scales.data_ptr(), down.data_ptr() if form else 0, la.data_ptr() if form else 0,
            1.0, m, k, kind, block, mode, form, native.DTYPE_CODE[dtype], native.stream_handle(DEV)), "xqt_b200_act_prologue")
        assert torch.equal(codes, want_codes)
        order = (lambda s: s.reshape(-1, k // 64, 128).permute(0, 2, 1).reshape(-1, k // 64)[:m]) if mode == 6 else (lambda s: s)
        assert torch.equal(order(scales), order(want_scales))        # no scale is NaN


@pytest.mark.parametrize("k", [51200, 169984])             # the longest token of the separate kernels, and of the cluster form
def test_longest_tokens(k):
    lib, x = native.library(), (torch.randn((5, k), generator=seeded(k)) * 3).to(DEV, torch.bfloat16)
    assert lib.xqt_b200_act_prologue_supported(k, 0, 0, 8) and not lib.xqt_b200_act_prologue_supported(169984 + 16, 0, 0, 8)
    codes, scales = rotate_quantize(x, None, bits=8)
    want_scales = x.float().abs().amax(dim=1) / torch.full((5,), 127.0, device=DEV)      # by a scalar, torch multiplies by its reciprocal
    assert torch.equal(scales, want_scales)
    assert torch.equal(codes, torch.round(x.float() / want_scales[:, None]).clamp(-128, 127).to(torch.int8))


@pytest.mark.parametrize("m,k,rotation,mode", [(9, 768, "r256", 8), (600, 512, "s128", 8), (9, 768, "s32", 6), (1300, 512, "r64", 6)])
def test_column_factors_read_before_and_after_the_wait(m, k, rotation, mode):
    rot, dtype = ROTATIONS[rotation], torch.bfloat16
    x, column_scale = torch.randn((m, k), generator=seeded(m)).to(DEV, dtype), _column_scale(rot, DEV)
    down = torch.randn((32, k), generator=seeded(k)).to(DEV, dtype)
    got = []
    for ready in (0, 256):                                 # 256: XQT_B200_ROT_FACTORS_READY
        codes, la = torch.full((m, k), 99, device=DEV, dtype=torch.int8), torch.zeros((m, 32), device=DEV)
        scales = torch.zeros((m,) if mode == 8 else (-(-m // 128) * 128, k // 64), device=DEV)
        native.check(native.library().xqt_b200_act_prologue(
            x.data_ptr(), column_scale.data_ptr(), codes.data_ptr(), scales.data_ptr(), down.data_ptr(), la.data_ptr(), 1.0, m, k, _KIND[rot.kind] | ready,
            rot.block, mode, 1, native.DTYPE_CODE[dtype], native.stream_handle(DEV)), "xqt_b200_act_prologue")
        got.append((codes, scales, la))
    assert all(torch.equal(a, b) for a, b in zip(*got))
    assert torch.equal(got[0][0], rotate_quantize(x, rot, bits=4 if mode == 6 else 8, sign_magnitude=mode == 6, tiled_scales=mode == 6, return_rotated=True)[0])
