"""SVDQuant W8A8 on B200: int8 x int8 GEMM with a rank-R low-rank branch, under the names of xqt's native op
(xqt/kernels/ops/_impl/cute/svdq_w8a8_sm89.py): ``pack_svdq_w8a8_linear``, ``allocate_svdq_w8a8_workspace``,
``svdq_w8a8_linear``, ``bind_svdq_w8a8_linear``, ``w8a8_linear`` and the ``native_svdq_w8a8_*`` probes.

    s_a[m] = T(amax_m / 127),  q_a = clamp(rint(x / s_a)),  la = T(lora_scale x down^T)     act_prologue_i8_kernel, mode 9
    y      = T(int32(q_a q_w^T) s_a s_w + bias + la up^T)                                   gemm_scaled_kernel: both products on
                                                                                            the tensor cores, fp32 sums for la up^T

The reference's kernels are svdq_w8a8_sm89_kernel.cu (quantize_act_lora / gemm_lora); it multiplies by approximate
reciprocals of the scales where this path divides (IEEE), which can move a code that sits on a rounding boundary."""

from __future__ import annotations

from dataclasses import dataclass

import torch

from .. import native
from ..errors import XQTBackendError
from ..hostcall import INPUT, OUTPUT, WORKSPACE, bound_call, float_bits, step
from .activation import rotate_quantize

RANK_PAD = 32          # the down projection's width
UP_PAD = 64            # the up projection's K extent (one 64-element tensor-core K block)


@dataclass(frozen=True)
class PackedSVDQW8A8Linear:
    qweight: torch.Tensor          # int8 [N, K]
    weight_scales: torch.Tensor    # fp32 [N] (values representable in the activation dtype)
    bias: torch.Tensor | None      # fp32 [N]
    down: torch.Tensor             # dtype [32, K], rows past the rank are zero
    up: torch.Tensor               # dtype [N, 64], columns past the rank are zero
    input_features: int
    output_features: int
    rank: int
    dtype: torch.dtype

    @property
    def padded_rank(self) -> int:
        return RANK_PAD


@dataclass(frozen=True)
class _Unallocated:
    """A workspace field that the layer's own kernels do not use: allocated when somebody reads it."""

    shape: tuple[int, int]
    dtype: torch.dtype
    device: torch.device


class _OnDemand:
    def __set_name__(self, owner, name: str) -> None:
        self.name = name

    def __get__(self, instance, owner=None) -> torch.Tensor:
        if instance is None:
            raise AttributeError(self.name)          # to the dataclass: a field without a default
        value = instance.__dict__[self.name]
        if isinstance(value, _Unallocated):
            value = instance.__dict__[self.name] = torch.empty(value.shape, dtype=value.dtype, device=value.device)
        return value

    def __set__(self, instance, value) -> None:
        instance.__dict__[self.name] = value


@dataclass
class W8A8SVDQWorkspace:
    quantized_activation: torch.Tensor     # int8 [rows, K]
    activation_scales: torch.Tensor        # fp32 [rows]
    lora_activation: torch.Tensor = _OnDemand()        # fp32 [rows, 32]: for callers of xqt_b200_lowrank_down / _up of their own
    lora_activation16: torch.Tensor        # dtype [rows, 64], columns past 32 stay zero
    low_rank_output: torch.Tensor = _OnDemand()        # fp32 [rows, N], likewise

    @property
    def padded_rows(self) -> int:
        return int(self.quantized_activation.shape[0])

    def _check(self, packed: PackedSVDQW8A8Linear, rows: int, low_rank: bool) -> None:
        k, n = packed.input_features, packed.output_features
        if self.padded_rows < rows or int(self.quantized_activation.shape[1]) != k or int(self.__dict__["low_rank_output"].shape[1]) != n:
            raise ValueError("workspace extent does not match inputs")
        for tensor, dtype, shape in ((self.quantized_activation, torch.int8, (rows, k)), (self.activation_scales, torch.float32, (rows,)),
                                     (self.lora_activation16, packed.dtype, (rows, UP_PAD))):
            if tensor is self.lora_activation16 and not low_rank:
                continue
            if tensor.dtype != dtype or tuple(tensor[:rows].shape) != shape or not tensor[:rows].is_contiguous():
                raise XQTBackendError("SVDQ W8A8: workspace buffers do not match the layer")


def native_svdq_w8a8_shape_supported(input_features: int, output_features: int, rank: int) -> bool:
    """K a multiple of 32 (the down projection's K step), N a multiple of 8, rank <= 32."""

    return int(input_features) > 0 and int(input_features) % 32 == 0 and int(output_features) > 0 \
        and int(output_features) % 8 == 0 and 0 <= int(rank) <= RANK_PAD


def native_svdq_w8a8_available(*, build: bool = False) -> bool:
    if not torch.cuda.is_available() or torch.cuda.get_device_capability() != (10, 0):
        return False
    return native.available() if build else native.LIBRARY_PATH.exists()


def native_svdq_w8a8_version() -> str:
    return native.version()


def pack_svdq_w8a8_linear(residual_weight: torch.Tensor, down_weight: torch.Tensor | None, up_weight: torch.Tensor | None,
                          bias: torch.Tensor | None = None) -> PackedSVDQW8A8Linear:
    """Per-output-channel int8 weights with ``scale = T(absmax/127)`` (1 for a zero row), as the reference's pack
    (svdq_w8a8_sm89.py:158-232); ``down_weight`` ``[rank, K]``, ``up_weight`` ``[N, rank]`` in the weight's dtype."""

    if residual_weight.ndim != 2 or residual_weight.dtype not in (torch.bfloat16, torch.float16) or not residual_weight.is_cuda:
        raise XQTBackendError("SVDQ W8A8: residual_weight must be a CUDA bf16/fp16 [N, K] tensor")
    n, k = (int(v) for v in residual_weight.shape)
    rank = 0 if down_weight is None else int(down_weight.shape[0])
    if not native_svdq_w8a8_shape_supported(k, n, rank):
        raise XQTBackendError("SVDQ W8A8 on B200 requires K % 32 == 0, N % 8 == 0 and rank <= 32")
    dtype, device = residual_weight.dtype, residual_weight.device
    if rank and (tuple(down_weight.shape) != (rank, k) or up_weight is None or tuple(up_weight.shape) != (n, rank)):
        raise ValueError("down_weight must be [rank, K] and up_weight [N, rank]")
    w = residual_weight.to(torch.float32)
    amax = w.abs().amax(dim=1)
    scale = torch.where(amax > 0, amax / 127.0, torch.ones_like(amax)).to(dtype).to(torch.float32)
    q = torch.round(w / scale[:, None]).clamp_(-128, 127).to(torch.int8).contiguous()
    down = torch.zeros((RANK_PAD, k), device=device, dtype=dtype)
    up = torch.zeros((n, UP_PAD), device=device, dtype=dtype)
    if rank:
        down[:rank] = down_weight.to(device=device, dtype=dtype)
        up[:, :rank] = up_weight.to(device=device, dtype=dtype)
    if bias is not None and (bias.ndim != 1 or int(bias.numel()) != n):
        raise ValueError("bias must match output_features")
    return PackedSVDQW8A8Linear(
        qweight=q, weight_scales=scale.contiguous(),
        bias=None if bias is None else bias.to(device=device, dtype=torch.float32).contiguous(),
        down=down, up=up, input_features=k, output_features=n, rank=rank, dtype=dtype)


def allocate_svdq_w8a8_workspace(rows: int, packed: PackedSVDQW8A8Linear) -> W8A8SVDQWorkspace:
    rows, k, n, device = int(rows), packed.input_features, packed.output_features, packed.qweight.device
    return W8A8SVDQWorkspace(
        quantized_activation=torch.empty((rows, k), dtype=torch.int8, device=device),
        activation_scales=torch.empty((rows,), dtype=torch.float32, device=device),
        lora_activation=_Unallocated((rows, RANK_PAD), torch.float32, device),
        lora_activation16=torch.zeros((rows, UP_PAD), dtype=packed.dtype, device=device),
        low_rank_output=_Unallocated((rows, n), torch.float32, device))


def _forward(inputs: torch.Tensor, packed: PackedSVDQW8A8Linear, workspace: W8A8SVDQWorkspace | None, lora_scale: float,
             low_rank: bool, return_parts: bool = False):
    if inputs.ndim != 2 or inputs.dtype != packed.dtype or not inputs.is_cuda:
        raise XQTBackendError("SVDQ W8A8: inputs must be a CUDA rank-2 tensor in the packed layer's dtype")
    if int(inputs.shape[1]) != packed.input_features:
        raise ValueError("inputs do not match packed input_features")
    if inputs.device != packed.qweight.device:
        raise XQTBackendError("inputs and packed weights must share a CUDA device")
    x = inputs.contiguous()
    m, k, n, device = int(x.shape[0]), packed.input_features, packed.output_features, x.device
    out = torch.empty((m, n), dtype=packed.dtype, device=device)
    if m == 0:
        return out
    ws = workspace or allocate_svdq_w8a8_workspace(m, packed)
    low_rank = low_rank and bool(packed.rank)
    ws._check(packed, m, low_rank)
    codes, scales, la = ws.quantized_activation[:m], ws.activation_scales[:m], ws.lora_activation16[:m]
    lib, stream, dcode = native.library(), native.stream_handle(device), native.DTYPE_CODE[packed.dtype]
    with torch.cuda.device(device):
        scratch = native.workspace(device, 256, "gemm")
        if low_rank:
            native.check(lib.xqt_b200_act_prologue(x.data_ptr(), 0, codes.data_ptr(), scales.data_ptr(), packed.down.data_ptr(), la.data_ptr(),
                                                   lora_scale, m, k, 0, 0, 9, 3, dcode, stream), "xqt_b200_act_prologue")
        else:                                                # serves an input at any address
            rotate_quantize(x, None, bits=8, out=(ws.quantized_activation, ws.activation_scales), scale_in_act_dtype=True)
        head = (codes.data_ptr(), packed.qweight.data_ptr(), scales.data_ptr(), packed.weight_scales.data_ptr(), native.ptr(packed.bias))
        tail = (out.data_ptr(), m, n, k, dcode, scratch.data_ptr(), scratch.numel(), stream)
        if low_rank:
            native.check(lib.xqt_b200_w8a8_gemm_lowrank(*head, la.data_ptr(), packed.up.data_ptr(), *tail), "xqt_b200_w8a8_gemm_lowrank")
        else:
            native.check(lib.xqt_b200_w8a8_gemm(*head, *tail), "xqt_b200_w8a8_gemm")
    if return_parts:
        return out, {"codes": codes, "scales": scales}
    return out


def svdq_w8a8_linear(inputs: torch.Tensor, packed: PackedSVDQW8A8Linear, *, workspace: W8A8SVDQWorkspace | None = None,
                     lora_scale: float = 1.0, return_parts: bool = False):
    """Dynamic per-token int8 activations x per-channel int8 weights + low-rank branch (svdq_w8a8_sm89.py:258-312)."""

    return _forward(inputs, packed, workspace, float(lora_scale), True, return_parts)


def w8a8_linear(inputs: torch.Tensor, packed: PackedSVDQW8A8Linear, *, workspace: W8A8SVDQWorkspace | None = None) -> torch.Tensor:
    """The same dynamic W8A8 path without the low-rank branch (svdq_w8a8_sm89.py:380-425)."""

    return _forward(inputs, packed, workspace, 1.0, False)


def bind_svdq_w8a8_linear(packed: PackedSVDQW8A8Linear, workspace: W8A8SVDQWorkspace | None = None, *, rows: int,
                          lora_scale: float = 1.0):
    """Validated state for the steady-state path (svdq_w8a8_sm89.py:314-377): the workspace is fixed here, a call
    allocates only its output."""

    rows = int(rows)
    if workspace is None:
        workspace = allocate_svdq_w8a8_workspace(rows, packed)
    if workspace.padded_rows < rows:
        raise ValueError("workspace row extent does not match rows")
    k, n, dtype, device, scale = packed.input_features, packed.output_features, packed.dtype, packed.qweight.device, float(lora_scale)
    # a workspace may be shared by layers of several sizes: its memory is what counts here
    for tensor, held, count in ((workspace.quantized_activation, torch.int8, rows * k), (workspace.activation_scales, torch.float32, rows),
                                (workspace.lora_activation16, dtype, rows * UP_PAD if packed.rank else 0)):
        if count and (tensor.dtype != held or not tensor.is_contiguous() or tensor.numel() < count):
            raise ValueError("workspace extent does not match the packed layer")
    native.workspace(device, 256, "gemm")            # the current stream's status word, made now
    dcode = native.DTYPE_CODE[dtype]
    codes, scales, la = workspace.quantized_activation, workspace.activation_scales, workspace.lora_activation16

    def run(inputs: torch.Tensor) -> torch.Tensor:
        if inputs.dtype != dtype or inputs.device != device or inputs.ndim != 2 or tuple(inputs.shape) != (rows, k) \
                or not inputs.is_contiguous():
            raise XQTBackendError("bound SVDQ W8A8 call: input shape, dtype, device or layout mismatch")
        if torch.cuda.current_device() != (device.index if device.index is not None else torch.cuda.current_device()):
            raise XQTBackendError("bound SVDQ W8A8 call: make the weight's device current before calling")
        return _forward(inputs, packed, workspace, scale, True)

    low_rank = bool(packed.rank)
    quantise = step("xqt_b200_act_prologue", ((INPUT, 0), 0, codes, scales, packed.down if low_rank else 0, la if low_rank else 0),
                    (float_bits(scale), rows, k, 0, 0, 9, 3 if low_rank else 0, dcode))
    if low_rank:
        gemm = step("xqt_b200_w8a8_gemm_lowrank", (codes, packed.qweight, scales, packed.weight_scales, packed.bias, la, packed.up, (OUTPUT, 0)),
                    (rows, n, k, dcode), (WORKSPACE, 0), 256)
    else:
        gemm = step("xqt_b200_w8a8_gemm_addend", (codes, packed.qweight, scales, packed.weight_scales, packed.bias, 0, (OUTPUT, 0)),
                    (rows, n, k, dcode), (WORKSPACE, 0), 256)
    return bound_call([quantise, gemm], run, dtype=dtype, device=device, rows=rows, k=k, n=n, workspace="gemm", keep=(packed, workspace),
                      symbols="bound SVDQ W8A8 (quantise / GEMM)")


__all__ = ["PackedSVDQW8A8Linear", "W8A8SVDQWorkspace", "allocate_svdq_w8a8_workspace", "bind_svdq_w8a8_linear",
           "native_svdq_w8a8_available", "native_svdq_w8a8_shape_supported", "native_svdq_w8a8_version",
           "pack_svdq_w8a8_linear", "svdq_w8a8_linear", "w8a8_linear"]
