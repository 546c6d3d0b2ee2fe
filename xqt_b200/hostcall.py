"""Building bound calls that run natively: see ``csrc/host.cpp``.

A bound layer is described once -- which input it takes, which output it makes, which library entries it calls with
which arguments -- and :func:`bound_call` turns that into a callable whose steady-state call runs no Python code.
Pointer arguments are addresses of tensors that the callable keeps, or one of the sources below with a byte offset.
"""

from __future__ import annotations

import ctypes
import struct
import weakref

import torch

from . import native

INPUT, OUTPUT, RESIDUAL, SCRATCH, WORKSPACE = 1, 2, 3, 4, 5      # csrc/host.cpp: Source

# entry -> the step's number in csrc/host.cpp (Op)
_OPS = {name: i for i, name in enumerate((
    "xqt_b200_w4a16_decode_lanes", "xqt_b200_w4a16_run", "xqt_b200_swiglu", "xqt_b200_rotate_quantize",
    "xqt_b200_w8a8_gemm_addend", "xqt_b200_lowrank_down", "xqt_b200_w4a4_gemm", "xqt_b200_act_prologue",
    "xqt_b200_w8a8_gemm_lowrank", "xqt_b200_w4a16_swiglu_mlp"))}


def step(symbol: str, pointers: tuple, integers: tuple, workspace=0, workspace_bytes: int = 0) -> tuple:
    """One library call.  ``pointers``: tensors, None, addresses or ``(source, byte offset)``, in the order of the C
    prototype; ``workspace``: the same for the entry's workspace argument."""

    resolved = tuple(p.data_ptr() if isinstance(p, torch.Tensor) else (0 if p is None else p) for p in pointers)
    address = ctypes.cast(getattr(native.library(), symbol), ctypes.c_void_p).value
    workspace = workspace.data_ptr() if isinstance(workspace, torch.Tensor) else workspace
    return (_OPS[symbol], address, resolved, tuple(int(v) for v in integers), workspace, int(workspace_bytes))


def float_bits(value: float) -> int:
    """The integer a step passes for a float argument."""

    return struct.unpack("i", struct.pack("f", float(value)))[0]


class ScratchPlan:
    """Offsets of a call's temporaries inside the one scratch allocation it makes."""

    def __init__(self) -> None:
        self.nbytes = 0

    def take(self, nbytes: int) -> tuple[int, int]:
        at = self.nbytes
        self.nbytes += (int(nbytes) + 255) // 256 * 256
        return (SCRATCH, at)


def weak_method(method):
    """A bound method that does not keep its object alive: what an object's own bound call falls back to (a strong
    reference would tie the object and its weights into a cycle that only the garbage collector frees)."""

    reference = weakref.WeakMethod(method)

    def call(*args, **kwargs):
        return reference()(*args, **kwargs)

    return call


def bound_call(steps: list, slow, *, dtype: torch.dtype, device: torch.device, rows: int, k: int, n: int, out_dtype: torch.dtype | None = None,
               any_rank: bool = False, residual: bool = False, scratch_bytes: int = 0, workspace: str | None = None, keep=(), symbols: str = ""):
    """``run(x[, out[, residual]])``: checks ``x`` (``[rows, k]``, or with ``any_rank`` any shape of that many elements
    with trailing dimension ``k``), allocates ``[rows, n]`` and makes the calls.  ``slow`` has the same signature and
    gets every call whose arguments the native path does not take: it raises, or serves it.  ``workspace``: the tag of the
    pool's buffer (:func:`native.workspace`) that steps with a ``WORKSPACE`` pointer use, looked up on every call."""

    index = device.index if device.index is not None else torch.cuda.current_device()

    def failed(code: int, at: int) -> None:
        native.check(code, symbols or f"bound call, step {at}")

    pool = None if workspace is None else lambda nbytes: native.workspace(device, nbytes, workspace)
    return native.host().Bound(
        tuple(steps), slow, failed, dtype, dtype if out_dtype is None else out_dtype, index, int(rows), int(k), int(n),
        any_rank=any_rank, takes_residual=residual, scratch_bytes=int(scratch_bytes), workspace=pool,
        tag=workspace or "run", keep=keep)


__all__ = ["INPUT", "OUTPUT", "RESIDUAL", "SCRATCH", "WORKSPACE", "ScratchPlan", "bound_call", "float_bits", "step", "weak_method"]
