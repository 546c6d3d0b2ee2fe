"""Building bound calls that run natively: see ``csrc/host.cpp``.

A bound layer is described once -- which input it takes, which output it makes, which library entries it calls with
which arguments -- and :func:`bound_call` turns that into a callable whose steady-state call runs no Python code.
Pointer arguments are addresses of tensors that the callable keeps, or one of the sources below with a byte offset (and bytes
per row of the call's input); an integer argument may be ``(constant, factor of the row count)``.
"""

from __future__ import annotations

import ctypes
import functools
import struct
import weakref

import torch

from . import native

INPUT, OUTPUT, RESIDUAL, SCRATCH, WORKSPACE = 1, 2, 3, 4, 5      # csrc/host.cpp: Source
ROWS = (0, 1)                                                    # the integer argument "rows of the input"
MANY_ROWS = 2 ** 31 - 1

# entry -> the step's number in csrc/host.cpp (Op)
_OPS = {name: i for i, name in enumerate((
    "xqt_b200_w4a16_decode_lanes", "xqt_b200_w4a16_run", "xqt_b200_swiglu", "xqt_b200_rotate_quantize",
    "xqt_b200_w8a8_gemm_addend", "xqt_b200_lowrank_down", "xqt_b200_w4a4_gemm", "xqt_b200_act_prologue",
    "xqt_b200_w8a8_gemm_lowrank", "xqt_b200_w4a16_swiglu_mlp"))}


@functools.cache
def _address(symbol: str) -> int:
    return ctypes.cast(getattr(native.library(), symbol), ctypes.c_void_p).value


def step(symbol: str, pointers: tuple, integers: tuple, workspace=0, workspace_bytes: int | tuple = 0) -> tuple:
    """One library call.  ``pointers``: tensors, None, addresses or ``(source, byte offset[, bytes per row])``, in the order of the
    C prototype; ``workspace``: the same for the entry's workspace argument; ``workspace_bytes``: its size, or
    ``(entry, a, b)`` for what ``entry(rows, a, b)`` returns."""

    resolved = tuple(p.data_ptr() if isinstance(p, torch.Tensor) else (0 if p is None else p) for p in pointers)
    workspace = workspace.data_ptr() if isinstance(workspace, torch.Tensor) else workspace
    need = (_address(workspace_bytes[0]), *workspace_bytes[1:]) if isinstance(workspace_bytes, tuple) else int(workspace_bytes)
    return (_OPS[symbol], _address(symbol), resolved, tuple(v if isinstance(v, tuple) else int(v) for v in integers), workspace, need)


def guard(symbol: str, rows, *integers: int) -> tuple:
    """The condition ``symbol(rows, *integers) != 0`` of a plan."""

    return (_address(symbol), rows, tuple(int(v) for v in integers))


def plan(steps, *, rows: tuple[int, int], guards: tuple = (), scratch: tuple[int, int] = (0, 0)) -> tuple:
    """The calls for row counts ``rows[0]`` to ``rows[1]`` where every guard holds; ``scratch``: bytes, and bytes per row."""

    return (*rows, tuple(guards), tuple(steps), *scratch)


def float_bits(value: float) -> int:
    """The integer a step passes for a float argument."""

    return struct.unpack("i", struct.pack("f", float(value)))[0]


def weak_method(method):
    """A bound method that does not keep its object alive: what an object's own bound call falls back to (a strong
    reference would tie the object and its weights into a cycle that only the garbage collector frees)."""

    reference = weakref.WeakMethod(method)

    def call(*args, **kwargs):
        return reference()(*args, **kwargs)

    return call


def bound_layer(plans: list, slow, *, dtype: torch.dtype, device: torch.device, rows: int | None, k: int, n: int,
                out_dtype: torch.dtype | None = None, any_rank: bool = False, residual: bool = False, workspace: str | None = None,
                keep=(), symbols: str = ""):
    """``run(x[, out[, residual]])``: checks ``x`` (``[rows, k]``, or with ``any_rank`` any shape of that many elements
    with trailing dimension ``k``; ``rows`` None: as many as one of the plans takes), allocates ``[rows, n]`` and makes the calls
    of the first plan that fits.  ``slow`` has the same signature and
    gets every call whose arguments the native path does not take: it raises, or serves it.  ``workspace``: the tag of the
    pool's buffer (:func:`native.workspace`) that steps with a ``WORKSPACE`` pointer use, looked up on every call."""

    index = device.index if device.index is not None else torch.cuda.current_device()

    def failed(code: int, at: int) -> None:
        native.check(code, symbols or f"bound call, step {at}")

    pool = None if workspace is None else lambda nbytes: native.workspace(device, nbytes, workspace)
    return native.host().Bound(
        tuple(plans), slow, failed, dtype, dtype if out_dtype is None else out_dtype, index, -1 if rows is None else int(rows), int(k), int(n),
        any_rank=any_rank, takes_residual=residual, workspace=pool, tag=workspace or "run", keep=keep)


def bound_call(steps: list, slow, *, rows: int, **options):
    """:func:`bound_layer` for one row count."""

    return bound_layer([plan(steps, rows=(int(rows), int(rows)))], slow, rows=rows, **options)


__all__ = ["INPUT", "MANY_ROWS", "OUTPUT", "RESIDUAL", "ROWS", "SCRATCH", "WORKSPACE", "bound_call", "bound_layer", "float_bits", "guard", "plan",
           "step", "weak_method"]
