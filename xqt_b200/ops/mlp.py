"""W4A16 SwiGLU MLP block on B200: ``y = down(silu(gate x) * up x)``.

The block shape is xqt's toy SwiGLU MLP (xqt/kernels/nn/fixtures/toy_models.py:87-121); the fusion
choices follow its ConvRot W8A8 backend, which fuses gate and up horizontally into one linear and
gates with one vectorised kernel (xqt/kernels/ops/_impl/cute/convrot_w8a8_sm89.py:664-917,
convrot_w8a8_sm89_kernel.cu:756-837).

Per call and rank: one linear for the concatenated ``[gate; up]`` shard, one SwiGLU kernel, one
linear for the down shard; at M <= 16 the linears are the cluster split-K decode kernel, above it
the tcgen05 GEMM.  With more than one rank gate/up are split over N, down over K, and the fp32 partial
sums of down are added with one NCCL all-reduce and rounded once.
"""

from __future__ import annotations

import os

import torch
import torch.distributed as dist

from .. import native
from ..contracts import PackedWeight, PackedWeightMetadata
from ..errors import XQTBackendError
from ..hostcall import INPUT, MANY_ROWS, OUTPUT, ROWS, SCRATCH, WORKSPACE, bound_layer, guard, plan, step, weak_method
from ..parallel import shard_packed_weight
from .w4a16 import (_integer_zero_points, bind_w4a16_decode, fused_preferred, glu_row_order, integer_zero_points_now, prepare_decode, version_of, w4a16_linear,
                    w4a16_step, with_version)


def swiglu(gate_up: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
    """``[M, 2I] -> [M, I]``: ``silu(gate_up[:, :I]) * gate_up[:, I:]`` in fp32, rounded once."""

    if gate_up.ndim != 2 or gate_up.shape[1] % 16 or gate_up.dtype not in (torch.float16, torch.bfloat16):
        raise XQTBackendError("swiglu expects a rank-2 fp16/bf16 tensor [M, 2*inter] with inter % 8 == 0")
    if not gate_up.is_cuda or not gate_up.is_contiguous():
        raise XQTBackendError("swiglu expects a contiguous CUDA tensor")
    m, inter = int(gate_up.shape[0]), int(gate_up.shape[1]) // 2
    if out is None:
        out = torch.empty((m, inter), device=gate_up.device, dtype=gate_up.dtype)
    if m:
        with torch.cuda.device(gate_up.device):
            native.check(native.library().xqt_b200_swiglu(
                gate_up.data_ptr(), out.data_ptr(), m, inter, native.DTYPE_CODE[gate_up.dtype],
                native.stream_handle(gate_up.device)), "xqt_b200_swiglu")
    return out


def _concat_rows(a: PackedWeight, b: PackedWeight) -> PackedWeight:
    ma, mb = a.metadata, b.metadata
    if (ma.logical_shape[1], ma.group_size, ma.nibble_signed) != (mb.logical_shape[1], mb.group_size, mb.nibble_signed):
        raise XQTBackendError("gate and up must share K, group size and signedness to be fused")
    if (a.zero_points is None) != (b.zero_points is None):
        raise XQTBackendError("gate and up must both carry zero points or neither")
    n = ma.logical_shape[0] + mb.logical_shape[0]
    values = {f: getattr(ma, f) for f in PackedWeightMetadata.__dataclass_fields__}
    values.update(logical_shape=(n, ma.logical_shape[1]), local_shape=None if ma.local_shape is None else (n, ma.logical_shape[1]))
    return PackedWeight(
        qweight=torch.cat((a.qweight, b.qweight)), scales=torch.cat((a.scales, b.scales)),
        zero_points=None if a.zero_points is None else torch.cat((a.zero_points, b.zero_points)),
        metadata=PackedWeightMetadata(**values))


CHUNKED_DECODE_MAX_ROWS = 32


class _Linear:
    """One W4A16 layer on a device with both execution forms: decode layout and canonical bytes."""

    def __init__(self, weight: PackedWeight, device: torch.device, dtype: torch.dtype, glu: bool = False) -> None:
        meta = weight.metadata
        self.n, self.k = meta.logical_shape
        self.group, self.signed, self.dtype = int(meta.group_size), bool(meta.nibble_signed), dtype
        self.qweight = weight.qweight.to(device).contiguous()
        self.scales = weight.scales.to(device).contiguous()
        self.zeros = with_version(None if weight.zero_points is None else weight.zero_points.to(device).contiguous())
        self._bound: dict[tuple[int, torch.dtype], object] = {}
        self._gated: dict[int, object] = {}
        # glu: this is a fused [gate; up] layer.  Where the decode layout is the lanes one its tiles are built from the
        # rows in glu_row_order, and `gated` runs linear + SwiGLU as one decode launch; `tiled` then serves only that.
        self.glu, self.tiled = False, None
        if glu and self.n % 128 == 0:
            order = glu_row_order(self.n // 2).to(device)
            tiled = prepare_decode(self.qweight[order], self.scales[order], None if self.zeros is None else self.zeros[order],
                                   group_size=self.group, nibble_signed=self.signed)
            if tiled.layout == "lanes":
                self.glu, self.tiled = True, tiled
        if self.tiled is None:
            self.tiled = prepare_decode(self.qweight, self.scales, self.zeros, group_size=self.group, nibble_signed=self.signed)

    def __getstate__(self) -> dict:
        # bound calls hold addresses of this layer's tensors: a copy makes its own
        return {**self.__dict__, "_bound": {}, "_gated": {}}

    def gated(self, x: torch.Tensor) -> torch.Tensor | None:
        """``silu(gate) * up`` of a fused gate/up layer in one decode launch per 16 rows, or None where that form does
        not apply (not a glu layer, too many rows)."""

        m = int(x.shape[0])
        if not self.glu or m > CHUNKED_DECODE_MAX_ROWS:
            return None
        out = torch.empty((m, self.n // 2), device=x.device, dtype=self.dtype)
        for r0 in range(0, m, 16):
            rows = min(16, m - r0)
            run = self._gated.get(rows)
            if run is None:
                run = bind_w4a16_decode(self.tiled, rows=rows, dtype=self.dtype, glu=True)
                self._gated[rows] = run
            run(x if rows == m else x[r0:r0 + rows], out if rows == m else out[r0:r0 + rows])
        return out

    def __call__(self, x: torch.Tensor, out_dtype: torch.dtype | None = None, out: torch.Tensor | None = None) -> torch.Tensor:
        m = int(x.shape[0])
        odt = self.dtype if out_dtype is None else out_dtype
        if self.glu and m <= CHUNKED_DECODE_MAX_ROWS:
            raise XQTBackendError("a glu layer's decode tiles are interleaved: call gated()")
        if m <= 16 and (odt == self.dtype or self.tiled.layout in ("rows128", "lanes")):
            run = self._bound.get((m, odt))
            if run is None:
                run = bind_w4a16_decode(self.tiled, rows=m, dtype=self.dtype, out_dtype=odt)
                self._bound[(m, odt)] = run
            return run(x, out) if out is not None else run(x)
        if m <= CHUNKED_DECODE_MAX_ROWS and self.tiled.layout == "lanes":
            # a few decode passes over 16-row chunks: the packed weights of a layer (tens of MB) stay in the 126 MB
            # L2 between passes, and each pass runs at the decode kernel's rate -- measured ahead of the GEMM forms
            # up to two passes (from 33 rows the fused tcgen05 GEMM is ahead)
            if out is None:
                out = torch.empty((m, self.n), device=x.device, dtype=odt)
            for r0 in range(0, m, 16):
                rows = min(16, m - r0)
                run = self._bound.get((rows, odt))
                if run is None:
                    run = bind_w4a16_decode(self.tiled, rows=rows, dtype=self.dtype, out_dtype=odt)
                    self._bound[(rows, odt)] = run
                run(x[r0:r0 + rows], out[r0:r0 + rows])
            return out
        return w4a16_linear(x, self.qweight, self.scales, self.zeros, group_size=self.group,
                            nibble_signed=self.signed, k=self.k, out_dtype=odt, out=out)

    @property
    def canonical_served(self) -> bool:
        """Whether the canonical tensors are what ``w4a16_linear`` takes (it refuses zero points that differ from the scales in
        dtype or shape; the decode layout, which converts them, serves such a weight up to 16 or 32 rows)."""

        shape = (self.n, int(self.qweight.shape[1]) * 2 // self.group)
        return self.qweight.dtype == torch.uint8 and tuple(self.qweight.shape) == (self.n, shape[1] * self.group // 2) \
            and self.scales.dtype in native.DTYPE_CODE and tuple(self.scales.shape) == shape \
            and (self.zeros is None or (self.zeros.dtype == self.scales.dtype and self.zeros.shape == self.scales.shape))

    def decode_step(self, first: int, rows, source: tuple, target: tuple, *, glu: bool) -> tuple:
        """The decode launch of ``rows`` rows from row ``first`` on as a step of a bound layer."""

        status, params = native.status_word(self.qweight.device), self.tiled.params
        code, width = native.DTYPE_CODE[self.dtype], self.n // 2 if glu else self.n
        return step("xqt_b200_w4a16_decode_lanes",
                    ((source[0], source[1] + 2 * first * self.k), self.tiled.weights, params[0], params[1] if self.tiled.has_zero_point else 0,
                     0, 0, (target[0], target[1] + 2 * first * width), status),
                    (rows, self.n, self.k, self.group, self.tiled.nibble_signed, code, native.DTYPE_CODE[params.dtype], code, 2 if glu else 0))

    def fused_preferred(self, m: int) -> bool:
        return fused_preferred(m, self.n, self.k, int(self.qweight.shape[1]) * 2, self.group)

    def gemm_step(self, source: tuple, target: tuple, integer: bool | None) -> tuple:
        """The canonical-weight GEMM of any number of rows as a step of a bound layer."""

        return w4a16_step(source, self.qweight, self.scales, self.zeros, None, target, k=self.k, group_size=self.group,
                          nibble_signed=self.signed, dtype=self.dtype, integer=integer)

    def partial_into(self, x: torch.Tensor, peer) -> None:
        """Decode-size fp32 partial sums of a K-sharded layer, written into the slot of ``peer`` (a counted
        :class:`xqt_b200.parallel.PeerAllReduce`) that its next reduction reads; the kernel picks the slot on the device."""

        m = int(x.shape[0])
        run = self._bound.get((m, "peer"))
        if run is None:
            run = bind_w4a16_decode(self.tiled, rows=m, dtype=self.dtype, out_dtype=torch.float32, out_select=peer.out_select)
            self._bound[(m, "peer")] = run
        run(x, peer.partial(m, self.n))

    def rows(self, x: torch.Tensor, n0: int, n1: int, out_dtype: torch.dtype | None = None) -> torch.Tensor:
        """The output channels [n0, n1) only: ``x @ W[n0:n1]^T`` (a row block of the canonical weight is contiguous)."""

        return w4a16_linear(x, self.qweight[n0:n1], self.scales[n0:n1], None if self.zeros is None else self.zeros[n0:n1],
                            group_size=self.group, nibble_signed=self.signed, k=self.k,
                            out_dtype=self.dtype if out_dtype is None else out_dtype)


class _InjectedLinear:
    """One layer served by a caller-supplied ``local_linear(x, weight, out_dtype=...)`` (the gloo tests run the
    block's sharding and reduction logic on the CPU with the oracle in this seat)."""

    def __init__(self, weight: PackedWeight, local_linear) -> None:
        self.weight, self.local_linear = weight, local_linear
        self.n, self.k = weight.metadata.logical_shape
        self.tiled = None

    def __call__(self, x: torch.Tensor, out_dtype: torch.dtype | None = None, out: torch.Tensor | None = None) -> torch.Tensor:
        y = self.local_linear(x, self.weight) if out_dtype is None else self.local_linear(x, self.weight, out_dtype=out_dtype)
        if out is not None:
            out.copy_(y)
            return out
        return y


class W4A16SwiGLUMLP:
    """The MLP block of one rank.  ``gate`` / ``up`` are canonical ``[inter, hidden]`` weights,
    ``down`` is ``[hidden, inter]``; they are sharded here for ``rank`` of ``world``.  ``local_linear`` /
    ``swiglu_fn`` replace the CUDA kernels (tests of the multi-rank logic on CPU ranks)."""

    def __init__(self, gate: PackedWeight, up: PackedWeight, down: PackedWeight, *, device: torch.device,
                 dtype: torch.dtype = torch.bfloat16, rank: int = 0, world: int = 1, group=None,
                 peer_reduce: bool | None = None, local_linear=None, swiglu_fn=None) -> None:
        if world > 1:
            gate = shard_packed_weight(gate, world=world, rank=rank, axis=0)
            up = shard_packed_weight(up, world=world, rank=rank, axis=0)
            down = shard_packed_weight(down, world=world, rank=rank, axis=1)
        self.world, self.group, self.dtype = world, group, dtype
        # single-GPU blocks: the bound calls by 16 rows up to CHUNKED_DECODE_MAX_ROWS, and the one above, with the state of the
        # tensors it was built from
        self._decode: dict[int, object] = {}
        self._gemm: tuple | None = None
        self._can_bind = world == 1 and local_linear is None and swiglu_fn is None
        self._swiglu = swiglu_fn or swiglu
        self._fuse_gating = swiglu_fn is None and os.environ.get("XQT_B200_FUSED_SWIGLU", "1") not in {"0", ""}
        if local_linear is not None:
            self.gate_up = _InjectedLinear(_concat_rows(gate, up), local_linear)
            self.down = _InjectedLinear(down, local_linear)
            peer_reduce = False
        else:
            self.gate_up = _Linear(_concat_rows(gate, up), device, dtype, glu=self._fuse_gating)
            self.down = _Linear(down, device, dtype)
        self.hidden, self.inter_local = self.down.n, self.down.k
        # decode sizes (M <= 16): the partial sums of down are added by our own kernel over NVLink peer
        # memory instead of an NCCL all-reduce (XQT_B200_PEER_REDUCE=0 or peer_reduce=False: NCCL)
        if peer_reduce is None:
            peer_reduce = os.environ.get("XQT_B200_PEER_REDUCE", "1") not in {"0", ""}
        self._peer = None
        if world > 1 and peer_reduce and self.down.tiled is not None and self.down.tiled.layout in ("rows128", "lanes"):
            from ..parallel import PeerAllReduce

            # on the lanes layout the reduction is the counted (graph-safe) form: the call number lives on the device
            self._peer = PeerAllReduce(device, 16 * self.hidden, group, counted=self.down.tiled.layout == "lanes")

    def __getstate__(self) -> dict:
        return {**self.__dict__, "_decode": {}, "_gemm": None}

    def __setstate__(self, state: dict) -> None:
        # a block saved before these fields existed
        gate_up = state["gate_up"]
        self.__dict__.update({"_can_bind": state["world"] == 1 and isinstance(gate_up, _Linear) and state["_swiglu"] is swiglu,
                              "_fuse_gating": getattr(gate_up, "glu", False), **state, "_decode": {}, "_gemm": None})

    def __call__(self, x: torch.Tensor) -> torch.Tensor:
        if self._can_bind:
            m = x.shape[0]
            if m <= CHUNKED_DECODE_MAX_ROWS:
                run = self._decode.get((m + 15) // 16)
                if run is None:
                    run = self._decode[(m + 15) // 16] = self._bind_decode((m + 15) // 16)
                return run(x)
            run = self._gemm_call(m)
            if run is not None:
                return run(x)
        return self._forward(x)

    def _separate(self, x: torch.Tensor, *rest) -> torch.Tensor:
        """A call that the single library call's bound layer does not take."""

        run = self._gemm_call(x.shape[0], every=True) if not rest and x.ndim == 2 and x.shape[0] > CHUNKED_DECODE_MAX_ROWS else None
        return self._forward(x, *rest) if run is None else run(x)

    def _bound(self, plans: list, keep: tuple = (), slow=None):
        return bound_layer(plans, weak_method(slow or self._forward), dtype=self.dtype, device=self.gate_up.qweight.device, rows=None, k=self.gate_up.k,
                           n=self.hidden, workspace="run", keep=(self.gate_up, self.down, *keep), symbols="bound W4A16 SwiGLU MLP")

    def _bind_decode(self, chunks: int):
        """The launches of :meth:`_forward` for decode sizes of ``chunks`` times 16 rows (the last chunk may have fewer) as one
        bound layer."""

        gate_up, down, device = self.gate_up, self.down, self.gate_up.qweight.device
        if device.type != "cuda" or not gate_up.glu or down.tiled.layout != "lanes" or chunks < 1:
            return weak_method(self._forward)
        h, last = (SCRATCH, 0), 16 * (chunks - 1)
        parts = [(first, 16) for first in range(0, last, 16)] + [(last, (-last, 1))]
        steps = [gate_up.decode_step(first, rows, (INPUT, 0), h, glu=True) for first, rows in parts]
        steps += [down.decode_step(first, rows, h, (OUTPUT, 0), glu=False) for first, rows in parts]
        served = tuple(guard("xqt_b200_w4a16_decode_lanes_supported", rows, layer.n, layer.k, layer.group)
                       for layer in (gate_up, down) for rows in {rows for _, rows in parts})
        return self._bound([plan(steps, rows=(last + 1, last + 16), guards=served, scratch=(0, 2 * self.inter_local))], (native.status_word(device),))

    def _gemm_call(self, m: int, every: bool = False):
        """The launches of :meth:`_forward` above the decode sizes as one bound layer, made when there is none or a tensor has changed
        since; None where ``w4a16_linear`` has to look at the tensors itself.  Whether the zero points are integers is asked when
        the first row count comes for which it matters; until then (and in a graph capture) it is left open.  A block whose first
        row count is one for the single library call has the separate launches bound when a row count needs them (``every``)."""

        gu, dn = self.gate_up, self.down
        static = (gu.qweight, gu.scales, gu.zeros, dn.qweight, dn.scales, dn.zeros)
        state = (version_of(gu.zeros), version_of(dn.zeros), *(None if t is None else t.data_ptr() for t in static))

        def integers() -> list | None:
            answers = [integer_zero_points_now(layer.zeros) for layer in (gu, dn)] if gu.fused_preferred(m) or dn.fused_preferred(m) else [None]
            return None if None in answers else answers

        if self._gemm is not None and self._gemm[0] == state and not every and (self._gemm[2] or integers() is None):
            return self._gemm[1]
        if gu.qweight.device.type != "cuda" or not (gu.canonical_served and dn.canonical_served) \
                or any(t is not None and t.is_inference() for t in (gu.zeros, dn.zeros)):
            return None
        plans, inter, known = [], self.inter_local, integers()
        if known and self._fuse_gating and self._one_entry_form():
            code = native.DTYPE_CODE
            entry = step("xqt_b200_w4a16_swiglu_mlp", ((INPUT, 0), gu.qweight, gu.scales, gu.zeros, dn.qweight, dn.scales, dn.zeros, (OUTPUT, 0)),
                         (ROWS, self.hidden, inter, gu.group, dn.group, gu.signed, dn.signed, code[self.dtype], code[gu.scales.dtype], code[dn.scales.dtype]),
                         (WORKSPACE, 0), ("xqt_b200_w4a16_swiglu_mlp_workspace_bytes", self.hidden, inter))
            plans.append(plan([entry], rows=(CHUNKED_DECODE_MAX_ROWS + 1, MANY_ROWS),
                              guards=(guard("xqt_b200_w4a16_swiglu_mlp_supported", ROWS, self.hidden, inter, gu.group, dn.group),)))
            if not every and native.library().xqt_b200_w4a16_swiglu_mlp_supported(m, self.hidden, inter, gu.group, dn.group):
                self._gemm = (state, self._bound(plans, static, slow=self._separate), True)
                return self._gemm[1]
        both, h = (SCRATCH, 0), (SCRATCH, 0, 4 * inter)          # [rows, 2 * inter], then [rows, inter]
        plans.append(plan([gu.gemm_step((INPUT, 0), both, known and known[0]), step("xqt_b200_swiglu", (both, h), (ROWS, inter, native.DTYPE_CODE[self.dtype])),
                           dn.gemm_step(h, (OUTPUT, 0), known and known[1])], rows=(CHUNKED_DECODE_MAX_ROWS + 1, MANY_ROWS), scratch=(0, 6 * inter)))
        self._gemm = (state, self._bound(plans, static), known is not None)
        return self._gemm[1]

    def _one_entry_form(self) -> bool:
        """Both weights are what the single library call of the block takes: unpadded, integer zero points."""

        gu, dn = self.gate_up, self.down
        exact = 2 * int(gu.qweight.shape[1]) == gu.k == self.hidden and 2 * int(dn.qweight.shape[1]) == dn.k and gu.n == 2 * self.inter_local
        return exact and _integer_zero_points(gu.zeros) and _integer_zero_points(dn.zeros)

    def _one_entry(self, m: int) -> bool:
        """Both projections take the CTA-pair GEMM: the block is then one library call with the gating in the gate/up epilogue
        (unless ``XQT_B200_FUSED_SWIGLU=0`` turned the fused gating off when the block was built)."""

        gu, dn = self.gate_up, self.down
        return self._fuse_gating and self._one_entry_form() and bool(
            native.library().xqt_b200_w4a16_swiglu_mlp_supported(m, self.hidden, self.inter_local, gu.group, dn.group))

    def _forward(self, x: torch.Tensor) -> torch.Tensor:
        h = self.gate_up.gated(x) if isinstance(self.gate_up, _Linear) else None     # decode sizes: one launch
        if h is None:
            h = self._swiglu(self.gate_up(x))
        if self.world == 1:
            return self.down(h)
        m = int(h.shape[0])
        if self._peer is not None and m <= 16:
            if self._peer.counted:
                self.down.partial_into(h, self._peer)
            else:
                self.down(h, out_dtype=torch.float32, out=self._peer.partial(m, self.hidden))
            return self._peer.reduce(m, self.hidden, dtype=self.dtype)
        blocks = self._reduce_blocks(m)
        if blocks == 1 or not isinstance(self.down, _Linear):
            partial = self.down(h, out_dtype=torch.float32)
            dist.all_reduce(partial, op=dist.ReduceOp.SUM, group=self.group)
            return partial.to(self.dtype)
        # The down projection in column blocks of the output: block j's fp32 partial sums are all-reduced (NCCL, its
        # own stream) while block j + 1 is computed, so only the last block's reduction is exposed.  Blocks cut the
        # weight's rows, every packed weight is still dequantised once.
        width = self.hidden // blocks
        parts, works = [], []
        for j in range(blocks):
            part = self.down.rows(h, j * width, (j + 1) * width, out_dtype=torch.float32)
            works.append(dist.all_reduce(part, op=dist.ReduceOp.SUM, group=self.group, async_op=True))
            parts.append(part)
        out = torch.empty((m, self.hidden), device=h.device, dtype=self.dtype)
        for j, (part, work) in enumerate(zip(parts, works)):
            work.wait()
            out[:, j * width:(j + 1) * width].copy_(part)       # the cast to the activation dtype
        return out

    def capture(self, rows: int):
        """The block for a fixed row count as one CUDA graph (the decode kernels chain through programmatic dependent
        launch inside the graph, so the launches run without host gaps -- what xqt's graph decode runtime does around
        its modules, xqt/runtime/graph_decode.py).  Single-GPU blocks at any row count; with more ranks the decode
        sizes, whose reduction is the counted peer-memory kernel (every rank must then capture and replay in step: the
        same number of calls on every rank).  Returns ``replay`` with
        ``replay.input`` (``[rows, hidden]``, written by the caller, e.g. the target of its host-to-device copy) and
        ``replay.output``; ``replay()`` launches the graph on the current stream and returns ``replay.output``."""

        rows = int(rows)
        if self.world != 1 and not (self._peer is not None and self._peer.counted and rows <= 16):
            raise XQTBackendError("capture: with more than one rank only the decode sizes (rows <= 16) on the counted "
                                  "peer-memory reduction can be captured (NCCL collectives stay outside graphs here)")
        device = self.gate_up.qweight.device
        static_in = torch.zeros((rows, self.hidden), device=device, dtype=self.dtype)
        side = torch.cuda.Stream(device)
        side.wait_stream(torch.cuda.current_stream(device))
        with torch.cuda.stream(side):
            for _ in range(2):                      # bind the callables and load the kernels outside the capture
                self(static_in)
            side.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                static_out = self(static_in)
        torch.cuda.current_stream(device).wait_stream(side)

        def replay() -> torch.Tensor:
            graph.replay()
            return static_out

        replay.input, replay.output, replay.graph = static_in, static_out, graph
        return replay

    def _reduce_blocks(self, m: int) -> int:
        """Column blocks of the row-parallel reduction.  One block (the whole partial in one all-reduce) unless
        ``XQT_B200_REDUCE_BLOCKS`` asks for more: measured on two GPUs the blocked form is slower at every M (M = 4096:
        850 / 867 / 950 us with 1 / 2 / 4 blocks; M = 512: 242 / 293 / 460 us) -- the narrower GEMMs lose more than the
        overlapped part of a two-rank all-reduce gains.  More ranks shift that balance; it is a knob, not a default."""

        forced = os.environ.get("XQT_B200_REDUCE_BLOCKS")
        if forced and m >= 256 and self.hidden % (128 * max(1, int(forced))) == 0:
            return max(1, int(forced))
        return 1

    def execution_metadata(self) -> dict:
        """Which kernels serve this block (the report xqt's runtime modules expose,
        xqt/runtime/modules/composite_add_w4a4.py:304-318)."""

        return {
            "implementation": "b200_w4a16_swiglu_mlp", "world": self.world,
            "reduction": "none" if self.world == 1 else ("peer_allreduce_kernel (M <= 16) / " if self._peer else "") +
                         "NCCL all-reduce of fp32 partial sums (XQT_B200_REDUCE_BLOCKS: in column blocks overlapped with the down projection)",
            "decode_layout": None if self.gate_up.tiled is None else self.gate_up.tiled.layout, "hidden": self.hidden,
            "inter_local": self.inter_local,
            "kernels": {"m<=16": {"lanes": "w4a16_decode_cl_kernel", "rows128": "w4a16_decode_tc_kernel"}.get(
                            None if self.gate_up.tiled is None else self.gate_up.tiled.layout, "w4a16_decode_kernel"),
                        "17<=m<=128": "gemm_w4a16_fused_kernel",
                        "m>128": "gemm_w4a16_pair_kernel (m > 512: layers of 24 M weights or more) else dequant_w4_f16_kernel + gemm_f16_kernel",
                        "gating": "w4a16_decode_cl_kernel epilogue (m <= 32) / gemm_w4a16_pair_kernel epilogue (m > 128, single GPU) / swiglu_kernel" if getattr(self.gate_up, "glu", False) else "swiglu_kernel"},
        }


__all__ = ["W4A16SwiGLUMLP", "swiglu"]
