"""Block-level API of the B200 MoE layer.

`B200MoeBlock` is the object a serving loop holds per MoE layer: it owns the
layer's device weights, the scratch of the layer pass and (for expert
parallelism) the peer-memory buffers, and exposes

    forward_device(x_dev)          -> out_dev            inputs already in HBM
    forward_host(x_pinned, out_pinned)                    host buffers, copies included
    forward(hidden_states[B,S,H])  -> (out, router_logits) | out
                                      the `DistributedSparseMoeBlock.forward`
                                      contract (utils/eval_core.py:16418-16563)

Everything it computes goes through the C ABI; there is no eager fallback.
"""
from __future__ import annotations

from typing import Optional

import torch

from .layer import LayerRunner, LayerWeights


class B200MoeBlock:
    def __init__(self, weights: LayerWeights, top_k: int, max_tokens: int,
                 norm_topk_prob: bool = False, fp32_router_logits: bool = False,
                 return_router_logits: bool = True, ep_rank: int = 0, ep_size: int = 1,
                 process_group=None, owner=None, use_graphs: bool = False):
        self.weights = weights
        self.device = weights.device
        self.top_k = top_k
        self.ep_rank, self.ep_size = ep_rank, ep_size
        self.return_router_logits = return_router_logits
        self.runner = LayerRunner(weights, top_k, max_tokens, renorm=norm_topk_prob,
                                  fp32_logits=fp32_router_logits, want_logits=True)
        self._ep = None
        if ep_size > 1:
            from .ep import ExpertParallelLayer
            self._ep = ExpertParallelLayer(weights, top_k, max_tokens, ep_rank, ep_size,
                                           process_group, owner=owner, renorm=norm_topk_prob,
                                           fp32_logits=fp32_router_logits)
        self._x_stage: Optional[torch.Tensor] = None
        self.last_launches = 0
        # Replay each (input buffer, output buffer) pair's step from a CUDA graph
        # (see `forward_device`); off by default because a graph pins its buffers.
        self.use_graphs = use_graphs
        self._graphs = {}
        self._part_graphs = {}
        self._graph_reserve = self.runner.reserves

    @classmethod
    def from_block_weights(cls, w, device: torch.device, ep_rank: int = 0, ep_size: int = 1,
                           max_tokens: int = 4096, process_group=None, placement=None,
                           layer_idx: int = 0, stage: str = "prefill",
                           use_graphs: bool = False) -> "B200MoeBlock":
        """Build from seeded `synth.BlockWeights`; at ep_size > 1 only the
        experts this rank serves are loaded: round-robin (e % ep_size) by default,
        or every expert a `placement.Placement` lists `ep_rank` as a replica of,
        with that placement's per-source destination table."""
        s = w.shape
        owner = None
        if ep_size == 1:
            lw = LayerWeights.from_block_weights(w, device)
        else:
            if placement is not None:
                owned = sorted(placement.receive_experts(layer_idx, ep_rank, stage))
                owner = placement.dest_table(layer_idx, stage)
            else:
                owned = [e for e in range(s.num_experts) if e % ep_size == ep_rank]
            lw = LayerWeights(s.hidden, s.inter, s.num_experts, max(1, len(owned)), s.shared_inter, device)
            lw.set_router(w.router, w.router_bias)
            slot_of = [-1] * s.num_experts
            for slot, e in enumerate(owned):
                lw.load_expert(slot, w.gate[e], w.up[e], w.down[e])
                slot_of[e] = slot
            lw.set_slot_map(slot_of)
            if s.shared_inter:
                lw.set_shared(w.sh_gate, w.sh_up, w.sh_down, w.sh_scalar_gate)
        return cls(lw, s.top_k, max_tokens, norm_topk_prob=s.norm_topk_prob,
                   fp32_router_logits=not s.shared_gate and s.num_experts == 64,
                   ep_rank=ep_rank, ep_size=ep_size, process_group=process_group, owner=owner,
                   use_graphs=use_graphs)

    # -- the three entry points -----------------------------------------------------
    def forward_device(self, x: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
        """One layer pass on device-resident rows.  With `use_graphs` the launches
        of a pass are recorded once per (input buffer, row count, output buffer)
        and replayed afterwards: a serving loop that cycles through a few fixed
        buffers pays one graph launch per step instead of ten to twenty kernel
        launches from Python.  The block's first pass runs un-recorded (one-time
        set-up must not be captured), as do batches above `max_tokens`; under expert parallelism every
        rank has to make the same sequence of calls."""
        if self._ep is not None:
            if self.use_graphs and self._warm:
                res = self._ep.forward_graphed(x, out)
            else:
                res = self._ep.forward(x, out)
                self._warm = True
            self.last_launches = self._ep.last_launches
            return res
        if not self.use_graphs or not self._warm or x.shape[0] > self.runner.max_tokens:
            return self._pass(x, out)
        if self._graph_reserve != self.runner.reserves:
            self._drop_stale_graphs()
        dst = self.runner.out[:x.shape[0]] if out is None else out
        key = (x.data_ptr(), x.shape[0], dst.data_ptr())
        if key not in self._graphs and len(self._graphs) >= 32:
            self._graphs.clear()
        return self._replayed_pass(self._graphs, key, x, dst)

    _warm = False

    def _pass(self, x: torch.Tensor, out: Optional[torch.Tensor], first_row: int = 0) -> torch.Tensor:
        res, _, _, _ = self.runner.forward(x, out, first_row)
        self._warm = True
        self.last_launches = self.runner.last_launches
        return res

    def _replayed_pass(self, graphs: dict, key, x: torch.Tensor, dst: torch.Tensor, first_row: int = 0) -> torch.Tensor:
        ent = graphs.get(key)
        if ent is None:
            stream = torch.cuda.current_stream(self.device)
            cap = torch.cuda.Stream(device=self.device)
            cap.wait_stream(stream)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.stream(cap):
                with torch.cuda.graph(graph, stream=cap, capture_error_mode="thread_local"):
                    self.runner.forward(x, dst, first_row)
            stream.wait_stream(cap)
            ent = graphs[key] = (graph, self.runner.last_launches, x, dst)
        ent[0].replay()
        self.last_launches = ent[1]
        return ent[3]

    def _drop_stale_graphs(self) -> None:
        """A larger batch has replaced the runner's buffers, which the recorded passes write to."""
        torch.cuda.synchronize(self.device)
        self._graphs.clear()
        self._part_graphs.clear()
        self._graph_reserve = self.runner.reserves

    def forward_host(self, x_host: torch.Tensor, out_host: torch.Tensor) -> None:
        """x_host, out_host: pinned bf16 [T,H].  Copies in, runs the layer, copies
        the result out; returns when `out_host` is valid."""
        t, h = x_host.shape
        if self._x_stage is None or self._x_stage.shape[0] < t:
            self._x_stage = torch.empty((max(t, self.runner.max_tokens), h), dtype=torch.bfloat16,
                                        device=self.device)
        xd = self._x_stage[:t]
        parts = self._host_parts(x_host, out_host) if t >= 3072 else 1
        if parts == 1:
            xd.copy_(x_host, non_blocking=True)
            out = self.forward_device(xd)
            out_host.copy_(out, non_blocking=True)
            torch.cuda.current_stream(self.device).synchronize()
            return
        stream = torch.cuda.current_stream(self.device)
        # Part i + 1 comes in and part i - 1 goes out while part i is in the layer (a
        # row's result does not depend on the rows around it).
        graphs = self._graphs_of_parts(xd)
        if self._copy_lanes is None:
            self._copy_lanes = torch.cuda.Stream(device=self.device), torch.cuda.Stream(device=self.device)
        inward, outward = self._copy_lanes
        inward.wait_stream(stream)
        launches = 0
        rows = [t * i // parts // 16 * 16 for i in range(parts)] + [t]
        arrived = []
        try:
            with torch.cuda.stream(inward):
                for r0, r1 in zip(rows, rows[1:]):
                    xd[r0:r1].copy_(x_host[r0:r1], non_blocking=True)
                    arrived.append(inward.record_event())
            for r0, r1, there in zip(rows, rows[1:], arrived):
                stream.wait_event(there)
                dst = self.runner.out[r0:r1]
                if graphs is None:
                    self._pass(xd[r0:r1], dst, r0)
                else:
                    self._replayed_pass(graphs, r0, xd[r0:r1], dst, r0)
                launches += self.last_launches
                outward.wait_stream(stream)
                with torch.cuda.stream(outward):
                    out_host[r0:r1].copy_(dst, non_blocking=True)
        finally:                                  # also when a part is refused: no copy outlives the call
            stream.wait_stream(inward)
            stream.wait_stream(outward)
            stream.synchronize()
        self.last_launches = launches

    _copy_lanes = None

    def _graphs_of_parts(self, xd: torch.Tensor) -> Optional[dict]:
        """The recorded passes of the parts of a staged host batch, to be replayed or to be
        recorded on the way; None where the batch runs un-recorded: without `use_graphs`
        and the first time that its size comes.  Replayed, 4096 rows in two parts take
        1060 us, launched kernel by kernel 1099 us.  Eight sizes are kept, apart from the
        graphs of `forward_device`."""
        if not self.use_graphs:
            return None
        if self._graph_reserve != self.runner.reserves:
            self._drop_stale_graphs()
        key = (xd.data_ptr(), xd.shape[0])
        if key in self._part_graphs:
            return self._part_graphs[key]
        if len(self._part_graphs) >= 8:
            self._part_graphs.clear()
        self._part_graphs[key] = {}
        return None

    def _host_parts(self, x_host: torch.Tensor, out_host: torch.Tensor) -> int:
        """Parts a host batch of at least 3072 rows is passed in.  Splitting hides all copies
        but the first part's in and the last part's out (75 ns a row each way), and costs
        the layer time that two half batches take longer than one: from 3072 rows the
        copies win (a batch below streams the expert weights twice for little).  A result
        that is not row for row the input's counterpart, or that lies over other rows of
        it, is copied as a whole."""
        tokens = x_host.shape[0]
        if self._ep is not None or tokens > self.runner.max_tokens:
            return 1
        if out_host.shape != x_host.shape:
            return 1
        if out_host.untyped_storage().data_ptr() == x_host.untyped_storage().data_ptr() and (
                out_host.data_ptr() != x_host.data_ptr() or out_host.stride() != x_host.stride()
                or out_host.dtype != x_host.dtype):
            return 1
        return max(2, tokens // 4096)

    def host_pipeline(self, depth: int = 3) -> "HostPipeline":
        """A queue for host-resident batches: copy-in, layer and copy-out of
        successive batches overlap (see `HostPipeline`)."""
        return HostPipeline(self, depth)

    def forward(self, hidden_states: torch.Tensor):
        b, s, h = hidden_states.shape
        x = hidden_states.reshape(-1, h)
        if x.dtype != torch.bfloat16:
            raise RuntimeError("B200MoeBlock computes in bf16; got %s" % x.dtype)
        out = torch.empty_like(x)
        self.forward_device(x.contiguous(), out)
        out = out.view(b, s, h)
        if not self.return_router_logits:
            return out
        return out, self.router_logits(x.shape[0])

    def router_logits(self, tokens: int) -> torch.Tensor:
        src = self._ep.logits if self._ep is not None else self.runner.logits
        return src[:tokens]

    def topk(self, tokens: int):
        r = self._ep if self._ep is not None else self.runner
        return r.topk_idx[:tokens], r.topk_w[:tokens]

    def check_status(self) -> None:
        (self._ep or self.runner).check_status()


class HostPipeline:
    """Streams host batches through a block: batch i+1 is copied to the device
    and batch i-1 is copied back while batch i is in the layer.

    `submit(x_host, out_host)` enqueues one batch (pinned bf16 [T,H] buffers) and
    returns at once; `out_host` is valid after `wait(ticket)` or `drain()`.  Each
    of `depth` slots owns a device input and output buffer; a slot is reused only
    after its copy-out has finished (an event wait on the copy-in stream, not a
    host sync).  The layer itself runs on the stream that was current when the
    pipeline was built."""

    def __init__(self, block: B200MoeBlock, depth: int = 3):
        if depth < 2:
            raise ValueError("a pipeline needs at least 2 slots")
        self.block = block
        dev = block.device
        t, h = block.runner.max_tokens, block.weights.hidden
        with torch.cuda.device(dev):
            self.compute = torch.cuda.current_stream(dev)
            self.h2d = torch.cuda.Stream(device=dev)
            self.d2h = torch.cuda.Stream(device=dev)
            self.x_dev = [torch.empty((t, h), dtype=torch.bfloat16, device=dev) for _ in range(depth)]
            self.out_dev = [torch.empty((t, h), dtype=torch.bfloat16, device=dev) for _ in range(depth)]
            self.ev_in = [torch.cuda.Event() for _ in range(depth)]
            self.ev_done = [torch.cuda.Event() for _ in range(depth)]
            self.ev_out = [torch.cuda.Event() for _ in range(depth)]
        self.depth = depth
        self.count = 0

    def submit(self, x_host: torch.Tensor, out_host: torch.Tensor) -> int:
        t = x_host.shape[0]
        if t > self.x_dev[0].shape[0]:
            raise RuntimeError("pipeline was sized for %d rows, got %d" % (self.x_dev[0].shape[0], t))
        slot = self.count % self.depth
        xd, od = self.x_dev[slot][:t], self.out_dev[slot][:t]
        if self.count >= self.depth:
            self.h2d.wait_event(self.ev_out[slot])          # the slot's previous result has left the device
        with torch.cuda.stream(self.h2d):
            xd.copy_(x_host, non_blocking=True)
            self.ev_in[slot].record(self.h2d)
        self.compute.wait_event(self.ev_in[slot])
        with torch.cuda.stream(self.compute):
            self.block.forward_device(xd, od)
            self.ev_done[slot].record(self.compute)
        self.d2h.wait_event(self.ev_done[slot])
        with torch.cuda.stream(self.d2h):
            out_host.copy_(od, non_blocking=True)
            self.ev_out[slot].record(self.d2h)
        self.count += 1
        return self.count - 1

    def wait(self, ticket: int) -> None:
        """Blocks until the result of `submit` number `ticket` is in its host buffer
        (only the last `depth` tickets can still be waited for)."""
        if ticket < self.count - self.depth or ticket >= self.count:
            raise ValueError("ticket %d is not in flight" % ticket)
        self.ev_out[ticket % self.depth].synchronize()

    def drain(self) -> None:
        self.d2h.synchronize()
        self.compute.synchronize()
