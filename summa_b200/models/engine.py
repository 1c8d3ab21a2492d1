"""Inference engine: prefill + greedy decode over a KV cache, optionally tensor-parallel and
4-bit group-quantised.

`InferenceEngine.build` creates the model directly on the device (random-init or from a
state dict), shards it across the tensor-parallel group, quantises the block projections to
int4 g128 and allocates the KV cache. `prefill` uses the sequence-parallel fused
all-gather->GEMM / GEMM->reduce-scatter kernels when the token count allows and falls back
to the all-reduce form otherwise; `decode` runs one token per sequence per step: weight-
streaming int4 GEMV, split-KV decode attention, one-shot peer-memory all-reduce, device
argmax. The reference's generator is single-device (`summa-llm/src/generate.rs:127-250`).
"""
from __future__ import annotations

import os
from typing import Optional

import torch

from .. import ops
from .transformer import Transformer

# SUMMA_DECODE_FUSED_EPILOGUES=0: separate RoPE-append and SwiGLU kernels behind plain decode projections instead
# of the streaming kernel's fused epilogues
_FUSED_EPILOGUES = os.environ.get("SUMMA_DECODE_FUSED_EPILOGUES", "1") == "1"


class InferenceEngine:
    def __init__(self, model: Transformer, tp=None):
        self.model = model
        self.tp = tp
        self.state = None
        self.device = model.embedding.weight.device
        self.use_graph = True
        self._graph = None

    @classmethod
    def build(cls, cfg, device: torch.device, tp_group=None, quantize: Optional[str] = "int4",
              init_std: float = 0.02, seed: int = 0, max_prefill_tokens: int = 0, state_dict=None,
              quantize_head: bool = False):
        torch.manual_seed(seed)                      # every rank draws the same full model, then keeps its shard
        with torch.device(device):
            model = Transformer(cfg, init_std=init_std)
        if state_dict is not None:
            model.load_state_dict(state_dict)
        model.prepare_inference(torch.bfloat16)
        tp = None
        if tp_group is not None:
            import torch.distributed as dist
            from ..parallel.tp import TensorParallelGroup, shard_model
            if dist.get_world_size(tp_group) > 1:
                mt = max_prefill_tokens
                if mt:
                    step = 128 * dist.get_world_size(tp_group)
                    mt = -(-mt // step) * step
                tp = TensorParallelGroup(tp_group, device, mode="fused", max_tokens=mt, hidden=cfg.hidden_size)
                shard_model(model, tp)
                torch.cuda.empty_cache()
        if quantize == "int4":
            from .quantized import quantize_model_int4
            quantize_model_int4(model, include_head=quantize_head)
            torch.cuda.empty_cache()
        elif quantize not in (None, "none"):
            raise ValueError(f"unknown quantisation `{quantize}`")
        return cls(model, tp)

    def reset(self, batch: int, capacity: int):
        """Start a new set of sequences. A state of the same shape is recycled (the KV caches are
        overwritten as the new sequences grow, recurrent states start anew), which also keeps the captured decode graph."""
        st = self.state
        if st is not None and st.capacity == capacity and st.layers \
                and all((l.k if hasattr(l, "length") else l.conv).shape[0] == batch for l in st.layers):
            for i, l in enumerate(st.layers):
                if hasattr(l, "length"):
                    l.length = 0
                else:
                    st.layers[i] = self.model.layers[i].ssm.make_state(batch, l.h.device, l.conv.dtype)
            st.pos = 0
            return
        self.state = self.model.make_state(batch, capacity)
        self._graph = None

    @torch.no_grad()
    def prefill(self, tokens: torch.Tensor) -> torch.Tensor:
        """Consumes the prompt `[B, S]`; returns the greedy next token `[B, 1]`."""
        if self.state is None:
            raise RuntimeError("call reset(batch, capacity) first")
        if self.tp is not None:
            from ..parallel.tp import prefill_sequence_parallel
            logits = prefill_sequence_parallel(self.model, self.tp, tokens, self.state)
        else:
            logits = self.model.forward_next_logits_with_state(tokens, self.state)
        return ops.argmax(logits).view(-1, 1)

    @torch.no_grad()
    def decode(self, first: torch.Tensor, steps: int) -> torch.Tensor:
        """Greedy-decodes `steps` tokens after `first` `[B, 1]`; returns `[B, steps]` (the
        tokens produced, not including `first`). No steps: an empty tensor, and the state stays as it is."""
        if steps < 0:
            raise ValueError(f"cannot decode {steps} tokens")
        if steps == 0:
            return torch.empty(first.shape[0], 0, dtype=torch.long, device=first.device)
        if self.use_graph and self.device.type == "cuda" and not _has_hooks(self.model):
            if self._graph is None:
                self._graph = _GraphDecoder.try_build(self.model, self.state, steps)
            if self._graph is not None and self._graph.max_steps >= steps:
                return self._graph.run(first, steps)
        out = []
        tok = first
        for _ in range(steps):
            logits = self.model.forward_next_logits_with_state(tok, self.state)
            tok = ops.argmax(logits).view(-1, 1)
            out.append(tok)
        return torch.cat(out, dim=1)


def _has_hooks(model) -> bool:
    """Whether something watches or changes module calls: the captured step goes past the modules, so such a model decodes eagerly."""
    from torch.nn.modules import module as M
    return bool(M._global_forward_hooks or M._global_forward_pre_hooks
                or any(m._forward_hooks or m._forward_pre_hooks for m in model.modules()))


class _GraphDecoder:
    """One decode step captured in a CUDA graph. Everything that changes from step to step (the
    token, the position, the output column) lives in device memory: RoPE + cache append and the
    split-KV attention read the position on the device, the tensor-parallel all-reduce keeps its
    call number on the device, so a replay needs no host input at all."""

    @classmethod
    def try_build(cls, model, state, max_steps: int):
        from .layers import FeedForward, MultiHeadAttention
        from ..ops import cuda_ops
        cfgm = model.cfg
        for blk in model.layers:
            if not blk.pre_norm or not blk.residual or blk.memory is not None or not isinstance(blk.feed_forward, FeedForward):
                return None
            a = blk.attention
            if blk.ssm is not None:
                if not cuda_ops.mamba_decode_usable(blk.ssm):
                    return None
            elif (not isinstance(a, MultiHeadAttention) or a.head_dim != 128 or a.window is not None or a.q_norm is not None
                    or not a.use_rope or not a.causal or a.num_heads // a.num_kv_heads > 8):
                return None
        table = model.embedding.weight
        if (cfgm.embeddings.scale is not None or model.stream_dtype != torch.bfloat16 or table.dtype != torch.bfloat16
                or not table.is_contiguous() or table.shape[1] % 2):
            return None
        return cls(model, state, max_steps)

    def __init__(self, model, state, max_steps: int):
        from ..ops import native
        self.model, self.state, self.max_steps = model, state, max_steps
        self.attn = [i for i, blk in enumerate(model.layers) if blk.ssm is None]
        self.ssm = [i for i, blk in enumerate(model.layers) if blk.ssm is not None]
        dev = model.embedding.weight.device
        st0 = state.layers[0]
        self.B = (st0.conv if self.ssm and self.ssm[0] == 0 else st0.k).shape[0]
        self.cap = state.layers[self.attn[0]].k.shape[1] if self.attn else state.capacity
        # The captured step updates recurrent states of its own: a prefill leaves its results in fresh tensors, which `run`
        # copies in, and callers get copies back.
        self.rec = {i: (torch.empty_like(state.layers[i].conv, dtype=torch.bfloat16), torch.empty_like(state.layers[i].h))
                    for i in self.ssm}
        self.tok = torch.zeros(self.B, 1, dtype=torch.long, device=dev)
        self.pos = torch.zeros(1, dtype=torch.int32, device=dev)
        self.col = torch.zeros(1, 1, dtype=torch.long, device=dev)
        self.out = torch.zeros(self.B, max_steps, dtype=torch.long, device=dev)
        if self.attn:                            # (the largest of the blocks: their head counts may differ)
            heads = {model.layers[i].attention.num_kv_heads for i in self.attn}
            self.splits = {k: native.call_value("sb_attention_decode_splits", self.B, k, self.cap) for k in heads}
            need = max(native.call_value("sb_attention_decode_workspace", self.B, k, n) for k, n in self.splits.items())
            self.ws = torch.empty(need, dtype=torch.float32, device=dev)
        P, I, L, F = native.P, native.I, native.L, native.F
        native.register("sb_decode_rope_append", [P] * 6 + [I, I, I, I, L, P, I, P])
        native.register("sb_decode_embed", [P, P, P, I, I, L, P, P, P])
        native.register("sb_decode_pick", [P, P, I, I, L, I, P, P, L, P])
        native.register("sb_attention_decode_dyn", [P] * 5 + [I, I, I, P, I, I, I] + [P] * 4 + [F, I, P])
        self.graph = None

    def _step(self):
        from ..ops import native
        from .quantized import QuantLinear, in_proj_swiglu
        m, B = self.model, self.B
        table = m.embedding.weight
        h = torch.empty(B, table.shape[1], dtype=torch.bfloat16, device=table.device)
        native.call("sb_decode_embed", self.tok.data_ptr(), table.data_ptr(), h.data_ptr(), B, table.shape[1], table.shape[0],
                    self.pos.data_ptr(), self.col.data_ptr(), native.stream())
        cos, sin = m.rope(h.device) or (None, None)
        for i, (blk, st) in enumerate(zip(m.layers, self.state.layers)):
            if blk.ssm is not None:
                from ..ops import cuda_ops
                xz = self._norm_proj(blk.attn_norm, blk.ssm.in_proj, h)
                h = self._proj_add(blk.ssm.out_proj, cuda_ops.mamba_decode_step(blk.ssm, xz, *self.rec[i]), h)
            else:
                h = self._attend(blk, st, h, cos, sin)
            ff = blk.feed_forward
            if _FUSED_EPILOGUES and ff.gated and ff.act in ("swiglu", "silu") and getattr(blk.ffn_norm, "kind", None) == "rmsnorm" and h.shape[0] <= 4 and isinstance(ff.in_proj, QuantLinear):
                u = in_proj_swiglu(ff.in_proj, h, norm=(blk.ffn_norm.gamma, blk.ffn_norm.eps))
            else:
                u = self._norm_proj(blk.ffn_norm, ff.in_proj, h)
                u = ops.gated_act(u, ff.act) if ff.gated else ops.activation(ff.act, u)
            h = self._proj_add(ff.down_proj, u, h)
        head = m.lm_head
        logits = (m.project_logits(m.final_norm(h)) if head is None
                  else self._norm_proj(m.final_norm, head, h)[..., :m.cfg.vocab_size])
        native.call("sb_decode_pick", logits.data_ptr(), self.out.data_ptr(), B, logits.shape[1], logits.stride(0),
                    1 if logits.dtype == torch.bfloat16 else 0, self.tok.data_ptr(), self.col.data_ptr(), self.out.stride(0),
                    native.stream())

    def _attend(self, blk, st, h, cos, sin):
        """The attention branch of a block with its residual: qkv projection, RoPE, cache append, split-KV attention, o_proj."""
        import ctypes
        from ..ops import native
        B, a = self.B, blk.attention
        cs = (ctypes.c_long * 3)(st.k.stride(0), st.k.stride(1), st.k.stride(2))
        if self._rope_fusable(blk, h):
            from ..ops import cuda_ops
            k8, scales, settled = a.qkv_proj.decode_operands()
            qkv = cuda_ops.int4_gemv_rope_append(h, k8, scales, (blk.attn_norm.gamma, blk.attn_norm.eps), cos, sin, st.k, st.v,
                                                 self.pos, a.num_heads, a.num_kv_heads, a.head_dim, self.cap, settled)
        else:
            qkv = self._norm_proj(blk.attn_norm, a.qkv_proj, h)
            native.call("sb_decode_rope_append", qkv.data_ptr(), cos.data_ptr(), sin.data_ptr(), st.k.data_ptr(),
                        st.v.data_ptr(), self.pos.data_ptr(), B, a.num_heads, a.num_kv_heads, a.head_dim,
                        qkv.stride(0), cs, self.cap, native.stream())
        o = torch.empty(B, a.q_dim, dtype=torch.bfloat16, device=h.device)
        qs = (ctypes.c_long * 2)(qkv.stride(0), a.head_dim)
        os_ = (ctypes.c_long * 2)(o.stride(0), a.head_dim)
        native.call("sb_attention_decode_dyn", qkv.data_ptr(), st.k.data_ptr(), st.v.data_ptr(), o.data_ptr(),
                    self.ws.data_ptr(), B, a.num_heads, a.num_kv_heads, self.pos.data_ptr(), 1, self.cap, a.head_dim,
                    qs, cs, cs, os_, 1.0 / a.head_dim ** 0.5, self.splits[a.num_kv_heads], native.stream())
        return self._proj_add(a.o_proj, o, h)

    @staticmethod
    def _rope_fusable(blk, h) -> bool:
        """RMSNorm -> quantised qkv projection -> RoPE -> cache append as one kernel (<= 4 rows)."""
        from .quantized import QuantLinear
        a = blk.attention
        p = a.qkv_proj
        return (_FUSED_EPILOGUES and isinstance(p, QuantLinear) and p.bias is None and h.shape[0] <= 4
                and h.dtype == torch.bfloat16
                and getattr(blk.attn_norm, "kind", None) == "rmsnorm" and a.q_norm is None and a.k_norm is None
                and a.use_rope
                and p.d_in % 128 == 0 and p.d_in <= 20480 and h.is_contiguous()
                and p.d_out == (a.num_heads + 2 * a.num_kv_heads) * a.head_dim)

    @staticmethod
    def _norm_proj(norm, proj, h):
        """proj(norm(h)); an RMSNorm in front of a projection runs inside its GEMV kernel."""
        from .layers import Linear
        from .quantized import QuantLinear
        if getattr(norm, "kind", None) == "rmsnorm":
            if isinstance(proj, QuantLinear) and h.shape[0] <= 4:
                return proj(h, norm=(norm.gamma, norm.eps))
            if type(proj) is Linear and h.is_cuda:
                from ..ops import cuda_ops
                return cuda_ops.decode_linear(h, proj.weight, proj.bias, norm=(norm.gamma, norm.eps))
        return proj(norm(h))

    @staticmethod
    def _proj_add(proj, x, h):
        """h + proj(x), with the add fused into the projection's epilogue when it can be."""
        from .layers import Linear
        from .quantized import QuantLinear
        from ..parallel.tp import RowParallelLinear
        if isinstance(proj, (QuantLinear, RowParallelLinear)):
            return proj(x, residual=h)
        if type(proj) is Linear and x.is_cuda:
            from ..ops import cuda_ops
            return cuda_ops.decode_linear(x, proj.weight, proj.bias, residual=h)
        return h + proj(x)

    def _capture(self, step_bytes: int):
        """Captures the step. `torch.cuda.graph` hands the allocator's cached blocks back to the driver first, about 2 ms per GB
        of them (a first hybrid request behind 40 GB of cache: 96 to 119 ms, 66 without a graph). That only happens here if what
        the step allocates in all (`step_bytes`, counted over the eager step) would not surely fit the free memory."""
        torch.cuda.synchronize()
        if torch.cuda.mem_get_info()[0] < 2 * step_bytes + (1 << 30):
            torch.cuda.empty_cache()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.stream(torch.cuda.Stream()):
            g.capture_begin()
            try:
                self._step()
            finally:
                g.capture_end()
        self.graph = g

    def run(self, first: torch.Tensor, steps: int) -> torch.Tensor:
        start = self.state.layers[self.attn[0]].length if self.attn else self.state.pos
        if self.attn and start + steps > self.cap:
            raise RuntimeError(f"KV cache overflow: {start + steps} > capacity {self.cap}")
        for i, (conv, hid) in self.rec.items():
            conv.copy_(self.state.layers[i].conv)
            hid.copy_(self.state.layers[i].h)
        self.tok.copy_(first)
        self.pos.fill_(start - 1)                         # the step's first kernel moves both on
        self.col.fill_(-1)
        done = 0
        if self.graph is None:
            allocated = "allocated_bytes.all.allocated"
            before = torch.cuda.memory_stats().get(allocated, 0)
            self._step()                                  # eager: warms every lazy allocation and attribute
            done = 1
            if steps > 1:
                self._capture(torch.cuda.memory_stats().get(allocated, 0) - before)
        for _ in range(steps - done):
            self.graph.replay()
        for i in self.attn:
            self.state.layers[i].length = start + steps
        for i, (conv, hid) in self.rec.items():
            self.state.layers[i].conv = conv.to(self.state.layers[i].conv.dtype, copy=True)
            self.state.layers[i].h = hid.clone()
        self.state.pos += steps
        return self.out[:, :steps].clone()
