"""Decoder forward / backward on the flat parameter layout.

Two executors over the SAME parameters and the SAME packed-batch contract:

* ``OracleDecoder``  - plain PyTorch (autograd), any device, any float dtype. It is the CPU plumbing
  path and the numerical oracle.
* ``NativeDecoder``  - sm_100a kernels with an explicit, hand-scheduled backward (no autograd graph):
  tcgen05 GEMMs with fused bias / residual epilogues, RMSNorm / RoPE / SwiGLU kernels, varlen
  flash-attention forward / backward, fused lm_head loss. Gradients accumulate in fp32 into a
  ``GradSink`` so the sharded optimizer can reduce them unit by unit.

Both replace the HF Qwen2 body + loss shim the reference runs (grpo_loss.py:40-144,
gpu_process_worker.py:963-1050).
"""
from __future__ import annotations

import math
from dataclasses import dataclass
from typing import Any, List, Optional, Tuple

import torch

from ..ops import reference as R
from ..packing import PackedBatch
from .config import ModelConfig
from .layout import ParamLayout


@dataclass
class LossConfig:
    clip_low: float = 0.2
    clip_high: float = 0.28
    clip_ratio_c: float = 3.0
    kl_beta: float = 0.0
    temperature: float = 1.0
    entropy_coeff: float = 0.0
    apply_entropy_bonus: bool = True


# =====================================================================================================
# Oracle
# =====================================================================================================
class OracleDecoder:
    def __init__(self, cfg: ModelConfig, layout: ParamLayout, params: torch.Tensor):
        self.cfg, self.layout, self.params = cfg, layout, params
        self._rope: Optional[Tuple[torch.Tensor, torch.Tensor]] = None

    def _rope_tables(self, device, need: int):
        if self._rope is None or self._rope[0].shape[0] < need or self._rope[0].device != device:
            n = max(need, min(self.cfg.max_position_embeddings, 4096))
            self._rope = R.rope_tables(self.cfg.head_dim, n, self.cfg.rope_theta, device)
        return self._rope

    def w(self, name: str) -> torch.Tensor:
        return self.layout.view(self.params, name)

    def hidden(self, ids: torch.Tensor, pos: torch.Tensor, cu_seqlens: List[int]) -> torch.Tensor:
        cfg = self.cfg
        cos_t, sin_t = self._rope_tables(ids.device, int(pos.max().item()) + 1 if pos.numel() else 1)
        x = self.w("embed")[ids.long()]
        T = x.shape[0]
        for i in range(cfg.num_hidden_layers):
            p = f"layers.{i}."
            h = R.rmsnorm(x, self.w(p + "ln1"), cfg.rms_norm_eps)
            qkv = h @ self.w(p + "wqkv").t()
            if cfg.attention_bias:
                qkv = qkv + self.w(p + "bqkv")
            q = qkv[:, :cfg.q_dim].reshape(T, cfg.num_attention_heads, cfg.head_dim)
            k = qkv[:, cfg.q_dim:cfg.q_dim + cfg.kv_dim].reshape(T, cfg.num_key_value_heads, cfg.head_dim)
            v = qkv[:, cfg.q_dim + cfg.kv_dim:].reshape(T, cfg.num_key_value_heads, cfg.head_dim)
            q = R.apply_rope(q, pos, cos_t, sin_t)
            k = R.apply_rope(k, pos, cos_t, sin_t)
            a = R.attention_varlen(q, k, v, cu_seqlens).reshape(T, cfg.q_dim)
            x = x + a @ self.w(p + "wo").t()
            h2 = R.rmsnorm(x, self.w(p + "ln2"), cfg.rms_norm_eps)
            x = x + R.swiglu(h2 @ self.w(p + "wgu").t()) @ self.w(p + "wd").t()
        return R.rmsnorm(x, self.w("final_norm"), cfg.rms_norm_eps)

    def logprobs(self, batch: PackedBatch, temperature: float) -> Tuple[torch.Tensor, torch.Tensor]:
        cu = batch.cu_seqlens.tolist()
        hn = self.hidden(batch.ids, batch.pos, cu)
        return R.lmhead_logprob_entropy(hn, self.w(self.layout.lm_head_name()), batch.labels, temperature)

    def loss(self, batch: PackedBatch, lc: LossConfig, loss_scale: float) -> Tuple[torch.Tensor, torch.Tensor]:
        """Scaled microbatch loss (token mean * loss_scale) and the stats sums vector."""
        logp, ent = self.logprobs(batch, lc.temperature)
        ref = batch.ref_logprobs if lc.kl_beta > 0 else None
        loss_sum, stats = R.grpo_token_loss(logp, batch.old_logprobs, ref, batch.advantages, batch.labels, lc.clip_low,
                                            lc.clip_high, lc.clip_ratio_c, lc.kl_beta, ent, batch.old_entropies)
        denom = max(1.0, float(stats[0]))
        return loss_sum / denom * loss_scale, stats


# =====================================================================================================
# Native
# =====================================================================================================
class GradSink:
    """Where weight gradients go. ``unit_grads(u)`` returns an fp32 buffer covering unit ``u`` of the layout
    (kernels accumulate into it); ``unit_done(u)`` tells the owner that the unit's backward has finished."""

    def __init__(self, layout: ParamLayout, device, flat: Optional[torch.Tensor] = None):
        self.layout = layout
        self.flat = flat if flat is not None else torch.zeros(layout.total, dtype=torch.float32, device=device)

    def view(self, name: str) -> torch.Tensor:
        return self.layout.view(self.flat, name)

    def unit_done(self, unit: int) -> None:  # overridden by the sharded trainer
        pass

    def zero_(self) -> None:
        self.flat.zero_()


# Work of the output matrix on rows without a loss from which on those rows are left out: 50 us at 1.4 PFLOP/s, twice what the
# gather, the scatter and their allocations take (a model of 2048 x 512: 1.56 ms an update with all rows, 1.61 without).
LOSS_ROWS_MIN_FLOPS = 7e10


def vocab_chunk(T: int, asked: Optional[int] = None) -> int:
    """Columns of the dlogits buffer of ``T`` rows: what the caller asks for, else 15360 but at most 1 GiB, and at least 4096. A
    wide chunk reads and writes the fp32 dH sum seldom and fills the pairs' waves: 10 chunks of 151936 columns take about 0.8 of
    the time of 38."""
    if asked is not None:
        return asked
    return max(4096, min(15360, (1 << 29) // max(T, 1) // 256 * 256))


def kept_columns(rows: int, V: int, memory: float, step: int) -> int:
    """Leading columns of [rows, V] fp32 logits that ``memory`` bytes hold: all (rounded up to 8), or whole chunks of ``step``, since
    the backward pass reads no part of one."""
    cols = max(0, int(memory)) // (4 * rows)
    every = (V + 7) // 8 * 8
    return every if cols >= every else cols // step * step


class NativeDecoder:
    def __init__(self, cfg: ModelConfig, layout: ParamLayout, params: Optional[torch.Tensor], recompute: bool = False,
                 lmhead_chunk: Optional[int] = None, weights: Any = None):
        """``params`` is the resident flat bf16 parameter buffer. With ``weights`` (parallel/zero3.py::ShardedWeights)
        there is no resident copy: each unit is gathered from its owners just before use, the gather of the next unit
        riding on a GEMM launch of the current one. ``lmhead_chunk`` is the width of the dlogits buffer in columns of the
        vocabulary (None: by the number of rows, see ``vocab_chunk``)."""
        from ..ops import native

        self.C = native()
        self.weights = weights
        if weights is None:
            assert params is not None and params.is_cuda and params.dtype == torch.bfloat16
            self.dev = params.device
        else:
            self.dev = weights.device
        self.cfg, self.layout, self.params = cfg, layout, params
        self.recompute = recompute
        self.lmhead_chunk = lmhead_chunk
        self.status = torch.zeros(1, dtype=torch.int32, device=self.dev)
        if weights is not None:
            weights.status = self.status
        self._rope: Optional[Tuple[torch.Tensor, torch.Tensor]] = None
        self.n_stats = int(self.C.grpo_num_loss_stats())
        # resident parameters: a layer is one native call (offsets of its tensors in the flat buffer)
        self._dims = [cfg.hidden_size, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim, cfg.intermediate_size]
        self._offs = [[layout.segments[f"layers.{i}.{n}"].offset if f"layers.{i}.{n}" in layout.segments else -1
                       for n in ("ln1", "wqkv", "bqkv", "wo", "ln2", "wgu", "wd")] for i in range(cfg.num_hidden_layers)]
        self.launches = 0  # kernels of this package launched (bench bookkeeping)
        self.memory_share = 1.0  # of the device, what this process's roles are to stay within (kept logits only)
        self._asked = (-1, 0)  # what the allocator held when the device was last asked, and the free memory then

    # ---- helpers ----
    def w(self, name: str) -> torch.Tensor:
        if self.weights is not None:
            return self.weights.view(name)
        return self.layout.view(self.params, name)

    def _enter_unit(self, unit: int, then: Optional[int]) -> None:
        """Sharded weights only: ``unit`` must be staged now; ``then`` is the unit needed after it (prefetched by the
        next large GEMM launch)."""
        if self.weights is not None:
            self.launches += self.weights.enter(unit, then)

    def rope_tables(self, need: int = 1):
        if self._rope is None or self._rope[0].shape[0] < need:
            n = max(need, min(self.cfg.max_position_embeddings, 131072))
            cos_t, sin_t = R.rope_tables(self.cfg.head_dim, n, self.cfg.rope_theta, "cpu")
            self._rope = (cos_t.to(self.dev), sin_t.to(self.dev))
        return self._rope

    def check_status(self) -> None:
        code = int(self.status.item())
        if code != 0:
            self.status.zero_()
            raise RuntimeError(f"device kernel reported status {code} (bounded wait ran out or bad index)")

    def _gemm(self, a, b, out, a_mn=False, b_mn=False, bias=None, accumulate=False, residual=None):
        if self.weights is not None and self.weights.wants_ride(a, b):
            self.weights.gemm_with_prefetch(a, b, out, a_mn, b_mn, bias, accumulate, self.status, residual)
        else:
            self.C.gemm_bf16(a, b, out, a_mn, b_mn, bias, 1.0, accumulate, self.status, residual)
        self.launches += 1
        return out

    def _wgrad(self, dy, x, name: str, sink) -> None:
        """dW[name] += dy^T x. A scatter sink adds the tile straight into the owners' gradient shards (GEMM fused with
        the reduce-scatter); the plain sink accumulates into the local fp32 buffer."""
        if getattr(sink, "scatter", False):
            sink.wgrad(dy, x, name, self.status)
        else:
            self.C.gemm_bf16(dy, x, sink.view(name), True, True, None, 1.0, True, self.status, None)
        self.launches += 1

    def _qkv(self, h: torch.Tensor, p: str, qkv: torch.Tensor, pos: torch.Tensor, cos_t: torch.Tensor, sin_t: torch.Tensor) -> None:
        """Rotated q, k and v of the rows: one launch, or the plain GEMM and the rotation kernel, with the same bits."""
        cfg = self.cfg
        rot = cfg.num_attention_heads + cfg.num_key_value_heads
        w, bias = self.w(p + "wqkv"), self.w(p + "bqkv") if cfg.attention_bias else None
        if self.weights is None and self.C.gemm_qkv_rope(h, w, qkv, bias, pos, cos_t, sin_t, rot, cfg.head_dim, self.status):
            self.launches += 1
            return
        self._gemm(h, w, qkv, bias=bias)
        self.C.rope_inplace(qkv, pos, cos_t, sin_t, rot, cfg.head_dim, False)
        self.launches += 1

    def _mlp_in(self, h: torch.Tensor, w: torch.Tensor, keep: bool) -> Tuple[Optional[torch.Tensor], torch.Tensor]:
        """(gate / up projections if they are to be kept for the backward pass, SwiGLU activation): one launch, or the plain
        GEMM (which carries the prefetch of sharded weights) and the elementwise kernel, with the same bits."""
        T, F = h.shape[0], self.cfg.intermediate_size
        act = self._new(T, F)
        gu = self._new(T, 2 * F) if keep else None
        if self.weights is None and self.C.gemm_mlp_in(h, w, act, gu, self.status):
            self.launches += 1
            return gu, act
        if gu is None:
            gu = self._new(T, 2 * F)
        self._gemm(h, w, gu)
        self.C.swiglu_fwd(gu, act)
        self.launches += 1
        return gu, act

    def _new(self, *shape, dtype=torch.bfloat16):
        return torch.empty(shape, dtype=dtype, device=self.dev)

    # ---- layer forward ----
    def _layer_fwd(self, i: int, x: torch.Tensor, batch: PackedBatch, cos_t, sin_t, save: Optional[dict],
                   kv_write: Optional[tuple] = None, next_unit: Optional[int] = None):
        cfg, C = self.cfg, self.C
        if self.weights is None:
            k_cache, v_cache, slots, head0 = (tuple(kv_write) + (0,))[:4] if kv_write is not None else (None, None, None, 0)
            out, slab, n = C.layer_fwd(self.params, self._offs[i], self._dims, cfg.rms_norm_eps, x, batch.pos, batch.tiles, cos_t, sin_t,
                                       self.status, save is not None, slots, k_cache, v_cache, head0)
            self.launches += n
            if save is not None:
                save.update(x=x, slab=slab)
            return out
        T = x.shape[0]
        p = f"layers.{i}."
        self._enter_unit(i + 1, next_unit)
        h1 = self._new(T, cfg.hidden_size)
        rstd1 = self._new(T, dtype=torch.float32)
        C.rmsnorm_fwd(x, self.w(p + "ln1"), h1, rstd1, cfg.rms_norm_eps)
        qkv = self._new(T, cfg.qkv_dim)
        self._qkv(h1, p, qkv, batch.pos, cos_t, sin_t)
        if kv_write is not None:  # rollout prefill: K/V of every prompt token go to their cache slots
            k_cache, v_cache, slots, head0 = (tuple(kv_write) + (0,))[:4]  # tensor-parallel engine rank: its share of the kv heads
            C.kv_cache_write(qkv, slots, k_cache, v_cache, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim,
                             self.status, head0)
            self.launches += 1
        attn = self._new(T, cfg.q_dim)
        lse = self._new(cfg.num_attention_heads, T, dtype=torch.float32)
        C.attn_varlen_fwd(qkv, attn, lse, batch.tiles, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim,
                          1.0 / math.sqrt(cfg.head_dim), self.status)
        x1 = self._new(T, cfg.hidden_size)
        self._gemm(attn, self.w(p + "wo"), x1, residual=x)
        h2 = self._new(T, cfg.hidden_size)
        rstd2 = self._new(T, dtype=torch.float32)
        C.rmsnorm_fwd(x1, self.w(p + "ln2"), h2, rstd2, cfg.rms_norm_eps)
        gu, act = self._mlp_in(h2, self.w(p + "wgu"), save is not None)
        x2 = self._new(T, cfg.hidden_size)
        self._gemm(act, self.w(p + "wd"), x2, residual=x1)
        self.launches += 3
        if save is not None:
            save.update(x=x, h1=h1, rstd1=rstd1, qkv=qkv, attn=attn, lse=lse, x1=x1, h2=h2, rstd2=rstd2, gu=gu, act=act)
        return x2

    def layer_fwd_suffix(self, i: int, x: torch.Tensor, batch: PackedBatch, sfx: torch.Tensor, pfx: torch.Tensor,
                         pos_s: torch.Tensor, cos_t, sin_t, k_cache: torch.Tensor, v_cache: torch.Tensor, slots: torch.Tensor,
                         pfx_blk: torch.Tensor, pfx_off: torch.Tensor) -> torch.Tensor:
        """Layer forward for a rollout prefill whose leading prompt tokens are already in the KV cache (prefix caching).
        ``x`` holds the rows of the tokens that still have to be computed (packed positions ``sfx`` of ``batch``, which
        describes the whole prompts). Projections and MLP run on those rows only; attention runs over the whole prompts
        with the keys / values of the cached tokens (packed positions ``pfx``, cache block / offset ``pfx_blk`` /
        ``pfx_off``) gathered from the cache. The query rows of cached tokens are zero and their outputs are dropped."""
        cfg, C = self.cfg, self.C
        Ts, T = x.shape[0], batch.T
        Hq, Hkv, D = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim
        p = f"layers.{i}."
        self._enter_unit(i + 1, None)
        h1 = self._new(Ts, cfg.hidden_size)
        C.rmsnorm_fwd(x, self.w(p + "ln1"), h1, None, cfg.rms_norm_eps)
        qkv_s = self._new(Ts, cfg.qkv_dim)
        self._qkv(h1, p, qkv_s, pos_s, cos_t, sin_t)
        C.kv_cache_write(qkv_s, slots, k_cache, v_cache, Hq, Hkv, D, self.status, 0)
        qkv = torch.zeros(T, cfg.qkv_dim, dtype=torch.bfloat16, device=x.device)
        qkv.index_copy_(0, sfx, qkv_s)
        heads = qkv.view(T, Hq + 2 * Hkv, D)
        heads[pfx, Hq:Hq + Hkv] = k_cache[pfx_blk, :, pfx_off]   # [cached tokens, Hkv, D]
        heads[pfx, Hq + Hkv:] = v_cache[pfx_blk, :, pfx_off]
        attn = self._new(T, cfg.q_dim)
        lse = self._new(Hq, T, dtype=torch.float32)
        C.attn_varlen_fwd(qkv, attn, lse, batch.tiles, Hq, Hkv, D, 1.0 / math.sqrt(D), self.status)
        attn_s = attn.index_select(0, sfx)
        x1 = self._new(Ts, cfg.hidden_size)
        self._gemm(attn_s, self.w(p + "wo"), x1, residual=x)
        h2 = self._new(Ts, cfg.hidden_size)
        C.rmsnorm_fwd(x1, self.w(p + "ln2"), h2, None, cfg.rms_norm_eps)
        _, act = self._mlp_in(h2, self.w(p + "wgu"), False)
        x2 = self._new(Ts, cfg.hidden_size)
        self._gemm(act, self.w(p + "wd"), x2, residual=x1)
        self.launches += 4
        return x2

    def _layer_bwd(self, i: int, dx: torch.Tensor, s: dict, batch: PackedBatch, cos_t, sin_t, sink: GradSink):
        """dx (bf16 [T, H]) is the gradient w.r.t. the layer output; it is updated in place to the gradient w.r.t. the input."""
        cfg, C = self.cfg, self.C
        if self.weights is None:
            self.launches += C.layer_bwd(self.params, sink.flat, self._offs[i], self._dims, cfg.rms_norm_eps, dx, s["x"], s["slab"], batch.pos,
                                         batch.tiles, cos_t, sin_t, self.status)
            sink.unit_done(i + 1)
            return
        T = dx.shape[0]
        p = f"layers.{i}."
        self._enter_unit(i + 1, i if i > 0 else None)
        # ---- MLP ----
        dgu = self._new(T, 2 * cfg.intermediate_size)
        dact = self._new(T, cfg.intermediate_size)
        self._gemm(dx, self.w(p + "wd"), dact, b_mn=True)
        C.swiglu_bwd(s["gu"], dact, dgu)
        del dact
        self._wgrad(dx, s["act"], p + "wd", sink)
        dh2 = self._new(T, cfg.hidden_size)
        self._gemm(dgu, self.w(p + "wgu"), dh2, b_mn=True)
        self._wgrad(dgu, s["h2"], p + "wgu", sink)
        del dgu
        C.rmsnorm_bwd(dh2, s["x1"], self.w(p + "ln2"), s["rstd2"], dx, sink.view(p + "ln2"), True)
        # ---- attention ----
        dattn = self._new(T, cfg.q_dim)
        self._gemm(dx, self.w(p + "wo"), dattn, b_mn=True)
        self._wgrad(dx, s["attn"], p + "wo", sink)
        dqkv = self._new(T, cfg.qkv_dim)
        delta = self._new(cfg.num_attention_heads, T, dtype=torch.float32)
        dq_acc = self._new(T, cfg.q_dim, dtype=torch.float32)
        C.attn_varlen_bwd(s["qkv"], s["attn"], dattn, s["lse"], delta, dq_acc, dqkv, batch.tiles, cfg.num_attention_heads,
                          cfg.num_key_value_heads, cfg.head_dim, 1.0 / math.sqrt(cfg.head_dim), self.status, batch.pos, cos_t, sin_t)
        del dattn, delta, dq_acc
        if cfg.attention_bias:
            C.colsum(dqkv, sink.view(p + "bqkv"))
        dh1 = dh2  # reuse
        self._gemm(dqkv, self.w(p + "wqkv"), dh1, b_mn=True)
        self._wgrad(dqkv, s["h1"], p + "wqkv", sink)
        C.rmsnorm_bwd(dh1, s["x"], self.w(p + "ln1"), s["rstd1"], dx, sink.view(p + "ln1"), True)
        # SwiGLU, two norms of two kernels, attention with its row products and its conversions (one more for shared kv heads)
        spread = C.attn_bwd_pieces(batch.tiles.shape[0], cfg.num_attention_heads, cfg.num_key_value_heads) > 1
        self.launches += 8 + spread + cfg.attention_bias
        sink.unit_done(i + 1)

    # ---- public ----
    def hidden(self, batch: PackedBatch, saves: Optional[List[dict]] = None) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
        """Returns (normed final hidden, pre-norm hidden, final rstd)."""
        x = self._body(batch, saves)
        hn, rstd = self._final_norm(x)
        return hn, x, rstd

    def _final_norm(self, x: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
        hn = torch.empty_like(x)
        rstd = self._new(x.shape[0], dtype=torch.float32)
        self.C.rmsnorm_fwd(x, self.w("final_norm"), hn, rstd, self.cfg.rms_norm_eps)
        self.launches += 1
        return hn, rstd

    def _chunk(self, rows: int) -> int:
        """Columns of the dlogits buffer of ``rows`` rows."""
        return min(vocab_chunk(rows, self.lmhead_chunk), (self.cfg.vocab_size + 255) // 256 * 256)

    def _keep_columns(self, rows: int) -> int:
        """Columns of the fp32 logits of ``rows`` rows that a training step may keep beside what it holds when it asks (its layers'
        activations). The allocator is asked first, the device only if this stream's unused blocks do not hold the logits and the head's
        buffers, and then not again until the allocator has taken or given back memory: on a machine with other users that question
        takes 0.1 to 100 ms."""
        V, H = self.cfg.vocab_size, self.cfg.hidden_size
        if rows <= 0 or torch.cuda.is_current_stream_capturing() or torch.cuda.get_allocator_backend() != "native":
            return 0  # a graph's memory stays taken between its replays; other allocators do not say what they hold
        chunk = self._chunk(rows)
        step = int(self.C.lmhead_chunk_step(V, chunk))
        if 4 * rows * V <= 64 << 20:
            return kept_columns(rows, V, 64 << 20, step)
        # rows of the head, dlogits, dH. As exact as it can be: more, and a step would not find what the same step has left in the allocator
        head = rows * (2 * chunk + 6 * H)
        device = self.dev.index if self.dev.index is not None else torch.cuda.current_device()
        cached, block, reserved = self.C.cached_memory(device, 2 * rows * H)
        cols = kept_columns(rows, V, min(block, cached - head), step)
        if cols >= V:
            return cols
        if reserved != self._asked[0]:
            free, total = torch.cuda.mem_get_info(self.dev)
            limit = int(torch.cuda.get_per_process_memory_fraction(self.dev) * total) - reserved
            self._asked = (reserved, max(0, min(free - int((1.0 - self.memory_share) * total), limit)))
        # Of what the process could still get a quarter, since other streams and roles grow as well. For the head's buffers, or for a new
        # block, which is not more than the device has beside what the head asks it for: else the allocator would give back all that
        # it holds and begin anew.
        free = self._asked[1]
        cols = kept_columns(rows, V, min(block, cached + free // 4 - head), step)
        return max(cols, kept_columns(rows, V, min((cached + free - head) // 4, free - max(0, head - cached)), step))

    def _body(self, batch: PackedBatch, saves: Optional[List[dict]]) -> torch.Tensor:
        """Embedding and all layers."""
        cfg, C = self.cfg, self.C
        T = batch.T
        cos_t, sin_t = self.rope_tables()
        x = self._new(T, cfg.hidden_size)
        self._enter_unit(0, None)
        C.embedding_fwd(batch.ids, self.w("embed"), x)
        n_layers = cfg.num_hidden_layers
        for i in range(n_layers):
            save = None
            if saves is not None:
                save = {}
                saves.append(save)
            x_in = x
            x = self._layer_fwd(i, x, batch, cos_t, sin_t, save if not self.recompute else None,
                                next_unit=i + 2 if i + 1 < n_layers else None)
            if saves is not None and self.recompute:
                save["x"] = x_in
        self.launches += 1
        return x

    def ensure_rope(self, max_pos: int) -> None:
        if self._rope is None or self._rope[0].shape[0] < max_pos:
            self._rope = None
            self.rope_tables(max_pos)

    def logprobs(self, batch: PackedBatch, temperature: float) -> Tuple[torch.Tensor, torch.Tensor]:
        """Per-row logprob of the next token and entropy (fp32 [T]); forward only."""
        C = self.C
        hn, _, _ = self.hidden(batch)
        T = batch.T
        wl = self.w(self.layout.lm_head_name())
        groups = int(C.lmhead_num_groups(wl.shape[0], T))
        partials = self._new(3 * groups * T, dtype=torch.float32)
        ll = torch.zeros(T, dtype=torch.float32, device=self.dev)
        logp = self._new(T, dtype=torch.float32)
        ent = self._new(T, dtype=torch.float32)
        C.lmhead_logprob(hn, wl, batch.labels, temperature, partials, ll, logp, ent, None, self.status)
        self.launches += 2
        return logp, ent

    def forward_backward(self, batch: PackedBatch, lc: LossConfig, loss_scale: float, sink: GradSink) -> torch.Tensor:
        """One microbatch: forward, fused loss, full backward into ``sink``. Returns the device stats vector
        (sums over valid tokens, see ops.reference.LOSS_STAT_NAMES). The scalar loss is
        stats[loss_sum] / max(1, stats[count]) * loss_scale; nothing here synchronises with the host."""
        cfg, C = self.cfg, self.C
        T = batch.T
        cos_t, sin_t = self.rope_tables()
        saves: List[dict] = []
        # From the final norm to its gradient only rows with a label take part: prompts and the last row of a sample have none
        # (a third of the rows where answers are short), and their gradient is zero. Work that is saved: logits twice, two gradients.
        compact = (batch.loss_rows and batch.total_out > 0
                   and 8.0 * (T - batch.total_out) * cfg.vocab_size * cfg.hidden_size > LOSS_ROWS_MIN_FLOPS)
        x_last = self._body(batch, saves)
        # The backward pass needs the logits again: kept in fp32 (31287 x 151936: 19 GB) they are read once, 2 ms, instead of
        # recomputed, 10 ms. Columns for which there is no memory are recomputed. Decided here, when the activations have what they
        # need and the device has work: the question takes the host 0.2 ms.
        n_head = batch.total_out if compact else T
        keep = self._keep_columns(n_head)
        try:
            logits = self._new(n_head, keep, dtype=torch.float32) if keep > 0 else None
        except torch.OutOfMemoryError:
            logits = None
        labels, advantages, old_logp, old_ent = batch.labels, batch.advantages, batch.old_logprobs, batch.old_entropies
        ref = batch.ref_logprobs if (lc.kl_beta > 0 and batch.has_ref) else None
        rows = None
        if compact:
            rows, x_all, n = batch.output_indices, x_last, batch.total_out
            x_last, labels, cols = self._new(n, cfg.hidden_size), self._new(n, dtype=torch.int32), self._new(4, n, dtype=torch.float32)
            C.gather_loss_rows(rows, x_all, batch.labels, batch.float_buf[:4 * T].view(4, T), x_last, labels, cols)
            advantages, old_logp, old_ent = cols[0], cols[1], cols[2]
            ref = cols[3] if ref is not None else None
            T = n
            del x_all
        hn, rstd_f = self._final_norm(x_last)
        wl_name = self.layout.lm_head_name()
        wl = self.w(wl_name)
        V = wl.shape[0]
        groups = int(C.lmhead_num_groups(V, T))
        partials = self._new(3 * groups * T, dtype=torch.float32)
        ll = torch.zeros(T, dtype=torch.float32, device=self.dev)
        logp = self._new(T, dtype=torch.float32)
        ent = self._new(T, dtype=torch.float32)
        lse = self._new(T, dtype=torch.float32)
        C.lmhead_logprob(hn, wl, labels, lc.temperature, partials, ll, logp, ent, lse, self.status, logits)
        del partials
        stats = torch.zeros(self.n_stats, dtype=torch.float32, device=self.dev)
        dlogp = self._new(T, dtype=torch.float32)
        n_valid = max(1.0, batch.scalars.get("num_output_tokens_non_masked", float(batch.total_out)))
        C.grpo_token_loss(logp, old_logp, ref, advantages, labels, ent, old_ent,
                          lc.clip_low, lc.clip_high, lc.clip_ratio_c, lc.kl_beta, loss_scale / n_valid, dlogp, stats)
        chunk = self._chunk(T)
        dz = self._new(T, chunk)
        dh_acc = self._new(T, cfg.hidden_size, dtype=torch.float32)
        C.lmhead_backward(hn, wl, labels, lse, dlogp, lc.temperature, dz, dh_acc, sink.view(wl_name), self.status, logits)
        del dz, logits
        dhn = self._new(T, cfg.hidden_size)
        C.cast_f32_bf16(dh_acc, dhn)
        del dh_acc
        dx = self._new(T, cfg.hidden_size)
        C.rmsnorm_bwd(dhn, x_last, self.w("final_norm"), rstd_f, dx, sink.view("final_norm"), False)
        del dhn
        self.launches += 6 + 3 * ((V + chunk - 1) // chunk)
        if rows is not None:
            dx_rows, dx = dx, torch.zeros(batch.T, cfg.hidden_size, dtype=torch.bfloat16, device=self.dev)
            C.scatter_rows(rows, dx_rows, dx)
            del dx_rows
            self.launches += 2
        for i in reversed(range(cfg.num_hidden_layers)):
            s = saves[i]
            if self.recompute:
                full: dict = {}
                self._layer_fwd(i, s["x"], batch, cos_t, sin_t, full, next_unit=i if i > 0 else None)
                s = full
            self._layer_bwd(i, dx, s, batch, cos_t, sin_t, sink)
            saves[i] = None  # free activations of this layer
        C.embedding_bwd(batch.ids, dx, sink.view("embed"))
        self.launches += 1
        sink.unit_done(0)
        return stats
