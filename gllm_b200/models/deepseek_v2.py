"""DeepSeek-V2 / V3 / R1 (and Moonlight / Kimi-K2, same architecture): MLA attention + DeepSeek MoE
(reference: gllm/models/deepseek_v2.py:61-548, gllm/layers/attention.py:65-492).

MLA here stores the *latent* KV cache — `[kv_c (kv_lora_rank, RMS-normed) | k_pe (rope dims, rotated)]`
per token, one "head", replicated on every TP rank (like the reference's MLA `Segment`,
gllm/memory_manager.py:38-42) — and q heads are split over TP. Routing uses the group-limited top-k
kernel (sigmoid + bias-corrected `noaux_tc` for V3), experts run through the grouped tcgen05 GEMMs,
shared experts are an ordinary gated MLP whose partial output is reduced together with the routed one.

On sm_100a the attention runs in the *absorbed* form: q_nope·W_UK per head (batched tcgen05 GEMM over strided
views, written straight into the 576-wide query), fused RoPE + latent-cache write, split-KV multi-query attention
over the paged latent cache (csrc/attn/mla_attention.cu), then out_lat·W_UV per head (the same batched GEMM,
written in the [T, heads·v] layout o_proj reads). No cuBLAS and no host synchronisation on that path, so decode
batches run inside CUDA graphs. Prompt portions of 32 tokens and more take the
*expanded* form instead: the cached latents are gathered, a GEMM makes every head's keys and values, and the tcgen05
prefill attention runs on them. The CPU / odd-shape path below evaluates the expanded form with PyTorch ops per sequence
(the numerical oracle of the GPU path).
"""
from __future__ import annotations

from typing import Optional

import numpy as np
import torch
import torch.nn.functional as F
from torch import nn

from gllm_b200.layers import functional as Fn
from gllm_b200.layers.moe import SparseMoeBlock
from gllm_b200.layers.rotary import build_rope
from gllm_b200.models import weight_utils as wu
from gllm_b200.models.decoder import (CausalLM, DenseMLP, ModelSpec, MoESpec, _linear_params, _param, _qw,
                                      _store_linear)
from gllm_b200.models.registry import _dtype
from gllm_b200.ops import ref
from gllm_b200.parallel import state as ps
from gllm_b200.parallel.tp import TPComm


def _joined(a: torch.Tensor, b: torch.Tensor):
    """[a ; b] without a copy if b's rows follow a's in the same storage, else None."""
    if b.data_ptr() != a.data_ptr() + a.nbytes or b.dtype != a.dtype or not (a.is_contiguous() and b.is_contiguous()):
        return None
    (n, k), (m, l) = a.shape, b.shape
    if l != k or a.untyped_storage().nbytes() < (a.storage_offset() + (n + m) * k) * a.itemsize:
        return None
    return a.as_strided((n + m, k), (k, 1))


class MLAAttention(nn.Module):
    def __init__(self, spec: ModelSpec, layer_id: int, rope, device):
        super().__init__()
        x = spec.extra
        st = ps.get_state()
        tp = st.tp_size
        self.layer_id = layer_id
        self.tp, self.tr = tp, st.tp_rank
        self.num_heads = spec.num_heads // tp
        self.nope, self.rope_dim, self.v_dim = x["qk_nope_head_dim"], x["qk_rope_head_dim"], x["v_head_dim"]
        self.qk_dim = self.nope + self.rope_dim
        self.kv_lora, self.q_lora = x["kv_lora_rank"], x.get("q_lora_rank")
        self.rope = rope
        self.eps = spec.rms_eps
        self.scaling = self.qk_dim ** -0.5 * rope.attn_mscale
        h, dt = spec.hidden_size, spec.dtype
        # The projections follow the checkpoint's quantisation (fp8 block-scaled for V3 / R1: (weight, scale_inv)
        # pairs on the UTCQMMA GEMM — reference plumbs quant_config into them, gllm/models/deepseek_v2.py:280-440).
        # kv_b_proj stays bf16: it is only ever used absorbed, as the per-head W_UK / W_UV operands.
        # The two projections of the hidden state lie in one tensor, [q_a rows ; kv_a rows], of which the parameters are views: one GEMM
        # of 2112 columns instead of two of 1536 and 576, neither of which fills the machine (K = 7168, 4096 rows: 87 us instead of
        # 78 + 43, 128 rows: 17 instead of 16.5 + 16.4). Block scales must not straddle the border. Only the parameters hold them:
        # `_qkv_a` looks in each call whether they still lie so (one that was replaced, moved or converted does not).
        self.joined = bool(self.q_lora) and self.q_lora % 128 == 0
        if self.joined:
            w, s = _linear_params(self.q_lora + self.kv_lora + self.rope_dim, h, spec, device)

            def cut(x, n):
                return (None, None) if x is None else [nn.Parameter(v, requires_grad=False) for v in (x.data[:n], x.data[n:])]
            self.q_a_w, self.kv_a_w = cut(w, self.q_lora)
            self.q_a_ws, self.kv_a_ws = cut(s, self.q_lora // 128)
        if self.q_lora:
            if not self.joined:
                self.q_a_w, self.q_a_ws = _linear_params(self.q_lora, h, spec, device)
            self.q_a_norm_w = _param(self.q_lora, dtype=dt, device=device, fill=1.0)
            self.q_b_w, self.q_b_ws = _linear_params(self.num_heads * self.qk_dim, self.q_lora, spec, device)
        else:
            self.q_w, self.q_ws = _linear_params(self.num_heads * self.qk_dim, h, spec, device)
        if not self.joined:
            self.kv_a_w, self.kv_a_ws = _linear_params(self.kv_lora + self.rope_dim, h, spec, device)
        self.kv_a_norm_w = _param(self.kv_lora, dtype=dt, device=device, fill=1.0)
        self.kv_b_w = _param(self.num_heads * (self.nope + self.v_dim), self.kv_lora, dtype=dt, device=device)
        self.o_w, self.o_ws = _linear_params(h, self.num_heads * self.v_dim, spec, device)
        self.o_b = None
        # attributes the generic runner looks at
        self.num_kv_heads = 1
        self.head_dim = self.kv_lora + self.rope_dim

    def _qkv_a(self):
        """q_a and kv_a as the weight of one product, or None if their tensors do not follow each other in memory."""
        if not self.joined:
            return None
        w = _joined(self.q_a_w, self.kv_a_w)
        if w is None or self.q_a_ws is None:
            return w
        s = _joined(self.q_a_ws, self.kv_a_ws)
        return None if s is None else (w, s)

    def forward(self, inp, h: torch.Tensor, kv_cache, tpc: TPComm) -> torch.Tensor:
        t = h.shape[0]
        hl = self.num_heads
        h = tpc.materialize(h)
        qkv_a = self._qkv_a()
        if kv_cache is not None and self._one_call(inp, h, qkv_a):
            return self._forward_one_call(inp, h, qkv_a, kv_cache.k_cache[self.layer_id])
        if qkv_a is not None:
            both = Fn.linear(h, qkv_a)
            kv_a = both[:, self.q_lora:]
            qa, kv_c = Fn.rmsnorm_two(both[:, : self.q_lora], self.q_a_norm_w, kv_a[:, : self.kv_lora], self.kv_a_norm_w, self.eps)
            q = Fn.linear(qa, _qw(self.q_b_w, self.q_b_ws))
        else:
            if self.q_lora:
                qa, _ = Fn.rmsnorm(Fn.linear(h, _qw(self.q_a_w, self.q_a_ws)), self.q_a_norm_w, self.eps)
                q = Fn.linear(qa, _qw(self.q_b_w, self.q_b_ws))
            else:
                q = Fn.linear(h, _qw(self.q_w, self.q_ws))
            kv_a = Fn.linear(h, _qw(self.kv_a_w, self.kv_a_ws))
            lat = kv_a[:, : self.kv_lora]
            kv_c, _ = Fn.rmsnorm(lat if lat.is_cuda and kv_a.shape[1] % 8 == 0 else lat.contiguous(), self.kv_a_norm_w, self.eps)
        q = q.view(t, hl, self.qk_dim)
        if kv_cache is None:
            return q[:, :, : self.v_dim].reshape(t, hl * self.v_dim).contiguous()
        cache = kv_cache.k_cache[self.layer_id]
        if h.is_cuda and self.kv_lora == 512 and self.rope_dim == 64:
            return self._forward_absorbed(inp, q, kv_c, kv_a[:, self.kv_lora:], cache)
        k_pe = kv_a[:, self.kv_lora:].contiguous().view(t, 1, self.rope_dim)
        q_pe = q[:, :, self.nope:].contiguous()
        # GPT-J style (interleaved) rotary on the rope dims only; oracle op (strided sub-views)
        ref.rope_kv_write(q_pe, k_pe, None, inp.positions, self.rope.cos_sin, self.rope_dim, False, None, None,
                          self.eps, None, None, None)
        latent = torch.cat([kv_c, k_pe.view(t, self.rope_dim)], dim=-1).view(t, 1, self.head_dim)
        ref.write_kv_cache(latent, None, cache, None, inp.slot_mapping)
        q = torch.cat([q[:, :, : self.nope], q_pe], dim=-1)
        out = torch.empty(t, hl, self.v_dim, dtype=h.dtype, device=h.device)
        qsl = inp.query_start_loc.tolist()
        sls = inp.seq_lens.tolist()
        for s in range(inp.num_seqs):
            q0, q1 = qsl[s], qsl[s + 1]
            ql, sl = q1 - q0, sls[s]
            if ql <= 0:
                continue
            lat = ref.gather_kv(cache, inp.block_table[s], sl)[:, 0]  # [L, 576]
            kvb = F.linear(lat[:, : self.kv_lora], self.kv_b_w).view(sl, hl, self.nope + self.v_dim)
            k = torch.cat([kvb[:, :, : self.nope], lat[:, None, self.kv_lora:].expand(sl, hl, self.rope_dim)], dim=-1)
            v = kvb[:, :, self.nope:]
            att = torch.einsum("qhd,khd->hqk", q[q0:q1].float(), k.float()) * self.scaling
            qi = torch.arange(ql, device=h.device).view(ql, 1) + (sl - ql)
            kj = torch.arange(sl, device=h.device).view(1, sl)
            att = att.masked_fill((kj > qi).unsqueeze(0), float("-inf"))
            out[q0:q1] = torch.einsum("hqk,khd->qhd", torch.softmax(att, -1), v.float()).to(h.dtype)
        return out.view(t, hl * self.v_dim)

    def process_weights(self):
        """W_UK [hl, nope, 512] and W_UV [hl, 512, v] views of kv_b_proj, made contiguous once, eagerly, after
        the weights are final and BEFORE any CUDA-graph capture (tensors created inside a capture only get
        their contents when the graph replays). Reference: MLAAttention.process_weights,
        gllm/layers/attention.py:106-127."""
        if not self.kv_b_w.is_cuda:
            return
        kvb = self.kv_b_w.data.view(self.num_heads, self.nope + self.v_dim, self.kv_lora)
        # both in the [batch, N, K] (nn.Linear) layout the batched GEMM reads:
        #   q_lat[:, h] = q_nope[:, h] @ W_UK[h]      -> weight [512 (N), nope (K)] = W_UK[h]^T
        #   out[:, h]   = out_lat[:, h] @ W_UV[h]^T   -> weight [v (N), 512 (K)]    = kv_b rows of the value part
        w_uk_nk, w_uv_nk = kvb[:, : self.nope, :].transpose(1, 2), kvb[:, self.nope:, :]
        old = getattr(self, "_w_abs", None)
        if old is not None:   # keep the addresses: captured CUDA graphs point at these tensors
            old[0].copy_(w_uk_nk)
            old[1].copy_(w_uv_nk)
        else:
            self._w_abs = (w_uk_nk.contiguous(), w_uv_nk.contiguous())

    def _absorbed_weights(self):
        if getattr(self, "_w_abs", None) is None:
            assert not torch.cuda.is_current_stream_capturing(), "call model.process_weights() before capture"
            self.process_weights()
        return self._w_abs

    # Expanded heads cost a GEMM of 2 * 256 * 512 operations per cached row and head, and then 640 per (query, key) pair
    # instead of 2176 on a kernel eight times as fast: they win from some twenty new tokens per sequence on; below that a portion
    # is a few rows of one 128-row tile. 5 prompts of 4096 tokens together, 16 heads: 2459 -> 479 us. A sequence's own portion
    # decides: its length, and its (query, key) pairs over all heads. Below 2^18 of them the absorbed form takes at most 4 us
    # (16 per 2^20), less than the host needs for the launches that the expanded form and the picking of rows add: 12 portions of 6
    # to 50 tokens over some hundred cached ones, 16 heads, took 250 us for the block where all absorbed they take 166.
    # What a call holds at a time is bounded: the gathered latents (more sequences take another round) and the keys
    # and values of as many heads as fit.
    _EXPAND_MIN_TOKENS = 32
    _EXPAND_MIN_PAIRS = 1 << 18
    _EXPAND_KV_BYTES = 1 << 30
    _EXPAND_LATENT_BYTES = 256 << 20
    _LATENT_ROW_BYTES = 576 * 2

    def _expands(self) -> bool:
        return (self.kv_lora, self.rope_dim, self.nope, self.v_dim) == (512, 64, 128, 128)

    def _expand_min_work(self) -> int:
        return -(-2 * self._EXPAND_MIN_PAIRS // self.num_heads)

    def expand_scratch_bytes(self, max_len: int) -> int:
        """What the expanded form allocates beside the cache at most, for sequences of up to `max_len` tokens."""
        if not self._expands():
            return 0
        return self._EXPAND_KV_BYTES + max(self._EXPAND_LATENT_BYTES, (max_len + 63) // 64 * 64 * self._LATENT_ROW_BYTES)

    def _expanded_plan(self, inp):
        """(rounds, rest) of this batch. rounds: (first sequence, end, rows of latents) of the prompt portions to expand, each
        sequence rounded up to 64 rows; empty: all attend in the absorbed form. rest: None if the rows in the absorbed form are
        the leading ones of the decoding sequences, else [their rows ; their sequences]."""
        n0, b = inp.num_decode_seqs, getattr(inp, "batch", None)
        if b is None or inp.padded_tokens or n0 == inp.num_seqs or inp.max_q_len < self._EXPAND_MIN_TOKENS or \
                not self._expands():
            return [], None
        q_lens = np.diff(b.query_start_loc[:inp.num_seqs + 1].astype(np.int64))
        lens = b.seq_lens[:inp.num_seqs].astype(np.int64)
        expand = (q_lens >= self._EXPAND_MIN_TOKENS) & (q_lens * (2 * lens - q_lens) >= self._expand_min_work())
        expand[:n0] = False
        rows = np.where(expand, (lens + 63) // 64 * 64, 0)
        total = int(rows.sum())
        if total * self._LATENT_ROW_BYTES <= self._EXPAND_LATENT_BYTES:
            rounds = [(n0, inp.num_seqs, total)] if total else []
        else:
            rounds, first, held = [], n0, 0
            for s in range(n0, inp.num_seqs):
                if held and (held + int(rows[s])) * self._LATENT_ROW_BYTES > self._EXPAND_LATENT_BYTES:
                    rounds.append((first, s, held))
                    first, held = s, 0
                held += int(rows[s])
            if held:
                rounds.append((first, inp.num_seqs, held))
        if not rounds or expand[n0:].all():
            return rounds, None
        keep = ~np.repeat(expand, q_lens)
        return rounds, np.stack([np.flatnonzero(keep), np.repeat(np.arange(inp.num_seqs), q_lens)[keep]]).astype(np.int32)

    def _plan_on_device(self, inp, device):
        """`_expanded_plan` with `rest` as tensors (rows, sequences), kept on the step's input for the layers behind the first:
        `InputData.load` drops it."""
        plan = getattr(inp, "latent_plan", None)
        if plan is None:
            rounds, rest = self._expanded_plan(inp)
            if rest is not None:
                rows, seqs = torch.from_numpy(rest).to(device, non_blocking=True)
                rest = (rows.long(), seqs)
            plan = (rounds, rest)
            if hasattr(inp, "latent_plan"):
                inp.latent_plan = plan
        return plan

    def _one_call(self, inp, h, qkv_a) -> bool:
        """Whether the block is the plain absorbed one on bf16 weights, which one native call launches as a whole."""
        if not (h.is_cuda and isinstance(qkv_a, torch.Tensor)) or h.shape[0] == 0 or self._plan_on_device(inp, h.device)[0]:
            return False
        from gllm_b200.ops import sm100
        return self.q_b_ws is None and self._expands() and self.q_lora <= 8192 and self.q_b_w.is_contiguous() and \
            h.dtype == qkv_a.dtype == self.q_b_w.dtype == torch.bfloat16 and not sm100.gemm_forced()

    def _forward_one_call(self, inp, h, qkv_a, cache):
        from gllm_b200.ops import sm100
        pos = inp.positions if inp.positions.dim() == 1 else inp.positions[0]
        w_uk, w_uv = self._absorbed_weights()
        out = sm100.mla_block(h, self.num_heads, qkv_a, self.q_a_norm_w, self.kv_a_norm_w, self.eps, self.q_b_w, w_uk, w_uv,
                              self.rope.cos_sin, pos, inp.slot_mapping, cache, inp.block_table, inp.tok_seq, self.scaling)
        return out.view(h.shape[0], self.num_heads * self.v_dim)

    def _forward_absorbed(self, inp, q, kv_c, k_pe, cache):
        """sm_100a path: multi-query attention over the latent cache (csrc/attn/mla_attention.cu) for decoding sequences and
        short portions, expanded heads on the tcgen05 prefill kernel for prompts. No host synchronisation, so decode batches
        run inside CUDA graphs."""
        from gllm_b200.ops import sm100
        t, hl = q.shape[0], self.num_heads
        out = torch.empty(t, hl, self.v_dim, dtype=q.dtype, device=q.device)
        pos = inp.positions if inp.positions.dim() == 1 else inp.positions[0]
        rounds, rest = self._plan_on_device(inp, q.device)
        n = inp.num_decode_seqs if rounds else t         # leading rows in the absorbed form
        if rest is not None:
            # short portions among long ones: everything is rotated in place, their rows are picked out
            sm100.mla_rope_cache(q[:, :, self.nope:], None, k_pe, kv_c, self.rope.cos_sin, pos, inp.slot_mapping, cache)
            rows, seqs = rest
            w_uk, w_uv = self._absorbed_weights()
            some = q.index_select(0, rows)
            q_full = torch.empty(rows.shape[0], hl, 576, dtype=q.dtype, device=q.device)
            sm100.gemm_batched(some[:, :, : self.nope], w_uk, q_full[:, :, :512])
            q_full[:, :, 512:] = some[:, :, self.nope:]
            out_lat = sm100.mla_attention(q_full, cache, inp.block_table, seqs, pos.index_select(0, rows), self.scaling)
            part = torch.empty(rows.shape[0], hl, self.v_dim, dtype=q.dtype, device=q.device)
            sm100.gemm_batched(out_lat, w_uv, part)
            out.index_copy_(0, rows, part)
        elif n:
            w_uk, w_uv = self._absorbed_weights()
            q_full = torch.empty(n, hl, 576, dtype=q.dtype, device=q.device)
            sm100.gemm_batched(q[:n, :, : self.nope], w_uk, q_full[:, :, :512])   # per head: q_nope · W_UK
            sm100.mla_rope_cache(q[:n, :, self.nope:], q_full, k_pe[:n], kv_c[:n], self.rope.cos_sin, pos[:n],
                                 inp.slot_mapping[:n], cache)
            out_lat = sm100.mla_attention(q_full, cache, inp.block_table, None if rounds else inp.tok_seq, pos[:n],
                                          self.scaling)
            sm100.gemm_batched(out_lat, w_uv, out[:n])                            # per head: out_lat · W_UV
        if rounds and rest is None:
            sm100.mla_rope_cache(q[n:, :, self.nope:], None, k_pe[n:], kv_c[n:], self.rope.cos_sin, pos[n:],
                                 inp.slot_mapping[n:], cache)
        for first, end, held in rounds:
            sm100.mla_expanded_attention(q, cache, inp.block_table, inp.seq_lens, inp.query_start_loc, self.kv_b_w, held, first,
                                         inp.max_q_len, self.scaling, out, end, self._EXPAND_MIN_TOKENS, self._EXPAND_KV_BYTES,
                                         self._expand_min_work())
        return out.view(t, hl * self.v_dim)


class DeepseekDecoderLayer(nn.Module):
    def __init__(self, spec: ModelSpec, layer_id: int, local_id: int, rope, device):
        super().__init__()
        self.spec, self.layer_id, self.local_id = spec, layer_id, local_id
        dt, h = spec.dtype, spec.hidden_size
        self.input_norm_w = _param(h, dtype=dt, device=device, fill=1.0)
        self.post_norm_w = _param(h, dtype=dt, device=device, fill=1.0)
        self.attn = MLAAttention(spec, local_id, rope, device)
        self.is_moe = spec.is_moe_layer(layer_id)
        self.mlp = SparseMoeBlock(spec, layer_id, device) if self.is_moe else \
            DenseMLP(h, spec.intermediate_size, dt, device, spec=spec)

    def forward(self, inp, h, residual, kv_cache, tpc: TPComm, next_norm_w):
        eps = self.spec.rms_eps
        a = self.attn(inp, h, kv_cache, tpc)
        h, residual = tpc.row_linear_add_norm(a, _qw(self.attn.o_w, self.attn.o_ws), residual, self.post_norm_w, eps)
        if self.is_moe:
            partial = self.mlp(tpc.materialize(h), tpc)
            if next_norm_w is None:
                return tpc.all_reduce(partial), residual
            return tpc.reduce_add_norm(partial, residual, next_norm_w, eps)
        act = self.mlp.act(h, tpc)
        if next_norm_w is None:
            return tpc.row_linear(act, self.mlp.down_weight()), residual
        return tpc.row_linear_add_norm(act, self.mlp.down_weight(), residual, next_norm_w, eps)


class DeepseekForCausalLM(CausalLM):
    def __init__(self, spec: ModelSpec, device="cpu"):
        # build the generic skeleton with zero layers, then install MLA layers
        nn.Module.__init__(self)
        self.spec = spec
        st = ps.get_state()
        self.device = torch.device(device)
        self.layers_range = ps.get_pp_layers(spec.num_layers)
        self.is_first, self.is_last = ps.is_first_pp_rank(), ps.is_last_pp_rank()
        self.tp_size, self.tp_rank = st.tp_size, st.tp_rank
        x = spec.extra
        self.rope = build_rope(x["qk_rope_head_dim"], spec.max_position, spec.rope_theta, spec.rope_scaling,
                               x["qk_rope_head_dim"], False, device=device)
        dt, h = spec.dtype, spec.hidden_size
        self.vocab_padded = wu.pad_vocab(spec.vocab_size, self.tp_size)
        self.vocab_per_rank = self.vocab_padded // self.tp_size
        self.vocab_start = self.tp_rank * self.vocab_per_rank
        need_embed = self.is_first or (spec.tie_word_embeddings and self.is_last)
        self.embed_w = _param(self.vocab_per_rank, h, dtype=dt, device=device) if need_embed else None
        self.layers = nn.ModuleList([DeepseekDecoderLayer(spec, gid, lid, self.rope, device)
                                     for lid, gid in enumerate(self.layers_range)])
        if self.is_last:
            self.final_norm_w = _param(h, dtype=dt, device=device, fill=1.0)
            self.lm_head_w = self.embed_w if spec.tie_word_embeddings else _param(self.vocab_per_rank, h, dtype=dt,
                                                                                   device=device)
        else:
            self.final_norm_w = self.lm_head_w = None
        self.kv_latent_dim = x["kv_lora_rank"] + x["qk_rope_head_dim"]

    @property
    def num_kv_heads(self): return 1

    @property
    def head_dim(self): return self.kv_latent_dim

    def step_scratch_bytes(self, max_len: int) -> int:
        """What a step allocates beside the cache that the memory probe, which runs without one, does not see."""
        return max((L.attn.expand_scratch_bytes(max_len) for L in self.layers), default=0)

    def _load_attention(self, reader, pre, nm, at: MLAAttention):
        tp, tr = self.tp_size, self.tp_rank
        p = pre + "self_attn."
        if at.q_lora:
            _store_linear(at.q_a_w, at.q_a_ws, reader.get(p + "q_a_proj.weight"))
            at.q_a_norm_w.data.copy_(reader.get(p + "q_a_layernorm.weight"))
            _store_linear(at.q_b_w, at.q_b_ws, wu.shard_rows(reader.get(p + "q_b_proj.weight"), tr, tp))
        else:
            _store_linear(at.q_w, at.q_ws, wu.shard_rows(reader.get(p + "q_proj.weight"), tr, tp))
        _store_linear(at.kv_a_w, at.kv_a_ws, reader.get(p + "kv_a_proj_with_mqa.weight"))
        at.kv_a_norm_w.data.copy_(reader.get(p + "kv_a_layernorm.weight"))
        at.kv_b_w.data.copy_(wu.shard_rows(reader.get(p + "kv_b_proj.weight"), tr, tp))
        _store_linear(at.o_w, at.o_ws, wu.shard_cols(reader.get(p + "o_proj.weight"), tr, tp))


def spec_deepseek(cfg) -> ModelSpec:
    heads = cfg["num_attention_heads"]
    moe = None
    moe_layers = None
    if cfg.get("n_routed_experts"):
        is_v3_arch = "V3" in (cfg.get("architectures") or [""])[0]
        v3 = cfg.get("topk_method") == "noaux_tc" or (is_v3_arch and cfg.get("topk_method") is None)
        if is_v3_arch and cfg.get("scoring_func") is None:
            cfg["scoring_func"] = "sigmoid"  # transformers >= 5 configs drop the field; V3 is always sigmoid
        n_shared = cfg.get("n_shared_experts") or 0
        moe = MoESpec(num_experts=cfg["n_routed_experts"], top_k=cfg["num_experts_per_tok"],
                      intermediate_size=cfg["moe_intermediate_size"], norm_topk_prob=bool(cfg.get("norm_topk_prob", False)),
                      shared_intermediate_size=cfg["moe_intermediate_size"] * n_shared, shared_gate=False,
                      scoring=cfg.get("scoring_func", "softmax"), n_group=cfg.get("n_group") or 1,
                      topk_group=cfg.get("topk_group") or 1, routed_scaling=cfg.get("routed_scaling_factor", 1.0),
                      has_bias_correction=v3)
        first_dense, freq = cfg.get("first_k_dense_replace", 0), cfg.get("moe_layer_freq", 1)
        moe_layers = [i for i in range(cfg["num_hidden_layers"]) if i >= first_dense and i % freq == 0]
    rope_scaling = cfg.get("rope_scaling") or None
    rp = cfg.get("rope_parameters")
    rope_theta = cfg.get("rope_theta", 10000.0)
    if rp:
        rope_theta = rp.get("rope_theta", rope_theta)
        if rp.get("rope_type", "default") != "default":
            rope_scaling = dict(rp)
    spec = ModelSpec(
        arch="deepseek", hidden_size=cfg["hidden_size"], num_layers=cfg["num_hidden_layers"], num_heads=heads,
        num_kv_heads=heads, head_dim=cfg["kv_lora_rank"] + cfg["qk_rope_head_dim"],
        intermediate_size=cfg["intermediate_size"], vocab_size=cfg["vocab_size"],
        rms_eps=cfg.get("rms_norm_eps", 1e-6), tie_word_embeddings=bool(cfg.get("tie_word_embeddings", False)),
        max_position=cfg.get("max_position_embeddings", 4096), rope_theta=rope_theta,
        rope_scaling=dict(rope_scaling) if rope_scaling else None, moe=moe, moe_layers=moe_layers, dtype=_dtype(cfg),
        use_mla=True, eos_token_id=cfg.get("eos_token_id"))
    spec.extra = {k: cfg.get(k) for k in ("q_lora_rank", "kv_lora_rank", "qk_nope_head_dim", "qk_rope_head_dim",
                                          "v_head_dim")}
    spec.names = {"shared": "mlp.shared_experts.", "router_bias": "mlp.gate.e_score_correction_bias"}
    qc = cfg.get("quantization_config") or {}
    if qc.get("quant_method") == "fp8" and list(qc.get("weight_block_size") or []) == [128, 128]:
        # routed experts, MLA projections (q_a / q_b / kv_a / o) and dense / shared MLPs stay block-scaled e4m3 as in
        # the checkpoint; kv_b_proj is de-quantised once into the bf16 W_UK / W_UV absorption operands
        spec.quant = "fp8"
    return spec


def build_deepseek(cfg, device):
    if cfg.get("kv_lora_rank") is None:
        raise NotImplementedError("non-MLA DeepSeek checkpoints are not supported")
    return DeepseekForCausalLM(spec_deepseek(cfg), device)
