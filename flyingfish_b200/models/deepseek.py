"""DeepSeek-V3-style decoder: multi-head latent attention (MLA) + dense / MoE feed-forward.

Attention runs in the absorbed form for prefill and decode alike: the cache holds one latent row
per token (``kv_lora_rank`` compressed KV + the shared RoPE key), queries are projected into the
latent space with W_UK, attention is multi-query over the latent rows, and the latent output is
expanded with W_UV before ``o_proj``. The FFN side (first dense layers, then grouped no-aux routed
experts + shared expert) reuses the decoder's MoE block. Reference for the operator sequence:
src/backend/cuda/engine_deepseek.rs:1119-1700 (latent mixer) and kernels/moe_route.cu:316-390.
"""
from __future__ import annotations

import math
from dataclasses import dataclass

import torch

from .. import ops
from ..config import ModelSpec
from ..ops import mla_ops
from .decoder import DecoderModel
from .weights import LayerWeights, ModelWeights, TPInfo, build_decoder_weights


EXPAND_MAX_BYTES = 2 << 30       # most memory that a layer's expanded keys and values take (out of the planner's reserve)
# A step's portions are expanded from this many query rows per visible key on (a portion's rows, weighted by its context). The expansion costs
# by the key, the latent space by the row and key. One layer at the published widths, latent space against expanded: 64 rows in front of 16,000
# tokens 1748 / 855 us, 23 rows per key 553 / 622, 10 rows 634 / 1314, a portion of 64 rows beside fifteen of 8 rows behind 2000 tokens 612 / 1612.
EXPAND_MIN_ROWS_PER_KEY = 32


@dataclass
class MlaWeights:
    q_a: torch.Tensor | None        # [q_lora, h]
    q_a_ln: torch.Tensor | None
    q_b: torch.Tensor               # [heads*(nope+rope), q_lora or h]
    kv_a: torch.Tensor              # [kv_lora + rope, h]
    kv_a_ln: torch.Tensor
    w_uk_t: torch.Tensor            # [heads, kv_lora, nope]   (absorb: q_lat = q_nope @ W_UK)
    w_kv: torch.Tensor              # [heads * nope | heads * v, kv_lora]: all key matrices, then all value matrices
    wo: torch.Tensor                # [h, heads*v]

    def w_uv(self, heads: int) -> torch.Tensor:
        """[heads, v, kv_lora]"""
        return self.w_kv[heads * self.w_uk_t.shape[2]:].view(heads, -1, self.w_kv.shape[1])


def build_deepseek_weights(spec: ModelSpec, source, device, tp: TPInfo | None = None, ep: TPInfo | None = None
                           ) -> ModelWeights:
    """FFN / norms / embeddings come from the common builder (with a stub attention geometry);
    the MLA projections are attached per layer as ``lw.extra['mla']``."""
    a = spec.mla
    heads = spec.heads

    # build with attention disabled: temporarily a spec whose attention tensors are tiny
    import copy
    stub = copy.copy(spec)
    stub.heads, stub.kv_heads, stub.head_dim = 1, 1, 16
    stub.qk_norm = False
    fp8 = spec.linear_format == "fp8_block"
    fp8_experts = spec.moe is not None and spec.moe.expert_format == "fp8_block"
    if fp8 != fp8_experts and spec.moe is not None:
        raise ValueError("FP8 DeepSeek-style checkpoints quantise the linears and the experts together")
    from .weights import pack_ffn_fp8
    w = build_decoder_weights(stub, source_with_stub_attention(source, device), device, tp, ep, fuse_swiglu=not fp8,
                              layer_hook=pack_ffn_fp8 if fp8 else None)
    w.spec = spec
    h = spec.hidden
    qk = a.qk_nope_dim + a.qk_rope_dim
    for i, lw in enumerate(w.layers):
        p = f"model.layers.{i}.self_attn."
        lw.wqkv = None
        if a.q_lora_rank:
            q_a = source(p + "q_a_proj.weight", (a.q_lora_rank, h))
            q_a_ln = source(p + "q_a_layernorm.weight", (a.q_lora_rank,))
            q_b = source(p + "q_b_proj.weight", (heads * qk, a.q_lora_rank))
        else:
            q_a, q_a_ln = None, None
            q_b = source(p + "q_proj.weight", (heads * qk, h))
        kv_a = source(p + "kv_a_proj_with_mqa.weight", (a.kv_lora_rank + a.qk_rope_dim, h))
        kv_a_ln = source(p + "kv_a_layernorm.weight", (a.kv_lora_rank,))
        kv_b = source(p + "kv_b_proj.weight", (heads * (a.qk_nope_dim + a.v_head_dim), a.kv_lora_rank))
        kv_b = kv_b.view(heads, a.qk_nope_dim + a.v_head_dim, a.kv_lora_rank)
        w_uk = kv_b[:, : a.qk_nope_dim]                         # [heads, nope, kv_lora]
        w_kv = torch.cat([w_uk.reshape(-1, a.kv_lora_rank), kv_b[:, a.qk_nope_dim:].reshape(-1, a.kv_lora_rank)])
        wo = source(p + "o_proj.weight", (h, heads * a.v_head_dim))
        w_uk_t = w_uk.transpose(1, 2).contiguous()
        if fp8:
            # the projections stay in the checkpoint's E4M3 block format; the two absorbed factors of kv_b are small
            # and are applied per head in BF16
            from ..ops.quant_ops import Fp8Weight
            q_a = Fp8Weight.from_dense(q_a) if q_a is not None else None
            q_b, kv_a, wo = Fp8Weight.from_dense(q_b), Fp8Weight.from_dense(kv_a), Fp8Weight.from_dense(wo)
        lw.extra["mla"] = MlaWeights(q_a, q_a_ln, q_b, kv_a, kv_a_ln, w_uk_t, w_kv, wo)
        lw.wo = wo
    return w


def source_with_stub_attention(source, device):
    def src(name: str, shape):
        if any(k in name for k in (".self_attn.q_proj", ".self_attn.k_proj", ".self_attn.v_proj", ".self_attn.o_proj")):
            return torch.zeros(shape, dtype=torch.bfloat16, device=device)
        return source(name, shape)
    return src


class DeepseekModel(DecoderModel):
    """Same driver loop as :class:`DecoderModel`; only the attention block differs."""

    def __init__(self, weights: ModelWeights, comm=None, trace=None):
        super().__init__(weights, comm, trace)
        a = self.spec.mla
        self.mla = a
        self.scale = 1.0 / math.sqrt(a.qk_nope_dim + a.qk_rope_dim)
        self.latent_dim = a.kv_lora_rank + a.qk_rope_dim

    def _attention(self, i: int, n: torch.Tensor, b, kv) -> torch.Tensor:
        lw, s, a = self.w.layers[i], self.spec, self.mla
        m: MlaWeights = lw.extra["mla"]
        rows = n.shape[0]
        heads = s.heads
        if m.q_a is not None:
            qa = ops.rmsnorm(ops.linear(n, m.q_a), m.q_a_ln, s.rms_eps)
            q = ops.linear(qa, m.q_b)
        else:
            q = ops.linear(n, m.q_b)
        kva = ops.linear(n, m.kv_a)
        if n.is_cuda:
            o = self._attend(i, q, kva, m, b, kv)
        else:
            o = self._attend_oracle(i, q, kva, m, b, kv)
        if self.trace is not None:
            self.trace.record(f"layer.{i}.attn", o.view(rows, heads, a.v_head_dim))
        return self.comm.row_linear(o, m.wo)

    def _attend(self, i: int, q: torch.Tensor, kva: torch.Tensor, m: MlaWeights, b, kv) -> torch.Tensor:
        """[rows, heads * v] on the GPU. Portions of prompts expand the visible latents to keys and values; decoded tokens, portions that
        are short against what they see, and contexts beyond the expansion's memory go through the latent space. The step decides for all
        its portions, and the forms round at different places: a portion's bits may depend on the portions beside it."""
        s, a, heads, rows = self.spec, self.mla, self.spec.heads, q.shape[0]
        cache, nope, dv = kv.k[i], a.qk_nope_dim, a.v_head_dim
        form = (kva, m.kv_a_ln, b.positions, b.slots, cache, heads, nope, s.rope_theta, s.rms_eps)
        pages = None
        if not b.is_decode and mla_ops.expands(q, self.latent_dim, nope, a.qk_rope_dim, dv, b.max_q_len):
            pages = self._key_pages(b, kv)
        if pages is not None:
            mla_ops.norm_rope_cache(q, *form)
            out = torch.empty(rows, heads * dv, dtype=q.dtype, device=q.device)
            return mla_ops.expanded_attention(q, q.view(rows, heads, -1), cache, m.w_kv, pages, b.block_table, b.q_start, b.q_lens, b.ctx_lens,
                                              b.max_q_len, nope, dv, a.kv_lora_rank, self.scale, 0, None, out)
        q_full = torch.empty(rows, heads, self.latent_dim, dtype=q.dtype, device=q.device)
        mla_ops.norm_rope_cache(q, *form, q_full)
        ops.head_linear(q, m.w_uk_t, out=q_full.view(rows, -1), x_cols=nope + a.qk_rope_dim, out_cols=self.latent_dim)
        lat = mla_ops.attention(q_full, cache, b.block_table, b.q_start, b.q_lens, b.ctx_lens, b.nq if b.is_decode else b.max_q_len, b.max_ctx,
                                self.scale, a.kv_lora_rank)
        return ops.head_linear(lat.view(rows, -1), m.w_uv(heads))

    def _key_pages(self, b, kv):
        """The pages of a step's portions, or None where expanding them does not pay or would take over ``EXPAND_MAX_BYTES``. Listed by the
        step's first layer and kept with the step: one model serves several engines, also from several threads."""
        if b.key_pages is None:
            L, h, n = b.layout, b.host, b.batch
            table = h[L.block_table: L.block_table + L.max_batch * L.max_blocks].view(L.max_batch, L.max_blocks)[:n]
            ctx = h[L.ctx_lens: L.ctx_lens + n].tolist()
            lens = h[L.q_lens: L.q_lens + n].tolist()
            keys = sum((c + kv.block_size - 1) // kv.block_size for c in ctx) * kv.block_size
            fits = 2 * keys * self.spec.heads * (self.mla.qk_nope_dim + self.mla.v_head_dim) <= EXPAND_MAX_BYTES
            pays = sum(q * c for q, c in zip(lens, ctx)) >= EXPAND_MIN_ROWS_PER_KEY * sum(ctx)
            b.key_pages = (mla_ops.KeyPages.of(lens, ctx, table, 0, kv.block_size, b.device) if fits and pays else None,)
        return b.key_pages[0]

    def _attend_oracle(self, i: int, q: torch.Tensor, kva: torch.Tensor, m: MlaWeights, b, kv) -> torch.Tensor:
        """[rows, heads * v] through the latent space, operator by operator (CPU)."""
        s, a, heads, rows = self.spec, self.mla, self.spec.heads, q.shape[0]
        q = q.view(rows, heads, a.qk_nope_dim + a.qk_rope_dim)
        c = ops.rmsnorm(kva[:, : a.kv_lora_rank], m.kv_a_ln, s.rms_eps)
        k_rope = kva[:, a.kv_lora_rank:].contiguous()
        q_rope = q[:, :, a.qk_nope_dim:].reshape(rows, heads * a.qk_rope_dim).contiguous()
        ops.rope_inplace(q_rope, b.positions, heads, a.qk_rope_dim, s.rope_theta)
        ops.rope_inplace(k_rope, b.positions, 1, a.qk_rope_dim, s.rope_theta)
        mla_ops.cache_write(c, k_rope, b.slots, kv.k[i])
        q_lat = mla_ops.per_head_linear(q[:, :, : a.qk_nope_dim].contiguous(), m.w_uk_t)      # [rows, heads, kv_lora]
        q_full = torch.cat([q_lat, q_rope.view(rows, heads, a.qk_rope_dim)], dim=2).contiguous()
        lat = mla_ops.attention(q_full, kv.k[i], b.block_table, b.q_start, b.q_lens, b.ctx_lens, b.nq if b.is_decode else b.max_q_len, b.max_ctx,
                                self.scale, a.kv_lora_rank)
        return mla_ops.per_head_linear(lat, m.w_uv(heads)).reshape(rows, heads * a.v_head_dim)
