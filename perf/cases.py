"""The work a serving process has this framework do, as cases that can be timed and compared.

A case is one engine call of a loaded model: a decode step of a batch that already has its context in the paged cache
(``Engine.decode``) or the prefill of requests that have just arrived (``Engine.prefill``). Three model families at the
published layer sizes, with fewer layers than the published models so that a model loads in seconds (the lm_head is that of the
full vocabulary; every layer is far larger than the L2 cache):

* ``dense``: Llama-3-8B shape, BF16, 8 layers -- the headline model of the benchmark;
* ``fp4``: Qwen3-MoE-235B shape, BF16 attention and NVFP4 experts, 4 layers, all experts resident;
* ``fp8``: DeepSeek-V3 shape, FP8 blocks, latent attention, 3 dense layers and 1 with experts.

Weights are seeded random values that the quantised formats hold exactly, as those of a published quantised checkpoint are. A
process loads a model once and serves many batches from it; an engine (cache, step metadata, captured step) belongs to a state.
"""
from __future__ import annotations

import copy
import math
import zlib

import torch

from flyingfish_b200.config import Settings, named_shape
from flyingfish_b200.engine.engine import Engine, bucket_for
from flyingfish_b200.models.decoder import DecoderModel
from flyingfish_b200.models.deepseek import DeepseekModel, build_deepseek_weights
from flyingfish_b200.models.weights import build_decoder_weights
from flyingfish_b200.ops.moe_cuda import pack_experts_nvfp4

SHAPES = {"dense": ("llama3-8b-shape", 8), "fp4": ("qwen3-moe-235b-shape", 4), "fp8": ("deepseek-v3-shape", 4)}
PAGE = 64
CHUNK = 8192                # rows of a prefill call
MAX_BATCH = 128
MAX_CACHED = 90_000         # tokens of context in a decode batch


# ------------------------------------------------------------------------------------------
# cases
# ------------------------------------------------------------------------------------------
def _case(name, family, kind, seqs, tokens, spread):
    c = {"family": family, "kind": kind, "seqs": seqs, "tokens": tokens, "spread": spread}
    return {"name": name, **c} if name else c


def listed():
    return [
        # one user's chat: a token for a single sequence, the latency floor of every generation
        _case("dense decode 1", "dense", "decode", 1, 1024, 0.0),
        # a few users with histories of very different lengths; the batch is padded to its bucket
        _case("dense decode 7 ragged", "dense", "decode", 7, 1500, 0.9),
        # the benchmark's batch: 64 sequences, a 1024-token prompt each and up to 256 new tokens behind it
        _case("dense decode 64", "dense", "decode", 64, 1152, 0.11),
        # a full server with short conversations
        _case("dense decode 113 short", "dense", "decode", 113, 300, 0.6),
        # a short question arrives alone: time to first token of a small prompt
        _case("dense prefill 1 x 37", "dense", "prefill", 1, 37, 0.0),
        # an ordinary prompt
        _case("dense prefill 1 x 1000", "dense", "prefill", 1, 1000, 0.0),
        # a burst of requests packed into one prefill chunk
        _case("dense prefill 8 x 1000", "dense", "prefill", 8, 1000, 0.2),
        # a document: one long prompt, where attention counts
        _case("dense prefill 1 x 8191", "dense", "prefill", 1, 8191, 0.0),
        # a decode batch of a mixture model with packed 4-bit experts
        _case("fp4 decode 32", "fp4", "decode", 32, 1000, 0.3),
        # prompts of that model: enough rows that every expert serves more than a hundred
        _case("fp4 prefill 3 x 700", "fp4", "prefill", 3, 700, 0.3),
        # a decode batch with latent attention, 8-bit weights and 8-bit experts
        _case("fp8 decode 64", "fp8", "decode", 64, 1024, 0.2),
        # prompts of that model
        _case("fp8 prefill 2 x 900", "fp8", "prefill", 2, 900, 0.3),
    ]


def draw(rng):
    family = rng.choice(["dense", "dense", "dense", "fp4", "fp8"])
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    spread = round(rng.choice([0.0, rng.uniform(0.0, 0.9)]), 3)
    if rng.random() < 0.5:
        seqs = log(1, MAX_BATCH) if family == "dense" else log(1, 64)
        tokens = log(16, min(7000, MAX_CACHED // (2 * seqs)))
        return _case(None, family, "decode", seqs, tokens, spread)
    rows = CHUNK if family == "dense" else 2200
    seqs = log(1, 16)
    return _case(None, family, "prefill", seqs, log(16, rows // (2 * seqs) if seqs > 1 else rows), spread)


def _lengths(case):
    """Tokens of every sequence: spread evenly over ``tokens * (1 +- spread)``, in a shuffled order."""
    n, t, s = case["seqs"], case["tokens"], case["spread"]
    most = 8191 if n == 1 else 16000
    return [min(max(1, round(t * (1 + s * (2 * ((0.5 + i * 0.6180339887) % 1.0) - 1)))), most) for i in range(n)]


# ------------------------------------------------------------------------------------------
# weights
# ------------------------------------------------------------------------------------------
def _spec(family):
    shape, layers = SHAPES[family]
    spec = copy.deepcopy(named_shape(shape))
    spec.layers, spec.mtp_layers = layers, 0
    return spec


def _normal(name, shape, std):
    g = torch.Generator(device="cuda")
    g.manual_seed(zlib.crc32(name.encode()))
    return torch.empty(shape, dtype=torch.float32, device="cuda").normal_(0.0, std, generator=g)


def _on_fp8_grid(w):
    """E4M3 values times 2^-13, with the largest code in every 64 x 128 block: what 128 x 128 block scales hold exactly."""
    q = (w * 8192.0).clamp(-448.0, 448.0).to(torch.float8_e4m3fn).to(torch.float32)
    q[::64, ::128] = torch.where(w[::64, ::128] < 0, -448.0, 448.0)
    return q / 8192.0


def _on_fp4_grid(w):
    """E2M1 values times an E4M3 scale per 16 times 2^-14, with the largest scale somewhere: what NVFP4 holds exactly."""
    g = w.view(w.shape[0], -1, 16)
    top = g.abs().amax(-1, keepdim=True)
    s = (top / 6.0 * 16384.0).to(torch.float8_e4m3fn).to(torch.float32).clamp_min(2.0 ** -6)
    s[0, 0] = 448.0
    grid = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], device=w.device)
    mids = (grid[1:] + grid[:-1]) / 2
    q = grid[torch.bucketize(g.abs() * 16384.0 / s, mids)]
    q = torch.where(g.abs() == top, 6.0, q) * torch.where(g < 0, -1.0, 1.0)
    return (q * s / 16384.0).view(w.shape)


def _weight(family, name, shape):
    """One tensor of a checkpoint, by its published name."""
    if "norm" in name:
        return (1.0 + _normal(name, shape, 0.1)).to(torch.bfloat16)
    # a residual stream that the layers add to rather than make up, and routers that prefer some experts clearly, as training leaves them
    w = _normal(name, shape, (4.0 if family == "fp8" else 1.0) if "embed_tokens" in name else 0.06 if family == "fp4" and "mlp.gate." in name else 0.02)
    if family == "fp4" and ".experts." in name:
        w = _on_fp4_grid(w)
    elif family == "fp8" and ("mlp." in name or "self_attn." in name) and "mlp.gate." not in name and "kv_b_proj" not in name:
        w = _on_fp8_grid(w)
    return w.to(torch.bfloat16)


_loaded = {}


def _model(family):
    """The loaded model of a family; the process holds one at a time."""
    if family not in _loaded:
        _loaded.clear()
        torch.cuda.empty_cache()
        spec, dev = _spec(family), torch.device("cuda", torch.cuda.current_device())
        source = lambda name, shape: _weight(family, name, shape)
        if family == "fp8":
            net = DeepseekModel(build_deepseek_weights(spec, source, dev))
        else:
            weights = build_decoder_weights(spec, source, dev)
            if family == "fp4":
                pack_experts_nvfp4(weights)
            net = DecoderModel(weights)
        _loaded[family] = (spec, net)
    return _loaded[family]


# ------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------
def _tokens(spec, lens, seed):
    g = torch.Generator()
    g.manual_seed(seed)
    return [torch.randint(0, spec.vocab, (n,), generator=g).tolist() for n in lens]


def _cached(spec, layer, blocks, seed):
    """Keys and values of a decode batch's context, at the sizes that this model's projections of normed rows give them."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1009 + layer)
    rand = lambda *shape: torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, 1.0, generator=g)
    if spec.mla is not None:
        rows = rand(blocks, 1, PAGE, spec.mla.kv_lora_rank + spec.mla.qk_rope_dim)
        return rows, None
    k, v = rand(blocks, spec.kv_heads, PAGE, spec.head_dim), rand(blocks, spec.kv_heads, PAGE, spec.head_dim)
    return k, v


def _blocks(lens):
    return [(n + PAGE - 1) // PAGE for n in lens]


class _State:
    pass


def prepare(case, seed):
    spec, net = _model(case["family"])
    lens = _lengths(case)
    longest = max(lens) + 1
    settings = Settings(capacity=max(4096, (longest + 255) // 256 * 256), max_batch=MAX_BATCH, chunk=CHUNK)
    st = _State()
    st.kind = case["kind"]
    st.engine = eng = Engine(net, spec, settings, sum(_blocks(lens)) + len(lens) + 1, net.w.embed.device, max_prefill_rows=CHUNK)
    if st.kind == "prefill":
        st.prompts = _tokens(spec, lens, seed)
        return st
    # the batch as its prefill left it: context in the cache, one sampled token per sequence not yet fed
    st.pending = [t[0] for t in _tokens(spec, [1] * len(lens), seed)]
    st.lens = lens
    st.seqs = []
    for n, tok in zip(lens, st.pending):
        s = eng.add_sequence([0] * n)
        eng.kv.reserve(s.seq_id, n)
        eng.kv.commit(s.seq_id, n)
        s.prefilled, s.pending = n, tok
        st.seqs.append(s)
    used = sum(_blocks(lens))
    for i in range(spec.layers):
        k, v = _cached(spec, i, used, seed)
        eng.kv.k[i][:used] = k
        if v is not None:
            eng.kv.v[i][:used] = v
    st.logits = eng.capture(bucket_for(len(lens))).logits[: len(lens)]
    return st


def run(state):
    """One decode step or one prefill through the engine; the logits it ranked and the cache it wrote. (Ids are the largest
    logits' indexes: two correct roundings may rank close ones differently, so the logits are what is compared.)"""
    eng = state.engine
    cache = [t for t in eng.kv.k + eng.kv.v if t is not None]
    if state.kind == "decode":
        eng.decode(state.seqs)
        for s, n, tok in zip(reversed(state.seqs), reversed(state.lens), reversed(state.pending)):     # the same step again
            eng.kv.truncate(s.seq_id, n)
            s.output.pop()
            s.pending = tok
        return {"logits": state.logits, "cache": cache}
    seqs = [eng.add_sequence(p) for p in state.prompts]
    eng.prefill(seqs)
    for s in reversed(seqs):                                       # the requests end here: their pages go back in order
        eng.kv.truncate(s.seq_id, 0)
        eng.free_sequence(s.seq_id)
    return {"logits": eng.model.last_logits, "cache": cache}


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------
def work(case):
    spec, lens = _spec(case["family"]), _lengths(case)
    decode = case["kind"] == "decode"
    new = [1] * len(lens) if decode else lens
    rows, h, vocab = sum(new), spec.hidden, spec.vocab
    seen = [n + 1 for n in lens] if decode else lens
    pairs = sum(seen) if decode else sum(n * (n + 1) // 2 for n in lens)
    nbytes = 2 * vocab * h + 2 * len(lens) * vocab + 2 * rows * h          # lm_head, logits, embedding rows
    flops = 2 * len(lens) * vocab * h
    moe = spec.moe
    for i in range(spec.layers):
        if spec.mla is not None:
            a = spec.mla
            qk = a.qk_nope_dim + a.qk_rope_dim
            proj = a.q_lora_rank * (h + spec.heads * qk) + (a.kv_lora_rank + a.qk_rope_dim) * h + spec.heads * a.v_head_dim * h
            kv_b = spec.heads * (a.qk_nope_dim + a.v_head_dim) * a.kv_lora_rank
            row = 2 * (a.kv_lora_rank + a.qk_rope_dim)
            nbytes += proj + 2 * kv_b
            flops += 2 * rows * (proj + kv_b)
            # over cached latents in the latent space; in a prompt with keys and values expanded once
            flops += 2 * pairs * spec.heads * ((2 * a.kv_lora_rank + a.qk_rope_dim) if decode else (qk + a.v_head_dim))
        else:
            proj = h * spec.qkv_dim + spec.q_dim * h
            row = 4 * spec.kv_heads * spec.head_dim
            nbytes += 2 * proj
            flops += 2 * rows * proj + 4 * pairs * spec.heads * spec.head_dim
        nbytes += row * ((sum(lens) if decode else 0) + rows)
        if moe is None or i < moe.first_dense_layers:
            ffn = 3 * h * (moe.dense_ffn if moe is not None and moe.dense_ffn else spec.ffn)
            nbytes += ffn * (1 if spec.linear_format == "fp8_block" else 2)
            flops += 2 * rows * ffn
        else:
            expert, shared = 3 * h * moe.expert_ffn, 3 * h * moe.n_shared * moe.shared_ffn
            touched = moe.num_experts * (1 - (1 - moe.top_k / moe.num_experts) ** rows)
            nbytes += touched * expert * {"fp8_block": 1.0, "nvfp4": 0.5625}[moe.expert_format] + 2 * moe.num_experts * h
            nbytes += shared * (1 if moe.expert_format == "fp8_block" else 2)
            flops += 2 * rows * (moe.top_k * expert + shared + moe.num_experts * h)
    return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
    # BF16 activations and an 8- to 10-fold rounded residual stream: GEMM splits, fused roundings and another attention kernel were
    # seen to change the logits by 0.012 to 0.02 (largest element 0.1) and the cache by 0.02. With experts, a choice that rounding
    # turns exchanges one of a row's eight experts (largest element 0.5)
    return {"dense": {"rel": 0.03, "max": 0.4}, "fp4": {"rel": 0.03, "max": 1.0 - 1e-9}, "fp8": {"rel": 0.03, "max": 1.0 - 1e-9}}[case["family"]]


# ------------------------------------------------------------------------------------------
# the same in 64 bits
# ------------------------------------------------------------------------------------------
def _norm64(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rope64(x, pos, theta):
    """x [rows, heads, d]: halves rotated against each other."""
    d = x.shape[-1]
    inv = theta ** (-torch.arange(0, d, 2, dtype=torch.float64, device=x.device) / d)
    ang = pos.double()[:, None, None] * inv
    c, s = torch.cos(ang), torch.sin(ang)
    a, b = x[..., : d // 2], x[..., d // 2:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _attend64(q, k, v, scale):
    """q [n, heads, d] at the last n positions, k and v [ctx, kv heads, .]."""
    n, heads, _ = q.shape
    ctx, group = k.shape[0], heads // k.shape[1]
    out = q.new_empty(n, heads, v.shape[-1])
    hidden = torch.arange(ctx, device=q.device)[None] > torch.arange(ctx - n, ctx, device=q.device)[:, None]
    for h in range(heads):
        s = (q[:, h] @ k[:, h // group].t()) * scale
        out[:, h] = torch.softmax(s.masked_fill_(hidden, float("-inf")), -1) @ v[:, h // group]
    return out


def _ffn64(x, get, p):
    g = x @ get(p + "gate_proj.weight").t()
    return (g * torch.sigmoid(g) * (x @ get(p + "up_proj.weight").t())) @ get(p + "down_proj.weight").t()


def _experts64(x, spec, get, p):
    moe = spec.moe
    logits = x @ get(p + "gate.weight", (moe.num_experts, spec.hidden)).t()
    if moe.score == "softmax":
        score = torch.softmax(logits, -1)
        ids = score.topk(moe.top_k, -1).indices
    else:
        score = torch.sigmoid(logits)
        groups = score.view(len(x), moe.n_groups, -1)
        best = groups.topk(2, -1).values.sum(-1).topk(moe.topk_groups, -1).indices
        keep = torch.zeros(len(x), moe.n_groups, dtype=torch.bool, device=x.device).scatter_(1, best, True)
        ids = groups.masked_fill(~keep[..., None], -1.0).reshape(len(x), -1).topk(moe.top_k, -1).indices
    w = score.gather(1, ids)
    w = w / w.sum(-1, keepdim=True) * moe.routed_scaling
    out = torch.zeros_like(x)
    f = moe.expert_ffn
    shape = lambda n: (spec.hidden, f) if "down" in n else (f, spec.hidden)
    for e in range(moe.num_experts):
        r, c = torch.nonzero(ids == e, as_tuple=True)
        if r.numel():
            out[r] += w[r, c, None] * _ffn64(x[r], lambda n: get(n, shape(n)), p + f"experts.{e}.")
    if moe.n_shared:
        sf = moe.shared_ffn
        shape = lambda n: (spec.hidden, sf) if "down" in n else (sf, spec.hidden)
        out += _ffn64(x, lambda n: get(n, shape(n)), p + "shared_experts.")
    return out


@torch.no_grad()
def exact(case, seed):
    """The same step in 64 bits. Dense layers of thousands of rows are the cost: about 10 seconds for the largest."""
    _loaded.clear()
    torch.cuda.empty_cache()
    family, spec, lens = case["family"], _spec(case["family"]), _lengths(case)
    get = lambda name, shape: _weight(family, name, shape).double()
    decode = case["kind"] == "decode"
    new = [1] * len(lens) if decode else lens
    ids = torch.tensor(sum(_tokens(spec, new, seed), []), device="cuda")
    pos = torch.cat([torch.arange(n, n + 1) if decode else torch.arange(n) for n in lens]).cuda()
    starts = [sum(new[:i]) for i in range(len(new))]
    used = _blocks(lens)
    total = sum(used) + len(lens) + 1
    # pages in the order they are handed out: every sequence's context, then those the new tokens open
    pages, nxt = [], 0
    for u in used:
        pages.append(list(range(nxt, nxt + u)))
        nxt += u
    if decode:
        for i, n in enumerate(lens):
            if n % PAGE == 0:
                pages[i].append(nxt)
                nxt += 1
    x = get("model.embed_tokens.weight", (spec.vocab, spec.hidden))[ids]
    h, d, a = spec.hidden, spec.head_dim, spec.mla
    caches = [[], []]
    for i in range(spec.layers):
        p = f"model.layers.{i}."
        n = _norm64(x, get(p + "input_layernorm.weight", (h,)), spec.rms_eps)
        att = p + "self_attn."
        lin = lambda y, name, out: y @ get(att + name, (out, y.shape[1])).t()
        if a is not None:
            qk = a.qk_nope_dim + a.qk_rope_dim
            qa = _norm64(lin(n, "q_a_proj.weight", a.q_lora_rank), get(att + "q_a_layernorm.weight", (a.q_lora_rank,)), spec.rms_eps)
            q = lin(qa, "q_b_proj.weight", spec.heads * qk).view(-1, spec.heads, qk)
            q = torch.cat([q[..., : a.qk_nope_dim], _rope64(q[..., a.qk_nope_dim:], pos, spec.rope_theta)], -1)
            kva = lin(n, "kv_a_proj_with_mqa.weight", a.kv_lora_rank + a.qk_rope_dim)
            lat = _norm64(kva[:, : a.kv_lora_rank], get(att + "kv_a_layernorm.weight", (a.kv_lora_rank,)), spec.rms_eps)
            rows = [torch.cat([lat, _rope64(kva[:, None, a.kv_lora_rank:], pos, spec.rope_theta)[:, 0]], -1)[:, None]]
            scale, vdim = qk ** -0.5, a.v_head_dim
            kv_b = get(att + "kv_b_proj.weight", (spec.heads * (a.qk_nope_dim + vdim), a.kv_lora_rank)).view(spec.heads, -1, a.kv_lora_rank)
        else:
            q, k = lin(n, "q_proj.weight", spec.q_dim).view(-1, spec.heads, d), lin(n, "k_proj.weight", spec.kv_dim).view(-1, spec.kv_heads, d)
            if spec.qk_norm:
                q, k = _norm64(q, get(att + "q_norm.weight", (d,)), spec.rms_eps), _norm64(k, get(att + "k_norm.weight", (d,)), spec.rms_eps)
            q = _rope64(q, pos, spec.rope_theta)
            rows = [_rope64(k, pos, spec.rope_theta), lin(n, "v_proj.weight", spec.kv_dim).view(-1, spec.kv_heads, d)]
            scale, vdim = d ** -0.5, d
        ctx = [t.double() for t in _cached(spec, i, sum(used), seed) if t is not None] if decode else [None] * len(rows)
        pools = []
        for t, c in zip(rows, ctx):
            pool = t.new_zeros(total, t.shape[1], PAGE, t.shape[2])
            if c is not None:
                pool[: sum(used)] = c
            pools.append(pool)
        o = x.new_empty(len(x), spec.heads, vdim)
        for b, m in enumerate(new):
            at = pos[starts[b]: starts[b] + m]
            pg = torch.tensor(pages[b], device="cuda")
            for pool, t in zip(pools, rows):
                pool[pg[at // PAGE], :, at % PAGE] = t[starts[b]: starts[b] + m]
            seen = lens[b] + 1 if decode else lens[b]
            got = [pool[pg].transpose(1, 2).reshape(-1, pool.shape[1], pool.shape[3])[:seen] for pool in pools]
            if a is not None:
                r = got[0][:, 0]
                both = torch.einsum("tl,hol->tho", r[:, : a.kv_lora_rank], kv_b)
                keys = torch.cat([both[..., : a.qk_nope_dim], r[:, None, a.kv_lora_rank:].expand(-1, spec.heads, -1)], -1)
                got = [keys, both[..., a.qk_nope_dim:]]
            o[starts[b]: starts[b] + m] = _attend64(q[starts[b]: starts[b] + m], got[0], got[1], scale)
        for kind, pool in zip(caches, pools):
            kind.append(pool)
        x = x + o.reshape(len(x), -1) @ get(att + "o_proj.weight", (h, spec.heads * vdim)).t()
        n = _norm64(x, get(p + "post_attention_layernorm.weight", (h,)), spec.rms_eps)
        moe = spec.moe
        if moe is None or i < moe.first_dense_layers:
            f = moe.dense_ffn if moe is not None and moe.dense_ffn else spec.ffn
            x = x + _ffn64(n, lambda name: get(name, (h, f) if "down" in name else (f, h)), p + "mlp.")
        else:
            x = x + _experts64(n, spec, get, p + "mlp.")
    last = torch.tensor([s + m - 1 for s, m in zip(starts, new)], device="cuda")
    n = _norm64(x[last], get("model.norm.weight", (h,)), spec.rms_eps)
    logits = n @ get("lm_head.weight", (spec.vocab, h)).t()
    return {"logits": logits, "cache": caches[0] + caches[1]}
