"""Row-wise kernels between the products of a layer, against the operators they stand for."""
import pytest
import torch

from flyingfish_b200.ops import ref

BF16 = torch.bfloat16


def _packed(rows, heads, dim, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(rows, heads * dim, generator=g).to(BF16)


def _batch(rows, hq, hkv, dim):
    g = torch.Generator().manual_seed(rows + dim)
    nb = (rows + 63) // 64 + 1
    slots = torch.randperm(nb * 64, generator=g)[:rows].to(torch.int32)
    slots[rows // 2] = -1 if rows > 1 else slots[0]
    pos = torch.randint(0, 9000, (rows,), generator=g).to(torch.int32)
    return _packed(rows, hq + 2 * hkv, dim, rows + dim), pos, slots, [torch.zeros(nb, hkv, 64, dim, dtype=BF16) for _ in range(2)]


ROWS = [1, 7, 299, 600, 2368, 2371, 4741]   # one row per CTA, two and four for few heads, the first size with four for all, ragged ones, more for one head
HEADS = [(4, 1, 128, 128), (64, 4, 128, 128), (3, 2, 128, 64), (5, 1, 64, 64), (2, 2, 48, 32), (1, 1, 16, 16)]


@pytest.mark.gpu
@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("hq,hkv,dim,rot", HEADS)
def test_rotation_and_cache_write(rows, hq, hkv, dim, rot):
    """With the angles given, rotation and cache write are the oracle's bits; the kernel that makes the angles itself turns by those of the
    table kernel, which differ from the host's by a last bit of BF16 (and by what FP32 gives an angle of up to 9000)."""
    from flyingfish_b200 import ops
    from flyingfish_b200.ops import vision_ops
    qkv, pos, slots, caches = _batch(rows, hq, hkv, dim)
    table = ops.rope_table(pos, rot, 1e6)
    want, got = [[qkv.to(d), *(c.to(d) for c in caches)] for d in ("cpu", "cuda")]
    vision_ops.rope_table_apply_(want[0], table, hq, dim, rot, slots, want[1], want[2], hkv)
    vision_ops.rope_table_apply_(got[0], table.cuda(), hq, dim, rot, slots.cuda(), got[1], got[2], hkv)
    assert all(torch.equal(a.cpu(), b) for a, b in zip(got, want))
    own, by_table = [[qkv.cuda(), *(c.cuda() for c in caches)] for _ in range(2)]
    angles = ops.rope_table(pos.cuda(), rot, 1e6)
    ops.rope_kv_paged(own[0], pos.cuda(), slots.cuda(), own[1], own[2], hq, hkv, dim, 1e6, rot)
    vision_ops.rope_table_apply_(by_table[0], angles, hq, dim, rot, slots.cuda(), by_table[1], by_table[2], hkv)
    assert all(torch.equal(a, b) for a, b in zip(own, by_table))
    assert (angles.cpu() - table).abs().max() <= 2.0 ** -8 + 9000 * 2.0 ** -22
    torch.cuda.synchronize()
    ops.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("hq,hkv,dim,rot", HEADS)
def test_head_norms_before_the_rotation(rows, hq, hkv, dim, rot):
    """At position 0 what is left is the norm: the oracle's up to its last bit (2^-7 of a value at most), since the sums of squares meet in
    another order. Elsewhere the pass gives the bits of that norm followed by the plain rotation."""
    from flyingfish_b200 import ops
    qkv, pos, slots, caches = _batch(rows, hq, hkv, dim)
    g = torch.Generator().manual_seed(1)
    w = [(1 + 0.1 * torch.randn(dim, generator=g)).to(BF16) for _ in range(2)]
    kw = dict(q_norm=w[0].cuda(), k_norm=w[1].cuda(), eps=1e-6)

    def turned(x, positions, **norms):
        out = [x.cuda(), *(c.cuda() for c in caches)]
        ops.rope_kv_paged(out[0], positions.cuda(), slots.cuda(), out[1], out[2], hq, hkv, dim, 1e6, rot, **norms)
        return out
    normed = turned(qkv, torch.zeros_like(pos), **kw)[0].cpu()
    heads = qkv.view(rows, -1, dim)
    want = torch.cat([ref.rmsnorm(heads[:, :hq], w[0], 1e-6), ref.rmsnorm(heads[:, hq: hq + hkv], w[1], 1e-6)], 1).view(rows, -1).float()
    assert ((normed[:, : want.shape[1]].float() - want).abs() <= 2.0 ** -7 * want.abs()).all()
    assert torch.equal(normed[:, want.shape[1]:], qkv[:, want.shape[1]:])                        # values are copies
    assert all(torch.equal(a, b) for a, b in zip(turned(qkv, pos, **kw), turned(normed, pos)))
    torch.cuda.synchronize()
    ops.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("rows,hidden,top_k", [(1, 8, 1), (3, 1032, 3), (70, 4104, 9), (5, 2048, 16)])      # parts of a CTA, of its loads, the most choices
@pytest.mark.parametrize("accumulate", [False, True])
def test_expert_rows_dispatched_and_combined(rows, hidden, top_k, accumulate):
    """Rows reach every choice's place; the weighted sum skips choices served elsewhere."""
    from flyingfish_b200 import ops
    from flyingfish_b200.ops import moe_cuda
    experts, g = 24, torch.Generator().manual_seed(rows)
    x = torch.randn(rows, hidden, generator=g).to(BF16)
    ids = torch.stack([torch.randperm(experts, generator=g)[:top_k] for _ in range(rows)]).to(torch.int32)
    w = torch.rand(rows, top_k, generator=g)
    lo, hi = 3, experts - 2                                   # the others' choices belong to another rank
    xs, pos, _, _, cap = moe_cuda.dispatch_local(x.cuda(), ids.cuda(), experts, lo, hi)
    served = ((ids >= lo) & (ids < hi)).view(-1)
    assert torch.equal(pos.cpu() >= 0, served)
    assert torch.equal(xs[pos.long()[served.cuda()]].cpu(), x.repeat_interleave(top_k, 0)[served])
    y, out = torch.randn(cap, hidden, generator=g).to(BF16).cuda(), torch.randn(rows, hidden, generator=g).to(BF16).cuda()
    before = out.double().cpu()
    got = moe_cuda.combine(y, pos, ids.cuda(), w.cuda(), rows, hidden, **(dict(out=out, accumulate=True) if accumulate else {}))
    torch.cuda.synchronize()
    ops.check_status()
    terms = y.cpu().double()[pos.long().cpu().clamp_min(0)].view(rows, top_k, hidden) * (w.double() * served.view(rows, top_k))[..., None]
    want, size = terms.sum(1), terms.abs().sum(1)
    if accumulate:
        want, size = want + before, size + before.abs()
    # one rounding of the result, a rounding of FP32 per addition
    assert ((got.double().cpu() - want).abs() <= 2.0 ** -8 * want.abs() + (top_k + 1) * 2.0 ** -23 * size).all()


def _mla_batch(q_lens, pasts, seed):
    g = torch.Generator().manual_seed(seed)
    ql = torch.tensor(q_lens, dtype=torch.int32)
    ctx = ql + torch.tensor(pasts, dtype=torch.int32)
    blocks = int(((ctx + 63) // 64).sum()) + 1
    width = int(((ctx + 63) // 64).max())
    table, free = torch.zeros(len(q_lens), width, dtype=torch.int32), torch.randperm(blocks, generator=g).tolist()
    for b, c in enumerate(ctx.tolist()):
        n = (c + 63) // 64
        table[b, :n] = torch.tensor([free.pop() for _ in range(n)], dtype=torch.int32)
    pos = torch.cat([torch.arange(p, p + n) for n, p in zip(q_lens, pasts)]).to(torch.int32)
    slots = torch.cat([table[b, torch.arange(p, p + n) // 64].long() * 64 + torch.arange(p, p + n) % 64 for b, (n, p) in enumerate(zip(q_lens, pasts))])
    return g, ql, (torch.cumsum(ql, 0) - ql).to(torch.int32), ctx, table, blocks, pos, slots.to(torch.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 3, 200])
def test_latent_row_step_equals_its_operators(rows):
    """The fused step gives the bits of the rotation kernel and the cache write, and the norm's up to its order of additions."""
    from flyingfish_b200 import ops
    from flyingfish_b200.ops import mla_ops
    heads, nope = 5, 128
    g, *_, blocks, pos, slots = _mla_batch([rows], [37], 2)
    q, kva = torch.randn(rows, heads * (nope + 64), generator=g).to(BF16), torch.randn(rows, 576, generator=g).to(BF16)
    w = (1 + 0.1 * torch.randn(512, generator=g)).to(BF16)
    slots[rows // 2] = -1 if rows > 1 else slots[0]
    q_rope = q.view(rows, heads, -1)[:, :, nope:].reshape(rows, -1).cuda()
    k_rope = kva[:, 512:].cuda()
    ops.rope_inplace(q_rope, pos.cuda(), heads, 64, 1e4)
    ops.rope_inplace(k_rope, pos.cuda(), 1, 64, 1e4)
    want = torch.zeros(blocks, 1, 64, 576, dtype=BF16)
    mla_ops.cache_write(ops.rmsnorm(kva[:, :512], w, 1e-6), k_rope.cpu(), slots, want)
    for full in (False, True):
        qd, cache = q.cuda(), torch.zeros_like(want).cuda()
        q_full = torch.zeros(rows, heads, 576, dtype=BF16, device="cuda") if full else None
        mla_ops.norm_rope_cache(qd, kva.cuda(), w.cuda(), pos.cuda(), slots.cuda(), cache, heads, nope, 1e4, 1e-6, q_full)
        torch.cuda.synchronize()
        ops.check_status()
        got = q_full[:, :, 512:] if full else qd.view(rows, heads, -1)[:, :, nope:]
        assert torch.equal(got.reshape(rows, -1), q_rope)
        cache = cache.cpu()
        assert torch.equal(cache[..., 512:], want[..., 512:])
        a, b = cache[..., :512].float(), want[..., :512].float()
        assert ((a - b).abs() <= 2.0 ** -7 * b.abs()).all()                                     # one last bit
        assert torch.equal(qd.view(rows, heads, -1)[:, :, :nope].cpu(), q.view(rows, heads, -1)[:, :, :nope])


@pytest.mark.gpu
@pytest.mark.parametrize("q_lens,pasts", [([64], [0]), ([1, 130, 63], [70, 0, 129]), ([65, 64], [64, 1])])
def test_expanded_attention_over_packed_heads(q_lens, pasts):
    """Keys and values expanded from the latents, queries as the projection leaves them, against attention in 64 bits."""
    from flyingfish_b200 import ops
    from flyingfish_b200.ops import mla_ops
    heads, nope, rot, dv, rank = 3, 128, 64, 128, 512
    g, ql, qs, ctx, table, blocks, *_ = _mla_batch(q_lens, pasts, 5)
    rows = int(ql.sum())
    q = torch.randn(rows, heads * (nope + rot), generator=g).to(BF16)
    cache = torch.randn(blocks, 1, 64, rank + rot, generator=g).to(BF16)
    w_kv = (0.02 * torch.randn(heads * (nope + dv), rank, generator=g)).to(BF16)
    scale = (nope + rot) ** -0.5
    pages = mla_ops.KeyPages.of(ql.tolist(), ctx.tolist(), table, 0, 64, "cuda")
    out = torch.empty(rows, heads * dv, dtype=BF16, device="cuda")
    qd = q.cuda()
    mla_ops.expanded_attention(qd, qd.view(rows, heads, -1), cache.cuda(), w_kv.cuda(), pages, table.cuda(), qs.cuda(), ql.cuda(), ctx.cuda(), max(q_lens),
                               nope, dv, rank, scale, 0, None, out)
    torch.cuda.synchronize()
    ops.check_status()
    for b in range(len(q_lens)):
        lat = cache[table[b].long(), 0].reshape(-1, rank + rot)[: int(ctx[b])].double()
        n, s0 = q_lens[b], int(qs[b])
        hide = torch.arange(len(lat))[None] > torch.arange(len(lat) - n, len(lat))[:, None]
        for h in range(heads):
            k = torch.cat([lat[:, :rank] @ w_kv[h * nope: (h + 1) * nope].double().t(), lat[:, rank:]], 1)
            v = lat[:, :rank] @ w_kv[heads * nope + h * dv: heads * nope + (h + 1) * dv].double().t()
            s = (q[s0: s0 + n].view(n, heads, -1)[:, h].double() @ k.t()) * scale
            want = torch.softmax(s.masked_fill(hide, float("-inf")), -1) @ v
            got = out[s0: s0 + n].view(n, heads, dv)[:, h].cpu().double()
            # keys, values, weights and results are rounded to BF16 (2^-9 each): four roundings of values of about 0.5
            assert ((got - want).abs() <= 1e-2 + 1e-2 * want.abs()).all()


@pytest.mark.gpu
@pytest.mark.parametrize("vocab", [8, 1000, 16384, 40008, 49160])          # parts of a round of two and of four vectors, a tail of single logits
def test_argmax_by_rows_of_an_sm(vocab):
    """Both instances: a row per SM at most, and more. Equal logits give the lower id."""
    from flyingfish_b200 import ops
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for rows in (1, sms, sms + 1, 2 * sms + 3):
        lg = (torch.randn(rows, vocab, generator=torch.Generator().manual_seed(rows)) * 4).round().to(BF16)       # many ties
        got = ops.argmax_rows(lg.cuda()).cpu().long()
        top = lg == lg.amax(1, keepdim=True)
        assert torch.equal(got, top.int().argmax(1))
    ops.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("hidden", [8200, 16384])                # parts of a thread's vectors, all of them
@pytest.mark.parametrize("waves", [1, 4, 5, 6])
def test_norm_of_wide_rows(hidden, waves):
    """Rows around the waves at which another instance runs: the bits of the same rows normed a few at a time, and those near 64 bits."""
    from flyingfish_b200 import ops
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    w = (1 + 0.1 * torch.randn(hidden, generator=torch.Generator().manual_seed(1))).to(BF16)
    for rows in (waves * sms, waves * sms + 1):
        x = torch.randn(rows, hidden, generator=torch.Generator().manual_seed(rows)).to(BF16).cuda()
        got = ops.rmsnorm(x, w.cuda(), 1e-6)
        few = torch.cat([ops.rmsnorm(part.contiguous(), w.cuda(), 1e-6) for part in x.split(100)])
        assert torch.equal(got, few)
        some = x[:: max(1, rows // 20)].cpu().double()
        want = some * torch.rsqrt(some.square().mean(-1, keepdim=True) + 1e-6) * w.double()
        # one rounding of the result; the sum and its root in FP32
        assert ((got[:: max(1, rows // 20)].cpu().double() - want).abs() <= (2.0 ** -8 + 2.0 ** -20) * want.abs()).all()
    ops.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("rows,hidden,top_k", [(319, 2056, 1), (320, 2056, 1), (330, 1032, 2), (320, 520, 3), (400, 4104, 4), (511, 2056, 6), (512, 2056, 6), (600, 1032, 16)])
def test_expert_rows_of_many_rows_combined(rows, hidden, top_k):
    """A CTA per row and several: the weighted sum of a row's choices, some of them served elsewhere, vectors left over behind the last round."""
    from flyingfish_b200 import ops
    from flyingfish_b200.ops import moe_cuda
    g = torch.Generator().manual_seed(rows)
    ids = torch.stack([torch.randperm(40, generator=g)[:top_k] for _ in range(rows)]).to(torch.int32)
    pos = torch.randperm(rows * top_k, generator=g).to(torch.int32)
    pos[torch.rand(rows * top_k, generator=g) < 0.2] = -1
    w, y = torch.rand(rows, top_k, generator=g), torch.randn(rows * top_k, hidden, generator=g).to(BF16)
    got = moe_cuda.combine(y.cuda(), pos.cuda(), ids.cuda(), w.cuda(), rows, hidden).cpu().double()
    ops.check_status()
    terms = y.double()[pos.long().clamp_min(0)].view(rows, top_k, hidden) * (w.double() * (pos >= 0).view(rows, top_k))[..., None]
    want, size = terms.sum(1), terms.abs().sum(1)
    # one rounding of the result, a rounding of FP32 per addition
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + (top_k + 1) * 2.0 ** -23 * size).all()
