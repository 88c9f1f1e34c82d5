"""Products and reductions at the sizes where a tile, a chunk or a split ends."""
import subprocess

import pytest
import torch

from flyingfish_b200.loaders import quant as qref
from flyingfish_b200.ops import ref

BF16 = torch.bfloat16


def _rand(shape, seed, dtype=BF16):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(dtype)


def _check(got, want, k, dtype=BF16):
    """One rounding to the result's type, and FP32 sums of k products of unit size (k 2^-24 of their root k norm, with room for the
    tensor core's alignment of partial products)."""
    got = got.cpu().double()
    rounding = 2.0 ** -8 if dtype == BF16 else 0.0
    assert ((got - want).abs() <= rounding * want.abs() + 2.0 ** -20 * k).all(), (got - want).abs().max()


@pytest.mark.gpu
@pytest.mark.parametrize("m", [129, 255, 256, 257, 1000])        # second row tile of a pair empty, ragged, full; several pairs
@pytest.mark.parametrize("n,k", [(136, 72), (256, 64), (520, 520), (6144, 512)])
@pytest.mark.parametrize("odt", [BF16, torch.float32])
def test_pair_gemm(m, n, k, odt):
    from flyingfish_b200 import ops
    x, w = _rand((m, k), m), _rand((n, k), n)
    y = ops.linear(x.cuda(), w.cuda(), out_dtype=odt)
    torch.cuda.synchronize()
    ops.check_status()
    _check(y, x.double() @ w.double().t(), k, odt)


@pytest.mark.gpu
@pytest.mark.parametrize("kblocks", [1, 5, 6, 7, 8, 9, 12, 13, 16, 17])          # rings of six and eight stages: not full, full, begun again
@pytest.mark.parametrize("m,n", [(129, 256), (1536, 4096)])                      # one tile per pair, several
def test_pair_gemm_ends_with_its_last_stages(m, n, kblocks):
    """The producers wait for the last commit of every stage they used: a phase that never completes would show in the status word."""
    from flyingfish_b200 import ops
    k = 64 * kblocks
    x, w = _rand((m, k), m), _rand((n, k), n)
    y = ops.linear(x.cuda(), w.cuda())
    torch.cuda.synchronize()
    ops.check_status()
    _check(y, x.double() @ w.double().t(), k)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(200, 264, 128), (300, 4096, 200)])
def test_pair_gemm_tail(m, n, k):
    from flyingfish_b200 import ops
    x, w, bias = _rand((m, k), 1), _rand((n, k), 2), _rand((n,), 3)
    y = ops.linear(x.cuda(), w.cuda(), bias=bias.cuda(), act="relu2")
    want = (x.double() @ w.double().t() + bias.double()).clamp_min(0) ** 2
    # the square doubles the sum's relative error: absolute 2 |sum| times it
    assert ((y.cpu().double() - want).abs() <= 2.0 ** -8 * want + 2.0 ** -19 * k * want.sqrt() + 1e-3).all()


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["plain", "fp32", "pitches", "bias relu2", "bias gelu factors", "swiglu", "gated 3", "gated 5"])
@pytest.mark.parametrize("k", [64, 520, 584, 2048])
def test_pairs_and_single_ctas_give_the_same_bits(form, k):
    """Sixteen column tiles: 1000 rows are one wave of pairs and 1100 rows two, where 128-row tiles of one CTA need one (of K up to 512
    both sizes take those). The rows that both calls have must agree, whatever the epilogue and the pitches."""
    from flyingfish_b200 import ops
    x = _rand((1100, k + 8), 1).cuda()[:, : k]                                  # rows 16 bytes apart from being contiguous
    n = 4096 if form.startswith(("swiglu", "gated")) else 4072                   # a ragged last tile where the form takes one
    w = (_rand((n, k + 16), 2) * 0.1).cuda()[:, 8: k + 8]
    bias, table, ids = _rand((n,), 3).cuda(), _rand((7, n), 4).cuda(), torch.randint(0, 7, (1100,), generator=torch.Generator().manual_seed(5)).to(torch.int32).cuda()

    def run(m):
        if form == "fp32":
            return ops.linear(x[:m], w, out_dtype=torch.float32)
        if form == "pitches":
            out = torch.full((m, n + 24), 7.0, dtype=BF16, device="cuda")
            ops.linear(x[:m], w, out=out[:, 8: n + 8])
            assert (out[:, :8] == 7).all() and (out[:, n + 8:] == 7).all()
            return out
        if form == "bias relu2":
            return ops.linear(x[:m], w, bias=bias, act="relu2")
        if form == "bias gelu factors":
            return ops.linear(x[:m], w, bias=bias, act="gelu_tanh", mul=(table, ids[:m].contiguous()))
        if form == "swiglu" or form.startswith("gated"):
            mode = 0 if form == "swiglu" else int(form[-1])
            return ops.linear_swiglu(x[:m], w, mode=mode, limit=1.5)
        return ops.linear(x[:m], w)
    many, few = run(1100), run(1000)
    torch.cuda.synchronize()
    ops.check_status()
    assert torch.equal(many[:1000], few)
    if form in ("plain", "fp32"):
        want = x.cpu().double() @ w.cpu().double().t()
        _check(many, want, k, torch.float32 if form == "fp32" else BF16)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n", [(129, 256), (700, 5888), (256, 19200)])       # narrow and wide column tiles
def test_pair_gemm_gate(m, n):
    from flyingfish_b200 import ops
    x, w = _rand((m, 128), 4), _rand((n, 128), 5)
    got = ops.linear_swiglu(x.cuda(), w.cuda()).cpu().float()
    want = ref.linear_swiglu(x, w).float()
    # gate and up are rounded to BF16 before the product: sums on either side of a rounding boundary differ by a last bit each
    assert ((got - want).abs() <= 3 * 2.0 ** -8 * want.abs() + 2e-2).all()


def _pair_tiles(m, n, epi, pairs=74):
    import ctypes
    from flyingfish_b200.ops.lib import kernels
    out = (ctypes.c_int * 3)()
    assert kernels().ff_gemm_bf16_pair_tiles(m, n, epi, pairs, out) == 0
    return tuple(out)


@pytest.mark.parametrize("epi", [0, 1])
def test_pair_tiles_cover_the_columns(epi):
    """Widths the tensor cores and the epilogue take, wide columns that leave something to the narrow ones or nothing, no empty column."""
    mixed = 0
    for m in (129, 256, 257, 700, 1000, 2500, 8191, 70000):
        for n in (256, 512, 768, 4096, 6144, 28672) + (() if epi else (1, 31, 32, 63, 65, 136, 257, 576, 129280)):
            for pairs in (1, 16, 74):
                w1, wide, w2 = _pair_tiles(m, n, epi, pairs)
                step = 128 if epi else 32
                assert w1 % step == w2 % step == 0 and 64 <= w2 <= w1 <= 256
                rest = n - wide * w1
                assert rest > -w1 and wide * w1 + max(0, -(-rest // w2)) * w2 >= n
                mixed += 0 < wide and rest > 0 and w1 != w2
    assert mixed > 10


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,mixed", [(1000, 6144, 128, True), (2500, 4096, 704, True), (300, 6144, 832, False), (600, 4104, 64, False)])
def test_pair_gemm_of_two_widths(m, n, k, mixed):
    """Wide and narrow tiles in one launch and tiles of one odd width, rings of 7 to 11 stages begun again, a last tile past the columns."""
    from flyingfish_b200 import ops
    w1, wide, w2 = _pair_tiles(m, n, 0)
    assert (0 < wide * w1 < n and w1 != w2) if mixed else wide == 0 and w2 < 256
    x, w = _rand((m, k), m), _rand((n, k), n)
    y = ops.linear(x.cuda(), w.cuda())
    torch.cuda.synchronize()
    ops.check_status()
    _check(y, x.double() @ w.double().t(), k)


@pytest.mark.gpu
def test_pair_gemm_gate_of_two_widths():
    from flyingfish_b200 import ops
    m, n = 300, 28672
    w1, wide, w2 = _pair_tiles(m, n, 1)
    assert 0 < wide * w1 < n and (w1, w2) == (256, 128)
    x, w = _rand((m, 64), 4), _rand((n, 64), 5)
    got, want = ops.linear_swiglu(x.cuda(), w.cuda()), ops.silu_mul_interleaved(ops.linear(x.cuda(), w.cuda()))
    torch.cuda.synchronize()
    ops.check_status()
    assert torch.equal(got, want)                                # the activation kernel rounds at the same places


@pytest.mark.gpu
@pytest.mark.parametrize("counts", [[64, 1, 65, 0, 50, 33, 63, 47], [16, 17, 0, 32, 33, 1, 31, 30], [100, 128, 129, 16]])   # chunks of 64, 32, 128
@pytest.mark.parametrize("epi", [0, 1])
def test_grouped_fp8_chunks(counts, epi):
    from flyingfish_b200 import ops
    from flyingfish_b200.ops import quant_ops
    e, n, k = len(counts), 256, 384
    pad = [(c + 15) // 16 * 16 for c in counts]
    off = [sum(pad[:i]) for i in range(e + 1)]
    x = _rand((off[-1], k), 7)
    w = [qref.quantize_fp8_block_weight(_rand((n, k), 10 + i).float()) for i in range(e)]
    codes, scale = torch.stack([c for c, _ in w]), torch.stack([s for _, s in w])
    xq, xs = qref.quantize_fp8_act(x)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    y = quant_ops.grouped_gemm_fp8(xq.cuda(), xs.cuda(), codes.cuda(), scale.cuda(), i32(off), i32(counts), off[-1], epi).cpu().float()
    torch.cuda.synchronize()
    ops.check_status()
    for i, c in enumerate(counts):
        if c:
            rows = qref.fp8_block_linear(x[off[i]: off[i] + c], codes[i], scale[i])
            want = ref.silu_mul(quant_ops._deinterleave_cols(rows)).float() if epi else rows.float()
            got = y[off[i]: off[i] + c]
            assert ((got - want).abs() <= 3 * 2.0 ** -8 * want.abs() + 2e-2).all()      # roundings as in the gated product above


@pytest.mark.gpu
@pytest.mark.parametrize("rows,hidden,experts,top_k", [(1, 128, 4, 1), (64, 1152, 32, 8), (200, 512, 7, 3), (3000, 256, 1000, 4)])
def test_quantised_rows_dispatched(rows, hidden, experts, top_k):
    """Rows quantised in front of the dispatch, and rows of segments, have the codes and scales of rows quantised behind it."""
    from flyingfish_b200 import ops
    from flyingfish_b200.ops import moe_cuda, quant_ops
    x = _rand((rows, hidden), rows).cuda()
    g = torch.Generator().manual_seed(rows)
    ids = torch.stack([torch.randperm(experts, generator=g)[:top_k] for _ in range(rows)]).to(torch.int32).cuda()
    xq, xs, pos, seg_off, counts, cap = moe_cuda.dispatch_fp8(*quant_ops.quant_fp8_act(x), ids, experts, 0, experts)
    want_q, want_s = quant_ops.quant_fp8_act(x)
    row = torch.arange(rows, device="cuda").repeat_interleave(top_k)
    at = pos.long()
    assert at.unique().numel() == rows * top_k
    assert torch.equal(xq[at], want_q[row]) and torch.equal(xs[at], want_s[row])
    assert torch.equal(counts.long(), torch.bincount(ids.view(-1).long(), minlength=experts))
    assert torch.equal(seg_off[1:].long() - seg_off[:-1].long(), (counts.long() + 15) // 16 * 16)
    lo, n = seg_off[:-1].long()[ids.view(-1).long()], counts.long()[ids.view(-1).long()]
    assert bool(((at >= lo) & (at < lo + n)).all())
    h = _rand((cap, hidden), 5).cuda()
    hq, hs = quant_ops.quant_fp8_segments(h, seg_off, counts, max(1, rows * top_k // experts))
    want_q, want_s = quant_ops.quant_fp8_act(h)
    torch.cuda.synchronize()
    ops.check_status()
    assert torch.equal(hq[at], want_q[at]) and torch.equal(hs[at], want_s[at])


@pytest.mark.gpu
@pytest.mark.parametrize("rows,experts,top_k", [(64, 256, 8), (5, 8, 2)])
def test_grouped_fp8_waits_for_its_offsets(rows, experts, top_k):
    """Counts and offsets by a kernel that lets the next ones start before it has written them. The buffers hold zeros until then: a product
    that read too early would store nothing."""
    from flyingfish_b200 import ops
    from flyingfish_b200.ops import moe_cuda, quant_ops
    from flyingfish_b200.ops.lib import check, kernels, ptr, status_tensor, stream_ptr
    n, k, cap = 256, 512, (rows * top_k + 16 * experts + 15) // 16 * 16
    logits, x = torch.randn(rows, experts, generator=torch.Generator().manual_seed(1)).cuda(), _rand((rows, 8), 2).cuda()
    xq, xs = quant_ops.quant_fp8_act(_rand((1, k), 3).cuda().expand(cap, k).contiguous())      # all rows alike: their order in a segment is free
    codes = torch.randint(0, 120, (experts, n, k), generator=torch.Generator().manual_seed(4), dtype=torch.uint8).cuda()
    scale = torch.rand(experts, n // 128, k // 128, generator=torch.Generator().manual_seed(5)).cuda()
    i32 = lambda m: torch.zeros(m, dtype=torch.int32, device="cuda")
    ids, pos, weights, sorted_x = i32(rows * top_k), i32(rows * top_k), torch.empty(rows * top_k, device="cuda"), torch.empty(cap, 8, dtype=BF16, device="cuda")
    full = lambda: torch.full((cap, n), 5.0, dtype=BF16, device="cuda")
    for _ in range(5):
        counts, seg_off, y = i32(experts), i32(experts + 1), full()
        torch.cuda._sleep(1_000_000)                          # so that the launches below are all queued before the first runs
        check(kernels().ff_moe_plan(ptr(logits), None, ptr(weights), ptr(ids), ptr(counts), ptr(seg_off), ptr(pos), rows, experts, experts, top_k,
                                    moe_cuda.SCORE_MODES["softmax"], experts, 1, ptr(x), ptr(sorted_x), 8, 8, 2, cap, ptr(status_tensor("cuda")), stream_ptr()), "plan")
        quant_ops.grouped_gemm_fp8(xq, xs, codes, scale, seg_off, counts, cap, 0, out=y)
        torch.cuda.synchronize()
        ops.check_status()
        assert int(counts.sum()) == rows * top_k
        assert torch.equal(y, quant_ops.grouped_gemm_fp8(xq, xs, codes, scale, seg_off, counts, cap, 0, out=full()))
        assert int((y != 5).any(1).sum()) == rows * top_k


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 16, 33, 64, 100])
@pytest.mark.parametrize("n,k", [(576, 7168), (136, 2048), (1536, 1152)])       # fourteen, four and two splits, a ragged edge
def test_fp8_partials_of_many_splits(m, n, k):
    from flyingfish_b200 import ops
    from flyingfish_b200.ops import quant_ops
    x = _rand((m, k), m)
    codes, scale = qref.quantize_fp8_block_weight(_rand((n, k), n).float())
    y = quant_ops.linear_fp8(x.cuda(), codes.cuda(), scale.cuda())
    torch.cuda.synchronize()
    ops.check_status()
    xq, xs = qref.quantize_fp8_act(x)
    wide = lambda c: c.view(torch.float8_e4m3fn).double()
    want = (wide(xq) * xs.double().repeat_interleave(128, 1)[:, :k]) @ (wide(codes) * scale.double().repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)[:, :k]).t()
    # one rounding of the result; the products of a K block are aligned to its largest partial sum (13 bits, a few times root 128)
    assert ((y.cpu().double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -11 * k ** 0.5).all()


@pytest.mark.gpu
@pytest.mark.parametrize("n,k", [(130, 272), (5, 132), (1, 16), (300, 4)])
def test_fp8_expansion_is_exact(n, k):
    from flyingfish_b200.ops import quant_ops
    codes, scale = qref.quantize_fp8_block_weight(_rand((n, k), 3).float())
    assert torch.equal(quant_ops.dequant_fp8_block(codes.cuda(), scale.cuda()).cpu(), qref.dequantize_fp8_block(codes, scale))


@pytest.mark.gpu
@pytest.mark.parametrize("counts", [[1, 8, 0, 9], [16, 17, 32, 33], [70, 0, 0, 2]])      # column tiles of 8, 16 and 32 tokens, further passes
@pytest.mark.parametrize("k", [128, 384, 768, 2304])         # scale rows of no whole 16 bytes, a ragged stage, token slabs that end inside K
@pytest.mark.parametrize("epi", [0, 1])
def test_grouped_nvfp4_passes(counts, k, epi):
    from flyingfish_b200 import ops
    from flyingfish_b200.ops import moe_cuda
    e, n = len(counts), 256
    pad = [(c + 15) // 16 * 16 for c in counts]
    off = [sum(pad[:i]) for i in range(e + 1)]
    x = _rand((off[-1], k), 7)
    q = [qref.quantize_nvfp4(_rand((n, k), 20 + i).float()) for i in range(e)]
    w = moe_cuda.Nvfp4Experts(*(torch.stack([p[j] for p in q]).cuda() for j in range(3)))
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    y = moe_cuda.grouped_gemm_nvfp4(x.cuda(), w, i32(off), i32(counts), off[-1], epi).cpu().float()
    torch.cuda.synchronize()
    ops.check_status()
    for i, c in enumerate(counts):
        if c:
            full = (qref.e2m1_decode(qref.e2m1_unpack(q[i][0])).view(n, -1, 16) * qref.e4m3_decode(q[i][1])[..., None]).view(n, k).double()
            rows = x[off[i]: off[i] + c].double() @ full.t() * float(q[i][2])
            got = y[off[i]: off[i] + c]
            if epi:
                g = rows.float().view(c, n // 128, 2, 64)
                want = ref.silu_mul(torch.cat([g[:, :, 0].reshape(c, -1), g[:, :, 1].reshape(c, -1)], 1).to(BF16)).float()
                assert ((got - want).abs() <= 3 * 2.0 ** -8 * want.abs() + 2e-2).all()  # roundings as in the gated product above
            else:
                _check(got, rows, k)


@pytest.mark.gpu
@pytest.mark.parametrize("counts,n,k", [
    ([1, 16, 0, 17, 63], 256, 256),                          # one K chunk, boxes of 64 rows that reach past a segment and past the buffer
    ([64, 65, 255], 384, 768),                               # whole boxes and one row more, an odd number of chunks
    ([256, 257, 0, 600], 256, 1280),                         # whole passes and further ones
    ([33] * 50, 512, 512),                                   # more tiles than CTAs: accumulators and rings begun again
])
@pytest.mark.parametrize("epi", [0, 1])
def test_grouped_nvfp4_for_prompts(counts, n, k, epi):
    """The tcgen05 kernel against 64 bits, and rows that belong to no segment untouched."""
    from flyingfish_b200 import ops
    from flyingfish_b200.ops import moe_cuda
    e = len(counts)
    pad = [(c + 15) // 16 * 16 for c in counts]
    off = [sum(pad[:i]) for i in range(e + 1)]
    x = _rand((off[-1], k), 7)
    kinds = [qref.quantize_nvfp4(_rand((n, k), 20 + i).float()) for i in range(min(e, 5))]
    q = [kinds[i % len(kinds)] for i in range(e)]
    w = moe_cuda.Nvfp4Experts(*(torch.stack([p[j] for p in q]).cuda() for j in range(3)))
    assert w.prompts()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    out = torch.full((off[-1], n // (2 if epi else 1)), 5.0, dtype=BF16, device="cuda")
    y = moe_cuda.grouped_gemm_nvfp4(x.cuda(), w, i32(off), i32(counts), off[-1], epi, out=out, rows_per_expert=1e6).cpu().float()
    torch.cuda.synchronize()
    ops.check_status()
    for i, c in enumerate(counts):
        assert (y[off[i] + c: off[i + 1]] == 5).all()
        if c:
            full = (qref.e2m1_decode(qref.e2m1_unpack(q[i][0])).view(n, -1, 16) * qref.e4m3_decode(q[i][1])[..., None]).view(n, k).double()
            rows = x[off[i]: off[i] + c].double() @ full.t() * float(q[i][2])
            got = y[off[i]: off[i] + c]
            if epi:
                g = rows.float().view(c, n // 128, 2, 64)
                g, u = g[:, :, 0].reshape(c, -1).double(), g[:, :, 1].reshape(c, -1).double()
                # gate (slope of silu at most 1.1), up, silu and the product are each rounded to BF16, 2^-9 of themselves; twice that, and FP32 sums
                act = torch.nn.functional.silu(g)
                bound = 2.0 ** -8 * (1.1 * g.abs() + 3 * act.abs()) * u.abs() + 2.0 ** -20 * k * (1 + g.abs() + u.abs())
                assert ((got - act * u).abs() <= bound).all()
            else:
                _check(got, rows, k)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,prompts", [(256, True), (300, True), (40, True), (32, False), (5, False)])
def test_packed_experts_repeat_their_bits(rows, prompts):
    """Rings refilled many times while the tensor cores hold the warps up that read them: every launch the bits of the first, and those near 64 bits."""
    from flyingfish_b200 import ops
    from flyingfish_b200.ops import moe_cuda
    e, n, k = 24, 2048, 4096
    g = torch.Generator(device="cuda").manual_seed(rows)
    codes = torch.randint(0, 256, (e, n, k // 2), dtype=torch.uint8, device="cuda", generator=g)
    scales = torch.randint(40, 60, (e, n, k // 16), dtype=torch.uint8, device="cuda", generator=g)
    w = moe_cuda.Nvfp4Experts(codes, scales, torch.ones(e, device="cuda"))
    pad = (rows + 15) // 16 * 16
    x = torch.randn(e * pad, k, device="cuda", generator=g).to(BF16)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    off, counts = i32([pad * i for i in range(e + 1)]), i32([rows] * e)
    run = lambda: moe_cuda.grouped_gemm_nvfp4(x, w, off, counts, e * pad, 0, rows_per_expert=1e6 if prompts else 0.0).view(e, pad, n)[:, :rows]
    first = run().clone()
    assert all(torch.equal(run(), first) for _ in range(20))
    ops.check_status()
    for i in (0, e - 1):
        full = (qref.e2m1_decode(qref.e2m1_unpack(codes[i].cpu())).view(n, -1, 16) * qref.e4m3_decode(scales[i].cpu())[..., None]).view(n, k).double()
        want = x[i * pad: i * pad + rows].cpu().double() @ full.t()
        # one rounding of the result; FP32 sums of k products of the size of the weights
        assert ((first[i].cpu().double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20 * k * full.abs().max()).all()


_WALK = r"""
#include <atomic>
#include <barrier>
#include <cstdio>
#include <thread>
#include <vector>
#include "pass_walk.h"
constexpr int WARPS = 8;
int main() {
  int bad = 0;
  for (int chunks : {1, 2, 5, 9})
    for (int per_slab : {1, 2, 8})
      for (int warp = -1; warp < WARPS; ++warp)            // -1: nobody gives up
        for (int at = 0; at < (warp < 0 ? 1 : chunks); ++at) {
          std::barrier sync(WARPS);
          std::atomic<int> failed{0}, held{0}, done{0};
          std::vector<std::thread> ts;
          for (int w = 0; w < WARPS; ++w)
            ts.emplace_back([&, w] {
              auto meet = [&] { sync.arrive_and_wait(); };
              auto any = [&](bool f) { failed += f; meet(); return failed.load() > 0; };
              held += ff::walk_pass(chunks, per_slab, meet, [](int) {}, [&](int c) { return w != warp || c != at; }, [&](int) { ++done; }, any);
            });
          for (auto& t : ts) t.join();
          const int want = warp < 0 ? WARPS * chunks : (WARPS - 1) * chunks + at;      // a warp that gave up multiplies nothing more
          bad += held != (warp < 0 ? WARPS : 0) || done != want;
        }
  std::printf("%d", bad);
  return bad != 0;
}
"""


def test_warps_of_a_packed_pass_leave_together(tmp_path):
    """The kernel's own walk on eight host threads: whichever warp's wait gives up at whichever stage, all eight come out of the pass (a
    barrier that one of them no longer meets would hold the rest for good) and all say that it does not hold."""
    from flyingfish_b200.ops import build
    src, exe = tmp_path / "walk.cpp", tmp_path / "walk"
    src.write_text(_WALK)
    subprocess.run(["g++", "-std=c++20", "-O1", "-pthread", "-I", str(build.CSRC), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=60, capture_output=True, text=True, check=True).stdout == "0"


@pytest.mark.gpu
@pytest.mark.parametrize("ctx", [1, 64, 65, 4000])
def test_merge_of_many_splits(ctx):
    """A single sequence is cut into as many splits as it has pages: partials of all, one and most splits without keys."""
    from flyingfish_b200 import ops
    hq, hkv, d, blocks = 8, 2, 128, 64
    q, k, v = _rand((1, hq * d), 1), _rand((blocks, hkv, 64, d), 2), _rand((blocks, hkv, 64, d), 3)
    table = torch.randperm(blocks, generator=torch.Generator().manual_seed(4)).to(torch.int32)[None]
    one = torch.ones(1, dtype=torch.int32)
    want = ref.attention_paged(q, k, v, table, 0 * one, one, ctx * one, hq, hkv, d, d ** -0.5).float()
    got = ops.attn_decode(q.cuda(), k.cuda(), v.cuda(), table.cuda(), (ctx * one).cuda(), hq, hkv, d, d ** -0.5, max_ctx=blocks * 64)
    torch.cuda.synchronize()
    ops.check_status()
    assert ((got.cpu().float() - want).abs() <= 1e-2 + 1e-2 * want.abs()).all()  # BF16 weights and result


@pytest.mark.gpu
@pytest.mark.parametrize("m", [129, 300, 1000])
@pytest.mark.parametrize("hq,hkv,k,rot", [(8, 2, 1024, 128), (32, 8, 256, 128), (5, 1, 520, 64)])      # tiles of pairs and of single CTAs, a part turned
def test_rotation_in_the_product_of_prompts(m, hq, hkv, k, rot, monkeypatch):
    """The bits of the product followed by the rotation kernel, in the rows and in the cache; padding rows are not cached."""
    from flyingfish_b200 import ops
    monkeypatch.setattr(ops, "rope_in_product", lambda *a: True)           # also at sizes where the kernels apart are quicker
    n, blocks = (hq + 2 * hkv) * 128, 20
    x, w = _rand((m, k), 1).cuda(), (_rand((n, k), 2) * 0.1).cuda()
    g = torch.Generator().manual_seed(m)
    pos = torch.randint(0, 9000, (m,), generator=g).to(torch.int32).cuda()
    slots = torch.randperm(blocks * 64, generator=g)[:m].to(torch.int32)
    slots[::7] = -1
    slots = slots.cuda()
    cache = lambda: [torch.full((blocks, hkv, 64, 128), 3.0, dtype=BF16, device="cuda") for _ in range(2)]
    (k0, v0), (k1, v1) = cache(), cache()
    want = ops.linear(x, w)
    ops.rope_kv_paged(want, pos, slots, k0, v0, hq, hkv, 128, 5e5, rot)
    got = ops.linear_rope_kv(x, w, pos, slots, k1, v1, hq, hkv, 128, 5e5, rot)
    torch.cuda.synchronize()
    ops.check_status()
    assert torch.equal(got, want) and torch.equal(k0, k1) and torch.equal(v0, v1)


@pytest.mark.gpu
@pytest.mark.parametrize("rot", [2, 66, 94, 96])                 # an odd number of angles, which lie on 8 bytes; ends inside a group of columns
def test_part_rotation_in_the_product_of_prompts(rot, monkeypatch):
    test_rotation_in_the_product_of_prompts(300, 6, 3, 512, rot, monkeypatch)


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 1, 2, 3])                 # floats in front of the table: 16, 4 and 8 byte boundaries
def test_rotation_in_the_product_takes_any_table(offset, monkeypatch):
    from flyingfish_b200 import ops
    monkeypatch.setattr(ops, "rope_in_product", lambda *a: True)
    m, hq, hkv, k, blocks = 140, 4, 2, 256, 3
    x, w = _rand((m, k), 1).cuda(), (_rand(((hq + 2 * hkv) * 128, k), 2) * 0.1).cuda()
    pos = torch.arange(m, dtype=torch.int32).cuda()
    table = ops.rope_table(pos, 128, 5e5)
    moved = torch.cat([torch.zeros(offset, device="cuda"), table.view(-1)])[offset:].view(table.shape)
    assert moved.data_ptr() % 16 == 4 * offset
    out = []
    for t in (None, moved):
        kc, vc = (torch.zeros(blocks, hkv, 64, 128, dtype=BF16, device="cuda") for _ in range(2))
        out.append((ops.linear_rope_kv(x, w, pos, pos, kc, vc, hq, hkv, 128, 5e5, cos_sin=t), kc, vc))
    torch.cuda.synchronize()
    ops.check_status()
    assert all(torch.equal(a, b) for a, b in zip(*out))


def test_rotation_joins_the_products_that_hide_it():
    from flyingfish_b200 import ops
    shapes = [((hq + 2 * hkv) * 128, k) for hq, hkv, k in ((32, 8, 4096), (8, 2, 1024), (64, 8, 8192), (16, 16, 2048))]
    assert all(ops.rope_in_product(m, n, k) for n, k in shapes for m in (1, 128, 4096, 8191))
    assert not any(ops.rope_in_product(m, n, k) for n, k in shapes for m in (129, 512))


@pytest.mark.gpu
@pytest.mark.parametrize("lens,hq,hkv", [
    ([0, 1, 64, 65, 320, 321, 384, 640], 8, 2),              # padding, whole pages, one page more; one split and several in a launch
    ([2000, 63, 700], 16, 1),                                # more than eight splits beside one
    ([300] * 100 + [900, 0], 32, 8),                         # so many rows that short sequences are not split
])
@pytest.mark.parametrize("nq", [1, 3])
@pytest.mark.parametrize("sinks", [False, True])
def test_splits_by_length(lens, hq, hkv, nq, sinks):
    """A sequence is cut by its own length: results against the oracle, and the bits of a row beside sequences of other lengths."""
    from flyingfish_b200 import ops
    d, blocks, batch = 128, 64, len(lens)
    lens = [max(n, nq) if n else 0 for n in lens]
    pool = 40
    q, k, v = _rand((batch * nq, hq * d), 1), _rand((pool, hkv, 64, d), 2), _rand((pool, hkv, 64, d), 3)
    table = torch.stack([torch.randint(0, pool, (blocks,), generator=torch.Generator().manual_seed(b)) for b in range(batch)]).to(torch.int32)
    ctx = torch.tensor(lens, dtype=torch.int32)
    sk = torch.randn(hq, generator=torch.Generator().manual_seed(9)) if sinks else None
    run = lambda c: ops.attn_decode(q.cuda(), k.cuda(), v.cuda(), table.cuda(), c.cuda(), hq, hkv, d, d ** -0.5, nq=nq, max_ctx=blocks * 64, sinks=sk.cuda() if sinks else None)
    got = run(ctx)
    torch.cuda.synchronize()
    ops.check_status()
    live = [b for b in range(batch) if lens[b]]
    for b in live[:12] + live[-2:]:
        one = torch.ones(1, dtype=torch.int32)
        want = ref.attention_paged(q[b * nq: (b + 1) * nq], k, v, table[b: b + 1], 0 * one, nq * one, ctx[b: b + 1], hq, hkv, d, d ** -0.5, None, 0, sk).float()
        assert ((got[b * nq: (b + 1) * nq].cpu().float() - want).abs() <= 1e-2 + 1e-2 * want.abs()).all()      # BF16 weights and result
    other = torch.where(ctx > 0, (ctx * 3) // 4 + nq, ctx)
    for first in (True, False):                              # the first sequence beside others, the others beside another first one
        mixed = torch.cat([ctx[:1], other[1:]]) if first else torch.cat([other[:1], ctx[1:]])
        again = run(mixed)
        for b in range(batch):
            if int(mixed[b]) == lens[b]:
                assert torch.equal(again[b * nq: (b + 1) * nq], got[b * nq: (b + 1) * nq])


@pytest.mark.gpu
@pytest.mark.parametrize("lens,hq,hkv", [
    ([0, 1, 64, 65, 320, 1000, 4096], 8, 2),                 # more splits than most of them have pages: some leave, some are alone
    ([1500, 150, 2850], 32, 8),
    ([300, 64, 700] * 40, 32, 8),                            # two splits, one of them without pages
])
@pytest.mark.parametrize("nq", [1, 2])
def test_splits_share_the_pages_evenly(lens, hq, hkv, nq):
    """A window that reaches past every context hides nothing, and its launch writes and merges all splits: the same bits. They fix how a
    sequence is cut, which fixes how its probabilities are rounded."""
    from flyingfish_b200 import ops
    d, blocks, pool = 128, 64, 40
    lens = [max(n, nq) if n else 0 for n in lens]
    q, k, v = _rand((len(lens) * nq, hq * d), 1), _rand((pool, hkv, 64, d), 2), _rand((pool, hkv, 64, d), 3)
    table = torch.stack([torch.randint(0, pool, (blocks,), generator=torch.Generator().manual_seed(b)) for b in range(len(lens))]).to(torch.int32).cuda()
    run = lambda window: ops.attn_decode(q.cuda(), k.cuda(), v.cuda(), table, torch.tensor(lens, dtype=torch.int32, device="cuda"), hq, hkv, d, d ** -0.5,
                                         nq=nq, max_ctx=blocks * 64, window=window)
    full, wide = run(0), run(1 << 20)
    torch.cuda.synchronize()
    ops.check_status()
    assert torch.equal(full, wide)


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [[5, 64, 66, 300, 1000], [70] * 40])         # one split with keys, several, two of which one has pages
@pytest.mark.parametrize("nq", [3, 8])
def test_splits_of_draft_trees(lens, nq):
    """Rows of a draft tree see the context and their ancestors, wherever the last pages fall among the splits."""
    from flyingfish_b200 import ops
    hq, hkv, d, blocks, pool = 8, 2, 128, 32, 30
    lens = [max(n, nq) for n in lens]
    b, g = len(lens), torch.Generator().manual_seed(nq)
    masks = torch.zeros(b, nq, dtype=torch.int64)
    for i in range(nq):                                      # a parent among the rows before, and the row itself
        masks[:, i] = 1 << i
        if i:
            masks[:, i] |= masks.gather(1, torch.randint(0, i, (b, 1), generator=g))[:, 0]
    q, k, v = _rand((b * nq, hq * d), 1), _rand((pool, hkv, 64, d), 2), _rand((pool, hkv, 64, d), 3)
    table = torch.randint(0, pool, (b, blocks), generator=g).to(torch.int32)
    ctx = torch.tensor(lens, dtype=torch.int32)
    got = ops.attn_decode(q.cuda(), k.cuda(), v.cuda(), table.cuda(), ctx.cuda(), hq, hkv, d, d ** -0.5, nq=nq, tree_mask=masks.view(-1).cuda(), max_ctx=blocks * 64)
    ops.check_status()
    want = ops.attn_decode(q, k, v, table, ctx, hq, hkv, d, d ** -0.5, nq=nq, tree_mask=masks.view(-1), max_ctx=blocks * 64).float()
    assert ((got.cpu().float() - want).abs() <= 1e-2 + 1e-2 * want.abs()).all()      # BF16 weights and result


@pytest.mark.parametrize("n,k", [(7168, 18432), (7168, 2560), (4096, 7168), (6144, 4096), (34048, 512), (33920, 512), (576, 2560), (128, 128)])
def test_fp8_split_does_not_depend_on_the_rows(n, k):
    import ctypes
    from flyingfish_b200.ops.lib import kernels
    assert len({kernels().ff_gemm_fp8_plan(m, n, k, *(ctypes.byref(ctypes.c_longlong()) for _ in range(2))) for m in range(1, 129)}) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("n,k", [(7168, 2560), (4096, 7168), (34048, 512), (33920, 512)])      # splits, none with one and two CTAs per SM
def test_fp8_rows_keep_their_bits_in_any_decode_batch(n, k):
    from flyingfish_b200 import ops
    from flyingfish_b200.ops import quant_ops
    x = _rand((128, k), 1).cuda()
    codes, scale = (t.cuda() for t in qref.quantize_fp8_block_weight(_rand((n, k), 2).float()))
    y = quant_ops.linear_fp8(x, codes, scale)
    for m in (1, 5, 32, 33, 64, 65):
        assert torch.equal(quant_ops.linear_fp8(x[:m].contiguous(), codes, scale), y[:m]), m
    ops.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("m", [32, 33, 64, 65])                                 # two CTAs per SM between 33 and 64 rows
@pytest.mark.parametrize("n,k", [(7168, 2560), (35072, 128), (576, 2560)])      # two splits, none, too few tiles for it
def test_dense_fp8_pairs(m, n, k):
    from flyingfish_b200 import ops
    from flyingfish_b200.ops import quant_ops
    x, w = _rand((m, k), m), _rand((n, k), 5)
    codes, scale = qref.quantize_fp8_block_weight(w.float())
    y = quant_ops.linear_fp8(x.cuda(), codes.cuda(), scale.cuda()).cpu().float()
    torch.cuda.synchronize()
    ops.check_status()
    want = qref.fp8_block_linear(x, codes, scale).float()
    # exact block products, FP32 sums of k / 128 of them; device and host quantise activations alike up to a last bit of the scale
    assert ((y - want).abs() <= 2.0 ** -7 * want.abs() + 2e-3 * k ** 0.5).all()


@pytest.mark.parametrize("m", [1, 16, 17, 32, 33, 48, 64, 65, 128])
def test_fp8_scales_leave_a_stage(m):
    """The longest K whose scales are taken still leaves the ring a stage; beyond it a product is refused. (Refusals come in front of the tensor
    maps, which need a driver: where there is none, anything but "too large" was accepted.)"""
    from flyingfish_b200.ops.lib import kernels, ptr
    too_large, cap = -5, (m + 15) // 16 * 16
    buf, ints = torch.zeros(64, dtype=torch.uint8), torch.zeros(4, dtype=torch.int32)

    def call(k):
        return kernels().ff_gemm_fp8(ptr(buf), ptr(buf), ptr(buf), ptr(buf), ptr(buf), None, None, 1, m, 128, k, 128, 0, 1, None, None, ptr(ints), None)
    longest = 64 * 1024 // (4 * cap) * 128
    assert call(longest + 128) == too_large
    if not torch.cuda.is_available():
        assert call(longest) != too_large
