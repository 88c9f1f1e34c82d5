"""The host side of a step: packed metadata, reserved slots, results read back with the device status."""
import random

import pytest
import torch

from flyingfish_b200.engine.batch import BatchLayout, ForwardBatch
from flyingfish_b200.engine.kv_cache import OutOfBlocks, PagedKVCache


def _field(fb, off, n):
    return fb.host[off: off + n].tolist()


@pytest.mark.parametrize("batch", [1, 3, 8])
def test_fields_of_a_step(batch):
    L = BatchLayout(8, 24, 6, 2)
    fb = ForwardBatch(L, "cpu")
    rng = random.Random(batch)
    for step in range(3):                                        # block rows that stay, grow and are replaced
        q_lens = [rng.randint(1, 3) for _ in range(batch)]
        rows = sum(q_lens)
        ids, pos, slots = ([rng.randint(0, 1 << 20) for _ in range(rows)] for _ in range(3))
        blocks = [list(range(7 * i, 7 * i + rng.randint(0, 6))) for i in range(batch)]
        ctx = [rng.randint(1, 300) for _ in range(batch)]
        masks = [rng.getrandbits(64) for _ in range(rows)]
        fb.fill(ids=ids, positions=pos, slots=slots, q_lens=q_lens, ctx_lens=ctx, block_rows=blocks, logit_rows=range(rows), is_decode=False,
                tree_mask=masks, kv_start=[5] * (batch - 1), group_rows=[[1], [2, 3]][:batch], state_slots=list(range(batch)))
        starts = [sum(q_lens[:i]) for i in range(batch)]
        assert _field(fb, L.ids, rows) == ids and _field(fb, L.positions, rows) == pos and _field(fb, L.slots, rows) == slots
        assert _field(fb, L.q_start, batch) == starts and _field(fb, L.row_start, batch + 1) == starts + [rows]
        assert _field(fb, L.q_lens, batch) == q_lens and _field(fb, L.ctx_lens, batch) == ctx and _field(fb, L.logit_rows, rows) == list(range(rows))
        assert _field(fb, L.kv_start, batch) == [5] * (batch - 1) + [0] and _field(fb, L.state_slots, batch) == list(range(batch))
        for i, b in enumerate(blocks):
            assert _field(fb, L.block_table + i * L.max_blocks, len(b)) == b
            b.append(99)                                         # the caller's lists go on growing
        assert [m & (1 << 64) - 1 for m in fb.host[L.tree_mask: L.tree_mask + 2 * rows].view(torch.int64).tolist()] == masks
        assert (fb.max_q_len, fb.max_ctx) == (max(q_lens), max(ctx))


def test_a_step_reserves_for_all_or_none():
    kv = PagedKVCache(1, 1, 8, 6, 64)
    for i, n in enumerate((64, 10, 128)):
        kv.add_sequence(i)
        kv.reserve(i, n)
        kv.commit(i, n)
    before = [list(kv.seqs[i].blocks) for i in range(3)]
    free = kv.alloc.free_blocks
    assert free == 2
    taken = kv.alloc.alloc()
    with pytest.raises(OutOfBlocks):
        kv.reserve_step([0, 1, 2])
    assert [kv.seqs[i].blocks for i in range(3)] == before
    kv.alloc.release(taken)
    held, at, slots = kv.reserve_step([2, 1, 0])
    assert [h.seq_id for h in held] == [2, 1, 0] and at.tolist() == [128, 10, 64]
    assert slots.tolist() == [kv.seqs[2].blocks[2] * 64, kv.seqs[1].blocks[0] * 64 + 10, kv.seqs[0].blocks[1] * 64]
    assert kv.reserve_step([0])[2].tolist() == kv.reserve(0, 1)      # nothing is committed: the same slot again


@pytest.mark.gpu
def test_a_replayed_step_reports_the_device_status():
    from flyingfish_b200 import ops
    from flyingfish_b200.api import Model
    from flyingfish_b200.config import Settings
    m = Model.load("tiny-llama", Settings(capacity=256, max_batch=4), device="cuda:0", seed=0)
    eng = m.engine
    seqs = [eng.add_sequence([1, 2, 3, 4 + i]) for i in range(3)]
    eng.prefill(seqs)
    first = eng.decode(seqs)
    assert first == [s.output[-1] for s in seqs] and len(first) == 3
    seqs[1].pending = eng.spec.vocab + 7                          # refused by the embedding's own check
    with pytest.raises(ops.DeviceStatusError):
        eng.decode(seqs)
    assert ops.read_status("cuda:0")[0] == 0 and eng.poisoned
    eng.reset()
    seqs = [eng.add_sequence([1, 2, 3, 4 + i]) for i in range(3)]
    eng.prefill(seqs)
    assert eng.decode(seqs) == first


@pytest.mark.gpu
def test_a_captured_step_reads_the_device_buffer():
    """Steps staged in device memory and replayed, the ids fed back there, are those of ``Engine.decode``: ids, logits and cache."""
    from flyingfish_b200 import ops
    from flyingfish_b200.api import Model
    from flyingfish_b200.config import Settings
    from flyingfish_b200.engine.engine import bucket_for
    m = Model.load("tiny-llama", Settings(capacity=256, max_batch=4), device="cuda:0", seed=0)
    eng, steps, bucket = m.engine, 5, bucket_for(3)

    def start():
        eng.reset()
        for t in eng.kv.k + eng.kv.v:
            t.zero_()
        seqs = [eng.add_sequence([1, 2, 3, 4 + i][: 2 + i]) for i in range(3)]
        eng.prefill(seqs)
        return seqs
    seqs = start()
    g = eng.capture(bucket)
    want = [(eng.decode(seqs), g.logits[:3].clone()) for _ in range(steps)]
    cached = lambda: [t[eng.kv.seqs[s.seq_id].blocks] for t in eng.kv.k + eng.kv.v for s in seqs]
    cache = cached()
    seqs = start()
    fb, staged = g.batch, []
    for _ in range(steps):
        eng._fill_decode(fb, seqs, bucket)
        staged.append(fb.host.to("cuda"))
        for s in seqs:
            eng.kv.commit(s.seq_id, 1)
    ids, prev = fb.dev[fb.layout.ids: fb.layout.ids + bucket], torch.tensor([s.pending for s in seqs] + [0] * (bucket - 3), dtype=torch.int32, device="cuda")
    for meta, (toks, logits) in zip(staged, want):
        fb.dev.copy_(meta)
        ids.copy_(prev)
        g.graph.replay()
        prev = g.out
        assert g.out[:3].tolist() == toks and torch.equal(g.logits[:3], logits)
    ops.check_status()
    assert all(torch.equal(a, b) for a, b in zip(cache, cached()))
