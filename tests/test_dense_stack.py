"""The layers of a dense decoder launched by one native call against the operators called one by one."""
import re
from pathlib import Path

import pytest
import torch

CSRC = Path(__file__).resolve().parent.parent / "flyingfish_b200" / "ops" / "csrc"


def test_launchers_have_one_declaration():
    """C linkage: a prototype copied by hand would go on linking against a definition whose parameters have changed. The header that declares
    them is included where they are defined and where they are called."""
    declared = set(re.findall(r"FF_EXPORT int (ff_\w+)\(", (CSRC / "launchers.h").read_text()))
    assert declared
    for src in CSRC.glob("*.cu"):
        text = src.read_text()
        assert not re.findall(r"\bint ff_\w+\([^;{}]*\)\s*;", text), src.name
        defined = set(re.findall(r"FF_EXPORT int (ff_\w+)\(", text))
        called = set(re.findall(r"\b(ff_\w+)\(", text)) - defined
        if defined & declared or src.stem == "dense_stack":
            assert '#include "launchers.h"' in text, src.name
        if src.stem == "dense_stack":
            assert called <= declared


@pytest.mark.gpu
@pytest.mark.parametrize("lens,pasts", [([1], [0]), ([37], [0]), ([5, 64, 59], [0, 70, 3]), ([129], [0]), ([300, 1, 211], [10, 0, 64])])
def test_native_layers_give_the_bits_of_the_operators(lens, pasts, monkeypatch):
    """One and several sequences, portions behind a context; more rows than the decode product takes are left to the operators."""
    import copy
    from flyingfish_b200 import ops
    from flyingfish_b200.config import Settings, named_shape
    from flyingfish_b200.engine.engine import Engine
    from flyingfish_b200.models import decoder
    from flyingfish_b200.models.weights import build_decoder_weights
    spec = copy.deepcopy(named_shape("llama3-8b-shape"))
    spec.layers, spec.vocab, spec.hidden, spec.heads, spec.kv_heads, spec.ffn = 3, 512, 1024, 8, 2, 2048
    gen = torch.Generator(device="cuda").manual_seed(1)
    source = lambda name, shape: (torch.randn(shape, device="cuda", generator=gen) * (0.02 if "norm" not in name else 0.1) + (1.0 if "norm" in name else 0.0)).bfloat16()
    net = decoder.DecoderModel(build_decoder_weights(spec, source, torch.device("cuda")))
    ids = [torch.randint(0, 512, (n + p,), generator=torch.Generator().manual_seed(n)).tolist() for n, p in zip(lens, pasts)]

    def run(native):
        eng = Engine(net, spec, Settings(capacity=1024, max_batch=8), 64, "cuda", max_prefill_rows=1024)
        monkeypatch.setattr(decoder, "STACK_MAX_ROWS", 0)
        seqs = [eng.add_sequence(t) for t in ids]
        for s, p in zip(seqs, pasts):
            if p:
                eng.prefill_some([s], p)
        if native:
            monkeypatch.setattr(decoder, "STACK_MAX_ROWS", 1024)
        calls = []
        real = ops.dense_stack
        monkeypatch.setattr(ops, "dense_stack", lambda *a, **k: calls.append(real(*a, **k)) or calls[-1])
        eng.prefill(seqs)
        monkeypatch.setattr(ops, "dense_stack", real)
        assert bool(calls) == native and all(n == (spec.layers if sum(lens) <= ops.SKINNY_MAX_M else 0) for n in calls)
        ops.check_status()
        return net.last_logits.clone(), net.last_residual.clone(), [t.clone() for t in eng.kv.k + eng.kv.v]
    a, b = run(False), run(True)
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1]) and all(torch.equal(x, y) for x, y in zip(a[2], b[2]))
