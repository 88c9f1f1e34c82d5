"""Row-wise kernels between the products of a layer, against the operators they stand for."""
import pytest
import torch

from flyingfish_b200.ops import ref

BF16 = torch.bfloat16


def _packed(rows, heads, dim, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(rows, heads * dim, generator=g).to(BF16)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 7, 2368, 2371])          # one row per CTA, the first size with four, a ragged last CTA
@pytest.mark.parametrize("hq,hkv,dim,rot", [(4, 1, 128, 128), (64, 4, 128, 128), (3, 2, 128, 64), (5, 1, 64, 64), (2, 2, 48, 32)])
@pytest.mark.parametrize("norm", [False, True])
def test_rotation_norm_and_cache_write(rows, hq, hkv, dim, rot, norm):
    """Rotation and cache write are the oracle's bits; with head norms the sums of squares meet in another order, which moves a normed
    value by at most its last bit (2^-8 relative) before it is turned."""
    from flyingfish_b200 import ops
    qkv = _packed(rows, hq + 2 * hkv, dim, rows + dim)
    g = torch.Generator().manual_seed(1)
    nb = (rows + 63) // 64 + 1
    slots = torch.randperm(nb * 64, generator=g)[:rows].to(torch.int32)
    slots[rows // 2] = -1 if rows > 1 else slots[0]
    pos = torch.randint(0, 9000, (rows,), generator=g).to(torch.int32)
    w = [(1 + 0.1 * torch.randn(dim, generator=g)).to(BF16) for _ in range(2)]
    kw = dict(q_norm=w[0], k_norm=w[1], eps=1e-6) if norm else {}
    want = [qkv.clone(), torch.zeros(nb, hkv, 64, dim, dtype=BF16), torch.zeros(nb, hkv, 64, dim, dtype=BF16)]
    ops.rope_kv_paged(want[0], pos, slots, want[1], want[2], hq, hkv, dim, 1e6, rot, **kw)       # CPU oracle
    got = [qkv.cuda(), torch.zeros_like(want[1]).cuda(), torch.zeros_like(want[2]).cuda()]
    ops.rope_kv_paged(got[0], pos.cuda(), slots.cuda(), got[1], got[2], hq, hkv, dim, 1e6, rot, **{k: v.cuda() if k != "eps" else v for k, v in kw.items()})
    torch.cuda.synchronize()
    ops.check_status()
    for a, b in zip(got, want):
        a, b = a.cpu().float(), b.float()
        # sine and cosine may differ by a last bit of BF16 between the host's and the device's functions: an absolute 2^-7 of the
        # largest element of the pair, as the rotation's own test allows
        assert ((a - b).abs() <= 2e-2 + 2e-2 * b.abs()).all()
    assert torch.equal(got[2].cpu(), want[2])                                                   # values are copies
