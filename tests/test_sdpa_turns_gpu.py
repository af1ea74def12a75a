"""The two tiles of an item take turns on one place for their scores: tiles of unequal length, items of one key step, several
items on a CTA."""
import numpy as np
import pytest
import torch

from oracle import sdpa as osdpa

pytestmark = pytest.mark.gpu


def check(out, q, k, v, causal, entries):
    # the rounding bound of test_key_split_gpu.py: probabilities and results in the tensors' type, float32 sums
    u = 2.0 ** -11 if out.dtype == torch.float16 else 2.0 ** -8
    for at in entries:
        pick = [t[at:at + 1].cpu() for t in (q, k, v)]
        ref = osdpa.sdpa_ref(*pick, causal=causal)
        spread = osdpa.sdpa_ref(pick[0], pick[1], pick[2].abs(), causal=causal)
        err = np.abs(out[at:at + 1].float().cpu().numpy() - ref)
        assert (err <= u * (spread + np.abs(ref)) + 1e-4).all(), (at, float((err - u * (spread + np.abs(ref))).max()))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("b,hq,hkv,s,causal", [
    (4, 200, 200, 100, True),    # items of one tile and one key step, five or six a CTA: a place per tile
    (20, 15, 5, 300, True),      # groups of three heads: tiles A and B of different rows, so of unequal length
    (10, 32, 16, 257, True),     # a last key tile of one key; three row blocks
    (5, 64, 8, 384, False),      # equal tiles, three key steps, more items than SMs
])
def test_against_the_oracle(dtype, b, hq, hkv, s, causal):
    import openvino_contrib_b200 as b2a
    g = torch.Generator(device="cuda").manual_seed(s)
    q, k, v = (torch.randn(b, h, s, 128, generator=g, device="cuda").to(dtype) for h in (hq, hkv, hkv))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = b2a.sdpa(q, k, v, causal=causal, status=status)
    assert int(status.item()) == 0
    check(out, q, k, v, causal, sorted({0, 1, b // 2, b - 1}))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("b,hq,hkv,sq,skv,causal", [
    (1, 8, 8, 17, 1, False),       # the smallest: one key
    (3, 32, 8, 127, 127, True),
    (3, 32, 8, 128, 128, True),    # the largest key count of one step
    (3, 32, 8, 129, 129, True),    # two steps: tiles in turn on one place
    (2, 33, 11, 200, 128, False),  # two row blocks and an odd number of tiles
    (9, 40, 40, 300, 100, False),  # several items a CTA, items of one tile among them
    (2, 32, 8, 128, 300, True),    # (a causal row sees at most Sq keys: one step)
])
def test_one_key_step(dtype, b, hq, hkv, sq, skv, causal):
    import openvino_contrib_b200 as b2a
    g = torch.Generator(device="cuda").manual_seed(sq + skv)
    q, k, v = (torch.randn(b, h, s, 128, generator=g, device="cuda").to(dtype) for h, s in ((hq, sq), (hkv, skv), (hkv, skv)))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = b2a.sdpa(q, k, v, causal=causal, status=status)
    assert int(status.item()) == 0
    check(out, q, k, v, causal, range(b))
    if causal and sq == skv and sq >= 128:
        # rows 0..126 see the same keys in the same step whichever kernel takes the call
        shorter = b2a.sdpa(*(t[:, :, :127].contiguous() for t in (q, k, v)), causal=True)
        assert torch.equal(shorter, out[:, :, :127])


@pytest.mark.parametrize("s", [100, 128])
def test_one_key_step_of_a_head_shard(s):
    # the sharded epilogue (slabs and tensor stores) in the form for one key step, several items a CTA
    import openvino_contrib_b200 as b2a
    from openvino_contrib_b200.sharding import HeadShard, ShardGroup
    b, hq, hkv = 4, 120, 40
    g = torch.Generator(device="cuda").manual_seed(s)
    q, k, v = (torch.randn(b, h, s, 128, generator=g, device="cuda").half() for h in (hq, hkv, hkv))
    group = ShardGroup(HeadShard(0, 1, hq, hkv), staging_bytes=2 * q.numel() * 2)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    for causal in (True, False):
        full = group.sdpa(q, k, v, causal=causal, status=status).clone()
        assert int(status.item()) == 0
        assert torch.equal(full, b2a.sdpa(q, k, v, causal=causal))
    group.close()
