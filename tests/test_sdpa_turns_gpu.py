"""The two tiles of an item take turns on one place for their scores: tiles of unequal length, items of one key step, several
items on a CTA."""
import numpy as np
import pytest
import torch

from oracle import sdpa as osdpa

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("b,hq,hkv,s,causal", [
    (4, 200, 200, 100, True),    # an item of one tile and one key step; two items on some CTAs
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
    # the rounding bound of test_key_split_gpu.py: probabilities and results in the tensors' type, float32 sums
    u = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    for at in (0, b - 1):
        pick = [t[at:at + 1].cpu() for t in (q, k, v)]
        ref = osdpa.sdpa_ref(*pick, causal=causal)
        spread = osdpa.sdpa_ref(pick[0], pick[1], pick[2].abs(), causal=causal)
        err = np.abs(out[at:at + 1].float().cpu().numpy() - ref)
        assert (err <= u * (spread + np.abs(ref)) + 1e-4).all(), float((err - u * (spread + np.abs(ref))).max())
