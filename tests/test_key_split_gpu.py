"""Small problems on the tensor cores: a tile's keys shared out over the two softmax groups, merged in the epilogue."""
import numpy as np
import pytest
import torch

from oracle import sdpa as osdpa
from tests.helpers import assert_close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def b2a():
    import openvino_contrib_b200 as m
    assert torch.cuda.is_available()
    return m


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("b,hq,hkv,sq,skv,d", [
    (1, 2, 1, 100, 128, 128), (1, 4, 2, 130, 129, 128), (1, 3, 1, 257, 300, 128),   # one to three key tiles: halves of 1+0, 1+1, 2+1
    (1, 32, 8, 777, 777, 128), (1, 8, 8, 64, 1500, 128),                            # more tiles than SMs; long keys, few rows
    (1, 4, 4, 200, 129, 64), (2, 6, 2, 300, 700, 64),
    (1, 40, 40, 512, 512, 128), (1, 37, 37, 512, 512, 128),                         # either side of the rule (pairs against SMs)
])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("layout", ["bhsd", "bshd"])
def test_against_the_oracle(b2a, dtype, b, hq, hkv, sq, skv, d, causal, layout):
    q, k, v = (torch.randn(b, h, s, d, generator=torch.Generator().manual_seed(i)).to(dtype)
               for i, (h, s) in enumerate(((hq, sq), (hkv, skv), (hkv, skv))))
    dev = [t.transpose(1, 2).contiguous().cuda().transpose(1, 2) if layout == "bshd" else t.cuda() for t in (q, k, v)]
    out = torch.full((b, sq, hq, d), 7.0, dtype=dtype, device="cuda").transpose(1, 2) if layout == "bshd" else \
        torch.full((b, hq, sq, d), 7.0, dtype=dtype, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    b2a.sdpa(*dev, causal=causal, out=out, status=status)
    assert int(status.item()) == 0
    # Rounding bounds of the arithmetic: each probability enters the second product rounded to the tensors' type (relative
    # error up to u = 2^-11 in f16, 2^-8 in bf16, so up to u * sum p |v| of the result) and the result is rounded once more
    # (u * |result|); 1e-4 for float32 sums and exponentials of values up to about five.
    u = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    ref, spread = osdpa.sdpa_ref(q, k, v, causal=causal), osdpa.sdpa_ref(q, k, v.abs(), causal=causal)
    err = np.abs(out.float().cpu().numpy() - ref)
    assert (err <= u * (spread + np.abs(ref)) + 1e-4).all(), float((err - u * (spread + np.abs(ref))).max())


@pytest.mark.parametrize("kind", ["bool", "add"])
def test_a_half_without_keys(b2a, kind):
    # a padding mask that leaves one half of the keys, or nothing at all, to a row's sequence
    q, k, v = (torch.randn(3, 2, 200, 64, generator=torch.Generator().manual_seed(i)).half() for i in range(3))
    keep = torch.zeros(3, 1, 1, 200, dtype=torch.bool)
    keep[0, ..., :90] = True   # keys of the first tile only
    keep[1, ..., 150:] = True  # of the second only
    m = keep if kind == "bool" else torch.where(keep, 0.0, float("-inf")).half()
    out = b2a.sdpa(q.cuda(), k.cuda(), v.cuda(), m.cuda())
    assert float(out[2].abs().max()) == 0.0
    assert_close(out[0], osdpa.sdpa_ref(q[:1], k[:1, :, :90], v[:1, :, :90])[0], torch.float16)
    assert_close(out[1], osdpa.sdpa_ref(q[1:2], k[1:2, :, 150:], v[1:2, :, 150:])[0], torch.float16)
