"""The float32 kernel: tile edges, every way it shares out the keys, masks and layouts."""
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


def _rand(shape, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed))


@pytest.mark.parametrize("b,hq,hkv,sq,skv,d", [
    (1, 1, 1, 1, 1, 4), (1, 2, 1, 15, 17, 64), (1, 4, 4, 16, 128, 64), (2, 2, 2, 33, 129, 80),   # four key ranges a tile
    (2, 12, 4, 190, 191, 64), (1, 16, 16, 300, 257, 128), (2, 25, 25, 65, 70, 100),              # two
    (8, 20, 20, 64, 65, 64), (4, 40, 8, 130, 63, 128), (3, 50, 50, 65, 200, 36),                 # one
])
@pytest.mark.parametrize("mask", ["none", "causal", "bool", "add", "add-full"])
@pytest.mark.parametrize("layout", ["bhsd", "bshd"])
def test_against_the_oracle(b2a, b, hq, hkv, sq, skv, d, mask, layout):
    q, k, v = _rand((b, hq, sq, d), 1), _rand((b, hkv, skv, d), 2), _rand((b, hkv, skv, d), 3)
    m = None
    if mask not in ("none", "causal"):
        keep = torch.rand((b, 1, sq if mask == "add-full" else 1, skv), generator=torch.Generator().manual_seed(4)) > 0.4
        keep[..., 0] = True
        m = keep if mask == "bool" else torch.where(keep, 0.25, torch.finfo(torch.float32).min)
    dev = [t.transpose(1, 2).contiguous().cuda().transpose(1, 2) if layout == "bshd" else t.cuda() for t in (q, k, v)]
    out = torch.full((b, sq, hq, d), 7.0, device="cuda").transpose(1, 2) if layout == "bshd" else \
        torch.full((b, hq, sq, d), 7.0, device="cuda")
    b2a.sdpa(*dev, None if m is None else m.cuda(), causal=mask == "causal", out=out)
    assert_close(out, osdpa.sdpa_ref(q, k, v, mask=m, causal=mask == "causal"), torch.float32)


@pytest.mark.parametrize("b", [1, 40])
def test_fully_masked_rows(b2a, b):
    # every key removed: zeros; every key at the type's lowest value: nothing of the scores is left, the plain average
    q, k, v = _rand((b, 4, 70, 64), 1), _rand((b, 4, 201, 64), 2), _rand((b, 4, 201, 64), 3)
    for value in (float("-inf"), torch.finfo(torch.float32).min):
        out = b2a.sdpa(q.cuda(), k.cuda(), v.cuda(), torch.full((1, 1, 1, 201), value, device="cuda"))
        want = torch.zeros(b, 4, 70, 64) if value == float("-inf") else v.mean(2, keepdim=True).expand(b, 4, 70, 64)
        assert_close(out, want.numpy(), torch.float32)
