"""Paths that only long tables reach: a warp's second window of block ids, a plan of more than 256 sequences, more than 32
splits of a sequence, chunks of the steps that fill the GPU."""
import numpy as np
import pytest
import torch

from oracle import paged as opaged
from oracle import sdpa as osdpa
from tests.helpers import PagedWorkload, assert_close

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def b2a():
    import openvino_contrib_b200 as m
    assert torch.cuda.is_available()
    return m


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_windows_of_block_ids_in_a_sixteen_bit_pool(b2a, dtype):
    # 128 sequences x 8 KV heads: one CTA each, so a warp walks a quarter of its sequence - 66 and 40 tiles of the two long ones,
    # through three and two windows of 32 block ids
    hq, hkv, d, bs, long = 16, 8, 64, 16, {3: 4200, 97: 2500}
    ctx = np.array([long.get(s, 1 + s % 37) for s in range(128)], np.int32)
    bi, bb, nb = opaged.build_block_tables(ctx, bs, seed=5, spare_blocks=3)
    gen = torch.Generator().manual_seed(3)
    k, v = (torch.randn(int(ctx.sum()), hkv, d, generator=gen).to(dtype) for _ in range(2))
    begins = np.zeros(129, np.int32)
    begins[1:] = np.cumsum(ctx)
    cache = b2a.PagedKvCache.allocate(nb, hkv, d, bs, dtype)
    t = [torch.from_numpy(a).cuda() for a in (np.zeros(128, np.int32), begins, bi, bb)]
    b2a.paged_kv_store(k.reshape(-1, hkv * d).cuda(), v.reshape(-1, hkv * d).cuda(), cache, *t)
    q = torch.randn(128, hq * d, generator=gen).to(dtype)
    t = [torch.from_numpy(a).cuda() for a in (ctx - 1, np.arange(129, dtype=np.int32), bi, bb)]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = b2a.paged_attention(q.cuda(), cache, *t, hq=hq, max_context_len=4200, max_q_len=1, status=status).float().cpu().numpy()
    assert int(status.item()) == 0
    for s in (0, 3, 36, 97, 127):
        rows = slice(int(begins[s]), int(begins[s + 1]))
        ref = osdpa.sdpa_ref(q[s].reshape(1, hq, 1, d), k[rows].transpose(0, 1)[None], v[rows].transpose(0, 1)[None])
        # the rounding of the result, and float32 sums of values up to about five
        np.testing.assert_allclose(out[s], ref.reshape(-1), atol=5e-5, rtol=2.0 ** -10 if dtype == torch.float16 else 2.0 ** -8)


@pytest.mark.parametrize("kv_hint", [True, False])
def test_a_mixed_step_of_more_than_256_sequences(b2a, kv_hint):
    many = {5: 40, 200: 130, 255: 17, 256: 33, 257: 2, 299: 150}
    q_len = [many.get(s, 1) for s in range(300)]
    ctx = [n + (7 * s) % 50 for s, n in enumerate(q_len)]
    w = PagedWorkload(ctx, q_len, 8, 2, 128, seed=6)
    q = torch.from_numpy(w.query).to(torch.float16)
    tokens = sum((ctx[s] + 127) // 128 * 128 for s in many)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = b2a.paged_attention(q.cuda(), w.device_cache(), *w.device_tables(), hq=8, max_context_len=256, max_q_len=150,
                              prefill_kv_tokens=tokens if kv_hint else 0, status=status)
    assert int(status.item()) == 0
    assert_close(out, w.reference(q.float().numpy()), torch.float16)


@pytest.mark.parametrize("scores", [False, True])
def test_more_than_32_splits(b2a, scores):
    # fourteen sequences of up to 68000 tokens: chunks of 128 blocks, 34 of them; with scores 64 blocks and twice as many
    ctx = [68000, 1000] + [30 * s + 1 for s in range(12)]
    w = PagedWorkload(ctx, [1] * 14, 8, 2, 128, seed=8)
    q = torch.from_numpy(w.query).to(torch.float16)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    args = dict(hq=8, max_context_len=68000, status=status)
    if scores:
        out, got, begins = b2a.paged_attention_scores(q.cuda(), w.device_cache(), *w.device_tables(), **args)
        ref, ref_begins = opaged.last_token_scores_ref(q.float().numpy(), w.k_cache, w.past, w.sb, w.bi, w.bb, 8, 2, 128, 16)
        assert np.array_equal(begins.cpu().numpy(), ref_begins)
        np.testing.assert_allclose(got.cpu().numpy()[: ref_begins[-1]], ref, atol=2e-5 * 8, rtol=2e-3)
    else:
        out = b2a.paged_attention(q.cuda(), w.device_cache(), *w.device_tables(), max_q_len=1, **args)
    assert int(status.item()) == 0
    assert_close(out, w.reference(q.float().numpy()), torch.float16)
