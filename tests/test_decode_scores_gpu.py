"""Attention and score output of a step of one-token sequences from one walk over the cache."""
import numpy as np
import pytest
import torch

from oracle import paged as opaged
from tests.helpers import PagedWorkload

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def b2a():
    import openvino_contrib_b200 as m
    assert torch.cuda.is_available()
    return m


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("ctx,hq,hkv,window", [
    ([1, 16, 17, 300], 32, 8, 0),             # one key; exactly one block; one key into the second block
    ([511, 512, 513, 2048, 4099], 64, 8, 0),  # edges of a score CTA's positions, several chunks, eight heads a group
    ([7, 300], 8, 8, 0),                      # no grouping
    ([40, 9000], 12, 4, 0),                   # three heads a group
    ([20 + 3 * i for i in range(150)], 4, 1, 0),  # more sequences than a CTA has threads
    ([9, 250, 1500], 32, 8, 1), ([9, 250, 1500], 32, 8, 100), ([9, 250, 1500], 16, 8, 4096),
])
def test_both_outputs(b2a, dtype, ctx, hq, hkv, window):
    # the attention rows are the bits of paged_attention wherever both calls cut the sequences alike: in steps that leave the plan
    # below 96 blocks a chunk, as these do (beyond, the scores halve the chunks: test_more_than_32_splits compares with the
    # oracle).  The scores agree with the oracle like those of the call of their own
    w = PagedWorkload(ctx, [1] * len(ctx), hq, hkv, 128, seed=3 * hq + len(ctx))
    q = torch.from_numpy(w.query).to(dtype)
    cache, tables, status = w.device_cache(), w.device_tables(), torch.zeros(1, dtype=torch.int32, device="cuda")
    done = b2a.paged_attention_scores(q.cuda(), cache, *tables, hq=hq, max_context_len=int(w.ctx.max()), sliding_window=window,
                                      status=status)
    assert done is not None and int(status.item()) == 0
    out, scores, begins = done
    alone = b2a.paged_attention(q.cuda(), cache, *tables, hq=hq, max_context_len=int(w.ctx.max()), max_q_len=1, sliding_window=window)
    assert torch.equal(out, alone)
    ref, ref_begins = opaged.last_token_scores_ref(q.float().numpy(), w.k_cache, w.past, w.sb, w.bi, w.bb, w.hq, w.hkv, w.d,
                                                   w.bs, None, window)
    assert np.array_equal(begins.cpu().numpy(), ref_begins)
    # probabilities: f32 accumulation of exact f16 products, ex2.approx (2 ulp) - the floating-point bar of f32 outputs
    np.testing.assert_allclose(scores.cpu().numpy()[: ref_begins[-1]], ref, atol=2e-5 * w.hq, rtol=2e-3)


def test_inconsistent_tables_and_a_small_buffer(b2a):
    # a sequence with a negative length and one beyond the admitted context have no entries and are reported; nothing
    # is written beyond the caller's buffer
    w = PagedWorkload([100, 200, 60, 500], [1] * 4, 16, 2, 128, seed=9)
    q = torch.from_numpy(w.query).to(torch.float16).cuda()
    past = w.past.copy()
    past[0] = -3
    tables = list(w.device_tables())
    tables[0] = torch.from_numpy(past).cuda()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    scores = torch.full((230,), -7.0, device="cuda")
    call = lambda t, s: b2a.paged_attention_scores(q, w.device_cache(), *t, hq=16, max_context_len=256, scores=s, status=status)  # noqa: E731
    _, _, begins = call(tables, scores)
    assert begins.tolist() == [0, 0, 200, 260, 260] and int(status.item()) & 4  # B2A_DEV_BAD_LEN
    got = scores.cpu().numpy()
    assert abs(got[:200].sum() - 16) < 0.1 and (got[200:] == -7).all()


def test_steps_it_does_not_take(b2a):
    w = PagedWorkload([100, 200], [1, 2], 16, 2, 128, seed=9)
    q = torch.from_numpy(w.query).to(torch.float16).cuda()
    assert b2a.paged_attention_scores(q, w.device_cache(), *w.device_tables(), hq=16, max_context_len=256) is None
    w = PagedWorkload([100, 200], [1, 1], 32, 2, 128, seed=9)  # sixteen heads a group
    q = torch.from_numpy(w.query).to(torch.float16).cuda()
    assert b2a.paged_attention_scores(q, w.device_cache(), *w.device_tables(), hq=32, max_context_len=256) is None
