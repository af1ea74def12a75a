"""A block that one sequence holds as cached context and another sequence's new tokens of the same step go into (prefixes shared
within a step): the step stores first, so the first sequence attends over the rows that the second one brings."""
import numpy as np
import pytest
import torch

from oracle import paged as opaged
from tests.helpers import assert_close

pytestmark = pytest.mark.gpu
HQ, HKV, D, BS = 8, 2, 128, 16


def shared_step(writer_tokens, pairs, reader_ctx, seed):
    """Tables of `pairs` writers (`writer_tokens` new tokens that end at a block's end) and as many one-token readers whose tables
    begin with the blocks of their writer; and the pool's block count."""
    rng = np.random.default_rng(seed)
    per_writer = (writer_tokens + BS - 1) // BS
    per_reader = (reader_ctx + BS - 1) // BS
    nb = pairs * per_reader + 3
    ids = rng.permutation(nb)[:pairs * per_reader].reshape(pairs, per_reader)
    past, new, tables = [], [], []
    for w in range(pairs):
        past.append(per_writer * BS - writer_tokens)
        new.append(writer_tokens)
        tables.append(ids[w, :per_writer])
    for w in range(pairs):
        past.append(reader_ctx - 1)
        new.append(1)
        tables.append(ids[w])
    cum = lambda x: np.concatenate([[0], np.cumsum(x)])  # noqa: E731
    t = [past, cum(new), np.concatenate(tables), cum([len(x) for x in tables])]
    return [np.asarray(x, np.int32) for x in t], nb


@pytest.mark.parametrize("kv", ["f16", "bf16", "u8"])
@pytest.mark.parametrize("writer_tokens,pairs", [(1, 3), (64, 2), (1, 40)])
@pytest.mark.parametrize("reader_ctx", [33, 600, 4000])
def test_new_rows_of_another_sequence_are_seen(kv, writer_tokens, pairs, reader_ctx):
    import openvino_contrib_b200 as b2a
    dt = torch.bfloat16 if kv == "bf16" else torch.float16
    if writer_tokens > reader_ctx:
        pytest.skip("the reader's context is shorter than what the writer brings")
    t, nb = shared_step(writer_tokens, pairs, reader_ctx, 7)
    tokens = int(t[1][-1])
    g = torch.Generator().manual_seed(reader_ctx + writer_tokens)
    q, k, v = (torch.randn(tokens, h * D, generator=g).to(dt) for h in (HQ, HKV, HKV))
    k *= 2  # (new rows draw the attention, so that a stale one shows)
    cache = b2a.PagedKvCache.allocate(nb, HKV, D, BS, torch.uint8 if kv == "u8" else dt)
    rows = [torch.randn(nb * BS, HKV * D, generator=g).to(dt) for _ in range(2)]
    every = [np.asarray(x, np.int32) for x in ([0], [0, nb * BS], np.arange(nb), [0, nb])]
    b2a.paged_kv_store(rows[0].cuda(), rows[1].cuda(), cache, *[torch.from_numpy(x).cuda() for x in every])
    pools = [c.cpu().numpy().copy() for c in (cache.k, cache.v)]
    if kv == "u8":
        for new, pool in ((k, pools[0]), (v, pools[1])):
            opaged.kv_store_ref(new, pool, *t, HKV, D, BS)
        ref = opaged.paged_attention_ref(q.float().numpy(), *pools, *t, HQ, HKV, D, BS)
    else:
        ref = attention_16(q, k, v, rows, t, nb)
    op = b2a.PagedAttentionOp(HQ, HKV, D, BS, cache.kv_dtype, max_seqs=2 * pairs, max_context_len=4096, q_dtype=dt,
                              max_prefill_kv_tokens=4096)
    work = {"mutable": [torch.empty(n, dtype=torch.uint8, device="cuda") for n in op.GetWorkBufferRequest()["mutable_sizes"]]}
    first = [c.clone() for c in (cache.k, cache.v)]
    dev, ins = [torch.from_numpy(x).cuda() for x in t], [x.cuda() for x in (q, k, v)]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.empty(tokens, HQ * D, dtype=dt, device="cuda")
    u = 2.0 ** -11 if dt == torch.float16 else 2.0 ** -8
    for _ in range(5):  # from the same pool each time: what the step before stored is gone
        cache.k.copy_(first[0])
        cache.v.copy_(first[1])
        out.zero_()
        op.Execute([*ins, cache.k, cache.v, *dev, None, 0], [out], workbuffers=work, status=status)
        assert int(status.item()) == 0
        if kv == "u8":
            assert_close(out, ref, dt)
            continue
        # the result is rounded to the type; sums and probabilities are float32's
        err = np.abs(out.double().cpu().numpy() - ref)
        assert (err <= u * np.abs(ref) + 5e-5).all(), float((err - u * np.abs(ref)).max())


def attention_16(q, k, v, rows, t, nb):
    """Store, then attention, over pools of the rows' own type, in float64."""
    past, sb, bi, bb = t
    pool = [r.double().numpy().reshape(nb, BS, HKV, D).copy() for r in rows]
    for s in range(len(past)):
        for i in range(sb[s + 1] - sb[s]):
            p = past[s] + i
            for which, new in ((0, k), (1, v)):
                pool[which][bi[bb[s] + p // BS], p % BS] = new[sb[s] + i].double().numpy().reshape(HKV, D)
    out = np.zeros((len(q), HQ, D))
    for s in range(len(past)):
        kk, vv = (p[bi[bb[s]:bb[s + 1]]].reshape(-1, HKV, D) for p in pool)
        for i in range(sb[s + 1] - sb[s]):
            n = past[s] + i + 1
            for h in range(HQ):
                sc = kk[:n, h // (HQ // HKV)] @ q[sb[s] + i].double().numpy().reshape(HQ, D)[h] / np.sqrt(D)
                e = np.exp(sc - sc.max())
                out[sb[s] + i, h] = e / e.sum() @ vv[:n, h // (HQ // HKV)]
    return out.reshape(len(q), HQ * D)
