"""Rows copied into a pool of their own 16-bit type, and the attention that starts on cached blocks while the store drains."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def tables(past, new, block_size, seed):
    """past, begins, block ids and their begins of a step, the blocks in shuffled order."""
    per = [(p + n + block_size - 1) // block_size for p, n in zip(past, new)]
    ids = np.random.RandomState(seed).permutation(sum(per) + 3)[:sum(per)]
    cum = lambda x: np.concatenate([[0], np.cumsum(x)])  # noqa: E731
    return [np.asarray(t, np.int32) for t in (past, cum(new), ids, cum(per))]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("hkv,d,block_size", [(1, 128, 16), (2, 64, 16), (3, 128, 16), (8, 128, 32), (16, 8, 5), (16, 16, 8),
                                              # no whole warps a token: the general kernel
                                              (2, 8, 8), (1, 64, 16), (4, 12, 16)])
@pytest.mark.parametrize("new", [[1] * 5, [1, 7, 1, 40], [33]])
def test_rows_land_in_their_blocks(dtype, hkv, d, block_size, new):
    import openvino_contrib_b200 as b2a
    past = [3 * i * block_size // 2 for i in range(len(new))]
    t = tables(past, new, block_size, 1)
    cache = b2a.PagedKvCache.allocate(int(t[2].max()) + 4, hkv, d, block_size, dtype)
    rows = [torch.randn(sum(new), hkv * d, generator=torch.Generator().manual_seed(i)).to(dtype) for i in range(2)]
    rows[0][0, 0], rows[1][-1, -1] = float("inf"), 1e-7
    quiet = 0x7E01 if dtype == torch.float16 else 0x7FC1  # NaNs with a payload and a sign, which become the canonical one
    rows[0].view(torch.int16)[-1, 2], rows[1].view(torch.int16)[0, 3] = quiet, quiet - 0x8000
    before = [c.cpu().numpy().copy() for c in (cache.k, cache.v)]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    b2a.paged_kv_store(rows[0].cuda(), rows[1].cuda(), cache, *[torch.from_numpy(x).cuda() for x in t], status=status)
    assert int(status.item()) == 0
    for pool, was, r in zip((cache.k, cache.v), before, rows):
        want = was.view(np.uint16).reshape(-1, hkv, block_size, d)
        bits = r.view(torch.int16).numpy().view(np.uint16).reshape(-1, hkv, d).copy()
        bits[torch.isnan(r).numpy().reshape(bits.shape)] = 0x7FFF
        for s in range(len(new)):
            for i in range(new[s]):
                pos = past[s] + i
                want[t[2][t[3][s] + pos // block_size], :, pos % block_size] = bits[t[1][s] + i]
        np.testing.assert_array_equal(pool.cpu().numpy().view(np.uint16).reshape(want.shape), want)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("hkv,d", [(2, 64), (16, 8), (2, 8)])  # (the last: the general kernel)
@pytest.mark.parametrize("what", ["block id too large", "block id negative", "no block for the position", "negative past",
                                  "tokens that no sequence has"])
def test_bad_tables_are_reported_and_write_nothing(dtype, hkv, d, what):
    import openvino_contrib_b200 as b2a
    from openvino_contrib_b200._lib import DEV_BAD_BLOCK, DEV_BAD_LEN
    past, new = [20, 3, 40], [1, 30, 1]
    t = tables(past, new, 16, 4)
    cache = b2a.PagedKvCache.allocate(int(t[2].max()) + 4, hkv, d, 16, dtype, poison=0x5A)
    tokens, lost, status_bit = sum(new), set(), 0
    if what.startswith("block id"):
        t[2][t[3][1]] = cache.num_blocks if "large" in what else -1  # the second sequence's first block: its positions 3 to 15
        lost, status_bit = set(range(1, 14)), DEV_BAD_BLOCK
    elif what == "no block for the position":
        t[0][1] = 10  # positions 10 to 39, and two blocks instead of three
        t[3][2:] -= 1
        t[2] = np.delete(t[2], t[3][2])
        lost, status_bit = {1 + i for i in range(30) if 10 + i >= 32}, DEV_BAD_LEN
    elif what == "negative past":
        t[0][2] = -5
        lost, status_bit = {31}, DEV_BAD_LEN
    else:
        tokens += 9  # rows behind the last sequence's
        lost = set(range(32, 41))
    rows = [torch.randn(tokens, hkv * d, generator=torch.Generator().manual_seed(i)).to(dtype) for i in range(2)]
    before = [c.cpu().numpy().copy() for c in (cache.k, cache.v)]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    b2a.paged_kv_store(rows[0].cuda(), rows[1].cuda(), cache, *[torch.from_numpy(x).cuda() for x in t], status=status)
    assert int(status.item()) == status_bit
    for pool, was, r in zip((cache.k, cache.v), before, rows):
        want = was.view(np.uint16).reshape(-1, hkv, 16, d)
        bits = r.view(torch.int16).numpy().view(np.uint16).reshape(-1, hkv, d)
        for s in range(len(new)):
            for i in range(new[s]):
                if t[1][s] + i in lost:
                    continue
                pos = t[0][s] + i
                want[t[2][t[3][s] + pos // 16], :, pos % 16] = bits[t[1][s] + i]
        np.testing.assert_array_equal(pool.cpu().numpy().view(np.uint16).reshape(want.shape), want)


def attention_rows(q, pools, past, t, hq, hkv, d, block_size, window):
    """One new token per sequence over pools [blocks, hkv, block_size, d], in float64."""
    out = np.zeros((len(q), hq, d))
    for s, p in enumerate(past):
        blocks = t[2][t[3][s]:t[3][s + 1]]
        keys, values = (x[blocks].transpose(1, 0, 2, 3).reshape(hkv, -1, d)[:, :p + 1] for x in pools)
        lo = max(0, p + 1 - window) if window else 0
        for h in range(hq):
            sc = keys[h * hkv // hq, lo:] @ q[s].reshape(hq, d)[h] / np.sqrt(d)
            e = np.exp(sc - sc.max())
            out[s, h] = e / e.sum() @ values[h * hkv // hq, lo:]
    return out.reshape(len(q), hq * d)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("window", [0, 40])
@pytest.mark.parametrize("captured", [False, True])
def test_steps_through_the_operator_see_their_new_rows(dtype, d, window, captured):
    # Store, attention, store, attention ..: the attention reads block ids, and asks for its first tiles, while the store in front
    # of it drains.  The slots of all new tokens hold NaN in the beginning, so a row that was read too early shows; the new
    # row is the first of a block, its last, and one inside, in contexts of one tile and of many.
    import openvino_contrib_b200 as b2a
    past0, hkv, hq, steps = [0, 15, 16, 14, 300, 2047, 2048, 5000], 2, 8, 3
    n = len(past0)
    t = tables(past0, [steps] * n, 16, 2)
    begins = np.arange(n + 1, dtype=np.int32)
    g = torch.Generator().manual_seed(d + window)
    filled = torch.randn(2, int(t[2].max()) + 1, hkv, 16, d, generator=g).to(dtype)
    for s, p in enumerate(past0):
        for pos in range(p, p + steps):
            filled[:, t[2][t[3][s] + pos // 16], :, pos % 16] = float("nan")
    rows = [[torch.randn(n, h * d, generator=g).to(dtype) for h in (hq, hkv, hkv)] for _ in range(steps)]
    cache = b2a.PagedKvCache.allocate(filled.shape[1], hkv, d, 16, dtype)
    op = b2a.PagedAttentionOp(hq, hkv, d, 16, dtype, max_seqs=n, max_context_len=5100, sliding_window=window, q_dtype=dtype)
    work = {"mutable": [torch.empty(m, dtype=torch.uint8, device="cuda") for m in op.GetWorkBufferRequest()["mutable_sizes"]]}
    pasts = [torch.tensor(past0, dtype=torch.int32, device="cuda") + i for i in range(steps)]
    dev = [torch.from_numpy(x).cuda() for x in (begins, t[2], t[3])]
    ins = [[x.cuda() for x in r] for r in rows]
    outs = [torch.empty(n, hq * d, dtype=dtype, device="cuda") for _ in range(steps)]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    fresh = filled.cuda()

    def run():
        for pool, x in zip((cache.k, cache.v), fresh):
            pool.view(dtype).view(x.shape).copy_(x)
        for i in range(steps):
            op.Execute([*ins[i], cache.k, cache.v, pasts[i], *dev, None, window], [outs[i]], workbuffers=work, status=status)

    if captured:
        graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.graph(graph, stream=side):
            run()
        torch.cuda.synchronize()
        run = graph.replay
    for _ in range(2):  # (the second time from the pool with its NaNs again)
        run()
        assert int(status.item()) == 0
        pools = [x.double().numpy() for x in filled]
        u = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
        for i in range(steps):
            q, k, v = (x.double().numpy() for x in rows[i])
            for s, p in enumerate(past0):
                at = t[2][t[3][s] + (p + i) // 16], slice(None), (p + i) % 16
                pools[0][at], pools[1][at] = k[s].reshape(hkv, d), v[s].reshape(hkv, d)
            ref = attention_rows(q, pools, [p + i for p in past0], t, hq, hkv, d, 16, window)
            # the result is rounded to the type; sums and probabilities are float32's (5000 terms of order one)
            err = np.abs(outs[i].double().cpu().numpy() - ref)
            assert (err <= u * np.abs(ref) + 5e-5).all(), (i, float((err - u * np.abs(ref)).max()))
