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
@pytest.mark.parametrize("hkv,d,block_size", [(1, 128, 16), (2, 64, 16), (3, 128, 16), (8, 128, 32), (2, 8, 8), (16, 8, 5),
                                              (1, 64, 16), (4, 12, 16)])  # (the last two: the general kernel)
@pytest.mark.parametrize("new", [[1] * 5, [1, 7, 1, 40], [33]])
def test_rows_land_in_their_blocks(dtype, hkv, d, block_size, new):
    import openvino_contrib_b200 as b2a
    past = [3 * i * block_size // 2 for i in range(len(new))]
    t = tables(past, new, block_size, 1)
    cache = b2a.PagedKvCache.allocate(int(t[2].max()) + 4, hkv, d, block_size, dtype)
    rows = [torch.randn(sum(new), hkv * d, generator=torch.Generator().manual_seed(i)).to(dtype) for i in range(2)]
    rows[0][0, 0], rows[1][-1, -1] = float("inf"), 1e-7
    before = [c.cpu().numpy().copy() for c in (cache.k, cache.v)]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    b2a.paged_kv_store(rows[0].cuda(), rows[1].cuda(), cache, *[torch.from_numpy(x).cuda() for x in t], status=status)
    assert int(status.item()) == 0
    for pool, was, r in zip((cache.k, cache.v), before, rows):
        want = was.view(np.uint16).reshape(-1, hkv, block_size, d)
        bits = r.view(torch.int16).numpy().view(np.uint16).reshape(-1, hkv, d)
        for s in range(len(new)):
            for i in range(new[s]):
                pos = past[s] + i
                want[t[2][t[3][s] + pos // block_size], :, pos % block_size] = bits[t[1][s] + i]
        np.testing.assert_array_equal(pool.cpu().numpy().view(np.uint16).reshape(want.shape), want)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("window", [0, 40])
def test_settled_rows_give_the_same_bits(d, window):
    import openvino_contrib_b200 as b2a
    past, hkv, hq = [0, 15, 16, 17, 300, 2047, 2048, 5000], 2, 8
    t = tables(past, [1] * len(past), 16, 2)
    dev = [torch.from_numpy(x).cuda() for x in t]
    cache = b2a.PagedKvCache.allocate(int(t[2].max()) + 1, hkv, d, 16, torch.float16)
    cache.k.view(torch.float16).normal_(), cache.v.view(torch.float16).normal_()
    q, k, v = (torch.randn(len(past), h * d, device="cuda").half() for h in (hq, hkv, hkv))
    outs = []
    for settled in (False, True):
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        b2a.paged_kv_store(k, v, cache, *dev, status=status)
        outs.append(b2a.paged_attention(q, cache, *dev, hq=hq, max_context_len=5001, max_q_len=1, sliding_window=window, status=status,
                                        cache_rows_settled=settled))
        assert int(status.item()) == 0
        k, v = k.clone(), v.clone()
    assert torch.equal(*outs)
