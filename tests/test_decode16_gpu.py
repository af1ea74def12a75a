"""A few query rows over 16-bit keys and values on the GPU: dense tensors (any mask, any layout) and a 16-bit block pool."""
import numpy as np
import pytest
import torch

from oracle import paged as opaged
from oracle import sdpa as osdpa

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def b2a():
    import openvino_contrib_b200 as m
    assert torch.cuda.is_available()
    return m


def _check(out, ref, dtype, what=""):
    # the probabilities keep float32 precision, so what is left is the rounding of the result (half a unit in the last
    # place: 2^-11 of the value in f16, 2^-9 in bf16; twice that is allowed) and float32 sums of values up to about five
    rtol = 2.0 ** -10 if dtype == torch.float16 else 2.0 ** -8
    np.testing.assert_allclose(out.float().cpu().numpy().reshape(ref.shape), ref, rtol=rtol, atol=5e-5, err_msg=what)


def _rand(shape, seed, dtype):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("b,hq,hkv,sq,skv,d", [
    (1, 1, 1, 1, 1, 64), (1, 4, 4, 1, 15, 128), (2, 8, 2, 1, 17, 128),     # below and just above one 16-key tile
    (3, 32, 4, 1, 64, 64), (2, 64, 4, 1, 1027, 128),                       # 8 and 16 rows per KV head
    (1, 6, 2, 5, 333, 128), (1, 4, 1, 4, 100, 64),                         # several query positions
    (1, 8, 8, 1, 4097, 128), (40, 16, 8, 1, 130, 128),                     # eight CTAs per cluster; many small problems
])
@pytest.mark.parametrize("mask", ["none", "bool", "add", "causal"])
def test_few_rows_on_dense_tensors(b2a, dtype, b, hq, hkv, sq, skv, d, mask):
    q, k, v = _rand((b, hq, sq, d), 1, dtype), _rand((b, hkv, skv + 3, d), 2, dtype), _rand((b, hkv, skv + 3, d), 3, dtype)
    k, v = k[:, :, :skv], v[:, :, :skv]  # the filled part of a longer cache
    m = None
    if mask in ("bool", "add"):
        keep = torch.rand(b, 1, sq, skv, generator=torch.Generator().manual_seed(4)) > 0.4
        keep[..., -1] = True
        m = keep if mask == "bool" else torch.where(keep, torch.tensor(0.25), torch.tensor(torch.finfo(dtype).min)).to(dtype)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    store = torch.zeros(b, sq, hq, d, dtype=dtype, device="cuda")
    mk = None if m is None else m.cuda()
    kc, vc = k.cuda(), v.cuda()
    b2a.sdpa(q.cuda(), kc, vc, mk, causal=mask == "causal", out=store.transpose(1, 2), status=status)
    assert int(status.item()) == 0
    _check(store.transpose(1, 2), osdpa.sdpa_ref(q, k, v, mask=m, causal=mask == "causal"), dtype)


def test_fully_masked_rows(b2a):
    # every key removed: zeros; every key at one large negative value: softmax of the scores as float32 keeps them.
    # bf16's lowest value leaves nothing of the scores: the plain average of the values.  -60000 in f16 leaves multiples
    # of 2^-8 (the reference) or 2^-7 in base-2 units (the kernel): a score moves by at most 2^-9 or 2^-8 * ln 2, so the
    # probabilities of the two differ by at most a factor exp(2 * (0.0020 + 0.0027)) and the average by 0.0094 * mean|v|.
    for dtype in (torch.float16, torch.bfloat16):
        q, k, v = _rand((2, 8, 1, 128), 1, dtype), _rand((2, 2, 50, 128), 2, dtype), _rand((2, 2, 50, 128), 3, dtype)
        m = torch.zeros(2, 1, 1, 50, dtype=dtype)
        m[0] = float("-inf")
        m[1] = torch.finfo(torch.bfloat16).min if dtype == torch.bfloat16 else -60000.0
        out = b2a.sdpa(q.cuda(), k.cuda(), v.cuda(), m.cuda())
        assert float(out[0].abs().max()) == 0.0
        if dtype == torch.bfloat16:
            _check(out[1], v[1].float().mean(1, keepdim=True).repeat_interleave(4, 0).numpy(), dtype)
        else:
            ref = osdpa.sdpa_ref(q[1:], k[1:], v[1:], mask=m[1:])[0]
            bound = 0.0094 * float(v[1].float().abs().mean(1).max())
            assert float(np.abs(out[1].float().cpu().numpy() - ref).max()) <= bound


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("hq,hkv,d,bs", [(32, 8, 128, 16), (8, 8, 64, 32), (64, 4, 128, 16)])
def test_sixteen_bit_pool(b2a, dtype, hq, hkv, d, bs):
    # one-token sequences on the decode kernel, two multi-token ones (and an idle one) on the general kernel; with and
    # without a sliding window; the pool's unused slots hold NaN bytes
    past = np.array([0, 15, 16, 1000, 3, 40, 20, 2600], np.int32)
    qlen = np.array([1, 1, 1, 1, 9, 1, 0, 33], np.int32)
    ctx = past + qlen
    bi, bb, nb = opaged.build_block_tables(ctx, bs, seed=5, spare_blocks=3)
    sb = np.zeros(len(ctx) + 1, np.int32)
    sb[1:] = np.cumsum(qlen)
    rows_k = [_rand((int(c), hkv, d), 10 + s, dtype) for s, c in enumerate(ctx)]
    rows_v = [_rand((int(c), hkv, d), 50 + s, dtype) for s, c in enumerate(ctx)]
    cache = b2a.PagedKvCache.allocate(nb, hkv, d, bs, dtype)
    full = np.zeros(len(ctx) + 1, np.int32)
    full[1:] = np.cumsum(ctx)
    t = [torch.from_numpy(a).cuda() for a in (np.zeros(len(ctx), np.int32), full, bi, bb)]
    b2a.paged_kv_store(torch.cat(rows_k).reshape(-1, hkv * d).cuda(), torch.cat(rows_v).reshape(-1, hkv * d).cuda(), cache, *t)
    q = _rand((int(sb[-1]), hq * d), 99, dtype)
    t = [torch.from_numpy(a).cuda() for a in (past, sb, bi, bb)]
    for window in (0, 30):
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        out = b2a.paged_attention(q.cuda(), cache, *t, hq=hq, max_context_len=4096, max_q_len=33, sliding_window=window,
                                  status=status)
        assert int(status.item()) == 0
        for s in range(len(ctx)):
            n = int(qlen[s])
            if n == 0:
                continue
            pos = past[s] + np.arange(n)[:, None]
            at = np.arange(int(ctx[s]))[None]
            keep = (at <= pos) & ((pos - at < window) if window else True)
            ref = osdpa.sdpa_ref(q[sb[s]:sb[s + 1]].reshape(n, hq, d).transpose(0, 1)[None], rows_k[s].transpose(0, 1)[None],
                                 rows_v[s].transpose(0, 1)[None], mask=keep[None, None])
            _check(out[sb[s]:sb[s + 1]], ref[0].transpose(1, 0, 2).reshape(n, -1), dtype, f"sequence {s}, window {window}")
    # a block index outside the pool is reported and not followed
    bad = bi.copy()
    bad[int(bb[3]) + 2] = nb + 7
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = b2a.paged_attention(q.cuda(), cache, t[0], t[1], torch.from_numpy(bad).cuda(), t[3], hq=hq, max_context_len=4096,
                              max_q_len=33, status=status)
    assert int(status.item()) & 2 and torch.isfinite(out.float()).all()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("sq,d", [(1, 128), (1, 64), (12, 128)])
@pytest.mark.parametrize("gap", [10.0, 16.0, 17.4, 20.0])
def test_many_keys_far_below_one(b2a, dtype, sq, d, gap):
    # an attention sink: one key with a zero value row stands `gap` above 32768 equal ones, whose values are the result.
    # Their probabilities lie down to 2^-29 below the maximum, under f16's smallest value times 2^-4.  Bounds: the rounding of
    # the result (half a unit in the last place, 2^-25 where f16 has no smaller step; twice that is allowed), beside which the
    # 2^-20 of exponentials and split vanish.
    n = 32768
    q, k, v = torch.zeros(1, 2, sq, d), torch.zeros(1, 2, n, d), torch.ones(1, 2, n, d)
    q[..., 0], k[:, :, 5, 0], v[:, :, 5] = 1.0, gap, 0.0
    q, k, v = q.to(dtype), k.to(dtype), v.to(dtype)
    out = b2a.sdpa(q.cuda(), k.cuda(), v.cuda(), scale=1.0)
    np.testing.assert_allclose(out.float().cpu().numpy(), osdpa.sdpa_ref(q, k, v, scale=1.0), atol=2.0 ** -24,
                               rtol=2.0 ** -10 if dtype == torch.float16 else 2.0 ** -8)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("sq,d,n", [(1, 128, 100), (4, 64, 333), (12, 128, 3000)])
def test_an_infinity_in_the_values_stays_one(b2a, dtype, sq, d, n):
    q, k, v = _rand((1, 2, sq, d), 1, dtype), _rand((1, 2, n, d), 2, dtype), _rand((1, 2, n, d), 3, dtype)
    v[0, 0, 7, 3], v[0, 1, n - 1, d - 1] = float("inf"), float("-inf")
    out = b2a.sdpa(q.cuda(), k.cuda(), v.cuda()).float().cpu()
    assert (out[0, 0, :, 3] == float("inf")).all() and (out[0, 1, :, d - 1] == float("-inf")).all()
    v[0, 0, 7, 3] = v[0, 1, n - 1, d - 1] = 0.0
    out[0, 0, :, 3] = out[0, 1, :, d - 1] = 0.0
    ref = osdpa.sdpa_ref(q, k, v)
    ref[0, 0, :, 3] = ref[0, 1, :, d - 1] = 0.0
    _check(out, ref, dtype)
