"""The tensor-core form that keeps the probabilities' precision: head size 64, and masks that cannot be read in 16-byte pieces."""
import numpy as np
import pytest
import torch

from oracle import sdpa as osdpa

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def b2a():
    import openvino_contrib_b200 as m
    assert torch.cuda.is_available()
    return m


def _check(out, ref, dtype, what=""):
    # the result's own rounding (half a unit in the last place: 2^-11 of the value in f16, 2^-9 in bf16; twice that is
    # allowed), and float32 sums of values up to about five.  The probabilities keep 22 (f16) or 24 bits (bf16)
    rtol = 2.0 ** -10 if dtype == torch.float16 else 2.0 ** -8
    np.testing.assert_allclose(out.float().cpu().numpy().reshape(ref.shape), ref, rtol=rtol, atol=5e-5, err_msg=what)


def _rand(shape, seed, dtype):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(dtype)


def _masks(b, hq, sq, skv, dtype, kind):
    """kind: none, causal, then {bool, add} x {keys: one row per batch entry, heads: one row per head, full, strided:
    every second key of a wider mask}."""
    if kind in ("none", "causal"):
        return None
    what, form = kind.split("-")
    shape = {"keys": (b, 1, 1, skv), "heads": (1, hq, 1, skv), "full": (b, 1, sq, skv), "strided": (b, hq, sq, 2 * skv)}[form]
    keep = torch.rand(shape, generator=torch.Generator().manual_seed(4)) > 0.4
    if form == "strided":
        keep = keep[..., ::2]
    keep[..., 0] = True
    if what == "bool":
        return keep
    low = torch.tensor(torch.finfo(dtype).min)
    add = torch.where(keep, torch.tensor(0.25), low).to(dtype)
    return add


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("b,hq,hkv,sq,skv,d", [
    (1, 4, 4, 33, 31, 64), (2, 2, 2, 127, 129, 64), (2, 4, 2, 128, 128, 64),    # around one tile
    (1, 3, 1, 257, 511, 64), (3, 12, 12, 300, 300, 64), (1, 2, 2, 1030, 1153, 64),  # odd groups; several tiles
    (2, 40, 40, 520, 260, 64),                                                  # more items than SMs
    (1, 4, 2, 150, 131, 128), (2, 2, 2, 129, 257, 128),                         # head size 128, odd key counts
])
@pytest.mark.parametrize("mask", ["none", "causal", "bool-keys", "add-keys", "bool-heads", "add-heads", "bool-full", "add-full",
                                  "add-strided"])
@pytest.mark.parametrize("layout", ["bhsd", "bshd"])
def test_against_the_oracle(b2a, dtype, b, hq, hkv, sq, skv, d, mask, layout):
    if d == 128 and mask in ("none", "causal"):
        pytest.skip("the other tensor-core form")
    if layout == "bshd" and mask in ("bool-full", "add-heads", "add-strided"):
        pytest.skip("covered in the other layout")
    q, k, v = _rand((b, hq, sq, d), 1, dtype), _rand((b, hkv, skv, d), 2, dtype), _rand((b, hkv, skv, d), 3, dtype)
    m = _masks(b, hq, sq, skv, dtype, mask)
    dev = [t.transpose(1, 2).contiguous().cuda().transpose(1, 2) if layout == "bshd" else t.cuda() for t in (q, k, v)]
    out = torch.full((b, sq, hq, d), 7.0, dtype=dtype, device="cuda").transpose(1, 2) if layout == "bshd" else \
        torch.full((b, hq, sq, d), 7.0, dtype=dtype, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    b2a.sdpa(*dev, None if m is None else m.cuda(), causal=mask == "causal", out=out, status=status)
    assert int(status.item()) == 0
    _check(out, osdpa.sdpa_ref(q, k, v, mask=m, causal=mask == "causal"), dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d", [64, 128])
def test_fully_masked_rows(b2a, dtype, d):
    # every key removed: zeros.  Every key at bf16's lowest value, whose product with log2(e) is not finite: nothing of the
    # scores is left, the plain average of the values.  The first key tile masked and the second not: only the second.
    q, k, v = _rand((3, 4, 140, d), 1, dtype), _rand((3, 4, 201, d), 2, dtype), _rand((3, 4, 201, d), 3, dtype)
    low = torch.finfo(dtype).min
    for rows in (1, 140):
        m = torch.zeros(3, 1, rows, 201, dtype=dtype)
        m[0] = float("-inf")
        m[1] = low
        m[2, :, :, :150] = low
        out = b2a.sdpa(q.cuda(), k.cuda(), v.cuda(), m.cuda())
        assert float(out[0].abs().max()) == 0.0
        if dtype == torch.bfloat16:
            _check(out[1], v[1].float().mean(1, keepdim=True).expand(4, 140, d).numpy(), dtype)
        _check(out[2], osdpa.sdpa_ref(q[2:, :, :, :], k[2:, :, 150:], v[2:, :, 150:])[0], dtype)
        keep = torch.ones(3, 1, rows, 201, dtype=torch.bool)
        keep[0] = False
        keep[2, :, :, :150] = False
        out = b2a.sdpa(q.cuda(), k.cuda(), v.cuda(), keep.cuda())
        assert float(out[0].abs().max()) == 0.0
        _check(out[2], osdpa.sdpa_ref(q[2:, :, :, :], k[2:, :, 150:], v[2:, :, 150:])[0], dtype)


def test_precision_is_that_of_float32_probabilities(b2a):
    b, h, s, d = 1, 2, 512, 64
    q, k = _rand((b, h, s, d), 1, torch.float16), _rand((b, h, s, d), 2, torch.float16)
    v = _rand((b, h, s, d), 3, torch.float16)
    out = b2a.sdpa(q.cuda(), k.cuda(), v.cuda()).double().cpu()
    p = torch.softmax((q.double() @ k.double().transpose(-1, -2)) / 8.0, -1)
    ref = p @ v.double()
    # rounding the result errs by at most 2^-11 of each value and, spread evenly over that, by 2^-11 / sqrt(3) times at most
    # 1 / sqrt(2)..1 of it in the 2-norm: below 2^-11.8 in all.  Probabilities in f16 alone would add their own 2^-12.3.
    assert float((out - ref).norm() / ref.norm()) < 2.0 ** -11.8


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("heads,sq,d,mask", [(2, 140, 64, "none"), (160, 140, 64, "none"), (2, 140, 64, "keys"), (2, 140, 64, "rows"),
                                             (2, 140, 128, "keys"), (2, 140, 128, "rows")])
@pytest.mark.parametrize("gap", [10.0, 16.0, 17.4, 20.0])
def test_many_keys_far_below_one(b2a, dtype, heads, sq, d, mask, gap):
    # an attention sink: one key with a zero value row stands `gap` above thousands of equal ones, whose values are the result.
    # Their probabilities lie down to 2^-29 below the maximum, under f16's smallest value times 2^-4.  Bounds: the rounding of
    # the result (half a unit in the last place, 2^-25 where f16 has no smaller step; twice that is allowed), beside which the
    # 2^-14 of exponentials and split vanish.  (160 heads: pairs of tiles; 2: their keys shared out)
    n = 2047 if heads > 2 else 32767
    q, k, v = torch.zeros(1, heads, sq, d), torch.zeros(1, heads, n, d), torch.ones(1, heads, n, d)
    q[..., 0], k[:, :, 5, 0], v[:, :, 5] = 1.0, gap, 0.0
    q, k, v = q.to(dtype), k.to(dtype), v.to(dtype)
    m = None if mask == "none" else torch.zeros(1, 1, 1 if mask == "keys" else sq, n, dtype=dtype)
    out = b2a.sdpa(q.cuda(), k.cuda(), v.cuda(), None if m is None else m.cuda(), scale=1.0)
    ref = osdpa.sdpa_ref(q[:, :2, :1], k[:, :2], v[:, :2], scale=1.0)
    np.testing.assert_allclose(out.float().cpu().numpy(), np.broadcast_to(ref[:, :1], out.shape), atol=2.0 ** -24,
                               rtol=2.0 ** -10 if dtype == torch.float16 else 2.0 ** -8)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("d,n,masked", [(64, 128, False), (64, 333, False), (64, 333, True), (128, 333, True)])
def test_an_infinity_in_the_values_stays_one(b2a, dtype, d, n, masked):
    q, k, v = _rand((1, 2, 150, d), 1, dtype), _rand((1, 2, n, d), 2, dtype), _rand((1, 2, n, d), 3, dtype)
    v[0, 0, 7, 3], v[0, 1, n - 1, d - 1] = float("inf"), float("-inf")
    m = torch.ones(1, 1, 1, n, dtype=torch.bool) if masked else None
    out = b2a.sdpa(q.cuda(), k.cuda(), v.cuda(), None if m is None else m.cuda()).float().cpu()
    assert (out[0, 0, :, 3] == float("inf")).all() and (out[0, 1, :, d - 1] == float("-inf")).all()
    v[0, 0, 7, 3] = v[0, 1, n - 1, d - 1] = 0.0
    out[0, 0, :, 3] = out[0, 1, :, d - 1] = 0.0
    ref = osdpa.sdpa_ref(q, k, v)
    ref[0, 0, :, 3] = ref[0, 1, :, d - 1] = 0.0
    _check(out, ref, dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("heads,sq,skv,d", [(2, 140, 300, 64), (100, 140, 300, 64), (2, 140, 300, 128), (100, 140, 300, 128),
                                            (2, 129, 130, 64), (2, 4, 60, 128)])
def test_causal_reads_no_key_beyond_the_queries(b2a, dtype, heads, sq, skv, d):
    # the unfilled rows of a cache hold anything: causal attention stops at key Sq - 1
    q, k, v = _rand((1, heads, sq, d), 1, dtype), _rand((1, heads, skv, d), 2, dtype), _rand((1, heads, skv, d), 3, dtype)
    k[:, :, sq:] = float("nan")
    v[:, :, sq:] = float("nan")
    out = b2a.sdpa(q.cuda(), k.cuda(), v.cuda(), causal=True)
    assert torch.equal(out, b2a.sdpa(q.cuda(), k[:, :, :sq].contiguous().cuda(), v[:, :, :sq].contiguous().cuda(), causal=True))


@pytest.mark.parametrize("skv", [200, 201, 1000])
@pytest.mark.parametrize("rows", [1, 140])
def test_the_lowest_value_in_every_place_is_an_average(b2a, skv, rows):
    # bf16's lowest value times log2(e) is not finite; nothing of the scores is left, whatever form reads the mask
    q, k, v = (_rand((2, 4, n, 128), s, torch.bfloat16) for n, s in ((140, 1), (skv, 2), (skv, 3)))
    m = torch.full((2, 1, rows, skv), torch.finfo(torch.bfloat16).min, dtype=torch.bfloat16)
    m[1, :, :, :150] = float("-inf")
    out = b2a.sdpa(q.cuda(), k.cuda(), v.cuda(), m.cuda())
    for i, lo in ((0, 0), (1, 150)):
        _check(out[i], v[i, :, lo:].float().mean(1, keepdim=True).expand(4, 140, 128).numpy(), torch.bfloat16)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("sq,rows,skv,d", [(1, 1, 100, 128), (140, 1, 201, 64), (140, 140, 201, 64), (140, 140, 200, 128)])
def test_a_nan_in_the_mask_stays_one(b2a, dtype, sq, rows, skv, d):
    q, k, v = _rand((2, 2, sq, d), 1, dtype), _rand((2, 2, skv, d), 2, dtype), _rand((2, 2, skv, d), 3, dtype)
    m = torch.zeros(2, 1, rows, skv, dtype=dtype)
    m[1, :, rows // 2, 70] = float("nan")
    out = b2a.sdpa(q.cuda(), k.cuda(), v.cuda(), m.cuda()).float().cpu()
    hit = torch.zeros(sq, dtype=torch.bool)
    hit[rows // 2 if rows > 1 else slice(None)] = True
    assert torch.isnan(out[1][:, hit]).all() and torch.isfinite(out[1][:, ~hit]).all() and torch.isfinite(out[0]).all()
