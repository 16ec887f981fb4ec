"""Decode attention over pages on the matrix instructions against 64-bit attention over the same (dequantised) pages:
every head count and size it is built for, both page types, sequences that end at, before and behind tiles of 16 keys
and splits, page sizes that tiles do not line up with.  Everything in the pool that no sequence owns is NaN."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

LENS = [1, 15, 16, 17, 64, 65, 333]


def _case(hq, hk, hd, bs, int8, lens=LENS, q_size=1.0):
    g = torch.Generator("cuda").manual_seed(hq * 1000 + hd + bs)
    B, mb = len(lens), -(-max(lens) // bs)
    nb = B * mb
    tables = torch.randperm(nb, device="cuda", generator=g).to(torch.int32).reshape(B, mb)
    q = (q_size * torch.randn(B, hq * hd, device="cuda", generator=g)).bfloat16()
    pos = torch.arange(mb * bs, device="cuda")
    owned = torch.zeros(nb, bs, dtype=torch.bool, device="cuda")
    for b, n in enumerate(lens):
        owned[tables[b, pos[:n] // bs].long(), pos[:n] % bs] = True
    owned = owned[:, None, :].expand(nb, hk, bs)
    if int8:
        pools = [torch.randint(-127, 128, (nb, hk, bs, hd), device="cuda", dtype=torch.int8, generator=g) for _ in range(2)]
        # value scales over six powers of ten: a weight times its scale is far from 1
        scales = [torch.rand(nb, hk, bs, device="cuda", generator=g) * 0.02 + 0.005,
                  10.0 ** (torch.rand(nb, hk, bs, device="cuda", generator=g) * 6 - 5)]
        real = [p.double() * s.double()[..., None] for p, s in zip(pools, scales)]
        scales = [torch.where(owned, s, math.nan) for s in scales]
    else:
        pools = [torch.randn(nb, hk, bs, hd, device="cuda", generator=g).bfloat16() for _ in range(2)]
        real = [p.double() for p in pools]
        pools = [torch.where(owned[..., None], p, math.nan).bfloat16() for p in pools]
        scales = [None, None]
    want = []
    for b, n in enumerate(lens):
        k, v = (r[tables[b, pos[:n] // bs].long(), :, pos[:n] % bs].repeat_interleave(hq // hk, 1) for r in real)
        s = torch.einsum("hd,shd->hs", q[b].double().reshape(hq, hd), k) * hd ** -0.5
        want.append(torch.einsum("hs,shd->hd", torch.softmax(s, -1), v).reshape(-1))
    return B, tables, q, pools, scales, torch.tensor(lens, device="cuda", dtype=torch.int32), torch.stack(want)


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("hd,ratio,hk,bs,splits", [(128, 1, 2, 16, 1), (128, 2, 3, 16, 4), (128, 4, 2, 16, 1), (128, 4, 2, 24, 3),
                                                   (128, 8, 2, 16, 2), (64, 1, 2, 16, 1), (64, 2, 2, 5, 2), (64, 3, 2, 16, 1), (64, 4, 1, 64, 7)])
def test_decode_attention_against_64_bit(hd, ratio, hk, bs, splits, int8):
    from brain_b200.ops._cuda import call, check_error, stream_ptr
    hq = hk * ratio
    B, tables, q, (kc, vc), (ks, vs), lens, want = _case(hq, hk, hd, bs, int8)
    out = torch.full((B, hq * hd + 8), 7.0, device="cuda", dtype=torch.bfloat16)
    po = torch.empty(B * hq * splits * hd, device="cuda")
    pm = torch.empty(B * hq * splits * 2, device="cuda")
    tail = (tables, tables.shape[1], lens, out, out.stride(0), po, pm, B, hq, hk, hd, bs, splits, float(hd ** -0.5), stream_ptr())
    if int8:
        call("paged_decode_i8", q, q.stride(0), kc, vc, ks, vs, *tail)
    else:
        call("paged_decode", q, q.stride(0), kc, vc, *tail)
    check_error()
    assert bool((out[:, hq * hd:] == 7.0).all())
    got = out[:, :hq * hd].double()
    # rounding the result to bf16: at most 2^-9 of each value.  bf16 pages: weights to 17 bits, sums in fp32.  int8
    # pages: the query is kept to 2^-15 of its largest component, |dq.k| <= hd 2^-15 max|q| max|k| / sqrt(hd) < 0.02
    # in the exponent for these keys (|k| <= 3.2, |q| < 5) and in the mean two orders less
    err = (got - want).norm(dim=1) / want.norm(dim=1)
    assert float(err.max()) < (2 ** -9 + 2e-3 if int8 else 2 ** -9 + 2 ** -14), err


@pytest.mark.parametrize("hd,ratio", [(128, 4), (128, 8), (64, 3), (64, 1)])
def test_windowed_capped_decode_against_64_bit(hd, ratio):
    from brain_b200.ops._cuda import call, check_error, stream_ptr
    hk, bs, splits, window, cap = 2, 16, 2, 50, 5.0
    hq = hk * ratio
    B, tables, q, (kc, vc), _, lens, _ = _case(hq, hk, hd, bs, False)
    out = torch.empty(B, hq * hd, device="cuda", dtype=torch.bfloat16)
    po = torch.empty(B * hq * splits * hd, device="cuda")
    pm = torch.empty(B * hq * splits * 2, device="cuda")
    call("paged_decode_x", q, q.stride(0), kc, vc, tables, tables.shape[1], lens, out, out.stride(0), po, pm, B, hq, hk, hd, hd, bs,
         splits, float(hd ** -0.5), cap, None, 0, 0, 1.0, window, stream_ptr())
    check_error()
    pos = torch.arange(tables.shape[1] * bs, device="cuda")
    for b, n in enumerate(LENS):
        keys = pos[max(0, n - window):n]
        k, v = (r[tables[b, keys // bs].long(), :, keys % bs].double().repeat_interleave(ratio, 1) for r in (kc, vc))
        s = cap * torch.tanh(torch.einsum("hd,shd->hs", q[b].double().reshape(hq, hd), k) * hd ** -0.5 / cap)
        want = torch.einsum("hs,shd->hd", torch.softmax(s, -1), v).reshape(-1)
        assert float((out[b].double() - want).norm() / want.norm()) < 2 ** -9 + 2 ** -14


def _run(int8, tables, q, pools, scales, lens, hq, hk, hd, bs, splits):
    """(rows, parts [B, hq, splits, hd], maxima and sums [B, hq, splits, 2])"""
    from brain_b200.ops._cuda import call, check_error, stream_ptr
    B = q.shape[0]
    out = torch.empty(B, hq * hd, device="cuda", dtype=torch.bfloat16)
    po = torch.zeros(B, hq, splits, hd, device="cuda")
    pm = torch.zeros(B, hq, splits, 2, device="cuda")
    tail = (tables, tables.shape[1], lens, out, out.stride(0), po, pm, B, hq, hk, hd, bs, splits, float(hd ** -0.5), stream_ptr())
    if int8:
        call("paged_decode_i8", q, q.stride(0), *pools, *scales, *tail)
    else:
        call("paged_decode", q, q.stride(0), *pools, *tail)
    check_error()
    return out, po, pm


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("hd,ratio,hk,bs,splits,times", [(128, 4, 2, 16, 8, 1), (128, 2, 2, 16, 9, 1), (64, 3, 2, 16, 16, 1), (128, 8, 1, 24, 16, 1),
                                                         (128, 4, 4, 16, 3, 10), (64, 1, 4, 16, 3, 10)])
def test_splits_in_clusters_and_behind_a_merge_kernel(hd, ratio, hk, bs, splits, times, int8):
    """Eight splits are the last that merge in their cluster; more, or more than two CTAs an SM (here 840), leave parts to a
    second kernel.  Sequences of fewer keys than splits among them."""
    lens = LENS * times
    hq = hk * ratio
    _, tables, q, pools, scales, n, want = _case(hq, hk, hd, bs, int8, lens)
    out, _, _ = _run(int8, tables, q, pools, scales, n, hq, hk, hd, bs, splits)
    err = (out.double() - want).norm(dim=1) / want.norm(dim=1)
    assert float(err.max()) < (2 ** -9 + 2e-3 if int8 else 2 ** -9 + 2 ** -14), err      # as above


@pytest.mark.parametrize("hd,ratio", [(128, 1), (128, 2), (128, 4), (128, 8), (64, 1), (64, 2), (64, 3), (64, 4)])
def test_weights_keep_their_24_bits(hd, ratio):
    """The fp32 parts, merged in 64 bits.  A weight is good to 2^-22 (two units of exp2, scores of size 1 summed in fp32) and
    its errors are independent from key to key, as the values are: the result's relative error is no larger.  Weights of 17
    bits err by up to 2^-18, 5e-7 in the mean."""
    hk, bs, splits = 2, 16, 9
    hq = hk * ratio
    _, tables, q, pools, scales, n, want = _case(hq, hk, hd, bs, False, q_size=0.2)
    _, po, pm = _run(False, tables, q, pools, scales, n, hq, hk, hd, bs, splits)
    m, l = pm[..., 0].double(), pm[..., 1].double()
    w = torch.exp2(m - m.max(-1, keepdim=True).values)
    got = ((po.double() * w[..., None]).sum(2) / (l * w).sum(2)[..., None]).reshape(want.shape)
    assert float((got - want).norm() / want.norm()) < 2 ** -22


@pytest.mark.parametrize("hd,ratio", [(128, 1), (128, 4), (128, 8), (64, 3)])
def test_small_values_beside_a_large_one_without_weight(hd, ratio):
    """int8 pages: a row whose scale is ten powers of ten above the others', at a score 60 below theirs."""
    hk, bs = 2, 16
    hq = hk * ratio
    _, tables, q, pools, scales, n, _ = _case(hq, hk, hd, bs, True)
    q = q.abs()                                            # so that a key of -127 scores lowest for every head
    pos = torch.arange(tables.shape[1] * bs, device="cuda")
    blk, off = tables[-1, 100 // bs].long(), 100 % bs      # one key of the longest sequence
    scales[0].fill_(0.002)
    scales[1].fill_(1e-3)
    pools[0][blk, :, off] = -127
    low = 127 * q[-1].double().reshape(hq, hd).sum(1) * hd ** -0.5
    scales[0][blk, :, off] = 60.0 / float(low.min())
    scales[1][blk, :, off] = 1e7
    out, _, _ = _run(True, tables, q, pools, scales, n, hq, hk, hd, bs, 1)
    k, v = (p[tables[-1, pos[:LENS[-1]] // bs].long(), :, pos[:LENS[-1]] % bs].double() *
            s[tables[-1, pos[:LENS[-1]] // bs].long(), :, pos[:LENS[-1]] % bs].double()[..., None] for p, s in zip(pools, scales))
    s = torch.einsum("hd,shd->hs", q[-1].double().reshape(hq, hd), k.repeat_interleave(ratio, 1)) * hd ** -0.5
    want = torch.einsum("hs,shd->hd", torch.softmax(s, -1), v.repeat_interleave(ratio, 1)).reshape(-1)
    assert float((out[-1].double() - want).norm() / want.norm()) < 2 ** -9 + 2e-3      # as for every int8 page


@pytest.mark.parametrize("hd,ratio", [(128, 1), (128, 2), (128, 4), (128, 8), (64, 3)])
@pytest.mark.parametrize("splits", [1, 3, 9])
def test_an_infinite_value_stays_infinite(hd, ratio, splits):
    """A weighted sum with an infinity in it is that infinity, whatever the weight's bits; other columns do not see it."""
    hk, bs = 2, 16
    hq = hk * ratio
    _, tables, q, pools, scales, n, want = _case(hq, hk, hd, bs, False)
    want = want.clone()
    for b, length in enumerate(LENS):
        for at, col, value in ((0, 5, math.inf), (length - 1, 40, -math.inf)):
            pools[1][tables[b, at // bs].long(), :, at % bs, col] = value
            want.reshape(len(LENS), hq, hd)[b, :, col] = value
    out, _, _ = _run(False, tables, q, pools, scales, n, hq, hk, hd, bs, splits)
    finite = torch.isfinite(want)
    assert torch.equal(out.double()[~finite], want[~finite])
    err = torch.where(finite, out.double() - want, 0.0).norm() / torch.where(finite, want, 0.0).norm()
    assert float(err) < 2 ** -9 + 2 ** -14
