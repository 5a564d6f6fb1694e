"""The kernels whose fp32 products are sums of bf16 products, against 64-bit arithmetic: tile edges (rows of 1 to 9 blocks, so that a
step has 1 to 4 of them, every block size and head width, widths that are no multiple of a unit), every operand type, and what is
not finite or close to it, which must come out as plain fp32 arithmetic gives it."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TD = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
# Unit roundoff of what leaves a kernel, and of its fp32 sums.  A product of two split numbers is off by 2^-24 of it (three terms
# of 8 bits each, the products of the smallest left out), a sum of 16 of them is truncated at most six times by 2^-23 of the
# largest partial sum, and sums of 16 are added with one rounding each.
EPS = 2.0 ** -24


def _bound(terms):
    return (1 + 6 * 2 + math.ceil(terms / 16) + 1) * EPS


def _spmm_bound(terms, pt):
    """fp32 blocks go by FMAs: one rounding per term."""
    return max(_bound(terms), terms * EPS) if pt == "f32" else _bound(terms)


def _layout(sfb, nb, bs, seed):
    rng = np.random.RandomState(seed)
    keep = np.zeros((1, nb, nb), np.uint8)
    for i in range(nb):
        keep[0, i, rng.choice(nb, size=min(nb, i + 1), replace=False)] = 1     # rows of 1, 2, ... nb blocks
    lay = sfb.BlockLayout(torch.from_numpy(keep).cuda(), bs)
    return lay, keep[0].astype(bool)


def _blocks(keep, bs, x):
    """[B, H, L, L] -> [B, H, blocks, bs, bs] in row-major block order."""
    nb = keep.shape[0]
    i, j = np.nonzero(keep)
    return x.reshape(x.shape[0], x.shape[1], nb, bs, nb, bs)[:, :, i, :, j].permute(1, 2, 0, 3, 4)


def _dense(keep, bs, p):
    nb = keep.shape[0]
    i, j = np.nonzero(keep)
    out = torch.zeros(p.shape[0], p.shape[1], nb, nb, bs, bs, dtype=torch.float64, device="cuda")
    out[:, :, i, j] = p.double()
    return out.permute(0, 1, 2, 4, 3, 5).reshape(p.shape[0], p.shape[1], nb * bs, nb * bs)


def _heads(x):
    return x.double().permute(0, 2, 1, 3)


@pytest.mark.parametrize("dtype", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("bs,d,nb", [(32, 128, 9), (32, 64, 7), (32, 32, 5), (32, 40, 3), (64, 128, 5), (64, 64, 4), (64, 32, 3), (64, 72, 2), (32, 30, 2)])
def test_products_against_64_bits(sfb, bs, d, nb, dtype):
    if dtype != "f32" and bs == 64 and d == 64:
        pytest.skip("taken by the tcgen05 kernels")
    lay, keep = _layout(sfb, nb, bs, nb + d)
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn(2, nb * bs, 3, d, device="cuda", generator=g).to(TD[dtype]) for _ in range(3))
    Q, K, V = map(_heads, (q, k, v))
    S, A = Q @ K.transpose(-1, -2), Q.abs() @ K.abs().transpose(-1, -2)
    s = sfb.bst_sgemm_nt(q, k, lay, torch.float32)
    assert ((s.double() - _blocks(keep, bs, S)).abs() <= _bound(d) * _blocks(keep, bs, A)).all()
    for pt in ("f32", "bf16", "f16"):
        p = torch.randn(s.shape, device="cuda", generator=g).to(TD[pt])
        P = _dense(keep, bs, p)
        u = EPS if dtype == "f32" else 2.0 ** -8 if dtype == "bf16" else 2.0 ** -11
        for M, got in ((P, sfb.bst_sgemm_xn(p, v, lay)), (P.transpose(-1, -2), sfb.bst_sgemm_tn(p, v, lay))):
            want, size = M @ V, M.abs() @ V.abs()
            assert ((_heads(got) - want).abs() <= _spmm_bound(nb * bs, pt) * size + u * want.abs() + (2.0 ** -25 if dtype == "f16" else 0)).all()
    scale = 1 / math.sqrt(d)
    full = torch.from_numpy(np.kron(keep, np.ones((bs, bs), bool))).cuda()
    W = torch.softmax((S * scale).masked_fill(~full, -math.inf), -1)
    want, size = W @ V, W @ V.abs()
    # a score off by e moves its probability by e of it; ex2.approx and its argument: 2^-22 and the argument's rounding
    off = (_bound(d) * A * scale + (S * scale).abs() * 4 * EPS + 2.0 ** -21).masked_fill(~full, 0)
    err = (W * off) @ V.abs() + off.amax(-1, keepdim=True) * size + _bound(nb * bs) * size + u * want.abs()
    assert ((_heads(sfb.fused_attention(q, k, v, lay, scale)) - want).abs() <= err).all()
    if d in (32, 64, 128):
        rowptr, colidx = sfb.csr_from_layout(lay)
        got = _heads(sfb.csr_attention(q, k, v, rowptr, colidx, scale)[0])
        # the denominator's 1e-6; 16-bit tiles keep P to 16 (bf16) or 22 (fp16) bits and add their products on the tensor core, truncated
        extra = 2e-6 + (0 if dtype == "f32" else nb * bs * 2 * EPS + (2.0 ** -16 if dtype == "bf16" else 2.0 ** -22))
        assert ((got - want).abs() <= err + extra * size + (2.0 ** -25 if dtype == "f16" else 0)).all()


def _same(got, want, tol):
    """Finite where `want` is and close there (tol: of the value, or absolute below 1); the same infinities and NaN elsewhere."""
    fin = torch.isfinite(want)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(got[~fin & ~torch.isnan(want)], want[~fin & ~torch.isnan(want)])
    assert ((got[fin] - want[fin]).abs() <= tol * want[fin].abs().clamp_min(1)).all()


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("bs,d", [(32, 64), (64, 128)])
@pytest.mark.parametrize("value", [math.inf, -math.inf, math.nan, 3.4e38])
def test_values_that_are_not_finite_or_nearly(sfb, bs, d, value, dtype):
    if dtype == "f16" and value == 3.4e38:
        pytest.skip("not an fp16 number")
    nb = 4
    lay, keep = _layout(sfb, nb, bs, 1)
    g = torch.Generator(device="cuda").manual_seed(4)
    q, k, v = (torch.randn(1, nb * bs, 2, d, device="cuda", generator=g).to(TD[dtype]) for _ in range(3))
    q = q.where(q.abs() > 1e-2, torch.ones_like(q))
    k[0, 5, 0, 3] = value
    q[0, 2 * bs + 1, 1] = 0
    q[0, 2 * bs + 1, 1, 0] = 0.5
    k[0, bs + 2, 1, 0] = value
    full = torch.from_numpy(np.kron(keep, np.ones((bs, bs), bool))).cuda()
    S32 = (q.float().permute(0, 2, 1, 3)[..., None, :] * k.float().permute(0, 2, 1, 3)[:, :, None]).sum(-1)     # element by element: inf * 0 is NaN
    _same(sfb.bst_sgemm_nt(q, k, lay, torch.float32), _blocks(keep, bs, S32), 1e-4)
    # a score of -inf is a probability of 0, one of +inf or NaN a row of NaN
    scale = 1 / math.sqrt(d)
    W = torch.softmax((S32.double() * scale).masked_fill(~full, -math.inf), -1)
    want = (W @ v.double().permute(0, 2, 1, 3)).permute(0, 2, 1, 3).float()
    rowptr, colidx = sfb.csr_from_layout(lay)
    tol = 1e-5 if dtype == "f32" else 2.0 ** -9
    _same(sfb.fused_attention(q, k, v, lay, scale).float(), want, tol)
    _same(sfb.csr_attention(q, k, v, rowptr, colidx, scale)[0].float(), want, tol)
    # one value: the rows that keep its block, and no other
    k = torch.randn(k.shape, device="cuda", generator=g).to(TD[dtype])
    v[0, bs + 3, 1, d - 1] = value
    p = torch.rand(1, 2, int(keep.sum()), bs, bs, device="cuda", generator=g).add(0.01).to(torch.bfloat16)
    M = _dense(keep, bs, p).float()
    want = torch.where(full[None, None, :, :, None], M[..., None] * v.float().permute(0, 2, 1, 3)[:, :, None], torch.zeros((), device="cuda")).sum(3).permute(0, 2, 1, 3)
    none = torch.zeros((), device="cuda")
    V = v.float().permute(0, 2, 1, 3)[:, :, None]
    wantT = torch.where(full.T[None, None, :, :, None], M.transpose(-1, -2)[..., None] * V, none).sum(3).permute(0, 2, 1, 3)
    for pt in (p.to(TD[dtype]), p):                          # fp32 blocks go by FMAs, others as split products
        for got, ref in ((sfb.bst_sgemm_xn(pt, v, lay).float(), want), (sfb.bst_sgemm_tn(pt, v, lay).float(), wantT)):
            if dtype == "f16":
                assert torch.equal(torch.isfinite(got), torch.isfinite(ref))
            else:
                _same(got, ref, 1e-4)
    W = torch.softmax((_heads(q) @ _heads(k).transpose(-1, -2) * scale).masked_fill(~full, -math.inf), -1)
    want = torch.where(full[None, None, :, :, None], W[..., None] * V.double(), none.double()).sum(3).permute(0, 2, 1, 3).float()
    touched = torch.zeros_like(want, dtype=torch.bool)
    touched[0, :, 1, d - 1] = full[:, bs + 3]
    for o in (sfb.fused_attention(q, k, v, lay, scale).float(), sfb.csr_attention(q, k, v, rowptr, colidx, scale)[0].float()):
        _same(o[~touched], want[~touched], tol)
        _same(o[touched], want[touched], 1e-5)


def test_a_row_of_scores_that_are_not_numbers_is_not_a_row_of_zeros(sfb):
    lay = sfb.BlockLayout.generate(sfb.LAYOUT_FULL, 1, 2, 32)
    q, k, v = (torch.ones(1, 64, 1, 32, device="cuda") for _ in range(3))
    q[0, 7, 0, 0] = math.nan
    o = sfb.fused_attention(q, k, v, lay, 0.1)
    assert torch.isnan(o[0, 7]).all() and torch.isfinite(o[0, :7]).all() and torch.isfinite(o[0, 8:]).all()


def _us(f):
    times = []
    for _ in range(7):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        f()
        a.record()
        for _ in range(5):
            f()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b))
    return min(times)


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("bs,d", [(32, 128), (32, 64), (64, 128)])
def test_what_is_not_finite_does_not_set_the_time(sfb, bs, d, dtype):
    """An overflowed gradient or an infinite key must not make a call much longer: every result, or every row, is made again, and the
    call takes at most eight times what it takes on finite operands (two to five, measured; made again one by one, 7 to 70)."""
    lay = sfb.BlockLayout.generate(sfb.LAYOUT_SAWTOOTH, 1, 1024 // bs, bs, p0=8)
    lay.tn_lut
    g = torch.Generator(device="cuda").manual_seed(6)
    q, k, v = (torch.randn(8, 1024, 4, d, device="cuda", generator=g).to(TD[dtype]) for _ in range(3))
    p = torch.rand(8, 4, lay.blocks, bs, bs, device="cuda", generator=g).to(torch.bfloat16 if dtype == "f32" else TD[dtype])
    bad, key = torch.full_like(v, math.nan), k.clone()
    key[:, ::64, :, 3] = math.inf                            # in every row of blocks
    scale = 1 / math.sqrt(d)
    assert _us(lambda: sfb.bst_sgemm_nt(q, bad, lay, torch.float32)) <= 8 * _us(lambda: sfb.bst_sgemm_nt(q, k, lay, torch.float32))
    assert _us(lambda: sfb.bst_sgemm_xn(p, bad, lay)) <= 8 * _us(lambda: sfb.bst_sgemm_xn(p, v, lay))
    assert _us(lambda: sfb.bst_sgemm_tn(p, bad, lay)) <= 8 * _us(lambda: sfb.bst_sgemm_tn(p, v, lay))
    assert _us(lambda: sfb.fused_attention(q, key, v, lay, scale)) <= 8 * _us(lambda: sfb.fused_attention(q, k, v, lay, scale))


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("bs,d", [(32, 128), (32, 64), (32, 32), (32, 30), (64, 128), (64, 72), (64, 32)])
def test_rows_made_again(sfb, bs, d, dtype):
    """Infinities in several places of the keys and of the values, rows of 1 to 9 blocks with and without a mask, widths that are no
    multiple of a unit: what is not finite is what fp32 arithmetic gives, and what meets no infinity is bit for bit what it is without."""
    nb = 9
    lay, keep = _layout(sfb, nb, bs, d)
    lay.pack_mask(sfb.MASK_CAUSAL_DIAG)
    g = torch.Generator(device="cuda").manual_seed(7)
    q, k, v = (torch.randn(2, nb * bs, 3, d, device="cuda", generator=g).to(TD[dtype]) for _ in range(3))
    q, v = (x.where(x.abs() > 1e-2, torch.ones_like(x)) for x in (q, v))
    full = torch.from_numpy(np.kron(keep, np.ones((bs, bs), bool))).cuda()
    scale = 1 / math.sqrt(d)
    bad = k.clone()
    for j in range(nb):
        bad[:, j * bs + 3 * j + 1, :, (5 * j) % d] = math.inf if j % 2 else -math.inf
    S = torch.einsum("blhd,bmhd->bhlm", q.double(), bad.double())        # one infinity per key: no inf - inf
    assert not torch.isnan(S).any()
    _same(sfb.bst_sgemm_nt(q, bad, lay, torch.float32), _blocks(keep, bs, S.float()), 1e-4)
    inside = torch.ones(nb * bs, nb * bs, dtype=torch.bool, device="cuda")
    for i in range(nb):
        inside[i * bs:(i + 1) * bs, i * bs:(i + 1) * bs] = torch.ones(bs, bs, device="cuda").tril().bool()
    for use_mask in (False, True):
        W = torch.softmax((S * scale).masked_fill(~(full & inside if use_mask else full), -math.inf), -1)
        want = torch.einsum("bhlm,bmhd->blhd", W, v.double()).float()
        _same(sfb.fused_attention(q, bad, v, lay, scale, use_mask=use_mask).float(), want, 1e-5 if dtype == "f32" else 2.0 ** -9)
    p = torch.rand(2, 3, lay.blocks, bs, bs, device="cuda", generator=g).clamp_min(1e-2).to(torch.bfloat16 if dtype == "f32" else TD[dtype])
    badv, hit = v.clone(), torch.zeros(nb * bs, d, dtype=torch.float64, device="cuda")
    for j in range(0, nb, 2):
        badv[:, j * bs + 2 * j, :, (7 * j) % d] = math.inf
        hit[j * bs + 2 * j, (7 * j) % d] = 1
    for rows, f in ((full, sfb.bst_sgemm_xn), (full.T, sfb.bst_sgemm_tn)):
        got, clean = (f(p, x, lay).permute(0, 2, 1, 3) for x in (badv, v))
        met = rows.double() @ hit > 0
        assert (got[:, :, met] == math.inf).all()
        assert torch.equal(got[:, :, ~met], clean[:, :, ~met])


@pytest.mark.parametrize("bs,d", [(32, 128), (32, 64), (64, 64)])
@pytest.mark.parametrize("below", [100, 126, 127, 130, 132])
def test_weights_that_are_subnormal(sfb, bs, d, below):
    """A key whose weight is 2^-below of the row's largest, with the only values of its columns: subnormal weights count, as far as the
    terms of a product do (multiples of 2^-133)."""
    L = 4 * bs
    lay = sfb.BlockLayout.generate(sfb.LAYOUT_FULL, 1, 4, bs)
    q, k, v = (torch.zeros(1, L, 1, d, device="cuda") for _ in range(3))
    q[..., 0] = 1
    k[:, :, 0, 0] = -1000                                    # weights of 0
    k[:, 5, 0, 0] = 0
    k[:, L - 3, 0, 0] = -below
    v[:, L - 3, 0, : d // 2] = 2.0 ** 100
    v[:, 5, 0, d // 2:] = 1
    want = torch.cat([torch.full((d // 2,), 2.0 ** (100 - below)), torch.ones(d - d // 2)]).cuda()
    # score * scale is off by 2^-24 of itself, twice (the scale in units of log2), and ex2 by 2^-22
    tol = 2 * below * EPS + 2.0 ** -21
    rowptr, colidx = sfb.csr_from_layout(lay)
    for o in (sfb.fused_attention(q, k, v, lay, math.log(2)), sfb.csr_attention(q, k, v, rowptr, colidx, math.log(2))[0] * (1 + 1e-6)):
        assert ((o[0, :, 0] - want).abs() <= tol * want + (2.0 ** (100 - 134) if below > 109 else 0) * (want < 1)).all()
        assert (o[0, :, 0] > 0).all()


@pytest.mark.parametrize("down", [100, 109, 112, 118, 124])
def test_small_operands(sfb, down):
    """What is left of an operand below 2^-109 is a multiple of 2^-133, the last place of the smallest bf16 numbers: its products are
    off by up to 2^-134 of the other operand on top of what larger ones are."""
    bs, d, nb = 32, 64, 4
    lay, keep = _layout(sfb, nb, bs, 2)
    g = torch.Generator(device="cuda").manual_seed(9)
    q, k, v = (torch.randn(1, nb * bs, 2, d, device="cuda", generator=g) for _ in range(3))
    q, v = q * 2.0 ** -down, v * 2.0 ** -down
    Q, K, V = map(_heads, (q, k, v))
    S, A, lost = Q @ K.transpose(-1, -2), Q.abs() @ K.abs().transpose(-1, -2), torch.ones_like(Q) @ K.abs().transpose(-1, -2) * 2.0 ** -134
    s = sfb.bst_sgemm_nt(q, k, lay, torch.float32)
    assert ((s.double() - _blocks(keep, bs, S)).abs() <= _blocks(keep, bs, _bound(d) * A + lost)).all()
    p = torch.randn(1, 2, lay.blocks, bs, bs, device="cuda", generator=g).to(torch.bfloat16)
    P = _dense(keep, bs, p)
    for M, got in ((P, sfb.bst_sgemm_xn(p, v, lay)), (P.transpose(-1, -2), sfb.bst_sgemm_tn(p, v, lay))):
        assert ((_heads(got) - M @ V).abs() <= _bound(nb * bs) * (M.abs() @ V.abs()) + 2.0 ** -134 * (M.abs() @ torch.ones_like(V))).all()


def _attention64(q, k, v, keep, scale):
    """Outputs [B, H, L, d] in 64 bits and the error that scores and exponentials of fp32 leave in them."""
    d, n = q.shape[3], k.shape[1]
    Q, K, V = map(_heads, (q, k, v))
    S, A = Q @ K.transpose(-1, -2) * scale, Q.abs() @ K.abs().transpose(-1, -2) * scale
    W = torch.softmax(S.masked_fill(~keep, -math.inf), -1).nan_to_num(0)
    size = W @ V.abs()
    off = (_bound(d) * A + S.abs() * 4 * EPS + 2.0 ** -21).masked_fill(~keep, 0)
    return W @ V, (W * off) @ V.abs() + off.amax(-1, keepdim=True) * size + _bound(n) * size


@pytest.mark.parametrize("dtype", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("bs,d", [(32, 32), (32, 64), (32, 128), (64, 32), (64, 64), (64, 128)])
def test_attention_launches_of_more_than_one_wave(sfb, bs, d, dtype):
    """More CTAs than the SMs hold at once (up to three each): the kernels with short rings.  Against 64 bits with and without a mask,
    bit for bit what a slice of one head gives (the kernels with long rings), and with a key that is not finite."""
    if dtype != "f32" and bs == 64 and d == 64:
        pytest.skip("taken by the tcgen05 kernels")
    nb = 7
    B = 3 * torch.cuda.get_device_properties(0).multi_processor_count // (2 * nb) + 1
    lay, keep = _layout(sfb, nb, bs, bs + d)
    lay.pack_mask(sfb.MASK_CAUSAL_DIAG)
    g = torch.Generator(device="cuda").manual_seed(12)
    q, k, v = (torch.randn(B, nb * bs, 2, d, device="cuda", generator=g).to(TD[dtype]) for _ in range(3))
    full = torch.from_numpy(np.kron(keep, np.ones((bs, bs), bool))).cuda()
    tril = torch.ones(bs, bs, device="cuda").tril().bool()
    u = EPS if dtype == "f32" else 2.0 ** -8 if dtype == "bf16" else 2.0 ** -11
    scale = 1 / math.sqrt(d)
    for use_mask in (False, True):
        if use_mask:
            for i in range(nb):
                full[i * bs:(i + 1) * bs, i * bs:(i + 1) * bs] &= tril
        want, err = _attention64(q, k, v, full, scale)
        o = sfb.fused_attention(q, k, v, lay, scale, use_mask=use_mask)
        assert ((_heads(o) - want).abs() <= err + u * want.abs() + (2.0 ** -25 if dtype == "f16" else 0)).all()
        for b in (0, B // 2, B - 1):
            part = sfb.fused_attention_slice(q[b:b + 1, :, 1:], k[b:b + 1, :, 1:], v[b:b + 1, :, 1:], lay, scale, use_mask=use_mask)
            assert torch.equal(part, o[b:b + 1, :, 1:])
    bad = k.clone()
    bad[B // 2, bs + 5, 1, 3] = math.nan
    again = sfb.fused_attention(q, bad, v, lay, scale, use_mask=True)
    met = torch.zeros(o.shape[:3], dtype=torch.bool, device="cuda")
    met[B // 2, :, 1] = full[:, bs + 5]
    assert met.any() and torch.isnan(again[met]).all() and torch.equal(again[~met], o[~met])


@pytest.mark.parametrize("dtype", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("d,B", [(64, 1), (128, 1), (32, 1), (64, 5)])
def test_rows_longer_than_the_lanes(sfb, d, B, dtype):
    """A row's entries are held one per lane, 32 at a time: rows (and columns) of 31 to 97 blocks in no regular order."""
    nb, bs, H = 104, 32, 1
    rng = np.random.RandomState(d)
    keep = np.zeros((nb, nb), bool)
    for i, n in enumerate((31, 32, 33, 64, 65, 97, 1, 0)):
        keep[11 * i, rng.choice(nb, size=n, replace=False)] = True
    lay, layT = (sfb.BlockLayout(torch.from_numpy(np.ascontiguousarray(x)[None].astype(np.uint8)).cuda(), bs) for x in (keep, keep.T))
    g = torch.Generator(device="cuda").manual_seed(13)
    q, k, v = (torch.randn(B, nb * bs, H, d, device="cuda", generator=g).to(TD[dtype]) for _ in range(3))
    u, floor = (EPS if dtype == "f32" else 2.0 ** -8 if dtype == "bf16" else 2.0 ** -11), (2.0 ** -25 if dtype == "f16" else 0)
    rows = torch.arange(nb * bs, device="cuda").reshape(nb, bs)[::11][:8].reshape(-1)          # of the block-rows above
    V = _heads(v)
    # the blocks in the transposed layout's order
    at = np.zeros((nb, nb), np.int64)
    at[np.nonzero(keep)] = np.arange(lay.blocks)
    i, j = np.nonzero(keep.T)
    order = torch.from_numpy(at[j, i]).cuda()
    for pt in ("f32", "bf16"):
        p = torch.randn(B, H, lay.blocks, bs, bs, device="cuda", generator=g).to(TD[pt])
        M = _dense(keep, bs, p)
        want, size = M @ V, M.abs() @ V.abs()
        for got in (sfb.bst_sgemm_xn(p, v, lay), sfb.bst_sgemm_tn(p[:, :, order].transpose(-1, -2).contiguous(), v, layT)):
            assert ((_heads(got) - want).abs() <= _spmm_bound(97 * bs, pt) * size + u * want.abs() + floor).all()
    lay.pack_mask(sfb.MASK_CAUSAL_DIAG)
    full = torch.from_numpy(np.kron(keep, np.ones((bs, bs), bool))).cuda()[rows]
    rest = torch.ones(nb * bs, dtype=torch.bool, device="cuda")
    rest[rows] = False
    scale = 1 / math.sqrt(d)
    for use_mask in (False, True):
        if use_mask:
            for n in range(8):
                full[n * bs:(n + 1) * bs, 11 * n * bs:(11 * n + 1) * bs] &= torch.ones(bs, bs, device="cuda").tril().bool()
        want, err = _attention64(q[:, rows], k, v, full, scale)
        o = _heads(sfb.fused_attention(q, k, v, lay, scale, use_mask=use_mask))
        assert ((o[:, :, rows] - want).abs() <= err + u * want.abs() + floor).all()
        assert (o[:, :, rest] == 0).all()
