"""GPU parity of the element-sparse (CSR) attention path against the CPU oracle, and against the block-sparse path on
patterns both can express.  Tolerances: pattern arrays bit-exact; fp32 outputs max-abs 1e-5; 16-bit 2e-2 relative."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TD = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}


@pytest.mark.parametrize("kind,kw,dev,nb,bs", [
    ("stride", dict(band=2, every=4), ("LAYOUT_STRIDE", dict(p0=2, p1=4)), 8, 32),
    ("local", dict(left=1, right=1), ("LAYOUT_LOCAL", dict(p0=1, p1=1)), 5, 64),
    ("full", dict(causal=1), ("LAYOUT_FULL", dict(causal=1)), 4, 32),
])
def test_csr_pattern_from_layout_bit_exact(sfb, oracle, kind, kw, dev, nb, bs):
    lay = sfb.BlockLayout.generate(getattr(sfb, dev[0]), 1, nb, bs, **dev[1])
    rowptr, colidx = sfb.csr_from_layout(lay)
    wr, wc = oracle.csr_from_layout(oracle.layout(kind, 1, nb, **kw)[0], bs)
    assert np.array_equal(rowptr.cpu().numpy(), wr) and np.array_equal(colidx.cpu().numpy(), wc)


@pytest.mark.parametrize("dtype,d", [("f32", 64), ("f32", 32), ("bf16", 64), ("f16", 128)])
def test_csr_attention_against_oracle_on_an_irregular_pattern(sfb, oracle, dtype, d):
    """Rows of very different lengths, one empty row, unsorted columns."""
    B, L, H = 2, 200, 3
    rng = np.random.RandomState(5)
    rows = []
    for i in range(L):
        n = 0 if i == 7 else int(rng.randint(1, 90 if i % 5 else 200))
        rows.append(rng.choice(L, size=n, replace=False).astype(np.int32))
    rowptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    colidx = np.concatenate(rows).astype(np.int32)
    q, k, v = (torch.from_numpy(oracle.fill_normal((B, L, H, d), 500 + i)).cuda().to(TD[dtype]) for i in range(3))
    o, bad = sfb.csr_attention(q, k, v, torch.from_numpy(rowptr).cuda(), torch.from_numpy(colidx).cuda(), 0.125)
    assert int(bad.item()) == 0
    want = oracle.csr_attention(q.float().cpu().numpy(), k.float().cpu().numpy(), v.float().cpu().numpy(), rowptr, colidx, np.float32(0.125))
    got = o.float().cpu().numpy()
    if dtype == "f32":
        assert np.abs(got - want).max() < 1e-5
    else:
        assert np.abs(got - want).max() <= 2e-2 * np.abs(want).max()
    assert float(np.abs(got[:, 7]).max()) == 0.0


def test_csr_attention_equals_block_sparse_attention(sfb, oracle):
    """The same pattern through both formats: CSR of a block layout against the fused block-sparse kernel."""
    B, H, d, bs, nb = 2, 4, 64, 64, 16
    lay = sfb.BlockLayout.generate(sfb.LAYOUT_STRIDE, 1, nb, bs, p0=4, p1=8)
    rowptr, colidx = sfb.csr_from_layout(lay)
    q, k, v = (torch.from_numpy(oracle.fill_normal((B, nb * bs, H, d), 510 + i)).cuda() for i in range(3))
    a, _ = sfb.csr_attention(q, k, v, rowptr, colidx, 0.125)
    b = sfb.fused_attention(q, k, v, lay, 0.125)
    assert float((a - b).abs().max()) < 2e-5


def test_csr_columns_outside_the_sequence_are_counted_not_read(sfb):
    L, d = 8, 32
    q = torch.ones(1, L, 1, d, device="cuda")
    rowptr = torch.arange(0, 2 * L + 1, 2, dtype=torch.int32, device="cuda")
    colidx = torch.tensor([0, 1] * L, dtype=torch.int32, device="cuda")
    colidx[3], colidx[10] = -5, L
    o, bad = sfb.csr_attention(q, q, q, rowptr, colidx, 1.0)
    assert int(bad.item()) == 2
    assert torch.allclose(o, torch.ones_like(o), atol=1e-4)


@pytest.mark.parametrize("dtype", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("L,d", [(1, 64), (31, 32), (33, 128), (64, 64), (517, 64), (530, 128), (545, 32)])
def test_csr_tiles_against_oracle(sfb, oracle, dtype, L, d):
    """Tiles of 32 rows: a single row, ragged last tiles, lists shorter and longer than a chunk, rows that name a column
    twice (it counts twice), an empty tile, and the call without a workspace."""
    B, H = 2, 2
    rng = np.random.RandomState(L)
    rows = []
    for i in range(L):
        n = 0 if 96 <= i < 128 else int(rng.randint(0, min(L, 300) + 1))
        r = rng.choice(L, size=n, replace=False)
        if n and i % 4 == 0:
            r = np.r_[r, r[:3]]
        rows.append(r.astype(np.int32))
    rows[0] = np.array([0], np.int32)
    rowptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    colidx = np.concatenate(rows).astype(np.int32)
    q, k, v = (torch.from_numpy(oracle.fill_normal((B, L, H, d), 530 + i)).cuda().to(TD[dtype]) for i in range(3))
    rp, ci = torch.from_numpy(rowptr).cuda(), torch.from_numpy(colidx).cuda()
    o, bad = sfb.csr_attention(q, k, v, rp, ci, 0.125)
    assert int(bad.item()) == 0
    plain = torch.empty_like(q)
    p = lambda t: sfb.C.c_void_p(t.data_ptr())
    sfb._check(sfb.lib.sfb_csr_attention(sfb._stream(), p(rp), p(ci), p(q), p(k), p(v), p(plain), sfb.dtype_tag(q), B, L, H, d, 0.125, p(bad)))
    want = oracle.csr_attention(q.float().cpu().numpy(), k.float().cpu().numpy(), v.float().cpu().numpy(), rowptr, colidx, np.float32(0.125))
    for got in (o, plain):
        assert np.abs(got.float().cpu().numpy() - want).max() <= (1e-5 if dtype == "f32" else 2e-2 * np.abs(want).max())
    if dtype != "f32":   # 16-bit outputs of the two agree to their last bit nearly everywhere: nothing between them is rounded more
        assert float((o != plain).float().mean()) < 0.02


def test_csr_bad_columns_are_counted_per_batch_and_head(sfb):
    L, d = 70, 64
    q = torch.ones(2, L, 3, d, device="cuda", dtype=torch.bfloat16)
    rowptr = torch.arange(0, 2 * L + 1, 2, dtype=torch.int32, device="cuda")
    colidx = torch.tensor([0, 1] * L, dtype=torch.int32, device="cuda")
    colidx[3], colidx[100], colidx[139] = -5, L, 1 << 30
    o, bad = sfb.csr_attention(q, q, q, rowptr, colidx, 1.0)
    assert int(bad.item()) == 3 * 2 * 3
    assert torch.equal(o, q)


@pytest.mark.parametrize("upper,lower,both", [(0, 0, 40), (37, 0, 0), (0, 5, 0), (16, 16, 16), (3, 70, 1), (50, 1, 33)])
@pytest.mark.parametrize("twice", [False, True])
def test_csr_columns_of_half_a_tile(sfb, oracle, upper, lower, both, twice):
    """Tiles whose columns belong to the first 16 rows, to the last 16, or to both, in any proportion, with and without
    columns named twice, at the head width whose warps work for half a tile each."""
    L, d = 128, 128
    rng = np.random.RandomState(upper + lower)
    rows = []
    for t in range(L // 32):
        cols = rng.permutation(L)[:upper + lower + both]
        u, w, b = np.split(cols, [upper, upper + lower])
        for r in range(32):
            c = np.r_[u if r < 16 else w, b]
            c = c[rng.rand(len(c)) < (1.0 if r % 16 == 3 else 0.3)]
            rows.append(np.r_[c, c[:1] if twice and r % 8 == 3 else []].astype(np.int32))
    rowptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    colidx = np.concatenate(rows).astype(np.int32)
    q, k, v = (torch.from_numpy(oracle.fill_normal((1, L, 2, d), 640 + i)).cuda().to(torch.bfloat16) for i in range(3))
    o, bad = sfb.csr_attention(q, k, v, torch.from_numpy(rowptr).cuda(), torch.from_numpy(colidx).cuda(), 0.125)
    want = oracle.csr_attention(q.float().cpu().numpy(), k.float().cpu().numpy(), v.float().cpu().numpy(), rowptr, colidx, np.float32(0.125))
    assert int(bad.item()) == 0
    assert np.abs(o.float().cpu().numpy() - want).max() <= 2e-2 * np.abs(want).max()


def _random_rows(L, seed, most=60):
    rng = np.random.RandomState(seed)
    rows = [rng.choice(L, size=0 if 32 <= i < 40 else int(rng.randint(1, min(L, most) + 1)), replace=False).astype(np.int32) for i in range(L)]
    return rows, np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32), np.concatenate(rows).astype(np.int32)


@pytest.mark.parametrize("dtype", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("d", [32, 64, 128])
def test_csr_nan_query_gives_nan(sfb, dtype, d):
    """A query with a NaN has a NaN for every output, and no other row has one."""
    L, bad_row = 100, 70
    _, rowptr, colidx = _random_rows(L, 9)
    gen = torch.Generator(device="cuda").manual_seed(90)
    q, k, v = (torch.randn(1, L, 1, d, device="cuda", generator=gen).to(TD[dtype]) for _ in range(3))
    q[0, bad_row, 0, 5] = float("nan")
    o, _ = sfb.csr_attention(q, k, v, torch.from_numpy(rowptr).cuda(), torch.from_numpy(colidx).cuda(), 0.125)
    want = torch.zeros(L, d, dtype=torch.bool)
    want[bad_row] = True
    assert torch.equal(torch.isnan(o[0, :, 0]).cpu(), want)


@pytest.mark.parametrize("dtype", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("value", ["nan", "inf", "-inf"])
def test_csr_values_that_are_not_finite_stay_in_the_rows_that_have_them(sfb, oracle, dtype, d, value):
    """An infinity or a NaN among the values of a column reaches the rows that have the column, in that element, and no other:
    rows of the same tile are as they are without it.  Also in a column of its own that nobody has, in tiles of one row and
    in rows without elements."""
    B, L, H = 2, 193, 2                                      # the last tile has one row
    rows, rowptr, colidx = _random_rows(L, 11)
    cols = [3, 77, 192]
    nobody = [c for c in range(L) if not any(c in r for r in rows)]
    q, k, v = (torch.from_numpy(oracle.fill_normal((B, L, H, d), 700 + i)).cuda().to(TD[dtype]) for i in range(3))
    rp, ci = torch.from_numpy(rowptr).cuda(), torch.from_numpy(colidx).cuda()
    clean = sfb.csr_attention(q, k, v, rp, ci, 0.125)[0].float().cpu().numpy()
    dirty = v.clone()
    for n, c in enumerate(cols + nobody[:2]):
        dirty[:, c, :, (5 * n) % d] = float(value)
    got = sfb.csr_attention(q, k, dirty, rp, ci, 0.125)[0].float().cpu().numpy()
    has = np.zeros((L, d), bool)                             # elements of the output that one of the values belongs to
    for n, c in enumerate(cols):
        for i, r in enumerate(rows):
            has[i, (5 * n) % d] |= c in r
    assert has.any() and np.array_equal(~np.isfinite(got), np.broadcast_to(has[None, :, None], got.shape))
    keep = ~np.broadcast_to(has[None, :, None], got.shape)
    # two sums in a different order, rounded to the type of the output
    assert np.abs(got - clean)[keep].max() <= (1e-5 if dtype == "f32" else 2.0 ** -7) * np.abs(clean).max()


@pytest.mark.parametrize("dtype", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("what", ["inf", "-inf", "product"])
@pytest.mark.parametrize("scale", [0.125, -0.125])
def test_csr_keys_that_are_not_finite(sfb, dtype, d, what, scale):
    """A score that the scale makes -inf is a probability of 0 wherever in its row the column stands, among the first that a warp
    takes or behind them; one that it makes +inf gives NaN in the rows that have the column and in no other.
    what: the key's element, or `product`: finite operands whose product overflows fp32."""
    if what == "product" and dtype == "f16":
        pytest.skip("no product of fp16 numbers overflows fp32")
    L = 160
    gen = torch.Generator(device="cuda").manual_seed(60 + d)
    q, k, v = (torch.randn(1, L, 2, d, device="cuda", generator=gen).to(TD[dtype]) for _ in range(3))
    # rows of 1 to 97 columns, the bad one first, in place i, or last
    rng = np.random.RandomState(d)
    bad, rows = 5, []
    for i in range(L):
        r = rng.choice(np.delete(np.arange(L), bad), size=i % 97, replace=False)
        rows.append(np.insert(r, {0: 0, 1: min(i, len(r)), 2: len(r)}[i % 3], bad) if i % 4 else r)
    rowptr = torch.from_numpy(np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)).cuda()
    colidx = torch.from_numpy(np.concatenate(rows).astype(np.int32)).cuda()
    if what == "product":
        q[..., 3] = -2.0 ** 70
        k[..., 3] = 0
        k[0, bad, :, 3] = 2.0 ** 70
        sign = -1
    else:
        q[..., 3] = q[..., 3].abs() + 1
        k[0, bad, :, 3] = float(what)
        sign = 1 if what == "inf" else -1
    has = torch.zeros(L, L, device="cuda")
    has.index_put_((torch.repeat_interleave(torch.arange(L, device="cuda"), (rowptr[1:] - rowptr[:-1]).long()), colidx.long()), torch.ones((), device="cuda"), accumulate=True)
    keep = has.clone()
    keep[:, bad] = 0                                         # what the rows are without it
    S = torch.einsum("blhd,bmhd->bhlm", q.double(), k.double().nan_to_num(0, 0, 0)) * scale
    W = torch.softmax(S.masked_fill(keep == 0, -np.inf), -1).nan_to_num(0)
    want = torch.einsum("bhlm,bmhd->blhd", W, v.double())
    got = sfb.csr_attention(q, k, v, rowptr, colidx, scale)[0].double()
    plain = torch.empty_like(q)
    p = lambda t: sfb.C.c_void_p(t.data_ptr())
    n = torch.zeros(1, dtype=torch.int32, device="cuda")
    sfb._check(sfb.lib.sfb_csr_attention(sfb._stream(), p(rowptr), p(colidx), p(q), p(k), p(v), p(plain), sfb.dtype_tag(q), 1, L, 2, d, scale, p(n)))
    nan = torch.zeros(L, dtype=torch.bool, device="cuda") if sign * scale < 0 else has[:, bad] > 0
    for o in (got, plain.double()):
        assert torch.equal(torch.isnan(o), nan[None, :, None, None].expand_as(o))
        diff = (o - want)[:, ~nan].abs().max()
        assert diff <= (1e-5 if dtype == "f32" else 2.0 ** -7) * want.abs().max()


@pytest.mark.parametrize("dtype", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("L", [545, 1024])
def test_csr_scores_that_rise_and_fall(sfb, dtype, d, L):
    """The reference maximum of a row moves only when a score outgrows it by 2^8 (16-bit tiles): scores that rise or fall along the row by
    little, by a little less and a little more than 8 (log2) from one of a warp's chunks to its next, and by far more, row by row
    in the same tile, so that some rows of a tile rescale where others must not, and warps meet with very different maxima."""
    gen = torch.Generator(device="cuda").manual_seed(L + d)
    q, k, v = (0.25 * torch.randn(1, L, 2, d, device="cuda", generator=gen) for _ in range(3))
    v *= 4
    scale = 0.125
    # how many columns a warp's chunk and its next are apart, and by what their scores differ then
    apart = 32 if d == 128 else 128 if d == 32 else 64
    slopes = torch.tensor([0.5, 3, 7.75, 8.25, 20, 60, -0.5, -3, -7.75, -8.25, -20, -60], device="cuda")
    q[..., 0] = (slopes / (apart / 16 * scale * 1.4427))[torch.arange(L, device="cuda") % 12][None, :, None]
    q[..., 1] = q[..., 0] / 16
    j = torch.arange(L, device="cuda")
    k[..., 0], k[..., 1] = (j // 16).float()[None, :, None], (j % 16).float()[None, :, None]
    q, k, v = (x.to(TD[dtype]) for x in (q, k, v))
    keep = torch.rand(L, L, device="cuda", generator=gen) < 0.7
    keep[:, 0] = True
    rowptr = torch.zeros(L + 1, dtype=torch.int32, device="cuda")
    rowptr[1:] = keep.sum(1).cumsum(0)
    got = sfb.csr_attention(q, k, v, rowptr, keep.nonzero()[:, 1].to(torch.int32).contiguous(), scale)[0].double()
    Q, K, V = (x.double().permute(0, 2, 1, 3) for x in (q, k, v))
    S, A = Q @ K.transpose(-1, -2) * scale, Q.abs() @ K.abs().transpose(-1, -2) * scale
    W = torch.softmax(S.masked_fill(~keep, -np.inf), -1)
    want, size = (W @ V).permute(0, 2, 1, 3), (W @ V.abs()).permute(0, 2, 1, 3)
    # a score: fp32 sums of d products, truncated (2^-23 each), and two roundings of the exponent; P: two 16-bit terms
    off = ((d * 2.0 ** -23 + 4 * 2.0 ** -24) * A + 2.0 ** -21).masked_fill(~keep, 0).amax(-1)[..., None].permute(0, 2, 1, 3)
    u = {"f32": 2.0 ** -24, "bf16": 2.0 ** -8, "f16": 2.0 ** -11}[dtype]
    err = (2 * off + 2e-6 + L * 2.0 ** -23 + (2.0 ** -16 if dtype == "bf16" else 2.0 ** -22)) * size + u * want.abs() + (2.0 ** -25 if dtype == "f16" else 0)
    assert ((got - want).abs() <= err).all()
