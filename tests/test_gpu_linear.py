"""GPU parity of the tcgen05 dense projection (sfb_linear, sfb_linear_nt) and of the embedding front end against the CPU oracle.  Tolerance: 16-bit operands with
fp32 accumulation, 2e-2 relative to the largest reference value (the output itself is rounded to 16 bits)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TD = {"bf16": torch.bfloat16, "f16": torch.float16}


def _mk(oracle, shape, seed, dtype, std=1.0):
    t = torch.from_numpy(oracle.fill_normal(shape, seed, std)).cuda().to(TD[dtype])
    return t, t.float().cpu().numpy()


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("m,n,k,act,with_bias", [
    (128, 256, 64, 0, False),        # one tile, one k-block
    (128, 256, 768, 0, True),
    (300, 768, 768, 0, True),        # ragged rows, three column tiles
    (257, 3072, 768, 1, True),       # FFN up-projection with GELU
    (130, 768, 3072, 0, True),       # FFN down-projection: 48 k-blocks
    (64, 48, 40, 1, True),           # smaller than a tile in every direction; k not a multiple of 64
    (1000, 1024, 1024, 0, False),
])
def test_linear_against_oracle(sfb, oracle, dtype, m, n, k, act, with_bias):
    x, xn = _mk(oracle, (m, k), 400, dtype)
    w, wn = _mk(oracle, (k, n), 401, dtype, 0.05)
    b = torch.from_numpy(oracle.fill_normal((n,), 402, 0.5)).cuda() if with_bias else None
    got = sfb.linear(x, w, b, act)
    assert sfb.device_status() == 0
    want = oracle.linear(xn, wn, None if b is None else b.cpu().numpy(), act)
    assert got.shape == (m, n) and got.dtype == TD[dtype]
    assert np.abs(got.float().cpu().numpy() - want).max() <= 2e-2 * np.abs(want).max()


@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("m,n,k,act", [
    (1, 16, 8, 0),                   # the smallest: one row, one column group, an eighth of a k-block
    (129, 80, 72, 1),                # one row and 16 columns into the second tiles
    (64, 192, 520, 1),               # nine k-blocks in one CTA per tile
    (64, 192, 2056, 1),              # 33 k-blocks over four CTAs per tile, one of them with nine
    (320, 768, 3072, 0),             # two CTAs per 128 x 64 tile
    (640, 1040, 4096, 1),            # two CTAs per 128 x 128 tile, the last one 16 columns wide
    (2048, 1024, 1032, 0),           # 128 x 128 tiles, eight elements into the last k-block
])
def test_linear_few_tiles(sfb, oracle, m, n, k, act, transposed):
    x, xn = _mk(oracle, (m, k), 420, "bf16")
    w, wn = _mk(oracle, (n, k) if transposed else (k, n), 421, "bf16", 0.05)
    b = torch.from_numpy(oracle.fill_normal((n,), 422, 0.5)).cuda()
    got = (sfb.linear_nt if transposed else sfb.linear)(x, w, b, act)
    again = (sfb.linear_nt if transposed else sfb.linear)(x, w, b, act)
    assert sfb.device_status() == 0 and torch.equal(got, again)      # the shares of a tile are added in a fixed order
    rows = np.unique(np.r_[np.arange(0, m, 37), m - 1])
    want = oracle.linear(xn[rows], np.ascontiguousarray(wn.T) if transposed else wn, b.cpu().numpy(), act)
    assert np.abs(got[rows].float().cpu().numpy() - want).max() <= 2e-2 * np.abs(want).max()


@pytest.mark.parametrize("m,n,k", [(129, 80, 72), (64, 192, 520), (2048, 1040, 136), (3000, 2320, 64), (20000, 272, 64)])
def test_linear_residual(sfb, m, n, k):
    """The sum in the epilogue (one CTA per tile, several) and as a pass of its own equals the product and a separate add."""
    g = torch.Generator(device="cuda").manual_seed(7)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.float16)
    x, w, r, b = rn(m, k), rn(k, n), rn(m, n), torch.randn(n, device="cuda", generator=g)
    out = torch.empty_like(r)
    p = lambda t: sfb.C.c_void_p(t.data_ptr())
    sfb._check(sfb.lib.sfb_linear_residual(sfb._stream(), p(out), p(x), p(w), p(b), p(r), *(sfb.C.c_uint32(v) for v in (m, n, k)), sfb.F16))
    assert sfb.device_status() == 0 and torch.equal(out, r + sfb.linear(x, w, b))


def test_linear_more_tiles_than_sms_and_batched_input(sfb, oracle):
    """A [B, L, hidden] activation (leading dimensions flattened) with enough tiles that every CTA loops."""
    B, L, hidden, n = 2, 4096, 768, 2304
    x = torch.randn(B, L, hidden, device="cuda", generator=torch.Generator(device="cuda").manual_seed(9)).to(torch.bfloat16)
    w = (0.05 * torch.randn(hidden, n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(10))).to(torch.bfloat16)
    b = torch.randn(n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(11))
    got = sfb.linear(x, w, b)
    assert sfb.device_status() == 0 and got.shape == (B, L, n)
    # rows sampled across all tiles against the oracle; everything against a float32 matmul on the device
    rows = np.arange(0, B * L, 97)
    want = oracle.linear(x.view(-1, hidden)[rows].float().cpu().numpy(), w.float().cpu().numpy(), b.cpu().numpy())
    assert np.abs(got.view(-1, n)[rows].float().cpu().numpy() - want).max() <= 2e-2 * np.abs(want).max()
    full = x.view(-1, hidden).float() @ w.float() + b
    assert float((got.view(-1, n).float() - full).abs().max()) <= 2e-2 * float(full.abs().max())


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("m,n,k,act,transposed", [
    (19000, 256, 64, 0, False),      # one k-block, one column tile, every pair of CTAs busy
    (2500, 2320, 200, 1, False),     # ragged in m (last 256-row tile: 196 rows), n (16 columns into the last tile) and k
    (4096, 768, 3072, 0, False),     # 48 k-blocks: the stage ring wraps eight times per tile
    (2304, 4000, 512, 1, True),      # w as [n, k]; the odd CTA's half of the last column tile lies beyond n
    (129, 19200, 128, 0, True),      # a single row into the second CTA's half
    (8192, 768, 256, 0, True),
    (8192, 752, 200, 1, True),       # ragged n (the last tile's second half has 112 of its 128 columns) and k
    # from here on the estimated times send the product to the CTA pairs; the shapes above go to 128 x 256 tiles
    (400000, 256, 64, 0, False),     # one k-block, one column tile, 22 rounds of tiles
    (8100, 752, 1032, 1, False),     # ragged in m (last 256-row tile: 164 rows), n (the last tile's second half: 112 columns) and k
    (8192, 752, 1032, 1, True),      # the same with w as [n, k]
    (4096, 3968, 520, 1, True),      # the odd CTA's half of the last column tile lies beyond n
    (385, 19200, 1024, 0, True),     # a single row into the second CTA's half of the last row tile
    (8192, 768, 3072, 0, False),     # 48 k-blocks: the stage ring wraps eight times per tile
])
def test_linear_on_cta_pairs(sfb, dtype, m, n, k, act, transposed):
    """Persistent kernels, on shapes with about one tile per SM and more: against a float32 product on the device (the oracle
    checks the same entry point on small shapes above)."""
    gen = torch.Generator(device="cuda").manual_seed(77)
    x = torch.randn(m, k, device="cuda", generator=gen).to(TD[dtype])
    w = (0.05 * torch.randn(k, n, device="cuda", generator=gen)).to(TD[dtype])
    b = torch.randn(n, device="cuda", generator=gen)
    got = sfb.linear_nt(x, w.t().contiguous(), b, act) if transposed else sfb.linear(x, w, b, act)
    assert sfb.device_status() == 0
    t = x.float() @ w.float() + b
    want = t * torch.sigmoid(1.702 * t) if act else t
    assert got.shape == (m, n)
    assert float((got.float() - want).abs().max()) <= 2e-2 * float(want.abs().max())


@pytest.mark.parametrize("m,n,k", [
    (20, 592 * 256, 64),             # one-CTA tiles: only the first of the four epilogue warps of a column half has rows to store
    (160, 592 * 256, 256),           # CTA pairs: the odd CTA has 32 rows
    (20, 600 * 256 - 112, 64),       # the last column tile is ragged too
])
def test_linear_bias_over_many_tiles_of_few_rows(sfb, m, n, k):
    """Several tiles per CTA, one or two k-blocks each, and epilogue warps without rows: those run ahead of the others as far
    as the accumulators let them, and must not replace the bias of a tile that is still being written.  The bias steps by 8
    from one column tile to the next, far above the rounding of the result."""
    gen = torch.Generator(device="cuda").manual_seed(78)
    x = torch.randn(m, k, device="cuda", generator=gen).to(torch.bfloat16)
    w = (0.01 * torch.randn(k, n, device="cuda", generator=gen)).to(torch.bfloat16)
    b = (torch.arange(n, device="cuda") // 256 % 7 * 8).float()
    want = x.float() @ w.float() + b
    for _ in range(5):
        got = sfb.linear(x, w, b)
        assert float((got.float() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max()) + 1e-3
    assert sfb.device_status() == 0


@pytest.fixture(scope="module")
def refusing(tmp_path_factory):
    """The projections built so that every launch of a cluster is refused (refused_clusters.cu)."""
    out = str(tmp_path_factory.mktemp("refused") / "refused.so")
    here = os.path.dirname(os.path.abspath(__file__))
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    os.path.join(here, "refused_clusters.cu"), "-o", out], check=True)
    lib = ctypes.CDLL(out)
    lib.linear_refused.argtypes = [ctypes.c_void_p] * 6 + [ctypes.c_uint] * 3 + [ctypes.c_int] * 2 + [ctypes.POINTER(ctypes.c_int)]
    return lib


@pytest.mark.parametrize("m,n,k,act,transposed,residual", [
    (320, 768, 3072, 0, False, False),       # clusters of two on 128 x 64 tiles
    (320, 768, 3072, 0, False, True),        # their residual, which the kernel that takes over leaves to a pass of its own
    (64, 192, 2056, 1, True, False),         # clusters of four
    (640, 1040, 4096, 0, True, False),       # clusters of two on 128 x 128 tiles
    (8192, 752, 1032, 1, False, False),      # CTA pairs
])
def test_linear_where_clusters_are_refused(sfb, refusing, m, n, k, act, transposed, residual):
    gen = torch.Generator(device="cuda").manual_seed(79)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen).to(torch.bfloat16)
    x, w, b = rn(m, k), rn(*((n, k) if transposed else (k, n))), torch.randn(n, device="cuda", generator=gen)
    r, out, n_refused = rn(m, n) if residual else None, torch.empty(m, n, device="cuda", dtype=torch.bfloat16), ctypes.c_int(0)
    p = lambda t: None if t is None else t.data_ptr()
    rc = refusing.linear_refused(torch.cuda.current_stream().cuda_stream, p(out), p(x), p(w), p(b), p(r), m, n, k, act, int(transposed), ctypes.byref(n_refused))
    assert rc == 0 and n_refused.value > 0
    t = x.float() @ (w.t() if transposed else w).float() + b
    want = t * torch.sigmoid(1.702 * t) if act else t
    if residual:
        want = want + r.float()
    assert float((out.float() - want).abs().max()) <= 2e-2 * float(want.abs().max())
    status = ctypes.c_uint(1)
    assert refusing.linear_status(ctypes.byref(status)) == 0 and status.value == 0


def test_linear_rejects_what_it_cannot_do(sfb):
    x = torch.zeros(16, 64, device="cuda")
    w = torch.zeros(64, 64, device="cuda")
    with pytest.raises(sfb.SfbError):
        sfb.linear(x, w)                                   # fp32
    xb, wb = x.to(torch.bfloat16), torch.zeros(64, 24, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(sfb.SfbError):
        sfb.linear(xb, wb)                                 # n not a multiple of 16


@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("m,n,k,act", [(128, 256, 64, 0), (300, 1008, 768, 0), (257, 30528, 1024, 0), (64, 48, 40, 1)])
def test_linear_nt_against_oracle(sfb, oracle, dtype, m, n, k, act):
    """out = x . wt^T with wt [n, k] -- the logits over a (padded) tied embedding table."""
    x, xn = _mk(oracle, (m, k), 410, dtype)
    wt, wn = _mk(oracle, (n, k), 411, dtype, 0.05)
    b = torch.from_numpy(oracle.fill_normal((n,), 412, 0.5)).cuda()
    got = sfb.linear_nt(x, wt, b, act)
    assert sfb.device_status() == 0
    rows = np.arange(0, m, max(1, m // 40))
    want = oracle.linear_nt(xn[rows], wn, b.cpu().numpy(), act)
    assert got.shape == (m, n) and got.dtype == TD[dtype]
    assert np.abs(got[rows].float().cpu().numpy() - want).max() <= 2e-2 * np.abs(want).max()
    # the transposed-weight path and the plain one are the same product
    same = sfb.linear(x, wt.t().contiguous(), b, act)
    assert float((got.float() - same.float()).abs().max()) <= 2e-2 * float(same.float().abs().max())


@pytest.mark.parametrize("dtype,hidden", [("f32", 768), ("bf16", 1024), ("f16", 40)])
def test_embedding_bit_exact(sfb, oracle, dtype, hidden):
    td = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[dtype]
    vocab, B, L = 3000, 3, 257
    table = torch.from_numpy(oracle.fill_normal((vocab, hidden), 420, 0.02)).cuda().to(td)
    pos = torch.from_numpy(oracle.fill_normal((L, hidden), 421, 0.02)).cuda().to(td)
    ids = torch.from_numpy((np.arange(B * L, dtype=np.int64) * 7919 % vocab).astype(np.int32).reshape(B, L)).cuda()
    out, bad = sfb.embedding(table, ids, pos)
    assert int(bad.item()) == 0
    want = oracle.embedding(table.float().cpu().numpy(), ids.cpu().numpy(), pos.float().cpu().numpy())
    if dtype == "f32":
        assert np.array_equal(out.cpu().numpy(), want)
    else:   # one rounding of the sum to 16 bits
        assert np.array_equal(out.float().cpu().numpy(), torch.from_numpy(want).to(td).float().numpy())
    plain, _ = sfb.embedding(table, ids)
    assert torch.equal(plain, table[ids.long()])


@pytest.mark.parametrize("B,L,hidden", [(37, 8, 64), (5, 2, 1024), (130, 33, 128), (1, 4096, 768)])
def test_embedding_batch_runs(sfb, B, L, hidden):
    """A thread keeps one piece of a position row for a run of batch elements; short sequences split the batch over
    the grid.  Batches that are no multiple of the run length or of the steps inside it, and a batch of one."""
    gen = torch.Generator(device="cuda").manual_seed(31)
    vocab = 1000
    table = torch.randn(vocab, hidden, device="cuda", generator=gen).to(torch.bfloat16)
    pos = torch.randn(L, hidden, device="cuda", generator=gen).to(torch.bfloat16)
    ids = torch.randint(0, vocab, (B, L), device="cuda", generator=gen, dtype=torch.int32)
    ids[B // 2, L // 2] = vocab + 3          # one id outside the table: zeros + position, counted once
    out, bad = sfb.embedding(table, ids, pos)
    assert int(bad.item()) == 1
    rows = table[ids.clamp(0, vocab - 1).long()].float()
    rows[B // 2, L // 2] = 0.0
    want = (rows + pos.float().unsqueeze(0)).to(torch.bfloat16)
    assert torch.equal(out, want)


@pytest.mark.parametrize("dtype,B,L,hidden", [("bf16", 4, 4096, 8), ("bf16", 5, 4096, 64), ("f32", 1, 16385, 8), ("f16", 3001, 7, 40), ("bf16", 1, 70001, 16)])
def test_embedding_counts_bad_ids_on_both_sides_of_the_line(sfb, dtype, B, L, hidden):
    """Up to 16384 ids one CTA counts, beyond that every reader: first and last ids of the sequence and the batch among the bad."""
    td = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[dtype]
    gen = torch.Generator(device="cuda").manual_seed(32)
    table = torch.randn(500, hidden, device="cuda", generator=gen).to(td)
    ids = torch.randint(-50, 550, (B, L), device="cuda", generator=gen, dtype=torch.int32)
    ids[0, 0], ids[-1, -1], ids[0, -1], ids[-1, 0] = -1, 500, 1 << 30, -(1 << 31)
    ok = (ids >= 0) & (ids < 500)
    for _ in range(2):                       # the second call starts from the first one's count
        out, bad = sfb.embedding(table, ids)
        assert int(bad.item()) == int((~ok).sum())
        assert torch.equal(out, table[ids.clamp(0, 499).long()] * ok.unsqueeze(-1))
    none = torch.zeros_like(ids)
    assert int(sfb.embedding(table, none)[1].item()) == 0


def test_embedding_count_does_not_set_the_time_of_a_long_lookup(sfb):
    """A million ids on narrow rows: with the count at most three times the time without it (one CTA reading all ids took 28
    times as long)."""
    B, L, hidden = 256, 4096, 8
    table = torch.ones(1000, hidden, device="cuda", dtype=torch.bfloat16)
    ids = torch.zeros(B, L, device="cuda", dtype=torch.int32)
    out, bad = sfb.embedding(table, ids)
    p = lambda t: ctypes.c_void_p(None if t is None else t.data_ptr())

    def us(count):
        times = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(20):
                sfb._check(sfb.lib.sfb_embedding(sfb._stream(), p(out), p(table), p(ids), None, *(ctypes.c_uint32(v) for v in (B, L, hidden, 1000)),
                                                 sfb.BF16, p(count)))
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    us(bad)
    assert us(bad) <= 3 * us(None)


def test_embedding_ids_outside_the_table_are_counted_not_read(sfb):
    table = torch.ones(10, 16, device="cuda", dtype=torch.bfloat16)
    ids = torch.tensor([[0, 9, 10, -1, 5]], dtype=torch.int32, device="cuda")
    out, bad = sfb.embedding(table, ids)
    assert int(bad.item()) == 2
    assert out[0, :, 0].float().cpu().tolist() == [1.0, 1.0, 0.0, 0.0, 1.0]

