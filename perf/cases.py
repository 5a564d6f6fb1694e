"""The work that users of this library have it do, as cases to time: block-sparse attention forward and backward,
the separate operators, encoder layers and whole encoder forwards, and element-sparse attention, each through the
package's public calls on tensors and layouts that such a program already holds."""
import importlib
import math

import numpy as np
import torch

sfb = importlib.import_module("sf-bert_b200")
encoder = importlib.import_module("sf-bert_b200.encoder")

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
BYTES = {"f32": 4, "bf16": 2, "f16": 2}
KINDS = {"full": sfb.LAYOUT_FULL, "fixed": sfb.LAYOUT_FIXED, "stride": sfb.LAYOUT_STRIDE, "sawtooth": sfb.LAYOUT_SAWTOOTH,
         "local": sfb.LAYOUT_LOCAL, "bigbird": sfb.LAYOUT_BIGBIRD}


def _case(kind, dtype, B, H, L, d, bs, layout, p=(0, 0, 0, 0), causal=False, mask=False, **more):
    """kind: what a pass is (see run).  layout, p, causal: the block pattern, as sfb.BlockLayout.generate takes it.
    mask: an element mask on the diagonal blocks, which a causal model needs."""
    return dict(kind=kind, dtype=dtype, B=B, H=H, L=L, d=d, bs=bs, layout=layout, p0=p[0], p1=p[1], p2=p[2], p3=p[3],
                causal=causal, mask=mask, **more)


def listed():
    return [
        # One short fp32 sequence with a pattern per head: the smallest call, a single launch of a few blocks.
        dict(_case("attention", "f32", 1, 4, 512, 64, 32, "fixed", (4, 0, 0, 0), per_head=True), name="attention_fixed_f32"),
        # fp32 operands, 32x32 blocks, 128-wide heads: the shape of the operators' own micro-benchmark (bench.py --kernel dropin).
        dict(_case("attention", "f32", 32, 4, 1024, 128, 32, "sawtooth", (8, 0, 0, 0)), name="attention_sawtooth_f32"),
        # The library's headline: BERT-base heads over long sequences, band plus every 8th column, fp16.
        dict(_case("attention", "f16", 8, 12, 4096, 64, 64, "stride", (4, 8, 0, 0)), name="attention_stride_f16"),
        # BigBird: rows of very different length (global rows, window, random blocks), bf16.
        dict(_case("attention", "bf16", 16, 12, 4096, 64, 64, "bigbird", (1, 1, 1, 3)), name="attention_bigbird_bf16"),
        # A small causal batch with an odd number of blocks per sequence and an element mask on the diagonal.
        dict(_case("attention", "bf16", 3, 12, 832, 64, 64, "full", causal=True, mask=True), name="attention_causal_bf16"),
        # The three operators one after another, for programs that keep scores and probabilities (bf16, sliding window).
        dict(_case("operators", "bf16", 2, 16, 4096, 64, 64, "local", (8, 8, 0, 0)), name="operators_local_bf16"),
        # A training step of the attention: probabilities kept by the forward, then the gradients of Q, K and V, fp16.
        dict(_case("training", "f16", 8, 12, 4096, 64, 64, "stride", (4, 8, 0, 0)), name="training_stride_f16"),
        # The same in the operators' original types: fp32 activations, bf16 scores, 32x32 blocks, a pattern per head, L=320.
        dict(_case("training", "f32", 32, 4, 320, 128, 32, "fixed", (5, 0, 0, 0), per_head=True), name="training_fixed_f32"),
        # One BERT-base encoder layer over long sequences: projections, attention, LayerNorm, FFN.
        dict(_case("model", "f16", 8, 12, 4096, 64, 64, "stride", (4, 8, 0, 0), layers=1, ln="post", vocab=0), name="layer_stride_f16"),
        # A request-sized forward of a small model: embedding, two layers, logits; five blocks per sequence, pre-LN.
        dict(_case("model", "bf16", 1, 12, 320, 64, 64, "full", layers=2, ln="pre", vocab=30528), name="model_small_bf16"),
        # The largest: embedding, 24 BERT-large layers with full attention and the logits over the vocabulary, four sequences.
        dict(_case("model", "bf16", 4, 16, 1024, 64, 64, "full", layers=24, ln="post", vocab=30528), name="model_large_bf16"),
        # Element-sparse attention for masks without block structure: a causal window per token, strided and random columns.
        dict(_case("elements", "f16", 2, 12, 4096, 64, 64, "stride", (4, 8, 0, 0), window=256, every=64, nrand=16), name="elements_window_f16"),
    ]


# ---- the patterns on the host: what a case costs, without a GPU -------------------------------------------------------
def _kept(case):
    """Kept blocks of one head's layout (the random blocks of BigBird: their expected number)."""
    nb = case["L"] // case["bs"]
    i, j = np.arange(nb)[:, None], np.arange(nb)[None, :]
    p0, p1, p2, p3 = (case["p%d" % k] for k in range(4))
    kind = case["layout"]
    if kind == "full":
        keep = np.ones((nb, nb), bool)
    elif kind == "fixed":
        keep = ((j >= p0 - 1) & ((j - (p0 - 1)) % p0 == 0)) | (j // p0 == i // p0)
    elif kind == "stride":
        keep = ((j <= i) & (j + p0 > i)) | (j % p1 == 0)
    elif kind == "sawtooth":
        keep = (j + i % p0 >= i) & (j <= i)
    elif kind == "local":
        keep = (j + p0 >= i) & (j <= i + p1)
    else:
        keep = (abs(i - j) <= p0) | (i < p1) | (i + p2 >= nb) | (j < p1) | (j + p2 >= nb)
    if case["causal"] and kind != "bigbird":
        keep = keep & (j <= i)
    count = float(keep.sum())
    if kind == "bigbird":
        count += float(((nb - keep.sum(1)) * min(p3, nb) / nb).sum())
    return count


def _nonzeros(case):
    """Kept elements of an element-sparse case."""
    if not case["window"]:
        return _kept(case) * case["bs"] ** 2
    i = np.arange(case["L"])
    near = np.minimum(i + 1, case["window"])
    far = np.maximum(i + 1 - case["window"], 0)                     # earlier than the window
    strided = np.ceil(far / case["every"])
    return float((near + strided + (far - strided) * (1 - (1 - 1 / case["L"]) ** case["nrand"])).sum())


def work(case):
    B, H, L, d, bs, e = case["B"], case["H"], case["L"], case["d"], case["bs"], BYTES[case["dtype"]]
    act = B * L * H * d * e
    if case["kind"] == "elements":
        nnz = _nonzeros(case)
        return {"bytes": 4 * act + 4 * (nnz + L), "flops": 4 * d * nnz * B * H}
    blocks = _kept(case) * B * H
    pair = 2 * bs * bs * d * blocks                                 # one product per kept block
    if case["kind"] == "attention":
        return {"bytes": 4 * act, "flops": 2 * pair}
    blk = blocks * bs * bs
    if case["kind"] == "operators":                                 # Q, K, V in, P and O out
        return {"bytes": 4 * act + blk * 2, "flops": 2 * pair}
    if case["kind"] == "training":                                  # Q, K, V, dO in, P, O, dQ, dK, dV out
        return {"bytes": 8 * act + blk * 2, "flops": 6 * pair}
    hidden, m = H * d, B * L
    flops = case["layers"] * (2 * m * hidden * hidden * 12 + 2 * pair)
    nbytes = case["layers"] * 12 * hidden * hidden * e + 2 * act
    if case["vocab"]:
        flops += 2 * m * hidden * case["vocab"]
        nbytes += case["vocab"] * hidden * e + m * case["vocab"] * e + L * hidden * e + 4 * m
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["dtype"] == "f32":
        # fp32 attention is fp32 throughout; training keeps scores, probabilities and their gradients in bf16, where a sum
        # at a rounding boundary moves by a bf16 unit
        return {"rel": 1e-5} if case["kind"] in ("attention", "elements") else {"rel": 5e-3}
    if case["kind"] == "model":
        return {"rel": 2e-2 if case["dtype"] == "bf16" else 5e-3}   # every layer rounds its activations several times
    # the operators and training keep scores or probabilities in the 16-bit type (scores always in bf16)
    return {"rel": 2e-3 if case["dtype"] == "f16" and case["kind"] in ("attention", "elements") else 1e-2 if case["dtype"] == "bf16" or case["kind"] == "operators" else 5e-3}


# ---- more cases of the same ranges ------------------------------------------------------------------------------------
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pattern(rng, nb, H):
    """A block pattern for nb blocks: (layout, parameters, causal, one per head)."""
    kind = rng.choice(["full", "fixed", "stride", "stride", "sawtooth", "local", "local", "bigbird"])
    if kind == "full":
        return kind, (0, 0, 0, 0), rng.random() < 0.5, False
    if kind == "fixed":
        fits = [s for s in range(2, 17) if nb % s == 0]
        if not fits:
            return "local", (2, 0, 0, 0), False, False
        s = rng.choice(fits)
        return kind, (s, 0, 0, 0), False, H <= s and rng.random() < 0.5
    if kind == "stride":
        return kind, (rng.randint(1, 8), rng.randint(4, 16), 0, 0), rng.random() < 0.3, False
    if kind == "sawtooth":
        return kind, (rng.randint(2, 12), 0, 0, 0), False, False
    if kind == "local":
        return kind, (rng.randint(1, 10), rng.randint(0, 10), 0, 0), rng.random() < 0.3, False
    return kind, (rng.randint(1, 2), 1, 1, min(3, nb)), False, False


def _drawn(rng):
    kind = rng.choice(["attention"] * 7 + ["operators"] * 2 + ["training"] * 4 + ["model"] * 5 + ["elements"] * 2)
    if kind == "model":
        H = rng.choice([4, 8, 12, 12, 16])
        nb = _log(rng, 2, 64)
        layout, p, causal, _ = _pattern(rng, nb, H)
        vocab = rng.choice([0, 30528, 16 * rng.randint(64, 1024)])
        return _case(kind, rng.choice(["bf16", "f16"]), _log(rng, 1, 16), H, 64 * nb, 64, 64, layout, p, causal,
                     layers=_log(rng, 1, 12), ln=rng.choice(["pre", "post"]), vocab=vocab)
    if kind == "elements":
        nb = _log(rng, 4, 64)
        layout, p, causal, _ = _pattern(rng, nb, 1)
        window = rng.choice([0, _log(rng, 16, 512)])                # 0: the elements of a block pattern
        return _case(kind, rng.choice(["f16", "bf16", "f32"]), _log(rng, 1, 4), _log(rng, 1, 16), 64 * nb, rng.choice([64, 64, 32, 128]), 64, layout, p,
                     causal, window=window, every=rng.randint(16, 128), nrand=rng.randint(0, 32))
    dtype = rng.choice(["f16", "bf16", "bf16", "f32", "f32"] if kind != "operators" else ["f16", "bf16", "bf16", "f32"])
    H = _log(rng, 1, 16)
    if dtype == "f32":                                              # the block sizes and head widths of the fp32 operators
        bs, d = rng.choice([32, 32, 64]), rng.choice([64, 64, 128, 32])
    elif kind == "attention" and rng.random() < 0.15:               # 16-bit operands at the other block size or head width
        bs, d = rng.choice([(32, 64), (64, 128), (32, 128)])
    else:
        bs, d = 64, 64
    nb = _log(rng, 2, 256 if kind == "attention" else 64)
    layout, p, causal, per_head = _pattern(rng, nb, H)
    mask = causal and layout != "bigbird" and rng.random() < 0.7
    return _case(kind, dtype, _log(rng, 1, 32), H, bs * nb, d, bs, layout, p, causal, mask, per_head=per_head)


def draw(rng):
    while True:
        case = _drawn(rng)
        w = work(case)
        small = case["dtype"] == "f32" or case["kind"] == "elements" or case["bs"] != 64 or case["d"] != 64
        most = 1.2e12 if case["kind"] == "model" else 2e10 if small else 3e11
        if w["flops"] <= most and w["bytes"] <= 2e9:
            return case


# ---- a user's program --------------------------------------------------------------------------------------------------
def _element_pattern(case, seed):
    """rowptr and colidx of a causal pattern per token: the last `window` tokens, every `every`-th earlier one, and
    `nrand` random earlier ones."""
    L = case["L"]
    i, j = torch.arange(L, device="cuda")[:, None], torch.arange(L, device="cuda")[None, :]
    keep = (i - j < case["window"]) | (j % case["every"] == 0)
    if case["nrand"]:
        g = torch.Generator(device="cuda").manual_seed(seed)
        keep.scatter_(1, torch.randint(0, L, (L, case["nrand"]), device="cuda", generator=g), True)
    keep &= j <= i
    rowptr = torch.zeros(L + 1, dtype=torch.int32, device="cuda")
    rowptr[1:] = keep.sum(1).cumsum(0)
    return rowptr, keep.nonzero()[:, 1].to(torch.int32).contiguous()


def prepare(case, seed):
    B, H, L, d, bs, t = case["B"], case["H"], case["L"], case["d"], case["bs"], DTYPES[case["dtype"]]
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = {"case": case, "scale": 1.0 / math.sqrt(d)}
    lay = sfb.BlockLayout.generate(KINDS[case["layout"]], H if case.get("per_head") else 1, L // bs, bs, case["p0"], case["p1"],
                                   case["p2"], case["p3"], int(case["causal"]), seed=1236)
    if case["mask"]:
        lay.pack_mask(sfb.MASK_CAUSAL_DIAG)
    if case["kind"] == "training":
        lay.tn_lut                                                  # the backward's table is built once with the layout
    s["lay"] = lay
    if case["kind"] == "model":
        hidden = H * d
        s["w"] = [encoder.EncoderLayerWeights(hidden, 4 * hidden, t, seed=seed + 1 + n) for n in range(case["layers"])]
        if case["vocab"]:
            s["table"] = (0.02 * torch.randn(case["vocab"], hidden, device="cuda", generator=g)).to(t)
            s["pos"] = (0.02 * torch.randn(L, hidden, device="cuda", generator=g)).to(t)
            s["ids"] = torch.randint(0, case["vocab"], (B, L), device="cuda", dtype=torch.int32, generator=g)
        else:
            s["x"] = torch.randn(B, L, hidden, device="cuda", generator=g).to(t)
        return s
    names = ("q", "k", "v", "do") if case["kind"] == "training" else ("q", "k", "v")
    for n in names:
        s[n] = torch.randn(B, L, H, d, device="cuda", generator=g).to(t)
    if case["kind"] == "elements":
        s["rowptr"], s["colidx"] = _element_pattern(case, seed) if case["window"] else sfb.csr_from_layout(lay)
    return s


def run(s):
    case, lay, scale = s["case"], s["lay"], s["scale"]
    kind, masked = case["kind"], case["mask"]
    if kind == "attention":
        return sfb.fused_attention(s["q"], s["k"], s["v"], lay, scale, use_mask=masked)
    if kind == "elements":
        return sfb.csr_attention(s["q"], s["k"], s["v"], s["rowptr"], s["colidx"], scale)[0]
    if kind == "model":
        x = sfb.embedding(s["table"], s["ids"], s["pos"])[0] if case["vocab"] else s["x"]
        for w in s["w"]:
            x = encoder.encoder_layer(sfb, x, w, lay, case["H"], case["ln"], "tensor")
        return {"hidden": x, "logits": sfb.linear_nt(x, s["table"])} if case["vocab"] else {"hidden": x}
    q, k, v, f32 = s["q"], s["k"], s["v"], case["dtype"] == "f32"
    if kind == "operators" or f32:
        # scores and probabilities in bf16 beside fp32 activations, in the activations' type beside 16-bit ones
        p = sfb.masked_softmax(sfb.bst_sgemm_nt(q, k, lay), lay, scale, torch.bfloat16 if f32 else q.dtype, masked)
    else:
        p = sfb.fused_sddmm_softmax(q, k, lay, scale, q.dtype, masked)
    o = sfb.bst_sgemm_xn(p, v, lay)
    if kind == "operators":
        return {"p": p, "o": o}
    if f32:
        dq, dk, dv = sfb.attention_backward(q, k, v, p, s["do"], lay, scale)
    else:
        dq, dk, dv = sfb.attention_backward_fused(q, k, v, p, o, s["do"], lay, scale)
    return {"p": p, "o": o, "dq": dq, "dk": dk, "dv": dv}
