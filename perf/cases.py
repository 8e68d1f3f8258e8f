"""The attention calls that a user of this framework makes, as a list of measurable cases.

A case is a dict of plain values.  ``op`` names the path it takes through ``flashck_b200.ops``:

* ``dense``   -- ``fmha_fwd``: one rectangular batch (training forward, encoders), with the masks and score additions
* ``varlen``  -- ``fmha_fwd_var_len`` / ``fmha_fwd_fp8``: packed prompts of unequal lengths (serving prefill)
* ``chunk``   -- ``fmha_fwd_paged_kv_prefill`` / ``batch_prefill``: a chunk of new tokens per sequence against a paged cache
* ``decode``  -- ``fmha_fwd_splitkv``: one token per sequence, or a few drafted ones, against a paged or contiguous cache
* ``append``  -- ``fmha_fwd_append_kv`` + ``fmha_fwd_splitkv``: RoPE and cache write of the new tokens, then their decode

``lo`` / ``hi`` bound the sequence lengths; ``lens_seed`` fixes them, so that the work of a case does not depend on the
seed of its values.  Head geometries, length ranges and page sizes are those of the repository's benchmark and tests.
"""
import torch

from flashck_b200 import ops
from flashck_b200.utils.inputs import iota_shuffle, rotary_cos_sin, to_seqstarts, uniform_seqlens

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "e4m3": torch.float8_e4m3fn}
_BYTES = {"bf16": 2, "fp16": 2, "e4m3": 1}
_MOST_FLOPS, _MOST_BYTES = 8.3e11, 8.6e9  # of a drawn case: what the largest listed ones take


def _case(name, op, dtype, batch, hq, hkv, d, **more):
    return dict(name=name, op=op, dtype=dtype, batch=batch, hq=hq, hkv=hkv, d=d, **more)


def listed():
    return [
        # the smallest call: two short fp16 prompts, where the call itself is what takes the time
        _case("dense_tiny", "dense", "fp16", 2, 8, 8, 64, sq=128, mask="causal", add="none", cap=0.0, lse=True),
        # an encoder layer: no mask, head dim 64, a length that no tile divides
        _case("encoder_hdim64", "dense", "bf16", 32, 16, 16, 64, sq=1025, mask="none", add="none", cap=0.0, lse=False),
        # training forward with a sliding window and a logits soft cap (LSE is kept for the backward pass)
        _case("window_softcap", "dense", "bf16", 2, 32, 8, 128, sq=5000, mask="window", window=1023, add="none", cap=30.0,
              lse=True),
        # a relative-position bias tensor with a plane per head
        _case("bias_per_head", "dense", "bf16", 2, 16, 16, 128, sq=2048, mask="none", add="bias1", cap=0.0, lse=False),
        # serving prefill of a batch of prompts of unequal lengths; the same on 8-bit operands
        _case("varlen_prefill", "varlen", "bf16", 16, 32, 8, 128, lo=512, hi=4096, lens_seed=1234, mask="causal", lse=True),
        _case("varlen_prefill_fp8", "varlen", "e4m3", 16, 32, 8, 128, lo=512, hi=4096, lens_seed=1234, mask="causal", lse=True),
        # chunked prefill: a few hundred new tokens per sequence over what the paged cache already holds
        _case("chunked_prefill", "chunk", "bf16", 6, 32, 8, 128, lo=1024, hi=16384, new_lo=128, new_hi=768, page=16,
              lens_seed=21, table="block", lse=False),
        # decode: a full serving batch, one short conversation, a few very long contexts, a contiguous fp16 cache of hdim 64
        _case("decode_batch", "decode", "bf16", 64, 32, 8, 128, lo=1024, hi=32768, tokens=1, page=16, lens_seed=4321),
        _case("decode_single", "decode", "bf16", 1, 32, 8, 128, lo=2000, hi=4000, tokens=1, page=16, lens_seed=5),
        _case("decode_long", "decode", "bf16", 4, 64, 8, 128, lo=524288, hi=524288, tokens=1, page=64, lens_seed=9),
        _case("decode_hdim64", "decode", "fp16", 48, 32, 8, 64, lo=300, hi=8000, tokens=1, page=0, lens_seed=77),
        # the decode step of a speculative or chunked scheduler: append 1-16 tokens with RoPE, then attend
        _case("append_decode", "append", "bf16", 32, 32, 8, 128, lo=2048, hi=16384, new_lo=1, new_hi=16, page=16, lens_seed=99),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _draw_once(rng):
    op = rng.choice(["dense", "dense", "varlen", "chunk", "decode", "decode", "append"])
    hq, hkv = rng.choice([(32, 8), (32, 8), (64, 8), (16, 16), (8, 8), (16, 2), (12, 4)])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    seed = rng.randrange(1 << 20)
    if op == "dense":
        mask, add = rng.choice(["none", "causal", "causal", "window"]), rng.choice(["none", "none", "none", "alibi", "bias0", "bias1"])
        d = rng.choice([128, 128, 64])
        case = _case("", op, dtype, _log_int(rng, 1, 32), hq, hkv, d, sq=_log_int(rng, 64, 16384), mask=mask, add=add,
                     cap=rng.choice([0.0, 0.0, 0.0, 30.0]), lse=rng.random() < 0.5)
        if mask == "window":
            case["window"] = _log_int(rng, 128, 4096)
    elif op == "varlen":
        lo = _log_int(rng, 32, 1024)
        case = _case("", op, rng.choice([dtype, dtype, "e4m3"]), _log_int(rng, 1, 64), hq, hkv, 128, lo=lo,
                     hi=lo * rng.randint(2, 8), lens_seed=seed, mask=rng.choice(["causal", "causal", "none"]), lse=rng.random() < 0.5)
    elif op == "chunk":
        lo, new = _log_int(rng, 256, 8192), _log_int(rng, 64, 2048)
        case = _case("", op, dtype, _log_int(rng, 1, 32), hq, hkv, 128, lo=lo, hi=lo * rng.randint(1, 4), new_lo=max(1, new // 4),
                     new_hi=new, page=rng.choice([16, 16, 32, 64]), lens_seed=seed, table=rng.choice(["block", "indptr"]),
                     lse=rng.random() < 0.3)
    elif op == "decode":
        lo = _log_int(rng, 128, 65536)
        case = _case("", op, dtype, _log_int(rng, 1, 128), hq, hkv, rng.choice([128, 128, 64]), lo=lo, hi=lo * rng.randint(1, 8),
                     tokens=rng.choice([1, 1, 1, 2, 4]), page=rng.choice([0, 16, 16, 64]), lens_seed=seed)
    else:
        lo = _log_int(rng, 256, 16384)
        case = _case("", op, dtype, _log_int(rng, 1, 64), hq, hkv, 128, lo=lo, hi=lo * rng.randint(1, 8), new_lo=1,
                     new_hi=rng.choice([1, 4, 16]), page=rng.choice([16, 16, 64]), lens_seed=seed)
    del case["name"]
    return case


def draw(rng):
    while True:
        case = _draw_once(rng)
        w = work(case)
        dear = case.get("cap", 0.0) > 0 or case.get("add", "none") != "none"  # (score additions: more time per FLOP)
        if w["flops"] <= _MOST_FLOPS / (5 if dear else 1) and w["bytes"] <= _MOST_BYTES:
            return case


# ---- sizes of a case -----------------------------------------------------------------------------------------------
def _lens(case):
    """(query lengths, key lengths) of every sequence; the keys include the new tokens."""
    b, op = case["batch"], case["op"]
    if op == "dense":
        return [case["sq"]] * b, [case["sq"]] * b
    ctx = uniform_seqlens(b, case["lo"], case["hi"], case["lens_seed"])
    if op == "varlen":
        return ctx, ctx
    if op == "decode":
        return [case["tokens"]] * b, ctx
    new = uniform_seqlens(b, case["new_lo"], case["new_hi"], case["lens_seed"] + 1)
    return new, [c + n for c, n in zip(ctx, new)]


def _pairs(case, nq, nk):
    """Visible (query, key) pairs of one sequence: bottom-right aligned causal or window masks, or everything."""
    mask = case.get("mask", "causal" if nq > 1 else "none")
    if mask == "none":
        return nq * nk
    full = nq * (nk - nq) + nq * (nq + 1) // 2
    if mask == "causal":
        return full
    hidden = max(0, nk - case["window"] - 1)  # keys the last row no longer sees; one fewer for each row before it
    rows = min(nq, hidden)
    return full - (rows * hidden - rows * (rows - 1) // 2)


def work(case):
    nq, nk = _lens(case)
    b, hq, hkv, d, size = case["batch"], case["hq"], case["hkv"], case["d"], _BYTES[case["dtype"]]
    flops = 4 * d * hq * sum(_pairs(case, q, k) for q, k in zip(nq, nk))
    tq, tk = sum(nq), sum(nk)
    nbytes = tq * hq * d * size + tk * hkv * 2 * d * size + tq * hq * d * 2  # Q, K and V read, O written
    if case.get("lse"):
        nbytes += 4 * tq * hq
    if case["op"] == "dense" and case["add"].startswith("bias"):
        nbytes += case["sq"] ** 2 * size * (hq if case["add"] == "bias1" else 1)
    if case.get("page"):
        nbytes += 4 * sum(-(-k // case["page"]) for k in nk)
    if case["op"] == "append":  # the new tokens' K and V read and written, their cos / sin rows; Q rotated in place
        nbytes += tq * hkv * 2 * d * size * 2 + tq * d * size + tq * hq * d * size * 2
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # About four times what the path differs by from the same attention with every sum in 64 bits: 2.3e-3 (max 3.5e-2, rows
    # that a long window leaves small) in bf16, 2.9e-4 in fp16; on 8-bit operands P keeps 3 bits: 2.0e-2 (max 0.4).
    if case["dtype"] == "e4m3":
        return {"rel": 3e-2, "max": 0.8}
    return {"rel": 1e-2, "max": 0.14} if case["dtype"] == "bf16" else {"rel": 1.2e-3, "max": 2e-2}


# ---- inputs ----------------------------------------------------------------------------------------------------------
def _pool(lens, page, seed):
    """(block table [batch, pages of the longest], number of pages): a shuffled hand-out of the pool's pages."""
    pages = [-(-n // page) for n in lens]
    perm, off = iota_shuffle(sum(pages), seed), 0
    table = torch.zeros((len(lens), max(pages)), dtype=torch.int32)
    for b, n in enumerate(pages):
        table[b, :n] = perm[off:off + n]
        off += n
    return table, sum(pages)


def prepare(case, seed):
    dev, dtype = torch.device("cuda"), _DTYPES[case["dtype"]]
    op, b, hq, hkv, d = case["op"], case["batch"], case["hq"], case["hkv"], case["d"]
    g = torch.Generator(device=dev).manual_seed(seed)
    nq, nk = _lens(case)
    s = {"case": case, "causal": case.get("mask", "causal") != "none"}

    def randn(*shape):
        return torch.randn(shape, generator=g, device=dev, dtype=torch.bfloat16 if dtype == torch.float8_e4m3fn else dtype)

    if op == "dense":
        n = case["sq"]
        s["q"], s["k"], s["v"] = randn(b, n, hq, d), randn(b, n, hkv, d), randn(b, n, hkv, d)
        s["kw"] = {"causal": s["causal"], "return_lse": case["lse"], "logits_soft_cap": case["cap"]}
        if case["mask"] == "window":
            s["kw"]["window_size"] = (case["window"], 0)
        if case["add"] == "alibi":
            s["kw"]["alibi_slopes"] = 2.0 ** (-8.0 * torch.arange(1, hq + 1, device=dev, dtype=torch.float32) / hq).view(1, hq)
        elif case["add"] != "none":
            s["kw"]["bias"] = randn(1, hq if case["add"] == "bias1" else 1, n, n)
        return s
    s["max_q"] = max(nq)
    s["cu_q"] = to_seqstarts(nq).to(dev)
    if op == "varlen":
        s["q"], s["k"], s["v"] = randn(sum(nq), hq, d), randn(sum(nk), hkv, d), randn(sum(nk), hkv, d)
        if case["dtype"] == "e4m3":
            (s["q"], dq), (s["k"], dk), (s["v"], dv) = (ops.quantize_fp8(s[n], dtype) for n in ("q", "k", "v"))
            s["scales"] = {"scale_s": dq * dk / d ** 0.5, "scale_p": 256.0, "scale_o": dv / 256.0}
        return s
    page = case["page"]
    s["seqlen"] = torch.tensor(nk, dtype=torch.int32, device=dev)
    if page:
        table, pages = _pool(nk, page, seed)
        s["k"], s["v"], s["table"] = randn(pages, page, hkv, d), randn(pages, page, hkv, d), table.to(dev)
    else:
        s["k"], s["v"], s["table"] = randn(b, max(nk), hkv, d), randn(b, max(nk), hkv, d), None
    if op == "decode":
        s["q"] = randn(b, case["tokens"], hq, d)
        return s
    s["q"] = randn(sum(nq), hq, d)
    if op == "chunk":
        if case["table"] == "indptr":  # the page table as one list per batch
            pages = [-(-n // page) for n in nk]
            s["indptr"] = to_seqstarts(pages).to(dev, torch.int32)
            s["indices"] = torch.cat([table[i, :n] for i, n in enumerate(pages)]).to(dev)
            s["last"] = torch.tensor([n - (p - 1) * page for n, p in zip(nk, pages)], dtype=torch.int32, device=dev)
        return s
    s["knew"], s["vnew"] = randn(sum(nq), hkv, d), randn(sum(nq), hkv, d)
    s["cached"] = torch.tensor([k - n for k, n in zip(nk, nq)], dtype=torch.int32, device=dev)
    cos, sin = rotary_cos_sin(max(nk) + 1, d, dtype)
    s["cos"], s["sin"] = cos.to(dev), sin.to(dev)
    return s


# ---- one pass ----------------------------------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    op = case["op"]
    if op == "dense":
        return ops.fmha_fwd(s["q"], s["k"], s["v"], **s["kw"])
    if op == "varlen":
        if case["dtype"] == "e4m3":
            return ops.fmha_fwd_fp8(s["q"], s["k"], s["v"], cu_seqlens_q=s["cu_q"], cu_seqlens_k=s["cu_q"],
                                    max_seqlen_q=s["max_q"], causal=s["causal"], out_dtype=torch.bfloat16,
                                    return_lse=case["lse"], **s["scales"])
        return ops.fmha_fwd_var_len(s["q"], s["k"], s["v"], s["cu_q"], s["cu_q"], s["max_q"], causal=s["causal"],
                                    return_lse=case["lse"])
    if op == "chunk":
        if case["table"] == "indptr":
            return ops.batch_prefill(s["q"], s["k"], s["v"], s["cu_q"], s["indptr"], s["indices"], s["last"], s["max_q"],
                                     causal=True, return_lse=case["lse"])
        return ops.fmha_fwd_paged_kv_prefill(s["q"], s["k"], s["v"], s["table"], s["seqlen"], cu_seqlens_q=s["cu_q"],
                                             max_seqlen_q=s["max_q"], causal=True, return_lse=case["lse"])
    if op == "decode":
        return ops.fmha_fwd_splitkv(s["q"], s["k"], s["v"], seqlen_k=s["seqlen"], block_table=s["table"],
                                    causal=case["tokens"] > 1)
    ops.fmha_fwd_append_kv(s["q"], s["k"], s["v"], s["knew"], s["vnew"], s["cached"], s["cos"], s["sin"],
                           block_table=s["table"], cu_seqlens_q=s["cu_q"], cu_seqlens_knew=s["cu_q"])
    o = ops.fmha_fwd_splitkv(s["q"], s["k"], s["v"], seqlen_k=s["seqlen"], block_table=s["table"], cu_seqlens_q=s["cu_q"],
                             max_seqlen_q=s["max_q"], causal=True)
    return {"o": o, "q": s["q"], "k_cache": s["k"], "v_cache": s["v"]}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------
def _rope64(x, cos, sin):
    """Interleaved pairs of x [n, heads, d] rotated by the n rows of cos / sin."""
    x, c, s = x.double(), cos.double()[:, None], sin.double()[:, None]
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack((a * c - b * s, a * s + b * c), -1).flatten(-2)


def _attend64(case, q, k, v, bias=None, slopes=None, scale=None):
    """Attention of one sequence, q [nq, hq, d] over k, v [nk, hkv, d]: (o, lse [hq, nq]), a block of rows of one head at a time."""
    (nq, hq, d), nk, group = q.shape, k.shape[0], q.shape[1] // k.shape[1]
    o = torch.empty((nq, hq, d), dtype=torch.float64, device=q.device)
    lse = torch.empty((hq, nq), dtype=torch.float64, device=q.device)
    step, keys = max(1, (1 << 27) // nk), torch.arange(nk, device=q.device)
    for h in range(hq):
        if h % group == 0:
            kh, vh = k[:, h // group].double(), v[:, h // group].double()
        for r in range(0, nq, step):
            rows = torch.arange(r, min(nq, r + step), device=q.device)[:, None] + (nk - nq)
            x = (q[r:r + step, h].double() @ kh.T) * (scale or d ** -0.5)
            if case.get("cap", 0.0) > 0:
                x = case["cap"] * torch.tanh(x / case["cap"])
            if bias is not None:
                x += bias[0, h if bias.shape[1] > 1 else 0, r:r + step].double()
            if slopes is not None:
                x -= slopes[0, h].double() * (rows - keys).abs()
            if case.get("mask", "causal" if nq > 1 else "none") != "none":
                x.masked_fill_(keys > rows, float("-inf"))
                if case.get("mask") == "window":
                    x.masked_fill_(keys < rows - case["window"], float("-inf"))
            lse[h, r:r + step] = torch.logsumexp(x, -1)
            o[r:r + step, h] = torch.softmax(x, -1) @ vh
    return o, lse


def exact(case, seed):
    nq, nk = _lens(case)
    if case["hq"] * sum(q * k for q, k in zip(nq, nk)) > 2.5e10:
        return None
    s = prepare(case, seed)
    op = case["op"]
    if op == "dense":
        kw = s["kw"]
        parts = [_attend64(case, s["q"][i], s["k"][i], s["v"][i], kw.get("bias"), kw.get("alibi_slopes")) for i in range(case["batch"])]
        o, lse = torch.stack([p[0] for p in parts]), torch.stack([p[1] for p in parts])
        return (o, lse) if case["lse"] else o
    cq = [sum(nq[:i]) for i in range(len(nq) + 1)]
    if op == "varlen":
        sc = s.get("scales")
        parts = [_attend64(case, s["q"][a:b], s["k"][a:b], s["v"][a:b], scale=sc and sc["scale_s"]) for a, b in zip(cq, cq[1:])]
        o, lse = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts], 1)
        if sc:
            o *= sc["scale_p"] * sc["scale_o"]
        return (o, lse) if case["lse"] else o

    def cached(pool, b):
        if not case["page"]:
            return pool[b, :nk[b]]
        return pool[s["table"][b, :-(-nk[b] // case["page"])].long()].flatten(0, 1)[:nk[b]]

    q, out = s["q"].flatten(0, 1) if op == "decode" else s["q"], {}
    if op == "append":
        pos = torch.cat([torch.arange(k - n, k) for n, k in zip(nq, nk)]).to(q.device)
        knew = _rope64(s["knew"], s["cos"][pos], s["sin"][pos])
        q = _rope64(q, s["cos"][pos], s["sin"][pos])
        out = {"q": q, "k_cache": None, "v_cache": None}  # (whole pools: copies of the new rows, and the rest as it was)
    parts = []
    for b in range(case["batch"]):
        k, v = cached(s["k"], b).double(), cached(s["v"], b).double()
        if op == "append":
            k[nk[b] - nq[b]:], v[nk[b] - nq[b]:] = knew[cq[b]:cq[b + 1]], s["vnew"][cq[b]:cq[b + 1]].double()
        parts.append(_attend64(case, q[cq[b]:cq[b + 1]] if op != "decode" else s["q"][b], k, v))
    o, lse = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts], 1)
    if op == "append":
        return {"o": o, **out}
    if op == "decode":
        return o.view(s["q"].shape)
    return (o, lse) if case["lse"] else o
