"""Sizes that the kernels index one tensor by and take from another: a call whose tensors do not fit is refused on the host.  The
tensors are fake (no memory, no device), so nothing can be launched; the compiled binding is asked on a GPU box with real ones, directly
and for its answer alone."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from flashck_b200 import ops
from flashck_b200.ops import fmha

BF, I32, I64, F32, F8 = torch.bfloat16, torch.int32, torch.int64, torch.float32, torch.float8_e4m3fn


def _append(form):
    """Two sequences, three new tokens each, 2 kv heads of 64 (V: 128), pages of 16."""
    s = {"q": (2, 3, 4, 64), "k_cache": (9, 16, 2, 64), "v_cache": (9, 16, 2, 128), "knew": (2, 3, 2, 64), "vnew": (2, 3, 2, 128),
         "seqlen_k": (2,), "rotary_cos": (40, 32), "rotary_sin": (40, 32), "block_table": (2, 4)}
    if form == "packed":
        s |= {"q": (6, 4, 64), "knew": (6, 2, 64), "vnew": (6, 2, 128), "cu_seqlens_q": (3,), "cu_seqlens_knew": (3,)}
    if form == "contiguous":
        s |= {"k_cache": (2, 50, 2, 64), "v_cache": (2, 50, 2, 128), "block_table": None}
    return s


def _prefill(form):
    s = {"q": (2, 30, 4, 64), "k_pool": (9, 16, 2, 64), "v_pool": (9, 16, 2, 64), "block_table": (2, 4), "seqlen_k": (2,)}
    if form == "packed":
        s |= {"q": (60, 4, 64), "cu_seqlens_q": (3,), "max_seqlen_q": 30}
    return s


def _decode(form):
    s = {"q": (2, 1, 4, 64), "k_cache": (9, 16, 2, 64), "v_cache": (9, 16, 2, 64), "block_table": (2, 4), "seqlen_k": (2,)}
    if form == "contiguous":
        s |= {"k_cache": (2, 50, 2, 64), "v_cache": (2, 50, 2, 64), "block_table": None}
    if form == "packed keys":
        s |= {"q": (2, 4, 64), "cu_seqlens_q": (3,), "max_seqlen_q": 1, "k_cache": (70, 2, 64), "v_cache": (70, 2, 64), "block_table": None,
              "seqlen_k": None, "cu_seqlens_k": (3,)}
    return s


def _fp8(form):
    s = {"q": (2, 30, 4, 64), "k": (2, 50, 2, 64), "v": (2, 50, 2, 64)}
    if form == "packed":
        s = {"q": (60, 4, 64), "k": (70, 2, 64), "v": (70, 2, 64), "cu_seqlens_q": (3,), "cu_seqlens_k": (3,)}
    return s


def _tensors(sizes, device, elem=BF):
    kind = {"seqlen_k": I32, "block_table": I32, "cu_seqlens_q": I64, "cu_seqlens_k": I64, "cu_seqlens_knew": I64, "cache_batch_idx": I64}
    out = {}
    for n, v in sizes.items():
        if n == "workspace":
            out[n] = tuple(torch.empty(x, dtype=F32, device=device) for x in v)
        else:
            out[n] = torch.zeros(v, dtype=kind.get(n, elem), device=device) if isinstance(v, tuple) else v
    return out


APPEND = [
    ("paged", {"knew": (2, 3, 4, 64), "vnew": (2, 3, 4, 128)}),      # more kv heads than the caches have
    ("paged", {"k_cache": (9, 16, 2, 32)}), ("paged", {"v_cache": (9, 16, 2, 64)}), ("paged", {"v_cache": (9, 16, 4, 128)}),
    ("paged", {"v_cache": (9, 8, 2, 128)}), ("paged", {"v_cache": (8, 16, 2, 128)}),
    ("paged", {"vnew": (2, 2, 2, 128)}), ("paged", {"vnew": (1, 3, 2, 128)}), ("paged", {"knew": (1, 3, 2, 64), "vnew": (1, 3, 2, 128)}),
    ("paged", {"seqlen_k": (3,)}), ("paged", {"block_table": (1, 4)}), ("paged", {"q": (1, 3, 4, 64)}), ("paged", {"q": (2, 3, 4, 32)}),
    ("paged", {"rotary_sin": (40, 16)}), ("paged", {"rotary_cos": (40, 16), "rotary_sin": (40, 16), "rotary_dim": 64}),
    ("packed", {"cu_seqlens_knew": (2,)}), ("packed", {"cu_seqlens_q": (2,)}), ("packed", {"seqlen_k": (3,), "block_table": (3, 4)}),
    ("packed", {"vnew": (5, 2, 128)}),
    ("contiguous", {"k_cache": (1, 50, 2, 64), "v_cache": (1, 50, 2, 128)}), ("contiguous", {"v_cache": (2, 40, 2, 128)}),
    ("contiguous", {"cache_batch_idx": (1,)}),
]
PREFILL = [
    ("paged", {"k_pool": (9, 16, 2, 128), "v_pool": (9, 16, 2, 128)}), ("paged", {"v_pool": (9, 16, 1, 64)}),
    ("paged", {"v_pool": (9, 8, 2, 64)}), ("paged", {"v_pool": (8, 16, 2, 64)}), ("paged", {"seqlen_k": (1,)}),
    ("paged", {"cache_batch_idx": (1,)}), ("packed", {"cu_seqlens_q": (2,)}), ("packed", {"block_table": (3, 4), "seqlen_k": (3,)}),
]
DECODE = [
    ("paged", {"v_cache": (9, 16, 1, 64)}), ("paged", {"v_cache": (9, 8, 2, 64)}), ("paged", {"v_cache": (8, 16, 2, 64)}),
    ("paged", {"seqlen_k": (1,)}), ("paged", {"cache_batch_idx": (1,)}),
    ("paged", {"workspace": ((2, 4, 8, 1), (2, 4, 8, 1, 32))}), ("paged", {"workspace": ((2, 4, 7, 1), (2, 4, 8, 1, 64))}),
    ("paged", {"workspace": ((1, 4, 8, 1), (1, 4, 8, 1, 64))}),
    ("contiguous", {"k_cache": (1, 50, 2, 64), "v_cache": (1, 50, 2, 64)}), ("contiguous", {"v_cache": (2, 40, 2, 64)}),
    ("packed keys", {"cu_seqlens_k": (2,)}), ("packed keys", {"v_cache": (69, 2, 64)}),
]
FP8 = [
    ("batch", {"k": (1, 50, 2, 64), "v": (1, 50, 2, 64)}), ("batch", {"v": (2, 49, 2, 64)}), ("batch", {"v": (2, 50, 1, 64)}),
    ("batch", {"k": (2, 50, 2, 32)}), ("packed", {"cu_seqlens_k": (2,)}), ("packed", {"v": (69, 2, 64)}), ("packed", {"k": (70, 2, 32)}),
]
CALLS = {"append": (ops.fmha_fwd_append_kv, _append, APPEND, BF), "prefill": (ops.fmha_fwd_paged_kv_prefill, _prefill, PREFILL, BF),
         "decode": (ops.fmha_fwd_splitkv, _decode, DECODE, BF), "fp8": (ops.fmha_fwd_fp8, _fp8, FP8, F8)}


@pytest.mark.parametrize("what,n", [(w, n) for w, c in CALLS.items() for n in range(len(c[2]))])
def test_refused_on_the_host(what, n):
    fn, sizes, wrong, elem = CALLS[what]
    form, other = wrong[n]
    with FakeTensorMode(), pytest.raises(ValueError):
        fn(**_tensors(sizes(form) | other, "cuda", elem))


class Launched(Exception):
    pass


# ... and what fits is not: the sizes above, and larger tensors than a call needs where the rest of them is not looked at
FITS = [("append", f, {}) for f in ("paged", "packed", "contiguous")] + [("prefill", f, {}) for f in ("paged", "packed")] + \
       [("decode", f, {}) for f in ("paged", "contiguous", "packed keys")] + [("fp8", f, {}) for f in ("batch", "packed")] + [
    ("append", "paged", {"knew": (3, 3, 2, 64), "vnew": (3, 3, 2, 128), "q": (3, 3, 4, 64), "block_table": (3, 4)}),
    ("append", "packed", {"cu_seqlens_q": (5,), "cu_seqlens_knew": (5,)}), ("append", "paged", {"q": None}),
    ("append", "paged", {"q": (1, 3, 4, 32), "rope": 0}), ("append", "paged", {"k_cache": (9, 16, 128), "v_cache": (9, 16, 256)}),
    ("append", "contiguous", {"k_cache": (7, 50, 2, 64), "v_cache": (7, 50, 2, 128), "cache_batch_idx": (2,)}),
    ("append", "paged", {"rotary_cos": (40, 16), "rotary_sin": (40, 16)}), ("append", "contiguous", {"k_cache": (3, 50, 2, 64), "v_cache": (3, 50, 2, 128)}),
    ("append", "paged", {"v_cache": (10, 16, 2, 128)}), ("append", "packed", {"vnew": (7, 2, 128)}), ("prefill", "paged", {"v_pool": (10, 16, 2, 64)}),
    ("decode", "paged", {"v_cache": (10, 16, 2, 64)}), ("decode", "contiguous", {"v_cache": (3, 50, 2, 64)}),
    ("decode", "packed keys", {"v_cache": (71, 2, 64)}), ("fp8", "packed", {"v": (71, 2, 64)}),
    ("prefill", "paged", {"seqlen_k": (5,)}), ("prefill", "packed", {"cu_seqlens_q": (6,)}),
    ("decode", "paged", {"seqlen_k": (5,)}), ("decode", "contiguous", {"k_cache": (3, 50, 2, 64), "v_cache": (3, 50, 2, 64)}),
    ("decode", "contiguous", {"k_cache": (1, 50, 2, 64), "v_cache": (1, 50, 2, 64), "cache_batch_idx": (2,)}),
    ("decode", "paged", {"workspace": ((2, 4, 8, 1), (2, 4, 8, 1, 64))}), ("fp8", "batch", {"k": (3, 50, 2, 64), "v": (3, 50, 2, 64)}),
]


@pytest.mark.parametrize("what,form,other", FITS)
def test_accepted(monkeypatch, what, form, other):
    def stop(device):
        raise Launched
    monkeypatch.setattr(fmha, "_on", stop)  # (the last step before the C call)
    fn, sizes, _, elem = CALLS[what]
    with FakeTensorMode(), pytest.raises(Launched):
        fn(**_tensors(sizes(form) | other, "cuda", elem))


_ORDER = {
    "append": ("_call_append_kv", lambda s: [s["q"], s["k_cache"], s["v_cache"], s["knew"], s["vnew"], s["seqlen_k"], s["rotary_cos"],
                                             s["rotary_sin"], 1, s.get("rotary_dim"), s["block_table"], s.get("cu_seqlens_q"),
                                             s.get("cu_seqlens_knew")]),
    "prefill": ("_call_paged_prefill", lambda s: [s["q"], s["k_pool"], s["v_pool"], s["block_table"], s["seqlen_k"], s.get("cu_seqlens_q"),
                                                  s.get("max_seqlen_q", 0), None, True, (-1, -1), None, False]),
    "decode": ("_call_splitkv", lambda s: [s["q"], s["k_cache"], s["v_cache"], s["seqlen_k"], s["block_table"], s.get("cu_seqlens_q"),
                                           s.get("max_seqlen_q", 0), 0, None, False, (-1, -1), None, False]),
}


@pytest.mark.gpu
@pytest.mark.parametrize("what,n", [(w, n) for w in _ORDER for n in range(len(CALLS[w][2]))])
def test_left_alone_by_the_binding(what, n):
    _, sizes, wrong, elem = CALLS[what]
    form, other = wrong[n]
    if form == "packed keys" or "workspace" in other or "cache_batch_idx" in other:
        pytest.skip("a form that the binding is not asked for")
    name, order = _ORDER[what]
    native = fmha._native()
    assert native and getattr(native, name)(*order(_tensors(sizes(form) | other, "cuda", elem))) is None


@pytest.mark.parametrize("what,other", [
    ("prefill", {"v_pool": (9, 16, 1, 64)}), ("prefill", {"v_pool": (8, 16, 2, 64)}), ("prefill", {"seqlen_k": (1,)}),
    ("decode", {"v_cache": (9, 16, 1, 64)}), ("decode", {"v_cache": (9, 8, 2, 64)}), ("decode", {"seqlen_k": (1,)}),
    ("append", {"knew": (2, 3, 4, 64), "vnew": (2, 3, 4, 128)}), ("append", {"k_cache": (9, 16, 2, 32)}), ("append", {"v_cache": (9, 8, 2, 128)}),
    ("append", {"v_cache": (9, 16, 2, 64)}), ("append", {"rotary_sin": (40, 16)}), ("append", {"q": (2, 3, 4, 32)}),
    ("append", {"block_table": None, "k_cache": (1, 50, 2, 64), "v_cache": (1, 50, 2, 128)}),
])
def test_refused_by_the_binding_functions(what, other):
    from flashck_b200 import flash_ck
    with FakeTensorMode(), pytest.raises(RuntimeError, match="inconsistent|must have|must fit|do not fit|one row per sequence|one shape"):
        s = _tensors(CALLS[what][1]("paged") | other, "cuda")
        if what == "prefill":
            flash_ck.fmha_fwd_paged_kv_prefill(s["q"], s["k_pool"], s["v_pool"], s["block_table"], s["seqlen_k"])
        elif what == "decode":
            flash_ck.fmha_fwd_splitkv(s["q"], s["k_cache"], s["v_cache"], s["seqlen_k"], s["block_table"])
        else:
            flash_ck.fmha_fwd_appendkv(s["q"], s["k_cache"], s["v_cache"], s["knew"], s["vnew"], s["seqlen_k"], s["rotary_cos"],
                                       s["rotary_sin"], 1, s["block_table"])
