"""The compiled calls (csrc/pybind/calls.cpp) against the Python of ops/fmha.py: what they take gives the same bits, what they
cannot check completely they leave alone, and what was refused is refused with the same words."""
import pytest
import torch

from flashck_b200 import ops
from flashck_b200.ops import fmha
from flashck_b200.utils import flags
from flashck_b200.utils.inputs import make_paged_cache, normal_tensor, rotary_cos_sin, to_seqstarts


def _binding():
    native = fmha._native()
    assert native, "the binding has not been built"
    return native


def test_number_of_splits():
    native = _binding()
    for batch in [*range(1, 300), 1000]:
        for rows in (1, 4, 16, 17, 128):
            assert native._num_splits(batch, rows) == ops.default_num_splits(batch, rows_per_kv_head=rows)


def test_leaves_alone_what_is_not_plain():
    native, x = _binding(), torch.zeros(2, 8, 2, 64, dtype=torch.bfloat16)
    for q in (x, x[:, ::2], None, "q", x.to_sparse()):
        assert native._call_forward(q, q, q, None, None, 0, None, False, (-1, -1), None, False, 0.0) is None
    assert native._call_forward(x, x) is None
    with pytest.raises(ValueError, match="must be a CUDA tensor"):
        ops.fmha_fwd(x, x, x)


def test_tuning_takes_the_python_path(monkeypatch):
    monkeypatch.setattr(flags.flag("FC_TUNING_DB_DIR"), "value", "/tmp")
    assert not fmha._native()


def _both(monkeypatch, call, state):
    """The call through the binding and through Python, each on copies of the state: (result or error, state) twice."""
    out, taken = [], []
    native = _binding()
    for on in (True, False):
        s = {k: v.clone() if isinstance(v, torch.Tensor) and v.is_contiguous() else v for k, v in state.items()}
        with monkeypatch.context() as m:
            if on:
                class Spy:
                    def __getattr__(self, name):
                        def f(*a):
                            r = getattr(native, name)(*a)
                            taken.append(r is not None)
                            return r
                        return f
                m.setattr(fmha, "_NATIVE", Spy())
            else:
                m.setattr(fmha, "_NATIVE", False)
            try:
                r = call(**s)
            except (RuntimeError, ValueError, TypeError) as e:
                r = (type(e), str(e))
        out.append((r, s))
    return out, taken


def _same(a, b):
    if isinstance(a, torch.Tensor):
        return a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)
    if isinstance(a, (tuple, list)):
        return len(a) == len(b) and all(_same(x, y) for x, y in zip(a, b))
    return a == b


def _check(monkeypatch, call, state, native):
    (a, b), taken = _both(monkeypatch, call, state)
    assert _same(a[0], b[0])
    for k, v in state.items():
        if isinstance(v, torch.Tensor):
            assert torch.equal(a[1][k], b[1][k])
    assert taken == [native]


def _qkv(b, n, m, hq, hkv, d, dtype=torch.bfloat16):
    return {"q": normal_tensor((b, n, hq, d), dtype, 1).cuda(), "k": normal_tensor((b, m, hkv, d), dtype, 2).cuda(),
            "v": normal_tensor((b, m, hkv, d), dtype, 3).cuda()}


@pytest.mark.gpu
@pytest.mark.parametrize("kw,native", [
    ({}, True), ({"causal": True, "return_lse": True}, True), ({"window_size": (64, 3)}, True), ({"window_size": [64, 3]}, False),
    ({"causal": True, "window_size": (20, 9)}, True), ({"mask_type": 1, "window_size": (-1, 0)}, True), ({"mask_type": 3}, True),
    ({"mask_type": 7}, False), ({"scale": 0.5}, True), ({"scale": 1}, False), ({"logits_soft_cap": 20.0}, True),
    ({"logits_soft_cap": 20}, False), ({"causal": 1}, False), ({"return_lse": 1}, False),
])
def test_dense(monkeypatch, kw, native):
    _check(monkeypatch, lambda **s: ops.fmha_fwd(s["q"], s["k"], s["v"], **kw), _qkv(2, 130, 200, 4, 2, 64), native)


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["heads", "hdim", "batch", "dtype", "strided", "keys", "three", "grad", "fp16", "empty", "one"])
def test_dense_forms(monkeypatch, form):
    s = _qkv(2, 70, 70, 4, 2, 128, torch.float16 if form == "fp16" else torch.bfloat16)
    native = form in ("heads", "hdim", "grad", "fp16", "empty", "one")
    if form == "heads":
        s["q"] = normal_tensor((2, 70, 5, 128), torch.bfloat16, 1).cuda()  # refused: 5 heads over 2
    elif form == "hdim":
        s = {k: v[..., :65].contiguous() for k, v in s.items()}            # refused: no instance
    elif form == "batch":
        s["k"] = s["k"][:1].contiguous()
    elif form == "dtype":
        s["v"] = s["v"].half()
    elif form == "strided":
        s["q"] = s["q"].transpose(1, 2)
    elif form == "keys":
        s["v"] = s["v"][:, :69].contiguous()
    elif form == "three":
        s = {k: v[0].contiguous() for k, v in s.items()}
    elif form == "grad":
        s["q"] = s["q"].requires_grad_()
    elif form == "empty":
        s = {k: v[:0].contiguous() for k, v in s.items()}
    elif form == "one":
        s = {k: v[:1, :1].contiguous() for k, v in s.items()}
    _check(monkeypatch, lambda **s: ops.fmha_fwd(s["q"], s["k"], s["v"], return_lse=True), s, native)


@pytest.mark.gpu
def test_modes_and_transforms_stay_in_python(monkeypatch):
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    class Seen(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    class Fn(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(getattr(func, "__name__", ""))
            return func(*args, **(kwargs or {}))

    class Sub(torch.Tensor):
        pass

    s, native = _qkv(1, 40, 40, 2, 2, 64), _binding()
    args = (None, None, 0, None, False, (-1, -1), None, False, 0.0)
    assert native._call_forward(s["q"], s["k"], s["v"], *args) is not None
    assert native._call_forward(s["q"].as_subclass(Sub), s["k"], s["v"], *args) is None
    for mode in (Seen, Fn):
        seen = []
        with mode():
            assert native._call_forward(s["q"], s["k"], s["v"], *args) is None
            ops.fmha_fwd(s["q"], s["k"], s["v"])
        assert any("empty" in x for x in seen)

    def inside(x):
        assert native._call_forward(x, x, x, *args) is None
        assert native._call_forward(s["q"], s["k"], s["v"], *args) is None
        return x * 1
    torch.func.vmap(inside)(torch.stack([s["q"], s["q"]]))


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["plain", "int32", "cpu", "short"])
def test_varlen(monkeypatch, form):
    lens = [100, 1, 0, 77]
    n = sum(lens)
    cu = to_seqstarts(lens).cuda()
    s = {k: v[0] for k, v in _qkv(1, n, n, 4, 2, 128).items()}
    s["cu"] = cu.int() if form == "int32" else cu.cpu() if form == "cpu" else cu
    s["cu_k"] = cu[:-1].contiguous() if form == "short" else s["cu"]
    _check(monkeypatch, lambda **s: ops.fmha_fwd_var_len(s["q"], s["k"], s["v"], s["cu"], s["cu_k"], 100, causal=True,
                                                         return_lse=True), s, form == "plain")


def _paged(lens, tokens, d=128):
    c = make_paged_cache(lens, 2, d, d, 16, torch.bfloat16, seed=5)
    return {"q": normal_tensor((len(lens), tokens, 8, d), torch.bfloat16, 6).cuda(), "k": c.k.cuda(), "v": c.v.cuda(),
            "bt": c.block_table.cuda(), "sl": c.seqlen_k.cuda()}


@pytest.mark.gpu
@pytest.mark.parametrize("tokens", [1, 4, 20])
@pytest.mark.parametrize("form", ["paged", "lse", "splits", "varlen", "contiguous", "no_lens", "int64", "alibi", "rows", "no_table_lens"])
def test_splitkv(monkeypatch, tokens, form):
    s = _paged([500, 33, 2000], tokens)
    kw, native = {"causal": tokens > 1}, form not in ("int64", "alibi", "rows", "no_table_lens")
    if form == "lse":
        kw["return_lse"] = True
    if form == "splits":
        kw["num_splits"] = 5
    if form == "varlen":
        s["q"], s["cu"] = s["q"].flatten(0, 1), to_seqstarts([tokens] * 3).cuda()
        kw["max_seqlen_q"] = tokens
    if form in ("contiguous", "no_lens"):
        s["k"], s["v"] = (normal_tensor((3, 2000, 2, 128), torch.bfloat16, i).cuda() for i in (7, 8))
        s["bt"] = None
    if form in ("no_lens", "no_table_lens"):
        s["sl"] = None
    if form == "int64":
        s["sl"] = s["sl"].long()
    if form == "rows":
        s["bt"] = s["bt"][:2].contiguous()
    if form == "alibi":
        kw["alibi_slopes"] = torch.full((1, 8), 0.1, device="cuda")
    _check(monkeypatch, lambda **s: ops.fmha_fwd_splitkv(s["q"], s["k"], s["v"], seqlen_k=s["sl"], block_table=s["bt"],
                                                         cu_seqlens_q=s.get("cu"), **kw), s, native) if form != "alibi" else \
        ops.fmha_fwd_splitkv(s["q"], s["k"], s["v"], seqlen_k=s["sl"], block_table=s["bt"], **kw)


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["batch", "varlen", "int64", "page"])
def test_paged_prefill(monkeypatch, form):
    s = _paged([500, 133, 200], 100)
    kw = {}
    if form == "varlen":
        s["q"], s["cu"] = s["q"].flatten(0, 1), to_seqstarts([100] * 3).cuda()
        kw["max_seqlen_q"] = 100
    if form == "int64":
        s["bt"] = s["bt"].long()
    if form == "page":  # refused: a table of another batch
        s["bt"] = s["bt"][:2].contiguous()
    _check(monkeypatch, lambda **s: ops.fmha_fwd_paged_kv_prefill(s["q"], s["k"], s["v"], s["bt"], s["sl"], return_lse=True,
                                                                  cu_seqlens_q=s.get("cu"), **kw), s, form in ("batch", "varlen"))


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["batch", "varlen", "no_q", "no_rope", "missing", "half", "contiguous"])
def test_append_kv(monkeypatch, form):
    s = _paged([500, 133, 200], 4)
    s["kn"], s["vn"] = (normal_tensor((3, 4, 2, 128), torch.bfloat16, i).cuda() for i in (7, 8))
    s["cos"], s["sin"] = (t.cuda() for t in rotary_cos_sin(2048, 128, torch.bfloat16))
    s["sl"] = s["sl"] - 4
    kw, native = {}, form != "missing"
    if form == "varlen":
        s["q"], s["kn"], s["vn"] = (s[n].flatten(0, 1) for n in ("q", "kn", "vn"))
        kw = {n: to_seqstarts([4] * 3).cuda() for n in ("cu_seqlens_q", "cu_seqlens_knew")}
    if form == "no_q":
        s["q"] = None
    if form == "no_rope":
        kw["rope"], s["cos"], s["sin"] = 0, None, None
    if form == "missing":
        s["cos"] = None
    if form == "half":
        kw["rope"], kw["rotary_dim"] = 2, 64
        s["cos"], s["sin"] = s["cos"][:, :32].contiguous(), s["sin"][:, :32].contiguous()
    if form == "contiguous":
        s["k"], s["v"] = (normal_tensor((3, 600, 2, 128), torch.bfloat16, i).cuda() for i in (9, 10))
        s["bt"] = None
    _check(monkeypatch, lambda **s: ops.fmha_fwd_append_kv(s["q"], s["k"], s["v"], s["kn"], s["vn"], s["sl"], s["cos"], s["sin"],
                                                           block_table=s["bt"], **kw), s, native)
