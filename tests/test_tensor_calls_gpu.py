"""The C++ calls that take tensors against the Python front-ends' own path: same results, same refusals."""
import contextlib

import pytest
import torch

from fluidmoe_b200.ops import elementwise, flash, gemm, norm, rope

pytestmark = pytest.mark.gpu
BF, F32 = torch.bfloat16, torch.float32


@contextlib.contextmanager
def _general(monkeypatch):
    with monkeypatch.context() as m:
        for mod in (gemm, elementwise, flash):
            for name in [n for n in vars(mod) if n.startswith("_t_")]:
                m.setattr(mod, name, lambda *a: None)
        yield


def _same(x, y, exact=True):
    if isinstance(x, (tuple, list)):
        assert len(x) == len(y)
        for a, b in zip(x, y):
            _same(a, b, exact)
    elif x is None:
        assert y is None
    else:
        assert x.shape == y.shape and x.dtype == y.dtype and x.stride() == y.stride()
        if exact:
            assert torch.equal(x, y)
        else:
            # sums of n fp32 parts in two orders: n * 2^-24 of the sum of magnitudes; parts are of one size here
            assert (x - y).abs().max() <= 1e-5 * y.abs().max()


@contextlib.contextmanager
def _recorded(monkeypatch):
    """Names of the C++ calls in the order made, with whether they took their arguments."""
    made = []

    def recorder(name, call):
        def run(*args):
            res = call(*args)
            made.append((name, res is not None))
            return res
        return run
    with monkeypatch.context() as m:
        for mod in (gemm, elementwise, flash):
            for name in [n for n in vars(mod) if n.startswith("_t_")]:
                m.setattr(mod, name, recorder(name, getattr(mod, name)))
        yield made


def _both(monkeypatch, fn, exact=True, native=True):
    """``fn`` by a C++ call and by the general path: the same results.  ``native``: the call takes this form; else it
    hands it back, and the general path does it both times."""
    before = gemm.LAUNCHES + elementwise.LAUNCHES + flash.LAUNCHES
    with _recorded(monkeypatch) as made:
        got = fn()
    assert made and all(taken == native for _, taken in made), made
    mid = gemm.LAUNCHES + elementwise.LAUNCHES + flash.LAUNCHES
    with _general(monkeypatch):
        want = fn()
    assert gemm.LAUNCHES + elementwise.LAUNCHES + flash.LAUNCHES - mid == mid - before > 0
    _same(got, want, exact)
    gemm.check_status()


def _r(*s, dtype=BF):
    return torch.randn(*s, device="cuda", dtype=F32).to(dtype)


@pytest.mark.parametrize("layout", ["kn", "nk"])
@pytest.mark.parametrize("form", ["plain", "fp32", "wide_a", "wide_b", "out", "out_fp32", "accumulate", "residual", "alpha",
                                  "stacked", "grouped", "grouped_hole"])
def test_gemm_forms(monkeypatch, layout, form):
    torch.manual_seed(0)
    M, K, N, G = 200, 128, 136, 3
    a = _r(M, K + 8)[:, :K] if form == "wide_a" else _r(M, K)
    shape = (K, N) if layout == "kn" else (N, K)
    if form in ("stacked", "grouped", "grouped_hole"):
        b = _r(G, *shape)
    elif form == "wide_b":
        b = _r(shape[0], shape[1] + 8)[:, :shape[1]]
    else:
        b = _r(*shape)
    kw = dict(b_layout=layout)
    if form == "fp32":
        kw.update(out_dtype=F32)
    if form == "stacked":
        a = _r(G * 72, K)
        kw.update(uniform_rows=72)
    if form.startswith("grouped"):
        a = _r(256, K)
        kw.update(group_rows=torch.tensor([64, 5, 60], dtype=torch.int32, device="cuda"),
                  group_offs=torch.tensor([0, 64, 128], dtype=torch.int32, device="cuda"), zero_fill=form == "grouped")
    if form == "alpha":
        kw.update(alpha=0.5, alpha_dev=torch.tensor(3.0, device="cuda"))
    if form == "residual":
        kw.update(residual=_r(M, N))
    base = _r(M, N + 8)

    def run():
        if form in ("out", "accumulate"):
            out = base.clone()[:, :N]
            gemm.grouped_gemm(a, b, out=out, accumulate=form == "accumulate", **kw)
            return out
        if form == "out_fp32":
            out = base.float()[:, :N]
            gemm.grouped_gemm(a, b, out=out, **kw)
            return out
        got = gemm.grouped_gemm(a, b, **kw)
        if form == "grouped_hole":       # rows outside the groups are undefined
            return got[:64], got[64:69], got[128:188]
        return got
    if form == "grouped_hole":
        with _recorded(monkeypatch) as made:
            got = run()
        assert made == [("_t_gemm", True)]
        with _general(monkeypatch):
            _same([g.clone() for g in got], [g.clone() for g in run()])
        return
    _both(monkeypatch, run)


@pytest.mark.parametrize("activation", ["gelu", "silu", "swiglu", "none"])
@pytest.mark.parametrize("probs,save,grouped", [(True, True, False), (False, False, False), (True, True, True)])
def test_expert_forms(monkeypatch, activation, probs, save, grouped):
    torch.manual_seed(1)
    G, H, F = 2, 128, 136 if activation == "swiglu" else 72
    M = 192
    a, w1 = _r(M, H), _r(G, H, F * (2 if activation == "swiglu" else 1))
    w2, p = _r(G, F, H), torch.rand(M, device="cuda") if probs else None
    kw = dict(uniform_rows=M // G)
    if grouped:
        kw = dict(group_rows=torch.tensor([70, 60], dtype=torch.int32, device="cuda"),
                  group_offs=torch.tensor([0, 128], dtype=torch.int32, device="cuda"))
    _both(monkeypatch, lambda: gemm.grouped_gemm_act(a, w1, p, activation=activation, save_pre=save, **kw))
    pre = _r(M, w1.shape[2])
    _both(monkeypatch, lambda: gemm.grouped_gemm_dact(a, w2, pre, p, activation=activation, **kw)[0])
    _both(monkeypatch, lambda: gemm.grouped_gemm_dact(a, w2, pre, p, activation=activation, **kw)[1], exact=False)


@pytest.mark.parametrize("dtype,accumulate,grouped", [(F32, False, False), (F32, True, False), (BF, False, False),
                                                      (F32, False, True)])
def test_weight_gradient_forms(monkeypatch, dtype, accumulate, grouped):
    torch.manual_seed(2)
    a, dy = _r(192, 72), _r(192, 264)
    kw = dict(uniform_rows=64)
    if grouped:
        kw = dict(group_rows=torch.tensor([64, 0, 64], dtype=torch.int32, device="cuda"),
                  group_offs=torch.tensor([0, 64, 128], dtype=torch.int32, device="cuda"))
    base = _r(3, 72, 264, dtype=dtype)

    def run():
        out = base.clone()
        gemm.grouped_gemm_wgrad(a, dy, 3, out=out, accumulate=accumulate, **kw)
        return out
    _both(monkeypatch, run)
    _both(monkeypatch, lambda: gemm.grouped_gemm_wgrad(a, dy, 3, **kw))


@pytest.mark.parametrize("T", [1, 200])
@pytest.mark.parametrize("kind,bias,residual", [("layernorm", True, True), ("layernorm", False, False),
                                                ("rmsnorm", False, True), ("rmsnorm", True, False)])
def test_norm_forms(monkeypatch, T, kind, bias, residual):
    torch.manual_seed(3)
    x, w, b = _r(T, 264), _r(264), _r(264) if bias else None
    _both(monkeypatch, lambda: norm.norm_fwd(x, w, b, 1e-5, kind))
    y, mean, rstd = norm.norm_fwd(x, w, b, 1e-5, kind)
    dy, res = _r(T, 264), _r(T, 264) if residual else None
    _both(monkeypatch, lambda: norm.norm_bwd(dy, x, w, mean, rstd, kind, bias, res))
    wide = _r(T, 528)[:, :264]                     # a strided gradient takes the general path
    _both(monkeypatch, lambda: norm.norm_bwd(wide, x, w, mean, rstd, kind, bias, res), native=T == 1)


def test_row_and_routing_forms(monkeypatch):
    torch.manual_seed(4)
    x, idx = _r(50, 72), torch.randint(0, 50, (77,), device="cuda")
    _both(monkeypatch, lambda: elementwise.gather_rows(x, idx))
    _both(monkeypatch, lambda: elementwise.gather_rows(x, idx.int()), native=False)
    _both(monkeypatch, lambda: elementwise.gather_rows(x, idx, torch.empty(77, 72, device="cuda", dtype=BF)))
    slot = torch.randint(-1, 50, (33, 3), device="cuda", dtype=torch.int32)
    res = _r(33, 72)
    _both(monkeypatch, lambda: elementwise.unpermute_reduce(x, slot, res))
    _both(monkeypatch, lambda: elementwise.unpermute_reduce(x, slot.long()), native=False)
    logits = _r(40, 16, dtype=F32)
    _both(monkeypatch, lambda: elementwise.topk_softmax(logits, 3))
    _both(monkeypatch, lambda: elementwise.topk_softmax(_columns(logits), 3), native=False)
    top, pr = elementwise.topk_softmax(logits, 3)
    _both(monkeypatch, lambda: elementwise.moe_plan(top, pr, 16, 8))


def _columns(t):
    return t.t().contiguous().t()


@pytest.mark.parametrize("s,b,G,qpg", [(130, 2, 1, 2), (1, 1, 2, 1)])
def test_attention_forms(monkeypatch, s, b, G, qpg):
    torch.manual_seed(5)
    qkv = _r(s, b, G, (qpg + 2) * 128)
    freqs = rope.make_rope_freqs(s, 64, device="cuda")
    _both(monkeypatch, lambda: rope.rope_packed_(qkv.clone(), freqs, qpg, 128))
    _both(monkeypatch, lambda: rope.rope_packed_(qkv.clone(), freqs, qpg, 128, backward=True))
    _both(monkeypatch, lambda: flash.flash_attn_fwd_packed(qkv, qpg, 128, 0.1))
    out, lse = flash.flash_attn_fwd_packed(qkv, qpg, 128, 0.1)
    dout = _r(s, b, G * qpg, 128)
    # one K/V block walks its query tiles in one order; dQ of two blocks is a sum of two terms, in either order the same
    _both(monkeypatch, lambda: flash.flash_attn_bwd_packed(dout, qkv, out, lse, qpg, 128, 0.1, head_split=False))


def test_refusals_stay():
    a, b = _r(16, 64), _r(64, 32)
    with pytest.raises(AssertionError):
        gemm.grouped_gemm(a.float(), b)
    with pytest.raises(AssertionError):
        gemm.grouped_gemm(a, _r(64, 33))
    with pytest.raises(AssertionError):
        gemm.grouped_gemm(a.t().contiguous().t(), b)
    with pytest.raises(AssertionError):
        gemm.grouped_gemm(a, b, residual=_r(16, 24))
    with pytest.raises(AssertionError):
        gemm.grouped_gemm(a, _r(2, 64, 32))
    with pytest.raises(AssertionError):
        gemm.grouped_gemm(a, b, alpha_dev=torch.ones(2, device="cuda"))
    with pytest.raises(RuntimeError):
        gemm.grouped_gemm(_r(17, 64).view(-1)[1:1 + 16 * 64].view(16, 64), b)      # operand off 16 bytes
    with pytest.raises(RuntimeError):
        flash.flash_attn_fwd_packed(_r(16, 1, 1, 192), 1, 64, 0.1)


def test_deterministic_mode_still_fills(monkeypatch):
    """torch.empty fills with NaN in deterministic mode; so does the allocation of these calls."""
    a, w = _r(64, 64), _r(1, 64, 32)
    torch.use_deterministic_algorithms(True, warn_only=True)
    try:
        out = gemm.grouped_gemm(a, w, group_rows=torch.tensor([8], dtype=torch.int32, device="cuda"),
                                group_offs=torch.tensor([0], dtype=torch.int32, device="cuda"), zero_fill=False)
        assert out[8:].isnan().all()
    finally:
        torch.use_deterministic_algorithms(False)


def test_status_words_are_those_of_the_tensor_s_device(monkeypatch):
    """A call reports where ``check_status(tensor.device)`` looks, also when words for a device without an index came
    first."""
    monkeypatch.setattr(gemm, "_STATUS", {})
    monkeypatch.setattr(gemm, "_STATUS_PTR", {})
    x = _r(8, 8)
    unnamed = gemm.status_buffer("cuda")
    assert gemm.status_ptr(x) == gemm.status_buffer(x.device).data_ptr() != unnamed.data_ptr()
    gemm.status_buffer(x.device)[0] = 1
    gemm.check_status("cuda")
    with pytest.raises(gemm.FluidKernelTimeout):
        gemm.check_status(x.device)
