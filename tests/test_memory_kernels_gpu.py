"""Memory-bound kernels at the edges of their work split, against 64-bit arithmetic."""
import pytest
import torch

from fluidmoe_b200.ops import norm, permute

pytestmark = pytest.mark.gpu


def _rand(*shape):
    return torch.randn(*shape, device="cuda").to(torch.bfloat16)


@pytest.mark.parametrize("T", [1, 295, 297, 600])
@pytest.mark.parametrize("H", [8, 520, 2048, 2056, 4104, 8192])
@pytest.mark.parametrize("kind", ["rmsnorm", "layernorm"])
@pytest.mark.parametrize("with_res", [False, True])
def test_norm_backward(T, H, kind, with_res):
    torch.manual_seed(T + H)
    x, dy, w, res = _rand(T, H), _rand(T, H), _rand(H), _rand(T, H)
    b = _rand(H) if kind == "layernorm" else None
    _, mean, rstd = norm.norm_fwd(x, w, b, 1e-5, kind)
    dx, dw, db = norm.norm_bwd(dy, x, w, mean, rstd, kind, b is not None, res if with_res else None)
    r = rstd.double()[:, None]
    xh = (x.double() - (mean.double()[:, None] if mean is not None else 0.0)) * r
    g = dy.double() * w.double()
    c2 = g.mean(-1, keepdim=True) if mean is not None else 0.0
    ref = (g - c2 - xh * (g * xh).mean(-1, keepdim=True)) * r + (res.double() if with_res else 0.0)
    # one rounding of bf16; fp32 sums of H terms before it
    assert ((dx.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * ref.abs().max()).all()
    terms = (dy.double() * xh).abs().sum(0)
    assert ((dw.double() - (dy.double() * xh).sum(0)).abs() <= 2e-6 * terms + 1e-6).all()
    if db is not None:
        assert ((db.double() - dy.double().sum(0)).abs() <= 2e-6 * dy.double().abs().sum(0) + 1e-6).all()


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 6, 7, 8, 9, 16])
@pytest.mark.parametrize("T,H", [(1, 8), (65, 72), (130, 2048)])
@pytest.mark.parametrize("with_res", [False, True])
def test_unpermute(k, T, H, with_res):
    """fp32 sums in the order residual, choice 0, 1, ...: the same bytes as that loop gives."""
    torch.manual_seed(k)
    rows, res = _rand(T * k, H), _rand(T, H)
    slot = torch.randperm(T * k, device="cuda").view(T, k).to(torch.int32)
    slot[torch.rand(T, k, device="cuda") < 0.2] = -1
    got = permute.unpermute_reduce(rows, slot, res if with_res else None)
    acc = res.float() if with_res else torch.zeros(T, H, device="cuda")
    for j in range(k):
        s = slot[:, j].long()
        acc = torch.where((s >= 0)[:, None], acc + rows[s.clamp(min=0)].float(), acc)
    assert torch.equal(got, acc.to(torch.bfloat16))


@pytest.mark.parametrize("T", [1, 31, 33, 1531])
@pytest.mark.parametrize("H,E", [(4, 1), (2, 3), (264, 8), (512, 16), (520, 17), (1028, 64), (2048, 70)])
def test_router_weight_gradient(T, H, E):
    from fluidmoe_b200.ops import router
    torch.manual_seed(T + E)
    x, dl = _rand(T, H), torch.randn(T, E, device="cuda")
    got = router.router_wgrad(x, dl)
    ref = x.double().t() @ dl.double()
    # fp32 sums of T products in an order of their own
    assert ((got.double() - ref).abs() <= 1e-6 * (x.double().abs().t() @ dl.double().abs()) + 1e-30).all()


@pytest.mark.parametrize("T", [1535, 1536, 1537, 2111])
@pytest.mark.parametrize("H,E", [(8, 1), (120, 8), (264, 17), (520, 64), (2048, 66), (136, 200), (1028, 64)])
@pytest.mark.parametrize("offset", [0, 4])
def test_router_weight_gradient_of_many_tokens(T, H, E, offset):
    """Edges of the tensor core's tiles and rule; rows of 8 bytes and a base of 8 bytes, which it does not take."""
    from fluidmoe_b200.ops import elementwise
    torch.manual_seed(T + E)
    x = _rand(T * H + offset)[offset:].view(T, H)
    dl = torch.randn(T, E, device="cuda") * torch.logspace(-3, 3, E, device="cuda")
    got, ref = elementwise.router_wgrad(x, dl), x.double().t() @ dl.double()
    # sums of 64 tokens cut off at 2^-23 five times at the most, then few dozens of them rounded to 2^-24
    assert ((got.double() - ref).abs() <= 2.4e-6 * (x.double().abs().t() @ dl.double().abs())).all()


@pytest.mark.parametrize("T", [1536, 1600, 2048, 8192])
@pytest.mark.parametrize("H,E", [(264, 8), (520, 64), (2048, 16)])
@pytest.mark.parametrize("signs", ["one", "both"])
def test_router_weight_gradient_has_every_bit_of_its_operand(T, H, E, signs):
    """All three bf16 parts of a gradient count.  Two of them hold 16 bits, cut off, which loses 2^-16 of a value of [1, 2)
    on average and 1e-5 of the sum.  The kernel's own error: sums of 32 tokens, cut off at 2^-23 in each of two steps, and
    the roundings of the running sum of those, 2^-24 of it each and of random sign, for which as much again is left."""
    from fluidmoe_b200.ops import elementwise
    torch.manual_seed(T + E)
    x, dl = _rand(T, H), torch.randn(T, E, device="cuda")
    if signs == "one":
        x, dl = x.abs(), 1.0 + torch.rand(T, E, device="cuda")
    got, ref = elementwise.router_wgrad(x, dl).double(), x.double().t() @ dl.double()
    cut = (dl.view(torch.int32) & ~0xff).view(torch.float32)              # two parts: 16 bits
    lost = x.double().t() @ cut.double()
    bound = 4 * 2.0 ** -23
    assert (lost - ref).norm() > 5 * bound * ref.norm()
    assert (got - ref).norm() <= bound * ref.norm()


def test_router_weight_gradient_keeps_what_is_not_finite():
    from fluidmoe_b200.ops import elementwise
    torch.manual_seed(0)
    x, dl = _rand(2048, 256), torch.randn(2048, 24, device="cuda")
    x[7, 3], x[100, 9], x[2047, 200] = float("inf"), float("nan"), float("-inf")
    dl[:, 5] = 1.0                                   # its small parts are zeros
    dl[50, 2], dl[60, 3], dl[70, 4], dl[80, 6] = float("inf"), float("nan"), 3.4e38, -1e-40
    x[70, 3] = x[70, 200] = 0                        # or infinities would meet an overflow of the other sign
    got, ref = elementwise.router_wgrad(x, dl), x.double().t() @ dl.double()
    assert torch.equal(got.isnan(), ref.isnan())
    big = ref.abs() > 3.4028235e38
    assert torch.equal(got[big & ~ref.isnan()], ref[big & ~ref.isnan()].float())
    ok = ~big & ~ref.isnan()
    assert ((got.double() - ref).abs()[ok] <= 2.4e-6 * (x.double().abs().t() @ dl.double().abs())[ok]).all()


@pytest.mark.parametrize("T,V,H", [(1, 3, 8), (700, 5, 264), (513, 1000, 1024)])
def test_embedding_gradient(T, V, H):
    from fluidmoe_b200.ops import elementwise
    torch.manual_seed(T)
    ids, dy = torch.randint(0, V, (T,), device="cuda"), _rand(T, H)
    main = torch.randn(V, H, device="cuda")
    ref = main.double().index_add_(0, ids, dy.double())
    terms = main.double().abs().index_add_(0, ids, dy.double().abs())
    assert elementwise.embedding_grad_(main, ids, dy)
    assert ((main.double() - ref).abs() <= 2e-6 * terms).all()


@pytest.mark.parametrize("state", [torch.float32, torch.bfloat16])
def test_adam_over_many_tensors_equals_one_by_one(state):
    """More tensors than one launch's table holds, sizes around the chunk and off the vector width, one base
    off its alignment.  The compiler may contract either kernel's products and sums into fused ones, which
    saves a rounding of 2^-24 of a term; the terms of a moment have one sign or stay below 4 here."""
    from fluidmoe_b200.ops import elementwise
    torch.manual_seed(0)
    sizes = [1, 3, 4, 5, 8191, 8192, 8193, 8195, 40000, 2] + [16] * 60
    kw = dict(lr=1e-2, beta1=0.9, beta2=0.99, eps=1e-8, weight_decay=0.1, step=3, grad_scale=0.5)
    sets = []
    for off, n in enumerate(sizes):
        lead = 1 if off == 6 else 0
        mk = lambda t: torch.cat([torch.zeros(lead, device="cuda"), t]).to(state)[lead:]    # noqa: E731
        p = torch.cat([torch.zeros(lead, device="cuda"), torch.randn(n, device="cuda")]).bfloat16()[lead:]
        sets.append((p, torch.randn(n, device="cuda"), mk(torch.randn(n, device="cuda")), mk(torch.rand(n, device="cuda"))))
    ones = [tuple(t.clone() if i != 6 else torch.cat([t[:1], t])[1:] for t in s) for i, s in enumerate(sets)]
    for p, g, m, v in ones:
        elementwise.adam_step(p, None, g, m, v, **kw)
    elementwise.adam_multi(sets, state == torch.bfloat16, **kw)
    for a, b in zip(sets, ones):
        for x, y in zip(a, b):
            # 4 * 2^-23 of absolute error in fp32 (four roundings), then one rounding of bf16
            rtol = 0.0 if x.dtype == torch.float32 else 2.0 ** -7
            torch.testing.assert_close(x.float(), y.float(), rtol=rtol, atol=4 * 2.0 ** -23 * 4)


@pytest.mark.parametrize("T,H,E", [(1, 8, 8), (33, 264, 16), (700, 2048, 64), (257, 512, 12)])
def test_router_input_gradient(T, H, E):
    from fluidmoe_b200.ops import router
    torch.manual_seed(T)
    dl, w = torch.randn(T, E, device="cuda"), _rand(H, E)
    got = router.router_dgrad(dl, w, torch.bfloat16)
    ref = dl.bfloat16().double() @ w.double().t()
    # fp32 sums of E products, then one rounding of bf16
    assert ((got.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * E ** 0.5).all()


@pytest.mark.parametrize("s,b,G,qpg,d,rot", [(1, 1, 1, 1, 128, 128), (37, 2, 3, 5, 64, 32), (65, 3, 2, 4, 128, 128), (300, 1, 1, 8, 128, 64)])
@pytest.mark.parametrize("backward", [False, True])
def test_rope(s, b, G, qpg, d, rot, backward):
    """Angles of the two halves differ here, as the layout allows; the value head stays as it was."""
    from fluidmoe_b200.ops import rope
    torch.manual_seed(s)
    x, f = _rand(s, b, G, (qpg + 2) * d), torch.randn(s, 1, 1, rot, device="cuda")
    got = rope.rope_packed_(x.clone(), f, qpg, d, backward=backward).view(s, b, G, qpg + 2, d)
    v = x.view(s, b, G, qpg + 2, d).double()
    c, sn = torch.cos(f.double()).view(s, 1, 1, 1, rot), torch.sin(f.double()).view(s, 1, 1, 1, rot)
    (c1, c2), (s1, s2) = c.chunk(2, -1), sn.chunk(2, -1)
    x1, x2 = v[..., :rot].chunk(2, -1)
    o = (x1 * c1 + x2 * s2, x2 * c2 - x1 * s1) if backward else (x1 * c1 - x2 * s1, x2 * c2 + x1 * s2)
    ref = torch.cat((*o, v[..., rot:]), -1)
    ref[..., -1, :] = v[..., -1, :]
    assert ((got.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5).all()
    assert torch.equal(got[..., -1, :], x.view(s, b, G, qpg + 2, d)[..., -1, :])


@pytest.mark.parametrize("T", [1, 295, 593, 1500])
@pytest.mark.parametrize("H", [8, 520, 2048, 2056, 4104, 8192, 8200])
@pytest.mark.parametrize("kind", ["rmsnorm", "layernorm", "layernorm without bias"])
def test_norm_forward(T, H, kind):
    torch.manual_seed(T + H)
    x, w = _rand(T, H) + 0.5, _rand(H)
    b = _rand(H) if kind == "layernorm" else None
    y, mean, rstd = norm.norm_fwd(x, w, b, 1e-5, kind.split()[0])
    xd = x.double()
    mu = xd.mean(-1, keepdim=True) if kind != "rmsnorm" else torch.zeros(T, 1, device="cuda", dtype=torch.float64)
    r = torch.rsqrt((xd - mu).pow(2).mean(-1, keepdim=True) + 1e-5)
    ref = (xd - mu) * r * w.double() + (b.double() if b is not None else 0.0)
    # fp32 sums of H terms, then one rounding of bf16
    assert ((y.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * ref.abs().max()).all()
    assert ((rstd.double() - r.squeeze(1)).abs() <= 1e-5 * r.squeeze(1)).all()
    assert mean is None or ((mean.double() - mu.squeeze(1)).abs() <= 1e-5).all()


@pytest.mark.parametrize("H", [520, 4096, 8192])
def test_rms_norm_backward_with_a_bias_gradient(H):
    """RMSNorm has no bias, but the call returns the column sums of dy when asked for a bias gradient."""
    torch.manual_seed(H)
    x, dy, w = _rand(300, H), _rand(300, H), _rand(H)
    _, _, rstd = norm.norm_fwd(x, w, None, 1e-5, "rmsnorm")
    dx, dw, db = norm.norm_bwd(dy, x, w, None, rstd, "rmsnorm", True)
    dx2, dw2, none = norm.norm_bwd(dy, x, w, None, rstd, "rmsnorm", False)
    assert none is None and torch.equal(dx, dx2) and torch.equal(dw, dw2)
    assert ((db.double() - dy.double().sum(0)).abs() <= 2e-6 * dy.double().abs().sum(0) + 1e-6).all()


def test_adam_updates_tied_parameters_one_after_the_other():
    """A parameter that is listed twice, and two parameters over one array (moments of their own each)."""
    from fluidmoe_b200.ops import elementwise
    from fluidmoe_b200.ops.optim import FusedAdam
    torch.manual_seed(9)
    n, hyper = 100_000, dict(lr=1e-2, weight_decay=0.1)
    w, w0, g, g2 = _rand(n), _rand(n), torch.randn(n, device="cuda"), torch.randn(n, device="cuda")
    w.copy_(w0)
    p, tied, others = torch.nn.Parameter(w), torch.nn.Parameter(w), [torch.nn.Parameter(_rand(64)) for _ in range(3)]
    p.main_grad, tied.main_grad = g, g2
    for o in others:
        o.main_grad = torch.randn(64, device="cuda")
    opt = FusedAdam([p, others[0], tied, others[1], p, others[2]], **hyper)
    opt.step()
    m, v, m2, v2 = (torch.zeros(n, device="cuda") for _ in range(4))
    for grad, a, b in ((g, m, v), (g2, m2, v2), (g, m, v)):
        elementwise.adam_multi([(w0, grad, a, b)], False, hyper["lr"], 0.9, 0.999, 1e-8, hyper["weight_decay"], 1)
    assert torch.equal(w, w0)
    for q, a, b in ((p, m, v), (tied, m2, v2)):
        assert torch.equal(opt.state[id(q)]["m"], a) and torch.equal(opt.state[id(q)]["v"], b)


@pytest.mark.parametrize("count", [1, 2])
def test_adam_of_one_tensor_takes_the_kernel_for_one(count, monkeypatch):
    from fluidmoe_b200.ops import elementwise
    from fluidmoe_b200.ops.optim import FusedAdam
    calls = []
    for name in ("adam_step", "adam_multi"):
        real = getattr(elementwise, name)
        monkeypatch.setattr(elementwise, name, lambda *a, _n=name, _f=real, **kw: (calls.append(_n), _f(*a, **kw)))
    params = [torch.nn.Parameter(_rand(1000 + i)) for i in range(count)]
    start = [p.detach().double() for p in params]
    for p in params:      # gradients well above eps
        p.main_grad = torch.where(torch.rand(p.shape, device="cuda") < 0.5, -1.0, 1.0) * (torch.rand(p.shape, device="cuda") + 0.1)
    FusedAdam(params, lr=1e-2, weight_decay=0.1).step()
    assert calls == (["adam_step"] if count == 1 else ["adam_multi"])
    for p, s in zip(params, start):
        # the first step moves a weight by lr * (sign of the gradient + decay), then one rounding of bf16
        ref = s - 1e-2 * (torch.sign(p.main_grad.double()) + 0.1 * s)
        assert ((p.detach().double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5).all()


@pytest.mark.parametrize("s,G,qpg,d,rot", [(1, 1, 32, 128, 128), (64, 1, 32, 128, 128), (300, 1, 7, 128, 64), (590, 2, 32, 64, 64),
                                           (595, 1, 70, 128, 128), (64, 8, 4, 128, 128), (4700, 1, 2, 128, 128)])
@pytest.mark.parametrize("backward", [False, True])
def test_rope_with_the_heads_split_over_threads(s, G, qpg, d, rot, backward):
    """Few rows and many heads: each head once, also where the split does not divide them; the same bytes as with
    every group as a tensor of its own."""
    from fluidmoe_b200.ops import rope
    torch.manual_seed(s)
    x, f = _rand(s, 1, G, qpg + 2, d), torch.randn(s, 1, 1, rot, device="cuda")
    got = rope.rope_packed_(x.clone().view(s, 1, G, -1), f, qpg, d, backward=backward).view_as(x)
    for h in range(qpg + 1):
        # one rotated head and a value head
        one = torch.cat((x[:, :, :, h:h + 1], x[:, :, :, h:h + 1], x[:, :, :, -1:]), 3).contiguous()
        ref = rope.rope_packed_(one.view(s, 1, G, -1), f, 1, d, backward=backward).view_as(one)
        assert torch.equal(got[:, :, :, h], ref[:, :, :, 0])
    assert torch.equal(got[:, :, :, -1], x[:, :, :, -1])


@pytest.mark.parametrize("T", [1, 31, 33, 1531])
@pytest.mark.parametrize("H,E", [(4, 1), (2, 3), (264, 8), (512, 16), (520, 17), (1028, 64), (2048, 70)])
def test_router_weight_gradient_kernel(T, H, E):
    """The kernel itself, also at the sizes that ``ops.router`` leaves to the library."""
    from fluidmoe_b200.ops import elementwise
    torch.manual_seed(T + E)
    x, dl = _rand(T, H), torch.randn(T, E, device="cuda")
    got = elementwise.router_wgrad(x, dl)
    assert (got is None) == (H % 4 != 0)
    if got is not None:
        ref, terms = x.double().t() @ dl.double(), x.double().abs().t() @ dl.double().abs()
        # fp32 sums of T terms, a few hundred at a time
        assert ((got.double() - ref).abs() <= 2e-6 * terms).all()


@pytest.mark.parametrize("T,H,E,kernel", [(127, 64, 8, False), (128, 64, 8, True), (511, 512, 32, False), (512, 512, 32, True),
                                          (512, 2048, 64, True), (512, 2056, 64, False), (1024, 2056, 64, True),
                                          (600, 1024, 128, True), (600, 1032, 128, False), (600, 256, 161, False)])
def test_router_weight_gradient_takes_the_kernel_where_it_pays(T, H, E, kernel):
    from fluidmoe_b200.ops import elementwise, router
    torch.manual_seed(T)
    x, dl = _rand(T, H), torch.randn(T, E, device="cuda")
    before = elementwise.LAUNCHES
    got = router.router_wgrad(x, dl)
    assert (elementwise.LAUNCHES > before) == kernel
    ref, terms = x.double().t() @ dl.double(), x.double().abs().t() @ dl.double().abs()
    # fp32 sums of T terms in either path: 2^-24 of their absolute sum a step, T steps at the worst, sqrt(T) as a rule
    assert ((got.double() - ref).abs() <= 4 * T ** 0.5 * 2.0 ** -24 * terms).all()


@pytest.mark.parametrize("k", [9, 10, 11, 12, 13, 14, 15, 16])
@pytest.mark.parametrize("T,H", [(1, 8), (65, 72), (130, 2048)])
@pytest.mark.parametrize("with_res", [False, True])
def test_unpermute_in_rounds(k, T, H, with_res):
    """More choices than one round holds: whole rounds, cut ones and choices without a row anywhere; the same
    bytes as the loop over the choices gives."""
    torch.manual_seed(k)
    rows, res = _rand(T * k, H), _rand(T, H)
    slot = torch.randperm(T * k, device="cuda").view(T, k).to(torch.int32)
    slot[torch.rand(T, k, device="cuda") < 0.2] = -1
    slot[::3, :8] = -1
    got = permute.unpermute_reduce(rows, slot, res if with_res else None)
    acc = res.float() if with_res else torch.zeros(T, H, device="cuda")
    for j in range(k):
        s = slot[:, j].long()
        acc = torch.where((s >= 0)[:, None], acc + rows[s.clamp(min=0)].float(), acc)
    assert torch.equal(got, acc.to(torch.bfloat16))


@pytest.mark.parametrize("T", [1, 700, 5000, 20_000])
@pytest.mark.parametrize("k", [2, 10])
def test_waiting_unpermute_gives_the_same(T, k):
    """The form that waits for peers, with counters that have arrived: its grid is smaller, so its threads take
    several pieces each."""
    from fluidmoe_b200.ops import elementwise, gemm
    torch.manual_seed(T)
    H = 512
    rows, res = _rand(T * k, H), _rand(T, H)
    slot = torch.randperm(T * k, device="cuda").view(T, k).to(torch.int32)
    flags, waited = torch.full((2,), 5, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int64, device="cuda")
    wait = dict(flags=flags.data_ptr(), n=2, expected=5, wait_ns=waited.data_ptr(), timeout_ns=1_000_000_000,
                status=gemm.status_buffer(rows.device).data_ptr())
    assert torch.equal(elementwise.unpermute_reduce(rows, slot, res, wait), elementwise.unpermute_reduce(rows, slot, res))
    gemm.check_status()


@pytest.mark.parametrize("T,H,E,own", [(64, 512, 8, True), (4095, 2048, 64, True), (4096, 2048, 64, False), (4096, 4096, 8, False)])
def test_router_input_gradient_of_many_rows_goes_to_the_library(T, H, E, own):
    from fluidmoe_b200.ops import gemm, router
    torch.manual_seed(T)
    dl, w = torch.randn(T, E, device="cuda"), _rand(H, E)
    before = gemm.LAUNCHES
    got = router.router_dgrad(dl, w, torch.bfloat16)
    assert (gemm.LAUNCHES > before) == own
    ref = dl.bfloat16().double() @ w.double().t()
    # fp32 sums of E products, then one rounding of bf16
    assert ((got.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * E ** 0.5).all()
