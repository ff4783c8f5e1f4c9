"""tcgen05 GEMM against a PyTorch fp32 reference of the same op."""
import pytest
import torch

from fluidmoe_b200.ops import gemm

pytestmark = pytest.mark.gpu


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(torch.bfloat16)


def _close(got, ref, tol=2e-2):
    got, ref = got.float(), ref.float()
    err = (got - ref).abs().max().item()
    denom = ref.abs().max().item() + 1e-6
    assert err / denom < tol, f"max err {err} vs scale {denom}"


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (128, 128, 128), (256, 512, 256), (300, 520, 192), (1024, 1024, 1024), (77, 72, 72)])
@pytest.mark.parametrize("layout", ["nk", "kn"])
def test_dense(M, N, K, layout):
    torch.manual_seed(0)
    a = _rand(M, K)
    w = _rand(N, K) if layout == "nk" else _rand(K, N)
    out = gemm.grouped_gemm(a, w, b_layout=layout)
    torch.cuda.synchronize()
    gemm.check_status()
    ref = a.float() @ (w.float().t() if layout == "nk" else w.float())
    _close(out, ref)


def test_dense_fp32_accumulate():
    a, w = _rand(256, 128), _rand(384, 128)
    out = torch.ones(256, 384, device="cuda", dtype=torch.float32)
    gemm.grouped_gemm(a, w, b_layout="nk", out=out, accumulate=True, alpha=0.5)
    torch.cuda.synchronize()
    gemm.check_status()
    _close(out, 1.0 + 0.5 * (a.float() @ w.float().t()))


@pytest.mark.parametrize("layout", ["nk", "kn"])
def test_grouped_variable_rows(layout):
    torch.manual_seed(1)
    G, K, N = 4, 128, 320
    rows = torch.tensor([130, 0, 64, 257], dtype=torch.int32)
    offs = torch.tensor([0, 192, 192, 256], dtype=torch.int32)
    total = 256 + 320
    a = _rand(total, K)
    w = _rand(G, N, K) if layout == "nk" else _rand(G, K, N)
    out = gemm.grouped_gemm(a, w, b_layout=layout, group_rows=rows.cuda(), group_offs=offs.cuda())
    torch.cuda.synchronize()
    gemm.check_status()
    for g in range(G):
        o, r = offs[g].item(), rows[g].item()
        wg = w[g].float().t() if layout == "nk" else w[g].float()
        _close(out[o:o + r], a[o:o + r].float() @ wg) if r else None


@pytest.mark.parametrize("act", ["gelu", "silu", "swiglu"])
def test_fc1_act_prob(act):
    torch.manual_seed(2)
    G, H, F, cap = 2, 256, 384, 192
    a = _rand(G * cap, H)
    w = _rand(G, H, 2 * F if act == "swiglu" else F, scale=0.05)
    probs = torch.rand(G * cap, device="cuda")
    out, pre = gemm.grouped_gemm_act(a, w, probs, activation=act, uniform_rows=cap)
    torch.cuda.synchronize()
    gemm.check_status()
    for g in range(G):
        x = a[g * cap:(g + 1) * cap].float() @ w[g].float()
        _close(pre[g * cap:(g + 1) * cap], x)
        ref = gemm.act_ref(x, act) * probs[g * cap:(g + 1) * cap, None]
        _close(out[g * cap:(g + 1) * cap], ref)


@pytest.mark.parametrize("act", ["gelu", "swiglu"])
def test_fc2_dx_dact(act):
    torch.manual_seed(3)
    G, H, F, cap = 2, 256, 384, 160
    dy = _rand(G * cap, H)
    w2 = _rand(G, F, H, scale=0.05)
    pre = _rand(G * cap, 2 * F if act == "swiglu" else F)
    probs = torch.rand(G * cap, device="cuda")
    dpre, dprobs = gemm.grouped_gemm_dact(dy, w2, pre, probs, activation=act, uniform_rows=cap)
    torch.cuda.synchronize()
    gemm.check_status()
    rdpre, rdprobs = gemm.grouped_gemm_dact(dy.cpu(), w2.cpu(), pre.cpu(), probs.cpu(), activation=act, uniform_rows=cap)
    _close(dpre.cpu(), rdpre)
    _close(dprobs.cpu(), rdprobs)


def test_wgrad_grouped():
    torch.manual_seed(4)
    G, M, N = 3, 256, 320
    rows = torch.tensor([128, 70, 200], dtype=torch.int32)
    offs = torch.tensor([0, 128, 256], dtype=torch.int32)
    total = 512
    a, dy = _rand(total, M), _rand(total, N)
    # rows outside the groups must be zero (64-row contraction blocks)
    mask = torch.zeros(total, dtype=torch.bool)
    for o, r in zip(offs.tolist(), rows.tolist()):
        mask[o:o + r] = True
    a[~mask.cuda()] = 0
    out = torch.full((G, M, N), 2.0, device="cuda")
    gemm.grouped_gemm_wgrad(a, dy, G, group_rows=rows.cuda(), group_offs=offs.cuda(), out=out, accumulate=True)
    torch.cuda.synchronize()
    gemm.check_status()
    for g in range(G):
        o, r = offs[g].item(), rows[g].item()
        _close(out[g], 2.0 + a[o:o + r].float().t() @ dy[o:o + r].float())


def test_large_perf_smoke():
    a, w = _rand(4096, 4096), _rand(4096, 4096)
    for _ in range(3):
        out = gemm.grouped_gemm(a, w, b_layout="nk")
    torch.cuda.synchronize()
    s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s.record()
    for _ in range(10):
        out = gemm.grouped_gemm(a, w, b_layout="nk")
    e.record()
    torch.cuda.synchronize()
    gemm.check_status()
    ms = s.elapsed_time(e) / 10
    print(f"\n4096^3 bf16: {ms:.3f} ms, {2 * 4096**3 / ms / 1e9:.1f} TFLOP/s")
    _close(out, a.float() @ w.float().t())


@pytest.fixture
def cta_pair():
    old = gemm.CTA_PAIR
    gemm.CTA_PAIR = 1
    yield
    gemm.CTA_PAIR = old


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (512, 512, 256), (300, 520, 192), (1024, 1024, 1024)])
@pytest.mark.parametrize("layout", ["nk", "kn"])
def test_cta_pair_dense(cta_pair, M, N, K, layout):
    torch.manual_seed(0)
    a = _rand(M, K)
    w = _rand(N, K) if layout == "nk" else _rand(K, N)
    out = gemm.grouped_gemm(a, w, b_layout=layout)
    torch.cuda.synchronize()
    gemm.check_status()
    _close(out, a.float() @ (w.float().t() if layout == "nk" else w.float()))


def test_cta_pair_grouped_fused_epilogues(cta_pair):
    torch.manual_seed(2)
    G, H, F, cap = 2, 256, 384, 320
    a = _rand(G * cap, H)
    w = _rand(G, H, 2 * F, scale=0.05)
    probs = torch.rand(G * cap, device="cuda")
    out, pre = gemm.grouped_gemm_act(a, w, probs, activation="swiglu", uniform_rows=cap)
    dy = _rand(G * cap, H)
    w2 = _rand(G, F, H, scale=0.05)
    dpre, dprobs = gemm.grouped_gemm_dact(dy, w2, pre, probs, activation="swiglu", uniform_rows=cap)
    g1 = gemm.grouped_gemm_wgrad(a, dpre, G, uniform_rows=cap)
    torch.cuda.synchronize()
    gemm.check_status()
    for g in range(G):
        x = a[g * cap:(g + 1) * cap].float() @ w[g].float()
        _close(pre[g * cap:(g + 1) * cap], x)
        _close(out[g * cap:(g + 1) * cap], gemm.act_ref(x, "swiglu") * probs[g * cap:(g + 1) * cap, None])
        _close(g1[g], a[g * cap:(g + 1) * cap].float().t() @ dpre[g * cap:(g + 1) * cap].float())
    rdpre, rdprobs = gemm.grouped_gemm_dact(dy.cpu(), w2.cpu(), pre.cpu(), probs.cpu(), activation="swiglu", uniform_rows=cap)
    _close(dpre.cpu(), rdpre)
    _close(dprobs.cpu(), rdprobs)


def test_cta_pair_speed(cta_pair):
    a, w = _rand(8192, 8192), _rand(8192, 8192)
    for _ in range(3):
        out = gemm.grouped_gemm(a, w, b_layout="nk")
    torch.cuda.synchronize()
    s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s.record()
    for _ in range(10):
        out = gemm.grouped_gemm(a, w, b_layout="nk")
    e.record()
    torch.cuda.synchronize()
    gemm.check_status()
    ms = s.elapsed_time(e) / 10
    print(f"\n8192^3 bf16 (CTA pair): {ms:.3f} ms, {2 * 8192**3 / ms / 1e9:.1f} TFLOP/s")


@pytest.mark.parametrize("cta_pair", [0, 1])
@pytest.mark.parametrize("G,rows_per,M,N", [(2, 256, 256, 512), (3, 128, 384, 264)])
def test_wgrad_adam_epilogue_matches_fp32_reference(G, rows_per, M, N, cta_pair, monkeypatch):
    """Optimizer in the weight-gradient epilogue == fp32 gradient followed by an fp32 AdamW update
    (the PyTorch reference of the same op), up to the bf16 rounding of parameter and moments."""
    monkeypatch.setattr(gemm, "CTA_PAIR", cta_pair)
    torch.manual_seed(5)
    a = torch.randn(G * rows_per, M, device="cuda").bfloat16()
    dy = torch.randn(G * rows_per, N, device="cuda").bfloat16()
    p = (torch.randn(G, M, N, device="cuda") * 0.05).bfloat16()
    m = (torch.randn(G, M, N, device="cuda") * 0.1).bfloat16()
    v = (torch.rand(G, M, N, device="cuda") * 0.1).bfloat16()
    lr, b1, b2, eps, wd, step, gs = 1e-2, 0.9, 0.95, 1e-8, 0.1, 3, 0.25
    g = torch.stack([a[i * rows_per:(i + 1) * rows_per].float().t() @ dy[i * rows_per:(i + 1) * rows_per].float()
                     for i in range(G)]) * gs
    m_ref = b1 * m.float() + (1 - b1) * g
    v_ref = b2 * v.float() + (1 - b2) * g * g
    w = p.float()
    w_ref = w - lr * ((m_ref / (1 - b1 ** step)) / ((v_ref / (1 - b2 ** step)).sqrt() + eps) + wd * w)
    gemm.grouped_gemm_wgrad_adam(a, dy, G, p, m, v, lr=lr, beta1=b1, beta2=b2, eps=eps, weight_decay=wd,
                                 step=step, grad_scale=gs, uniform_rows=rows_per)
    torch.cuda.synchronize()
    gemm.check_status()
    for name, got, ref in (("m", m, m_ref), ("v", v, v_ref), ("p", p, w_ref)):
        err = ((got.float() - ref).norm() / ref.norm()).item()
        assert err < 6e-3, (name, err)


def test_cta_pair_claimed_tile_order_few_pairs_many_launches(cta_pair):
    """Two CTA pairs claim the 64 tiles of the problem one by one (the order is dynamic whenever
    there are more tiles than pairs); 80 launches walk the claim counters round more than once,
    and a second stream, with a workspace of its own, runs beside the first."""
    torch.manual_seed(3)
    a = _rand(2048, 256)
    w = _rand(2048, 256)
    ref = a.float() @ w.float().t()
    side = torch.cuda.Stream()
    outs = []
    for i in range(80):
        outs.append(gemm.grouped_gemm(a, w, b_layout="nk", max_ctas=4))
        if i % 8 == 0:
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                outs.append(gemm.grouped_gemm(a, w, b_layout="nk", max_ctas=6))
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    gemm.check_status()
    for o in (outs[0], outs[1], outs[40], outs[-1]):
        _close(o, ref)
    assert all(torch.equal(o, outs[0]) for o in outs[1:])


def test_cta_pair_claimed_tile_order_with_row_counts_on_the_device(cta_pair):
    """Row counts in device memory: the host only knows a bound of the tile count, pairs stop at
    the first claim past the last tile, and empty groups contribute no tile."""
    torch.manual_seed(4)
    G, K, N = 6, 128, 1024
    rows = torch.tensor([700, 0, 256, 1, 1030, 0], dtype=torch.int32)
    offs = torch.tensor([0, 768, 768, 1024, 1280, 2560], dtype=torch.int32)
    a = _rand(2560, K)
    w = _rand(G, N, K)
    out = gemm.grouped_gemm(a, w, b_layout="nk", group_rows=rows.cuda(), group_offs=offs.cuda(), max_ctas=4)
    torch.cuda.synchronize()
    gemm.check_status()
    for g in range(G):
        o, r = offs[g].item(), rows[g].item()
        if r:
            _close(out[o:o + r], a[o:o + r].float() @ w[g].float().t())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,K", [(32, 128, 64), (31, 264, 64), (33, 40, 128), (257, 328, 64), (512, 192, 128)])
@pytest.mark.parametrize("where", ["whole", "columns", "unaligned"])
@pytest.mark.parametrize("cta_pair", [0, 1])
def test_store_writes_its_block_and_nothing_else(dtype, M, N, K, where, cta_pair, monkeypatch):
    """Bulk tensor stores and the stores from registers they fall back to (partial row blocks, bases off
    16 bytes) at tile edges; a column block of a wider buffer keeps what lies around it."""
    monkeypatch.setattr(gemm, "CTA_PAIR", cta_pair)
    torch.manual_seed(M + N)
    a, w = _rand(M, K), _rand(N, K)
    lead = {"whole": 0, "columns": 8, "unaligned": 1}[where]
    buf = torch.full((M + 2, N + 2 * lead), 7.0, dtype=dtype, device="cuda")
    if where == "unaligned":
        buf = torch.full(((M + 2) * (N + 8) + 1,), 7.0, dtype=dtype, device="cuda")[1:].view(M + 2, N + 8)
    out = buf[1:M + 1, lead:lead + N]
    gemm.grouped_gemm(a, w, b_layout="nk", out=out, alpha=0.5)
    torch.cuda.synchronize()
    gemm.check_status()
    ref = 0.5 * (a.double() @ w.double().t())
    # fp32 sums of K products, then one rounding: 2^-8 of the value in bf16
    tol = (2.0 ** -8 if dtype == torch.bfloat16 else 1e-6) * ref.abs() + 1e-5 * K ** 0.5
    assert ((out.double() - ref).abs() <= tol).all()
    keep = torch.ones_like(buf, dtype=torch.bool)
    keep[1:M + 1, lead:lead + N] = False
    assert (buf[keep] == 7.0).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("cta_pair", [0, 1])
def test_stores_of_ragged_groups(dtype, cta_pair, monkeypatch):
    """Groups that end inside a 32-row block next to rows of the following group, and a weight gradient
    per group with rows past M cut off."""
    monkeypatch.setattr(gemm, "CTA_PAIR", cta_pair)
    torch.manual_seed(3)
    rows, K, N = [33, 0, 64, 1, 31, 300], 64, 328
    offs = [0, 33, 33, 97, 98, 129]
    total = 429 + 16
    a, w = _rand(total, K), _rand(len(rows), K, N)
    out = torch.full((total, N), 7.0, dtype=dtype, device="cuda")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")   # noqa: E731
    gemm.grouped_gemm(a, w, group_rows=i32(rows), group_offs=i32(offs), out=out)
    for g, (o, r) in enumerate(zip(offs, rows)):
        ref = a[o:o + r].double() @ w[g].double()
        tol = (2.0 ** -8 if dtype == torch.bfloat16 else 1e-6) * ref.abs() + 1e-5 * K ** 0.5
        assert ((out[o:o + r].double() - ref).abs() <= tol).all()
    assert (out[429:] == 7.0).all()
    M, G = 200, 3
    x, dy = _rand(G * 128, M), _rand(G * 128, N)
    buf = torch.full((G * M * N + 8,), 7.0, dtype=dtype, device="cuda")
    gw = buf[4 if dtype == torch.float32 else 8:][:G * M * N].view(G, M, N)
    gemm.grouped_gemm_wgrad(x, dy, G, uniform_rows=128, out=gw)
    torch.cuda.synchronize()
    gemm.check_status()
    ref = x.view(G, 128, M).double().transpose(1, 2) @ dy.view(G, 128, N).double()
    tol = (2.0 ** -8 if dtype == torch.bfloat16 else 1e-6) * ref.abs() + 1e-5 * 128 ** 0.5
    assert ((gw.double() - ref).abs() <= tol).all()
    assert int((buf == 7.0).sum()) >= 8 and (buf[:4] == 7.0).all()


@pytest.mark.parametrize("G,rows,M,N", [(2, 64, 256, 512), (3, 128, 200, 328), (2, 192, 160, 1024), (1, 64, 8, 264)])
@pytest.mark.parametrize("cta_pair", [0, 1])
def test_wgrad_adam_in_boxes_agrees_with_the_path_through_registers(G, rows, M, N, cta_pair, monkeypatch):
    """Whole blocks move by bulk copies, edges and bases off 16 bytes through registers: results agree to one
    rounding of bf16 (the unaligned path takes the exact square root and division), and what lies around
    the arrays stays."""
    monkeypatch.setattr(gemm, "CTA_PAIR", cta_pair)
    torch.manual_seed(M)
    x, dy = _rand(G * rows, M), _rand(G * rows, N)
    start = [_rand(G, M, N), _rand(G, M, N, scale=0.1), _rand(G, M, N, scale=0.1).abs()]
    results = []
    for lead in (8, 1):
        bufs = [torch.full((G * M * N + 16,), 7.0, dtype=torch.bfloat16, device="cuda") for _ in start]
        arrays = [b[lead:lead + G * M * N].view(G, M, N) for b in bufs]
        for a, s in zip(arrays, start):
            a.copy_(s)
        for step in (1, 2):
            gemm.grouped_gemm_wgrad_adam(x, dy, G, *arrays, lr=1e-2, beta1=0.9, beta2=0.99, eps=1e-8,
                                         weight_decay=0.1, step=step, uniform_rows=rows, grad_scale=0.5)
        torch.cuda.synchronize()
        gemm.check_status()
        for b in bufs:
            assert (b[:lead] == 7.0).all() and (b[lead + G * M * N:] == 7.0).all()
        results.append([a.clone() for a in arrays])
    for s, box, reg in zip(start, *results):
        assert not torch.equal(s, box)
        torch.testing.assert_close(box.float(), reg.float(), rtol=2.0 ** -7, atol=1e-6)


@pytest.mark.parametrize("act", ["gelu", "silu", "swiglu"])
@pytest.mark.parametrize("rows,F", [([64, 33, 0, 31], 264), ([32, 96, 1, 256], 512), ([300, 20, 64, 64], 128)])
@pytest.mark.parametrize("cta_pair", [0, 1])
@pytest.mark.parametrize("lead", [0, 1])
def test_activation_epilogues_at_ragged_groups_and_edges(act, rows, F, cta_pair, lead, monkeypatch):
    """FC1 and the FC2 input gradient: whole blocks move in boxes, the rest and bases off 16 bytes (`lead`)
    through registers; rows of no group stay as they were."""
    monkeypatch.setattr(gemm, "CTA_PAIR", cta_pair)
    torch.manual_seed(F)
    if act == "swiglu" and F <= 128:
        F = 136          # gated tiles are 256 wide
    G, H = len(rows), 128
    offs = [sum(rows[:g]) for g in range(G)]
    total = sum(rows) + 40
    Fw = 2 * F if act == "swiglu" else F
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")   # noqa: E731

    def fresh(n):
        return torch.full((total * n + 8,), 7.0, dtype=torch.bfloat16, device="cuda")[lead:lead + total * n].view(total, n)

    x, w1, w2 = _rand(total, H), _rand(G, H, Fw, scale=0.1), _rand(G, F, H, scale=0.1)
    probs, dy = torch.rand(total, device="cuda"), _rand(total, H)
    kw = dict(activation=act, group_rows=i32(rows), group_offs=i32(offs))
    a, pre = gemm.grouped_gemm_act(x, w1, probs, act_out=fresh(F), pre_out=fresh(Fw), **kw)
    a2, none = gemm.grouped_gemm_act(x, w1, probs, act_out=fresh(F), save_pre=False, **kw)
    dpre, dprobs = gemm.grouped_gemm_dact(dy, w2, pre, probs, dpre_out=fresh(Fw), **kw)
    torch.cuda.synchronize()
    gemm.check_status()
    assert none is None and torch.equal(a, a2)
    for t in (a, pre, dpre):
        assert (t[sum(rows):] == 7.0).all()
    for g in range(G):
        r = slice(offs[g], offs[g] + rows[g])
        p = probs[r].double()[:, None]
        ref_pre = x[r].double() @ w1[g].double()
        # one rounding of bf16 (2^-8) after fp32 sums and fast exponentials
        def close(got, ref, rel=2.0 ** -8, floor=2e-4):
            assert ((got.double() - ref).abs() <= rel * ref.abs() + floor * ref.abs().max().clamp(min=1e-9)).all()
        if rows[g] == 0:
            continue
        close(pre[r], ref_pre)
        close(a[r], gemm.act_ref(ref_pre, act) * p)
        z = pre[r].double().requires_grad_(True)
        y = gemm.act_ref(z, act)
        d = dy[r].double() @ w2[g].double().t()
        (dz,) = torch.autograd.grad(y, z, d * p)
        close(dpre[r], dz)
        close(dprobs[r], (d * y.detach()).sum(1), rel=1e-5)


@pytest.mark.parametrize("M,N,K", [(32, 128, 64), (31, 264, 64), (33, 40, 128), (257, 328, 64), (512, 192, 128)])
@pytest.mark.parametrize("how", ["whole", "columns", "unaligned", "in place"])
@pytest.mark.parametrize("cta_pair", [0, 1])
def test_residual_and_device_scalar(M, N, K, how, cta_pair, monkeypatch):
    """``alpha * alpha_dev * a @ w + residual`` with one rounding, for residuals of any row stride and base and
    for the accumulating form, which reads C itself."""
    monkeypatch.setattr(gemm, "CTA_PAIR", cta_pair)
    torch.manual_seed(M + N)
    a, w = _rand(M, K), _rand(N, K)
    scale = torch.tensor(0.375, device="cuda")
    lead = {"whole": 0, "columns": 8, "unaligned": 1, "in place": 0}[how]
    r = _rand(M + 1, N + 16)[1:, lead:lead + N]
    ref = 0.5 * 0.375 * (a.double() @ w.double().t()) + r.double()
    if how == "in place":
        out = gemm.grouped_gemm(a, w, b_layout="nk", out=r, accumulate=True, alpha=0.5, alpha_dev=scale)
    else:
        out = gemm.grouped_gemm(a, w, b_layout="nk", residual=r, alpha=0.5, alpha_dev=scale)
    g = gemm.grouped_gemm_wgrad(a, _rand(M, 72).fill_(1.0), 1, alpha_dev=scale) if M % 64 == 0 else None
    torch.cuda.synchronize()
    gemm.check_status()
    # fp32 sums of K products, then one rounding: 2^-8 of the value
    assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * K ** 0.5).all()
    if g is not None:
        want = 0.375 * a.double().sum(0)[:, None].expand(K, 72)
        assert ((g[0].double() - want).abs() <= 1e-5 * a.double().abs().sum(0)[:, None]).all()


@pytest.mark.parametrize("N", [200, 328, 1000])
@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("cta_pair", [0, 1])
def test_residual_store_with_a_cut_last_block(N, in_place, cta_pair, monkeypatch):
    """A warp that stores a whole 64-column block and then the cut last one (N mod 128 between 64 and 128): the
    second must not refill the box that the first store still reads.  Rows enough for every SM to store at
    once; every element against 64 bits, and the same bytes each time."""
    monkeypatch.setattr(gemm, "CTA_PAIR", cta_pair)
    torch.manual_seed(N)
    M, K = 40_000, 64
    a, w, r = _rand(M, K), _rand(N, K), _rand(M, N)
    ref = a.double() @ w.double().t() + r.double()
    first = None
    for _ in range(8):
        if in_place:
            out = gemm.grouped_gemm(a, w, b_layout="nk", out=r.clone(), accumulate=True)
        else:
            out = gemm.grouped_gemm(a, w, b_layout="nk", residual=r)
        if first is None:
            first = out
            # fp32 sums of K products, then one rounding: 2^-8 of the value
            assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5 * K ** 0.5).all()
        assert torch.equal(out, first)
    torch.cuda.synchronize()
    gemm.check_status()


@pytest.mark.parametrize("F", [128, 104, 64, 40])
@pytest.mark.parametrize("act", ["gelu", "silu", "none"])
def test_activation_gradient_of_narrow_tiles(F, act):
    """Tiles of 128 columns, three a CTA: the boxes' barriers change phase with every tile.  Blocks that reach past F
    (104: those of the second half of the columns) and groups' ends go through registers."""
    torch.manual_seed(F)
    rows = [30_000, 33, 0, 20_015]
    G, H, total = len(rows), 64, sum(rows)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")   # noqa: E731
    offs = [sum(rows[:g]) for g in range(G)]
    w2, dy, pre, probs = _rand(G, F, H, scale=0.1), _rand(total, H), _rand(total, F), torch.rand(total, device="cuda")
    results = []
    for lead in (0, 1):      # bases off 16 bytes go through registers
        dpre = torch.full((total * F + 8,), 7.0, dtype=torch.bfloat16, device="cuda")[lead:lead + total * F].view(total, F)
        src = torch.empty(total * F + 8, dtype=torch.bfloat16, device="cuda")[lead:lead + total * F].view(total, F)
        src.copy_(pre)
        results.append(gemm.grouped_gemm_dact(dy, w2, src, probs, activation=act, group_rows=i32(rows),
                                              group_offs=i32(offs), dpre_out=dpre))
    torch.cuda.synchronize()
    gemm.check_status()
    for g in range(G):
        r = slice(offs[g], offs[g] + rows[g])
        if rows[g] == 0:
            continue
        z = pre[r].double().requires_grad_(True)
        y = gemm.act_ref(z, act)
        d = dy[r].double() @ w2[g].double().t()
        ref = torch.autograd.grad(y, z, d * probs[r].double()[:, None])[0]
        dp = (d * y.detach()).sum(1)
        for dpre, dprobs in results:
            # one rounding of bf16 (2^-8) after fp32 sums and fast exponentials
            assert ((dpre[r].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2e-4 * ref.abs().max()).all()
            assert ((dprobs[r].double() - dp).abs() <= 1e-5 * dp.abs() + 2e-4 * dp.abs().max()).all()


@pytest.mark.parametrize("N", [128, 104, 64])
def test_wgrad_adam_of_narrow_tiles(N):
    """Tiles of 128 columns, three a CTA: see above.  From the same start both paths agree to one rounding of bf16 (2^-7
    between neighbours); before it they differ by a few 2^-23 of terms below 8, which is what is left where a weight
    and its update cancel."""
    torch.manual_seed(N)
    G, rows, M = 2, 128, 30_000
    x, dy = _rand(G * rows, M), _rand(G * rows, N)
    start = [_rand(G, M, N), _rand(G, M, N, scale=0.1), _rand(G, M, N, scale=0.1).abs()]
    results = []
    for lead in (0, 1):
        arrays = [torch.empty(G * M * N + 8, dtype=torch.bfloat16, device="cuda")[lead:lead + G * M * N].view(G, M, N)
                  for _ in start]
        for a, s in zip(arrays, start):
            a.copy_(s)
        gemm.grouped_gemm_wgrad_adam(x, dy, G, *arrays, lr=1e-2, beta1=0.9, beta2=0.99, eps=1e-8,
                                     weight_decay=0.1, step=1, uniform_rows=rows, grad_scale=0.5)
        results.append(arrays)
    torch.cuda.synchronize()
    gemm.check_status()
    for s, box, reg in zip(start, *results):
        assert not torch.equal(s, box)
        torch.testing.assert_close(box.float(), reg.float(), rtol=2.0 ** -7, atol=4 * 8 * 2.0 ** -23)


@pytest.mark.parametrize("cta_pair", [0, 1])
@pytest.mark.parametrize("rows,N,expected", [(200, 264, 1), (333, 128, 3), (129, 520, 2)])
def test_gated_rows_and_gated_columns_that_have_arrived(rows, N, expected, cta_pair, monkeypatch):
    """The producers behind a gate, on counters that stand at their targets: blocks of 128 rows of a group, and
    column blocks by their source, begun at another source than the first."""
    monkeypatch.setattr(gemm, "CTA_PAIR", cta_pair)
    torch.manual_seed(8)
    G, K, per_src = 3, 256, 2
    blocks = (rows + 127) // 128
    a, w = _rand(G * rows, K), _rand(G, K, N)
    in_block = torch.tensor([min(128, rows - 128 * i) for i in range(blocks)], dtype=torch.int32, device="cuda")
    waited = torch.zeros(1, dtype=torch.int64, device="cuda")
    common = dict(gate_blocks_per_group=blocks, gate_expected=expected, timeout_ns=10 ** 9, wait_ns=waited.data_ptr())
    flags = (in_block * expected).repeat(G)
    got = gemm.grouped_gemm(a, w, uniform_rows=rows, gate=dict(gate_flags=flags.data_ptr(), **common))
    gemm.check_status()
    for g in range(G):
        _close(got[g * rows:(g + 1) * rows], a[g * rows:(g + 1) * rows].float() @ w[g].float())
    flags = (in_block * expected).repeat(K // 64 // per_src)
    got = gemm.grouped_gemm(a[:rows], w[:1], gate=dict(gate_flags=flags.data_ptr(), gate_k_blocks_per_src=per_src,
                                                       k_rotate=per_src, **common))
    gemm.check_status()
    _close(got, a[:rows].float() @ w[0].float())
