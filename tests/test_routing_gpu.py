"""Router kernels against the PyTorch statements of the same rules: integers and probabilities of the
plans are copies, so they are compared exactly."""
import math

import pytest
import torch

from fluidmoe_b200.models import moe_dropless
from fluidmoe_b200.ops import elementwise, permute, router

pytestmark = pytest.mark.gpu


def serial_topk(row, k):
    """The selection rule, spelled out: first candidate, or a strictly larger one after it."""
    taken = []
    for _ in range(k):
        best, bi = -math.inf, -1
        for e, v in enumerate(row):
            if e not in taken and (v > best or bi < 0):
                best, bi = v, e
        taken.append(bi)
    return taken


@pytest.mark.parametrize("E,k", [(1, 1), (8, 2), (31, 16), (32, 4), (33, 2), (64, 8), (65, 6), (200, 8), (256, 16),
                                 (257, 3)])
@pytest.mark.parametrize("kind", ["normal", "ties", "special"])
def test_topk_softmax(E, k, kind):
    g = torch.Generator().manual_seed(E * 17 + k)
    T = 67
    x = torch.randn(T, E, generator=g)
    if kind == "ties":
        x = torch.randint(-1, 2, (T, E), generator=g).float() * \
            torch.where(torch.rand(T, E, generator=g) < 0.5, -1.0, 1.0)
    if kind == "special":
        pick = torch.rand(T, E, generator=g)
        x[pick < 0.2] = -math.inf
        x[(pick > 0.8) & (torch.arange(T)[:, None] % 3 == 0)] = math.nan
        x[(pick > 0.95) & (torch.arange(T)[:, None] % 3 == 1)] = math.inf
        x[5] = -math.inf
    idx, probs = elementwise.topk_softmax(x.cuda(), k)
    want = torch.tensor([serial_topk(r.tolist(), k) for r in x])
    assert torch.equal(idx.cpu(), want)
    # winners less the first one, as the kernel subtracts; 16 terms of a fast exponential: 1e-5
    v = x.gather(1, want).double()
    ex = torch.exp(v - v[:, :1])
    torch.testing.assert_close(probs.cpu().double(), ex / ex.sum(1, keepdim=True), rtol=1e-5, atol=1e-7, equal_nan=True)


@pytest.mark.parametrize("E,k", [(1, 1), (2, 2), (7, 3), (8, 8), (9, 3), (16, 2)])
@pytest.mark.parametrize("ties", [False, True])
def test_topk_of_many_tokens_equals_that_of_few(E, k, ties):
    """From 1024 * E * k tokens on a thread takes a token, below a warp; the same choices and, but for the order of
    k terms, the same probabilities."""
    T = 1024 * E * k
    g = torch.Generator().manual_seed(E)
    x = torch.randn(T, E, generator=g)
    if ties:
        x = torch.randint(-1, 2, (T, E), generator=g).float()
        x[::5] = -math.inf
        x[1::5, 0] = math.nan
    x = x.cuda()
    idx, probs = elementwise.topk_softmax(x, k)
    for part in (slice(0, T // 2), slice(T // 2, T)):
        i2, p2 = elementwise.topk_softmax(x[part], k)
        assert torch.equal(idx[part], i2)
        torch.testing.assert_close(probs[part], p2, rtol=2e-6, atol=0.0, equal_nan=True)


def _routing(T, E, k, seed, skew=0.0):
    g = torch.Generator().manual_seed(seed)
    logits = torch.randn(T, E, generator=g) - skew * torch.arange(E)
    logits = (logits * 4).round() / 4 if seed % 2 else logits      # odd seeds: many equal probabilities
    top, idx = torch.topk(logits, k, dim=1)
    return idx, torch.softmax(top, dim=1)


@pytest.mark.parametrize("T,E,k,cf,skew", [
    (1, 1, 1, 1.0, 0.0), (31, 8, 2, 1.0, 0.0), (64, 8, 2, 1.0, 0.5), (1023, 8, 2, 1.0, 0.0), (1025, 16, 1, 1.0, 0.3),
    (2048, 64, 8, 1.0, 0.05), (4096, 8, 2, 0.5, 0.0), (4096, 8, 2, 2.0, 0.0), (8192, 64, 8, 1.0, 0.02),
    (12289, 4, 2, 1.0, 0.0), (39715, 8, 2, 1.0, 0.1), (39720, 8, 2, 1.0, 0.1), (45000, 4, 2, 1.0, 0.1)])
@pytest.mark.parametrize("seed", [2, 3])
def test_padded_plan(T, E, k, cf, skew, seed):
    idx, probs = _routing(T, E, k, seed, skew)
    cap = min(T, router.expert_capacity(T, k, E, cf))
    got = router.build_padded_plan(idx.cuda(), probs.cuda(), E, cap)
    # the rule: of equal probabilities at the threshold the lower token ids stay
    rmap = torch.zeros(T, E, dtype=torch.bool).scatter(1, idx, True)
    pr = torch.zeros(T, E).scatter(1, idx, probs)
    keep = torch.zeros(T, E, dtype=torch.bool)
    order = torch.sort(torch.where(rmap, pr, torch.full_like(pr, -1.0)), dim=0, descending=True, stable=True).indices
    keep.scatter_(0, order[:cap], True)
    keep &= rmap
    pad = ~rmap & (torch.cumsum(~rmap, 0) - 1 < (cap - keep.sum(0)))
    sel = keep | pad
    pos = torch.cumsum(sel, 0) - 1
    for e in range(E):
        toks = sel[:, e].nonzero().squeeze(1)
        n = toks.numel()      # below cap only where fewer tokens than slots are left to pad with
        assert torch.equal(got.sorted_indices.cpu()[e * cap:e * cap + n], toks)
        assert torch.equal(got.permuted_probs.cpu()[e * cap:e * cap + n], (pr[:, e] * keep[:, e])[toks])
    slot = torch.where(keep, pos + torch.arange(E) * cap, torch.full_like(pos, -1)).gather(1, idx)
    assert torch.equal(got.slot_of_token.cpu().long(), slot)
    assert torch.equal(got.routed_per_expert.cpu().long(), keep.sum(0))
    assert got.tokens_per_expert.cpu().tolist() == [cap] * E


def test_padded_plan_counts_a_repeated_choice_once():
    idx = torch.tensor([[0, 0], [1, 0], [0, 1], [1, 1]]).cuda()
    probs = torch.tensor([[0.75, 0.25], [0.5, 0.5], [0.625, 0.375], [0.875, 0.125]]).cuda()
    got = router.build_padded_plan(idx, probs, 2, 3)
    assert got.routed_per_expert.tolist() == [3, 3]
    assert got.sorted_indices.tolist() == [0, 1, 2, 1, 2, 3]
    assert got.permuted_probs.tolist() == [0.75, 0.5, 0.625, 0.5, 0.375, 0.875]


@pytest.mark.parametrize("T", [4, 1000, 50_000])     # the last takes the kernel for rows beyond shared memory
@pytest.mark.parametrize("k", [2, 5])
def test_padded_plan_gives_repeated_choices_no_slot(T, k):
    """Every entry of ``slot_of_token`` is written: the slot of a kept first choice, -1 for a dropped one and for
    every later choice of the same expert (the un-permute takes any value from 0 up as a row)."""
    E = 3
    g = torch.Generator().manual_seed(T)
    idx = torch.randint(0, E, (T, k), generator=g)
    probs = torch.rand(T, k, generator=g) + 0.01
    cap = max(1, T // 2)
    # blocks of the plan's sizes, filled and given back, so that what a kernel leaves out shows
    filled = [torch.full((T, k), 7, dtype=torch.int32, device="cuda") for _ in range(4)]
    del filled
    got = router.build_padded_plan(idx.cuda(), probs.cuda(), E, cap)
    slot, tok = got.slot_of_token.cpu().long(), got.sorted_indices.cpu()
    first = torch.ones(T, k, dtype=torch.bool)
    for j in range(1, k):
        first[:, j] = (idx[:, :j] != idx[:, j:j + 1]).all(1)
    assert (slot[~first] == -1).all()
    kept = slot >= 0
    assert torch.equal(tok[slot[kept]], torch.arange(T)[:, None].expand(T, k)[kept])
    assert torch.equal(slot[kept] // cap, idx[kept])
    assert torch.equal(got.permuted_probs.cpu()[slot[kept]], probs[kept])
    assert torch.bincount(idx[kept], minlength=E).tolist() == got.routed_per_expert.tolist()


@pytest.mark.parametrize("T,E,k,skew", [(1, 1, 1, 0.0), (1, 8, 2, 0.0), (63, 8, 2, 3.0), (64, 1, 1, 0.0),
                                        (683, 64, 6, 0.1), (1531, 64, 6, 0.05), (4096, 8, 2, 0.0), (4097, 1024, 8, 0.0)])
def test_dropless_plan_local(T, E, k, skew):
    idx, probs = _routing(T, E, k, 4, skew)
    p = moe_dropless.build_local_plan(idx.cuda(), probs.cuda(), E)
    counts = torch.bincount(idx.reshape(-1), minlength=E)
    rows = (counts + 63) // 64 * 64
    offs = torch.cumsum(rows, 0) - rows
    tok = torch.full((p.rows_em,), -2)
    prob = torch.zeros(p.rows_em)
    slot = torch.empty(T * k, dtype=torch.long)
    order = torch.sort(idx.reshape(-1), stable=True).indices
    first = torch.cumsum(counts, 0) - counts
    e_of = idx.reshape(-1)[order]
    r = offs[e_of] + torch.arange(T * k) - first[e_of]
    for e in range(E):
        tok[int(offs[e] + counts[e]):int(offs[e] + rows[e])] = -1
    tok[r], prob[r], slot[order] = order // k, probs.reshape(-1)[order], r
    assert torch.equal(p.sorted_indices.cpu(), tok) and torch.equal(p.permuted_probs.cpu(), prob)
    assert torch.equal(p.slot_of_token.cpu().long().reshape(-1), slot)
    assert torch.equal(p.counts.cpu().long(), counts)
    assert torch.equal(p.group_rows.cpu().long(), rows) and torch.equal(p.group_offs.cpu().long(), offs)
    x = torch.randn(T, 72, device="cuda").bfloat16()
    out = torch.full((p.rows_em, 72), 7.0, device="cuda", dtype=torch.bfloat16)
    permute.permute_rows(x, p.sorted_indices, out)
    want = torch.full((p.rows_em, 72), 7.0, dtype=torch.bfloat16)
    want[tok == -1] = 0
    want[tok >= 0] = x.cpu()[tok[tok >= 0]]
    assert torch.equal(out.cpu(), want)


@pytest.mark.parametrize("T,E,k", [(5, 8, 2), (333, 64, 6)])
def test_dropless_layer_passes_equal_the_plan_of_the_host(T, E, k, monkeypatch):
    """The same dropless layer with either plan: the same rows meet the same weights, so results agree to
    the order of fp32 sums inside a weight gradient (K blocks of 64 rows start elsewhere): 1e-5."""
    from fluidmoe_b200.models.transformer import TransformerModel
    from fluidmoe_b200.parallel.scheduler import get_backward_scheduler
    torch.manual_seed(0)
    model = TransformerModel(1, 128, 1, 1, 192, E, k, activation_func="swiglu", norm_type="rmsnorm",
                             capacity_factor=0.0, router_dtype=torch.float32, has_attention=False,
                             num_shared_experts=1, dtype=torch.bfloat16, device="cuda")
    x0 = torch.randn(T, 1, 128, device="cuda").bfloat16()
    dy = torch.randn(T, 1, 128, device="cuda").bfloat16()
    sched = get_backward_scheduler()
    results = []
    for local in (True, False):
        if not local:
            monkeypatch.setattr(moe_dropless, "local_plan_applies", lambda *a: False)
        for p in model.parameters():
            p.grad = None
        x = x0.clone().requires_grad_(True)
        y = model(x)
        y.backward(dy)
        sched.finish_batch()
        sched.clear_iteration()
        results.append([y.detach(), x.grad] + [p.grad for n, p in model.named_parameters()
                                               if not n.split(".")[-1].startswith(("qkv", "proj", "ln1"))])
    for a, b in zip(*results):
        a, b = a.double(), b.double()
        assert torch.isfinite(a).all()
        assert (a - b).norm() <= 1e-5 * b.norm() + 1e-12
