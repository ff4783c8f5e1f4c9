"""GEMM for few rows per group and few tiles against fp32 products; edges of tiles, parts, row chunks and rules.

Bounds: products of bf16 are exact in fp32 and K of them are summed in fp32, 2^-24 K relative to the sum of
magnitudes, far below the rounding of a bf16 result, 2^-9 of it (twice for the activation's product with the
probability): 4e-3 of the norm; fp32 results 1e-5."""
import pytest
import torch

from fluidmoe_b200 import _native
from fluidmoe_b200.ops import gemm

pytestmark = pytest.mark.gpu


def _r(*s):
    return torch.randn(*s, device="cuda").bfloat16()


def _close(got, want, tol):
    assert got.shape == want.shape
    assert (got.float() - want).norm() <= tol * want.norm()


def _alone(monkeypatch, fn):
    """The same call without scratch: no tile is shared by several CTAs."""
    with monkeypatch.context() as m:
        m.setattr(gemm, "_t_gemm", lambda *a: None)
        m.setattr(gemm, "_t_gemm_act", lambda *a: None)
        return fn()


def _taken(monkeypatch, fn):
    """The call with scratch, which only the C++ call gives."""
    made = []
    with monkeypatch.context() as m:
        for name in ("_t_gemm", "_t_gemm_act"):
            def record(*args, call=getattr(gemm, name)):
                made.append(call(*args))
                return made[-1]
            m.setattr(gemm, name, record)
        res = fn()
    assert len(made) == 1 and made[0] is not None
    return res


def _shared(monkeypatch, fn):
    """Whether CTAs share tiles in this call: the launcher asks for scratch."""
    descs = []
    with monkeypatch.context() as m:
        m.setattr(gemm, "_launch", lambda d: descs.append(dict(d, cta_pair=gemm.CTA_PAIR)))
        _alone(monkeypatch, fn)
    return _native.lib().gemm_workspace(descs[0]) > 0


@pytest.mark.parametrize("rows", [1, 31, 32, 33, 63, 64, 65])
@pytest.mark.parametrize("groups,K,N,layout", [(1, 520, 8, "nk"), (1, 4096, 264, "nk"), (3, 128, 136, "kn"),
                                               (8, 1024, 512, "kn"), (1, 72, 128, "kn"), (8, 4096, 4096, "kn"),
                                               (3, 8192, 4104, "kn")])
def test_store(monkeypatch, rows, groups, K, N, layout):
    torch.manual_seed(0)
    a = _r(groups * rows, K)
    w = _r(groups, K, N) if layout == "kn" else _r(N, K)
    b = w if groups > 1 else (w[0] if layout == "kn" else w)
    want = torch.bmm(a.float().view(groups, rows, K), w.float() if layout == "kn" else w.float().t().unsqueeze(0))
    want = want.view(groups * rows, N)

    def run(dtype):
        return gemm.grouped_gemm(a, b, b_layout=layout, uniform_rows=rows, out_dtype=dtype, alpha=0.5)
    # 2 and 51 tiles with sums of 64 and 128 blocks; the others go round once as evenly or have short sums
    shares = {(1, 4096): rows <= 32, (3, 8192): rows <= 64}.get((groups, K), False)
    assert _shared(monkeypatch, lambda: run(None)) == shares
    for got in (_taken(monkeypatch, lambda: run(torch.float32)), _alone(monkeypatch, lambda: run(torch.float32))):
        _close(got, 0.5 * want, 1e-5)
    for got in (_taken(monkeypatch, lambda: run(None)), _alone(monkeypatch, lambda: run(None))):
        _close(got, 0.5 * want, 4e-3)
    gemm.check_status()


@pytest.mark.parametrize("have,rows,N", [(40, 16, 4096), (17, 16, 264), (100, 60, 512), (16, 16, 4096)])
def test_groups_beyond_the_rows(monkeypatch, have, rows, N):
    """``uniform_rows`` of three groups may come to more rows than there are: the last groups are cut or empty, and
    nothing behind the results is written."""
    torch.manual_seed(5)
    a, w, p = _r(have, 1024), _r(3, 1024, N), torch.rand(have, device="cuda")
    want = torch.cat([a[g * rows:(g + 1) * rows].float() @ w[g].float() for g in range(3)])

    def run(dtype):
        room = torch.full((have + 2 * rows, N), 7.0, device="cuda", dtype=dtype)
        gemm.grouped_gemm(a, w, uniform_rows=rows, out=room[:have])
        assert (room[have:] == 7.0).all()
        return room[:have]
    for got in (run(torch.float32), _alone(monkeypatch, lambda: run(torch.float32))):
        _close(got, want, 1e-5)
    act, pre = gemm.grouped_gemm_act(a, w, p, activation="silu", uniform_rows=rows)
    _close(act, gemm.act_ref(want, "silu") * p.unsqueeze(1), 4e-3)
    _close(pre, want, 4e-3)
    gemm.check_status()


@pytest.mark.parametrize("rows", [33, 64, 100, 1000, 2016, 2017])
@pytest.mark.parametrize("K,N,layout", [(2048, 8, "nk"), (2056, 72, "nk"), (2048, 128, "kn"), (4096, 64, "nk"),
                                        (2040, 64, "kn")])
def test_narrow_products_in_row_chunks(monkeypatch, rows, K, N, layout):
    torch.manual_seed(2)
    a, b = _r(rows, K), (_r(K, N) if layout == "kn" else _r(N, K))
    want = a.float() @ (b.float() if layout == "kn" else b.float().t())

    def run(dtype):
        return gemm.grouped_gemm(a, b, b_layout=layout, uniform_rows=rows, out_dtype=dtype)
    assert _shared(monkeypatch, lambda: run(None)) == (K == 4096 and rows <= 100)      # 1000 rows go the other way
    for got in (_taken(monkeypatch, lambda: run(torch.float32)), _alone(monkeypatch, lambda: run(torch.float32))):
        _close(got, want, 1e-5)
    _close(_taken(monkeypatch, lambda: run(None)), want, 4e-3)
    gemm.check_status()


@pytest.mark.parametrize("activation", ["gelu", "silu", "swiglu", "none"])
@pytest.mark.parametrize("rows,groups,K,F,probs,save", [(16, 8, 1024, 200, True, True), (32, 2, 128, 128, False, False),
                                                        (5, 3, 4096, 384, True, False), (17, 8, 2048, 3000, True, True),
                                                        (33, 3, 2048, 200, True, True), (64, 8, 1024, 1000, True, False),
                                                        (49, 2, 128, 128, False, True), (65, 2, 192, 136, True, True),
                                                        (61, 3, 4096, 200, True, True)])
def test_activation(monkeypatch, activation, rows, groups, K, F, probs, save):
    torch.manual_seed(1)
    a, w = _r(groups * rows, K), _r(groups, K, F * (2 if activation == "swiglu" else 1))
    p = torch.rand(groups * rows, device="cuda") if probs else None
    pre = torch.bmm(a.float().view(groups, rows, K), w.float()).view(groups * rows, -1)
    want = gemm.act_ref(pre, activation) * (p.unsqueeze(1) if probs else 1.0)

    def run():
        return gemm.grouped_gemm_act(a, w, p, activation=activation, uniform_rows=rows, save_pre=save)
    # 9, 6 and 192 tiles of 64 and 32 blocks; 6 of 32 blocks where a block is 36 KB
    assert _shared(monkeypatch, run) == ((groups, K) in ((3, 4096), (8, 2048)) or
                                         (groups, K, activation) == (3, 2048, "swiglu"))
    for act, kept in (_taken(monkeypatch, run), _alone(monkeypatch, run)):
        _close(act, want, 4e-3)
        assert (kept is None) == (not save)
        if save:
            _close(kept, pre, 4e-3)
    gemm.check_status()


@pytest.mark.parametrize("rows", [16, 60])
def test_repeats_streams_and_graphs(monkeypatch, rows):
    """Shared tiles are summed in the order of their parts: every launch gives the same bytes, also more launches than
    there are counter sets, from two streams at once, products of other sizes between them, and from a captured graph."""
    torch.manual_seed(3)
    a, w = _r(8 * rows, 2048), _r(8, 2048, 2 * 3072)
    a2, w2 = _r(100, 4096), _r(64, 4096)

    def run():
        return gemm.grouped_gemm_act(a, w, None, activation="swiglu", uniform_rows=rows, save_pre=False)[0]

    def other():
        return gemm.grouped_gemm(a2, w2, b_layout="nk", uniform_rows=100, out_dtype=torch.float32)
    assert _shared(monkeypatch, run) and _shared(monkeypatch, other)
    first, second = run(), other()
    # nothing is read on the host before all is queued: launches of both streams are under way together
    side, got = torch.cuda.Stream(), []
    side.wait_stream(torch.cuda.current_stream())
    for i in range(150):
        for stream in (side, torch.cuda.current_stream()):
            with torch.cuda.stream(stream):
                got.append((run(), first))
                if i % 3 == 0:
                    got.append((other(), second))
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in got)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = run()
    for _ in range(3):
        out.zero_()
        graph.replay()
        assert torch.equal(out, first)
    gemm.check_status()


@pytest.mark.parametrize("M,N", [(72, 136), (512, 4736), (520, 4736), (2048, 1152), (2048, 1160), (2304, 4096), (2312, 4104)])
@pytest.mark.parametrize("K", [512, 1024, 1032, 2048])
def test_few_tiles(M, N, K):
    """Edges of the rule that gives few tiles to single CTAs: stored with its options, and weight gradients."""
    torch.manual_seed(4)
    a, w, d = _r(M, K), _r(K, N), _r(M, N)
    want = a.float() @ w.float()
    _close(gemm.grouped_gemm(a, w), want, 4e-3)
    _close(gemm.grouped_gemm(a, w.t().contiguous(), b_layout="nk", residual=d), want + d.float(), 4e-3)
    _close(gemm.grouped_gemm(a, w, out_dtype=torch.float32), want, 1e-5)
    grad = torch.ones(1, K, N, device="cuda")
    gemm.grouped_gemm_wgrad(a, d, 1, uniform_rows=M, out=grad, accumulate=True)
    _close(grad[0], a.float().t() @ d.float() + 1.0, 1e-5)
    gemm.check_status()
