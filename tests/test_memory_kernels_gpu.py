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
