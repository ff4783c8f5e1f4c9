"""Options of the op front-ends that need no GPU."""
import pytest
import torch

from fluidmoe_b200.ops import elementwise, gemm


def test_residual_is_added_and_refuses_what_the_kernel_refuses():
    torch.manual_seed(0)
    a, w, r = torch.randn(6, 8), torch.randn(5, 8), torch.randn(6, 5)
    torch.testing.assert_close(gemm.gemm_nt(a, w, residual=r), a @ w.t() + r)
    torch.testing.assert_close(gemm.gemm_nt(a, w, residual=r, alpha=0.5, alpha_dev=torch.tensor(3.0)), 1.5 * a @ w.t() + r)
    for kw in (dict(residual=r, out=torch.ones(6, 5), accumulate=True), dict(residual=r[:1]), dict(residual=r.double())):
        with pytest.raises(AssertionError):
            gemm.gemm_nt(a, w, **kw)


def test_rope_table_follows_its_angles():
    """Angles that come to the address of released ones, other strides over one array, and an update in place."""
    def check(f):
        tab = elementwise._cos_sin_table(f, f.shape[-1])
        assert torch.equal(tab, torch.stack((torch.cos(f), torch.sin(f)), -1).view_as(tab))
    for i in range(12):
        f = torch.full((64, 1, 1, 16), 0.1 * i)      # released at the next turn
        check(f)
        del f
    f = torch.rand(16, 1, 1, 16)
    check(f)
    check(f.transpose(0, 3))
    f.mul_(2.0)
    check(f)
