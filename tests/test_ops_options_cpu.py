"""Options of the op front-ends that need no GPU."""
import pytest
import torch

from fluidmoe_b200.ops import gemm


def test_residual_is_added_and_refuses_what_the_kernel_refuses():
    torch.manual_seed(0)
    a, w, r = torch.randn(6, 8), torch.randn(5, 8), torch.randn(6, 5)
    torch.testing.assert_close(gemm.gemm_nt(a, w, residual=r), a @ w.t() + r)
    torch.testing.assert_close(gemm.gemm_nt(a, w, residual=r, alpha=0.5, alpha_dev=torch.tensor(3.0)), 1.5 * a @ w.t() + r)
    for kw in (dict(residual=r, out=torch.ones(6, 5), accumulate=True), dict(residual=r[:1]), dict(residual=r.double())):
        with pytest.raises(AssertionError):
            gemm.gemm_nt(a, w, **kw)
