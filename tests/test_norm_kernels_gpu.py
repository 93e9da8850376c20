"""RMSNorm forward and backward at the widths where the kernels change (lanes per row, threads and registers per row), against
64 bits."""
import pytest
import torch

from gcore_b200.ops import fused

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [8, 64, 72, 128, 136, 256, 264, 1024, 1032, 2048, 2056, 4096, 4104, 6144, 6152, 7168, 8192])
@pytest.mark.parametrize("T", [1, 17, 297, 2401])
@pytest.mark.parametrize("residual", [False, True])
def test_rmsnorm(H, T, residual):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(H + T)
    x, r, dy, dr = (torch.randn(T, H, generator=g, device="cuda").bfloat16() for _ in range(4))
    w = (1 + 0.1 * torch.randn(H, generator=g, device="cuda")).bfloat16()
    x.requires_grad_()
    w.requires_grad_()
    r.requires_grad_(residual)
    y, s = fused.rmsnorm(x, w, 1e-6, r if residual else None)
    sd = (x.detach().float() + r.detach().float()).bfloat16().double() if residual else x.detach().double()
    if residual:
        assert torch.equal(s.detach().double(), sd)
    rs = torch.rsqrt(sd.square().mean(-1, keepdim=True) + 1e-6)
    ref = sd * rs * w.detach().double()
    u, f = 2.0 ** -8, H * 2.0 ** -24 + 2.0 ** -20     # rounding to bf16; fp32 sums of H terms and the fast square root
    assert ((y.double() - ref).abs() <= (u + f) * ref.abs()).all()
    torch.autograd.backward([y, s] if residual else [y], [dy, dr] if residual else [dy])
    gw, n = dy.double() * w.detach().double(), sd * rs
    c = (gw * n).mean(-1, keepdim=True)
    dx = rs * (gw - n * c)
    mag = rs * (gw.abs() + n.abs() * (gw * n).abs().mean(-1, keepdim=True))
    if residual:
        dx, mag = dx + dr.double(), mag + dr.double().abs()
        assert torch.equal(x.grad, r.grad)
    assert ((x.grad.double() - dx).abs() <= u * dx.abs() + 4 * f * mag).all()
    dw = (dy.double() * n).sum(0)
    assert ((w.grad.double() - dw).abs() <= u * dw.abs() + (T * 2.0 ** -24 + 4 * f) * (dy.double() * n).abs().sum(0)).all()
