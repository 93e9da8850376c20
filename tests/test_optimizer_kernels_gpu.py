"""AdamW and the squared norm on aligned and unaligned shards, with and without a remainder, against 64 bits."""
import pytest
import torch

from gcore_b200.ops import optim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 1030, 70001])
@pytest.mark.parametrize("shift", [0, 1, 4])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_adam(n, shift, dtype):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(n + shift)

    def buf(dt=torch.float32):
        return torch.randn(n + shift + 5, generator=g, device="cuda").to(dt)

    whole = [buf(), buf(), buf().abs(), buf(dtype), buf(torch.bfloat16)]
    kept = [t.clone() for t in whole]
    master, m, v, grad, param = (t[shift:shift + n] for t in whole)
    lr, b1, b2, eps, wd, step, sc = 0.01, 0.9, 0.95, 1e-8, 0.1, 3, 0.25
    gd = grad.double() * sc * 2.0
    m2, v2 = b1 * m.double() + (1 - b1) * gd, b2 * v.double() + (1 - b2) * gd * gd
    p2 = master.double()
    p2 = p2 - lr * ((m2 / (1 - b1 ** step)) / ((v2 / (1 - b2 ** step)).sqrt() + eps) + wd * p2)
    optim.adam_step(master, m, v, grad, param, lr=lr, beta1=b1, beta2=b2, eps=eps, weight_decay=wd, step=step,
                    grad_scale=torch.tensor([sc], device="cuda"), scale_val=2.0)
    # a handful of fp32 roundings of values of at most 10 (the bias corrections lose two bits more)
    for have, want in ((master, p2), (m, m2), (v, v2)):
        assert ((have.double() - want).abs() <= 2.0 ** -19 * (want.abs() + 1)).all()
    assert torch.equal(param, master.bfloat16())
    for t, k in zip(whole, kept):
        assert torch.equal(t[:shift], k[:shift]) and torch.equal(t[shift + n:], k[shift + n:])


@pytest.mark.parametrize("n", [1, 7, 8, 4100, 3000001])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_sumsq(n, shift, dtype):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n + shift, generator=g, device="cuda").to(dtype)[shift:]
    out = torch.full((1,), 2.0, device="cuda")
    optim.sumsq(x, out)
    want = x.double().square().sum() + 2
    # chains of at most a few hundred fp32 additions of positive numbers
    assert (out.double() - want).abs() <= 256 * 2.0 ** -24 * want
