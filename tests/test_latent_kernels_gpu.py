"""Rotation of aligned rows, keys and values out of the latent, the decode step's cache rows and block-fp8 dequantisation, against
their plain definitions."""
import pytest
import torch

from gcore_b200.ops import fused, quant

pytestmark = pytest.mark.gpu
THETA = 10000.0


def _angles_bound(pos, x):
    # the angle is pos * theta^(-2 i / rot) in fp32 with the fast power (a few units of 2^-22) and the fast sine
    return (pos.double()[:, None, None] * 2.0 ** -20 + 2.0 ** -20) * x.double().abs().amax() * 2


@pytest.mark.parametrize("T", [1, 5, 301])
@pytest.mark.parametrize("heads,D,rot", [(1, 64, 64), (3, 128, 128), (36, 128, 64), (5, 192, 32), (2, 24, 24)])
@pytest.mark.parametrize("interleaved", [False, True])
def test_rope_rows(T, heads, D, rot, interleaved):
    """In place at the front of packed heads, as the query and key rotation does; the rest is not touched.  (rot = 24, not
    interleaved: the scalar kernel.)"""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(T + D)
    rows = torch.randn(T, heads + 2, D, generator=g, device="cuda").bfloat16()
    pos = torch.randint(0, 2000, (T,), generator=g, device="cuda", dtype=torch.int32)
    ref = fused.rope_ref(rows[:, :heads].float(), pos, THETA, rot, interleaved).double()
    back = fused.rope_ref(rows[:, :heads].float(), pos, THETA, rot, interleaved, True).double()
    old = rows.clone()
    fused.rope_inplace(rows[:, :heads], pos, THETA, rot, interleaved)
    assert ((rows[:, :heads].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + _angles_bound(pos, old)).all()
    assert torch.equal(rows[:, heads:], old[:, heads:]) and torch.equal(rows[..., rot:], old[..., rot:])
    again = old.clone()
    fused.rope_inplace(again[:, :heads], pos, THETA, rot, interleaved, True)
    assert ((again[:, :heads].double() - back).abs() <= 2.0 ** -8 * back.abs() + _angles_bound(pos, old)).all()


# a thread per pair, one below and at the line; several tokens of few heads a CTA, as many as the angles allow; shares of the heads
@pytest.mark.parametrize("T,heads,D,rot", [(1535, 2, 64, 64), (1536, 2, 64, 64), (9001, 1, 64, 64), (3503, 4, 128, 128),
                                           (2000, 1, 512, 512), (25, 128, 64, 64), (599, 37, 128, 128)])
@pytest.mark.parametrize("interleaved", [False, True])
def test_rope_launches(T, heads, D, rot, interleaved):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(T)
    rows = torch.randn(T, heads + 1, D, generator=g, device="cuda").bfloat16()
    pos = torch.randint(0, 2000, (T,), generator=g, device="cuda", dtype=torch.int32)
    old = rows.clone()
    ref = fused.rope_ref(old[:, :heads].float(), pos, THETA, rot, interleaved).double()
    fused.rope_inplace(rows[:, :heads], pos, THETA, rot, interleaved)
    assert ((rows[:, :heads].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + _angles_bound(pos, old)).all()
    assert torch.equal(rows[:, heads:], old[:, heads:])


@pytest.mark.parametrize("T", [0, 1, 6, 301])
@pytest.mark.parametrize("heads,D,rot", [(0, 192, 64), (1, 32, 16), (5, 192, 64), (128, 192, 64)])
@pytest.mark.parametrize("interleaved", [False, True])
def test_rotated_tail(T, heads, D, rot, interleaved):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(T + heads)
    x, dy = (torch.randn(T, heads, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    pos = torch.randint(0, 2000, (T,), generator=g, device="cuda", dtype=torch.int32)
    x.requires_grad_()
    y = fused.RotateTail.apply(x, pos, THETA, rot, interleaved)
    y.backward(dy)
    for have, src, back in ((y, x.detach(), False), (x.grad, dy, True)):
        tail = src[..., D - rot:].contiguous()
        fused.rope_inplace(tail, pos, THETA, rot, interleaved, back)
        assert torch.equal(have[..., :D - rot], src[..., :D - rot]) and torch.equal(have[..., D - rot:], tail)


@pytest.mark.parametrize("T,h,dn,dr,dv", [(0, 3, 128, 64, 128), (1, 1, 8, 8, 8), (5, 3, 128, 64, 128), (301, 128, 128, 64, 128), (7, 9, 64, 256, 40)])
def test_expanded_latent(T, h, dn, dr, dv):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(T)
    kvu = torch.randn(T, h, dn + dv, generator=g, device="cuda").bfloat16().requires_grad_()
    kr = torch.randn(T, dr, generator=g, device="cuda").bfloat16().requires_grad_()
    k, v = fused.ExpandLatent.apply(kvu, kr, dn)
    assert torch.equal(k, torch.cat([kvu[..., :dn], kr[:, None].expand(T, h, dr)], -1)) and torch.equal(v, kvu[..., dn:])
    dk, dv_ = torch.randn_like(k), torch.randn_like(v)
    torch.autograd.backward([k, v], [dk, dv_])
    assert torch.equal(kvu.grad, torch.cat([dk[..., :dn], dv_], -1))
    ref, mag = dk[..., dn:].double().sum(1), dk[..., dn:].double().abs().sum(1)
    assert ((kr.grad.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + h * 2.0 ** -24 * mag).all()


@pytest.mark.parametrize("B", [1, 33])
@pytest.mark.parametrize("C,dr", [(512, 64), (8, 8), (1024, 32), (520, 64)])
@pytest.mark.parametrize("interleaved", [False, True])
def test_latent_append(B, C, dr, interleaved):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(C)
    kv = torch.randn(B, C + dr + 8, generator=g, device="cuda").bfloat16()[:, :C + dr]
    gain = torch.randn(C, generator=g, device="cuda").bfloat16()
    pos = torch.randint(0, 900, (B,), generator=g, device="cuda", dtype=torch.int32)
    slots = torch.randperm(B + 3, generator=g, device="cuda")[:B]
    cache = torch.full((B + 3, C + dr), 9.0, device="cuda", dtype=torch.bfloat16)
    fused.latent_append(kv, gain, pos, slots, cache, C, 1e-6, THETA, interleaved)
    x = kv[:, :C].double()
    ref = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * gain.double()
    assert ((cache[slots, :C].double() - ref).abs() <= (2.0 ** -8 + C * 2.0 ** -24 + 2.0 ** -20) * ref.abs()).all()
    key = kv[:, C:].reshape(B, 1, dr).contiguous()
    ref = fused.rope_ref(key.float(), pos, THETA, dr, interleaved).double()
    have = cache[slots, C:][:, None].double()
    assert ((have - ref).abs() <= 2.0 ** -8 * ref.abs() + _angles_bound(pos, key)).all()
    left = torch.ones(B + 3, dtype=torch.bool, device="cuda")
    left[slots] = False
    assert bool((cache[left] == 9).all())


@pytest.mark.parametrize("N,K", [(1, 128), (300, 640), (4096, 7168)])
def test_dequantised_weights(N, K):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(N)
    codes = torch.randint(0, 256, (N, K), generator=g, device="cuda", dtype=torch.uint8)
    codes[codes % 128 == 127] = 3                       # no NaN codes
    q, s = codes.view(torch.float8_e4m3fn), torch.rand((N + 127) // 128, K // 128, generator=g, device="cuda")
    before = quant.LAUNCHES["quant"]
    out = quant.dequant_128x128_as(q, s, torch.bfloat16)
    assert quant.LAUNCHES["quant"] == before + 1 and torch.equal(out, quant.dequant_128x128(q, s).bfloat16())
