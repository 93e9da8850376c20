"""Token movement of mixture-of-experts layers, forward and backward, and the decode step's layer, against plain PyTorch."""
import pytest
import torch

from gcore_b200.models import moe as M
from gcore_b200.models.config import ModelConfig
from gcore_b200.ops import _lib, moe

pytestmark = pytest.mark.gpu


def _ids(g, T, K, E, skew):
    score = torch.rand(T, E, generator=g, device="cuda")
    if skew:
        score[:, E // 3] += 1          # every token takes this expert
        score[:, -1] -= 1              # hardly any the last one
    return score.topk(K, -1).indices


@pytest.mark.parametrize("T,K,E", [(1, 1, 3), (5, 2, 8), (300, 8, 128), (2049, 2, 33), (700, 9, 512)])
@pytest.mark.parametrize("seg", [16, 128])
@pytest.mark.parametrize("skew", [False, True])
def test_plan(T, K, E, seg, skew):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    ids = _ids(torch.Generator(device="cuda").manual_seed(T + E), T, K, E, skew)
    dest, src, off = moe.plan_rows(ids, E, seg)
    flat = ids.reshape(-1).cpu()
    counts = torch.bincount(flat, minlength=E)
    want_off = torch.cat([torch.zeros(1, dtype=torch.long), ((counts + seg - 1) // seg * seg).cumsum(0)])
    assert torch.equal(off.cpu().long(), want_off) and src.numel() >= int(want_off[-1])
    want_src = torch.full((int(want_off[-1]),), -1)
    for e in range(E):
        n = (flat == e).nonzero()[:, 0]
        want_src[want_off[e]:want_off[e] + len(n)] = n
    assert torch.equal(src[:len(want_src)].cpu().long(), want_src)
    assert torch.equal(want_src[dest.reshape(-1).cpu().long()], torch.arange(T * K))


@pytest.mark.parametrize("T,K,E,H", [(1, 1, 3, 8), (37, 3, 8, 264), (513, 8, 32, 2048)])
def test_movement_and_gradients(T, K, E, H):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(T)
    ids = _ids(g, T, K, E, True)
    x = torch.randn(T, H, generator=g, device="cuda").bfloat16().requires_grad_()
    w = torch.rand(T, K, generator=g, device="cuda").requires_grad_()
    dy = torch.randn(T, H, generator=g, device="cuda").bfloat16()
    dest, src, off = moe.plan_rows(ids, E)
    used = int(off[-1])
    rows = moe.GatherRows.apply(x, dest, src, off)
    want = torch.zeros(used, H, device="cuda", dtype=torch.bfloat16)
    want[dest.reshape(-1).long()] = x.detach().repeat_interleave(K, 0)
    assert torch.equal(rows[:used], want)
    scale = torch.randn(rows.shape[0], 1, generator=g, device="cuda").bfloat16()
    z = (rows * scale).detach().requires_grad_()
    y = moe.CombineRows.apply(z, w, dest, src, off)
    at = dest.long()
    zd, wd = z.detach().double(), w.detach().bfloat16().double()
    ref = (wd[:, :, None] * zd[at]).sum(1)
    mag = (wd[:, :, None] * zd[at]).abs().sum(1)
    # every term and the sum are rounded to bf16 (8 significant bits: 2^-8 of the value at most), K additions in fp32
    u = 2.0 ** -8
    assert ((y.double() - ref).abs() <= u * (ref.abs() + (1 + u) * mag) + K * 2.0 ** -23 * mag).all()
    y.backward(dy)
    gz = torch.zeros(used, H, device="cuda", dtype=torch.double)
    gz[at.reshape(-1)] = (wd[:, :, None] * dy.double()[:, None]).reshape(T * K, H)
    assert ((z.grad[:used].double() - gz).abs() <= u * gz.abs()).all()      # padding rows: exactly zero
    gw = (zd[at] * dy.double()[:, None]).sum(-1)
    mag = (zd[at] * dy.double()[:, None]).abs().sum(-1)      # products and their sum are rounded to bf16
    assert ((w.grad.double() - gw).abs() <= u * (gw.abs() + (1 + u) * mag) + H * 2.0 ** -24 * mag).all()
    up = torch.randn(rows.shape[0], H, generator=g, device="cuda").bfloat16()
    rows.backward(up)
    gx = up.double()[at].sum(1)
    mag = up.double()[at].abs().sum(1)
    assert ((x.grad.double() - gx).abs() <= K * u * (1 + u) ** K * mag).all()      # K sums, each rounded to bf16


def _layer(H, F, E, K, kind, g):
    cfg = ModelConfig(arch="qwen3_moe", num_layers=1, hidden_size=H, num_attention_heads=2, num_kv_heads=2, head_dim=64,
                      ffn_hidden_size=F, vocab_size=128, num_experts=E, moe_top_k=K, moe_ffn_hidden_size=F,
                      moe_router_type=kind, moe_norm_topk_prob=True, **(
                          dict(moe_n_group=4, moe_topk_group=2, moe_router_bias=True, moe_routed_scaling_factor=2.5)
                          if kind != "softmax" else {}))
    layer = M.MoELayer(cfg, 0, 1, 1, "cuda")
    with torch.no_grad():
        for p in layer.parameters():
            p.copy_(torch.randn(p.shape, generator=g, device="cuda") * p.shape[-1] ** -0.5)
        if layer.router.expert_bias is not None:
            layer.router.expert_bias.copy_(0.1 * torch.randn(E, generator=g, device="cuda"))
    return layer.eval()


@pytest.mark.parametrize("T", [1, 16, 17, 128])
@pytest.mark.parametrize("H,F,E,K,kind", [(256, 64, 32, 4, "softmax"), (264, 192, 64, 8, "sigmoid"), (2048, 768, 128, 8, "softmax"),
                                          (136, 128, 32, 1, "softmax")])
@pytest.mark.parametrize("skew", [False, True])
def test_decode_layer(T, H, F, E, K, kind, skew):
    """Against 64 bits and against the general path; with ``skew`` all tokens share their experts (several segments)."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(T + H)
    layer = _layer(H, F, E, K, kind, g)
    x = torch.randn(1 if skew else T, H, generator=g, device="cuda").bfloat16().expand(T, H).contiguous()
    with torch.no_grad():
        assert layer._native(x) and layer._decode_ready(x)
        y, aux = layer(x)
        assert aux is None
        idx, w, _ = layer.router(x)
        dest, src, off = moe.plan_rows(idx, E)
        rows = layer.experts(moe.GatherRows.apply(x, dest, src, off), off)
        general = moe.CombineRows.apply(rows, w, dest, src, off)
        up, down = layer.experts.linear_fc1.weight.double(), layer.experts.linear_fc2.weight.double()
        ref, mag = torch.zeros(T, H, device="cuda", dtype=torch.double), torch.zeros(T, H, device="cuda", dtype=torch.double)
        for k in range(K):
            for t in range(T):
                e = int(idx[t, k])
                a, b = (up[e] @ x[t].double()).chunk(2)
                v = torch.nn.functional.silu(a) * b
                ref[t] += w[t, k].double() * (down[e] @ v)
                mag[t] += w[t, k].double() * (down[e].abs() @ v.abs())
    # roundings of 2^-8 each: activation, expert output, weight, term, sum (the last four act on |output| <= mag)
    assert ((y.double() - ref).abs() <= 5 * 2.0 ** -8 * mag + 1e-6).all()
    # and no further from 64 bits than the general path, which also rounds gate and up
    err, other = ((z.double() - ref).norm() / ref.norm() for z in (y, general))
    assert err <= 1.05 * other + 1e-4
    _lib.check_device_errors()


def test_decode_layer_ends_while_an_earlier_error_stands():
    """Another kernel's error makes waits give up early: the launches end, and the ones after the report are right."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(1)
    layer = _layer(1024, 256, 64, 8, "softmax", g)
    x = torch.randn(40, 1024, generator=g, device="cuda").bfloat16()
    with torch.no_grad():
        assert layer._decode_ready(x)
        ref, _ = layer(x)
        for _ in range(5):
            _lib.err_flag(x.device).fill_(1)
            layer(x)
            with pytest.raises(RuntimeError, match="timed-out wait"):
                _lib.check_device_errors()
            assert torch.equal(layer(x)[0], ref)
    _lib.check_device_errors()
