"""The embedding table's gradient in fp32 and the logits' gradient in 16-byte units, against 64 bits."""
import pytest
import torch

from gcore_b200.ops import fused, vocab

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,V,H", [(0, 5, 16), (1, 10, 8), (13, 4, 264), (900, 50, 2048), (5000, 3000, 2056)])
def test_embedding_gradient(n, V, H):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(n)
    w = torch.nn.Parameter(torch.randn(V, H, generator=g, device="cuda").bfloat16())
    w.main_grad = torch.randn(V, H, generator=g, device="cuda")
    old = w.main_grad.clone()
    ids = torch.randint(0, max(1, V - 1), (n,), generator=g, device="cuda")
    ids[:n // 3] = 2 % V                                    # a long run of one token
    dy = torch.randn(n, H, generator=g, device="cuda").bfloat16()
    y = fused.embedding(ids, w)
    assert torch.equal(y, w.detach()[ids])
    y.backward(dy)
    assert w.grad is None
    rows = torch.zeros(V, H, device="cuda", dtype=torch.double).index_add_(0, ids, dy.double())
    mag = torch.zeros(V, H, device="cuda", dtype=torch.double).index_add_(0, ids, dy.double().abs())
    assert ((w.main_grad.double() - old.double() - rows).abs() <= n * 2.0 ** -24 * (mag + old.double().abs())).all()
    assert torch.equal(w.main_grad[V - 1], old[V - 1]) or V == 1


@pytest.mark.parametrize("runs", [[128], [129], [1, 127, 1], [5, 250, 1, 128, 128, 3], [256, 256, 1], [1000, 2, 9000], [64, 192, 300]])
def test_runs_that_cross_blocks(runs):
    """Runs of equal tokens that end at, before and behind the borders of the kernel's blocks of 128; the same bits each time."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    H, n = 72, sum(runs)
    g = torch.Generator(device="cuda").manual_seed(n)
    ids = torch.cat([torch.full((r,), 3 * k, device="cuda") for k, r in enumerate(runs)])
    ids = ids[torch.randperm(n, generator=g, device="cuda")]
    w = torch.nn.Parameter(torch.zeros(3 * len(runs), H, device="cuda", dtype=torch.bfloat16))
    old = torch.randn(w.shape, generator=g, device="cuda")
    dy = torch.randn(n, H, generator=g, device="cuda").bfloat16()
    rows = torch.zeros(w.shape, device="cuda", dtype=torch.double).index_add_(0, ids, dy.double())
    mag = torch.zeros(w.shape, device="cuda", dtype=torch.double).index_add_(0, ids, dy.double().abs())
    got = []
    for _ in range(2):
        w.main_grad = old.clone()
        fused.embedding(ids, w).backward(dy)
        # blocks of 128 one after another, then their sums
        assert ((w.main_grad.double() - old.double() - rows).abs()
                <= (129 + n // 128) * 2.0 ** -24 * (mag + old.double().abs())).all()
        got.append(w.main_grad)
    assert torch.equal(*got)


@pytest.mark.parametrize("V,pad", [(40, 0), (1003, 0), (32768, 0), (32768, 3), (4100, 4)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("entropy", [False, True])
def test_logits_gradient(V, pad, dtype, entropy):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from gcore_b200.ops import _lib
    T = 5
    g = torch.Generator(device="cuda").manual_seed(V)
    whole = torch.randn(T, V + pad, generator=g, device="cuda").to(dtype)
    z = whole[:, :V]
    kept = whole.clone()
    tg = torch.randint(0, V, (T,), generator=g, device="cuda")
    tg[0] = V + 7                                            # another rank's target
    gl, gh = (torch.randn(T, generator=g, device="cuda") for _ in range(2))
    zd = z.double() / 0.7
    lse = torch.logsumexp(zd, -1)
    p = (zd - lse[:, None]).exp()
    H = lse - (p * zd).sum(-1)
    hot = torch.zeros(T, V, device="cuda", dtype=torch.double)
    hot[1:].scatter_(1, tg[1:, None], 1.0)
    ref = gl.double()[:, None] * (hot - p)
    if entropy:
        ref = ref - gh.double()[:, None] * p * (zd - lse[:, None] + H[:, None])
    ref = ref / 0.7
    ls, en = lse.float(), H.float()
    _lib.check(_lib.kernels().gk_logprob_entropy_bwd(
        _lib.ptr(z), int(dtype == torch.float32), z.stride(0), _lib.ptr(tg), _lib.ptr(ls), _lib.ptr(en), _lib.ptr(gl),
        _lib.ptr(gh if entropy else None), 1 / 0.7, 0, V, T, _lib.stream_ptr()), "logprob_entropy_bwd")
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23
    # fp32 of lse (2^-22 of about 10) inside the exponential, whose fast form has 2^-21
    assert ((z.double() - ref).abs() <= u * ref.abs() + 2e-5 * (ref.abs() + p * 10)).all()
    assert torch.equal(whole[:, V:], kept[:, V:])
