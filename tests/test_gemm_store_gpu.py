"""Results that leave a GEMM through TMA copies and reductions: ragged edges, results inside a larger buffer, sums into C,
expert planes without rows; against 64-bit products."""
import pytest
import torch

from gcore_b200.ops import _lib
from gcore_b200.ops import gemm as G

pytestmark = pytest.mark.gpu


def _rand(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda").bfloat16()


def _bound(a, b, K):
    # fp32 sums of K products of exact bf16 values: sqrt(K) roundings of 2^-24 of the sum of magnitudes
    return 4 * K ** 0.5 * 2.0 ** -24 * (a.double().abs() @ b.double().abs().t()) + 1e-12


# (M, N, K): 256 x 256 tiles with ragged rows and columns, a partial last wave, 128-row tiles, one narrow tile; more than half as
# many 128-row tiles as SMs, of several k-blocks and of one
@pytest.mark.parametrize("M,N,K", [(1100, 2052, 520), (2049, 4100, 264), (300, 200, 136), (129, 264, 72), (40, 36, 64),
                                   (1100, 2050, 520), (300, 201, 136), (900, 2600, 136), (900, 2600, 64)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_dense(M, N, K, dtype):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a, b, bias = _rand(g, M, K), _rand(g, N, K), _rand(g, N)
    ref, bound = a.double() @ b.double().t(), _bound(a, b, K)
    rnd = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23
    pad = torch.full((M + 2, N + 8 - N % 8 + 16), 3.0, device="cuda", dtype=dtype)
    out = pad[1:M + 1, 8:N + 8]
    G.gemm(a, b, out=out, bias=bias, alpha=0.5)
    want = 0.5 * ref + bias.double()
    assert ((out.double() - want).abs() <= bound + rnd * want.abs()).all()
    edge = pad.clone()
    edge[1:M + 1, 8:N + 8] = 3.0
    assert bool((edge == 3).all())
    if dtype == torch.float32:
        old = out.clone()
        G.gemm(a, b, out=out, accumulate=True)
        want = old.double() + ref
        assert ((out.double() - want).abs() <= bound + rnd * want.abs()).all()
        edge = pad.clone()
        edge[1:M + 1, 8:N + 8] = 3.0
        assert bool((edge == 3).all())
    _lib.check_device_errors()


@pytest.mark.parametrize("N,K", [(384, 264), (136, 40)])
def test_weight_gradient_of_experts(N, K):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(N + K)
    rows = [128, 0, 384, 128, 0]
    off = torch.tensor([0] + rows).cumsum(0).to(torch.int32).cuda()
    M = sum(rows)
    dy, x = _rand(g, M, N), _rand(g, M, K)
    old = torch.randn(len(rows), N, K, generator=g, device="cuda")
    out = old.clone()
    G.grouped_wgrad(dy, x, off, len(rows), out=out, accumulate=True)
    fresh = G.grouped_wgrad(dy, x, off, len(rows))
    for e in range(len(rows)):
        a, b = dy[off[e]:off[e + 1]].t(), x[off[e]:off[e + 1]].t()
        ref, bound = a.double() @ b.double().t(), _bound(a, b, max(rows[e], 1))
        assert ((fresh[e].double() - ref).abs() <= bound + 2.0 ** -23 * ref.abs()).all()
        want = old[e].double() + ref
        assert ((out[e].double() - want).abs() <= bound + 2.0 ** -23 * want.abs()).all()
        if not rows[e]:
            assert torch.equal(out[e], old[e])
    _lib.check_device_errors()


@pytest.mark.parametrize("N,K", [(384, 264), (200, 72), (48, 136), (4096, 136)])
def test_expert_rows(N, K):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(N + K)
    rows = [256, 0, 128]
    off = torch.tensor([0] + rows).cumsum(0).to(torch.int32).cuda()
    x, w = _rand(g, 512, K), _rand(g, 3, N, K)
    out = torch.full((512, N), 5.0, device="cuda", dtype=torch.bfloat16)
    G.grouped_gemm(x, w, off, out=out)
    for e in range(3):
        a = x[off[e]:off[e + 1]]
        ref = a.double() @ w[e].double().t()
        assert ((out[off[e]:off[e + 1]].double() - ref).abs() <= _bound(a, w[e], K) + 2.0 ** -8 * ref.abs()).all()
    assert bool((out[384:] == 5).all())       # rows behind the last segment are not written
    _lib.check_device_errors()


@pytest.mark.parametrize("N,K", [(384, 264), (48, 136), (4096, 136)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_segments_that_end_inside_a_tile(N, K, dtype):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(N + K)
    rows = [100, 0, 257, 32, 140, 1]
    off = torch.tensor([0] + rows).cumsum(0).to(torch.int32).cuda()
    x, w = _rand(g, 640, K), _rand(g, len(rows), N, K)
    for _ in range(5):
        out = torch.full((640, N), 5.0, device="cuda", dtype=dtype)
        G.grouped_gemm(x, w, off, out=out)
        rnd = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23
        for e in range(len(rows)):
            a = x[off[e]:off[e + 1]]
            ref = a.double() @ w[e].double().t()
            assert ((out[off[e]:off[e + 1]].double() - ref).abs() <= _bound(a, w[e], K) + rnd * ref.abs()).all()
        assert bool((out[sum(rows):] == 5).all())
    _lib.check_device_errors()
