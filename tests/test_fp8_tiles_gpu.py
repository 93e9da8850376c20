"""The block-fp8 GEMM where its tile widths meet their edges (ragged rows and columns, a last tile of one column block, groups)."""
import pytest
import torch

from gcore_b200.ops import _lib, quant

pytestmark = pytest.mark.gpu


def _close(y, a, b, K):
    """The tensor core adds the 128 exact products of a block with at least 13 bits below its largest term; then one fp32
    rounding per block, and the rounding of the result."""
    ref, mag = a @ b.t(), a.abs() @ b.abs().t()
    u = 2.0 ** -8 if y.dtype == torch.bfloat16 else 2.0 ** -23
    return ((y.double() - ref).abs() <= u * ref.abs() + (2.0 ** -13 + K // 128 * 2.0 ** -23) * mag).all()


# enough rows for the wide tiles to be taken, and few; N: whole and half wide tiles, ragged
@pytest.mark.parametrize("M", [130, 4000, 9472])
@pytest.mark.parametrize("N,K", [(512, 1024), (640, 1152), (1000, 1280), (1928, 640), (2304, 1024)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_dense(M, N, K, dtype):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(M + N)
    aq, sa = quant.quant_act_1x128(torch.randn(M, K, generator=g, device="cuda").bfloat16())
    bq, sb = quant.quant_weight_128x128(torch.randn(N, K, generator=g, device="cuda").bfloat16())
    y = quant.gemm_fp8_blockscaled(aq, sa, bq, sb, out_dtype=dtype)
    assert _close(y, quant.dequant_1x128(aq, sa).double(), quant.dequant_128x128(bq, sb).double(), K)
    _lib.check_device_errors()


@pytest.mark.parametrize("N", [512, 384, 640])
def test_groups(N):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    K, rows = 1024, [2560, 0, 6400, 128]
    g = torch.Generator(device="cuda").manual_seed(N)
    off = torch.tensor([0] + rows).cumsum(0).to(torch.int32).cuda()
    G = len(rows)
    aq, sa = quant.quant_act_1x128(torch.randn(sum(rows) + 128, K, generator=g, device="cuda").bfloat16())
    ws = [quant.quant_weight_128x128(torch.randn(N, K, generator=g, device="cuda").bfloat16()) for _ in range(G)]
    bq, sb = torch.cat([w[0].view(torch.uint8) for w in ws]).view(torch.float8_e4m3fn), torch.cat([w[1] for w in ws])
    y = quant.gemm_fp8_grouped(aq, sa, bq, sb, off, G, out_dtype=torch.float32)
    a = quant.dequant_1x128(aq, sa).double()
    for e in range(G):
        s = slice(int(off[e]), int(off[e + 1]))
        assert rows[e] == 0 or _close(y[s], a[s], quant.dequant_128x128(*ws[e]).double(), K)
    _lib.check_device_errors()
