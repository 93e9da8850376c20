"""What surrounds the model in a decode step: cache rows, contexts and embeddings in front, the drawn tokens behind, and the
sampler's vectors, against plain PyTorch."""
import pytest
import torch

from gcore_b200.ops import fused
from gcore_b200.ops.vocab import sample

pytestmark = pytest.mark.gpu


def _state(B, max_blocks, R, g):
    i32 = dict(dtype=torch.int32, device="cuda")
    return dict(tokens=torch.randint(0, 50, (B,), generator=g, device="cuda"), pos=torch.randint(0, 70, (B,), generator=g, **i32),
                active=torch.rand(B, generator=g, device="cuda") < 0.7, limit=torch.randint(0, 70, (B,), generator=g, **i32),
                block_table=torch.randint(0, 99, (B, max_blocks), generator=g, **i32),
                state=torch.arange(B, **i32), steps=torch.randint(0, 9, (B,), generator=g, **i32),
                ring_idx=torch.tensor([R + 1], device="cuda"), ring_tok=torch.zeros(R, B, dtype=torch.int64, device="cuda"),
                ring_lp=torch.zeros(R, B, device="cuda"))


@pytest.mark.parametrize("B", [1, 5, 300])
@pytest.mark.parametrize("width,dtype", [(None, None), (8, torch.bfloat16), (2056, torch.bfloat16), (12, torch.float32)])
def test_begin_and_end(B, width, dtype):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(B)
    st = _state(B, 4, 3, g)
    embed = None if width is None else torch.randn(50, width, generator=g, device="cuda").to(dtype)
    slots, ctx, states, sink, x = fused.decode_begin(st, 16, embed, 777)
    blk = st["block_table"].gather(1, (st["pos"] // 16).long()[:, None].clamp_max(3)).squeeze(1)
    live = st["active"] & (st["pos"] < st["limit"])
    want = torch.where(live, blk * 16 + st["pos"] % 16, -1)
    assert torch.equal(slots, want.int()) and torch.equal(sink, torch.where(want >= 0, want, 777).long())
    assert torch.equal(ctx, torch.where(live, st["pos"] + 1, 0).int())
    assert torch.equal(states, torch.where(live, st["state"], -1).int())
    assert x is None if embed is None else torch.equal(x, embed[st["tokens"]])
    tok, lp = torch.randint(0, 50, (B,), generator=g, device="cuda"), torch.randn(B, generator=g, device="cuda")
    old = {k: v.clone() for k, v in st.items()}
    fused.decode_end(st, tok, lp)
    assert torch.equal(st["tokens"], tok) and torch.equal(st["steps"], old["steps"] + 1) and int(st["ring_idx"]) == 5
    assert torch.equal(st["pos"], old["pos"] + st["active"].int())
    assert torch.equal(st["ring_tok"][1], tok) and torch.equal(st["ring_lp"][1], lp)      # (3 + 1) % 3
    assert not st["ring_tok"][[0, 2]].any() and not st["ring_lp"][[0, 2]].any()


@pytest.mark.parametrize("B,V", [(1, 40), (3, 16384), (2, 50257), (64, 32768), (1, 152064), (700, 20003)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("pad", [0, 1, 4])
def test_sample(B, V, dtype, pad):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    g = torch.Generator(device="cuda").manual_seed(V + B)
    z = (3 * torch.randn(B, V + pad, generator=g, device="cuda")).to(dtype)[:, pad // 2:pad // 2 + V]
    z[0, V // 2:] = float("-inf")          # masked tokens
    seeds, steps = torch.arange(B, device="cuda"), torch.full((B,), 5, dtype=torch.int32, device="cuda")
    ref = torch.log_softmax(z.double() / 0.8, -1)
    tok, lp = sample(z, 0.8, seeds, steps, True)
    best = z.double().amax(-1)
    assert torch.equal(z.double().gather(1, tok[:, None])[:, 0], best)
    assert torch.equal(tok, (z.double() == best[:, None]).int().argmax(-1))      # the first of equal ones
    # fp32 sums of V terms in chains of at most V / 256, and the fast exponentials' 2^-21
    assert ((lp.double() - ref.gather(1, tok[:, None])[:, 0]).abs() <= 2e-5).all()
    tok, lp = sample(z, 0.8, seeds, steps, False)
    assert ((lp.double() - ref.gather(1, tok[:, None])[:, 0]).abs() <= 2e-5).all()
    assert int(tok[0]) < V // 2
    # the draw does not depend on how the row is laid out or shared out
    again, _ = sample(z.clone(memory_format=torch.contiguous_format)[:1], 0.8, seeds[:1], steps[:1], False)
    assert torch.equal(again, tok[:1])
