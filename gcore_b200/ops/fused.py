"""Autograd wrappers for the bandwidth-bound block kernels (``csrc/elementwise.cu``): RMSNorm with fused residual
add, RoPE, SwiGLU.  Each has a plain PyTorch implementation used on CPU and as the test oracle."""
from __future__ import annotations

import ctypes

import torch

from . import _lib

LAUNCHES = {"elementwise": 0}


# ------------------------------------------------------------------------------------------------ RMSNorm
def rmsnorm_ref(x, w, eps, residual=None):
    if residual is not None:
        x = (x.float() + residual.float()).to(x.dtype)
    xf = x.float()
    y = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps) * w.float()
    return y.to(x.dtype), x


class _RmsNormFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, residual, eps):
        H = x.shape[-1]
        x2 = x.reshape(-1, H)
        T = x2.shape[0]
        y = torch.empty_like(x2)
        rstd = torch.empty(T, dtype=torch.float32, device=x.device)
        res_out = None
        r2 = None
        if residual is not None:
            r2 = residual.reshape(-1, H)
            res_out = torch.empty_like(x2)
        LAUNCHES["elementwise"] += 1
        _lib.check(_lib.kernels().gk_rmsnorm_fwd(_lib.ptr(x2), _lib.ptr(r2), _lib.ptr(w), _lib.ptr(y),
                                                 _lib.ptr(res_out), _lib.ptr(rstd), T, H, float(eps),
                                                 _lib.stream_ptr()), "rmsnorm_fwd")
        normed_in = res_out if residual is not None else x2
        ctx.save_for_backward(normed_in, w, rstd)
        ctx.shape = x.shape
        ctx.has_res = residual is not None
        if residual is not None:
            return y.reshape(x.shape), res_out.reshape(x.shape)
        return y.reshape(x.shape)

    @staticmethod
    def backward(ctx, gy, gres=None):
        xin, w, rstd = ctx.saved_tensors
        T, H = xin.shape
        lib = _lib.kernels()
        gy2 = gy.reshape(T, H).contiguous()
        gres2 = gres.reshape(T, H).contiguous() if gres is not None else None
        dx = torch.empty_like(xin)
        parts = lib.gk_rmsnorm_bwd_parts(T)
        partial = torch.empty(parts * H, dtype=torch.float32, device=xin.device)
        dw = torch.empty(H, dtype=torch.float32, device=xin.device)
        LAUNCHES["elementwise"] += 2
        _lib.check(lib.gk_rmsnorm_bwd(_lib.ptr(gy2), _lib.ptr(xin), _lib.ptr(w), _lib.ptr(rstd), _lib.ptr(gres2),
                                      _lib.ptr(dx), _lib.ptr(partial), _lib.ptr(dw), 0, T, H, _lib.stream_ptr()),
                   "rmsnorm_bwd")
        dx = dx.reshape(ctx.shape)
        return dx, dw.to(w.dtype), (dx if ctx.has_res else None), None


def rmsnorm(x: torch.Tensor, w: torch.Tensor, eps: float = 1e-6, residual: torch.Tensor | None = None):
    """Returns ``(norm(x + residual) * w, x + residual)``; with ``residual=None`` the second value is ``x``."""
    if x.dtype == torch.bfloat16 and _lib.use_native(x) and x.shape[-1] % 8 == 0 and x.shape[-1] <= 8192:
        if not x.is_contiguous():
            x = x.contiguous()
        if residual is not None and not residual.is_contiguous():
            residual = residual.contiguous()
        if residual is None:
            return _RmsNormFn.apply(x, w, None, eps), x
        return _RmsNormFn.apply(x, w, residual, eps)
    return rmsnorm_ref(x, w, eps, residual)


# ------------------------------------------------------------------------------------------------ embedding
class _EmbeddingFn(torch.autograd.Function):
    """Embedding rows; the table's gradient is added to its fp32 ``main_grad`` (rows of equal tokens in a fixed order),
    autograd sees none."""

    @staticmethod
    def forward(ctx, ids, weight, main_grad):
        ctx.save_for_backward(ids)
        ctx.main_grad = main_grad
        return torch.nn.functional.embedding(ids, weight)

    @staticmethod
    def backward(ctx, g):
        (ids,) = ctx.saved_tensors
        V, H = ctx.main_grad.shape
        g = g.reshape(-1, H)
        g = g if g.is_contiguous() and g.data_ptr() % 16 == 0 else g.clone(memory_format=torch.contiguous_format)
        order, rows = torch.sort(ids.reshape(-1), stable=True)
        lib = _lib.kernels()
        scratch = torch.empty(lib.gk_embedding_grad_scratch(rows.numel(), H), dtype=torch.float32, device=g.device)
        LAUNCHES["elementwise"] += 1
        _lib.check(lib.gk_embedding_grad(_lib.ptr(order), _lib.ptr(rows), _lib.ptr(g), _lib.ptr(ctx.main_grad),
                                         _lib.ptr(scratch), rows.numel(), H, V, _lib.stream_ptr()), "embedding_grad")
        return None, None, None


def embedding(ids: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    """``weight[ids]``; a bf16 table with an fp32 ``main_grad`` on a GPU collects its gradient there."""
    mg = getattr(weight, "main_grad", None) if weight.requires_grad and torch.is_grad_enabled() else None
    if (mg is not None and _lib.use_native(weight) and weight.dtype == torch.bfloat16 and ids.dtype == torch.int64
            and mg.dtype == torch.float32 and mg.is_contiguous() and mg.shape == weight.shape and mg.data_ptr() % 16 == 0
            and weight.shape[1] % 8 == 0):
        return _EmbeddingFn.apply(ids, weight, mg)
    return torch.nn.functional.embedding(ids, weight)


# ------------------------------------------------------------------------------------------------ RoPE
def mrope_tables(pos3: torch.Tensor, theta: float, rot: int, sections, interleaved_sections: bool = True):
    """Multi-axis rotary tables.  ``pos3`` [T, 3] = (temporal, height, width) index of every token; frequency ``i``
    of the ``rot / 2`` frequencies takes its angle from one of the three axes: chunked (``sections = (t, h, w)``
    consecutive frequencies per axis, Qwen2-VL) or interleaved (frequency ``i`` uses axis ``i % 3`` while that axis
    still has budget, the rest temporal, Qwen3-VL; gpatch_v4/extended_model/qwen3_vl.py).  Returns ``(cos, sin)``
    fp32 ``[T, rot / 2]``, accepted wherever a rotary op takes position ids."""
    half = rot // 2
    assert sum(sections) == half, f"mrope sections {sections} must sum to {half}"
    inv = theta ** (-torch.arange(0, half, device=pos3.device, dtype=torch.float32) * 2.0 / rot)
    axis = torch.zeros(half, dtype=torch.long, device=pos3.device)
    if interleaved_sections:
        idx = torch.arange(half, device=pos3.device)
        for a in (1, 2):
            axis[(idx % 3 == a) & (idx < 3 * sections[a])] = a
    else:
        o = 0
        for a, n in enumerate(sections):
            axis[o:o + n] = a
            o += n
    ang = pos3.float()[:, axis] * inv[None, :]
    return ang.cos().contiguous(), ang.sin().contiguous()


def rope_ref(x, pos, theta, rot=None, interleaved=False, backward=False):
    """x: [T, nheads, D]; rotate-half pairing (i, i + rot/2) unless ``interleaved``.  ``pos``: position ids [T] or a
    ``(cos, sin)`` pair of tables [T, rot / 2] (see ``mrope_tables``)."""
    D = x.shape[-1]
    rot = rot or D
    half = rot // 2
    if isinstance(pos, tuple):
        c, s = pos[0][:, None, :], pos[1][:, None, :]
    else:
        inv = theta ** (-torch.arange(0, half, device=x.device, dtype=torch.float32) * 2.0 / rot)
        ang = pos.float()[:, None] * inv[None, :]
        c, s = ang.cos()[:, None, :], ang.sin()[:, None, :]
    if backward:
        s = -s
    xf = x.float()
    xr = xf[..., :rot]
    if interleaved:
        a, b = xr[..., 0::2], xr[..., 1::2]
        o = torch.stack([a * c - b * s, b * c + a * s], dim=-1).flatten(-2)
    else:
        a, b = xr[..., :half], xr[..., half:]
        o = torch.cat([a * c - b * s, b * c + a * s], dim=-1)
    return torch.cat([o, xf[..., rot:]], dim=-1).to(x.dtype)


def rope_inplace(x: torch.Tensor, pos: torch.Tensor, theta: float, rot: int | None = None,
                 interleaved: bool = False, backward: bool = False):
    """In-place RoPE on ``x`` [T, nheads, D]; ``x`` may be a slice of a packed QKV buffer (any token stride)."""
    T, nh, D = x.shape
    rot = rot or D
    if x.dtype == torch.bfloat16 and _lib.use_native(x) and x.stride(2) == 1 and x.stride(1) == D:
        if isinstance(pos, tuple):
            LAUNCHES["elementwise"] += 1
            _lib.check(_lib.kernels().gk_rope_table(_lib.ptr(x), _lib.ptr(pos[0]), _lib.ptr(pos[1]), T, nh, D, rot,
                                                    x.stride(0), int(backward), int(interleaved), _lib.stream_ptr()),
                       "rope_table")
            return x
        p32 = pos if pos.dtype == torch.int32 else pos.to(torch.int32)
        LAUNCHES["elementwise"] += 1
        _lib.check(_lib.kernels().gk_rope(_lib.ptr(x), _lib.ptr(p32), T, nh, D, rot, x.stride(0), float(theta),
                                          int(backward), int(interleaved), _lib.stream_ptr()), "rope")
        return x
    x.copy_(rope_ref(x, pos, theta, rot, interleaved, backward))
    return x


class _RopeFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, pos, theta, rot, interleaved):
        ctx.pos = pos   # position ids or (cos, sin) tables: never differentiated
        ctx.args = (theta, rot, interleaved)
        return rope_inplace(x.clone(), pos, theta, rot, interleaved, False)

    @staticmethod
    def backward(ctx, g):
        pos = ctx.pos
        theta, rot, interleaved = ctx.args
        return rope_inplace(g.clone(), pos, theta, rot, interleaved, True), None, None, None, None


def rope(x, pos, theta, rot=None, interleaved=False):
    return _RopeFn.apply(x, pos, theta, rot, interleaved)


class RotateTail(torch.autograd.Function):
    """``x`` [T, heads, D] (bf16 on a GPU, contiguous) with the last ``rot`` values of every head rotated; ``pos`` int32."""

    @staticmethod
    def forward(ctx, x, pos, theta, rot, interleaved):
        ctx.save_for_backward(pos)
        ctx.args = (theta, rot, interleaved)
        return RotateTail._turn(x, pos, theta, rot, interleaved, 0)

    @staticmethod
    def backward(ctx, g):
        (pos,) = ctx.saved_tensors
        return RotateTail._turn(g.contiguous(), pos, *ctx.args, 1), None, None, None, None

    @staticmethod
    def _turn(x, pos, theta, rot, interleaved, backward):
        (T, nh, D), y = x.shape, torch.empty_like(x)
        LAUNCHES["elementwise"] += 1
        _lib.check(_lib.kernels().gk_rope_copy(_lib.ptr(x), _lib.ptr(y), _lib.ptr(pos), T, nh, D, D - rot, rot, float(theta),
                                               backward, int(interleaved), _lib.stream_ptr()), "rope_copy")
        return y


class ExpandLatent(torch.autograd.Function):
    """Keys ``[T, heads, dn + dr]`` and values ``[T, heads, dv]`` from the up-projected latent ``kvu`` [T, heads, dn + dv] and
    the shared rotated key ``kr`` [T, dr] (bf16 on a GPU, contiguous)."""

    @staticmethod
    def forward(ctx, kvu, kr, dn):
        (T, h, w), dr = kvu.shape, kr.shape[1]
        k = torch.empty(T, h, dn + dr, dtype=kvu.dtype, device=kvu.device)
        v = torch.empty(T, h, w - dn, dtype=kvu.dtype, device=kvu.device)
        ctx.sizes = (T, h, dn, dr, w - dn)
        LAUNCHES["elementwise"] += 1
        _lib.check(_lib.kernels().gk_mla_expand(_lib.ptr(kvu), _lib.ptr(kr), _lib.ptr(k), _lib.ptr(v), T, h, dn, dr, w - dn,
                                                _lib.stream_ptr()), "mla_expand")
        return k, v

    @staticmethod
    def backward(ctx, dk, dv):
        T, h, dn, dr, w = ctx.sizes
        dk, dv = dk.contiguous(), dv.contiguous()
        dkvu = torch.empty(T, h, dn + w, dtype=dk.dtype, device=dk.device)
        dkr = torch.empty(T, dr, dtype=dk.dtype, device=dk.device)
        LAUNCHES["elementwise"] += 1
        _lib.check(_lib.kernels().gk_mla_expand_bwd(_lib.ptr(dk), _lib.ptr(dv), _lib.ptr(dkvu), _lib.ptr(dkr), T, h, dn, dr, w,
                                                    _lib.stream_ptr()), "mla_expand_bwd")
        return dkvu, dkr, None


def latent_append(kv, gain, pos, slots, cache, kv_lora: int, eps: float, theta: float, interleaved: bool):
    """One decode token per request: RMSNorm of the latent ``kv[:, :kv_lora]`` and the rotation of the shared key behind it,
    written to the rows ``slots`` (int64) of ``cache`` [rows, kv_lora + dr] (bf16 on a GPU)."""
    LAUNCHES["elementwise"] += 1
    _lib.check(_lib.kernels().gk_latent_append(_lib.ptr(kv), kv.stride(0), _lib.ptr(gain), _lib.ptr(pos), _lib.ptr(slots),
                                               _lib.ptr(cache), kv.shape[0], kv_lora, cache.shape[1] - kv_lora, float(eps),
                                               float(theta), int(interleaved), _lib.stream_ptr()), "latent_append")


# ------------------------------------------------------------------------------------------------ SwiGLU
def qk_headnorm_(qkv: torch.Tensor, wq: torch.Tensor, wk: torch.Tensor, Hq: int, Hk: int, D: int, eps: float):
    """In-place per-head RMSNorm of the query and key heads of packed ``[T, (Hq + 2 Hk) * D]`` rows (inference: no
    autograd).  One kernel on a GPU; the same arithmetic through ``rmsnorm`` elsewhere."""
    T = qkv.shape[0]
    if (qkv.dtype == torch.bfloat16 and _lib.use_native(qkv) and D % 8 == 0 and D <= 256 and qkv.stride(1) == 1
            and wq.dtype == torch.bfloat16 and hasattr(_lib.kernels(), "gk_qk_headnorm")):
        LAUNCHES["elementwise"] += 1
        _lib.check(_lib.kernels().gk_qk_headnorm(_lib.ptr(qkv), _lib.ptr(wq), _lib.ptr(wk), T, Hq, Hk, D,
                                                 qkv.stride(0), float(eps), _lib.stream_ptr()), "qk_headnorm")
        return qkv
    v = qkv.view(T, Hq + 2 * Hk, D)
    v[:, :Hq] = rmsnorm(v[:, :Hq].reshape(-1, D), wq, eps)[0].view(T, Hq, D)
    v[:, Hq:Hq + Hk] = rmsnorm(v[:, Hq:Hq + Hk].reshape(-1, D), wk, eps)[0].view(T, Hk, D)
    return qkv


def swiglu_ref(x):
    g, u = x.float().chunk(2, dim=-1)
    return (torch.nn.functional.silu(g) * u).to(x.dtype)


class _SwigluFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        F = x.shape[-1] // 2
        x2 = x.reshape(-1, 2 * F)
        out = torch.empty(x2.shape[0], F, dtype=x.dtype, device=x.device)
        LAUNCHES["elementwise"] += 1
        _lib.check(_lib.kernels().gk_swiglu_fwd(_lib.ptr(x2), _lib.ptr(out), x2.shape[0], F, _lib.stream_ptr()),
                   "swiglu_fwd")
        ctx.save_for_backward(x2)
        ctx.shape = x.shape
        return out.reshape(*x.shape[:-1], F)

    @staticmethod
    def backward(ctx, g):
        (x2,) = ctx.saved_tensors
        F = x2.shape[1] // 2
        g2 = g.reshape(-1, F).contiguous()
        din = torch.empty_like(x2)
        LAUNCHES["elementwise"] += 1
        _lib.check(_lib.kernels().gk_swiglu_bwd(_lib.ptr(g2), _lib.ptr(x2), _lib.ptr(din), x2.shape[0], F,
                                                _lib.stream_ptr()), "swiglu_bwd")
        return din.reshape(ctx.shape)


def swiglu(x: torch.Tensor, n_rows: torch.Tensor = None) -> torch.Tensor:
    """``silu(x[..., :F]) * x[..., F:]`` for ``x = [gate | up]``.  ``n_rows`` (one int32 on the device, inference only):
    rows of the 2-D ``x`` at or beyond it are not computed and their output is undefined - for expert-sorted buffers
    that are sized for the worst case and carry the count of rows in use on the device."""
    if x.dtype == torch.bfloat16 and _lib.use_native(x) and (x.shape[-1] // 2) % 8 == 0:
        if not x.is_contiguous():
            x = x.contiguous()
        if n_rows is not None and x.dim() == 2 and not (torch.is_grad_enabled() and x.requires_grad) \
                and n_rows.dtype == torch.int32 and hasattr(_lib.kernels(), "gk_swiglu_fwd_rows"):
            F = x.shape[1] // 2
            out = torch.empty(x.shape[0], F, dtype=x.dtype, device=x.device)
            LAUNCHES["elementwise"] += 1
            _lib.check(_lib.kernels().gk_swiglu_fwd_rows(_lib.ptr(x), _lib.ptr(out), x.shape[0], F, _lib.ptr(n_rows),
                                                         _lib.stream_ptr()), "swiglu_fwd_rows")
            return out
        return _SwigluFn.apply(x)
    return swiglu_ref(x)


def decode_begin(st, block: int, embed=None, sink=None):
    """In front of a decode step over the batch state ``st`` (GPU tensors): ``(slots, ctx, states, sink_slots, x)``, the cache
    row of every request's token (-1 where nothing is stored: a row that rests or has reached its limit), the tokens it sees,
    its recurrent state's slot or -1, with ``sink`` the rows once more with ``sink`` for -1 (int64), and with ``embed`` the
    tokens' embedding rows."""
    B, max_blocks = st["block_table"].shape
    dev = st["pos"].device
    slots, ctx, states = (torch.empty(B, dtype=torch.int32, device=dev) for _ in range(3))
    sink_slots = torch.empty(B, dtype=torch.int64, device=dev) if sink is not None else None
    x = torch.empty(B, embed.shape[1], dtype=embed.dtype, device=dev) if embed is not None else None
    ptrs = (ctypes.c_void_p * 12)(*[t.data_ptr() if t is not None else None for t in (
        st["tokens"], st["pos"], st["active"], st["limit"], st["block_table"], st["state"], embed, slots, ctx, states,
        sink_slots, x)])
    dims = (ctypes.c_longlong * 6)(B, max_blocks, block, embed.shape[1] * embed.element_size() if embed is not None else 0,
                                   embed.shape[0] if embed is not None else 0, sink if sink is not None else 0)
    LAUNCHES["elementwise"] += 1
    _lib.check(_lib.kernels().gk_decode_begin(ptrs, dims, _lib.stream_ptr()), "decode_begin")
    return slots, ctx, states, sink_slots, x


def decode_end(st, tok, lp):
    """Behind a decode step: the drawn tokens into the batch state and, with their log-probs, into the output ring; active
    rows advance."""
    ptrs = (ctypes.c_void_p * 9)(*[t.data_ptr() for t in (tok, lp, st["active"], st["tokens"], st["pos"], st["steps"],
                                                         st["ring_idx"], st["ring_tok"], st["ring_lp"])])
    LAUNCHES["elementwise"] += 1
    _lib.check(_lib.kernels().gk_decode_end(ptrs, st["tokens"].numel(), st["ring_tok"].shape[0], _lib.stream_ptr()),
               "decode_end")
