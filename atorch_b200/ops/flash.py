"""Front end of the sm_100a flash-attention kernels (csrc/flash_attn.cu, csrc/flash_attn_bwd.cu).

All masks are lowered to one per-row key interval ``[lo, hi)``:

=====================  ==========================================================
causal                 ``hi = i + 1 + (Sk - Sq)``
GLM break-point g[b]   ``hi = max(i + 1, g[b])``
packed GLM [b, 2, P]   ``hi = max(i + 1, max{e_p : s_p <= i})``
key padding            ``[lo, hi) = [first valid key, last valid key + 1)`` when the valid keys of a row are
                       contiguous (right or left padding); masks with holes are unpadded into packed
                       sequences (``cu_seqlens``) like the reference's varlen path
packed sequences       ``lo = start of the row's sequence`` (``cu_seqlens``)
=====================  ==========================================================

(Reference semantics: atorch/modules/transformer/layers.py:1283-1408, docs/FA-glm.md:52-160.)
"""
from __future__ import annotations

import collections
import ctypes
import math
from typing import Optional, Tuple

import torch

from .. import _lib
from .function import call


import os
import weakref

# forward kernel with two 128-row query tiles per CTA that share every K/V tile (csrc/flash_attn_v2.cu): the
# default from 256 query rows on for head dims 128 and 64 (measured at S=4096, H=32, D=128, causal: 118 us against
# 232 us for the single-tile kernel; at B=16, S=512, H=16, D=64, all keys: 40 us against 68 us); ATB_FLASH_V2=0
# keeps the single-tile kernel everywhere
FWD_TWO_TILES = os.environ.get("ATB_FLASH_V2", "1") == "1"
# Head dim 64 keeps the single-tile kernel while its CTAs (128 rows) fit one wave: two tiles a CTA then leave half of the SMs
# without work (16 heads, all keys, single / two tiles: 512 rows, 64 CTAs, 12.4 / 12.8 us; 1024, 128 CTAs, 17.5 / 21.2; two waves,
# 64 heads of 512: 20.7 / 13.9; 32 heads of 1024: 32.5 / 22.3).
ONE_WAVE = 148
# backward as two kernels (dK/dV per key block + dQ per query block; no atomics, no fp32 scratch) where there is neither
# dropout nor a bias. ATB_FLASH_BWD_SPLIT=0 selects the one key-block kernel with TMA reduce-adds of dQ everywhere.
BWD_SPLIT = os.environ.get("ATB_FLASH_BWD_SPLIT", "1") == "1"
# dK/dV kernel: a CTA sums the query heads of its group in tensor memory, as many of them (a divisor of the group) as still
# leave this many CTAs; what is left of a group is summed by a pass over the bf16 results. A CTA per SM will do while a
# head is short (10 x 512, 16 heads on 4, causal, backward in all: 75 us with 160 CTAs, 83 with 320, 89 with 640). From 12 query
# blocks on the last CTAs weigh more, and it takes FOLD_LONG_CTAS (2 x 1536, 32 on 4: 167 us with 192, 156 with 384; 2560, 32 on 8:
# 222 with 160, 188 with 320, 192 with 640; 3584: 338 with 224, 327 with 448, 333 with 896; 4096: 400 with 256, 403 with 512), with
# every key visible too (2 x 1536, 32 on 8: 306 with 192, 281 with 384; 1664, 64 on 16: 335 with 208, 304 with 416; 3 x 1792, 32 on
# 4: 632 with 168, 550 with 336; 4 x 1920, 12 on 3: 343 with 180, 310 with 360; head dim 64, 2 x 1536, 32 on 8: 263 and 237).
# Long heads that all see every key fold whole groups or none (4000, 32 on 4: 758 us unfolded, 807 by 4, 996 by 2).
FOLD_MIN_CTAS = 148
FOLD_LONG_CTAS = 240


def kernels_built() -> bool:
    L = _lib.lib()
    return L is not None and L.has("atb_flash_fwd")


def backward_built() -> bool:
    L = _lib.lib()
    return L is not None and L.has("atb_flash_bwd")


def supported(q, k, v, dropout_p=0.0, additive_mask=None, additive_bias=None, key_padding_mask=None) -> bool:
    if not _lib.use_kernels(q, k, v) or not kernels_built():
        return False
    if additive_mask is not None or additive_bias is not None:
        # soft masks / biases run in the kernels when they can be read as one bf16 tensor without a gradient
        if not _lib.lib().has("atb_flash_fwd_bias") or k.shape[1] % 8 != 0:
            return False
        for t in (additive_mask, additive_bias):
            if t is not None and (t.requires_grad or t.dim() < 2 or t.dim() > 4 or t.shape[-1] != k.shape[1]
                                  or t.shape[-2] not in (1, q.shape[1])):
                return False
    if dropout_p != 0.0 and not (0.0 < dropout_p < 1.0 and _lib.lib().has("atb_flash_fwd_dropout")):
        return False
    if (q.requires_grad or k.requires_grad or v.requires_grad) and torch.is_grad_enabled() and not backward_built():
        return False
    B, Sq, Hq, D = q.shape
    ok = q.dtype == torch.bfloat16 and Hq % k.shape[2] == 0 and \
        (D == 128 or (D == 64 and _lib.lib().has("atb_flash_fwd_ex")))
    if not ok:
        return False
    for t in (q, k, v):
        s0, s1, s2, s3 = t.stride()
        if s3 != 1 or s2 != D or s1 % 8 or s0 != s1 * t.shape[1]:
            return False
    return True


def supported_qkv(qkv: torch.Tensor, num_heads: int) -> bool:
    """:func:`supported` for the three thirds of a contiguous ``qkv [B, S, 3*H, D]`` without dropout, mask tensors or biases."""
    return (_lib.use_kernels(qkv) and kernels_built() and backward_built() and qkv.dtype == torch.bfloat16
            and qkv.is_contiguous() and qkv.shape[2] == 3 * num_heads
            and (qkv.shape[3] == 128 or (qkv.shape[3] == 64 and _lib.lib().has("atb_flash_fwd_ex"))))


def row_intervals(B: int, Sq: int, Sk: int, device, causal: bool = False, glm_mask=None, pack_glm_mask=None,
                  key_padding_mask=None, cu_seqlens=None) -> Tuple[Optional[torch.Tensor], Optional[torch.Tensor]]:
    """Lower the mask arguments to int32 ``(row_lo, row_hi)`` of shape [B, Sq]; ``(None, None)`` when the
    analytic causal / full form inside the kernel is enough."""
    if glm_mask is None and pack_glm_mask is None and key_padding_mask is None and cu_seqlens is None:
        return None, None
    out = _row_intervals_kernel(B, Sq, Sk, device, causal, glm_mask, pack_glm_mask, key_padding_mask, cu_seqlens)
    return out if out is not None else row_intervals_reference(B, Sq, Sk, device, causal, glm_mask, pack_glm_mask,
                                                               key_padding_mask, cu_seqlens)


def _launch_row_intervals(B, Sq, Sk, device, causal, glm_mask, pack_glm_mask, key_padding_mask, cu_seqlens):
    """The lowering in one launch (csrc/masks.cu): ``(row_lo, row_hi, holes)``, or ``None`` for arguments it does not read
    as they are. ``holes`` (int32 per sample, None without a key padding mask) is for the host to look at: an interval can
    only describe valid keys that lie next to each other."""
    device = torch.device(device)
    if device.type != "cuda" or B < 1 or B > 65535 or Sq < 1 or Sk < 1 or _lib.lib() is None:
        return None
    ints = (torch.int32, torch.int64)
    glm, pack, kp, cu = (None if t is None else t.to(device) for t in (glm_mask, pack_glm_mask, key_padding_mask, cu_seqlens))
    if not ((glm is None or (glm.dtype in ints and glm.numel() == B))
            and (pack is None or (pack.dtype in ints and pack.dim() == 3 and pack.shape[0] == B and pack.shape[1] >= 2
                                  and pack.shape[2] > 0))
            and (kp is None or (kp.dtype in (torch.bool, torch.uint8) and kp.shape == (B, Sk)))
            and (cu is None or (cu.dtype in ints and cu.dim() == 1 and cu.numel() >= 2))):
        return None
    glm, kp, cu = (None if t is None else t.contiguous() for t in (glm, kp, cu))
    pack = None if pack is None else pack[:, :2].contiguous()
    is64 = lambda t: int(t is not None and t.dtype == torch.int64)
    buf = torch.empty(2 * B * Sq + B, dtype=torch.int32, device=device)
    lo, hi, holes = buf[: B * Sq].view(B, Sq), buf[B * Sq: 2 * B * Sq].view(B, Sq), buf[2 * B * Sq:]
    with torch.cuda.device(device):
        p = _lib.addr
        rc = _lib.lib().atb_row_intervals(
            p(lo), p(hi), p(holes), B, Sq, Sk, int(causal or glm is not None or pack is not None), p(glm), is64(glm),
            p(pack), is64(pack), 0 if pack is None else pack.shape[2], p(kp), p(cu), is64(cu),
            0 if cu is None else cu.numel(), _lib.stream())
    _lib.check(rc, "atb_row_intervals")
    return lo, hi, holes if kp is not None else None


def _row_intervals_kernel(B, Sq, Sk, device, causal, glm_mask, pack_glm_mask, key_padding_mask, cu_seqlens):
    """``(row_lo, row_hi)`` of the launch; with a key padding mask one host synchronisation."""
    out = _launch_row_intervals(B, Sq, Sk, device, causal, glm_mask, pack_glm_mask, key_padding_mask, cu_seqlens)
    if out is None:
        return None
    if out[2] is not None and any(out[2].tolist()):
        raise NonContiguousKeyMask()
    return out[:2]


class _HolesOnTheWay:
    """The holes that the mask kernel found, on their way to the host: ``device`` for the attention kernel, which does
    nothing if there are any, :meth:`check` for the host, which waits for the mask kernel only."""

    def __init__(self, holes: torch.Tensor):
        self.device = holes
        self.host = holes.to("cpu", non_blocking=True)
        self.event = torch.cuda.Event()
        self.event.record(torch.cuda.current_stream(holes.device))

    def check(self) -> None:
        self.event.synchronize()
        if any(self.host.tolist()):
            raise NonContiguousKeyMask()


# From two waves of forward CTAs on, the forward kernel goes ahead of the host's look at the holes of a key padding mask.
# Forward and backward, right padding, against a look that waits first: 16 x 512, 16 heads of 64 (512 CTAs) 273 -> 236 us,
# 8 x 1024 335 -> 305, 2 x 4096, 32 heads of 128 1820 -> 1750; below two waves the event and the separate copy cost more
# than the wait (4 x 512, 128 CTAs: 191 -> 203).
AHEAD_MIN_CTAS = 296


def _padded_intervals(q, heads, Sk, causal, scale, key_padding_mask, others, drop):
    """``(row_lo, row_hi, look)`` for a key padding mask of self-attention in front of the two-query-tile forward. The host
    has to know whether the mask has holes (those are unpadded), but the forward kernel need not wait for it: it is
    launched first and leaves at once if there are any, and ``look.check()`` comes after it, so that the GPU has work while
    the host waits and starts up again. ``None`` where another forward kernel would run, the mask comes with others or the
    forward is too short."""
    if key_padding_mask is None:
        return None
    B, S = q.shape[:2]
    if drop or any(o is not None for o in others) or Sk != S or S < 256 or not FWD_TWO_TILES or not scale > 0 \
            or B * heads * ((S + 255) // 256) < AHEAD_MIN_CTAS:
        return None
    out = _launch_row_intervals(B, S, S, q.device, causal, None, None, key_padding_mask, None)
    return None if out is None else (out[0], out[1], _HolesOnTheWay(out[2]))


def row_intervals_reference(B: int, Sq: int, Sk: int, device, causal: bool = False, glm_mask=None, pack_glm_mask=None,
                            key_padding_mask=None, cu_seqlens=None):
    """The same in tensor operations: any device, any argument dtype (and the oracle of the kernel's test)."""
    i = torch.arange(Sq, device=device, dtype=torch.int64)
    shift = Sk - Sq
    causal_like = causal or glm_mask is not None or pack_glm_mask is not None
    hi = (i + 1 + shift).clamp(max=Sk)[None].expand(B, Sq).clone() if causal_like else \
        torch.full((B, Sq), Sk, device=device, dtype=torch.int64)
    lo = torch.zeros(B, Sq, device=device, dtype=torch.int64)
    if glm_mask is not None:
        hi = torch.maximum(hi, glm_mask.to(device).long().view(B, 1).expand(B, Sq))
    if pack_glm_mask is not None:
        pm = pack_glm_mask.to(device).long()
        s, e = pm[:, 0], pm[:, 1]                       # [B, P]
        valid = (s >= 0) & (e >= 0)
        applies = valid[:, None, :] & (s[:, None, :] <= i[None, :, None])   # [B, Sq, P]
        ext = torch.where(applies, e[:, None, :].expand(B, Sq, -1), torch.zeros((), device=device, dtype=torch.int64))
        hi = torch.maximum(hi, ext.max(dim=-1).values)
    if cu_seqlens is not None:
        cu = cu_seqlens.to(device).long()
        seg = torch.bucketize(i, cu[1:], right=True).clamp(max=cu.numel() - 2)
        lo = torch.maximum(lo, cu[seg][None].expand(B, Sq))
        if not causal_like:
            hi = torch.minimum(hi, cu[seg + 1][None].expand(B, Sq))
    if key_padding_mask is not None:
        kp = key_padding_mask.to(device).bool()
        cnt = kp.sum(dim=1)
        first = kp.int().argmax(dim=1)
        last = Sk - 1 - kp.flip(1).int().argmax(dim=1)
        # one host sync: an interval can only describe valid keys that lie next to each other
        if not bool(((cnt == 0) | (last - first + 1 == cnt)).all()):
            raise NonContiguousKeyMask()
        last1 = torch.where(cnt > 0, last + 1, torch.zeros_like(last))
        lo = torch.maximum(lo, first.view(B, 1).expand(B, Sq))
        hi = torch.minimum(hi, last1.view(B, 1).expand(B, Sq))
    hi = hi.clamp(max=Sk)
    return lo.to(torch.int32).contiguous(), hi.to(torch.int32).contiguous()


_INTERVAL_CACHE: "collections.OrderedDict" = collections.OrderedDict()   # the layers of one forward share one mask


def intervals_from_additive_mask(additive_mask: torch.Tensor, B: int, Sq: int, Sk: int, causal: bool = False):
    """Cached front of ``_intervals_from_additive_mask``: every layer of a forward pass is given the same mask
    tensor, so the lowering (one pass over the mask and one host synchronisation) runs once per mask, not per layer."""
    key = (additive_mask.data_ptr(), tuple(additive_mask.shape), additive_mask.dtype, additive_mask._version,
           str(additive_mask.device), B, Sq, Sk, bool(causal))
    hit = _INTERVAL_CACHE.get(key)
    if hit is not None and hit[0]() is additive_mask:
        return hit[1]
    out = _intervals_from_additive_mask(additive_mask, B, Sq, Sk, causal)
    try:
        _INTERVAL_CACHE[key] = (weakref.ref(additive_mask), out)
    except TypeError:
        return out
    while len(_INTERVAL_CACHE) > 8:
        _INTERVAL_CACHE.popitem(last=False)
    return out


def _intervals_from_additive_mask(additive_mask: torch.Tensor, B: int, Sq: int, Sk: int, causal: bool = False):
    """Lower a dense mask to per-row key intervals, or return ``None`` when it is not of that form.

    ``additive_mask``: broadcastable to ``[B, 1, Sq, Sk]`` (the same for every head), either boolean (True =
    visible) or additive with entries that are 0 (visible) or <= -1e4 (hidden) — the ``-65504 * (1 - ltor_mask)``
    and ``-inf`` conventions. Causal, GLM prefix, packed-sequence and padding masks all have one contiguous run of
    visible keys per row, which is what the kernels take; a mask with soft biases or holes is left to the dense
    path. Costs one pass over the mask and one host synchronisation."""
    m = additive_mask
    if m.dim() == 4:
        if m.shape[1] != 1:
            return None
        m = m[:, 0]
    elif m.dim() == 2:
        m = m[None]
    if m.dim() != 3 or m.shape[-2:] != (Sq, Sk) or m.shape[0] not in (1, B):
        return None
    if m.dtype == torch.bool:
        vis, binary = m, None
    else:
        vis = m > -1e4
        binary = ((m == 0) | ~vis).all()
    cnt = vis.sum(-1)
    first = vis.int().argmax(-1)
    last = Sk - 1 - vis.flip(-1).int().argmax(-1)
    ok = ((cnt == 0) | (last - first + 1 == cnt)).all()
    if binary is not None:
        ok = ok & binary
    if not bool(ok):
        return None
    lo = torch.where(cnt > 0, first, torch.zeros_like(first)).expand(B, Sq)
    hi = torch.where(cnt > 0, last + 1, torch.zeros_like(last)).expand(B, Sq)
    if causal:
        i = torch.arange(Sq, device=m.device)
        hi = torch.minimum(hi, (i + 1 + (Sk - Sq)).clamp(min=0)[None])
    return lo.to(torch.int32).contiguous(), hi.to(torch.int32).contiguous()


class NonContiguousKeyMask(ValueError):
    """The valid keys of some row are not contiguous: no per-row interval describes the mask."""


def _token_stride(t: torch.Tensor) -> int:
    return t.stride(1)


def bias_config(B: int, Hq: int, Sq: int, Sk: int, additive_mask=None, additive_bias=None):
    """``(tensor, stride_b, stride_h, stride_q)`` for the bias kernels: mask and bias summed into one bf16 tensor
    of shape ``[1|B, 1|H, 1|Sq, Sk]`` (2-D = ``[Sq, Sk]``, 3-D = ``[B, Sq, Sk]``), broadcast dims with stride 0."""
    t = None
    for x in (additive_mask, additive_bias):
        if x is None:
            continue
        if x.dtype == torch.bool:
            x = torch.zeros(x.shape, dtype=torch.float32, device=x.device).masked_fill(~x, float("-inf"))
        x = x[None, None] if x.dim() == 2 else x[:, None] if x.dim() == 3 else x
        t = x.float() if t is None else t + x.float()
    t = t.to(torch.bfloat16).contiguous()
    b, h, sq, sk = t.shape
    assert b in (1, B) and h in (1, Hq) and sq in (1, Sq) and sk == Sk, (t.shape, (B, Hq, Sq, Sk))
    return t, (0 if b == 1 else h * sq * sk), (0 if h == 1 else sq * sk), (0 if sq == 1 else sk)


def dropout_config(dropout_p: float, seed=None) -> Tuple[int, int, int]:
    """``(thr16, seed_lo, seed_hi)`` for the dropout kernels: an element is dropped when its 16 hash bits are below
    ``thr16 = round(p * 65536)`` (so the effective probability is ``thr16 / 65536``). The seed pair is drawn from
    torch's CPU generator (restored by activation checkpointing, so a recomputed forward draws the same mask)
    unless given."""
    thr = min(max(int(round(dropout_p * 65536.0)), 1), 65535)
    if seed is None:
        lo, hi = torch.randint(0, 2 ** 31 - 1, (2,)).tolist()
    else:
        lo, hi = int(seed) & 0xFFFFFFFF, (int(seed) >> 32) & 0xFFFFFFFF
    return thr, lo, hi


def _hash32(x: torch.Tensor) -> torch.Tensor:
    m = 0xFFFFFFFF
    x = x ^ (x >> 16)
    x = (x * 0x7FEB352D) & m
    x = x ^ (x >> 15)
    x = (x * 0x846CA68B) & m
    return x ^ (x >> 16)


def dropout_keep_mask(B: int, Hq: int, Sq: int, Sk: int, drop: Tuple[int, int, int], device="cpu") -> torch.Tensor:
    """The keep mask ``[B, Hq, Sq, Sk]`` (bool) the kernels use for ``drop = (thr16, seed_lo, seed_hi)``: the
    host restatement of ``drop_row_key`` / ``drop_pair_bits`` (csrc/common.cuh), used by the tests."""
    thr, lo, hi = drop
    m = 0xFFFFFFFF
    bh = torch.arange(B * Hq, dtype=torch.int64, device=device)
    base = _hash32(lo ^ ((bh * 0x9E3779B1) & m)) ^ hi                               # [B*Hq]
    rows = torch.arange(Sq, dtype=torch.int64, device=device)
    key = _hash32((base[:, None] + ((rows * 0x85EBCA77) & m)[None]) & m)             # [B*Hq, Sq]
    pairs = torch.arange((Sk + 1) // 2, dtype=torch.int64, device=device)
    w = _hash32(key[:, :, None] ^ ((pairs * 0xC2B2AE3D) & m)[None, None])            # [B*Hq, Sq, Sk/2]
    bits = torch.stack([w & 0xFFFF, w >> 16], dim=-1).reshape(B * Hq, Sq, -1)[:, :, :Sk]
    return (bits >= thr).view(B, Hq, Sq, Sk)


def _extra_args(drop, bias, head_dim=None):
    d = drop if drop is not None else (0, 0, 0)
    extra = tuple(ctypes.c_uint(x) for x in d)
    if bias is not None:
        extra += (_lib.ptr(bias[0]),) + tuple(ctypes.c_longlong(x) for x in bias[1:])
    elif head_dim is not None:
        extra += (None, ctypes.c_longlong(0), ctypes.c_longlong(0), ctypes.c_longlong(0))
    if head_dim is not None:
        extra += (ctypes.c_int(head_dim),)
    return extra


def _as_ctypes(name, args):
    """``args`` under the declared types of launcher ``name``, for a launcher that begins with the same arguments."""
    return tuple(_lib._CTYPE[c](x) for c, x in zip(_lib.SIGNATURES[name], args))


def flash_fwd_raw(q, k, v, causal, softmax_scale, row_lo, row_hi, drop=None, bias=None, holes=None):
    """Launch the forward kernel. Returns (out [B,Sq,Hq,D] bf16, lse [B,Hq,Sq] fp32). ``drop``: see
    ``dropout_config``; dropout runs in the single-tile kernel. ``holes``: see ``_padded_intervals`` (two-tile kernel)."""
    B, Sq, Hq, D = q.shape
    return _forward(q, (q.data_ptr(), k.data_ptr(), v.data_ptr()), (B, Sq, k.shape[1], Hq, k.shape[2]), D,
                    (_token_stride(q), _token_stride(k), _token_stride(v)), causal, softmax_scale, row_lo, row_hi, drop,
                    bias, holes)


def _fused_heads(qkv, H):
    """Addresses and token strides of the q, k and v heads of ``qkv [B, S, 3*H, D]`` (a slice takes longer to make than to
    read)."""
    step = H * qkv.shape[3] * qkv.element_size()
    base = qkv.data_ptr()
    return (base, base + step, base + 2 * step), (_token_stride(qkv),) * 3


def _forward(like, qkv, sizes, D, strides, causal, softmax_scale, row_lo, row_hi, drop=None, bias=None, holes=None):
    """:func:`flash_fwd_raw` on addresses ``qkv`` with token ``strides`` and ``sizes = (B, Sq, Sk, Hq, Hkv)``; ``like``: a
    tensor of their device and dtype."""
    B, Sq, _, Hq, _ = sizes
    out = torch.empty(B, Sq, Hq, D, dtype=like.dtype, device=like.device)
    lse = torch.empty(B, Hq, Sq, dtype=torch.float32, device=like.device)
    L = _lib.lib()
    # two-query-tile kernel (flash_attn_v2.cu) for long enough sequences (and enough blocks, see ONE_WAVE); the single-tile
    # kernel otherwise, and for
    # dropout, a bias, and a scale that is not positive (hidden scores are -inf before they are scaled)
    p = _lib.addr
    args = (*qkv, out.data_ptr(), lse.data_ptr(), p(row_lo), p(row_hi), *sizes, *strides, int(causal), softmax_scale,
            _lib.stream(), _lib.status_addr(like))
    if FWD_TWO_TILES and Sq >= 256 and drop is None and bias is None and softmax_scale > 0 \
            and (D == 128 or B * Hq * ((Sq + 127) // 128) > ONE_WAVE):
        rc = L.atb_flash_fwd_v2(*args, D, p(holes))
    elif D == 128 and bias is None and drop is None:
        rc = L.atb_flash_fwd(*args)
    else:
        fwd, extra = (L.atb_flash_fwd_ex, _extra_args(drop, bias, D)) if D != 128 else \
            (L.atb_flash_fwd_bias, _extra_args(drop, bias)) if bias is not None else \
            (L.atb_flash_fwd_dropout, _extra_args(drop, None))        # single-tile kernel
        rc = fwd(*_as_ctypes("atb_flash_fwd", args), *extra)
    _lib.check(rc, "atb_flash_fwd")
    return out, lse


def _fold(group: int, ctas: int, q_blocks: int, causal: bool) -> int:
    """Query heads per CTA of the dK/dV kernel (see FOLD_MIN_CTAS); ``ctas``: its CTAs with whole groups."""
    need = FOLD_MIN_CTAS if q_blocks < 12 else FOLD_LONG_CTAS
    return next((f for f in range(group, 1, -1) if group % f == 0 and ctas * (group // f) >= need
                 and (f == group or causal or q_blocks < 16)), 1)


def flash_bwd_raw(dout, q, k, v, out, lse, causal, softmax_scale, row_lo, row_hi, fused_out: bool = False,
                  drop=None, bias=None):
    """Launch the backward kernels. Returns (dq, dk, dv) shaped like q, k, v. With ``fused_out`` (and
    equal query / key-value head counts) the three are slices of ONE ``[B, S, 3*H, D]`` buffer laid out
    like a fused q|k|v projection output, so the gradient of that projection needs no concatenation."""
    B, Sq, Hq, D = q.shape
    return _backward(q, (q.data_ptr(), k.data_ptr(), v.data_ptr()), (B, Sq, k.shape[1], Hq, k.shape[2]), D,
                     (_token_stride(q), _token_stride(k), _token_stride(v)), dout, out, lse, causal, softmax_scale, row_lo,
                     row_hi, fused_out, drop, bias)


def _backward(like, qkv, sizes, D, strides, dout, out, lse, causal, softmax_scale, row_lo, row_hi, fused_out=False, drop=None,
              bias=None):
    """:func:`flash_bwd_raw` on addresses, see :func:`_forward`."""
    B, Sq, Sk, Hq, Hkv = sizes
    dev, dt = like.device, like.dtype
    split = BWD_SPLIT and drop is None and bias is None
    dq_acc = None if split else torch.zeros(B, Sq, Hq, D, dtype=torch.float32, device=dev)
    fold = _fold(Hq // Hkv, B * Hkv * ((Sk + 127) // 128), (Sq + 127) // 128, bool(causal)) if split else 1
    # row sums; the two-kernel form with intervals keeps two words per query block behind them
    rows = B * Hq * Sq
    ranges = 2 * B * ((Sq + 127) // 128) if split and (row_lo is not None or row_hi is not None) else 0
    delta = torch.empty(rows + (rows & 1) + ranges, dtype=torch.float32, device=dev)
    if fused_out and Hkv == Hq and Sq == Sk:
        fused = torch.empty(B, Sq, 3 * Hq, D, dtype=dt, device=dev)
        grads, (dq_stride, dkv_stride, _) = _fused_heads(fused, Hq)
    else:
        fused = None
        dq = torch.empty(B, Sq, Hq, D, dtype=dt, device=dev)
        dk = torch.empty(B, Sk, Hq // fold, D, dtype=dt, device=dev)
        dv = torch.empty(B, Sk, Hq // fold, D, dtype=dt, device=dev)
        grads, dq_stride, dkv_stride = (dq.data_ptr(), dk.data_ptr(), dv.data_ptr()), Hq * D, Hq // fold * D
    dout = dout if (dout.stride(-1) == 1 and dout.stride(2) == D and dout.stride(0) == dout.stride(1) * Sq) \
        else dout.contiguous()
    L, p = _lib.lib(), _lib.addr
    dims = (p(row_lo), p(row_hi), *sizes, *strides, _token_stride(dout), dq_stride, dkv_stride, int(causal), softmax_scale,
            _lib.stream(), _lib.status_addr(like))
    ins = (dout.data_ptr(), *qkv, out.data_ptr(), lse.data_ptr(), delta.data_ptr())
    if split:
        rc = L.atb_flash_bwd_split(*ins, *grads, *dims, fold, D)
    else:
        if D != 128:
            bwd, extra = L.atb_flash_bwd_ex, _extra_args(drop, bias, D)
        elif bias is not None:
            bwd, extra = L.atb_flash_bwd_bias, _extra_args(drop, bias)
        elif drop is not None:
            bwd, extra = L.atb_flash_bwd_dropout, _extra_args(drop, None)
        else:
            bwd, extra = L.atb_flash_bwd, ()
        args = _as_ctypes("atb_flash_bwd_split", (*ins, *grads, *dims))
        rc = bwd(*args[: len(ins)], _lib.ptr(dq_acc), *args[len(ins):], *extra)
    _lib.check(rc, "atb_flash_bwd")
    if fused is not None:
        return fused
    if Hkv * fold != Hq:
        parts, (dk, dv) = (dk, dv), (torch.empty(B, Sk, Hkv, D, dtype=dt, device=dev) for _ in range(2))
        rc = L.atb_head_sum(*map(p, parts), p(dk), p(dv), B * Sk * Hkv, Hq // Hkv // fold, D, _lib.stream())
        _lib.check(rc, "atb_head_sum")
    return dq, dk, dv


class _FlashAttn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, causal, scale, row_lo, row_hi, drop=None, bias=None, look=None):
        out, lse = flash_fwd_raw(q, k, v, causal, scale, row_lo, row_hi, drop, bias, None if look is None else look.device)
        if look is not None:
            look.check()
        ctx.save_for_backward(q, k, v, out, lse, row_lo, row_hi)
        ctx.cfg = (causal, scale, drop, bias)       # bias: (bf16 tensor, strides), not differentiated
        return out

    @staticmethod
    def backward(ctx, dout):
        q, k, v, out, lse, row_lo, row_hi = ctx.saved_tensors
        causal, scale, drop, bias = ctx.cfg
        dq, dk, dv = flash_bwd_raw(dout, q, k, v, out, lse, causal, scale, row_lo, row_hi, drop=drop, bias=bias)
        return dq, dk, dv, None, None, None, None, None, None, None


def flash_attention(q, k, v, causal=False, softmax_scale=None, glm_mask=None, pack_glm_mask=None,
                    key_padding_mask=None, cu_seqlens=None, dropout_p=0.0, dropout_seed=None,
                    additive_mask=None, additive_bias=None):
    """``dropout_p``: attention dropout inside the kernels (the mask is a counter-based hash of batch, head, row
    and column, see ``dropout_keep_mask``); ``dropout_seed`` fixes the mask, otherwise torch's CPU generator
    supplies the seed."""
    B, Sq, Hq, D = q.shape
    Sk = k.shape[1]
    scale = softmax_scale if softmax_scale is not None else 1.0 / math.sqrt(D)
    if Sq == 1:
        causal = False   # single-query decode sees every key
    padded = _padded_intervals(q, Hq, Sk, causal, scale, key_padding_mask,
                               (glm_mask, pack_glm_mask, cu_seqlens, additive_mask, additive_bias), dropout_p > 0.0)
    try:
        if padded is not None:
            return call(_FlashAttn, q, k, v, bool(causal), float(scale), padded[0], padded[1], None, None, padded[2])
        lo, hi = row_intervals(B, Sq, Sk, q.device, causal, glm_mask, pack_glm_mask, key_padding_mask, cu_seqlens)
    except NonContiguousKeyMask:
        if additive_mask is not None or additive_bias is not None:
            from .attention import attention_reference

            return attention_reference(q, k, v, causal, scale, glm_mask, pack_glm_mask, key_padding_mask, cu_seqlens,
                                       additive_mask, additive_bias, dropout_p)
        return _unpadded_attention(q, k, v, key_padding_mask, causal, scale, glm_mask, pack_glm_mask, cu_seqlens,
                                   dropout_p, dropout_seed)
    drop = dropout_config(dropout_p, dropout_seed) if dropout_p > 0.0 else None
    bias = None
    if additive_mask is not None or additive_bias is not None:
        bias = bias_config(B, Hq, Sq, Sk, additive_mask, additive_bias)
    return call(_FlashAttn, q, k, v, bool(causal), float(scale), lo, hi, drop, bias)


def _unpadded_attention(q, k, v, key_padding_mask, causal, scale, glm_mask, pack_glm_mask, cu_seqlens,
                        dropout_p=0.0, dropout_seed=None):
    """Key-padding mask with holes (self-attention): drop the padded tokens, run the batch as packed
    sequences, put the results back (padded positions get zeros). Mirrors the reference's unpad / pad
    path (atorch/modules/transformer/layers.py:76-95,1363-1408)."""
    B, S, H, D = q.shape
    if k.shape[1] != S or glm_mask is not None or pack_glm_mask is not None or cu_seqlens is not None:
        from .attention import attention_reference

        return attention_reference(q, k, v, causal, scale, glm_mask, pack_glm_mask, key_padding_mask, cu_seqlens,
                                   dropout_p=dropout_p)
    kp = key_padding_mask.to(q.device).bool()
    idx = kp.reshape(-1).nonzero(as_tuple=False)[:, 0]
    cu = torch.zeros(B + 1, dtype=torch.int32, device=q.device)
    cu[1:] = kp.sum(1).cumsum(0)
    pick = lambda t: t.reshape(B * S, t.shape[2], D).index_select(0, idx).unsqueeze(0)
    out_p = flash_attention(pick(q), pick(k), pick(v), causal=causal, softmax_scale=scale, cu_seqlens=cu,
                            dropout_p=dropout_p, dropout_seed=dropout_seed)
    out = torch.zeros(B * S, H, D, dtype=q.dtype, device=q.device)
    out = out.index_copy(0, idx, out_p[0])
    return out.view(B, S, H, D)


def _fused_forward(qkv, H, causal, scale, row_lo, row_hi, look):
    B, S, _, D = qkv.shape
    heads, strides = _fused_heads(qkv, H)
    return _forward(qkv, heads, (B, S, S, H, H), D, strides, causal, scale, row_lo, row_hi,
                    holes=None if look is None else look.device)


class _FlashAttnQKV(torch.autograd.Function):
    """Attention on a fused projection output ``qkv [B, S, 3*H, D]`` (q heads, then k, then v). The
    backward emits one fused gradient tensor in the same layout: no slice-backward zero fills or adds."""

    @staticmethod
    def forward(ctx, qkv, H, causal, scale, row_lo, row_hi, cached, look=None):
        if cached is not None:
            out, lse = cached          # output and log-sum-exp kept from the first pass of a checkpointed block
        else:
            out, lse = _fused_forward(qkv, H, causal, scale, row_lo, row_hi, look)
        if look is not None:
            look.check()
        ctx.save_for_backward(qkv, out, lse, row_lo, row_hi)
        ctx.cfg = (H, causal, scale)
        return out

    @staticmethod
    def backward(ctx, dout):
        qkv, out, lse, row_lo, row_hi = ctx.saved_tensors
        H, causal, scale = ctx.cfg
        B, S, _, D = qkv.shape
        heads, strides = _fused_heads(qkv, H)
        dqkv = _backward(qkv, heads, (B, S, S, H, H), D, strides, dout, out, lse, causal, scale, row_lo, row_hi,
                         fused_out=True)
        return dqkv, None, None, None, None, None, None, None


def flash_attention_qkv(qkv: torch.Tensor, num_heads: int, causal: bool = True, softmax_scale=None,
                        recompute_cache=None, **mask_kwargs):
    """qkv: ``[B, S, 3*num_heads, D]``; returns ``[B, S, num_heads, D]``.

    ``recompute_cache`` (an ``OrderedDict`` owned by the calling layer) lets an activation-checkpointed
    block keep the attention output and log-sum-exp of its first (no-grad) pass: that pass stores
    ``(out, lse)`` under the pass token of its checkpoint node (utils/checkpoint.py), the recomputation
    of the same node takes the entry with the same token and skips the forward kernel. A forward that
    is not the first pass of a checkpointed block has no token and neither stores nor reads, and an
    entry whose backward never ran is evicted once more than ``RECOMPUTE_CACHE_LIMIT`` are held.
    32 MB per layer at 7B scale buys one attention forward per layer per step."""
    from ..utils.checkpoint import current_pass

    B, S, _, D = qkv.shape
    scale = softmax_scale if softmax_scale is not None else 1.0 / math.sqrt(D)
    look = None
    padded = _padded_intervals(qkv, num_heads, S, causal, scale, mask_kwargs.get("key_padding_mask"),
                               [v for n, v in mask_kwargs.items() if n not in ("key_padding_mask", "dropout_p", "dropout_seed")],
                               mask_kwargs.get("dropout_p", 0.0) > 0.0)
    try:
        if padded is not None:
            lo, hi, look = padded
        else:
            lo, hi = row_intervals(B, S, S, qkv.device, causal, mask_kwargs.get("glm_mask"),
                                   mask_kwargs.get("pack_glm_mask"), mask_kwargs.get("key_padding_mask"),
                                   mask_kwargs.get("cu_seqlens"))
        cached = None
        cur = current_pass() if recompute_cache is not None else None
        if cur is not None:
            token, is_recompute = cur
            if not is_recompute and not torch.is_grad_enabled():
                out, lse = _fused_forward(qkv, num_heads, bool(causal), float(scale), lo, hi, look)
                if look is not None:
                    look.check()
                recompute_cache[token] = (out, lse)
                while len(recompute_cache) > RECOMPUTE_CACHE_LIMIT:
                    recompute_cache.popitem(last=False)
                return out
            if is_recompute:
                cached = recompute_cache.pop(token, None)
                if cached is not None and cached[0].shape != (B, S, num_heads, D):
                    cached = None
        return call(_FlashAttnQKV, qkv, num_heads, bool(causal), float(scale), lo, hi, cached, look)
    except NonContiguousKeyMask:
        H = num_heads
        return flash_attention(qkv[:, :, :H], qkv[:, :, H: 2 * H], qkv[:, :, 2 * H:], causal=causal,
                               softmax_scale=softmax_scale, **mask_kwargs)


RECOMPUTE_CACHE_LIMIT = 16   # first passes in flight per layer (pipeline micro-batches) before eviction
