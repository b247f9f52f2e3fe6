"""Second half of the CUDA op layer: attention, MoE, log-prob head, sampling, quantisation."""
from __future__ import annotations

import math
import os

import torch

from . import reference as ref
from .cuda import BF16, LIMIT_KV_BLOCKS, LIMIT_KV_SLOTS, LIMIT_MOE_PAIRS, C, _apply, _c, gemm_nn, gemm_nt, gemm_tn, publish_limit, transformed

# ---------------------------------------------------------------------------------------------
# attention
# ---------------------------------------------------------------------------------------------


USE_TC_ATTENTION = os.environ.get("MILES_TC_ATTENTION", "1") != "0"
USE_TC_ATTENTION_BWD = os.environ.get("MILES_TC_ATTENTION_BWD", "1") != "0"


class _FlashAttn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, cu_seqlens, max_seqlen, causal):
        T, Hq, D = q.shape
        assert q.stride(2) == 1 and q.stride(1) == D and k.stride(1) == D and v.stride(1) == D and v.stride(2) == 1
        scale = 1.0 / math.sqrt(D)
        o = torch.empty(T, Hq, D, dtype=q.dtype, device=q.device)
        lse = torch.empty(Hq, T, dtype=torch.float32, device=q.device)
        if T > 0 and cu_seqlens.numel() > 1:
            if max_seqlen <= 0:
                max_seqlen = int((cu_seqlens[1:] - cu_seqlens[:-1]).max().item())
            if D == 128 and USE_TC_ATTENTION and q.stride(0) % 8 == 0 and k.stride(0) % 8 == 0 and v.stride(0) % 8 == 0:
                # tcgen05 forward (TMA-fed, accumulators in tensor memory)
                C.flash_fwd_tc(q, k, v, o, lse, cu_seqlens, max_seqlen, scale, causal, C.error_flag(q), None)
            else:
                C.flash_fwd(q, k, v, o, lse, cu_seqlens, max_seqlen, scale, causal)
        ctx.save_for_backward(q, k, v, o, lse, cu_seqlens)
        ctx.max_seqlen, ctx.causal, ctx.scale = max_seqlen, causal, scale
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, o, lse, cu = ctx.saved_tensors
        do = _c(do)
        dq = torch.empty(q.shape, dtype=q.dtype, device=q.device)
        dk = torch.empty(k.shape, dtype=k.dtype, device=k.device)
        dv = torch.empty(v.shape, dtype=v.dtype, device=v.device)
        delta = torch.empty_like(lse)
        D = q.shape[-1]
        if (D == 128 and USE_TC_ATTENTION_BWD and q.stride(0) % 8 == 0 and k.stride(0) % 8 == 0 and v.stride(0) % 8 == 0
                and q.stride(1) == D and k.stride(1) == D and v.stride(1) == D):
            # tcgen05 backward: Sᵀ/dPᵀ and the dK, dV, dQ accumulators live in tensor memory
            C.flash_bwd_tc(q, k, v, o, do, lse, delta, dq, dk, dv, cu, ctx.max_seqlen, ctx.scale, ctx.causal, C.error_flag(q))
        else:
            C.flash_bwd(q, k, v, o, do, lse, delta, dq, dk, dv, cu, ctx.max_seqlen, ctx.scale, ctx.causal)
        return dq, dk, dv, None, None, None


def attention_varlen(q, k, v, cu_seqlens, max_seqlen=0, causal=True):
    if q.dtype != BF16 or q.shape[-1] not in (64, 128):
        return ref.attention_varlen(q, k, v, cu_seqlens, causal)
    return _apply(_FlashAttn, q, k, v, cu_seqlens.to(torch.int32), int(max_seqlen), bool(causal))


_DECODE_SPLITS = int(os.environ.get("MILES_DECODE_SPLITS", "8"))   # KV splits per (request, kv head) in paged decode
# whoever asks for a number of splits gets the form that has them: a request's sums are then cut in the same places whatever else is in the
# batch (one split, for rollouts that have to agree with the trainer)
_DECODE_BY_TILES = "MILES_DECODE_SPLITS" not in os.environ
# Up to so many (request, KV head) segments the form that splits each of them runs as one wave, eight CTAs per segment on 148 SMs × 2, and an
# even share of all tiles has nothing to even out, but a longer chain from length to page.  µs per layer, split / tiles, cache from memory:
# 8 requests × 4 KV heads of 300, 700, 1500, 3000 keys 8.8 / 10.2, 10.1 / 12.5, 11.9 / 13.7, 16.0 / 18.4; 4 × 8 7.9 / 9.1, 9.1 / 11.1,
# 10.8 / 11.8, 15.0 / 16.3; 7 × 4 of 430 to 3000 14.8 / 14.2; 1 × 4 8.4 / 7.6 (700), 13.2 / 12.8 (3000).  Beyond it the split form needs a
# second wave or longer splits: 10 × 4 10.6 / 10.2, 12.5 / 13.1, 18.0 / 14.8, 26.1 / 19.9, of 430 to 3000 17.9 / 15.2; 6 × 8 26.7 / 21.0 (3000).
_DECODE_TILES_FROM = 33


def extend_attention(q, k_cache, v_cache, block_table, seq_lens, q_lens, extend=None):
    """New tokens of each request attend to that request's whole paged KV (which already contains them): the keys and
    values are gathered from the cache into packed buffers and the tcgen05 forward kernel runs with separate query and key
    sequences — query i of a request sees keys ≤ i + (Lk − Lq)."""
    T, Hq, D = q.shape
    Hkv = k_cache.shape[2]
    if extend is None:                       # callers outside the engine: build the description here (host round trip)
        bs = k_cache.shape[1]
        sl, ql = seq_lens.tolist(), q_lens.tolist()
        slots = [int(block_table[b, p // bs]) * bs + p % bs for b, L in enumerate(sl) for p in range(L)]
        cu_q = torch.tensor([0] + list(torch.tensor(ql).cumsum(0).tolist()), dtype=torch.int32, device=q.device)
        cu_k = torch.tensor([0] + list(torch.tensor(sl).cumsum(0).tolist()), dtype=torch.int32, device=q.device)
        extend = {"cu_q": cu_q, "cu_k": cu_k, "kv_slots": torch.tensor(slots, dtype=torch.int64, device=q.device), "max_k": max(sl)}
    max_q = int(q_lens.max().item()) if "max_q" not in extend else extend["max_q"]
    if q.dtype != BF16 or D != 128 or not USE_TC_ATTENTION:
        return ref.paged_attention(q, k_cache, v_cache, block_table, seq_lens, q_lens=q_lens)
    slots = extend["kv_slots"]
    if (k_cache.dtype == v_cache.dtype == BF16 and k_cache.shape == v_cache.shape and k_cache.is_contiguous() and v_cache.is_contiguous()
            and slots.dtype == torch.int64 and slots.is_contiguous() and k_cache.data_ptr() % 16 == v_cache.data_ptr() % 16 == 0):
        kk, vv = C.kv_gather(k_cache, v_cache, slots, C.error_flag(q))
    else:
        kk = k_cache.view(-1, Hkv, D).index_select(0, slots)
        vv = v_cache.view(-1, Hkv, D).index_select(0, slots)
    q = _c(q)
    o = torch.empty(T, Hq, D, dtype=q.dtype, device=q.device)
    lse = torch.empty(Hq, T, dtype=torch.float32, device=q.device)
    C.flash_fwd_tc(q, kk, vv, o, lse, extend["cu_q"], max_q, 1.0 / math.sqrt(D), True, C.error_flag(q), extend["cu_k"])
    return o


# The one-launch form of a decode step's attention takes up to so many (request, KV head) segments with so many CTAs each: one of the chip's waves, and no more
# than an SM and a half of each, because the projection behind brings its weights to the SMs' memory meanwhile.  µs of a step of 8 layers, three launches / 6,
# 7, 8, 12 CTAs per segment: 16 segments of 700 to 3000 keys 606 / 586, 581, 576, 565; 24 of 300 to 900 596 / 585, 587, 582, 635; 28 of 128 to 4096 676 /
# 649, 648, 634, 657; 32 of 300 to 1500 606 / 594, 596, 615, 649, of 128 to 4096 658 / 635, 635, 621, 659; 4 and 8 segments 8 / 16 CTAs 660 / 645 (12 layers)
# and 547 / 523.  Beyond, even shares of all tiles: 40 of 128 to 4096 667 / 697 with 8, 687 with 4.
_ATTEND_SEGMENTS = 32


def _attend_split(segments: int) -> int:
    return 16 if segments <= 8 else 12 if segments <= 18 else 8 if segments <= 28 else 7


def decode_attention(q, k, v, q_w, k_w, positions, theta, eps, k_cache, v_cache, slot_mapping, block_table, seq_lens):
    """A decode step's attention from its projections (one new token per request): norm and rotation of q and k, the cache write of (k, v) and attention over the
    paged cache, in one launch for few (request, KV head) segments; None where that form does not apply."""
    B, Hq, D = q.shape
    Hkv = k.shape[1]
    segments = B * Hkv
    if (not _DECODE_BY_TILES or not 0 < segments <= _ATTEND_SEGMENTS or D != 128 or q.dtype != BF16 or k_cache.dtype != BF16 or Hq % Hkv or Hq // Hkv not in (1, 2, 4, 8)
            or torch.is_grad_enabled() or transformed() or k_cache.shape[1] % 16 or k_cache.shape[2] != Hkv or not k_cache.is_contiguous() or not v_cache.is_contiguous()
            or (q_w is None) != (k_w is None) or any(t.stride(2) != 1 or t.stride(1) != D for t in (q, k, v)) or k_cache.data_ptr() % 16 or v_cache.data_ptr() % 16
            or positions.dtype != torch.int32 or slot_mapping.dtype != torch.int64 or block_table.dtype != torch.int32 or seq_lens.dtype != torch.int32
            or not all(t.is_contiguous() for t in (positions, slot_mapping, block_table, seq_lens)) or positions.numel() != B or slot_mapping.numel() != B):
        return None
    publish_limit(LIMIT_KV_SLOTS, k_cache.shape[0] * k_cache.shape[1])
    publish_limit(LIMIT_KV_BLOCKS, k_cache.shape[0])
    out = torch.empty(B, Hq, D, dtype=q.dtype, device=q.device)
    split = _attend_split(segments)
    C.decode_attend(q, k, v, q_w, k_w, positions, float(theta), float(eps), k_cache, v_cache, slot_mapping, block_table, seq_lens, out, 1.0 / math.sqrt(D), split,
                    C.error_flag(q))
    return out


def paged_attention(q, k_cache, v_cache, block_table, seq_lens, q_lens=None, max_q_len=1, extend=None):
    """Decode (one new token per request) over the paged cache; with `q_lens` a prefill that continues cached KV
    (`extend_attention`)."""
    if q_lens is not None:
        if extend is not None:
            extend = dict(extend, max_q=int(max_q_len))
        return extend_attention(q, k_cache, v_cache, block_table, seq_lens, q_lens, extend)
    B, Hq, D = q.shape
    group = Hq // k_cache.shape[2]
    if q.dtype != BF16 or D not in (64, 128) or group not in (1, 2, 4, 8):
        return ref.paged_attention(q, k_cache, v_cache, block_table, seq_lens)
    q = _c(q)
    out = torch.empty_like(q)
    publish_limit(LIMIT_KV_BLOCKS, k_cache.shape[0])
    if (_DECODE_BY_TILES and B * k_cache.shape[2] >= _DECODE_TILES_FROM and k_cache.shape[1] % 64 == 0 and k_cache.is_contiguous()
            and v_cache.is_contiguous() and block_table.is_contiguous()):
        # whole 64-key tiles inside a page: an even share of all tiles per CTA
        C.paged_decode_tiles(q, k_cache, v_cache, block_table, seq_lens, out, 1.0 / math.sqrt(D), C.error_flag(q))
        return out
    # enough (request, kv head, split) CTAs for two waves of the 148 SMs, never more splits than that needs
    splits = max(1, min(_DECODE_SPLITS, -(-296 // (B * k_cache.shape[2]))))
    part_o = torch.empty(B * Hq * splits * D, dtype=torch.float32, device=q.device)
    part_ml = torch.empty(B * Hq * splits * 2, dtype=torch.float32, device=q.device)
    C.paged_decode(q, k_cache, v_cache, block_table, seq_lens, out, part_o, part_ml, 1.0 / math.sqrt(D), splits)
    return out


# ---------------------------------------------------------------------------------------------
# router
# ---------------------------------------------------------------------------------------------

class _RouterTopK(torch.autograd.Function):
    @staticmethod
    def forward(ctx, logits, k, normalize, replay):
        w, idx, probs = C.router_topk(_c(logits.float()), k, normalize, True, replay, C.error_flag(logits) if replay is not None else None)
        ctx.save_for_backward(probs, idx, w)
        ctx.normalize = normalize
        ctx.mark_non_differentiable(idx)
        return w, idx, probs

    @staticmethod
    def backward(ctx, gw, _gidx, gprobs):
        probs, idx, w = ctx.saved_tensors
        li = idx.long()
        gw = gw.float()
        if ctx.normalize:
            # w_j = p_j / S, S = Σ_sel p  ⇒  dL/dp_j = (g_j − Σ_i g_i w_i) / S
            S = probs.gather(1, li).sum(-1, keepdim=True).clamp_min(1e-20)
            gp_sel = (gw - (gw * w).sum(-1, keepdim=True)) / S
        else:
            gp_sel = gw
        gp = torch.zeros_like(probs).scatter_add_(1, li, gp_sel)
        if gprobs is not None:
            gp = gp + gprobs
        # softmax backward
        gl = probs * (gp - (gp * probs).sum(-1, keepdim=True))
        return gl, None, None, None


def router_topk(logits, k, normalize=True):
    if logits.shape[-1] > 256:
        return ref.router_topk(logits, k, normalize)
    return _apply(_RouterTopK, logits, int(k), bool(normalize), None)


# Most experts of the one-launch form, one per warp of a token's CTA.  µs per call as norm, logits and top-k / in one launch, weights from memory: hidden 2048,
# 16 experts, 1, 8, 16, 32, 64 rows 5.9 / 4.1, 9.0 / 4.3, 6.8 / 4.3, 7.4 / 4.3, 11.0 / 4.3; hidden 1024 4.7 / 3.6 to 8.9 / 3.8, hidden 4096 8.5 / 5.2 to
# 16.7 / 5.4.  With several experts per warp their rows come one after another: 64 experts 6.0 to 11.3 / 10.2, 128 experts 6.3 to 12.3 / 18.
_ROUTER_EXPERTS = 16


def few_token_router(x, router) -> bool:
    """True when `add_rmsnorm_router` applies: CUDA bf16, no autograd, the rows of a decode step, and sums over K that may take another order
    than a product's of many rows (MILES_SPLIT_K, MILES_SMALL_M)."""
    from . import cuda as _cuda

    H = x.shape[-1]
    T = x.numel() // H
    return (x.dtype == BF16 and router.dtype == BF16 and router.is_contiguous() and 0 < T <= _cuda.SMALL_M and _cuda.SPLIT_K and H <= 4096 and H % 8 == 0
            and router.shape[0] <= _ROUTER_EXPERTS and not torch.is_grad_enabled() and not transformed()
            and x.data_ptr() % 16 == 0 and router.data_ptr() % 16 == 0)


def add_rmsnorm_router(x, residual, norm_w, eps, router, k, normalize=True):
    """(rmsnorm(x + residual), x + residual, weights, choices): what add_rmsnorm, linear_fp32 and router_topk give, with logits of unrounded operands."""
    H = x.shape[-1]
    res, xn, w, idx = C.norm_router(_c(x).view(-1, H), _c(residual).view(-1, H) if residual is not None else None, norm_w, float(eps), router, int(k),
                                    bool(normalize), bool(router.is_leaf and router.requires_grad and norm_w.is_leaf and norm_w.requires_grad))
    return xn.view(x.shape), (res.view(x.shape) if residual is not None else x), w, idx


def router_replay(logits, idx, normalize=True):
    """A choice outside the experts, in a row that has any, raises the device error flag (72) and counts nothing."""
    if logits.shape[-1] > 256 or idx.shape[1] > 32:
        return ref.router_replay(logits, idx, normalize)
    idx = idx.to(torch.int32)
    return _apply(_RouterTopK, logits, idx.shape[1], bool(normalize), idx if idx.stride(1) == 1 else idx.contiguous())


# ---------------------------------------------------------------------------------------------
# MoE FFN (single rank or the local part of an expert-parallel layer)
# ---------------------------------------------------------------------------------------------

def moe_max_rows(n_pairs: int, num_experts: int) -> int:
    """Worst-case padded row count: every expert's segment rounded up to 128."""
    return (n_pairs + num_experts * 127 + 127) // 128 * 128


# Inference with few tokens per expert (decode): segments are padded to 16/32/64 rows instead of 128 and the grouped
# GEMMs run with the expert weights on the 128-row MMA side (gemm_small.cu).  MILES_SMALL_MOE=0 turns the path off.
SMALL_MOE_AVG = float(os.environ.get("MILES_SMALL_MOE_AVG", "32")) if os.environ.get("MILES_SMALL_MOE", "1") != "0" else 0.0


MOE_GEMV_T = min(8, int(os.environ.get("MILES_MOE_GEMV_T", "8")))


def small_moe_bt(n_pairs: int, num_experts: int, w13, w2) -> int:
    """Row granularity for an inference MoE call: 128 (general path) or a decode-sized tile."""
    if SMALL_MOE_AVG <= 0 or torch.is_grad_enabled() or w13.shape[1] % 8 or w2.shape[1] % 8:
        return 128
    avg = n_pairs / max(num_experts, 1)
    if avg > SMALL_MOE_AVG:
        return 128
    return 16 if avg <= 16 else 32          # measured: the finest tile wins (weight re-reads hit L2, padding rows do not)


def moe_max_rows_pad(n_pairs: int, num_experts: int, pad: int) -> int:
    return (n_pairs + num_experts * (pad - 1) + pad - 1) // pad * pad


def few_token_experts(x, w13, T: int, k: int, ungated: bool = False) -> bool:
    """A handful of tokens: two matrix-vector kernels, no sort / gather / combine (gemv.cu).  Both keep their activations in shared
    memory next to a weight ring of at least 66 KB.  `ungated`: w13 has no gate rows."""
    F = w13.shape[1] if ungated else w13.shape[1] // 2
    return (x.dtype == BF16 and 0 < T <= MOE_GEMV_T and T * k <= 64 and not torch.is_grad_enabled() and x.shape[1] % 32 == 0
            and F % 32 == 0 and (ungated or w13.shape[1] % 64 == 0)
            and 65536 + max(8 * (2 * x.shape[1] + 64), T * k * (2 * F + 64)) <= 200 * 1024 and 67584 + (T * k + 1) * (2 * F + 64) <= 210 * 1024)


def all_token_experts(x, w13, w2, T: int, k: int) -> bool:
    """A decode step's experts without a sort (moe_rows.cu): every expert with some token multiplies all of them.  Up to 32 tokens always, up to 64 where
    an expert has more than 8: beyond that the tokens that did not choose it are too much of what each CTA reads.  µs of a layer of hidden 2048 and 768
    features, 8 choices, sorted / all: 16 experts, 9, 32, 64 tokens 42.2 / 32.6, 43.1 / 36.6, 46.9 / 42.0; 64 experts 88 / 75, 113 / 105, 114 / 118; 128
    experts 104 / 91, 178 / 174, 204 / 216.  Not where sums over the features have to be a single product's (MILES_SPLIT_K)."""
    from . import cuda as _cuda

    E = w13.shape[0]
    return (x.dtype == BF16 and 0 < T <= min(64, _cuda.SMALL_M) and (T <= 32 or T * k > 8 * E) and _cuda.SPLIT_K and SMALL_MOE_AVG > 0 and E <= 256
            and x.shape[1] % 8 == 0 and w2.shape[2] % 64 == 0 and not torch.is_grad_enabled() and not transformed())


def _glu_in_place() -> bool:
    """The activation may be formed in the bf16 product's epilogue: no block-scaled projection stands in its place, and nothing that
    the autograd functions would refuse (forward-mode tangents, function transforms) is under way."""
    from . import cuda as _cuda

    return not _cuda.MXFP8_LINEAR and not _cuda._MXFP8_WEIGHTS and not transformed()


def linear_swiglu(x, w):
    """swiglu(x · wᵀ) with w [gate; up]; without autograd in one kernel where sizes allow."""
    from . import cuda as _cuda

    rows = x.numel() // x.shape[-1]
    if (0 < rows <= _cuda.SMALL_M and not torch.is_grad_enabled() and x.dtype == BF16 and w.dtype == BF16 and w.is_contiguous() and _glu_in_place()
            and _cuda._rows_glu(rows, w, x.shape[-1])):
        act = torch.empty(*x.shape[:-1], w.shape[0] // 2, dtype=BF16, device=x.device)
        C.gemm_rows(_c(x).view(rows, -1), w, act, rows, w.shape[0], x.shape[-1], act.shape[-1], None, _cuda._rows_glu(rows, w, x.shape[-1]),
                    bool(w.is_leaf and w.requires_grad), None, True)
        return act
    if (torch.is_grad_enabled() or x.numel() < 512 * x.shape[-1] or x.dtype != BF16 or w.dtype != BF16 or not w.is_contiguous()
            or x.shape[-1] % 8 or not _glu_in_place()):                 # below 512 rows the tiles of 256 are half empty
        return _cuda.swiglu(_cuda.linear(x, w))
    act = torch.empty(*x.shape[:-1], w.shape[0] // 2, dtype=BF16, device=x.device)
    if act.numel() and C.gemm_glu(_c(x).view(-1, x.shape[-1]), w, act.view(-1, act.shape[-1]), None):
        return act
    return _cuda.swiglu(_cuda.linear(x, w))


def sort_by_expert(x, idx, E: int, bt: int, expert_offset: int = 0):
    """Rows of `x` per (token, choice), sorted by expert, every expert's segment padded to `bt` rows: (rows, segment offsets, expert of
    each row tile, row of each (token, choice))."""
    T, k = idx.shape
    max_rows = moe_max_rows(T * k, E) if bt == 128 else moe_max_rows_pad(T * k, E, bt)
    seg, tile, row_src, dst_row = C.moe_align(_c(idx.to(torch.int32)).view(-1), E, expert_offset, max_rows, None, bt, False)
    x_perm = torch.empty(max_rows, x.shape[1], dtype=x.dtype, device=x.device)
    publish_limit(LIMIT_MOE_PAIRS, T * k)
    C.moe_gather(_c(x), x_perm, row_src, seg, k)
    return x_perm, seg, tile, dst_row


def experts_forward(x_perm, w13, w2, seg, tile, bt: int = 128, glu=None, keep: bool = True):
    """Grouped expert FFN on expert-sorted rows whose segments are padded to `bt`. Returns (h1 pre-activation, y_perm).  `glu`: (limit,
    alpha, shift) of a clamped activation instead of SwiGLU, or "relu2" for experts without a gate (inference).  `keep`: h1 is wanted (a
    backward follows); else it may be None."""
    max_rows, H = x_perm.shape
    E, F2, _ = w13.shape
    F = w2.shape[2]
    if not keep and glu is None and bt == 128 and _glu_in_place():
        act = torch.empty(max_rows, F, dtype=x_perm.dtype, device=x_perm.device)
        if C.gemm_glu(x_perm, w13, act, tile):
            y_perm = torch.empty(max_rows, H, dtype=x_perm.dtype, device=x_perm.device)
            C.gemm_grouped(act, w2, y_perm, max_rows, H, F, E, tile, False, 0)
            return None, y_perm
    h1 = torch.empty(max_rows, F2, dtype=x_perm.dtype, device=x_perm.device)
    act = h1 if glu == "relu2" else torch.empty(max_rows, F, dtype=x_perm.dtype, device=x_perm.device)      # squared in place
    y_perm = torch.empty(max_rows, H, dtype=x_perm.dtype, device=x_perm.device)

    def activate():
        if glu is None:
            C.swiglu_fwd(h1, act, seg[-1:])
        elif glu == "relu2":
            C.relu_square(h1, seg[-1:])
        else:
            C.clamped_glu(h1, act, glu[0], glu[1], seg[-1:], glu[2])

    if bt != 128:
        C.gemm_small_grouped(x_perm, w13, h1, max_rows, F2, H, E, tile, seg[-1:], bt)
        activate()
        C.gemm_small_grouped(act, w2, y_perm, max_rows, H, F, E, tile, seg[-1:], bt)
        return h1, y_perm
    from . import cuda as _cuda

    if glu is None and _cuda.MXFP8_LINEAR and H % 128 == 0 and F2 % 256 == 0 and max_rows >= 8 * _cuda.MXFP8_MIN_ROWS:
        # --fp8-recipe mxfp8: the expert GEMMs of the forward run block-scaled (activations quantised per call, expert weights
        # once per call); the backward uses the bf16 grouped GEMMs on the unquantised operands (straight-through), like the
        # dense projections of this recipe
        from . import extra

        xq, xs = mxfp8_quant(x_perm)
        wq, ws = mxfp8_quant(w13.reshape(E * F2, H))
        extra.gemm_mxfp8_grouped(xq, xs, wq.view(E, F2, H), ws.view(E, F2, H // 32), tile, out=h1)
        C.swiglu_fwd(h1, act, seg[-1:])
        aq, as_ = mxfp8_quant(act)
        w2q, w2s = mxfp8_quant(w2.reshape(E * H, F))
        extra.gemm_mxfp8_grouped(aq, as_, w2q.view(E, H, F), w2s.view(E, H, F // 32), tile, out=y_perm)
        return h1, y_perm
    C.gemm_grouped(x_perm, w13, h1, max_rows, F2, H, E, tile, False, 0)
    activate()
    C.gemm_grouped(act, w2, y_perm, max_rows, H, F, E, tile, False, 0)
    return h1, y_perm


def _moe_ffn_small(x, w13, w2, topk_w, topk_idx, expert_offset, bt):
    T, H = x.shape
    k = topk_idx.shape[1]
    x_perm, seg, tile, dst_row = sort_by_expert(x, topk_idx, w13.shape[0], bt, expert_offset)
    _, y_perm = experts_forward(x_perm, _c(w13), _c(w2), seg, tile, bt)
    out = torch.empty(T, H, dtype=x.dtype, device=x.device)
    C.moe_combine(y_perm, _c(topk_w.float()), dst_row, out, k)
    return out


def experts_backward(dy_perm, x_perm, h1, w13, w2, seg, tile):
    """Backward of `experts_forward`: returns (dx_perm, dw13, dw2)."""
    max_rows, H = x_perm.shape
    E, F2, _ = w13.shape
    F = F2 // 2
    dt, dev = x_perm.dtype, x_perm.device
    act = torch.empty(max_rows, F, dtype=dt, device=dev)
    C.swiglu_fwd(h1, act, seg[-1:])
    dact = torch.empty(max_rows, F, dtype=dt, device=dev)
    C.gemm_grouped(dy_perm, w2, dact, max_rows, F, H, E, tile, True, 0)
    dw2 = torch.empty_like(w2)
    C.gemm_grouped_wgrad(dy_perm, act, dw2, max_rows, H, F, E, seg, False, 0)
    dh1 = torch.empty(max_rows, F2, dtype=dt, device=dev)
    C.swiglu_bwd(h1, dact, dh1, seg[-1:])
    dw13 = torch.empty_like(w13)
    C.gemm_grouped_wgrad(dh1, x_perm, dw13, max_rows, F2, H, E, seg, False, 0)
    dx_perm = torch.empty(max_rows, H, dtype=dt, device=dev)
    C.gemm_grouped(dh1, w13, dx_perm, max_rows, H, F2, E, tile, True, 0)
    return dx_perm, dw13, dw2


class _MoEFFN(torch.autograd.Function):
    """y[t] = Σ_j w[t,j] · W2[e]·swiglu(W13[e]·x[t]) with e = idx[t,j] − expert_offset ∈ [0, E_local) (others skipped)."""

    @staticmethod
    def forward(ctx, x, w13, w2, topk_w, topk_idx, expert_offset, keep, values):
        T, H = x.shape
        E, F2, _ = w13.shape
        F = F2 // 2
        k = topk_idx.shape[1]
        x = _c(x)
        idx32 = _c(topk_idx.to(torch.int32)).view(-1)
        wf = _c(topk_w.float())
        max_rows = moe_max_rows(T * k, E)
        seg, tile, row_src, dst_row = C.moe_align(idx32, E, expert_offset, max_rows, None, 128, keep)     # weight gradients are sums over a segment's rows
        x_perm = torch.empty(max_rows, H, dtype=x.dtype, device=x.device)
        publish_limit(LIMIT_MOE_PAIRS, x.shape[0] * k)
        C.moe_gather(x, x_perm, row_src, seg, k)
        from . import cuda as _cuda

        out = torch.empty(T, H, dtype=x.dtype, device=x.device)
        if keep and not values and not _cuda.MXFP8_LINEAR:                         # only a backward follows: what it needs
            h1, y_perm = torch.empty(max_rows, F2, dtype=x.dtype, device=x.device), None
            C.gemm_grouped(x_perm, w13, h1, max_rows, F2, H, E, tile, False, 0)
        else:
            h1, y_perm = experts_forward(x_perm, w13, w2, seg, tile, keep=keep)    # bf16 grouped GEMMs, or block-scaled under the MXFP8 recipe
            C.moe_combine(y_perm, wf, dst_row, out, k)

        # the gate weights' gradient ⟨dout, W2 · act⟩ is taken as ⟨dout · W2, act⟩: y is not needed, except where it is not W2 · act (quantised)
        ctx.save_for_backward(x_perm, w13, w2, wf, seg, tile, row_src, dst_row, h1, y_perm if _cuda.MXFP8_LINEAR else None)
        ctx.k = k
        return out

    @staticmethod
    def backward(ctx, dout):
        x_perm, w13, w2, wf, seg, tile, row_src, dst_row, h1, y_perm = ctx.saved_tensors
        k = ctx.k
        T, H = dout.shape
        E, F2, _ = w13.shape
        F = F2 // 2
        max_rows = h1.shape[0]
        dout = _c(dout)
        new = lambda *shape: torch.empty(*shape, dtype=h1.dtype, device=h1.device)
        dw_flat = torch.zeros(T * k, dtype=torch.float32, device=h1.device)
        dy_perm, act, dh1 = new(max_rows, H), new(max_rows, F), new(max_rows, F2)
        if y_perm is None:
            # every row of dout as it is: the weight goes to the activation
            publish_limit(LIMIT_MOE_PAIRS, T * k)
            C.moe_gather(dout, dy_perm, row_src, seg, k)
            C.gemm_grouped(dy_perm, w2, act, max_rows, F, H, E, tile, True, 0)
            C.moe_glu_bwd(h1, act, dh1, wf.view(-1), row_src, seg, dw_flat)
        else:
            C.moe_combine_bwd(dout, y_perm, wf.view(-1), row_src, seg, dy_perm, dw_flat, k)
            dact = new(max_rows, F)
            C.swiglu_fwd(h1, act, seg[-1:])
            C.gemm_grouped(dy_perm, w2, dact, max_rows, F, H, E, tile, True, 0)
            C.swiglu_bwd(h1, dact, dh1, seg[-1:])
        dw2 = torch.empty_like(w2)
        C.gemm_grouped_wgrad(dy_perm, act, dw2, max_rows, H, F, E, seg, False, 0)
        dw13 = torch.empty_like(w13)
        C.gemm_grouped_wgrad(dh1, x_perm, dw13, max_rows, F2, H, E, seg, False, 0)
        C.gemm_grouped(dh1, w13, dy_perm, max_rows, H, F2, E, tile, True, 0)              # dy_perm has been read: the input rows' gradient in its place
        dx = new(T, H)
        C.moe_combine(dy_perm, None, dst_row, dx, k)
        return dx, dw13, dw2, dw_flat.view(T, k), None, None, None, None


class Combine:
    """The experts' rows of a forward pass without gradients, still to be weighted and added up per token: by the add and norm of the next layer
    (`combine_add_rmsnorm`) or by `value`."""

    def __init__(self, y_perm, w, dst_row, k, like):
        self.y_perm, self.w, self.dst_row, self.k, self.like = y_perm, w, dst_row, k, like

    def value(self):
        out = torch.empty_like(self.like)
        C.moe_combine(self.y_perm, self.w, self.dst_row, out, self.k)
        return out


def combine_add_rmsnorm(x: Combine, residual, norm_w, eps):
    """(rmsnorm(x + residual) · norm_w, x + residual)."""
    H = residual.shape[-1]
    if norm_w.data_ptr() % 16 or residual.data_ptr() % 16 or not norm_w.is_contiguous():
        from . import cuda as _cuda

        return _cuda.add_rmsnorm(x.value(), residual, norm_w, eps)
    y, total = C.moe_combine_norm(x.y_perm, x.w, x.dst_row, _c(residual).view(-1, H), norm_w, x.k, float(eps))
    return y.view(residual.shape), total.view(residual.shape)


def moe_ffn_rows(x, w13, w2, topk_w, topk_idx, expert_offset: int = 0):
    """`moe_ffn` without its last kernel (`Combine`) where the rows that follow are those of `combine_add_rmsnorm`, else its value."""
    T, k = topk_idx.shape
    E = w13.shape[0]
    if (x.dtype != BF16 or torch.is_grad_enabled() or transformed() or T < 64 or x.dim() != 2 or x.shape[1] % 8 or x.shape[1] > 4096
            or few_token_experts(x, w13, T, k) or all_token_experts(x, w13, w2, T, k) or small_moe_bt(T * k, E, w13, w2) != 128):
        return moe_ffn(x, w13, w2, topk_w, topk_idx, expert_offset)
    x = _c(x)
    max_rows = moe_max_rows(T * k, E)
    seg, tile, row_src, dst_row = C.moe_align(_c(topk_idx.to(torch.int32)).view(-1), E, expert_offset, max_rows, None, 128, False)
    x_perm = torch.empty(max_rows, x.shape[1], dtype=x.dtype, device=x.device)
    publish_limit(LIMIT_MOE_PAIRS, T * k)
    C.moe_gather(x, x_perm, row_src, seg, k)
    _, y_perm = experts_forward(x_perm, w13, w2, seg, tile, keep=False)
    return Combine(y_perm, _c(topk_w.float()), dst_row, k, x)


def moe_ffn(x, w13, w2, topk_w, topk_idx, expert_offset: int = 0, values: bool = True):
    """`values` False: the result is not read, it only stands in the graph."""
    if x.dtype != BF16:
        return ref.moe_ffn(x, w13, w2, topk_w, topk_idx)
    T, k = topk_idx.shape
    if few_token_experts(x, w13, T, k):
        act = torch.empty(T * k, w13.shape[1] // 2, dtype=x.dtype, device=x.device)
        out = torch.empty_like(x)
        C.moe_gemv(_c(x), _c(w13), _c(w2), _c(topk_idx.to(torch.int32)), _c(topk_w.float()), act, out, int(expert_offset))
        return out
    if all_token_experts(x, w13, w2, T, k):
        out = torch.empty_like(x)
        C.moe_rows(_c(x), _c(w13), _c(w2), _c(topk_idx.to(torch.int32)), _c(topk_w.float()), out, int(expert_offset))
        return out
    bt = small_moe_bt(topk_idx.numel(), w13.shape[0], w13, w2)
    if bt != 128 and x.shape[0]:
        return _moe_ffn_small(x, w13, w2, topk_w, topk_idx, int(expert_offset), bt)
    return _apply(_MoEFFN, x, w13, w2, topk_w, topk_idx, int(expert_offset), torch.is_grad_enabled(), values)


# ---------------------------------------------------------------------------------------------
# log-prob / entropy head: vocabulary streamed in chunks, logits never materialised in full
# ---------------------------------------------------------------------------------------------
_VOCAB_CHUNK = 16384
_ROW_CHUNK = 16384


def _vocab_chunks(V):
    return [(v0, min(V, v0 + _VOCAB_CHUNK)) for v0 in range(0, V, _VOCAB_CHUNK)]


def _head_in_place(rows: int, hidden, w) -> bool:
    """Statistics and gradients in the product's epilogue (head.cu): more rows than the decode-sized kernels take, TMA-readable operands."""
    return rows > 64 and hidden.shape[1] % 8 == 0 and w.is_contiguous() and w.dtype == BF16


class _LogProbEntropy(torch.autograd.Function):
    @staticmethod
    def forward(ctx, hidden, w, targets, temperature, with_entropy, vocab_offset):
        R, H = hidden.shape
        V = w.shape[0]
        hidden = _c(hidden)
        tg = _c(targets.to(torch.int64)) - vocab_offset
        inv_t = 1.0 / temperature
        logp = torch.empty(R, dtype=torch.float32, device=hidden.device)
        ent = torch.empty(R, dtype=torch.float32, device=hidden.device)
        lse = torch.empty(R, dtype=torch.float32, device=hidden.device)
        for r0 in range(0, R, _ROW_CHUNK):
            r1 = min(R, r0 + _ROW_CHUNK)
            if _head_in_place(r1 - r0, hidden, w):
                C.head_logprob(hidden[r0:r1], w, tg[r0:r1], inv_t, logp[r0:r1], ent[r0:r1], lse[r0:r1], C.error_flag(hidden))
                continue
            stats = torch.empty(r1 - r0, 4, dtype=torch.float32, device=hidden.device)
            for ci, (v0, v1) in enumerate(_vocab_chunks(V)):
                logits = gemm_nt(hidden[r0:r1], w[v0:v1], out_dtype=torch.float32)
                C.logit_stats(logits, tg[r0:r1], stats, v0, inv_t, ci == 0)
            C.logit_stats_finish(stats, logp[r0:r1], ent[r0:r1], lse[r0:r1])
        ctx.save_for_backward(hidden, w, tg, lse, ent)
        ctx.inv_t, ctx.with_entropy = inv_t, with_entropy
        ctx.mark_non_differentiable(lse)
        return logp, ent, lse

    @staticmethod
    def backward(ctx, g_lp, g_ent, _g_lse):
        hidden, w, tg, lse, ent = ctx.saved_tensors
        R, H = hidden.shape
        V = w.shape[0]
        g_lp = _c(g_lp.float()) if g_lp is not None else None
        g_ent = _c(g_ent.float()) if (g_ent is not None and ctx.with_entropy) else None
        dh = torch.zeros(R, H, dtype=torch.float32, device=hidden.device)
        dw = torch.empty_like(w)
        for (v0, v1) in _vocab_chunks(V):
            dwc = None
            for r0 in range(0, R, _ROW_CHUNK):
                r1 = min(R, r0 + _ROW_CHUNK)
                dl = torch.empty(r1 - r0, v1 - v0, dtype=BF16, device=hidden.device)
                in_place = _head_in_place(r1 - r0, hidden, w) and (v1 - v0) % 8 == 0
                if in_place:
                    C.head_grad(hidden[r0:r1], w[v0:v1], tg[r0:r1], lse[r0:r1], ent[r0:r1] if g_ent is not None else None,
                                g_lp[r0:r1] if g_lp is not None else None, g_ent[r0:r1] if g_ent is not None else None, dl, v0, ctx.inv_t,
                                C.error_flag(hidden))
                else:
                    logits = gemm_nt(hidden[r0:r1], w[v0:v1], out_dtype=torch.float32)
                    C.logit_grad(logits, tg[r0:r1], lse[r0:r1], ent[r0:r1] if g_ent is not None else None,
                                 g_lp[r0:r1] if g_lp is not None else None, g_ent[r0:r1] if g_ent is not None else None, dl, v0,
                                 ctx.inv_t)
                # dH[r0:r1] += dl · W_c   (fp32 accumulate in place)
                Mr, Kc, Nh = r1 - r0, v1 - v0, H
                C.gemm(dl, w[v0:v1], dh[r0:r1], Mr, Nh, Kc, Kc, Nh, H, False, True, True, None, 0)
                # dW_c (+)= dlᵀ · H
                if dwc is None:
                    dwc = torch.empty(v1 - v0, H, dtype=torch.float32, device=hidden.device) if R > _ROW_CHUNK else dw[v0:v1]
                    gemm_tn(dl, hidden[r0:r1], out=dwc)
                else:
                    gemm_tn(dl, hidden[r0:r1], out=dwc, accumulate=True)
            if dwc.dtype != dw.dtype:
                dw[v0:v1].copy_(dwc)
        return dh.to(hidden.dtype), dw, None, None, None, None


def logprob_entropy(hidden, w, targets, temperature=1.0, with_entropy=False, vocab_offset: int = 0, return_lse=False):
    if hidden.dtype != BF16:
        lp, ent = ref.logprob_entropy(hidden, w, targets, temperature, with_entropy=with_entropy)
        return lp, ent
    logp, ent, lse = _apply(_LogProbEntropy, hidden, w, targets, float(temperature), bool(with_entropy), int(vocab_offset))
    if return_lse:
        return logp, ent, lse
    return logp, (ent if with_entropy else None)


# ---------------------------------------------------------------------------------------------
# sampling / quantisation
# ---------------------------------------------------------------------------------------------

def sample_logprob(logits, temperature, greedy, seeds=None, step: int = 0):
    logits = _c(logits.float())
    return tuple(C.sample_logprob(logits, _c(temperature.float()), _c(greedy.to(torch.uint8)),
                                  _c(seeds.to(torch.int64)) if seeds is not None else None, int(step)))


def mxfp8_quant(x):
    assert x.dtype == BF16 and x.shape[-1] % 32 == 0
    q, s = C.mxfp8_quant(_c(x))
    return q, s


def fp8_blockwise_quant(w):
    assert w.dtype == BF16 and w.dim() == 2
    q, s = C.fp8_block_quant(_c(w))
    return q, s


def int4_fake_quant(x, block_m=1, block_n=32, symmetric=True):
    assert x.dtype == BF16 and x.dim() == 2
    y, s = C.int4_fake_quant(_c(x), block_m, block_n, symmetric)
    return y, s


def absmax(x):
    return C.absmax(_c(x))


def nvfp4_qdq(x, global_amax=None, four_over_six=False):
    assert x.dtype == BF16 and x.numel() % 16 == 0
    x = _c(x)
    if global_amax is None:
        global_amax = C.absmax(x)
    return C.nvfp4_qdq(x, global_amax.reshape(1).float(), bool(four_over_six))
