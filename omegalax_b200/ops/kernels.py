"""Tensor-level wrappers around the sm_100a launchers (no autograd here).

All functions take CUDA bf16 tensors unless noted, launch on the current stream and
return immediately.  ``launch_count`` counts every kernel of this library that was
launched since the last ``reset_launch_count()``.
"""
from __future__ import annotations

import os

import torch

from . import lib

bf16 = torch.bfloat16
_launches = 0


def reset_launch_count() -> None:
    global _launches
    _launches = 0


def launch_count() -> int:
    return _launches


def add_launches(n: int) -> None:
    """Count the launches of a replayed CUDA graph."""
    global _launches
    _launches += n


def _call(name, *args):
    global _launches
    _launches += 1
    lib.call(name, *args)


def _row_major_2d(t: torch.Tensor) -> torch.Tensor:
    if t.dim() != 2:
        t = t.reshape(-1, t.shape[-1])
    if t.stride(1) != 1 or (t.stride(0) % 8) or (t.data_ptr() % 16):
        t = t.contiguous()
    return t


_PAIR_MODE = os.environ.get("OMEGALAX_B200_GEMM_PAIR", "all")   # "0" never, "1" always, "all" / "auto" by shape


_PAIR_AG = os.environ.get("OMEGALAX_B200_GEMM_PAIR_AG", "1") == "1"   # gather mode on the pair kernel


def _use_pair(M: int, N: int, K: int, wgrad: bool = False) -> bool:
    """CTA-pair (256 x 256 tile) kernel for GEMMs with enough tiles to fill every SM pair."""
    if _PAIR_MODE == "0":
        return False
    if _PAIR_MODE == "1":
        return True
    big = (-(-M // 256)) * (-(-N // 256)) >= 74 and N >= 512 and K >= 256
    if _PAIR_MODE == "all":
        # Inside a training step (power-capped clocks) the pair kernel is the faster one on every
        # large GEMM: it needs about 10 % fewer SM cycles per step.
        return big
    # Timed alone in short bursts it wins on the attention-sized projections and loses on the
    # widest (MLP) ones and on weight gradients: "auto" keeps it to the former.
    return big and not wgrad and N <= 8192 and K <= 8192


def _use_few(M: int, N: int, K: int) -> bool:
    """The kernel for few rows, where streaming the weights or filling the SMs is the bound.  Up to 128 rows it
    reads every weight once (N 4096, K 12288: 22 us for one row, 81 on 128 x 128 tiles; N 151936, K 4096: 191,
    516); above, while its 128 x 128 panels fit the SMs in one wave of two (M 500, N 6144, K 4096: 33 us against
    51; M 1000, N 6144: 64 against 55, beyond the wave).  Short reductions leave nothing to share out
    (M 128, N 8192, K 512: 9.9 against 9.5; K 768, M 2048, N 1024, whose panels are just one wave of the others: 11.7 against
    10.4, while 192 panels, two waves of the others, take 13.3 against 15.5)."""
    if M <= 64:
        return K > 0
    panels = -(-M // 128) * -(-N // 128)
    return K >= 768 and (M <= 128 or panels <= 296) and (K >= 1024 or not 74 < panels <= 148)


def _read_ahead(w) -> int:
    """4 where the kernel for few rows may read these weights while the kernel before it still runs (recorded steps): those that no
    kernel of a step writes, parameters.  A tensor that the call made (padded, cast, computed by a parametrization) may come from that
    very kernel."""
    return 4 if isinstance(w, torch.nn.Parameter) else 0


def gemm(a, b, *, a_mn: bool = False, b_mn: bool = False, out=None, out_dtype=bf16,
         accumulate: bool = False, residual=None, bn: int = 0, pair: bool | None = None, bias=None,
         ce=None, few: bool | None = None, splits: int = 0):
    """C = op(A) op(B)^T on the tcgen05 kernel.

    a: [M,K] (a_mn False) or [K,M] (a_mn True); b: [N,K] (b_mn False) or [K,N] (b_mn True).
    out: optional preallocated [M,N] (bf16 or fp32); ``accumulate`` adds into an fp32 out.
    ``bias`` (bf16 [N]) and ``residual`` (bf16 [M,N]) are added in the epilogue.  ``ce`` =
    (targets int32 [M], stats fp32 [M, ceil(N/256), 2], target_logit fp32 [M]) asks the 512 x 256
    tile kernel for the cross-entropy statistics of the fp32 accumulator (bf16 output only).
    ``few`` (K-major operands) overrides the choice of the kernel for few rows, ``splits`` its CTAs per
    column panel.
    """
    a = _row_major_2d(a)
    b = _row_major_2d(b)
    M, K = (a.shape[1], a.shape[0]) if a_mn else (a.shape[0], a.shape[1])
    N, Kb = (b.shape[1], b.shape[0]) if b_mn else (b.shape[0], b.shape[1])
    if K != Kb:
        raise ValueError(f"reduction mismatch {K} vs {Kb}")
    if out is None:
        out = torch.empty(M, N, dtype=out_dtype, device=a.device)
    if out.stride(1) != 1:
        raise ValueError("out must be row-major")
    if out.dtype == bf16:
        mode = 0
        if accumulate:
            raise ValueError("accumulate needs an fp32 output")
    elif out.dtype == torch.float32:
        mode = 2 if accumulate else 1
    else:
        raise ValueError("out dtype must be bf16 or fp32")
    res_ptr, ldr = None, 0
    if residual is not None:
        residual = residual.reshape(M, N)
        if residual.stride(1) != 1:
            residual = residual.contiguous()
        res_ptr, ldr = residual.data_ptr(), residual.stride(0)
    st = lib.status_tensor(a.device)
    if bias is not None and (bias.dtype != bf16 or bias.numel() != N or not bias.is_contiguous()):
        raise ValueError("bias must be a contiguous bf16 vector of N elements")
    if few is None:
        few = bn == 0 and pair is None and ce is None and not (a_mn or b_mn) and _use_few(M, N, K)
    if few:
        _call("ob_gemm_few", a.data_ptr(), b.data_ptr(), out.data_ptr(), res_ptr, M, N, K, a.stride(0), b.stride(0), out.stride(0),
              ldr, mode | _read_ahead(b), lib.ptr(bias), splits, st.data_ptr(), lib.stream_ptr())
        return out
    if pair is None:
        pair = bn == 0 and _use_pair(M, N, K, wgrad=a_mn and b_mn)
    if ce is not None:
        tg, stats, tl = ce
        if mode != 0 or residual is not None or tuple(stats.shape) != (M, -(-N // 256), 2) or tl.numel() != M:
            raise ValueError("cross-entropy statistics need a bf16 output, no residual and [M, ceil(N/256), 2] stats")
        pair = True
    if pair:
        ce_ptrs = (None, None, None) if ce is None else (ce[0].data_ptr(), ce[1].data_ptr(), ce[2].data_ptr())
        _call("ob_gemm_bf16_pair", a.data_ptr(), b.data_ptr(), out.data_ptr(), res_ptr, M, N, K,
              a.stride(0), b.stride(0), out.stride(0), ldr, int(a_mn), int(b_mn), mode, lib.ptr(bias), *ce_ptrs,
              st.data_ptr(), lib.stream_ptr())
        return out
    _call("ob_gemm_bf16", a.data_ptr(), b.data_ptr(), out.data_ptr(), res_ptr, M, N, K,
          a.stride(0), b.stride(0), out.stride(0), ldr, int(a_mn), int(b_mn), mode, bn, lib.ptr(bias),
          st.data_ptr(), lib.stream_ptr())
    return out


def gemm_step(x, w, *, residual=None, norm=None, squares: bool = False, act: int = 0):
    """C = x w^T (+ residual) of a decode step's few rows (x [M,K], w [N,K], bf16, contiguous), with what stands beside
    the product.  ``norm`` = (weight [K], eps, sums): x passes an RMS norm first, whose sums of squares by panels of 128
    columns are ``sums`` (M <= 32, K % 128 == 0).  ``squares``: returns (C, such sums of C) (N % 128 == 0).  ``act`` 1: w is
    [gate | up] (N % 128 == 0) and C = silu(gate) * up; 2: C = max(., 0)^2."""
    M, K = x.shape
    N = w.shape[0]
    out = torch.empty(M, N // 2 if act == 1 else N, dtype=bf16, device=x.device)
    sums = torch.empty(M, N // 128, dtype=torch.float32, device=x.device) if squares else None
    weight, eps, given = (None, 0.0, None) if norm is None else norm
    _call("ob_gemm_step", x.data_ptr(), w.data_ptr(), out.data_ptr(), lib.ptr(residual), M, N, K, K, K, out.shape[1], N, lib.ptr(weight),
          lib.ptr(given), float(eps), lib.ptr(sums), int(act) | _read_ahead(w), lib.status_tensor(x.device).data_ptr(), lib.stream_ptr())
    return (out, sums) if squares else out


def gemm_relu_sq(x, w, few: bool | None = None):
    """max(x w^T, 0)^2 without the product in memory, or None where the kernels that ``gemm`` takes for these sizes do not have
    it: few rows do, and the 512 x 256 tiles."""
    x, w = _row_major_2d(x), _row_major_2d(w)
    (M, K), N = x.shape, w.shape[0]
    if K % 8 == 0 and (_use_few(M, N, K) if few is None else few):
        return gemm_step(x, w, act=2) if x.is_contiguous() and w.is_contiguous() else None
    if not _use_pair(M, N, K) or not lib.ask("ob_gemm_relu_sq_fits", M, N, K):
        return None
    out = torch.empty(M, N, dtype=bf16, device=x.device)
    _call("ob_gemm_relu_sq", x.data_ptr(), w.data_ptr(), out.data_ptr(), M, N, K, x.stride(0), w.stride(0), N,
          lib.status_tensor(x.device).data_ptr(), lib.stream_ptr())
    return out


def gemm_peer_reduce(a, b, peer_ptrs, rows_per_peer: int, ldc: int, *, a_mn=False, b_mn=False, bf16_out=False,
                     pair: bool | None = None, slot: int | None = None):
    """GEMM whose result rows are added into buffers owned by other GPUs (``peer_ptrs[r]`` holds
    rows [r*rows_per_peer, (r+1)*rows_per_peer)): fp32 buffers by default (gradient shards), bf16
    buffers with ``bf16_out`` (activations: half the NVLink bytes, bf16 accumulation).  With
    ``slot`` nothing is reduced: the bf16 rows are stored into slab ``slot`` of the owner's staging
    buffer ([senders, rows_per_peer, ldc]) and the owner sums the slabs with ``slab_sum``.
    A ``peer_ptrs`` list with a ``rank`` attribute (``SymmetricBuffer.peer_ptr_list``) makes the
    tiles start with this GPU's own rows and walk the owners from there, so that the GPUs of the
    group write to distinct owners at any moment."""
    import ctypes

    a = _row_major_2d(a)
    b = _row_major_2d(b)
    M, K = (a.shape[1], a.shape[0]) if a_mn else (a.shape[0], a.shape[1])
    N = b.shape[1] if b_mn else b.shape[0]
    arr = (ctypes.c_void_p * len(peer_ptrs))(*peer_ptrs)
    st = lib.status_tensor(a.device)
    if pair is None:
        pair = _use_pair(M, N, K, wgrad=a_mn and b_mn)
    name = "ob_gemm_bf16_pair_peer_reduce" if pair else "ob_gemm_bf16_peer_reduce"
    _call(name, a.data_ptr(), b.data_ptr(), ctypes.cast(arr, ctypes.c_void_p),
          len(peer_ptrs), rows_per_peer, M, N, K, a.stride(0), b.stride(0), ldc, int(a_mn),
          int(b_mn), (2 + int(slot)) if slot is not None else int(bf16_out), int(getattr(peer_ptrs, "rank", 0)),
          st.data_ptr(), lib.stream_ptr())


def slab_sum(staging, slots: int, out, residual=None):
    """out = sum of the ``slots`` equal slabs of ``staging`` (+ residual): bf16, fp32 accumulation."""
    _call("ob_slab_sum", staging.data_ptr(), int(slots), out.numel(), lib.ptr(residual), out.data_ptr(),
          lib.stream_ptr())
    return out


def ag_copy_ctas(M: int, N: int, Kd: int, total_bytes: float) -> int:
    """Copy CTAs for the gather mode.  The tiles walk the chunks in arrival order starting with this
    GPU's own chunk (read in place), so the chunks must arrive at the rate the tiles consume them:
    the whole operand within ~80 % of the GEMM's duration, at ~45 GB/s per copy thread (128 KB in
    flight)."""
    t_gemm = 2.0 * M * N * Kd / 1.1e15
    need = total_bytes / max(0.8 * t_gemm, 1e-6) / 45e9
    n = int(min(16, max(2, -(-need // 1))))
    return n + (n & 1)          # even: the CTA-pair kernel gives up whole clusters


def gemm_ag(other, full, src_ptrs, *, side: int, rank: int, rows_per_rank: int, flags, target: int,
            copy_ctas: int = 8, residual=None, out=None):
    """All-gather -> GEMM in one launch: y = A @ B^T with both operands [rows, K] row-major.
    side 1: A = ``full`` [rows_per_rank * W, K] is assembled from the ranks' row chunks at
    ``src_ptrs`` while the tiles run; side 2: B likewise.  ``other`` is the operand that is
    already complete.  ``flags`` (uint32 [W]) only grow: ``target`` is their value after this call."""
    import ctypes

    W = len(src_ptrs)
    Kd = full.shape[1]
    if side == 1:
        M, N = full.shape[0], other.shape[0]
    else:
        M, N = other.shape[0], full.shape[0]
    other = _row_major_2d(other)
    assert other.stride(0) == Kd and full.is_contiguous()
    if out is None:
        out = torch.empty(M, N, dtype=bf16, device=full.device)
    arr = (ctypes.c_void_p * W)(*src_ptrs)
    st = lib.status_tensor(full.device)
    name = "ob_gemm_bf16_ag"
    if _PAIR_AG and rows_per_rank % 256 == 0 and copy_ctas % 2 == 0 and _use_pair(M, N, Kd):
        name = "ob_gemm_bf16_pair_ag"
    _call(name, other.data_ptr(), full.data_ptr(), ctypes.cast(arr, ctypes.c_void_p), out.data_ptr(),
          lib.ptr(residual), M, N, Kd, out.stride(0), residual.stride(0) if residual is not None else 0, 0, side, W,
          rank, rows_per_rank, flags.data_ptr(), int(target) & 0xFFFFFFFF, copy_ctas, st.data_ptr(), lib.stream_ptr())
    return out


def gemm_grouped(a, b, group_offsets, *, b_mn: bool = False, out=None, out_dtype=bf16, pair: bool = False):
    """Ragged-row grouped GEMM.  a: [R,K] rows grouped by ``group_offsets`` (int32 [G+1],
    multiples of 128, R % 128 == 0); b: [G,N,K] (or [G,K,N] when b_mn).  ``pair``: run on CTA pairs
    (256 x 256 tiles); the caller guarantees that every group offset and R are multiples of 256."""
    a = _row_major_2d(a)
    G = b.shape[0]
    R, K = a.shape
    N = b.shape[2] if b_mn else b.shape[1]
    b2 = b.reshape(-1, b.shape[-1])
    lib.check_index("gemm_grouped group_offsets", group_offsets, R + 1)
    if out is None:
        out = torch.empty(R, N, dtype=out_dtype, device=a.device)
    mode = 0 if out.dtype == bf16 else 1
    st = lib.status_tensor(a.device)
    pair = pair and R % 256 == 0
    _call("ob_gemm_bf16_pair_grouped" if pair else "ob_gemm_bf16_grouped", a.data_ptr(), b2.data_ptr(), out.data_ptr(),
          group_offsets.data_ptr(), G, R, N, K, a.stride(0), out.stride(0), int(b_mn), mode,
          st.data_ptr(), lib.stream_ptr())
    return out


def gemm_grouped_wgrad(dy, x, group_offsets, out, accumulate: bool = True, pair: bool = False):
    """out[g] (+)= dy[rows of g]^T x[rows of g]; dy [R,N], x [R,K], out fp32 [G,N,K].  ``pair`` as in
    ``gemm_grouped``."""
    dy = _row_major_2d(dy)
    x = _row_major_2d(x)
    G, N, K = out.shape
    lib.check_index("gemm_grouped_wgrad group_offsets", group_offsets, dy.shape[0] + 1)
    mode = (2 if accumulate else 1) if out.dtype == torch.float32 else 0
    st = lib.status_tensor(dy.device)
    _call("ob_gemm_bf16_pair_grouped_wgrad" if pair else "ob_gemm_bf16_grouped_wgrad", dy.data_ptr(), x.data_ptr(), out.data_ptr(),
          group_offsets.data_ptr(), G, dy.shape[0], N, K, dy.stride(0), x.stride(0), mode,
          st.data_ptr(), lib.stream_ptr())
    return out


def rmsnorm_fwd(x, w, eps, one_plus=False, want_rstd=True):
    x2 = x.reshape(-1, x.shape[-1])
    if not x2.is_contiguous():
        x2 = x2.contiguous()
    y = torch.empty_like(x2)
    rstd = torch.empty(x2.shape[0], dtype=torch.float32, device=x.device) if want_rstd else None
    _call("ob_rmsnorm_fwd", x2.data_ptr(), w.data_ptr(), y.data_ptr(), lib.ptr(rstd), x2.shape[0],
          x2.shape[1], float(eps), int(one_plus), lib.stream_ptr())
    return y.view(x.shape), rstd


def rmsnorm_bwd(dy, x, w, rstd, eps, dw_out, one_plus=False):
    x2 = x.reshape(-1, x.shape[-1])
    dy2 = dy.reshape(-1, x.shape[-1])
    if not x2.is_contiguous():
        x2 = x2.contiguous()
    if not dy2.is_contiguous():
        dy2 = dy2.contiguous()
    dx = torch.empty_like(x2)
    _call("ob_rmsnorm_bwd", dy2.data_ptr(), x2.data_ptr(), w.data_ptr(), lib.ptr(rstd),
          dx.data_ptr(), lib.ptr(dw_out), x2.shape[0], x2.shape[1], float(eps), int(one_plus),
          lib.stream_ptr())
    return dx.view(x.shape)


def swiglu_fwd(gu, rows=None):
    """silu(gate) * up; ``rows`` (int32, on the device): only so many rows matter, the others stay unwritten."""
    g2 = gu.reshape(-1, gu.shape[-1])
    F = g2.shape[1] // 2
    act = torch.empty(g2.shape[0], F, dtype=gu.dtype, device=gu.device)
    _call("ob_swiglu_fwd", g2.data_ptr(), act.data_ptr(), lib.ptr(rows), g2.shape[0], F, lib.stream_ptr())
    return act.view(*gu.shape[:-1], F)


def swiglu_bwd(gu, dact, with_act: bool = False, inplace: bool = False, rows=None):
    """Gradient of silu(gate) * up (``rows`` as in ``swiglu_fwd``); ``with_act`` also returns the activation itself, recomputed in
    the same pass (for a caller that did not keep it); ``inplace`` writes the gradient over
    ``gu`` (contiguous), for a caller that is the last reader of it."""
    g2 = gu.reshape(-1, gu.shape[-1])
    F = g2.shape[1] // 2
    d2 = dact.reshape(-1, F)
    if not d2.is_contiguous():
        d2 = d2.contiguous()
    if inplace and not g2.is_contiguous():
        raise ValueError("swiglu_bwd(inplace=True) needs a contiguous [gate | up] tensor")
    dgu = g2 if inplace else torch.empty_like(g2)
    act = torch.empty(g2.shape[0], F, dtype=gu.dtype, device=gu.device) if with_act else None
    _call("ob_swiglu_bwd", g2.data_ptr(), d2.data_ptr(), dgu.data_ptr(), lib.ptr(act), lib.ptr(rows), g2.shape[0], F,
          lib.stream_ptr())
    return (dgu.view(gu.shape), act) if with_act else dgu.view(gu.shape)


def column_sum(x, scale: float = 1.0):
    """scale * x.sum(0) of a contiguous bf16 or fp32 matrix with a multiple of eight columns; fp32 sums."""
    M, N = x.shape
    out = torch.empty(N, dtype=x.dtype, device=x.device)
    _call("ob_column_sum", x.data_ptr(), out.data_ptr(), M, N, int(x.dtype == bf16), float(scale), lib.stream_ptr())
    return out


def qknorm_rope_fwd(qkv, qw, kw, cos, sin, H, G, K, rot, eps, one_plus=False, q_stride_heads=1):
    M = qkv.shape[0]
    q = torch.empty(M, H, K, dtype=qkv.dtype, device=qkv.device)
    k = torch.empty(M, G, K, dtype=qkv.dtype, device=qkv.device)
    _call("ob_qknorm_rope_fwd", qkv.data_ptr(), lib.ptr(qw), lib.ptr(kw), cos.data_ptr(),
          sin.data_ptr(), q.data_ptr(), k.data_ptr(), M, H, G, K, rot, float(eps), int(one_plus),
          q_stride_heads, lib.stream_ptr())
    return q, k


def qknorm_rope_bwd(qkv, qw, kw, cos, sin, dq, dk, dqkv, dqw, dkw, H, G, K, rot, eps,
                    one_plus=False, q_stride_heads=1, dv=None, dgate=None):
    """All of dqkv: its v and gate heads are ``dv`` and ``dgate`` (zeros without)."""
    M = qkv.shape[0]
    _call("ob_qknorm_rope_bwd", qkv.data_ptr(), lib.ptr(qw), lib.ptr(kw), cos.data_ptr(),
          sin.data_ptr(), dq.data_ptr(), dk.data_ptr(), lib.ptr(dv), lib.ptr(dgate), dqkv.data_ptr(), lib.ptr(dqw),
          lib.ptr(dkw), M, H, G, K, rot, float(eps), int(one_plus), q_stride_heads,
          lib.stream_ptr())


def attn_fwd(q, k, v, cu_seqlens, max_seqlen, scale, causal, want_lse=True):
    """q [N,H,K]; k,v [N,G,K] (row-strided views allowed).  Returns out [N,H,K], lse [H,N]."""
    N, H, K = q.shape
    G = k.shape[1]
    for t in (q, k, v):
        if t.stride(2) != 1 or t.stride(1) != K:
            raise ValueError("attention operands need contiguous heads")
    out = torch.empty(N, H, K, dtype=q.dtype, device=q.device)
    lse = torch.empty(H, N, dtype=torch.float32, device=q.device) if want_lse else None
    st = lib.status_tensor(q.device)
    _call("ob_attn_fwd", q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lib.ptr(lse),
          cu_seqlens.data_ptr(), cu_seqlens.numel() - 1, int(max_seqlen), N, H, G, K, q.stride(0),
          k.stride(0), v.stride(0), out.stride(0), float(scale), int(causal), st.data_ptr(),
          lib.stream_ptr())
    return out, lse


_attn_scratch: dict = {}


def attn_bwd_splits(tiles: int, H: int, G: int, steps: int, causal: bool = True, values: int = 0) -> int:
    """CTAs that share the query heads of a key tile: the number with the least estimated time, in steps of 64 queries (2 us at
    head_dim 128).  A CTA has the SM to itself and costs four steps beside its walk; the SMs end together where walks
    differ (causal) and in whole rounds where they do not; sharing costs two steps, and two more for every million fp32 partial
    sums (``values`` per part) that are stored and added.  It has to save a twentieth.  Measured over 24 batches of 5 head layouts:
    0.4 % above the best choice on average, and at worst 2 % slower than no sharing.  In us by CTAs 1 / 2 / 4: 32 heads on 4, one
    row of 4096 1053 576 575; on 8, one of 3001 420 368 388, one of 4096 561 579 637, two of 4096 1066 1146 1281, seven of
    512 139 196 256."""
    R = H // G

    def cost(n):
        ctas, own = tiles * G * n, 4 + R / n * steps
        if causal:      # the last tile of a sequence sees two steps, the first all of them
            time = max((4 * ctas + tiles * G * R * (steps + 2) / 2) / 148, own)
        else:
            time = -(-ctas // 148) * own
        return time if n == 1 else time + 2 + 2e-6 * n * values

    best = n = 1
    while n < 8 and R % (2 * n) == 0:
        n *= 2
        if cost(n) < 0.95 * cost(best):
            best = n
    return best


def attn_bwd(q, k, v, o, lse, do, cu_seqlens, max_seqlen, scale, causal, dk_out=None, dv_out=None, splits: int | None = None):
    """Gradients of ``attn_fwd`` (head_dim 128).  Returns dq [N,H,K], dk, dv [N,G,K].
    ``dk_out`` / ``dv_out`` may be row-strided views (e.g. slices of a fused dqkv buffer).
    The fp32 dq accumulation buffer and the delta vector are cached per shape and reused."""
    N, H, Kd = q.shape
    G = k.shape[1]
    dq = torch.empty(N, H, Kd, dtype=q.dtype, device=q.device)
    dk = dk_out if dk_out is not None else torch.empty(N, G, Kd, dtype=q.dtype, device=q.device)
    dv = dv_out if dv_out is not None else torch.empty(N, G, Kd, dtype=q.dtype, device=q.device)
    key = (q.device.index, N, H, Kd)
    scratch = _attn_scratch.get(key)
    if scratch is None:
        _attn_scratch.clear()
        scratch = (lib.scratch("attn_bwd dq_acc", N * H * Kd, torch.float32, q.device),
                   lib.scratch("attn_bwd delta", H * N, torch.float32, q.device))
        _attn_scratch[key] = scratch
    dq_acc, delta = scratch
    if splits is None:
        B = cu_seqlens.numel() - 1     # empty sequences (no padding on the left) among them
        tiles = min(-(-int(max_seqlen) // 128) * B, N // 128 + B)
        splits = attn_bwd_splits(tiles * (Kd // 128), H, G, -(-int(max_seqlen) // 64), causal, N * G * Kd)
    part = torch.empty(splits, 2, N, G * Kd, dtype=torch.float32, device=q.device) if splits > 1 else None
    st = lib.status_tensor(q.device)
    _call("ob_attn_bwd", q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), do.data_ptr(),
          lse.data_ptr(), delta.data_ptr(), dq_acc.data_ptr(), dq.data_ptr(), dk.data_ptr(),
          dv.data_ptr(), cu_seqlens.data_ptr(), cu_seqlens.numel() - 1, int(max_seqlen), N, H, G, Kd,
          q.stride(0), k.stride(0), v.stride(0), o.stride(0), do.stride(0), dk.stride(0), dv.stride(0),
          float(scale), int(causal), splits, lib.ptr(part), st.data_ptr(), lib.stream_ptr())
    return dq, dk, dv


def ce_fwd_bwd(logits, targets, mask, grad_scale, loss_sum, write_grad=True, lse_out=None):
    R, V = logits.shape
    _call("ob_ce_fwd_bwd", logits.data_ptr(), logits.stride(0), R, V, targets.data_ptr(),
          lib.ptr(mask), lib.ptr(grad_scale), loss_sum.data_ptr(), lib.ptr(lse_out),
          int(write_grad), lib.stream_ptr())


def sigmoid_gate_fwd(o, gate):
    """o [M,H,Kd] dense, gate [M,H,Kd] (any row / head stride, unit inner stride): o * sigmoid(gate)."""
    M, H, Kd = o.shape
    out = torch.empty_like(o)
    _call("ob_sigmoid_gate_fwd", o.data_ptr(), gate.data_ptr(), out.data_ptr(), M, H, Kd, gate.stride(0), gate.stride(1),
          lib.stream_ptr())
    return out


def sigmoid_gate_bwd(o, gate, dout):
    M, H, Kd = o.shape
    d_o, d_gate = torch.empty_like(o), torch.empty_like(o)
    _call("ob_sigmoid_gate_bwd", o.data_ptr(), gate.data_ptr(), dout.data_ptr(), d_o.data_ptr(), d_gate.data_ptr(), M, H,
          Kd, gate.stride(0), gate.stride(1), lib.stream_ptr())
    return d_o, d_gate


def ce_finish(stats, tgt_logit, mask, loss_sum, lse_out, counted=(None, 0)):
    """Row log-sum-exp and masked loss from the statistics the logits GEMM wrote (``gemm(..., ce=)``).
    ``counted`` as in ``gemm_counted``."""
    R, n_tiles = stats.shape[0], stats.shape[1]
    _call("ob_ce_finish", stats.data_ptr(), n_tiles, tgt_logit.data_ptr(), lib.ptr(mask), loss_sum.data_ptr(),
          lse_out.data_ptr(), R, lib.ptr(counted[0]), counted[1], lib.stream_ptr())


def ce_supervised(mask, targets):
    """Rows with a nonzero mask, in order: (count int32 [1], rows [M] of every number, place [M] of every
    row or -1, their targets, their mask)."""
    M, dev = mask.numel(), mask.device
    rows, place, tgt = torch.empty(3, M, dtype=torch.int32, device=dev).unbind(0)
    mk = torch.empty(M, dtype=torch.float32, device=dev)
    count = torch.empty(1, dtype=torch.int32, device=dev)
    _call("ob_ce_count", mask.data_ptr(), targets.data_ptr(), M, rows.data_ptr(), place.data_ptr(), tgt.data_ptr(), mk.data_ptr(),
          count.data_ptr(), lib.stream_ptr())
    return count, rows, place, tgt, mk


def ce_gather(h, rows, count):
    """The counted rows of h [M, D] first, then zeros up to their next multiple of 64; what follows stays unwritten."""
    out = torch.empty_like(h)
    _call("ob_ce_gather", h.data_ptr(), rows.data_ptr(), count.data_ptr(), out.data_ptr(), h.shape[0], h.shape[1], lib.stream_ptr())
    return out


def ce_scatter(dh, place, g, scale):
    """bf16 rows: g and what ``scale`` is beyond a power of two times row ``place`` of fp32 ``dh``, or zero."""
    out = torch.empty(dh.shape, dtype=bf16, device=dh.device)
    _call("ob_ce_scatter", dh.data_ptr(), place.data_ptr(), g.data_ptr(), scale.data_ptr(), out.data_ptr(), dh.shape[0], dh.shape[1],
          lib.stream_ptr())
    return out


def ce_counted_grad_(logits, targets, lse, mask, grad_scale, counted):
    """Logits -> dlogits over what ``grad_scale`` is beyond a power of two, in place for the counted rows; zeros up to
    their next multiple of 64."""
    R, V = logits.shape
    _call("ob_ce_counted_grad", logits.data_ptr(), R, V, logits.stride(0), targets.data_ptr(), lse.data_ptr(), mask.data_ptr(),
          grad_scale.data_ptr(), counted[0].data_ptr(), counted[1], lib.stream_ptr())


def head_gradient_is_one_sum(V: int, D: int, rows: int, counted: bool) -> bool:
    """Whether a weight gradient of the head over so many rows is added as one sum per element.  Only then does it round the same when
    it is stored: a sum that the kernels cut for the sake of their last wave is the more precise one."""
    return rows < 2048 or (counted and bool(lib.ask("ob_gemm_counted_one_sum", V, D, rows)))


def gemm_counted(kind: int, a, b, out, counted, ce=None, scale=None, accumulate: bool = True):
    """The head's products when only the first ``counted[0]`` (int32 [1] on the device) - ``counted[1]`` rows
    of ``a`` hold anything.  kind 0: out bf16 = a b^T with the statistics ``ce``; kind 1: out fp32 += a b;
    kind 2: out fp32 += a^T b, times what ``scale`` (fp32 [1]) is beyond a power of two (without ``accumulate``: =)."""
    (M, K) = (a.shape[1], a.shape[0]) if kind == 2 else a.shape
    N = b.shape[1] if kind else b.shape[0]
    ce_ptrs = (None, None, None) if ce is None else (ce[0].data_ptr(), ce[1].data_ptr(), ce[2].data_ptr())
    if b.shape[0 if kind else 1] != K or out.shape != (M, N) or out.dtype != (torch.float32 if kind else bf16):
        raise ValueError("operands or output do not fit")
    for t in (a, b, out):
        if t.stride(1) != 1:
            raise ValueError("row-major operands expected")
    _call("ob_gemm_counted_rows", kind, a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, a.stride(0), b.stride(0), out.stride(0),
          counted[0].data_ptr(), counted[1], *ce_ptrs, lib.ptr(scale), int(accumulate or kind != 2), lib.status_tensor(a.device).data_ptr(),
          lib.stream_ptr())
    return out


def embedding_fwd(ids, table):
    ids32 = ids.reshape(-1).to(torch.int32)
    lib.check_index("embedding_fwd ids", ids32, table.shape[0])
    out = torch.empty(ids32.numel(), table.shape[1], dtype=table.dtype, device=table.device)
    _call("ob_embedding_fwd", ids32.data_ptr(), table.data_ptr(), out.data_ptr(), ids32.numel(),
          table.shape[1], lib.stream_ptr())
    return out.view(*ids.shape, table.shape[1])


def embedding_bwd(ids, dy, dtable_f32, row_lo=0, row_hi=None):
    ids32 = ids.reshape(-1).to(torch.int32)
    d2 = dy.reshape(-1, dy.shape[-1])
    if not d2.is_contiguous():
        d2 = d2.contiguous()
    hi = dtable_f32.shape[0] + row_lo if row_hi is None else row_hi
    lib.check_index("embedding_bwd ids", ids32, 2 ** 31 - 1)      # rows outside [row_lo, hi) are skipped, negatives are not expected
    _call("ob_embedding_bwd", ids32.data_ptr(), d2.data_ptr(), dtable_f32.data_ptr(),
          ids32.numel(), d2.shape[1], row_lo, hi, lib.stream_ptr())


def embedding_bwd_peer(ids, dy, peer_ptrs, rows_per_rank: int):
    """Embedding gradient rows added into the owners' fp32 shards over NVLink (``peer_ptrs[r]`` holds
    table rows [r*rows_per_rank, (r+1)*rows_per_rank))."""
    import ctypes

    ids32 = ids.reshape(-1).to(torch.int32)
    d2 = dy.reshape(-1, dy.shape[-1])
    if not d2.is_contiguous():
        d2 = d2.contiguous()
    lib.check_index("embedding_bwd_peer ids", ids32, rows_per_rank * len(peer_ptrs))
    arr = (ctypes.c_void_p * len(peer_ptrs))(*peer_ptrs)
    _call("ob_embedding_bwd_peer", ids32.data_ptr(), d2.data_ptr(), ctypes.cast(arr, ctypes.c_void_p), len(peer_ptrs),
          int(rows_per_rank), ids32.numel(), d2.shape[1], lib.stream_ptr())


def sumsq(g, out, used=None):
    """out += sum of squares of g; ``used`` (uint8, ``used_blocks``) says of every 128 elements whether one is not zero."""
    _call("ob_sumsq", g.data_ptr(), g.numel(), out.data_ptr(), lib.ptr(used), lib.stream_ptr())


def used_blocks(g):
    return torch.empty(-(-g.numel() // 1024) * 8, dtype=torch.uint8, device=g.device)


def adamw(p, m, v, g, p16, *, lr, b1, b2, eps, wd, step, grad_mul=1.0, norm_sq=None,
          max_norm=0.0, zero_grad=True, used=None):
    """``used``: what ``sumsq`` found in g as it is now."""
    bc1 = 1.0 - b1 ** step
    bc2 = 1.0 - b2 ** step
    _call("ob_adamw", p.data_ptr(), m.data_ptr(), v.data_ptr(), g.data_ptr(), lib.ptr(p16),
          p.numel(), float(lr), float(b1), float(b2), float(eps), float(wd), float(bc1),
          float(bc2), float(grad_mul), lib.ptr(norm_sq), float(max_norm), int(zero_grad), lib.ptr(used),
          lib.stream_ptr())


def cast_f32_bf16(src, dst):
    _call("ob_cast_f32_bf16", src.data_ptr(), dst.data_ptr(), src.numel(), lib.stream_ptr())


def transpose(src):
    R, C = src.shape
    dst = torch.empty(C, R, dtype=src.dtype, device=src.device)
    _call("ob_transpose_bf16", src.data_ptr(), dst.data_ptr(), R, C, src.stride(0), dst.stride(0),
          lib.stream_ptr())
    return dst


def l2_flush(buf):
    _call("ob_l2_flush", buf.data_ptr(), buf.numel() * buf.element_size(), lib.stream_ptr())


def decode_append(qkv, qw, kw, positions, seq_of_token, slot_of_token, block_table, page_size, k_pages, v_pages,
                  H, G, HD, rot, theta, eps, one_plus=False):
    """Per-head RMSNorm + RoPE of the new tokens' q and k; k/v go to their page slots.  Returns q."""
    n = qkv.shape[0]
    q = torch.empty(n, H, HD, dtype=qkv.dtype, device=qkv.device)
    _call("ob_decode_append", qkv.data_ptr(), lib.ptr(qw), lib.ptr(kw), positions.data_ptr(),
          seq_of_token.data_ptr(), slot_of_token.data_ptr(), block_table.data_ptr(), block_table.shape[1],
          page_size, q.data_ptr(), k_pages.data_ptr(), v_pages.data_ptr(), n, H, G, HD, rot, float(theta),
          float(eps), int(one_plus), lib.stream_ptr())
    return q


def kv_store(k, v, rows, k_pages, v_pages):
    """k, v [N, G, HD] (row-strided views allowed) into rows ``rows`` (int32 [N]) of [*, G, HD] pages."""
    N, G, HD = k.shape
    lib.check_index("kv_store rows", rows, k_pages.numel() // (G * HD))
    for t in (k, v):
        if t.stride(2) != 1 or t.stride(1) != HD or t.dtype != k_pages.dtype:
            raise ValueError("keys and values need contiguous heads in the type of the pages")
    _call("ob_kv_store", k.data_ptr(), v.data_ptr(), k.stride(0), v.stride(0), rows.data_ptr(), k_pages.data_ptr(), v_pages.data_ptr(),
          N, G * HD, lib.stream_ptr())


def decode_splits(blocks: int, keys: int) -> int:
    """CTAs that share a sequence's keys: as many as fit at once (296: two on each of 148 SMs), with at least 128 keys of capacity each.  In us by
    splits, alone: 32 sequences of 2048 on 8 key heads 1 / 2 / 4: 48 54 62; one of 4096, 8 / 16 / 32 / 48: 13.8 11.3 11.8 16.2; eight of
    4096 on 4, 4 / 8 / 16: 23.8 19.9 25.1; 64 of 1000 on 4, 1 / 2: 28.9 36.6."""
    return max(1, min(32, 296 // max(blocks, 1), keys // 128))


def decode_attn(q, k_pages, v_pages, block_table, seq_lens, page_size, scale, splits=None):
    """q [B,H,HD] attends over each sequence's pages; returns [B,H,HD]."""
    B, H, HD = q.shape
    G = k_pages.shape[2]
    if splits is None:
        splits = decode_splits(B * G, block_table.shape[1] * page_size)
    sc = (torch.empty(B * H * splits * HD, dtype=torch.float32, device=q.device),
          torch.empty(B * H * splits * 2, dtype=torch.float32, device=q.device))
    out = torch.empty_like(q)
    _call("ob_decode_attn", q.data_ptr(), k_pages.data_ptr(), v_pages.data_ptr(), block_table.data_ptr(),
          seq_lens.data_ptr(), B, H, G, HD, block_table.shape[1], page_size, splits, float(scale),
          sc[0].data_ptr(), sc[1].data_ptr(), out.data_ptr(), lib.stream_ptr())
    return out


def causal_conv1d_fwd(x_BTC, w_CK):
    B, T, C = x_BTC.shape
    y = torch.empty_like(x_BTC)
    _call("ob_conv1d_silu_fwd", x_BTC.data_ptr(), w_CK.data_ptr(), y.data_ptr(), B, T, C, w_CK.shape[1], lib.stream_ptr())
    return y


def causal_conv1d_bwd(x_BTC, w_CK, dy, dw_f32):
    B, T, C = x_BTC.shape
    dx = torch.empty_like(x_BTC)
    _call("ob_conv1d_silu_bwd", x_BTC.data_ptr(), w_CK.data_ptr(), dy.data_ptr(), dx.data_ptr(), lib.ptr(dw_f32), B, T, C,
          w_CK.shape[1], lib.stream_ptr())
    return dx


def _gdn_ranges(B: int, H: int, T: int, floats: int):
    """Chunks of 64 tokens in ranges whose work buffers (``floats`` a chunk and head) stay below 2 GB."""
    J = T // 64
    n = max(1, min(J, (1 << 29) // (B * H * floats)))
    return n, [(j, min(J, j + n)) for j in range(0, J, n)]


def _gdn_work(B: int, H: int, T: int, floats: int, new):
    """Ranges of chunks and ``new(chunks of a range)``, their work buffers: half as many chunks where the device has no room for more."""
    n, ranges = _gdn_ranges(B, H, T, floats)
    while True:
        try:
            return ranges, new(n)
        except torch.cuda.OutOfMemoryError:
            if n == 1:
                raise
            n = -(-n // 2)
            ranges = [(j, min(T // 64, j + n)) for j in range(0, T // 64, n)]


def gdn_fwd(q, k, v, g, beta, s0=None, save=True, want_final=False):
    """Chunked gated delta rule, fp32.  q,k [B,T,Hk,128]; v [B,T,H,U]; g,beta [B,T,H]; T % 64 == 0."""
    B, T, Hk, A = q.shape
    H, U = v.shape[2], v.shape[3]
    new = lambda *shape: torch.empty(*shape, dtype=torch.float32, device=v.device)  # noqa: E731
    o = torch.empty_like(v)
    n_out = torch.empty_like(v) if save else None
    states = new(B, H, T // 64, U, A) if save else None
    s_final = new(B, H, A, U) if want_final else None
    ranges, (work, carry) = _gdn_work(B, H, T, 2 * 64 * 64, lambda n: (new(2, B, H, n, 64, 64), new(B, H, U, A) if n < T // 64 else None))
    for j0, j1 in ranges:
        _call("ob_gdn_fwd", q.data_ptr(), k.data_ptr(), v.data_ptr(), g.data_ptr(), beta.data_ptr(), lib.ptr(s0), o.data_ptr(),
              lib.ptr(n_out), lib.ptr(states), lib.ptr(s_final), work[0].data_ptr(), work[1].data_ptr(), lib.ptr(carry), B, T, H, Hk,
              A, U, j0, j1, lib.stream_ptr())
    return o, n_out, states, s_final


def gdn_bwd(q, k, v, g, beta, n_out, states, d_o, d_sfinal=None, want_ds0=False):
    B, T, Hk, A = q.shape
    H, U = v.shape[2], v.shape[3]
    new = lambda *shape: torch.empty(*shape, dtype=torch.float32, device=v.device)  # noqa: E731
    dq, dk = torch.zeros_like(q), torch.zeros_like(k)
    dv = torch.empty_like(v)
    dg, dbeta = torch.zeros_like(g), torch.zeros_like(beta)
    ds0 = new(B, H, A, U) if want_ds0 else None
    ranges, (work, dstate, carry) = _gdn_work(B, H, T, 4 * 64 * 64 + U * A, lambda n: (
        new(4, B, H, n, 64, 64), new(B, H, n, U, A), new(B, H, U, A) if n < T // 64 else None))
    for j0, j1 in reversed(ranges):
        _call("ob_gdn_bwd", q.data_ptr(), k.data_ptr(), v.data_ptr(), g.data_ptr(), beta.data_ptr(), n_out.data_ptr(), states.data_ptr(),
              d_o.data_ptr(), lib.ptr(d_sfinal), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), dg.data_ptr(), dbeta.data_ptr(),
              lib.ptr(ds0), *(w.data_ptr() for w in work), dstate.data_ptr(), lib.ptr(carry), B, T, H, Hk, A, U, j0, j1,
              lib.stream_ptr())
    return dq, dk, dv, dg, dbeta, ds0


def gdn_rows_in(mixed, b, a, neg_a, dt, Hk: int, H: int, U: int, eps: float = 1e-6):
    """Inputs of ``gdn_fwd`` from bf16 rows: mixed [B,T,(2 Hk) 128 + H U] = [q | k | v], b and a [B*T,H]; neg_a, dt fp32 [H].
    q (scaled by 128^-1/2) and k are normed, v cast, beta = sigmoid(b), g = neg_a softplus(a + dt); T is padded to whole chunks
    with zeros."""
    B, T = mixed.shape[:2]
    Tp = -(-T // 64) * 64
    new = lambda *shape: torch.empty(B, Tp, *shape, dtype=torch.float32, device=mixed.device)  # noqa: E731
    q, k, v, g, beta = new(Hk, 128), new(Hk, 128), new(H, U), new(H), new(H)
    _call("ob_gdn_rows_in", mixed.data_ptr(), b.data_ptr(), a.data_ptr(), neg_a.data_ptr(), dt.data_ptr(), q.data_ptr(), k.data_ptr(),
          v.data_ptr(), g.data_ptr(), beta.data_ptr(), B, T, Tp, Hk, H, H * U, 128 ** -0.5, float(eps), lib.stream_ptr())
    return q, k, v, g, beta


def gdn_rows_in_bwd(mixed, b, a, neg_a, dt, dq, dk, dv, dg, dbeta, eps: float = 1e-6):
    """Gradients (dmixed, db, da, dneg_a, ddt)."""
    B, T = mixed.shape[:2]
    Tp, Hk, H = dq.shape[1], dq.shape[2], dv.shape[2]
    dmixed, db, da = torch.empty_like(mixed), torch.empty_like(b), torch.empty_like(a)
    da32, dneg = (torch.empty(B * T, H, dtype=torch.float32, device=mixed.device) for _ in range(2))
    _call("ob_gdn_rows_in_bwd", mixed.data_ptr(), b.data_ptr(), a.data_ptr(), neg_a.data_ptr(), dt.data_ptr(), dq.data_ptr(), dk.data_ptr(),
          dv.data_ptr(), dg.data_ptr(), dbeta.data_ptr(), dmixed.data_ptr(), db.data_ptr(), da.data_ptr(), da32.data_ptr(), dneg.data_ptr(),
          B, T, Tp, Hk, H, H * dv.shape[3], 128 ** -0.5, float(eps), lib.stream_ptr())
    return dmixed, db, da, dneg.sum(0), da32.sum(0)


def gdn_rows_cast(x, T: int):
    """fp32 [B,Tp,H,U] -> bf16 [B,T,H,U] (rows past T dropped), or bf16 [B,T',H,U] -> fp32 [B,T,H,U] (zeros past T')."""
    B, t, H, U = x.shape
    pad = x.dtype == bf16
    y = torch.empty(B, T, H, U, dtype=torch.float32 if pad else bf16, device=x.device)
    _call("ob_gdn_rows_cast", x.data_ptr(), y.data_ptr(), B, min(t, T), max(t, T), H * U, int(pad), lib.stream_ptr())
    return y


def gated_rmsnorm_fwd(x, z, w, eps):
    M, D = x.shape
    y = torch.empty_like(x)
    rstd = torch.empty(M, dtype=torch.float32, device=x.device)
    _call("ob_gated_rmsnorm_fwd", x.data_ptr(), z.data_ptr(), w.data_ptr(), y.data_ptr(), rstd.data_ptr(), M, D,
          float(eps), lib.stream_ptr())
    return y, rstd


def gated_rmsnorm_bwd(dy, x, z, w, rstd, eps, dw_f32):
    M, D = x.shape
    dx, dz = torch.empty_like(x), torch.empty_like(z)
    _call("ob_gated_rmsnorm_bwd", dy.data_ptr(), x.data_ptr(), z.data_ptr(), w.data_ptr(), lib.ptr(rstd), dx.data_ptr(),
          dz.data_ptr(), dw_f32.data_ptr(), M, D, float(eps), lib.stream_ptr())
    return dx, dz


def layernorm_fwd(x, w, b, eps):
    M, D = x.shape
    y = torch.empty_like(x)
    mean = torch.empty(M, dtype=torch.float32, device=x.device)
    rstd = torch.empty(M, dtype=torch.float32, device=x.device)
    _call("ob_layernorm_fwd", x.data_ptr(), w.data_ptr(), b.data_ptr(), y.data_ptr(), mean.data_ptr(), rstd.data_ptr(),
          M, D, float(eps), lib.stream_ptr())
    return y, mean, rstd


def layernorm_bwd(dy, x, w, mean, rstd, dw_f32, db_f32):
    M, D = x.shape
    dx = torch.empty_like(x)
    _call("ob_layernorm_bwd", dy.data_ptr(), x.data_ptr(), w.data_ptr(), mean.data_ptr(), rstd.data_ptr(), dx.data_ptr(),
          dw_f32.data_ptr(), db_f32.data_ptr(), M, D, lib.stream_ptr())
    return dx


def router_topk(logits, k, renorm, counts=None):
    """logits [M,E] bf16 -> probs [M,E] fp32, weights [M,k] fp32, idx [M,k] int32; counts [E] int32 += picks."""
    M, E = logits.shape
    probs = torch.empty(M, E, dtype=torch.float32, device=logits.device)
    w = torch.empty(M, k, dtype=torch.float32, device=logits.device)
    idx = torch.empty(M, k, dtype=torch.int32, device=logits.device)
    _call("ob_router_topk", logits.data_ptr(), probs.data_ptr(), w.data_ptr(), idx.data_ptr(), lib.ptr(counts), M, E, k,
          int(renorm), lib.stream_ptr())
    return probs, w, idx


def router_topk_bwd(probs, w, idx, dw, dprobs, renorm):
    M, E = probs.shape
    dlogits = torch.empty(M, E, dtype=bf16, device=probs.device)
    _call("ob_router_topk_bwd", probs.data_ptr(), w.data_ptr(), idx.data_ptr(), dw.data_ptr(), lib.ptr(dprobs),
          dlogits.data_ptr(), M, E, idx.shape[1], int(renorm), lib.stream_ptr())
    return dlogits


def moe_plan(idx32, E, pad=128, counts=None, with_counts: bool = False):
    """idx [M,k] int32 -> offsets [E+1] int32 (segments padded to ``pad``), dest [M*k] int32, and ``with_counts`` the
    histogram [E].  ``counts`` [E] int32 may carry it already (from the router)."""
    have = counts is not None
    if not have:
        counts = torch.empty(E, dtype=torch.int32, device=idx32.device)
    Pn = idx32.numel()
    offsets = torch.empty(E + 1, dtype=torch.int32, device=idx32.device)
    cursor = torch.empty(E, dtype=torch.int32, device=idx32.device)
    dest = torch.empty(Pn, dtype=torch.int32, device=idx32.device)
    _call("ob_moe_plan", idx32.data_ptr(), counts.data_ptr(), offsets.data_ptr(), cursor.data_ptr(), dest.data_ptr(), Pn,
          E, pad, int(not have), lib.stream_ptr())
    return (offsets, dest, counts) if with_counts else (offsets, dest)


def moe_fill_(rows, counts, offsets):
    """Zeros in the rows of [R, D] between an expert's ``counts`` and the end of its segment."""
    _call("ob_moe_fill", counts.data_ptr(), offsets.data_ptr(), rows.data_ptr(), counts.numel(), rows.shape[1], lib.stream_ptr())
    return rows


def gather_rows(src, idx32):
    out = torch.empty(idx32.numel(), src.shape[1], dtype=src.dtype, device=src.device)
    _call("ob_gather_rows", src.data_ptr(), idx32.data_ptr(), out.data_ptr(), idx32.numel(), src.shape[1], lib.stream_ptr())
    return out


def scatter_rows_(dst, idx32, src, replace: bool):
    _call("ob_scatter_rows", dst.data_ptr(), idx32.data_ptr(), src.data_ptr(), idx32.numel(), dst.shape[1], int(replace),
          lib.stream_ptr())
    return dst


def gather4_fwd(table, idx32_N4, w_N4):
    n = idx32_N4.shape[0]
    lib.check_index("gather4 idx", idx32_N4, table.shape[0])
    out = torch.empty(n, table.shape[1], dtype=table.dtype, device=table.device)
    _call("ob_gather4_fwd", table.data_ptr(), idx32_N4.data_ptr(), w_N4.data_ptr(), out.data_ptr(), n, table.shape[1],
          lib.stream_ptr())
    return out


def gather4_bwd(dout, idx32_N4, w_N4, dtable_f32):
    lib.check_index("gather4 idx", idx32_N4, dtable_f32.shape[0])
    _call("ob_gather4_bwd", dout.data_ptr(), idx32_N4.data_ptr(), w_N4.data_ptr(), dtable_f32.data_ptr(), idx32_N4.shape[0],
          dout.shape[1], lib.stream_ptr())


def gelu_tanh_fwd(x):
    y = torch.empty_like(x)
    _call("ob_gelu_tanh_fwd", x.data_ptr(), y.data_ptr(), x.numel(), lib.stream_ptr())
    return y


def gelu_tanh_bwd(x, dy):
    dx = torch.empty_like(x)
    _call("ob_gelu_tanh_bwd", x.data_ptr(), dy.data_ptr(), dx.data_ptr(), x.numel(), lib.stream_ptr())
    return dx


def ce_vp_stats(logits, targets32, v0):
    R, V = logits.shape
    mx, sm, tg = (torch.empty(R, dtype=torch.float32, device=logits.device) for _ in range(3))
    _call("ob_ce_vp_stats", logits.data_ptr(), R, V, logits.stride(0), int(v0), targets32.data_ptr(), mx.data_ptr(),
          sm.data_ptr(), tg.data_ptr(), lib.stream_ptr())
    return mx, sm, tg


def ce_vp_grad_(logits, targets32, v0, lse, mask, grad_scale):
    R, V = logits.shape
    _call("ob_ce_vp_grad", logits.data_ptr(), R, V, logits.stride(0), int(v0), targets32.data_ptr(), lse.data_ptr(),
          lib.ptr(mask), lib.ptr(grad_scale), lib.stream_ptr())
    return logits
