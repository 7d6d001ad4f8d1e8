"""Qwen3 decoder (dense and MoE) as PyTorch modules over the op layer.

Activations travel as packed rows [M = B*T, D].  The hot ops (projections, norms, QK-norm +
RoPE, attention, SwiGLU, experts) go through ``omegalax_b200.ops.functional`` which picks
the sm_100a kernels for CUDA bf16 tensors and the PyTorch definitions otherwise.
Behavioural reference: omegalax/models/qwen3/{model,attention}.py.
"""
from __future__ import annotations

import dataclasses
import math
from types import SimpleNamespace

import torch
import torch.nn.functional as F
from torch import nn
from torch.nn.modules import module as _module_hooks

from ...ops import functional as Fn
from ...ops import moe as moe_ops
from ...ops import reference as R
from ...ops import lib
from ...parallel import tp as tp_lib
from ..decode_graph import DecodeGraph
from .cache import LayerCache
from .config import Qwen3Config
from .norms import RMSNorm
from .utils import compute_positions_from_segment_ids, count_left_pads


from ...utils.profiling import scoped


class Embedding(nn.Module):
    """Token embedding table, normal(0, 0.02) init."""

    def __init__(self, num: int, dim: int, device=None, dtype=None):
        super().__init__()
        self.weight = nn.Parameter(torch.empty(num, dim, device=device, dtype=dtype))
        self.reset_parameters()

    def reset_parameters(self):
        if self.weight.device.type != "meta":
            nn.init.normal_(self.weight, std=0.02)

    def forward(self, ids):
        return Fn.embedding(ids, self.weight)


class Linear(nn.Module):
    """Bias-free (by default) projection, weight [out, in], lecun-normal init."""

    def __init__(self, in_dim: int, out_dim: int, bias: bool = False, device=None, dtype=None):
        super().__init__()
        self.weight = nn.Parameter(torch.empty(out_dim, in_dim, device=device, dtype=dtype))
        self.bias = nn.Parameter(torch.zeros(out_dim, device=device, dtype=dtype)) if bias else None
        self.tp_sharded = False  # True when this rank holds only its tensor-parallel slice
        self.reset_parameters()

    def reset_parameters(self):
        if self.weight.device.type != "meta":
            nn.init.normal_(self.weight, std=1.0 / math.sqrt(self.weight.shape[1]))
            if self.bias is not None:
                nn.init.zeros_(self.bias)

    def forward(self, x, residual=None, tag=None):
        return Fn.linear(x, self.weight, residual=residual, bias=self.bias, tag=tag)


def left_pad_cu_seqlens(k_start, B: int, T: int) -> torch.Tensor:
    """Packed-sequence boundaries for B rows of T positions whose first ``k_start[b]`` positions are
    left padding: int32 [2B+1] = (b*T, b*T + k_start[b]) per row, then B*T.  Each row becomes two
    causal sequences, its pads and its real tokens, so a real query never sees a pad key (what the
    ``k_start`` mask of the PyTorch path does) while the kernels keep plain causal sequences.  Pad
    positions attend among themselves; nothing downstream reads them.  Built on the device."""
    if Fn.library_mode():   # the library baseline runs plain causal rows, as the reference does
        return torch.arange(B + 1, device=k_start.device, dtype=torch.int32) * T
    base = torch.arange(B, device=k_start.device, dtype=torch.int64) * T
    cu = torch.stack([base, base + k_start.to(torch.int64).clamp(0, T)], dim=1).reshape(-1)
    end = torch.full((1,), B * T, device=k_start.device, dtype=torch.int64)
    return torch.cat([cu, end]).to(torch.int32)


@dataclasses.dataclass
class ForwardCtx:
    """Per-call state shared by all layers."""
    B: int
    T: int
    sin: torch.Tensor            # [M, rot/2] fp32
    cos: torch.Tensor
    cu_seqlens: torch.Tensor     # int32 [B+1]
    segment_ids: torch.Tensor    # [B, T]
    k_start: torch.Tensor | None = None   # [B] first real key per row (left padding)
    positions: torch.Tensor | None = None
    extra: dict = dataclasses.field(default_factory=dict)


class Attention(nn.Module):
    def __init__(self, cfg: Qwen3Config, device=None, dtype=None, tp_size: int = 1):
        super().__init__()
        if cfg.num_heads % tp_size or cfg.num_kv_heads % tp_size:
            raise ValueError(f"heads ({cfg.num_heads} q / {cfg.num_kv_heads} kv) do not divide over tp_size={tp_size}")
        H, G, Kd, D = cfg.num_heads // tp_size, cfg.num_kv_heads // tp_size, cfg.head_dim, cfg.emb_dim
        self.H, self.G, self.Kd = H, G, Kd   # heads held by this tensor-parallel rank
        self.tp_size = tp_size
        self.qkv_proj = Linear(D, (H + 2 * G) * Kd, device=device, dtype=dtype)
        self.o_proj = Linear(H * Kd, D, device=device, dtype=dtype)
        self.q_norm = RMSNorm(Kd, cfg.norm_eps, device=device, dtype=dtype)
        self.k_norm = RMSNorm(Kd, cfg.norm_eps, device=device, dtype=dtype)
        self.eps = cfg.norm_eps
        self.scale = Kd ** -0.5
        self.qkv_proj.tp_sharded = self.o_proj.tp_sharded = tp_size > 1

    @scoped("attention")
    def forward(self, x, ctx: ForwardCtx, residual=None, cache: LayerCache | None = None):
        tp = tp_lib.current() if self.tp_size > 1 else None
        if tp is not None:
            x = tp_lib.all_gather_rows(x, tp)      # sequence-parallel rows -> all rows
        M = x.shape[0]
        qkv = self.qkv_proj(x, tag="qkv")
        q, k, v, _ = Fn.qk_norm_rope(qkv, self.q_norm.weight, self.k_norm.weight, ctx.sin, ctx.cos,
                                     self.H, self.G, self.Kd, eps=self.eps)
        B, T = ctx.B, ctx.T
        if cache is None:
            if Fn.use_kernels(q) or (Fn.library_mode() and q.is_cuda):
                o = Fn.flash_attention(q, k, v, ctx.cu_seqlens, T, scale=self.scale, causal=True, tag="attn")
            else:
                ks = None if ctx.k_start is None else ctx.k_start[:, None].expand(B, T)
                o = R.attention(q.reshape(B, T, self.H, self.Kd), k.reshape(B, T, self.G, self.Kd),
                                v.reshape(B, T, self.G, self.Kd), causal=True, scale=self.scale,
                                k_start=ks).reshape(M, self.H, self.Kd)
        else:
            o = self._decode(q, k, v, ctx, cache)
        o = o.reshape(M, self.H * self.Kd)
        if tp is not None:
            return tp_lib.row_parallel_linear(o, self.o_proj.weight, residual, tp)
        return self.o_proj(o, residual=residual, tag="o")

    def _decode(self, q, k, v, ctx: ForwardCtx, cache: LayerCache):
        """Append this call's K/V at the cursor and attend over the whole cache with the mask
        (key position <= query position, both relative to the row's first real token) and
        (key holds a real token).  Softmax in fp32 (reference: qwen3/attention.py:95-132)."""
        B, T = ctx.B, ctx.T
        cur = cache.cur_ind
        k4 = k.reshape(B, T, self.G, self.Kd)
        v4 = v.reshape(B, T, self.G, self.Kd)
        cache.k_cache[:, cur:cur + T] = k4.to(cache.k_cache.dtype)
        cache.v_cache[:, cur:cur + T] = v4.to(cache.v_cache.dtype)
        valid = ctx.extra["kv_valid"]  # [B, S] bool, maintained by the model
        S = cache.size
        kpos = torch.arange(S, device=q.device)[None, :]
        qpos = (cur + torch.arange(T, device=q.device))[None, :, None]
        mask = (kpos[:, None, :] <= qpos) & valid[:, None, :] & (kpos[:, None, :] >= cache.start_ind[:, None, None])
        qf = q.reshape(B, T, self.G, self.H // self.G, self.Kd).float()
        logits = torch.einsum("btgrk,bsgk->btsgr", qf, cache.k_cache.float()) * self.scale
        logits = logits.masked_fill(~mask[:, :, :, None, None], torch.finfo(torch.float32).min)
        p = torch.softmax(logits, dim=2)
        o = torch.einsum("btsgr,bsgk->btgrk", p, cache.v_cache.float())
        cache.cur_ind = cur + T
        return o.reshape(B * T, self.H, self.Kd).to(q.dtype)


class MLP(nn.Module):
    """SwiGLU feed-forward: down(silu(gate(x)) * up(x)) with gate and up fused row-wise."""

    def __init__(self, dim: int, hidden: int, device=None, dtype=None, tp_size: int = 1):
        super().__init__()
        if hidden % tp_size:
            raise ValueError(f"mlp width {hidden} does not divide over tp_size={tp_size}")
        hidden //= tp_size
        self.tp_size = tp_size
        self.gate_up_proj = Linear(dim, 2 * hidden, device=device, dtype=dtype)   # this rank's [gate | up]
        self.down_proj = Linear(hidden, dim, device=device, dtype=dtype)
        self.gate_up_proj.tp_sharded = self.down_proj.tp_sharded = tp_size > 1

    @scoped("feed_forward")
    def forward(self, x, residual=None):
        tp = tp_lib.current() if self.tp_size > 1 else None
        if tp is not None:
            h = Fn.swiglu(tp_lib.column_parallel_linear(x, self.gate_up_proj.weight, tp))
            return tp_lib.row_parallel_linear(h, self.down_proj.weight, residual, tp)
        # With a residual this call produces the decoder layer's output, whose value nothing in the
        # layer's own backward reads ("down" may then be skipped when the layer is re-run).  Without
        # one (e.g. a shared expert whose output is gated) the value is needed: no tag.
        return Fn.swiglu_linear(self.gate_up_proj(x, tag="gate_up"), self.down_proj.weight, residual,
                                tag="down" if residual is not None else None)


class MoEFeedForward(nn.Module):
    """Top-k routed SwiGLU experts with the Qwen3 load-balance loss."""

    def __init__(self, cfg: Qwen3Config, device=None, dtype=None):
        super().__init__()
        E, D, F_ = cfg.num_experts, cfg.emb_dim, cfg.moe_intermediate_size
        self.E, self.k = E, cfg.num_experts_per_tok
        self.norm_topk, self.coef = cfg.norm_topk_prob, cfg.aux_loss_coef
        self.router = Linear(D, E, device=device, dtype=dtype)
        self.experts_gate_up = nn.Parameter(torch.empty(E, 2 * F_, D, device=device, dtype=dtype))
        self.experts_down = nn.Parameter(torch.empty(E, D, F_, device=device, dtype=dtype))
        self.ep = None  # set by the expert-parallel runtime
        self.aux_group = None  # data ranks over which the load-balance statistics are taken
        self.reset_parameters()

    def reset_parameters(self):
        if self.experts_gate_up.device.type != "meta":
            nn.init.normal_(self.experts_gate_up, std=1.0 / math.sqrt(self.experts_gate_up.shape[2]))
            nn.init.normal_(self.experts_down, std=1.0 / math.sqrt(self.experts_down.shape[2]))

    @scoped("moe_feed_forward")
    def forward(self, x, residual=None):
        logits = self.router(x)
        probs, w, idx = moe_ops.route(logits, self.k, self.norm_topk)
        if self.ep is not None:
            y = self.ep.moe_mlp(x, w, idx, self.experts_gate_up, self.experts_down)
        else:
            y = moe_ops.moe_mlp(x, w, idx, self.experts_gate_up, self.experts_down)
        aux = moe_ops.load_balance_loss_qwen3(probs, idx, self.E, self.coef, self.aux_group)
        if residual is not None:
            y = y + residual
        return y, aux


class DecoderLayer(nn.Module):
    def __init__(self, cfg: Qwen3Config, layer_idx: int, device=None, dtype=None, tp_size: int = 1):
        super().__init__()
        self.input_norm = RMSNorm(cfg.emb_dim, cfg.norm_eps, device=device, dtype=dtype)
        self.attn = Attention(cfg, device=device, dtype=dtype, tp_size=tp_size)
        self.post_norm = RMSNorm(cfg.emb_dim, cfg.norm_eps, device=device, dtype=dtype)
        self.is_moe = cfg.is_moe_layer(layer_idx)
        if self.is_moe:
            self.mlp = MoEFeedForward(cfg, device=device, dtype=dtype)
        else:
            self.mlp = MLP(cfg.emb_dim, cfg.mlp_dim, device=device, dtype=dtype, tp_size=tp_size)

    def forward(self, x, ctx: ForwardCtx, cache: LayerCache | None = None):
        x = self.attn(self.input_norm(x), ctx, residual=x, cache=cache)
        h = self.post_norm(x)
        if self.is_moe:
            x, aux = self.mlp(h, residual=x)
        else:
            x, aux = self.mlp(h, residual=x), x.new_zeros((), dtype=torch.float32)
        return x, aux


def vocab_parallel_head(cfg, tp_size: int) -> bool:
    return tp_size > 1 and not cfg.tie_word_embeddings and cfg.vocab_size % (8 * tp_size) == 0


_FORWARDS = {c: c.forward for c in (Linear, RMSNorm, Attention, MLP, DecoderLayer)}
_STEP_METHODS = frozenset(("forward", "embed", "run_layers", "_after_attention"))
_PLAIN = frozenset((int, float, bool))


class Qwen3(nn.Module):
    """Returns the final hidden states (before lm_head) and the summed auxiliary loss; the
    lm_head is a separate projection applied by callers (loss, decode)."""

    def __init__(self, cfg: Qwen3Config, device=None, dtype=None, tp_size: int = 1):
        super().__init__()
        self.cfg = cfg
        self.tp_size = tp_size
        dtype = dtype or torch.float32
        self.embedder = Embedding(cfg.vocab_size, cfg.emb_dim, device=device, dtype=dtype)
        self.layers = nn.ModuleList(DecoderLayer(cfg, i, device=device, dtype=dtype, tp_size=tp_size)
                                    for i in range(cfg.num_layers))
        self.final_norm = RMSNorm(cfg.emb_dim, cfg.norm_eps, device=device, dtype=dtype)
        # untied head under tensor parallelism: split over the vocabulary (vocab-parallel loss)
        self.vocab_parallel = vocab_parallel_head(cfg, tp_size)
        self.lm_head = Linear(cfg.emb_dim, cfg.vocab_size // tp_size if self.vocab_parallel else cfg.vocab_size,
                              device=device, dtype=dtype)
        self.lm_head.tp_sharded = self.vocab_parallel
        self.layer_runner = None  # installed by the training engine (remat / FSDP gather)

    def make_ctx(self, token_ids, segment_ids, position_offset: int = 0, start_ind=None) -> ForwardCtx:
        B, T = token_ids.shape
        dev = token_ids.device
        if start_ind is None:
            positions = compute_positions_from_segment_ids(segment_ids)
            k_start = count_left_pads(segment_ids).to(torch.int64)
        else:
            t = torch.arange(T, device=dev, dtype=torch.int64)[None, :] + position_offset
            positions = torch.where(segment_ids != 0, t - start_ind[:, None].to(torch.int64),
                                    torch.full_like(t.expand(B, T), 2 ** 30))
            k_start = start_ind.to(torch.int64)
        sin, cos = R.rope_tables(positions.reshape(-1), self.cfg.head_dim, self.cfg.rope_theta)
        cu = left_pad_cu_seqlens(k_start, B, T)
        return ForwardCtx(B=B, T=T, sin=sin, cos=cos, cu_seqlens=cu, segment_ids=segment_ids,
                          k_start=k_start, positions=positions)

    def logits(self, hidden):
        return self.lm_head(hidden)

    def _recordable(self, cache):
        """Key under which a recorded single-token step may be replayed: all that ``run_layers`` reads besides its batch, so that a
        step whose key differs is recorded anew.  None: hooks or replaced methods want to see every call, experts are routed (their
        buffers follow the routing), weights are gathered from other GPUs, or layer outputs are being stashed."""
        if (_module_hooks._global_forward_hooks or _module_hooks._global_forward_pre_hooks or lib.debug_enabled()
                or Fn._ACTIVE_STASH is not None):
            return None
        key = [Fn.use_kernels(self.embedder.weight), Fn.library_mode(), self.cfg.rope_theta, cache.page_size, cache.B]
        key += [t.data_ptr() for t in (cache.block_table, *cache.k_pages, *cache.v_pages)]
        left = [self]
        while left:
            m = left.pop()
            own = m.__dict__
            if own["_forward_hooks"] or own["_forward_pre_hooks"] or own.get("is_moe") or not _STEP_METHODS.isdisjoint(own):
                return None
            key += (m, type(m).forward)
            key += [v for v in own.values() if v.__class__ in _PLAIN]      # eps, scale, heads, ...
            for p in own["_parameters"].values():
                if p is not None:
                    if hasattr(p, "ag_spec"):
                        return None
                    key += (p.data_ptr(), p.dtype, p.shape, p.stride())
            left += [c for c in own["_modules"].values() if c is not None]
        return key

    @torch.no_grad()
    def run_layers(self, batch, cache):
        """Residual rows of one new token per sequence, after the last layer."""
        from ...ops import kernels as K

        x, squares = self.embed(batch.ids), None
        fused = self._plain_step(cache, x)
        for li, layer in enumerate(self.layers):
            a, k, v = layer.attn, cache.k_pages[li], cache.v_pages[li]
            if squares is None:
                qkv = a.qkv_proj(layer.input_norm(x))
            else:
                qkv = K.gemm_step(x, a.qkv_proj.weight, norm=(layer.input_norm.weight, layer.input_norm.eps, squares))
            q = K.decode_append(qkv, a.q_norm.weight, a.k_norm.weight, batch.slot, batch.seq, batch.slot,
                                cache.block_table, cache.page_size, k, v, a.H, a.G, a.Kd, a.Kd, self.cfg.rope_theta, a.eps)
            if batch.every:
                o = K.decode_attn(q, k, v, cache.block_table, batch.lens, cache.page_size, a.scale)
            else:
                qb = torch.zeros(cache.B, a.H, a.Kd, dtype=q.dtype, device=q.device)
                qb[batch.seq.long()] = q
                o = K.decode_attn(qb, k, v, cache.block_table, batch.lens, cache.page_size, a.scale)[batch.seq.long()]
            if fused:
                n, m, sums = layer.post_norm, layer.mlp, x.shape[0] <= 32
                x = K.gemm_step(o.reshape(x.shape[0], -1), a.o_proj.weight, residual=x, squares=sums)
                x, squares = x if sums else (x, None)
                if sums:
                    h = K.gemm_step(x, m.gate_up_proj.weight, norm=(n.weight, n.eps, squares), act=True)
                else:
                    h = K.gemm_step(n(x), m.gate_up_proj.weight, act=True)
                x = K.gemm_step(h, m.down_proj.weight, residual=x, squares=sums and li + 1 < len(self.layers))
                x, squares = x if x.__class__ is tuple else (x, None)
            else:
                x = self._after_attention(layer, o, x)
        return x

    def _plain_step(self, cache, x):
        """Whether the products of a step may take norms, activation and sums of squares along: nothing wants to see the modules'
        calls, and all of them are dense and of this file's classes."""
        D = self.cfg.emb_dim
        if (x.shape[0] > 64 or x.dtype != torch.bfloat16 or not Fn.use_kernels(x) or Fn.library_mode() or self.tp_size > 1 or D % 128
                or self._recordable(cache) is None):
            return False
        for la in self.layers:
            a, m = la.attn, la.mlp
            if not (type(la) is DecoderLayer and type(a) is Attention and type(m) is MLP):
                return False
            for n in (la.input_norm, la.post_norm):
                if type(n) is not RMSNorm or n.one_plus or n.scale_in_dtype:
                    return False
            linears = (a.qkv_proj, a.o_proj, m.gate_up_proj, m.down_proj)
            if any(type(p) is not Linear or p.bias is not None or hasattr(p.weight, "main_grad") or p.weight.shape[0] % 128
                   or p.weight.shape[1] % 64 for p in linears):
                return False
            for p in (la.input_norm, la.post_norm, *linears):
                if p.weight.dtype != torch.bfloat16 or not p.weight.is_contiguous() or p.weight.data_ptr() % 16:
                    return False
        return all(c.forward is f for c, f in _FORWARDS.items())

    @staticmethod
    def _after_attention(layer, o, x):
        x = layer.attn.o_proj(o.reshape(x.shape[0], -1), residual=x)
        y = layer.mlp(layer.post_norm(x), residual=x)
        return y[0] if layer.is_moe else y

    @staticmethod
    def _indices(ids, real, cache):
        """Indices of a call's tokens (host [B, T]: ids, and which of them are tokens): parts by name, and all of them in one
        buffer, where every part starts on a 16-byte boundary."""
        ps, counts = cache.page_size, real.sum(-1)
        seq = real.nonzero()[:, 0]
        hist = torch.tensor(cache.seq_lens_host)
        slot = hist[seq] + (real.cumsum(-1) - 1)[real]
        rows = cache.block_table_host[seq, slot // ps] * ps + slot % ps
        cu = torch.cat([counts.new_zeros(1), counts.cumsum(0)])
        has = counts.nonzero()[:, 0]
        parts = dict(ids=ids[real], seq=seq, slot=slot, rows=rows, cu=cu, lens=hist + counts, has=has, last=cu[has + 1] - 1)
        return parts, torch.cat([F.pad(t.to(torch.int32), (0, -t.numel() % 4)) for t in parts.values()])

    def _run_ahead(self, graph, both, cache):
        """A recorded step before the host knows the ids (``both``: ids and marks [2, B, 1] on the device), for callers that had a
        token for every sequence the last time.  Where that holds again the device goes on without a gap: one sequence
        of 4096 tokens, 8 layers of 4096 channels, spent 0.25 of 1.33 ms waiting for the host.  Returns the residual rows; or, where a
        sequence got no token, None and ``both`` on the host, with the cache as it was: what was written for such
        a sequence lies behind its last token, where its next one will go, and its id counted as 0."""
        pages = cache.reserve_ahead()
        if pages is None:
            return None, both
        if graph.asked is None:
            graph.asked = torch.empty(both.shape, dtype=both.dtype, pin_memory=True)
        graph.asked.copy_(both, non_blocking=True)
        graph.arrived.record()
        cache.settle()
        one = torch.ones(cache.B, 1, dtype=torch.bool)
        graph.batch.flat.copy_(self._indices(one.to(torch.int32), one, cache)[1], non_blocking=True)
        torch.mul(both[0], both[1], out=graph.batch.ids.view(-1, 1))
        x = graph.replay()
        graph.arrived.synchronize()
        if bool(graph.asked[1].all()):
            cache.advance([1] * cache.B)
            return x, both
        graph.every = False
        cache.take_back(pages)
        return None, graph.asked.clone()

    @torch.no_grad()
    def decode_paged(self, token_ids, segment_ids, cache, select=None):
        """Prefill or one decode step against a ``PagedKVCache`` (CUDA bf16).  Only real tokens
        are processed and stored; returns the final hidden state of every sequence's last new
        token, [B, D] (zeros for sequences without a new token), or, with the bool mask ``select``
        [B, T], of the marked tokens in order."""
        from ...ops import kernels as K

        cfg = self.cfg
        B, T = token_ids.shape
        dev = token_ids.device
        key = self._recordable(cache) if T == 1 else None
        # The indices of the call are worked out on the host and travel in one copy: the ids are the only thing
        # waited for.  A step of one token per sequence is then one graph launch (8 layers of 4096 channels: 3.1 ms of
        # launches for 1.1 ms of kernels).
        both = torch.stack((token_ids.to(torch.int32), (segment_ids != 0).to(torch.int32)))
        graph = DecodeGraph.recorded(self, cache, key) if key is not None and select is None else None
        if graph is not None and graph.every and B == cache.B and dev == graph.batch.flat.device:
            x, both = self._run_ahead(graph, both, cache)
            if x is not None:
                return self.final_norm(x)
        both = both.cpu()
        real = both[1] != 0
        counts = real.sum(-1)
        new_tokens = counts.tolist()
        cache.reserve(new_tokens)
        cache.settle()
        N, single = sum(new_tokens), max(new_tokens) <= 1
        if not single and any(cache.seq_lens_host[b] > 0 and new_tokens[b] > 0 for b in range(B)):
            raise NotImplementedError("multi-token calls are only supported on an empty cache (prefill)")
        if N == 0:
            return torch.zeros(0 if select is not None else B, cfg.emb_dim, dtype=self.embedder.weight.dtype, device=dev)
        parts, flat = self._indices(both[0], real, cache)
        has = parts["has"]
        # pageable memory is staged before the copy returns
        batch, at = SimpleNamespace(flat=flat.to(dev, non_blocking=True), every=single and N == B), 0
        for name, t in parts.items():
            setattr(batch, name, batch.flat[at:at + t.numel()])
            at += t.numel() + -t.numel() % 4
        if batch.every and key is not None:
            x = DecodeGraph.step(self, cache, batch, key, alone=True)
            graph = DecodeGraph.recorded(self, cache, key)
            if graph is not None:
                graph.every = True
        elif single:
            x = self.run_layers(batch, cache)
        else:
            x = self.embed(batch.ids)
            sin, cos = R.rope_tables(batch.slot, cfg.head_dim, cfg.rope_theta)
            for li, layer in enumerate(self.layers):
                a = layer.attn
                q, k, v, _ = Fn.qk_norm_rope(a.qkv_proj(layer.input_norm(x)), a.q_norm.weight, a.k_norm.weight, sin, cos, a.H, a.G,
                                             a.Kd, eps=a.eps)
                o = Fn.flash_attention(q, k, v, batch.cu, T, scale=a.scale, causal=True)
                K.kv_store(k, v, batch.rows, cache.k_pages[li], cache.v_pages[li])
                x = self._after_attention(layer, o, x)
        cache.advance(new_tokens)
        if select is not None:
            marked = (select.cpu() & real)[real].nonzero()[:, 0]
            return self.final_norm(x[marked.to(dev)])
        if batch.every:
            return self.final_norm(x)
        end = self.final_norm(x[batch.last.long()])
        if has.numel() == B:
            return end
        out = torch.zeros(B, x.shape[1], dtype=x.dtype, device=dev)
        out[batch.has.long()] = end
        return out

    def embed(self, token_ids):
        return Fn.embedding(token_ids.reshape(-1), self.embedder.weight)

    def forward(self, token_ids, segment_ids, cache=None, num_right_pads: int = 0, return_local_rows: bool = False):
        """With tensor parallelism the activations between blocks are sequence-parallel: this rank
        carries rows [r*M/tp, (r+1)*M/tp) of the flattened [B*T] token rows.  By default the final
        hidden states are gathered back to [B,T,D]; ``return_local_rows`` returns this rank's
        rows [M/tp, D] instead (the trainer computes the loss on them)."""
        B, T = token_ids.shape
        if cache is None:
            ctx = self.make_ctx(token_ids, segment_ids)
        else:
            first = cache[0]
            if first.cur_ind == 0:
                start = count_left_pads(segment_ids)
                for lc in cache:
                    lc.start_ind = start.clone()
                valid = torch.zeros(B, first.size, dtype=torch.bool, device=token_ids.device)
            else:
                valid = first._kv_valid  # type: ignore[attr-defined]
            cur = first.cur_ind
            valid = valid.clone()
            valid[:, cur:cur + T] = segment_ids != 0
            first._kv_valid = valid  # type: ignore[attr-defined]
            ctx = self.make_ctx(token_ids, segment_ids, position_offset=cur, start_ind=first.start_ind)
            ctx.extra["kv_valid"] = valid
        x = self.embed(token_ids)
        tp = tp_lib.current() if self.tp_size > 1 else None
        if tp is not None and cache is not None:
            # inference with a KV cache (this rank's kv heads): all rows on every rank
            with tp_lib.replicated_rows(tp):
                aux_total = torch.zeros((), dtype=torch.float32, device=x.device)
                for i, layer in enumerate(self.layers):
                    x, aux = layer(x, ctx, cache[i])
                    aux_total = aux_total + aux
                return self.final_norm(x).view(B, T, -1), aux_total
        if tp is not None:
            if (B * T) % tp.size:
                raise ValueError("tensor parallelism needs B*T divisible by tp_size")
            m = B * T // tp.size
            x = x[tp.rank * m:(tp.rank + 1) * m]
        aux_total = torch.zeros((), dtype=torch.float32, device=x.device)
        for i, layer in enumerate(self.layers):
            lc = None if cache is None else cache[i]
            if self.layer_runner is not None and cache is None:
                x, aux = self.layer_runner(layer, x, ctx)
            else:
                x, aux = layer(x, ctx, lc)
            aux_total = aux_total + aux
        x = self.final_norm(x)
        if tp is not None:
            if return_local_rows:
                return x, aux_total
            x = tp_lib.all_gather_rows(x, tp)
        return x.view(B, T, -1), aux_total
