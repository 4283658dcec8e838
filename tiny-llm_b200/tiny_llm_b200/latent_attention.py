"""Latent attention: keys and values of all heads are up-projections of one cached low-rank latent per token.

Per token the layer caches ``c = rms_norm(W_dkv h)[:rank]`` and one rotated key part shared by all heads.  Head ``h``
scores ``q_plain_h . (W_uk_h c_j) + q_rot_h . k_rot_j`` and mixes values ``W_uv_h c_j``.  Both up-projections are
folded into the query and the output ("absorbed" form), so attention runs directly on the cache as multi-query
attention with key width ``rank + rot`` and value width ``rank``:

    q_lat_h = W_uk_h^T q_plain_h        o_h = W_uv_h (sum_j p_hj c_j)

which is what makes decoding cheap (no per-head keys are ever rebuilt) and is exact up to rounding.  Parameters:
``heads, dim`` (un-rotated), ``rot_dim`` (rotated), ``vdim``, ``kv_rank``, the rotary layout (``interleaved`` pairs
(2i, 2i+1) or half pairs (i, i + dims/2)), its ``base`` and ``dims``, an optional sliding ``window`` (a token sees
itself and the window-1 tokens before it) and ``scale``.  A layer built without ``w_dkv`` reads the cache of another
layer (its slab is handed in by the model) with its own up-projections, queries and mask.

Two more choices a design may make.  Queries through a latent of their own: with ``w_q_down`` (and ``q_down_norm``)
``q = W_q rms_norm(W_q_down h)``; the down projection is then the one fused with ``w_dkv``.  A learned ``sink`` per head:
the softmax's denominator holds one more term ``exp(sink[h])``, which stands for no token: it has neither key nor value.
"""

from __future__ import annotations

import os

import torch

from .basics import linear, linear_wide


PER_HEAD_ENTRIES = 1 << 30  # keys and values up-projected per head: at most 2 GiB of them


class LatentAttention:
    def __init__(self, *, heads: int, dim: int, rot_dim: int, vdim: int, kv_rank: int, scale: float, rot_dims: int, rot_base: float,
                 interleaved: bool, window: int | None, w_q, w_uk, w_uv, w_o, w_dkv=None, dkv_norm=None, eps: float = 1e-5,
                 w_q_down=None, q_down_norm=None, sink=None):
        self.heads, self.dim, self.rot_dim, self.vdim, self.rank = heads, dim, rot_dim, vdim, kv_rank
        self.scale, self.rot_dims, self.rot_base, self.interleaved = float(scale), int(rot_dims), float(rot_base), bool(interleaved)
        self.window = int(window) if window else 0
        self.eps = float(eps)
        if tuple(w_q.shape)[0] != heads * (dim + rot_dim) or tuple(w_uk.shape) != (heads * dim, kv_rank) or tuple(w_uv.shape) != (heads * vdim, kv_rank):
            raise ValueError("latent attention: projection shapes do not match the head sizes")
        if rot_dims > rot_dim or rot_dims % 2:
            raise ValueError("latent attention: rotary dims must be even and fit the rotated part")
        self.q_rank = 0 if w_q_down is None else int(w_q_down.shape[0])
        if self.q_rank and (tuple(w_q.shape)[1] != self.q_rank or q_down_norm is None or q_down_norm.numel() != self.q_rank):
            raise ValueError("latent attention: the query up projection and norm must match the query latent")
        self.q_down_norm = None if q_down_norm is None else q_down_norm.contiguous()
        self.sink = None if sink is None else sink.detach().float().contiguous()  # the softmax runs in fp32
        if self.sink is not None and self.sink.numel() != heads:
            raise ValueError("latent attention: one sink per head")
        first = w_q_down if self.q_rank else w_q  # what is projected from the layer's input beside the latent
        self.w_q, self.w_o = (None if (w_dkv is not None and not self.q_rank) else w_q.contiguous()), w_o.contiguous()
        self.w_first = first.contiguous() if w_dkv is None and self.q_rank else None
        self.w_uk = w_uk.reshape(heads, dim, kv_rank).contiguous()                    # q_lat_h = q_plain_h @ w_uk[h]
        self.w_uv_t = w_uv.reshape(heads, vdim, kv_rank).transpose(1, 2).contiguous()  # o_h = o_lat_h @ w_uv_t[h]
        self.dkv_norm = None if dkv_norm is None else dkv_norm.contiguous()
        if w_dkv is not None and tuple(w_dkv.shape)[0] != kv_rank + rot_dim:
            raise ValueError("latent attention: the down projection must have kv_rank + rot_dim rows")
        # a caching layer projects q and the latent in ONE product (rows of w_q, then rows of w_dkv)
        self.caches = w_dkv is not None
        self.w_qd = torch.cat([first, w_dkv], dim=0).contiguous() if self.caches else None
        self.tc = (self.w_o.dtype == torch.bfloat16 and dim % 64 == 0 and rot_dim % 8 == 0 and rot_dim <= 64 and dim + rot_dim <= 256 and vdim % 8 == 0 and vdim <= 256
                   and os.environ.get("TL_FLASH_TC", "1") != "0")

    @property
    def cache_width(self) -> int:
        return self.rank + self.rot_dim

    def attention_kernel(self, slab: torch.Tensor) -> tuple[str, int]:
        """(kernel name, tokens per work-list entry) for this layer on ``slab [P, page_size, rank + rot]``."""
        from extensions_b200.tiny_llm_ext_b200 import blocks

        return blocks.attention_kernel(slab.dtype, self.heads, self.rank, self.rot_dim, slab.shape[1])

    def _per_head(self, plan, q3: torch.Tensor) -> bool:
        """Whether this step's attention runs on keys and values up-projected per head instead of on the latents themselves.

        Per query, key and head the absorbed form multiplies ``2 rank + rot`` entries, this one ``dim + rot + vdim`` (1088 and 320 at
        the larger benchmark size), and it runs on tcgen05; its price is the up projection of every cached row that is seen and three more
        launches.  Measured (us): absorbed about 30 + its operations at 110 TFLOP/s; this one about 25 + the up projection at 600
        TFLOP/s + 1.75 for every 64-key tile of the longest sequence and wave of CTAs.  2048 tokens, 16 heads: 723 and 158; 128 tokens
        after 4000: 250 and 172; 64 after 4000: 147 and 168.  Below 38 us the calls are bound by the host and launches count."""
        counts = getattr(plan, "counts", None)
        if not self.tc or counts is None or plan.max_tokens == 1:
            return False
        from extensions_b200.tiny_llm_ext_b200 import blocks

        w = self.window or (1 << 60)
        pairs = sum(n * min(s, w) + n * min(n, w) // 2 for n, s in zip(counts, plan.starts))
        rows = sum(n + s - blocks.latent_first_row(s, self.window) for n, s in zip(counts, plan.starts))
        tiles = min(plan.max_context, w + 128) / 64 * max(1.0, sum(-(-n // 128) for n in counts) * self.heads / (2 * blocks.sm_count(q3.device)))
        absorbed = 30 + pairs * self.heads * (2 * self.rank + self.rot_dim) * 2 / 110e6
        per_head = 25 + 1.75 * tiles + rows * self.rank * self.heads * (self.dim + self.vdim) * 2 / 600e6
        if absorbed <= max(per_head, 38) or rows * self.heads * (self.dim + self.vdim) > PER_HEAD_ENTRIES:
            return False
        return blocks.tma_rows(q3)

    def _attend_heads(self, q3: torch.Tensor, plan, slab: torch.Tensor) -> torch.Tensor | None:
        """``[T, heads, vdim]``: the sequences' cached rows (those that a new token sees) side by side, keys and values of every head from
        them, per-head attention.  None where the memory for them cannot be had: the absorbed form needs none of it."""
        from extensions_b200.tiny_llm_ext_b200 import blocks

        contexts = [n + s - blocks.latent_first_row(s, self.window) for n, s in zip(plan.counts, plan.starts)]
        seen = torch.empty_like(plan.seq_info) if self.window else None
        try:
            rows, table = blocks.latent_rows(slab, plan.block_table, plan.seq_info, contexts, self.window, seen)
            c = rows[:, : self.rank]
            k = linear(c, self.w_uk.view(self.heads * self.dim, self.rank))
            v = torch.bmm(c.expand(self.heads, -1, -1), self.w_uv_t)  # [heads, rows, vdim]
        except torch.OutOfMemoryError:
            return None
        return blocks.latent_attention_heads(q3, k, v, rows[:, self.rank :], table, plan.seq_info if seen is None else seen, sum(-(-n // 128) for n in plan.counts), dim=self.dim,
                                             window=self.window, scale=self.scale, sink=self.sink)

    def __call__(self, h: torch.Tensor, plan, slab: torch.Tensor) -> torch.Tensor:
        from extensions_b200.tiny_llm_ext_b200 import blocks

        T, H, dn, dr = h.shape[0], self.heads, self.dim, self.rot_dim
        if self.q_rank:
            if self.caches:
                y = linear(h, self.w_qd)  # [T, q_rank | rank + dr]
                cq = y[:, : self.q_rank]
            else:
                cq = linear(h, self.w_first)
            blocks.kv_prepare(cq.unflatten(1, (1, self.q_rank)), None, None, q_norm=self.q_down_norm, eps=self.eps)  # the row's norm, in place
            q = linear(cq, self.w_q)
            if self.caches:
                blocks.latent_prepare_parts(q, y[:, self.q_rank :], self.dkv_norm, self.eps, heads=H, dim=dn, rot_dim=dr, rank=self.rank,
                                            rot_dims=self.rot_dims, interleaved=self.interleaved, base=self.rot_base, tok_pos=plan.tok_pos,
                                            tok_seq=plan.tok_seq, block_table=plan.block_table, slab=slab)
            else:
                blocks.rope_rows(q, plan.tok_pos, heads=H, head_stride=dn + dr, first=dn, dims=self.rot_dims, base=self.rot_base, interleaved=self.interleaved)
            q3 = q.view(T, H, dn + dr)
        elif self.caches:
            qd = linear(h, self.w_qd)  # [T, H (dn + dr) | rank + dr]
            blocks.latent_prepare(qd, self.dkv_norm, self.eps, heads=H, dim=dn, rot_dim=dr, rank=self.rank, rot_dims=self.rot_dims,
                                  interleaved=self.interleaved, base=self.rot_base, tok_pos=plan.tok_pos, tok_seq=plan.tok_seq,
                                  block_table=plan.block_table, slab=slab)
            q3 = qd[:, : H * (dn + dr)].unflatten(1, (H, dn + dr))
        else:
            q = linear(h, self.w_q)
            blocks.rope_rows(q, plan.tok_pos, heads=H, head_stride=dn + dr, first=dn, dims=self.rot_dims, base=self.rot_base, interleaved=self.interleaved)
            q3 = q.view(T, H, dn + dr)
        kernel, tile_tokens = self.attention_kernel(slab)
        if kernel == "mma" and self._per_head(plan, q3):
            o = self._attend_heads(q3, plan, slab)
            if o is not None:
                return linear_wide(o.view(T, H * self.vdim), self.w_o)
        q_lat = torch.bmm(q3[:, :, :dn].transpose(0, 1), self.w_uk)          # [H, T, rank]
        o_lat = torch.empty_like(q_lat)
        blocks.latent_attention(q_lat.transpose(0, 1), q3[:, :, dn:], slab, plan.block_table, plan.tiles_for(tile_tokens), plan.tok_pos,
                                window=self.window, scale=self.scale, out=o_lat.transpose(0, 1), kernel=kernel,
                                max_context=getattr(plan, "max_context", 0), sink=self.sink)
        o = torch.bmm(o_lat, self.w_uv_t)                                     # [H, T, vdim]
        return linear_wide(o.transpose(0, 1).reshape(T, H * self.vdim), self.w_o)  # fp32: the layer's norm reads it unrounded
