"""Attention over a compressed latent: per token the cache holds one short row instead of keys and values per head."""
from __future__ import annotations

import torch

from ..config.model_config import ConfigError
from ..csrc import ops
from ..weights.loader import TensorSpec
from .attention import plan_segments, portion_tiles
from .base import HostBatch, Mixer, PagedLatent, Plan
from .gathered_attention import PortionAttention
from .linear import Linear
from .registry import register_mixer, POSITION_ENCODINGS


@register_mixer("latent_attention")
class LatentAttention(PortionAttention, Mixer):
    """q = Wq x (with q_rank: q = Wuq (rms(Wdq x) * w_q), through a latent of q_rank numbers), per head [head_dim plain | rot_dim rotated].  (c | kr) = Wdkv x: c (kv_rank columns) is normalised,
    c = rms(c) * w_c; kr (rot_dim columns) is one rotated key part for all heads
    (the rotation in halves or in neighbouring pairs, as the position encoding says).  Head h has the key [Wuk_h c | kr]
    and the value Wuv_h c; score = scale * (q_plain . Wuk_h c + q_rot . kr); causal softmax over the last `window` keys
    (None: all); output matrix on the concatenated heads.  Only the row [c | kr] is kept per token.
    rot_dim may be 0: no position enters, there is no kr, and `position` is not given.  With sink the softmax's
    denominator has one more term exp(sink_h), a learned number per head without key or value.  With head_gate head
    h's output is multiplied by sigmoid(Wg x)_h, one more projection of the layer's input.

    Single tokens and short portions never expand the cache: q_plain is carried through Wuk_h once per query
    (q'_h = Wuk_h^T q_plain_h, so that q_plain . Wuk_h c = q'_h . c), every head then attends over the same rows [c | kr]
    with the query [q'_h | q_rot_h] and sums the rows' first kv_rank elements, and Wuv_h expands that sum.  The two
    small products per head are one grouped product each.

    In a bfloat16 engine a portion of EXPAND tokens or more is the other way round (heads of 128, a rotated part of 64 or none):
    the request's latents that it sees are expanded once, [keys, heads x (key | value)], one library product, and the
    tcgen05 attention kernel of the dense decoder takes keys of 128 + 64 and values of 128 from there.  A pair of a query and
    a key then costs 128 + 64 + 128 multiply-adds per head instead of 512 + 64 + 512, which the expansion repays from a few dozen
    queries on, and the scores stay in tensor memory.

    params: hidden, heads, head_dim, rot_dim, v_dim, kv_rank, q_rank (0: none), scale, window, eps, sink, head_gate, position (rope_live
    with rotary_dim = rot_dim; absent where rot_dim is 0), borrows (the layer has no Wdkv: its run reads the rows that another layer's run keeps), keep (the
    widest window among the layers that read this layer's rows: pages older than that go back to the pool).
    Tensors: <prefix>q [heads*(head_dim+rot_dim), hidden] (with q_rank: dq [q_rank, hidden], dq.norm [q_rank], uq
    [heads*(head_dim+rot_dim), q_rank]), dkv [kv_rank+rot_dim, hidden], dkv.norm [kv_rank],
    uk [heads*head_dim, kv_rank], uv [heads*v_dim, kv_rank], o [hidden, heads*v_dim]; sink [heads] where sink; g [heads,
    hidden] where head_gate."""

    graph_safe = True

    # Tokens of a portion from which its keys are expanded.  Measured, us a mixer at width 4,096, 32 heads, compressed
    # against expanded: 32 tokens behind 2,000: 84 / 91; 64 behind 2,000: 105 / 95; 64 behind 8,000: 183 / 166; 128 behind 8,000:
    # 283 / 164; a prompt of 2,048: 969 / 242.
    EXPAND = 64
    EXPANDED_BYTES = 1 << 30     # and the most that the expansion may take; longer contexts stay compressed

    def __init__(self, spec, prefix=""):
        super().__init__(spec, prefix)
        p = spec.params
        self.hidden, self.heads, self.head_dim = p["hidden"], p["heads"], p["head_dim"]
        self.rot_dim, self.v_dim, self.rank = p["rot_dim"], p["v_dim"], p["kv_rank"]
        self.scale, self.eps = float(p["scale"]), float(p.get("eps", 1e-6))
        self.window, self.borrows, self.chunk, self.sinks = p.get("window"), bool(p.get("borrows", False)), None, None
        self.keep = p.get("keep", self.window) if self.window else None
        self.q_rank = int(p.get("q_rank") or 0)
        self.sink, self.head_gate = bool(p.get("sink", False)), bool(p.get("head_gate", False))
        if self.rank + self.rot_dim > 640:
            raise ConfigError("unsupported", f"latent attention: rows of {self.rank + self.rot_dim} numbers: the "
                                             "attention kernel takes up to 640")
        pos = p.get("position")
        if (pos is None) != (self.rot_dim == 0):
            raise ConfigError("data_error", "latent attention: a rotated part needs a position encoding, and only it")
        self.position = None if pos is None else POSITION_ENCODINGS.get(pos.kind)(pos)

    def cache_needs(self):
        return () if self.borrows else (PagedLatent(self.rank + self.rot_dim, self.keep),)

    def tensor_specs(self):
        p, e, H = self.prefix, self.hidden, self.heads
        qw = H * (self.head_dim + self.rot_dim)
        specs = [TensorSpec(p + "q", (qw, e))] if not self.q_rank else \
            [TensorSpec(p + "dq", (self.q_rank, e)), TensorSpec(p + "dq.norm", (self.q_rank,), init="one_plus_normal", wide=True),
             TensorSpec(p + "uq", (qw, self.q_rank))]
        if not self.borrows:
            specs += [TensorSpec(p + "dkv", (self.rank + self.rot_dim, e)),
                      TensorSpec(p + "dkv.norm", (self.rank,), init="one_plus_normal", wide=True)]
        specs += [TensorSpec(p + "uk", (H * self.head_dim, self.rank)), TensorSpec(p + "uv", (H * self.v_dim, self.rank)),
                  TensorSpec(p + "o", (e, H * self.v_dim))]
        if self.sink:
            specs.append(TensorSpec(p + "sink", (H,), std=1.0, wide=True))
        if self.head_gate:
            specs.append(TensorSpec(p + "g", (H, e)))
        return specs + (self.position.tensor_specs() if self.position is not None else [])

    def load(self, tensors, rt):
        super().load(tensors, rt)
        p, H, d, R = self.prefix, self.heads, self.head_dim, self.rank
        # one product for all projections of the layer's input: q or the query's latent, then (where the layer makes its own
        # latent) the latent's rows, then the gates; rows of zeros fill the matrix up to a multiple of 8, which the
        # tensor-core kernels want
        ws = [tensors[p + ("dq" if self.q_rank else "q")]]
        self.c_weight = None
        if not self.borrows:
            ws.append(tensors[p + "dkv"])
            self.c_weight = tensors[p + "dkv.norm"].to(torch.float32).contiguous()
        self.c_column, self.gate_column = ws[0].shape[0], sum(w.shape[0] for w in ws)
        if self.head_gate:
            ws.append(tensors[p + "g"])
        self.q_up = self.q_weight = None
        if self.q_rank:
            self.q_up, self.q_weight = self._expansion(tensors[p + "uq"], rt), \
                tensors[p + "dq.norm"].to(torch.float32).contiguous()
        if len({w.dtype for w in ws}) != 1:
            raise ValueError(f"{p}: the projections are stored in different precisions")
        rows = sum(w.shape[0] for w in ws)
        if rows % 8:
            ws.append(torch.zeros((8 - rows % 8, self.hidden), dtype=ws[0].dtype, device=ws[0].device))
        self.proj = Linear(torch.cat(ws, dim=0).contiguous() if len(ws) > 1 else ws[0], rt.status)
        self.sinks = tensors[p + "sink"].to(torch.float32).contiguous() if self.sink else None
        # Wuk_h [d, R] is the product's [K, N]: the grouped product wants [N, K] per head
        self.uk_t = tensors[p + "uk"].view(H, d, R).transpose(1, 2).contiguous()
        self.uv = tensors[p + "uv"].view(H, self.v_dim, R).contiguous()
        # both expansions head by head, [heads x (d + v_dim), R], for portions (a tuple: the matrices above once more)
        self.expansion = ()
        if self.expands:
            self.expansion = (torch.cat([tensors[p + "uk"].view(H, d, R), self.uv], dim=1).reshape(-1, R).contiguous(),)
        self.o = Linear(tensors[p + "o"], rt.status)
        if self.position is not None:
            self.position.load(tensors, rt)
            if not hasattr(self.position, "frequencies64") or self.position.magnitude != 1.0:
                raise ConfigError("unsupported", "latent attention takes a rotation with 64-bit frequencies and no magnitude")
            if self.position.rotary_dim != self.rot_dim:
                raise ConfigError("data_error", "latent attention: the rotation covers the rotated part, all of it")

    @property
    def expands(self) -> bool:
        return (self.rt.dtype == torch.bfloat16 and self.head_dim == 128 and self.v_dim == 128 and self.rot_dim in (0, 64)
                and self.rank % 8 == 0)

    def plan_key(self):
        key = super().plan_key()
        return key + ("expanded", self.heads, self.window) if key is not None and self.expands else key

    def portions_key(self):
        return self.plan_key()

    def plan(self, batch: HostBatch) -> Plan:
        """PortionAttention's plan; where this layer expands, the portions that it expands are in `expanded` instead: (first
        row, tokens, first position, slot, number of slots of partial sums), their tile lists in tiles<i>, segments<i> and
        items<i> as TiledAttention.plan has them.  rows: how many of the step's leading rows the other roads need (all of them
        up to the last row that is not in an expanded portion)."""
        plan = super().plan(batch)
        if not self.expands:
            return plan
        expanded, kept = [], []
        for r0, n, pos0, slot in plan.values["portions"]:
            keys = pos0 + n - self.first_visible(pos0)
            if n < self.EXPAND or keys * self.heads * 512 > self.EXPANDED_BYTES:
                kept.append((r0, n, pos0, slot))
                continue
            tiles, key_tiles = portion_tiles(n, pos0, slot, r0, self.window)
            cut = plan_segments(key_tiles, self.heads)
            i, slots = len(expanded), 0
            plan.arrays[f"tiles{i}"] = tiles
            if cut is not None:
                plan.arrays[f"segments{i}"], plan.arrays[f"items{i}"], slots = cut
            expanded.append((r0, n, pos0, slot, slots))
        taken = {r0 for r0, *_ in expanded}
        rows = max((batch.q_start[i + 1] for i, r0 in enumerate(batch.q_start[:-1]) if r0 not in taken), default=0)
        plan.values.update(portions=kept, expanded=expanded, rows=rows)
        return plan

    def expanded_keys(self, pos0: int, n: int):
        """What is expanded for a portion of n tokens at pos0: (the first row's position, rows that stand ahead of the first
        visible key, rows).  The attention kernel's tiles want the first row at a multiple of 64; the keys from there to the
        first visible one may lie in pages that the request has given back, so their rows are zeros."""
        first = self.first_visible(pos0)
        origin = first // 64 * 64
        return origin, first - origin, pos0 + n - origin

    def _attend_expanded(self, plan, q, q_rot, latent, bt, ctx, out):
        """out rows of the plan's expanded portions."""
        for i, (r0, n, pos0, slot, slots) in enumerate(plan.expanded):
            lo, ahead, count = self.expanded_keys(pos0, n)
            keys = -(-count // 16) * 16
            rows = ops.empty((1, keys, self.rank + self.rot_dim), torch.bfloat16, q.device)
            ops.gather_keys(latent.rows, bt[slot], lo, count, rows, None, latent=True, ahead=ahead)
            kv = torch.mm(rows[0, :, :self.rank], self.expansion[0].t())
            cut = getattr(plan, f"segments{i}", None)
            ops.prefill_attention_expanded(q, q_rot, kv, rows[0], self.rank, lo, getattr(plan, f"tiles{i}"), out, self.window,
                                           self.scale, status=ctx.status, segments=cut, items=getattr(plan, f"items{i}", None),
                                           slots=slots, sink=self.sinks)

    @staticmethod
    def _expansion(w, rt):
        """The product that makes the heads' queries from their latent: its inner size filled up with zeros to a multiple of
        8, its rows to a multiple of 4, which the tensor-core kernels want."""
        rows, inner = w.shape
        if w.dtype == torch.bfloat16 and (rows % 4 or inner % 8):
            full = torch.zeros((rows + -rows % 4, inner + -inner % 8), dtype=w.dtype, device=w.device)
            full[:rows, :inner] = w
            w = full
        return Linear(w, rt.status)

    def _queries(self, proj):
        """float32 [T, heads * (head_dim + rot_dim)] (a band of columns) from the first projection."""
        width = self.heads * (self.head_dim + self.rot_dim)
        if not self.q_rank:
            return proj[:, :width]
        latent = ops.empty((proj.shape[0], self.q_up.in_features), self.rt.dtype, proj.device)
        ops.band_rmsnorm(proj[:, :self.q_rank], self.q_weight, self.eps, latent)
        return self.q_up.f32(latent)[:, :width]

    def forward(self, x, ctx, cache, owns_cache=True):
        if owns_cache == self.borrows:
            raise ops.KernelError("latent attention: the layer and the run list disagree on whose rows the layer reads")
        (latent,) = cache
        T, H, d, rot, R, dv = x.shape[0], self.heads, self.head_dim, self.rot_dim, self.rank, self.v_dim
        rt = self.rt
        dev = x.device
        bt = ctx.block_tables[latent.group]
        proj = self.proj.f32(x)
        plan = ctx.plans.get(self.plan_key()) if self.expands else None
        expanded = plan is not None and bool(plan.expanded)
        rows = plan.rows if expanded else T         # of the step, from its first on, that the other roads need
        q_plain = ops.empty((T, H, d), rt.dtype, dev)
        q_full = ops.empty((T, H, R + rot), torch.float32, dev) if rows else None
        q_rot = ops.empty((T, H, rot), rt.dtype, dev) if expanded and rot else None
        gate = ops.empty((T, H), torch.float32, dev) if self.head_gate else None
        pos = self.position
        ops.latent_prepare(self._queries(proj), proj[:, self.c_column:self.c_column + R + rot] if owns_cache else None,
                           self.c_weight, self.eps, pos.frequencies64() if pos is not None else None, ctx.positions,
                           ctx.token_seq, bt, q_plain, q_full, latent.rows, owns_cache, status=ctx.status,
                           gate=proj[:, self.gate_column:self.gate_column + H] if gate is not None else None,
                           gate_out=gate, pairing=pos.pairing if pos is not None else "half", q_rot=q_rot)
        out = ops.empty((T, H, dv), rt.dtype, dev)
        if rows:
            ops.grouped_gemm(q_plain, self.uk_t, q_full, R, d, lda=H * d, ldo=H * (R + rot), groups=H, a_group_stride=d,
                             o_group_stride=R + rot, a_local=True, o_local=True, rows_per_group=rows, w_ready=True)
            summed = ops.empty((T, H, R), rt.dtype, dev)
            self.attend(q_full, latent.rows, bt, ctx, summed, latent=True)
            ops.grouped_gemm(summed, self.uv, out, dv, R, lda=H * R, ldo=H * dv, groups=H, a_group_stride=R,
                             o_group_stride=dv, a_local=True, o_local=True, rows_per_group=rows, o_scale=gate, o_scale_ld=H, w_ready=True)
        if expanded:      # (behind the other roads' products, which write all of the leading rows)
            self._attend_expanded(plan, q_plain, q_rot, latent, bt, ctx, out)
            if gate is not None:
                for r0, n, *_ in plan.expanded:
                    ops.head_gate(out[r0:r0 + n], gate[r0:r0 + n], ctx.token_seq[r0:r0 + n])
        return self.o.f32_sums(out.view(T, H * dv))
