"""A mixture of gated experts with a router on the device, beside an optional shared expert."""
from __future__ import annotations

import torch

from ..config.model_config import ConfigError
from ..csrc import ops
from ..weights.loader import TensorSpec
from .base import FeedForward, GatedSum
from .linear import Linear, SMALL_ROWS
from .mlp import ClampedGLU, SwiGLU
from .registry import register_feed_forward
from .spec import PartSpec


@register_feed_forward("swiglu_plain_names")
class PlainNamesSwiGLU(SwiGLU):
    """SwiGLU whose three matrices are called <prefix>gate, up and down."""
    NAMES = {"gate": "gate", "up": "up", "down": "down"}


@register_feed_forward("routed_experts")
class RoutedExperts(FeedForward):
    """y = sum over the token's `top` experts e of expert_e(s_e x)  +  g shared(x).

    Router: z = Wr x in 32-bit; scores s = sigmoid(z) (score "sigmoid") or softmax(z); the `top` largest are chosen
    (of equal scores the lower index); the weights are the chosen scores, divided by their sum (+ norm_eps) where
    renormalize, times route_scale.  With groups = (count, keep) experts g * (experts / count) .. (g + 1) * (experts /
    count) - 1 make group g, a group's mark is its best score plus its second best (group_mark "two", the default) or its best
    score alone ("best"), and only experts of the `keep`
    groups with the highest marks can be chosen.  With weight_on "input" (the default) the weight multiplies the expert's INPUT (the
    scaled row is rounded to the compute dtype like any input of a product), which is not the same as weighting its
    output, since an expert is not linear; with "output" it multiplies the expert's output, in 32-bit.  expert(u) = Wdown (silu(Wgate u) *
    (Wup u)).  The shared expert (shared_intermediate > 0) has the same form and runs for every token; with shared_gate
    its output is multiplied by g = sigmoid(w_sg . x), one number per token, else g = 1.

    With activation "clamped_glu" an expert, and the shared one, is expert(u) = Wdown (a sigmoid(1.702 a) (b + 1)), a = min(Wgate
    u, limit), b = clamp(Wup u, -limit, limit); the shared expert has a limit of its own (shared_limit).

    With gated False an expert has no gate: expert(u) = Wdown act(Wup u) with act the square of the rectifier
    (activation "relu2").  With choice_bias the experts are chosen by score + bias (a learned number per expert, the
    tensor `correction`) while the weights stay the scores.  With identity = n the router has n more outputs behind the
    experts' own; they stand for experts without matrices whose output is their input (times the weight), and they
    take part in the softmax and in the choice like the others.

    params: hidden, experts, top, intermediate, shared_intermediate, shared_gate, score, renormalize, norm_eps,
    route_scale, groups, group_mark, weight_on, gated, activation, limit, shared_limit, choice_bias, identity.
    Tensors: <prefix>router [experts + identity, hidden], e<i>.gate, e<i>.up [intermediate, hidden], e<i>.down [hidden,
    intermediate], shared.gate, shared.up, shared.down, shared.sg [1, hidden], correction [experts + identity].

    Everything happens on the device: a kernel picks the experts, one orders the (token, choice) pairs by expert, and
    two grouped products (gate and up with the activation; down) walk the experts' rows.  The outputs of a token's
    choices land in `top` planes (times the parts of k, see _parts) that the norm behind the layer adds in order.  A
    row's sum does not depend on the batch in float32; in bfloat16, on the stream of weights, it is the same in all
    steps of up to SMALL_ROWS rows, and in all longer ones.  In a bfloat16 engine the two products are a stream of the chosen experts' weights on the tcgen05 tensor cores
    (ops.expert_stream; sizes that it does not take, and float32, run ops.grouped_gemm).  From so many rows per expert on (in the
    mean; LIBRARY_ROWS, STREAM_HOLDS) a bfloat16 step hands the two products to the library's
    grouped product (which also takes the experts' bounds from the device): there the experts' outputs are rounded to
    bfloat16 before they are added up in 32-bit."""

    # Rows per expert (in the mean) from which the library takes over from ops.grouped_gemm, and how many times as many the stream of
    # weights holds (130 rows).  From WIDE_ROWS on its tiles are of 128 slots: an expert's matrix then goes through the SMs once instead of two
    # times, until most experts have more rows than such a tile.  Measured, a mixture without a shared expert on the device, us, library /
    # tiles of 64 / tiles of 128, even loads: 16 experts of 2,048 at width 2,048, 64 rows per expert 139 / 113 / 111, 80 143 / 127 / 115, 112
    # 149 / 129 / 121, 128 154 / 143 / 135, 130 141 / - / 133, 136 141 / 143 / 152, 140 141 / 145 / 152; 16 of 3,584 at 4,096, 64 rows 360 / 291 / 291, 128 451 /
    # 408 / 354, 130 383 / - / 334, 134 385 / - / 365, 140 350 / 401 / 362; 64 experts of 768 at 2,048 (8 to a token), 64 rows 203 / 162 / 156, 112 225 / 199 / 184, 128 229 / 213 /
    # 217, 132 211 / - / 219, 140 219 / 229 / 229; 128 of them, 64 rows 348 / 293 / 291, 112 420 / 401 / 361, 132 377 / - / 399, 140 387 / 434 / 434; 64 of 1,536 at 4,096 (4 to a
    # token), 64 rows 573 / 489 / 477, 80 590 / 561 / 492, 128 721 / 743 / 647, 140 584 / 750 / 672.  Uneven loads (one expert with five to
    # ten times the mean): 64 of 768, 64 rows 207 / 168 / 176, 100 221 / 188 / 192, 140 227 / 219 / 221; 64 of 1,536, 64 rows 596 / 488 /
    # 500, 80 627 / 514 / 510, 128 774 / 789 / 655.
    LIBRARY_ROWS, STREAM_HOLDS, WIDE_ROWS = 64, 2.03, 64

    graph_safe = True

    def __init__(self, spec, prefix=""):
        super().__init__(spec, prefix)
        p = spec.params
        self.hidden, self.experts, self.top = p["hidden"], p["experts"], p["top"]
        self.inter, self.shared_inter = p["intermediate"], int(p.get("shared_intermediate") or 0)
        self.shared_gate = bool(p.get("shared_gate", False)) and self.shared_inter > 0
        self.score, self.renormalize = p.get("score", "sigmoid"), bool(p.get("renormalize", False))
        self.norm_eps, self.route_scale = float(p.get("norm_eps", 0.0)), float(p.get("route_scale", 1.0))
        self.groups, self.keep = tuple(p["groups"]) if p.get("groups") else (0, 0)
        self.weight_on = p.get("weight_on", "input")
        if self.weight_on not in ("input", "output"):
            raise ConfigError("data_error", f"routed experts: weight_on {self.weight_on!r} (input or output)")
        if self.groups > 1 and (self.experts % self.groups or not (0 < self.keep <= self.groups)
                                or self.top > self.keep * (self.experts // self.groups)):
            raise ConfigError("data_error", "routed experts: the groups must be equal, keep between 1 and their number, "
                                            "and the kept groups must hold at least `top` experts")
        self.gated, self.activation = bool(p.get("gated", True)), p.get("activation", "silu")
        self.choice_bias, self.identity = bool(p.get("choice_bias", False)), int(p.get("identity") or 0)
        self.outputs = self.experts + self.identity          # what the router chooses among
        if (self.gated, self.activation) not in ((True, "silu"), (True, "clamped_glu"), (False, "relu2")):
            raise ConfigError("unsupported", "routed experts: gated experts with SiLU or the clamped activation, or plain ones "
                                             "with the squared rectifier")
        self.act, self.group_mark = ops.SILU, p.get("group_mark", "two")
        if self.activation == "clamped_glu":
            self.act = (1.702, float(p["limit"]), 1.0)      # alpha, limit, shift
        if self.identity < 0 or (self.identity and (self.weight_on != "output" or self.groups > 1)):
            raise ConfigError("unsupported", "routed experts: identity experts take their weight on the output, and "
                                             "no groups")
        if self.top > self.outputs:
            raise ConfigError("data_error", "routed experts: more choices than experts")
        if self.outputs > 512 or self.top > 32:
            raise ConfigError("unsupported", "routed experts: up to 512 experts and 32 choices per token")
        self.shared = None
        if self.shared_inter and self.activation == "clamped_glu":
            self.shared = ClampedGLU(PartSpec("clamped_glu", {"hidden": self.hidden, "intermediate": self.shared_inter,
                                                              "limit": float(p["shared_limit"]), "alpha": 1.702}),
                                     prefix + "shared.")
        elif self.shared_inter:
            self.shared = PlainNamesSwiGLU(PartSpec("swiglu_plain_names", {"hidden": self.hidden,
                                                                           "intermediate": self.shared_inter}),
                                           prefix + "shared.")

    def tensor_specs(self):
        p, e, f = self.prefix, self.hidden, self.inter
        specs = [TensorSpec(p + "router", (self.outputs, e), wide=True)]
        if self.choice_bias:
            specs.append(TensorSpec(p + "correction", (self.outputs,), wide=True, std=0.01))
        for i in range(self.experts):
            specs += ([TensorSpec(f"{p}e{i}.gate", (f, e))] if self.gated else []) + \
                [TensorSpec(f"{p}e{i}.up", (f, e)), TensorSpec(f"{p}e{i}.down", (e, f))]
        if self.shared is not None:
            specs += self.shared.tensor_specs()
        if self.shared_gate:
            specs.append(TensorSpec(p + "shared.sg", (1, e), wide=True))
        return specs

    def load(self, tensors, rt):
        super().load(tensors, rt)
        p, n = self.prefix, self.experts
        rows = [tensors[p + "router"]] + ([tensors[p + "shared.sg"]] if self.shared_gate else [])
        # The router and the shared expert's gate are one product with 32-bit sums.  In a bfloat16 engine its operands
        # are the stored 16-bit weights and the stream's rows as the other products read them: their products are
        # exact in 32 bits, so the tensor cores' 32-bit accumulation is the 32-bit router (rows of zeros fill the matrix
        # up to a multiple of 8, which those kernels want).  A float32 engine runs the 32-bit product.
        w = torch.cat([r.to(rt.dtype) for r in rows], dim=0)
        if not rt.is_fp32 and w.shape[0] % 8:
            w = torch.cat([w, torch.zeros((8 - w.shape[0] % 8, w.shape[1]), dtype=w.dtype, device=w.device)], dim=0)
        self.router = Linear(w.contiguous(), rt.status)
        # gate and up of an expert are one matrix, in the dense feed-forward's arrangement (blocks of gate rows and of up
        # rows in turn), so that the same memory serves the grouped product and the dense products per expert
        F = self.inter
        block = next((b for b in (128, 64, 32) if F % b == 0), F) if rt.dtype == torch.bfloat16 else F
        self.block = block

        def arranged(g, u):
            if block == F:
                return torch.cat([g, u], dim=0)
            return torch.stack([g.view(F // block, block, -1), u.view(F // block, block, -1)], dim=1).reshape(2 * F, -1)

        if self.gated:
            self.gate_up = torch.stack([arranged(tensors[f"{p}e{i}.gate"], tensors[f"{p}e{i}.up"])
                                        for i in range(n)]).contiguous()             # [n, 2F, E]
        else:
            self.gate_up = torch.stack([tensors[f"{p}e{i}.up"] for i in range(n)]).contiguous()      # [n, F, E]
        self.correction = tensors[p + "correction"].to(torch.float32).contiguous() if self.choice_bias else None
        self.down = torch.stack([tensors[f"{p}e{i}.down"] for i in range(n)]).contiguous()      # [n, E, F]
        if self.gate_up.dtype != rt.dtype:
            raise ValueError(f"{p}: the experts are stored as {self.gate_up.dtype}, the engine computes in {rt.dtype}")
        if self.shared is not None:
            self.shared.load(tensors, rt)

    def forward(self, x, ctx):
        T, E, F, n, top = x.shape[0], self.hidden, self.inter, self.experts, self.top
        dev = x.device
        z = self.router.f32_sums(x)      # (few rows: a block per part of k instead of one for all of it)
        expert = ops.empty((T, top), torch.int32, dev)
        weight = ops.empty((T, top), torch.float32, dev)
        gate = ops.empty((T,), torch.float32, dev) if self.shared_gate else None
        ops.moe_route(z, self.outputs, top, expert, weight, gate, has_gate=self.shared_gate, score=self.score,
                      renormalize=self.renormalize, groups=self.groups, keep=self.keep, route_scale=self.route_scale,
                      norm_eps=self.norm_eps, choice_bias=self.correction, mark=self.group_mark)
        on_input = self.weight_on == "input"
        pairs = T * top
        # (three numbers ahead of `start`, so that the experts' ends, start[1:], lie on a 16-byte boundary)
        ints = ops.empty(3 + n + 1 + pairs + 2 * (pairs // ops.GROUP_TILE + n) + 1, torch.int32, dev)[3:]
        start, pair_of_slot = ints[:n + 1], ints[n + 1:n + 1 + pairs]
        tiles, num_tiles = ints[n + 1 + pairs:-1].view(-1, 2), ints[-1:]
        streams = ops.expert_stream_ok(x, self.gate_up, self.block, self.gated) and ops.expert_stream_ok(x, self.down, 0, False)
        by_library = x.dtype == torch.bfloat16 and self._for_the_library(pairs, streams) and E % 16 == 0 and F % 16 == 0
        streams = streams and not by_library
        tile_rows = ops.GROUP_WIDE if streams and pairs >= self.WIDE_ROWS * n else ops.GROUP_TILE
        ops.moe_sort(expert, n, start, pair_of_slot, tiles, num_tiles, tile_rows=tile_rows)
        parts = self._parts(T) if streams else 1
        y = ops.empty((parts * top, T, E), torch.float32, dev)
        if self.identity:
            # (pairs of an expert without matrices get no slot in the order by expert: their planes are written here)
            ops.moe_identity(x, expert, weight, n, y)
        if by_library:
            self._experts_by_the_library(x, start, pair_of_slot, weight, y)
        elif streams:
            rows = ops.rows_by_index(x, pair_of_slot, top, weight.view(-1) if on_input else None,
                                     ops.empty((pairs, E), x.dtype, dev))
            act = ops.empty((pairs, F), x.dtype, dev)
            lists = (start, tiles, num_tiles, T)       # (a token takes an expert once at most)
            ops.expert_stream(rows, self.gate_up, act, *lists, silu_mul=self.gated, relu2=not self.gated, act=self.act,
                              status=self.rt.status, tile_rows=tile_rows)
            ops.expert_stream(act, self.down, y, *lists, o_index=pair_of_slot, o_div=top, splits=parts,
                              o_scale=None if on_input else weight.view(-1), lists_ready=True, status=self.rt.status,
                              tile_rows=tile_rows)
        else:
            act = ops.empty((pairs, F), x.dtype, dev)
            ops.grouped_gemm(x, self.gate_up, act, F, E, lda=E, ldo=F, groups=n, a_index=pair_of_slot, a_div=top,
                             a_scale=weight.view(-1) if on_input else None, start=start, tiles=tiles,
                             num_tiles=num_tiles, silu_mul=self.gated, gate_block=self.block if self.gated else 0,
                             relu2=not self.gated, act=self.act)
            ops.grouped_gemm(act, self.down, y, E, F, lda=F, ldo=E, groups=n, o_index=pair_of_slot, o_div=top,
                             o_part_stride=T * E, start=start, tiles=tiles, num_tiles=num_tiles,
                             o_scale=None if on_input else weight.view(-1))
        if self.shared is None:
            return y
        return GatedSum(y, self.shared.forward(x, ctx), gate)

    def _for_the_library(self, pairs, streams):
        """Whether so many (token, choice) pairs are more than this package's own products hold."""
        most = self.LIBRARY_ROWS * self.experts
        return pairs > self.STREAM_HOLDS * most if streams else pairs >= most

    def _parts(self, T):
        """Parts of k of the second product: halves in a step of few rows, where they are 8 steps of the ring or more.  A step of
        one or two tokens reaches so few experts that whole ranges leave SMs idle; every part has planes of its own, so not with
        identity experts, which write a plane themselves, nor where the planes are many rows.  From the layer's sizes alone on
        either side of SMALL_ROWS (where the dense products change their kernels as well), so that a row's sum does not depend
        on how many others its step has.  Measured, a mixture of 16 experts with 1, 2 and 4 parts, us: width 2,048, one token 57.9, 55.5,
        55.6; 16 tokens 99, 100, 103; 64 tokens 126, 129, 137; width 4,096, one token 99.7, 98.1, 98.3; 8 tokens 209, 211, 216; 64
        tokens 315, 313, 329."""
        k_tiles = -(-self.inter // 64)
        return 1 if self.identity or T > SMALL_ROWS or k_tiles % 2 or k_tiles < 16 else 2

    def _experts_by_the_library(self, x, start, pair_of_slot, weight, y):
        """The road of steps with many rows per expert: the rows in the experts' order with their weights on them, the
        library's grouped product (it takes the experts' bounds from the device) for gate and up, the package's
        activation kernel, the grouped product for down, the results back to the planes."""
        top, (T, E) = self.top, x.shape
        pairs = T * top
        on_input = self.weight_on == "input"
        rows = ops.rows_by_index(x, pair_of_slot, top, weight.view(-1) if on_input else None,
                                 ops.empty((pairs, E), x.dtype, x.device))
        ends = start[1:]
        act = ops.empty((pairs, self.inter), x.dtype, x.device)
        hidden = torch._grouped_mm(rows, self.gate_up.transpose(1, 2), offs=ends)
        if self.activation == "clamped_glu":
            ops.glu(hidden, act, block=self.block, alpha=self.act[0], limit=self.act[1], shift=self.act[2])
        elif self.gated:
            ops.silu_mul(hidden, act, block=self.block)
        else:
            ops.relu2(hidden, act)
        ops.planes_by_index(torch._grouped_mm(act, self.down.transpose(1, 2), offs=ends), pair_of_slot, top, y,
                            scale=None if on_input else weight.view(-1))
