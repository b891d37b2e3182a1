"""Quantized mixture-of-experts MLP: ``QuantizedSwitchLinear`` / ``SwitchGLU`` / ``MoEBlock``.

The reference reaches MoE models (gpt-oss: 32 experts, top-4) through mlx-lm's ``SwitchGLU`` whose expert
projections are ``QuantizedSwitchLinear`` modules -- named in vllm_metal/quant/awq_loader.py:171-173 -- i.e.
``mx.gather_qmm(x, weight, scales, biases, rhs_indices=indices, transpose=True, group_size, bits)`` over stacked
expert weights ``[E, N, K*bits/32]`` (third-party arithmetic: mlx 0.32.0 / mlx-lm 254d153, not in
the reference's tree -> parity unpinned, semantics restated in oracle/moe.py).  Same attribute names and shapes here.

B200 form: choice of the experts, the sort of the (token, expert) pairs, ONE launch of the gate and up products of all
experts with the activation in their epilogue, ONE of the down products, the weighted sum (csrc/qexperts.cu).  Nothing is read
back to the host.  A block of 32 experts of 2880 x 2880, top 4, int4: 159 us for 32 tokens and 313 us for 1024, where a GEMM per
expert and projection with a read-back of the counts took 1210 and 2734.

Sizes and types that those kernels do not take (``SwitchGLU.grouped_tile_rows``), and the ``mx.gather_qmm`` form of a single
projection, run one affine quantized GEMM per expert that received rows (`b200_qlinear_experts`), with the row counts read back
once.
"""

from __future__ import annotations

import torch
from torch import nn
from torch.autograd import forward_ad
from torch.nn.modules.module import _has_any_global_hook as _any_global_hook

from ..metal import get_ops
from .affine import quantize


class QuantizedSwitchLinear(nn.Module):
    """Stacked expert linears: ``weight`` uint32 ``[E, N, K*bits/32]``, ``scales`` / ``biases`` ``[E, N, K/g]``,
    optional dense ``bias`` ``[E, N]`` (mlx-lm ``QuantizedSwitchLinear``)."""

    def __init__(self, in_features: int, out_features: int, num_experts: int, bias: bool = False,
                 group_size: int = 64, bits: int = 4, dtype: torch.dtype = torch.bfloat16, device=None) -> None:
        super().__init__()
        if in_features % group_size:
            raise ValueError(f"in_features {in_features} not divisible by group_size {group_size}")
        self.group_size, self.bits = group_size, bits
        e, n, k = num_experts, out_features, in_features
        self.register_buffer("weight", torch.zeros((e, n, k * bits // 32), dtype=torch.int32, device=device))
        self.register_buffer("scales", torch.zeros((e, n, k // group_size), dtype=dtype, device=device))
        self.register_buffer("biases", torch.zeros((e, n, k // group_size), dtype=dtype, device=device))
        if bias:
            self.register_buffer("bias", torch.zeros((e, n), dtype=dtype, device=device))
        else:
            self.bias = None

    @property
    def num_experts(self) -> int:
        return self.scales.shape[0]

    @property
    def out_features(self) -> int:
        return self.scales.shape[1]

    @property
    def in_features(self) -> int:
        return self.scales.shape[2] * self.group_size

    @classmethod
    def from_dense(cls, weight: torch.Tensor, bias: torch.Tensor | None = None, group_size: int = 64, bits: int = 4,
                   dtype: torch.dtype = torch.bfloat16) -> QuantizedSwitchLinear:
        """``weight`` ``[E, N, K]`` dense; every expert is quantized like a ``QuantizedLinear``."""
        e, n, k = weight.shape
        m = cls(k, n, e, bias is not None, group_size, bits, dtype, weight.device)
        for i in range(e):
            w, s, b = quantize(weight[i], group_size, bits, dtype)
            m.weight[i].copy_(w)
            m.scales[i].copy_(s)
            m.biases[i].copy_(b)
        if bias is not None:
            m.bias.copy_(bias.to(dtype))
        return m

    def _slice(self, rows: slice, groups: slice, words: slice, keep_bias: bool) -> QuantizedSwitchLinear:
        w, sc, bi = self.weight[:, rows, words], self.scales[:, rows, groups], self.biases[:, rows, groups]
        m = QuantizedSwitchLinear(sc.shape[2] * self.group_size, sc.shape[1], self.num_experts,
                                  self.bias is not None and keep_bias, self.group_size, self.bits, self.scales.dtype,
                                  self.weight.device)
        m.weight.copy_(w)
        m.scales.copy_(sc)
        m.biases.copy_(bi)
        if m.bias is not None:
            m.bias.copy_(self.bias[:, rows])
        return m

    def shard_rows(self, rank: int, world: int) -> QuantizedSwitchLinear:
        """Column-parallel: every expert's output rows [rank*N/world, ...) (gate / up of a tensor-parallel MoE)."""
        n = self.out_features
        if n % world:
            raise ValueError(f"out_features {n} not divisible by world size {world}")
        return self._slice(slice(rank * n // world, (rank + 1) * n // world), slice(None), slice(None), True)

    def shard_cols(self, rank: int, world: int) -> QuantizedSwitchLinear:
        """Row-parallel along K on group boundaries (down); the dense bias stays on rank 0."""
        k = self.in_features
        if k % world or (k // world) % self.group_size:
            raise ValueError(f"in_features {k} / {world} must be a multiple of group_size {self.group_size}")
        kw = k // world
        return self._slice(slice(None), slice(rank * kw // self.group_size, (rank + 1) * kw // self.group_size),
                           slice(rank * kw * self.bits // 32, (rank + 1) * kw * self.bits // 32), rank == 0)

    def forward_sorted(self, x_sorted: torch.Tensor, counts: list[int]) -> torch.Tensor:
        """``x_sorted`` ``[P, K]``: rows grouped by expert (``counts[e]`` consecutive rows for expert e).  One C-ABI call
        (``b200_qlinear_experts``) that launches one quantized GEMM per expert with rows; returns ``[P, N]``."""
        return get_ops().quantized_matmul_experts(x_sorted, self.weight, self.scales, self.biases, counts,
                                                  self.group_size, self.bits, bias=self.bias)

    def forward(self, x: torch.Tensor, indices: torch.Tensor) -> torch.Tensor:
        """``mx.gather_qmm`` form: ``x`` ``[T, K]`` (shared by a token's experts) or ``[T, k, K]``; ``indices``
        ``[T, k]`` -> ``[T, k, N]``."""
        t, k = indices.shape
        order, counts = _sort_pairs(indices, self.num_experts)
        rows = x if x.dim() == 3 else x[:, None, :].expand(t, k, x.shape[-1])
        xs = rows.reshape(t * k, -1).index_select(0, order)
        ys = self.forward_sorted(_f16_operand(xs.contiguous(), self), counts)
        out = torch.empty_like(ys)
        out.index_copy_(0, order, ys)
        return out.reshape(t, k, -1)


def _sort_pairs(indices: torch.Tensor, num_experts: int) -> tuple[torch.Tensor, list[int]]:
    flat = indices.reshape(-1).to(torch.int64)
    order = torch.argsort(flat, stable=True)
    counts = torch.bincount(flat, minlength=num_experts).tolist()  # the one host read-back of the block
    return order, counts


def _f16_operand(x: torch.Tensor, lin: QuantizedSwitchLinear) -> torch.Tensor:
    """The tensor-core linears multiply fp16 operands and would cast every expert's slice of a bf16 ``x`` on their own
    (one more launch per expert): cast the gathered rows once for all experts.  Exact: the values are bf16."""
    ops = get_ops()
    if (x.dtype == torch.bfloat16 and lin.scales.dtype == torch.bfloat16 and lin.in_features % 64 == 0
            and x.data_ptr() % 16 == 0 and x.stride(0) % 8 == 0 and getattr(ops, "_qlinear_kernel", 0) != 1):
        return ops.cast_f16(x)
    return x


def _act_silu(gate: torch.Tensor, up: torch.Tensor) -> torch.Tensor:
    return torch.nn.functional.silu(gate) * up


def _act_gpt_oss(gate: torch.Tensor, up: torch.Tensor, alpha: float = 1.702, limit: float = 7.0) -> torch.Tensor:
    """gpt-oss's clipped SwiGLU (mlx-lm gpt_oss.py ``swiglu``): ``g = min(gate, limit)``, ``u = clip(up, +-limit)``,
    ``g * sigmoid(alpha * g) * (u + 1)``."""
    g = gate.clamp(max=limit)
    u = up.clamp(min=-limit, max=limit)
    return g * torch.sigmoid(alpha * g) * (u + 1.0)


ACTIVATIONS = {"silu": _act_silu, "gpt_oss": _act_gpt_oss}
_GROUPED_ACTIVATIONS = {"silu": (_act_silu, 0), "gpt_oss": (_act_gpt_oss, 1)}  # those that the grouped kernels compute
_WORDS = (torch.int32, torch.uint32)


def _as_defined(m, cls: type, *methods: str) -> bool:
    """Whether a call of ``m`` runs nothing but ``cls``'s methods as they stand in their module: no class of its own, no method
    replaced on the instance or the class, no hooks.  The grouped kernels take the place of such modules only."""
    return (type(m) is cls and all(getattr(cls, n) is _DEFINED[cls][n] and n not in m.__dict__ for n in methods)
            and not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks)
            and not _any_global_hook())


def _differentiated(*tensors) -> bool:
    """Whether a derivative is being taken that reaches one of these: the grouped kernels leave no trace of theirs."""
    return forward_ad._current_level >= 0 or (torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in tensors))


class SwitchGLU(nn.Module):
    """``down(act(gate(x), up(x)))`` per selected expert (mlx-lm ``SwitchGLU``).  The activation runs in fp32 on the
    dtype-rounded projections and is rounded once."""

    def __init__(self, hidden: int, inter: int, num_experts: int, bias: bool = False, group_size: int = 64,
                 bits: int = 4, dtype: torch.dtype = torch.bfloat16, device=None, activation: str = "silu") -> None:
        super().__init__()
        mk = lambda i, o: QuantizedSwitchLinear(i, o, num_experts, bias, group_size, bits, dtype, device)  # noqa: E731
        self.gate_proj, self.up_proj, self.down_proj = mk(hidden, inter), mk(hidden, inter), mk(inter, hidden)
        self.activation = activation

    def grouped_tile_rows(self, x: torch.Tensor, top: int) -> int:
        """Rows per tile with which the grouped kernels take ``x [T, H]``, 0 if they do not.  They take bf16 rows and affine
        parameters, widths that are multiples of 64 and 16-byte aligned tensors, of projections that are nothing but a
        ``QuantizedSwitchLinear``; gradients pass through the other path."""
        g, u, d = self.gate_proj, self.up_proj, self.down_proj
        if (x.dtype != torch.bfloat16 or not x.is_cuda or x.shape[0] == 0 or self.activation not in _GROUPED_ACTIVATIONS
                or ACTIVATIONS[self.activation] is not _GROUPED_ACTIVATIONS[self.activation][0] or _differentiated(x)
                or not all(_as_defined(m, QuantizedSwitchLinear, "forward_sorted") for m in (g, u, d))):
            return 0
        ops = get_ops()
        if getattr(ops, "_qlinear_kernel", 0) == 1 or (g.bits, g.group_size) != (u.bits, u.group_size):
            return 0
        e, h, f = g.num_experts, x.shape[1], g.out_features
        rows = []
        for m, n, k in ((g, f, h), (u, f, h), (d, h, f)):
            group = m.group_size
            if (m.bits not in (4, 8) or group not in (32, 64, 128) or k % 64 or k % group or m.weight.shape != (e, n, k * m.bits // 32)
                    or m.scales.shape != (e, n, k // group) or m.biases.shape != m.scales.shape):
                return 0
            for t, dtypes in ((m.weight, _WORDS), (m.scales, (x.dtype,)), (m.biases, (x.dtype,)), (m.bias, (x.dtype,))):
                if t is not None and (t.dtype not in dtypes or t.device != x.device or not t.is_contiguous() or t.data_ptr() % 16):
                    return 0
            if m.bias is not None and m.bias.shape != (e, n):
                return 0
            rows.append(ops.qexpert_tile_rows(x.shape[0], top, e, n, k, group, m is not d))
        return min(rows)

    def grouped(self, x: torch.Tensor, indices: torch.Tensor, tile_rows: int) -> torch.Tensor:
        """``x [T, H]``, ``indices [T, k]`` int32, in range -> ``[T * k, H]``."""
        ops = get_ops()
        if x.stride(1) != 1 or x.stride(0) % 8 or x.data_ptr() % 16:
            x = x.clone(memory_format=torch.contiguous_format)
        plan = ops.expert_plan(indices.contiguous(), self.gate_proj.num_experts, tile_rows)
        xs = ops.qexpert_rows(x, plan[0], indices.shape[1], self.gate_proj.bits)
        h = ops.qexpert_product(xs, self.gate_proj, plan, up=self.up_proj, activation=_GROUPED_ACTIVATIONS[self.activation][1])
        if (self.down_proj.bits == 4) != (self.gate_proj.bits == 4):  # the way in left the columns in its own weights' order
            order = torch.tensor([0, 2, 4, 6, 1, 3, 5, 7] if self.gate_proj.bits == 4 else [0, 4, 1, 5, 2, 6, 3, 7], device=h.device)
            h = h.view(h.shape[0], -1, 8)[:, :, order].reshape(h.shape)
        return ops.qexpert_product(h, self.down_proj, plan)

    def forward(self, x: torch.Tensor, indices: torch.Tensor) -> torch.Tensor:
        t, k = indices.shape
        tile_rows = self.grouped_tile_rows(x, k) if x.dim() == 2 and x.shape[0] == t and k else 0
        if tile_rows:
            lo, hi = torch.stack(torch.aminmax(indices)).tolist()  # the one host read-back of this form
            if lo < 0 or hi >= self.gate_proj.num_experts:
                raise ValueError(f"expert indices must lie in [0, {self.gate_proj.num_experts}), got {lo} .. {hi}")
            return self.grouped(x, indices.to(torch.int32), tile_rows).reshape(t, k, -1)
        order, counts = _sort_pairs(indices, self.gate_proj.num_experts)
        token_of_pair = torch.div(order, k, rounding_mode="floor")
        xs = x.index_select(0, token_of_pair).contiguous()  # rows grouped by expert: gathered once for gate and up
        xs = _f16_operand(xs, self.gate_proj)
        g = self.gate_proj.forward_sorted(xs, counts)
        u = self.up_proj.forward_sorted(xs, counts)
        h = ACTIVATIONS[self.activation](g.float(), u.float()).to(g.dtype)
        ys = self.down_proj.forward_sorted(_f16_operand(h, self.down_proj), counts)
        out = torch.empty_like(ys)
        out.index_copy_(0, order, ys)
        return out.reshape(t, k, -1)


class Router(nn.Module):
    """Dense router ``x @ W^T (+ b)`` (mlx-lm: ``nn.Linear(hidden, num_experts)``): fp32 accumulate, logits rounded to
    the activation dtype."""

    def __init__(self, hidden: int, num_experts: int, bias: bool, dtype: torch.dtype = torch.bfloat16, device=None) -> None:
        super().__init__()
        self.register_buffer("weight", torch.zeros((num_experts, hidden), dtype=dtype, device=device))
        if bias:
            self.register_buffer("bias", torch.zeros((num_experts,), dtype=dtype, device=device))
        else:
            self.bias = None

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        y = x.float() @ self.weight.float().t()
        if self.bias is not None:
            y = y + self.bias.float()
        return y.to(x.dtype)


class MoEBlock(nn.Module):
    """Router + top-k experts + weighted sum.

    ``routing="topk_softmax"`` (gpt-oss): top-k of the router logits, softmax over the k selected logits.
    ``routing="softmax_topk"`` (Qwen3-MoE style): softmax over all experts, top-k, optionally renormalised.
    Logits are sums of 32 bits rounded to the activations' type, the softmax is in fp32 (the grouped kernels add logits up on the
    tensor cores and take the activations' exponentials fast); ``y = sum_j score_j * expert_j(x)`` accumulated in fp32, rounded once."""

    def __init__(self, router: nn.Module, experts: SwitchGLU, top_k: int, routing: str = "topk_softmax",
                 norm_topk_prob: bool = True) -> None:
        super().__init__()
        if routing not in ("topk_softmax", "softmax_topk"):
            raise ValueError(f"unknown routing {routing!r}")
        self.router, self.experts, self.top_k = router, experts, int(top_k)
        self.routing, self.norm_topk_prob = routing, norm_topk_prob
        self.trace: list | None = None  # tests: a list collects (indices, scores) of every forward

    def _choose(self, x: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor] | None:
        """Router product and choice in one launch, ``(int32, fp32)`` of ``[T, k]``; ``None`` where it does not apply."""
        r = self.router
        if not x.is_cuda or x.dtype != torch.bfloat16 or x.shape[0] == 0 or not _as_defined(r, Router, "forward"):
            return None
        w, b = r.weight, r.bias
        if (_differentiated(x, w, b) or x.stride(1) != 1 or x.stride(0) % 8 or x.data_ptr() % 16 or x.shape[1] % 32
                or w.shape[1] != x.shape[1] or w.dtype != x.dtype or not w.is_contiguous() or w.data_ptr() % 16 or w.device != x.device or w.shape[0] > 128
                or not 1 <= self.top_k <= min(32, w.shape[0])
                or (b is not None and (b.dtype != x.dtype or not b.is_contiguous() or b.device != x.device))):
            return None
        return get_ops().qexpert_route(x, w, b, self.top_k, self.routing == "softmax_topk", self.norm_topk_prob)

    def _whole(self, x: torch.Tensor) -> torch.Tensor | None:
        """The block in one call, ``None`` where that does not apply (what is checked here: code that a call would run beside the
        kernels', types, shapes and strides; sizes and alignment by the call)."""
        r, glu = self.router, self.experts
        if (x.dtype != torch.bfloat16 or not x.is_cuda or x.shape[0] == 0 or x.stride(1) != 1 or self.trace is not None
                or not self._routes_as_defined() or not _as_defined(r, Router, "forward") or not _as_defined(glu, SwitchGLU, "forward")):
            return None
        act = _GROUPED_ACTIVATIONS.get(glu.activation)
        lins = (glu.gate_proj, glu.up_proj, glu.down_proj)
        if act is None or ACTIVATIONS[glu.activation] is not act[0] or not all(_as_defined(m, QuantizedSwitchLinear, "forward_sorted")
                                                                               for m in lins):
            return None
        ops, dev, h = get_ops(), x.device, x.shape[1]
        bits, group = lins[0].bits, lins[0].group_size
        if (getattr(ops, "_qlinear_kernel", 0) == 1 or bits not in (4, 8) or group not in (32, 64, 128)
                or any(m.bits != bits or m.group_size != group for m in lins)):
            return None
        mats = [(m.weight, m.scales, m.biases, m.bias) for m in lins]
        e, f = mats[0][1].shape[:2]
        for (w, s, b, extra), n, k in zip(mats, (f, f, h), (h, h, f), strict=True):
            if (s.dtype is not torch.bfloat16 or b.dtype is not torch.bfloat16 or w.dtype not in _WORDS or s.shape != (e, n, k // group)
                    or b.shape != s.shape or w.shape != (e, n, k * bits // 32) or w.device != dev or s.device != dev or b.device != dev
                    or not (w.is_contiguous() and s.is_contiguous() and b.is_contiguous())):
                return None
            if extra is not None and (extra.dtype is not torch.bfloat16 or extra.shape != (e, n) or extra.device != dev
                                      or not extra.is_contiguous()):
                return None
        rw, rb = r.weight, r.bias
        if (rw.dtype is not torch.bfloat16 or rw.shape != (e, h) or rw.device != dev or not rw.is_contiguous() or (rb is not None and (
                rb.dtype is not torch.bfloat16 or rb.shape != (e,) or rb.device != dev or not rb.is_contiguous()))
                or _differentiated(x, rw, rb)):
            return None
        return ops.qexpert_block(x, (rw, rb), mats, bits, group, self.top_k, act[1], self.routing == "softmax_topk", self.norm_topk_prob)

    def _routes_as_defined(self) -> bool:
        return type(self).route is _DEFINED[MoEBlock]["route"] and "route" not in self.__dict__

    def route(self, x: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
        got = self._choose(x) if x.dim() == 2 else None
        if got is not None:
            return got[0].to(torch.int64), got[1]
        logits = self.router(x).float()
        # stable descending sort: equal scores (bf16-rounded logits do tie) go to the lowest expert id, on every rank
        # and in the oracle alike -- torch.topk leaves the order of ties unspecified
        if self.routing == "topk_softmax":
            vals, idx = torch.sort(logits, dim=-1, descending=True, stable=True)
            return idx[:, :self.top_k], torch.softmax(vals[:, :self.top_k], dim=-1)
        probs = torch.softmax(logits, dim=-1)
        vals, idx = torch.sort(probs, dim=-1, descending=True, stable=True)
        vals, idx = vals[:, :self.top_k], idx[:, :self.top_k]
        if self.norm_topk_prob:
            vals = vals / vals.sum(dim=-1, keepdim=True)
        return idx, vals

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        lead = x.shape[:-1]
        x2 = x.reshape(-1, x.shape[-1])
        y = self._whole(x2)
        if y is not None:
            return y.reshape(*lead, -1)
        tile_rows = self.experts.grouped_tile_rows(x2, self.top_k) if _as_defined(self.experts, SwitchGLU, "forward") else 0
        known = tile_rows and self._routes_as_defined()
        got = self._choose(x2) if known else None
        idx, scores = got if got is not None else self.route(x2)
        if self.trace is not None:
            self.trace.append((idx.to(torch.int64).cpu().numpy(), scores.cpu().numpy()))
        if (known and scores.dtype == torch.float32 and not _differentiated(scores)
                and (_as_defined(self.router, Router, "forward") or _as_defined(self.router, nn.Linear, "forward"))
                and self.router.weight.shape[0] <= self.experts.gate_proj.num_experts):
            # no more logits than there are experts: the choices are in range
            y = self.experts.grouped(x2, idx.to(torch.int32), tile_rows)
            return get_ops().qexpert_sum(y, scores.contiguous()).reshape(*lead, -1)
        y = self.experts(x2, idx)  # [T, k, hidden]
        out = (y.float() * scores[..., None]).sum(dim=1).to(x.dtype)
        return out.reshape(*lead, -1)


_DEFINED = {QuantizedSwitchLinear: {"forward_sorted": QuantizedSwitchLinear.forward_sorted}, SwitchGLU: {"forward": SwitchGLU.forward},
            Router: {"forward": Router.forward}, nn.Linear: {"forward": nn.Linear.forward}, MoEBlock: {"route": MoEBlock.route}}
