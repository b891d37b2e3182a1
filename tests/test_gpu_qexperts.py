"""The grouped quantized expert kernels (csrc/qexperts.cu) against float64 over their ranges' edges."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _values(m, e):
    """float64 values of an expert's affine weights."""
    w = m.weight[e].to(torch.int64) & 0xFFFFFFFF
    q = (w.unsqueeze(-1) >> (torch.arange(32 // m.bits, device=w.device) * m.bits)) & (2**m.bits - 1)
    q = q.flatten(-2).unflatten(-1, (-1, m.group_size)).double()
    return (q * m.scales[e].double().unsqueeze(-1) + m.biases[e].double().unsqueeze(-1)).flatten(-2)


def _block(hidden, inter, experts, top, bits, group, act, routing, bias, down_bits=None):
    from vllm_metal_b200.quant.switch_linear import MoEBlock, QuantizedSwitchLinear, Router, SwitchGLU

    g = torch.Generator(device="cuda").manual_seed(hidden + inter + bits)
    glu = SwitchGLU(hidden, inter, experts, bias, group, bits, torch.bfloat16, "cuda", activation=act)
    for name, n, k, b in (("gate_proj", inter, hidden, bits), ("up_proj", inter, hidden, bits), ("down_proj", hidden, inter, down_bits or bits)):
        dense = torch.randn((experts, n, k), device="cuda", generator=g) * k**-0.5
        extra = torch.randn((experts, n), device="cuda", generator=g) * 0.1 if bias else None
        setattr(glu, name, QuantizedSwitchLinear.from_dense(dense, extra, group, b, torch.bfloat16))
    router = Router(hidden, experts, bias, torch.bfloat16, "cuda")
    router.weight.copy_(torch.randn((experts, hidden), device="cuda", generator=g) * 2 * hidden**-0.5)
    return MoEBlock(router, glu, top, routing)


@pytest.mark.parametrize("tokens", [1, 15, 17, 64, 65, 192, 193, 500])
@pytest.mark.parametrize("bits,group,hidden,inter,top,act,routing,bias,down_bits", [
    (4, 64, 320, 192, 2, "gpt_oss", "topk_softmax", True, 4),   # odd rows of groups; half a tile of features on the way out
    (4, 32, 576, 448, 3, "silu", "softmax_topk", False, 8),     # a way out of other words than the way in
    (8, 128, 1024, 128, 1, "silu", "softmax_topk", False, 8),
    (8, 32, 4096, 64, 2, "silu", "topk_softmax", True, 8),      # scales of one item only fit beside large tiles
])
def test_grouped_block_vs_float64(tokens, bits, group, hidden, inter, top, act, routing, bias, down_bits):
    from vllm_metal_b200.metal import get_ops

    blk = _block(hidden, inter, 7, top, bits, group, act, routing, bias, down_bits)
    x = torch.randn((tokens, hidden), device="cuda", generator=torch.Generator(device="cuda").manual_seed(tokens)).bfloat16()
    before = get_ops().launches
    y = blk(x)
    assert get_ops().launches - before == 6  # route, plan, rows, two products, sum
    idx, scores = blk.route(x)
    # the choice: the block says fp32 logits rounded to bf16, ties to the lowest
    logits = blk.router(x).float()
    vals = torch.softmax(logits, -1) if routing == "softmax_topk" else logits
    best, want = torch.sort(vals, dim=-1, descending=True, stable=True)
    same = (idx == want[:, :top]).all(1)
    assert same.float().mean() >= 0.98  # a logit on the edge of two bf16 values may go either way
    part = torch.softmax(best[:, :top], -1) if routing == "topk_softmax" else best[:, :top] / best[:, :top].sum(-1, keepdim=True)
    off = ((scores[same] - part[same]).abs() / part[same]).double()
    # sums in another order put a logit now and then on the other side of a rounding edge: one step of bf16, 2^-8 of it
    assert (off <= 2e-5).double().mean() >= 0.98 and off.max() <= 2 * 2**-8 * float(logits.abs().max()) + 2e-5
    glu, ref = blk.experts, torch.zeros((tokens, hidden), dtype=torch.float64, device="cuda")
    for e in range(7):
        at, place = (idx == e).nonzero(as_tuple=True)
        if len(at):
            lin = lambda z, m, e=e: z @ _values(m, e).T + (m.bias[e].double() if bias else 0)  # noqa: E731
            g, u = lin(x[at].double(), glu.gate_proj), lin(x[at].double(), glu.up_proj)
            if act == "gpt_oss":
                g, u = g.clamp(max=7.0), u.clamp(-7.0, 7.0)
                h = g * torch.sigmoid(1.702 * g) * (u + 1)
            else:
                h = torch.nn.functional.silu(g) * u
            ref[at] += lin(h, glu.down_proj) * scores[at, place].double()[:, None]
    # four roundings to bf16 (gate, up, activation, result: 2^-9 each at most, a third of it in the mean) and weights of 11 bits
    assert (y.double() - ref).norm() <= 4 * 2**-9 * ref.norm()
    assert not get_ops().qexpert_failed()


def test_choices_of_ties_and_nan():
    """Ties go to the lowest expert; a row of NaN stays in range, as the sort of the general path has it."""
    blk = _block(64, 64, 7, 3, 4, 64, "silu", "topk_softmax", False)
    blk.router.weight.zero_()
    x = torch.randn((5, 64), device="cuda").bfloat16()
    x[3] = float("nan")
    idx, scores = blk.route(x)
    assert idx.tolist() == [[0, 1, 2]] * 5 and idx.dtype == torch.int64
    assert torch.isnan(scores[3]).all() and torch.allclose(scores[:3], torch.full((3, 3), 1 / 3, device="cuda"))


def test_indices_out_of_range_are_refused():
    blk = _block(64, 64, 7, 2, 4, 64, "silu", "topk_softmax", False)
    x = torch.randn((3, 64), device="cuda").bfloat16()
    for bad in (-1, 7):
        idx = torch.zeros((3, 2), dtype=torch.int64, device="cuda")
        idx[1, 1] = bad
        with pytest.raises((ValueError, RuntimeError)):
            blk.experts(x, idx)


@pytest.mark.parametrize("top,tokens", [(2, 33), (7, 5)])
def test_the_parts_and_the_whole_agree(top, tokens):
    """The block in one call and its parts one by one (as with a trace, or rows that cannot be read in 16-byte units)."""
    blk = _block(320, 192, 7, top, 4, 64, "gpt_oss", "topk_softmax", True)
    x = torch.randn((tokens, 2, 320), device="cuda").bfloat16()[:, 1]  # rows apart
    y = blk(x)
    blk.trace = []
    assert torch.equal(blk(x), y) and len(blk.trace) == 1
    wide = torch.nn.functional.pad(x, (1, 0))[:, 1:]  # rows that start off 16 bytes: copied
    torch.testing.assert_close(blk(wide), y)
    idx, scores = blk.route(x)
    parts = blk.experts(x, idx)
    want = (parts.float() * scores[..., None]).sum(1)
    torch.testing.assert_close(y.float(), want, rtol=2**-7, atol=1e-5)


def _by_parts(blk, x, idx, scores):
    """The block's result for choices that are given, each expert's GEMM by itself."""
    from vllm_metal_b200.quant import switch_linear as sl

    glu = blk.experts
    order, counts = sl._sort_pairs(idx, glu.gate_proj.num_experts)
    xs = sl._f16_operand(x.index_select(0, order // idx.shape[1]).contiguous(), glu.gate_proj)
    g, u = (sl.QuantizedSwitchLinear.forward_sorted(m, xs, counts) for m in (glu.gate_proj, glu.up_proj))
    h = sl.ACTIVATIONS[glu.activation](g.float(), u.float()).to(g.dtype)
    ys = sl.QuantizedSwitchLinear.forward_sorted(glu.down_proj, sl._f16_operand(h, glu.down_proj), counts)
    out = torch.empty_like(ys)
    out[order] = ys
    return (out.unflatten(0, idx.shape).float() * scores[..., None]).sum(1)


@pytest.mark.parametrize("how", ["subclass", "instance", "class"])
def test_a_route_of_ones_own_is_asked(how, monkeypatch):
    blk = _block(128, 64, 7, 2, 4, 64, "silu", "topk_softmax", False)
    x = torch.randn((9, 128), device="cuda").bfloat16()

    def route(self, x):
        idx = torch.tensor([[6, 0]], device=x.device).expand(x.shape[0], 2)
        return idx, torch.full(idx.shape, 0.5, device=x.device)

    if how == "subclass":
        blk.__class__ = type("Own", (type(blk),), {"route": route})
    elif how == "instance":
        blk.route = route.__get__(blk)
    else:
        monkeypatch.setattr(type(blk), "route", route)
    want = _by_parts(blk, x, *route(blk, x))
    torch.testing.assert_close(blk(x).float(), want, rtol=2**-7, atol=1e-3)


@pytest.mark.parametrize("where", ["router", "experts"])
def test_hooks_and_forwards_of_ones_own_run(where):
    blk = _block(128, 64, 7, 2, 4, 64, "silu", "softmax_topk", False)
    x = torch.randn((9, 128), device="cuda").bfloat16()
    plain = blk(x)
    m = getattr(blk, where)
    seen = []
    for add in (m.register_forward_hook, m.register_forward_pre_hook):
        handle = add(lambda *a: seen.append(1))
        torch.testing.assert_close(blk(x).float(), plain.float(), rtol=2**-7, atol=1e-3)
        handle.remove()
    handle = torch.nn.modules.module.register_module_forward_hook(lambda mod, a, out: seen.append(1) if mod is m else None)
    blk(x)
    handle.remove()
    assert len(seen) == 3
    m.forward = lambda *a: type(m).forward(m, *a) * 0
    y = blk(x)
    assert (y == 0).all() if where == "experts" else not torch.equal(y, plain)


@pytest.mark.parametrize("which", ["gate_proj", "up_proj", "down_proj"])
def test_a_projection_of_ones_own_is_asked(which):
    blk = _block(128, 64, 7, 2, 4, 64, "silu", "topk_softmax", False)
    x = torch.randn((9, 128), device="cuda").bfloat16()
    m = getattr(blk.experts, which)
    m.__class__ = type("Own", (type(m),), {"forward_sorted": lambda self, xs, counts: super(type(self), self).forward_sorted(xs, counts) * 0})
    assert (blk(x) == 0).all() and (blk.experts(x, blk.route(x)[0]) == 0).all()


def test_routers_that_are_no_buffers_of_a_router():
    """A weight that is a Parameter, with gradients through the scores as before; a plain function."""
    blk = _block(128, 64, 7, 2, 4, 64, "silu", "topk_softmax", False)
    x = torch.randn((9, 128), device="cuda").bfloat16()
    plain, w = blk(x), blk.router.weight
    del blk.router.weight
    blk.router.weight = torch.nn.Parameter(w)
    y = blk(x)
    y.float().square().sum().backward()
    assert blk.router.weight.grad.abs().sum() > 0
    with torch.no_grad():
        assert torch.equal(blk(x), plain)
    del blk.router
    blk.router = lambda z: z @ w.t()
    torch.testing.assert_close(blk(x), plain, rtol=2**-6, atol=2e-3)


def test_reads_back_to_the_host():
    """The block none, the experts with choices from elsewhere one."""
    import warnings

    blk = _block(128, 64, 7, 2, 4, 64, "silu", "topk_softmax", False)
    x = torch.randn((9, 128), device="cuda").bfloat16()
    idx = blk.route(x)[0]
    for call, most in ((lambda: blk(x), 0), (lambda: blk.experts(x, idx), 1)):
        call()
        torch.cuda.synchronize()
        with warnings.catch_warnings(record=True) as seen:
            warnings.simplefilter("always")
            torch.cuda.set_sync_debug_mode("warn")
            try:
                call()
            finally:
                torch.cuda.set_sync_debug_mode("default")
        assert sum("called a synchronizing" in str(w.message) for w in seen) <= most


def _product_operands(tokens=40, hidden=128, inter=192, experts=7, top=2, bits=4):
    from vllm_metal_b200.metal import get_ops

    ops, blk = get_ops(), _block(hidden, inter, experts, top, bits, 64, "silu", "topk_softmax", False)
    x = torch.randn((tokens, hidden), device="cuda").bfloat16()
    tile_rows = blk.experts.grouped_tile_rows(x, top)
    plan = ops.expert_plan(blk.route(x)[0].int().contiguous(), experts, tile_rows)
    return ops, blk.experts, plan, ops.qexpert_rows(x, plan[0], top, bits)


def _spoilt(plan, what):
    """The plan with running counts that do not fit together."""
    first, tiles = plan[1].clone(), plan[2].clone()
    if what == "a tile too many":
        tiles[1:] += 1
    elif what == "counts that fall":
        first[2] = first[3] + 5
    elif what == "more tiles than there can be":
        tiles[-1] = 10**6
    elif what == "a negative row":
        first[1] = -4
    elif what == "tiles that start late":
        tiles += 1
    elif what == "rows that start late":
        first[0] = 1
    elif what == "rows that end early":
        first[-1] -= 1
    return plan[0], first, tiles, plan[3]


@pytest.mark.parametrize("what", ["a tile too many", "counts that fall", "more tiles than there can be", "a negative row",
                                  "tiles that start late", "rows that start late", "rows that end early"])
def test_a_plan_that_does_not_fit_together(what):
    """Nothing is touched that the plan leads to, the results are NaN, the status says so until it is reset, and the next call is
    sound."""
    ops, glu, plan, xs = _product_operands()
    assert not ops.qexpert_failed()
    want = ops.qexpert_product(xs, glu.gate_proj, plan, up=glu.up_proj)
    down = ops.qexpert_product(want, glu.down_proj, plan)
    assert torch.isfinite(want).all() and torch.isfinite(down).all()
    bad = _spoilt(plan, what)
    try:
        h = ops.qexpert_product(xs, glu.gate_proj, bad, up=glu.up_proj)
        torch.cuda.current_stream().synchronize()
        assert ops.qexpert_status() and torch.isnan(h).all()
        assert ops.qexpert_status(reset=True) and not ops.qexpert_failed()
        assert torch.isnan(ops.qexpert_product(want, glu.down_proj, bad)).all()
        assert ops.qexpert_failed()
        assert torch.isnan(ops.qexpert_product(h, glu.down_proj, plan)).all()  # what follows shows it
    finally:
        torch.cuda.synchronize()
        ops.qexpert_status(reset=True)
    assert torch.equal(ops.qexpert_product(xs, glu.gate_proj, plan, up=glu.up_proj), want)
    assert not ops.qexpert_failed()


def test_a_step_after_a_failed_product_raises():
    import dataclasses

    from vllm_metal_b200.attention.caches.kv_cache import B200PagedKVCache
    from vllm_metal_b200.lm.decoder import PRESETS, Model
    from vllm_metal_b200.v1.model_runner import PagedModelRunner

    args = dataclasses.replace(PRESETS["tiny"], num_experts=4, experts_per_tok=2)
    cache = B200PagedKVCache(args.num_layers, args.n_kv_heads, args.head_dim, 4, 16, torch.bfloat16, "cuda",
                             sliding_window_per_layer=args.sliding_window_per_layer())
    runner = PagedModelRunner(Model(args, torch.bfloat16, "cuda", seed=0), cache, max_batch=1, max_model_len=32)
    ids, table = list(range(1, 9)), [1]
    want = runner.execute(ids, [], [(table, 8, 0)])
    ops, glu, plan, xs = _product_operands()
    try:
        ops.qexpert_product(xs, glu.gate_proj, _spoilt(plan, "a tile too many"), up=glu.up_proj)
        for step in (lambda: runner.execute(ids, [], [(table, 8, 0)]), lambda: runner.verify(ids, [(table, 0, 8)]),
                     lambda: runner.decode_step([1], [table], [8]), lambda: runner.submit_decode([1], [table], [8]).tokens()):
            with pytest.raises(RuntimeError, match="grouped expert product"):
                step()
    finally:
        torch.cuda.synchronize()
        ops.qexpert_status(reset=True)
    assert runner.execute(ids, [], [(table, 8, 0)]) == want


@pytest.mark.parametrize("experts,top", [(32, 4), (33, 1), (64, 32), (65, 8), (128, 32), (129, 8)])
@pytest.mark.parametrize("routing", ["topk_softmax", "softmax_topk"])
def test_choice_over_more_experts(experts, top, routing):
    """Rows and router of few bits, whose products and sums are exact in any order: the choices, of which many tie, are those of the
    sort; 129 experts are more than the kernel takes."""
    from vllm_metal_b200.metal import get_ops
    from vllm_metal_b200.quant.switch_linear import MoEBlock, Router

    g = torch.Generator(device="cuda").manual_seed(experts)
    router = Router(96, experts, True, torch.bfloat16, "cuda")
    router.weight.copy_(torch.randint(-2, 3, router.weight.shape, device="cuda", generator=g) / 4)
    router.bias.copy_(torch.randint(-2, 3, router.bias.shape, device="cuda", generator=g) / 4)
    x = torch.randint(-1, 2, (37, 96), device="cuda", generator=g).bfloat16()
    before = get_ops().launches
    idx, scores = MoEBlock(router, None, top, routing).route(x)
    assert get_ops().launches - before == (experts <= 128)
    logits = (x.double() @ router.weight.double().T + router.bias.double()).bfloat16().double()
    vals, want = torch.sort(logits, dim=-1, descending=True, stable=True)
    assert torch.equal(idx, want[:, :top])
    part = torch.softmax(vals if routing == "softmax_topk" else vals[:, :top], -1)[:, :top]
    # a few roundings of 32 bits, and an exponential of one or two of its last bits
    torch.testing.assert_close(scores.double(), part / part.sum(-1, keepdim=True), rtol=16 * 2**-24, atol=0)


@pytest.mark.parametrize("experts", [40, 100, 129])
def test_blocks_of_more_experts(experts):
    blk = _block(128, 64, experts, 3, 4, 64, "silu", "softmax_topk", True)
    x = torch.randn((50, 128), device="cuda", generator=torch.Generator(device="cuda").manual_seed(0)).bfloat16()
    # the operands round alike on both ways: what is left is the activation's last bit in 16, and the result's
    torch.testing.assert_close(blk(x).float(), _by_parts(blk, x, *blk.route(x)), rtol=2**-7, atol=2**-7)


@pytest.mark.parametrize("act", ["silu", "gpt_oss"])
def test_operands_beyond_fp16_and_infinite_projections(act):
    """Rows saturate at fp16's largest as the other path's; infinite gates and halves as the activations in fp32 have them."""
    blk = _block(128, 64, 7, 2, 4, 64, act, "topk_softmax", True)
    x = torch.randn((9, 128), device="cuda", generator=torch.Generator(device="cuda").manual_seed(0)).bfloat16()
    x[2, :5], x[3, 7] = 1e5, -3e38
    idx, scores = torch.arange(18, device="cuda").view(9, 2) % 7, torch.full((9, 2), 0.5, device="cuda")
    inf = float("inf")
    for e, (g, u) in enumerate([(inf, 0), (-inf, 0), (0, inf), (0, -inf), (inf, inf), (inf, -inf)]):
        blk.experts.gate_proj.bias[e, e], blk.experts.up_proj.bias[e, e] = g, u
    blk.route = lambda z: (idx, scores)  # the choices are given
    got = (blk.experts(x, idx).float() * scores[..., None]).sum(1)
    want = _by_parts(blk, x, idx, scores)
    for r in range(9):  # NaN (an infinite gate's, times nought) becomes a finite operand of the way out on both ways
        assert torch.isfinite(want[r]).all() and (got[r] - want[r]).norm() <= 2**-6 * want[r].norm()


def test_rows_of_another_stream_and_passes_that_repeat():
    blk = _block(320, 192, 7, 2, 4, 64, "gpt_oss", "topk_softmax", True)
    x = torch.randn((200, 320), device="cuda").bfloat16()
    want = blk(x)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        rows = torch.zeros((4096, 4096), device="cuda")
        for _ in range(8):
            rows = rows @ rows  # the rows are late
        late = x + rows[0, 0].bfloat16()
        got = [blk(late) for _ in range(3)]
    other = blk(x)  # meanwhile
    torch.cuda.synchronize()
    assert torch.equal(other, want) and all(torch.equal(y, want) for y in got)


@pytest.mark.parametrize("tokens,most", [(16, 0.0009), (32, 0.0009), (64, 0.0014)])
def test_long_sums_round_as_those_of_a_split_product(tokens, most):
    """Share of results that are not the rounding of the float64 sum over the same fp16 weights, K = 4096: 0.17 to 0.19 % for one chain
    in the accumulator, 0.05 to 0.06 for four, 0.10 for two; a million results leave a tenth of that to chance."""
    from vllm_metal_b200.metal import get_ops
    from vllm_metal_b200.quant.switch_linear import QuantizedSwitchLinear

    ops, g = get_ops(), torch.Generator(device="cuda").manual_seed(0)
    m = QuantizedSwitchLinear.from_dense(torch.randn((1, 1536, 4096), device="cuda", generator=g) / 64, None, 64, 4, torch.bfloat16)
    q = (m.weight[0].to(torch.int64) & 0xFFFFFFFF).unsqueeze(-1) >> (torch.arange(8, device="cuda") * 4) & 15
    s, b = (t[0].half().double().unsqueeze(-1) for t in (m.scales, m.biases))
    w = (q.flatten(-2).unflatten(-1, (-1, 64)).double() * s + b).half().double().flatten(-2)  # rounded once, as the kernel does
    off = total = 0
    for _ in range(2**20 // (1536 * tokens) + 1):
        x = torch.randn((tokens, 4096), device="cuda", generator=g).bfloat16()
        plan = ops.expert_plan(torch.zeros((tokens, 1), dtype=torch.int32, device="cuda"), 1,
                               ops.qexpert_tile_rows(tokens, 1, 1, 1536, 4096, 64, False))
        got = ops.qexpert_product(ops.qexpert_rows(x, plan[0], 1, 4), m, plan)
        off += int((got != (x.double() @ w.T).bfloat16()).sum())
        total += got.numel()
    assert off <= most * total
