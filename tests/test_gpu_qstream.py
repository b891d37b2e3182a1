"""GPU parity of the persistent stream-K quantized GEMM (csrc/qgemm_stream.cu) vs the oracle.

Reference anchors: mx.quantized_matmul as called from gguf/mlx_native.py:212-222 and
nn.QuantizedLinear (attention/impls/sdpa.py:297-343,739); SwiGLU fusion = compiled_mlp.py:1-22.
Bar: 2e-2 max-abs + 1e-2 relative (bf16 outputs); the integer part of the streaming
layout round-trips bit-exactly; results are identical for every persistent-grid size that cuts the
super-tiles differently (the finisher adds partials in k order, never in arrival order).
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import affine_quant as oq
from oracle._numeric import round_to
from oracle.decoder import silu_mul as oracle_silu_mul

from .gpu_helpers import TORCH_DT, assert_close, to_np

pytestmark = pytest.mark.gpu


def _quantized(n, k, bits, group, dtype="bfloat16", seed=0, std=0.02):
    rng = np.random.default_rng(seed)
    w = round_to((rng.standard_normal((n, k)) * std).astype(np.float32), dtype)
    wq, s, b = oq.quantize(w, group, bits, dtype)
    tdt = TORCH_DT[dtype]
    return (wq, s, b, torch.from_numpy(wq.view(np.int32)).cuda(), torch.from_numpy(s).to(tdt).cuda(),
            torch.from_numpy(b).to(tdt).cuda())


@pytest.mark.parametrize("bits,group", [(4, 64), (4, 32), (4, 128), (8, 64), (8, 32), (8, 128)])
@pytest.mark.parametrize("n,k", [(320, 1024), (256, 128), (700, 2880), (1024, 4096)])
def test_blob_round_trip_bit_exact(ops, bits, group, n, k):
    if k % group:
        pytest.skip("K not a multiple of the group")
    g = torch.Generator(device="cuda").manual_seed(n + k + bits)
    w = torch.randint(-2**31, 2**31 - 1, (n, k * bits // 32), dtype=torch.int64, device="cuda", generator=g).to(torch.int32)
    s = (torch.rand((n, k // group), device="cuda", generator=g) * 0.01 + 0.001).bfloat16()
    b = (-8 * s.float()).bfloat16()
    for swiglu in (False, True):
        blob = ops.qstream_prepack(w, s, b, group, bits, swiglu)
        assert torch.equal(ops.qstream_unpack(blob, n, k, group, bits, swiglu), w)


@pytest.mark.parametrize("m", [1, 3, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("bits,group", [(4, 64), (4, 32), (4, 128), (8, 64), (8, 32), (8, 128)])
def test_qstream_vs_oracle(ops, m, bits, group):
    n, k = 320, 1024
    wq, s, b, tw, ts, tb = _quantized(n, k, bits, group, seed=m)
    x = round_to(np.random.default_rng(m + 1).standard_normal((m, k)).astype(np.float32), "bfloat16")
    bias = round_to(np.random.default_rng(7).standard_normal(n).astype(np.float32), "bfloat16")
    blob = ops.qstream_prepack(tw, ts, tb, group, bits)
    got = ops.qstream_linear(torch.from_numpy(x).bfloat16().cuda(), blob, n, k, group, bits,
                             bias=torch.from_numpy(bias).bfloat16().cuda())
    want = oq.quantized_matmul(x, wq, s, b, group, bits, bias=bias, dtype="bfloat16")
    assert got.shape == (m, n) and got.dtype == torch.bfloat16
    assert_close(got, want, "bfloat16", f"M={m}")


@pytest.mark.parametrize("n,k,bits,group,m", [
    (4096, 4096, 4, 64, 64), (6144, 4096, 4, 64, 64), (4096, 14336, 4, 64, 64), (2880, 2880, 4, 64, 32),
    (136, 192, 4, 64, 5), (1000, 2048, 4, 128, 33), (384, 1536, 8, 64, 64), (5120, 25600, 8, 64, 64),
    (8192, 28672, 4, 64, 16), (151936, 1024, 4, 64, 1), (128, 2880, 4, 32, 8), (1280, 8192, 4, 64, 16)])
def test_qstream_model_shapes(ops, n, k, bits, group, m):
    """Projection shapes of the served models incl. ragged N (not a multiple of 256), K = 2880 = 22.5 slabs,
    the long-K cases (25600 int8, 28672 int4) and the Qwen3-0.6B tied head; oracle on a row subset."""
    gen = torch.Generator(device="cuda").manual_seed(n + k)
    w = torch.randint(-2**31, 2**31 - 1, (n, k * bits // 32), dtype=torch.int64, device="cuda", generator=gen).to(torch.int32)
    s = (torch.rand((n, k // group), device="cuda", generator=gen) * 0.5 + 0.75) * (0.12 / (2**bits - 1))
    b = -s * 2 ** (bits - 1) * (1.0 + 0.1 * torch.randn((n, k // group), device="cuda", generator=gen))
    s, b = s.bfloat16(), b.bfloat16()
    x = torch.randn((m, k), device="cuda", generator=gen).bfloat16()
    blob = ops.qstream_prepack(w, s, b, group, bits)
    got = ops.qstream_linear(x, blob, n, k, group, bits)
    torch.cuda.synchronize()
    rows = np.sort(np.random.default_rng(k).choice(n, size=min(n, 320), replace=False))
    rows[-1] = n - 1
    rows[0] = 0
    rt = torch.from_numpy(rows).cuda()
    want = oq.quantized_matmul(to_np(x), w[rt].cpu().numpy().view(np.uint32), to_np(s[rt]), to_np(b[rt]), group, bits,
                               dtype="bfloat16")
    assert_close(got[:, rt], want, "bfloat16", f"{n}x{k} int{bits} g{group} M={m}")


@pytest.mark.parametrize("grid", [1, 2, 3, 7, 31, 64, 148])
@pytest.mark.parametrize("n,k,m", [(1024, 4096, 64), (600, 1536, 9), (2048, 512, 16)])
def test_stream_k_cuts_do_not_change_the_result(ops, grid, n, k, m):
    """Any persistent grid (= any way of cutting super-tiles between CTAs, up to 32 pieces per tile) gives
    the same bits: partials are added in k order by the finisher."""
    wq, s, b, tw, ts, tb = _quantized(n, k, 4, 64, seed=n)
    x = torch.from_numpy(round_to(np.random.default_rng(3).standard_normal((m, k)).astype(np.float32), "bfloat16")).bfloat16().cuda()
    blob = ops.qstream_prepack(tw, ts, tb, 64, 4)
    try:
        ops.set_qstream_grid(grid)
        got = ops.qstream_linear(x, blob, n, k, 64, 4)
        again = ops.qstream_linear(x, blob, n, k, 64, 4)  # counters re-armed by the finisher
        torch.cuda.synchronize()
    finally:
        ops.set_qstream_grid(0)
    want = oq.quantized_matmul(to_np(x), wq, s, b, 64, 4, dtype="bfloat16")
    assert_close(got, want, "bfloat16", f"grid={grid}")
    assert torch.equal(got, again)
    # fp32 partial sums are grouped differently per cut, so compare against the oracle, not across grids,
    # except for grid sizes that do not cut inside a tile at all
    if grid == 1:
        ops.set_qstream_grid(0)
        base = ops.qstream_linear(x, blob, n, k, 64, 4)
        assert_close(base, to_np(got), "bfloat16", "default grid vs grid=1")


@pytest.mark.parametrize("m", [1, 16, 40, 64])
@pytest.mark.parametrize("inter,k,bits,group", [(1536, 1024, 4, 64), (200, 512, 4, 32), (3584, 2048, 8, 64), (14336, 4096, 4, 64)])
def test_swiglu_epilogue_matches_unfused_and_oracle(ops, m, inter, k, bits, group):
    """gate_up with the SiLU*up epilogue == silu_mul(gate_up(x)) bit for bit (same rounding points), and
    both within tolerance of the oracle's silu_mul(matmul)."""
    n = 2 * inter
    gen = torch.Generator(device="cuda").manual_seed(inter)
    if inter <= 3584:
        wq, s, b, tw, ts, tb = _quantized(n, k, bits, group, seed=inter)
    else:
        tw = torch.randint(-2**31, 2**31 - 1, (n, k * bits // 32), dtype=torch.int64, device="cuda", generator=gen).to(torch.int32)
        ts = ((torch.rand((n, k // group), device="cuda", generator=gen) * 0.5 + 0.75) * 0.008).bfloat16()
        tb = (-8 * ts.float()).bfloat16()
        wq = s = b = None
    x = torch.randn((m, k), device="cuda", generator=gen).bfloat16()
    blob_f, blob_p = ops.qstream_prepack(tw, ts, tb, group, bits, swiglu=True), ops.qstream_prepack(tw, ts, tb, group, bits)
    try:
        ops.set_qstream_grid(1)  # no super-tile is cut: both layouts accumulate every row in plain k order
        fused1 = ops.qstream_linear(x, blob_f, n, k, group, bits, swiglu=True)
        unfused1 = ops.silu_mul(ops.qstream_linear(x, blob_p, n, k, group, bits))
        torch.cuda.synchronize()
    finally:
        ops.set_qstream_grid(0)
    assert fused1.shape == (m, inter)
    assert torch.equal(fused1, unfused1)
    fused = ops.qstream_linear(x, blob_f, n, k, group, bits, swiglu=True)  # default grid: tiles cut between CTAs
    assert_close(fused, to_np(fused1), "bfloat16", f"swiglu default grid vs grid 1, M={m}")
    if wq is not None:
        gu = oq.quantized_matmul(to_np(x), wq, s, b, group, bits, dtype="bfloat16")
        want = oracle_silu_mul(gu, "bfloat16")
        assert_close(fused, want, "bfloat16", f"swiglu M={m}")


def test_qstream_m_above_64_tiles_over_m(ops):
    wq, s, b, tw, ts, tb = _quantized(512, 1024, 4, 64, seed=11)
    x = round_to(np.random.default_rng(2).standard_normal((200, 1024)).astype(np.float32), "bfloat16")
    blob = ops.qstream_prepack(tw, ts, tb, 64, 4)
    got = ops.qstream_linear(torch.from_numpy(x).bfloat16().cuda(), blob, 512, 1024, 64, 4)
    assert_close(got, oq.quantized_matmul(x, wq, s, b, 64, 4, dtype="bfloat16"), "bfloat16", "M=200")


def test_qstream_fp16_activations_and_strides(ops):
    wq, s, b, tw, ts, tb = _quantized(192, 512, 4, 64, "float16", seed=9)
    blob = ops.qstream_prepack(tw, ts, tb, 64, 4)
    xw = torch.randn((20, 1024), device="cuda").half()
    x = xw[:, 256:768]
    yw = torch.zeros((20, 400), dtype=torch.float16, device="cuda")
    ops.qstream_linear(x, blob, 192, 512, 64, 4, out=yw[:, 8:200])
    want = oq.quantized_matmul(to_np(x), wq, s, b, 64, 4, dtype="float16")
    assert_close(yw[:, 8:200], want, "float16", "fp16 strided")
    assert (yw[:, :8] == 0).all() and (yw[:, 200:] == 0).all()


def test_qstream_inside_cuda_graph_and_pdl_chain(ops):
    """Back-to-back launches (PDL: the second kernel's weight prefetch overlaps the first) replayed
    from a CUDA graph; y of launch 1 is x of launch 2."""
    wq1, s1, b1, tw1, ts1, tb1 = _quantized(512, 256, 4, 64, seed=1)
    wq2, s2, b2, tw2, ts2, tb2 = _quantized(384, 512, 4, 64, seed=2)
    bl1, bl2 = ops.qstream_prepack(tw1, ts1, tb1, 64, 4), ops.qstream_prepack(tw2, ts2, tb2, 64, 4)
    x = torch.randn((24, 256), device="cuda").bfloat16()
    h = torch.empty((24, 512), device="cuda", dtype=torch.bfloat16)
    y = torch.empty((24, 384), device="cuda", dtype=torch.bfloat16)

    def chain():
        ops.qstream_linear(x, bl1, 512, 256, 64, 4, out=h)
        ops.qstream_linear(h, bl2, 384, 512, 64, 4, out=y)

    chain()
    torch.cuda.synchronize()
    ref = y.clone()
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            chain()
        y.zero_()
        for _ in range(5):
            g.replay()
        torch.cuda.synchronize()
    assert torch.equal(y, ref)
    h_want = oq.quantized_matmul(to_np(x), wq1, s1, b1, 64, 4, dtype="bfloat16")
    assert_close(h, h_want, "bfloat16", "chain stage 1")
