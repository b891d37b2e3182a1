"""Few decode rows: partitions merged inside a cluster, against the general kernel over what the plan accepts."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("heads,kv,dim,lens,rows,window,sinks,planned", [
    (16, 8, 128, [513], 1, -1, False, 1024),          # half of the cluster beyond the row
    (16, 8, 64, [1], 1, -1, True, 512),               # one token: all but one CTA have nothing
    (4, 1, 128, [700, 3, 8000], 1, -1, True, 8192),   # the longest rows the plan takes
    (8, 2, 64, [100, 2000], 1, 128, False, 2048),     # a window shorter than the plan
    (8, 2, 128, [700, 65], 1, 1000, True, 2048),
    (8, 1, 64, [300, 17, 1000], 3, -1, False, 1024),  # verification windows
    (32, 2, 128, [129], 2, 100, True, 512),
    (128, 128, 64, [200], 1, -1, False, 256),         # as many heads as SMs: clusters of one, the plan without them
])
def test_cluster_merge(heads, kv, dim, lens, rows, window, sinks, planned, dtype):
    from vllm_metal_b200.metal import get_ops

    ops, g = get_ops(), torch.Generator(device="cuda").manual_seed(sum(lens))
    lens = [max(n, rows) for n in lens]
    pages = sum(-(-n // 16) for n in lens)
    width = -(-planned // 16)
    table = torch.zeros((len(lens), width), dtype=torch.int32, device="cuda")
    order, at = torch.randperm(pages, generator=g, device="cuda").int(), 0
    for i, n in enumerate(lens):
        table[i, :-(-n // 16)] = order[at:at - (-n // 16)]
        at -= -n // 16
    kc, vc = (torch.randn((pages, 16, kv, dim), device="cuda", generator=g).to(dtype) for _ in range(2))
    q = torch.randn((len(lens) * rows, heads, dim), device="cuda", generator=g).to(dtype)
    sl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    cu = torch.arange(len(lens) + 1, dtype=torch.int32, device="cuda") * rows
    sk = torch.randn(heads, device="cuda", generator=g) if sinks else None
    outs = []
    for kernel in (0, 1):
        out = torch.full_like(q, float("nan"))
        ops.paged_attention_primitive(q, kc, vc, kv, dim**-0.5, 0.0, table, sl, cu, 16, planned, window, out, sinks=sk,
                                      window_seqlen_q=rows, _kernel=kernel)
        outs.append(out.float())
    # weights and results round to 8 (bf16) or 11 bits; the general kernel keeps weights in 32
    assert torch.isfinite(outs[0]).all()
    eps = 2.0**-8 if dtype == torch.bfloat16 else 2.0**-11
    assert (outs[0] - outs[1]).norm() <= 2 * eps * outs[1].norm()
