"""Few decode rows: partitions merged inside a cluster, bit for bit as by the merge launch."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("heads,kv,dim,lens,rows,window,sinks,planned", [
    (16, 8, 128, [513], 1, -1, False, 1024),          # one token of the second partition
    (16, 8, 64, [1], 1, -1, True, 1536),              # one token: all but one CTA have nothing; a cluster of 3
    (4, 1, 128, [700, 3, 4000], 1, -1, True, 4096),   # a cluster of 8
    (8, 2, 64, [100, 2000], 1, 1500, False, 2048),    # a window shorter than the plan: 3 partitions of 512 (700 would be one of 704)
    (8, 2, 128, [1700, 65], 1, 1000, True, 2048),
    (8, 1, 64, [300, 17, 1000], 3, -1, False, 1024),  # verification windows, rows that end before a partition
    (32, 2, 128, [1029], 2, 1000, True, 1536),
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
    before = ops.launches
    for force in (0, -(-planned // 512)):
        out = torch.full_like(q, float("nan"))
        ops.paged_attention_primitive(q, kc, vc, kv, dim**-0.5, 0.0, table, sl, cu, 16, planned, window, out, sinks=sk,
                                      window_seqlen_q=rows, _force_partitions=force)
        outs.append(out)
    assert ops.launches - before == 3  # one, and one with a merge
    assert torch.isfinite(outs[0]).all() and torch.equal(outs[0], outs[1])
