"""The attention of a mixed step does not depend on the order of its entries: decoded tokens in front of a portion go to their kernel
as a batch of their own, in any other order with the whole step."""

import numpy as np
import pytest
import torch

import standins
from pyre_b200.engine.context import StepContext


@pytest.mark.parametrize("lens", [[1, 1, 1, 70], [1, 70, 1], [70, 1, 1], [5, 1, 63, 64, 130], [3, 3, 90], [64, 2], [1, 1], [80, 64], [2, 40, 65, 3]])
@pytest.mark.parametrize("window", [None, 33])
def test_order_of_entries(monkeypatch, lens, window):
    from pyre_b200.kernels import ops
    seen = []
    standins.install_bf16(monkeypatch)
    stand_in = ops.paged_attention_mma

    def watched(q, *a, **k):
        seen.append(q.shape[0])
        return stand_in(q, *a, **k)
    monkeypatch.setattr(ops, "paged_attention_mma", watched)
    nh, nkv, hd, page = 4, 2, 64, 16
    g = torch.Generator().manual_seed(sum(lens))
    starts = [17 * i + 3 for i in range(len(lens))]
    width = max(-(-(s + n) // page) for s, n in zip(starts, lens))
    table = torch.randperm(len(lens) * width, generator=g).to(torch.int32).view(len(lens), width)
    cache = torch.randn(len(lens) * width, 2, nkv, page, hd, generator=g).to(torch.bfloat16)
    q = [torch.randn(n, nh * hd, generator=g).to(torch.bfloat16) for n in lens]

    def run(order):
        cu = np.concatenate([[0], np.cumsum([lens[e] for e in order])]).astype(np.int32)
        pos = torch.cat([torch.arange(starts[e], starts[e] + lens[e]) for e in order]).to(torch.int32)
        z = torch.zeros(int(cu[-1]), dtype=torch.int32)
        ctx = StepContext(dtype=torch.bfloat16, device=torch.device("cpu"), num_tokens=int(cu[-1]), num_seqs=len(order), num_logit_rows=0,
                          token_ids=z, positions=pos, seq_of_token=z, cu_seqlens=torch.from_numpy(cu), logit_rows=z[:0],
                          cu_seqlens_host=cu, start_pos_host=np.asarray([starts[e] for e in order]))
        out = ops.paged_attention_bf16(ctx, torch.cat([q[e] for e in order]), cache, table[list(order)].contiguous(), nh, nkv, hd, hd ** -0.5, window)
        return {e: out[cu[i]:cu[i + 1]] for i, e in enumerate(order)}
    mixed = run(range(len(lens)))
    by_length = run(sorted(range(len(lens)), key=lambda e: lens[e]))
    for e in range(len(lens)):
        assert torch.equal(mixed[e], by_length[e]), f"entry {e} of {lens[e]} tokens"
    short = sum(n for n in lens if n < 64)
    if short:
        assert seen[-1] == short, "short entries in front are a batch of their own"
