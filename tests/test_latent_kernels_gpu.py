"""Shares of the latent attention's keys put together, at the edges of the kernel's variants, against 64-bit evaluations."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from pyre_b200.kernels import build, ops
    build.ensure_built(["latent_attention"])
    return ops


def batch(lens, row, kd, seed):
    """Sequences of ``lens`` cached rows on scattered pages of 16, one decoded token each."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    width = max(-(-n // 16) for n in lens)
    n_pages = sum(-(-n // 16) for n in lens) + 2
    order = torch.randperm(n_pages, generator=torch.Generator().manual_seed(seed)).tolist()
    table = torch.full((len(lens), width), -1, dtype=torch.int32)
    pool = torch.full((n_pages, 1, 1, 16, row), float("nan"), device="cuda")
    for b, n in enumerate(lens):
        for lp in range(-(-n // 16)):
            table[b, lp] = order.pop()
            used = min(16, n - 16 * lp)
            pool[int(table[b, lp]), 0, 0, :used] = 0
            pool[int(table[b, lp]), 0, 0, :used, :kd] = torch.randn(used, kd, device="cuda", generator=g) * 0.5
    cu = torch.arange(len(lens) + 1, dtype=torch.int32, device="cuda")
    pos = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device="cuda")
    return pool.to(torch.bfloat16), table, cu, pos, g


# latents of part of a warp's 128 columns, of whole and part slices, and of a number that is no multiple of four
@pytest.mark.parametrize("nh,rank,rope", [(3, 24, 8), (5, 128, 16), (2, 260, 12), (4, 38, 10), (8, 512, 64)])
@pytest.mark.parametrize("splits", [2, 11, 16, 17, 33, 40])
@pytest.mark.parametrize("extras", [False, True])
def test_shares_put_together(ops, nh, rank, rope, splits, extras):
    """Up to forty shares, most of them without a key for the shorter sequences."""
    kd = rank + rope
    row = -(-kd // 16) * 16
    lens = [1, 31, 32, 33, 400, 1300]
    pool, table, cu, pos, g = batch(lens, row, kd, seed=rank + splits)
    qa = torch.zeros(len(lens), nh, row, dtype=torch.bfloat16, device="cuda")
    qa[..., :kd] = torch.randn(len(lens), nh, kd, device="cuda", generator=g)
    sink = torch.randn(nh, device="cuda", generator=g) if extras else None
    gate = (torch.randn(len(lens), nh + 3, device="cuda", generator=g).to(torch.bfloat16), 2) if extras else None
    scale = kd ** -0.5
    got = ops.latent_attention_mma(qa, pool, table.cuda(), cu, pos, len(lens), rank, scale, None, n_splits=splits, sink=sink, gate=gate)
    ops.check_device_errors()
    for b, n in enumerate(lens):
        rows = pool[table[b, :-(-n // 16)].long().cuda(), 0, 0].reshape(-1, row)[:n].double()
        s = qa[b].double() @ rows.T * scale
        if extras:
            s = torch.cat([s, sink.double()[:, None]], -1)
        p, gates = torch.softmax(s, -1)[:, :n], torch.sigmoid(gate[0][b, 2:2 + nh].double())[:, None] if extras else 1.0
        want, size = p @ rows[:, :rank] * gates, p @ rows[:, :rank].abs() * gates
        # probabilities in bfloat16 (2^-9 each) before the second product, the result rounded to bfloat16
        assert ((got[b].double() - want).abs() <= 2.0 ** -9 * (want.abs() + size) + 1e-5).all(), f"{n} rows"


@pytest.mark.parametrize("splits", [3, 16])
@pytest.mark.parametrize("sinks", [False, True])
def test_scores_of_minus_infinity(ops, splits, sinks):
    """A row all of whose scores are minus infinity: without a sink not a number, with one zero, whether the keys are shared out or not."""
    nh, rank, rope, row = 2, 32, 16, 48
    pool, table, cu, pos, g = batch([200, 70], row, rank + rope, seed=5)
    pool = pool.abs() + 0.125
    qa = torch.full((2, nh, row), float("-inf"), dtype=torch.bfloat16, device="cuda")
    qa[1, 1] = 0.25
    sink = torch.zeros(nh, device="cuda") if sinks else None
    whole, shared = (ops.latent_attention_mma(qa, pool, table.cuda(), cu, pos, 2, rank, 0.1, None, n_splits=n, sink=sink) for n in (1, splits))
    for got in (whole, shared):
        assert torch.isfinite(got[1, 1]).all()
        assert (got[0] == 0).all() if sinks else torch.isnan(got[0]).all()
        assert (got[1, 0] == 0).all() if sinks else torch.isnan(got[1, 0]).all()
