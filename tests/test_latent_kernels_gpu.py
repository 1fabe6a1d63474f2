"""Kernels around the latent attention at the edges of their variants: shares of the keys put together, and norms of latents by how
many columns a thread holds, against 64-bit evaluations."""

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


# columns that a thread of 256 holds in its first piece of four (up to 1,024; one by one: 256), in its second, up to its fourth, and in the
# loop after them; multiples of four from aligned columns, and neither
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("q_rank,rank,col,parts", [(1024, 260, 8, 0), (1536, 512, 4, 16), (4200, 1100, 8, 0), (260, 4200, 0, 3), (8, 40, 4, 5), (0, 512, 4, 0),
                                                   (257, 1101, 1, 0), (1100, 261, 3, 2), (33, 4201, 2, 0)])
def test_norms_of_latents_of_any_width(ops, dtype, q_rank, rank, col, parts):
    """Query latent, cached row and rotated queries from one projection row, one token to many: each against 64 bits, and the same
    bits for a token whatever tokens are beside it."""
    nh, dq, rope, rot = 3, 12, 8, 8
    T = 700      # more than two tokens per SM: a block then takes all pieces of a token
    q_col, c_col = col, col + q_rank
    qh_col = c_col + rank + rope
    W = -(-(qh_col + nh * (dq + rope)) // 4) * 4 + (0 if col % 4 == 0 else 1)
    row = -(-(rank + rope) // 16) * 16
    g = torch.Generator(device="cuda").manual_seed(q_rank + rank)
    proj = torch.randn(max(parts, 1), T, W, device="cuda", generator=g)
    if not parts:
        proj = proj.to(dtype)
    full = proj.double().sum(0)
    wq, wc = (torch.randn(n, device="cuda", generator=g) for n in (max(q_rank, 1), rank))
    cos, sin = (torch.rand(T, rot // 2, device="cuda", generator=g) for _ in range(2))
    slots = torch.randperm(T + 9, device="cuda", generator=g)[:T].to(torch.int32)

    def run(rows):
        n = len(range(T)[rows])
        cache = torch.full((-(-(T + 9) // 16), 1, 1, 16, row), 7.0, dtype=dtype, device="cuda")
        qa = torch.full((n, nh, row), 5.0, dtype=dtype, device="cuda")
        piece = proj[:, rows].contiguous()
        cq = ops.latent_prepare(ops.PartialSums(piece, dtype) if parts else piece[0], q_col, q_rank, c_col, rank, rope, rot, wq if q_rank else None, wc, 1e-5,
                                cos[rows].contiguous(), sin[rows].contiguous(), cache, slots[rows].contiguous(), 16, dtype, q_out=qa, qh_col=qh_col, dq=dq)
        return cq, cache.view(-1, row)[slots[rows].long()], qa

    def near(got, want, what):
        # fp32: the sum of squares passes through at most 17 additions of a thread, 15 of the block (half of its error in the root), then four
        # roundings and the partial sums' own; bfloat16 results are rounded to 2^-9 of themselves
        tol = (16 + 4 + parts) * 2.0 ** -24 + (0 if dtype == torch.float32 else 2.0 ** -8)
        bad = (got.double() - want).abs() > tol * want.abs() + 1e-6 * (1 + parts)
        assert not bad.any(), f"{what}: {int(bad.sum())} entries"

    def norm(v, w):
        return v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5) * w.double()

    def turn(v):      # neighbouring pairs by the token's angles
        c, s = (t.double().view((T,) + (1,) * (v.dim() - 2) + (-1,)) for t in (cos, sin))
        return torch.stack([v[..., 0::2] * c - v[..., 1::2] * s, v[..., 1::2] * c + v[..., 0::2] * s], -1).flatten(-2)
    cq, cached, qa = run(slice(0, T))
    if q_rank:
        near(cq, norm(full[:, q_col:q_col + q_rank], wq), "query latent")
    near(cached[:, :rank], norm(full[:, c_col:c_col + rank], wc), "latent")
    near(cached[:, rank:rank + rope], turn(full[:, c_col + rank:qh_col]), "key part")
    near(qa[..., rank:rank + rope], turn(full[:, qh_col:qh_col + nh * (dq + rope)].view(T, nh, dq + rope)[..., dq:]), "rotated queries")
    assert (cached[:, rank + rope:] == 0).all() and (qa[..., rank + rope:] == 0).all() and (qa[..., :rank] == 5).all()
    for rows in (slice(0, 1), slice(5, 9), slice(40, 340)):
        for whole, part in zip((cq, cached, qa), run(rows)):
            assert whole is None or torch.equal(part, whole[rows])
