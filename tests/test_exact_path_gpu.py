"""The kernels of the 32-bit path at the edges of their variants, against 64-bit evaluations: the product by number of rows
(weight stream, tiles, tiles with a CTA per chain, scalar loads) and the exact attention by how rows share a CTA."""

import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


@pytest.fixture(scope="module")
def ops():
    from pyre_b200.kernels import build, ops
    build.ensure_built(["gemm_f32", "attention_generic"])
    return ops


# rows: the ends of the weight stream's variants (4, 8, 16, 32) and of the tiles (64); K: part of a run, of a stage of 256, the
# first K whose chains may go to the CTAs of a cluster (1024) and its neighbours; N: a lone feature, ragged tiles
@pytest.mark.parametrize("N,K", [(1, 4), (15, 36), (65, 252), (17, 260), (130, 1020), (130, 1024), (200, 1028), (64, 2100), (33, 101)])
@pytest.mark.parametrize("M", [1, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 150])
def test_product_at_the_edges(ops, M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M * 1000 + K)
    wide = torch.full((M, K + 8), float("nan"), device="cuda")
    wide[:, :K] = torch.randn(M, K, device="cuda", generator=g)
    a = wide[:, :K]                                 # rows further apart than they are long
    w = torch.randn(N, K, device="cuda", generator=g)
    bias = torch.randn(N, device="cuda", generator=g)
    out = torch.full((M + 1, N), float("nan"), device="cuda")
    got = ops.sgemm_nt(a, w, out=out[:M])
    want, size = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
    # a product term passes through at most 16 fused additions of its run, 1 of the run's halves, K / 256 + 1 of its chain, 8 of the chains
    terms = 16 + 1 + K // 256 + 2 + 8
    assert ((got.double() - want).abs() <= terms * EPS * size).all()
    assert torch.isnan(out[M]).all(), "nothing is stored past the last row"
    assert torch.equal(ops.sgemm_nt(a, w, bias), got + bias)
    for r in {0, M // 2, M - 1}:
        assert torch.equal(ops.sgemm_nt(a[r:r + 1].contiguous(), w), got[r:r + 1]), "a row's bits do not depend on the other rows"
    # rows that are not on 16-byte boundaries take the scalar kernel: the same bits
    odd = torch.empty(M, K + 1, device="cuda")[:, 1:].copy_(a)
    assert torch.equal(ops.sgemm_nt(odd, w), got)


def reference(q, cache, table, seq, pos, nh, nkv, hd, scale, window, keep, sink):
    page = cache.shape[3]
    out = torch.empty(len(seq), nh, hd, dtype=torch.float64, device="cuda")
    for t in range(len(seq)):
        p = int(pos[t])
        j = torch.arange(p + 1, device="cuda")
        if window:
            j = j[(j > p - window) | (j < keep)]
        rows = cache[table[int(seq[t])][j // page].long(), :, :, j % page].double()      # [keys, 2, nkv, hd]
        k, v = (rows[:, i].repeat_interleave(nh // nkv, dim=1) for i in range(2))
        s = torch.einsum("hd,khd->hk", q[t].double().view(nh, hd), k) * scale
        s = torch.cat([s, sink.double()[:, None]], -1)
        out[t] = torch.einsum("hk,khd->hd", torch.softmax(s, -1)[:, :-1], v)
    return out.view(len(seq), -1)


# query heads per key/value head: one, some that fill a CTA's rows with several tokens, an odd count, more than the rows
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,hd,page,window,keep", [(2, 2, 16, 16, None, 0), (6, 2, 48, 8, 40, 0), (4, 2, 128, 16, 70, 9), (7, 1, 128, 16, None, 0),
                                                        (9, 1, 64, 4, 33, 3), (16, 1, 32, 16, None, 0), (4, 2, 144, 16, 50, 0), (10, 2, 256, 16, None, 0)])
def test_attention_however_rows_share_a_cta(ops, dtype, nh, nkv, hd, page, window, keep):
    """Many tokens of several sequences (portions of prompts, short ones among them, and decoded tokens): with two sequences in
    one CTA, with one token per CTA, token by token: the same bits, and the values of an evaluation in 64 bits.  Keys that a row does
    not see hold infinities."""
    g = torch.Generator(device="cuda").manual_seed(nh * 100 + hd)
    lens, new = [301, 190, 6, 33, 64], [150, 190, 3, 33, 1]
    width = max(-(-n // page) for n in lens)
    n_pages = sum(-(-n // page) for n in lens) + 1
    order = torch.randperm(n_pages, generator=torch.Generator().manual_seed(3)).tolist()
    table = torch.full((len(lens), width), -1, dtype=torch.int32)
    cache = torch.full((n_pages, 2, nkv, page, hd), float("inf"), device="cuda")
    for s, n in enumerate(lens):
        for lp in range(-(-n // page)):
            table[s, lp] = order.pop()
            used = min(page, n - lp * page)
            cache[int(table[s, lp]), :, :, :used] = torch.randn(2, nkv, used, hd, device="cuda", generator=g)
    cache = cache.to(dtype)
    table = table.cuda()
    seq = torch.tensor(sum(([s] * n for s, n in enumerate(new)), []), dtype=torch.int32, device="cuda")
    pos = torch.tensor(sum((list(range(n - k, n)) for n, k in zip(lens, new)), []), dtype=torch.int32, device="cuda")
    T = len(seq)
    q = torch.randn(T, nh * hd, device="cuda", generator=g).to(dtype)
    sink = torch.randn(nh, device="cuda", generator=g)
    scale = hd ** -0.5

    def run(rows):
        return ops.paged_attention_generic(q[rows].contiguous(), cache, table, seq[rows], pos[rows], nh, nkv, hd, scale, window, sink=sink, keep_first=keep)
    whole = run(slice(0, T))
    want = reference(q, cache, table, seq, pos, nh, nkv, hd, scale, window, keep, sink)
    # fp32: scores and weighted sums of numbers around one, sums of up to a few hundred terms; bfloat16 results are rounded to 2^-9
    err = (whole.double() - want).abs()
    assert (err <= (2e-6 if dtype == torch.float32 else 2.0 ** -8 * want.abs() + 1e-5)).all(), float(err.max())
    for cut in ([0, 7, 150, 151, 340, 343, 376, T], [0, 2, 3, 4, 5, 200, 345, T]):
        parts = torch.cat([run(slice(lo, hi)) for lo, hi in zip(cut, cut[1:])])
        assert torch.equal(parts, whole), "a row's bits do not depend on the rows beside it"
    # the first token that sees nothing but itself and what is before it: later keys of its chunk may hold anything
    later = cache.clone()
    s, p = 1, 10                                    # row 150 + 10: position 10 of the second sequence
    for j in range(p + 1, 32):
        later[int(table[s, j // page]), 1, :, j % page] = float("inf")
    got = ops.paged_attention_generic(q, later, table, seq, pos, nh, nkv, hd, scale, window, sink=sink, keep_first=keep)
    assert torch.equal(got[150:150 + p + 1], whole[150:150 + p + 1])


@pytest.mark.parametrize("nh,nkv,hd", [(2, 2, 32), (6, 2, 64), (7, 1, 16)])
@pytest.mark.parametrize("window,keep", [(None, 0), (40, 5)])
def test_attention_of_tokens_without_a_position(ops, nh, nkv, hd, window, keep):
    """A token at a negative position sees no key: nothing is read for it, with a sink its result is zero (the sink takes all of the
    weight), and the tokens that share its CTA have the bits that they have without it."""
    g = torch.Generator(device="cuda").manual_seed(nh)
    T, page = 300, 16
    table = torch.arange(-(-T // page), dtype=torch.int32, device="cuda").view(1, -1).repeat(2, 1)
    cache = torch.randn(table.shape[1], 2, nkv, page, hd, device="cuda", generator=g)
    cache[0, 1, :, 3] = float("inf")                # a value that a row without keys must not touch
    pos = torch.arange(T, dtype=torch.int32, device="cuda")
    pos[[0, 5, 6, 40]] = torch.tensor([-1, -1, -7, -2147483648], dtype=torch.int32, device="cuda")
    pos[64:96] = -1                                 # whole CTAs of them
    seq = (torch.arange(T, device="cuda") >= 200).to(torch.int32)
    q, sink = torch.randn(T, nh * hd, device="cuda", generator=g), torch.randn(nh, device="cuda", generator=g)

    def run(rows):
        return ops.paged_attention_generic(q[rows].contiguous(), cache, table, seq[rows], pos[rows], nh, nkv, hd, hd ** -0.5, window, sink=sink, keep_first=keep)
    got, none = run(slice(0, T)), pos < 0
    assert torch.equal(got[none], torch.zeros_like(got[none]))
    keep_rows = (~none).nonzero()[:, 0]
    # bytes, since the infinite value makes some results infinite or not a number
    assert torch.equal(got[keep_rows].view(torch.int32), run(keep_rows).view(torch.int32))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,hd", [(2, 2, 32), (4, 1, 144), (7, 1, 16)])
@pytest.mark.parametrize("low", [[32], [33, 34, 35], list(range(64, 96)), list(range(32)), list(range(96, 101)), list(range(40))])
def test_attention_with_scores_of_minus_infinity(ops, dtype, nh, nkv, hd, low):
    """Keys whose score overflows to minus infinity have no weight, also where they are all that a chunk of 32 keys holds; without any
    other key a row is not a number, or zero where a sink takes all of the weight."""
    g = torch.Generator(device="cuda").manual_seed(hd + len(low))
    page, T = 16, 101
    table = torch.randperm(-(-T // page), generator=torch.Generator().manual_seed(1)).to(torch.int32).cuda()[None]
    cache = torch.randn(table.shape[1], 2, nkv, page, hd, device="cuda", generator=g).to(dtype)
    cache[:, 0, :, :, 0] = 0
    for j in low:
        cache[int(table[0, j // page]), 0, :, j % page, 0] = -1e30
    q = torch.randn(T, nh * hd, device="cuda", generator=g).to(dtype)
    q[:, ::hd] = 1e30
    pos, seq = torch.arange(T, dtype=torch.int32, device="cuda"), torch.zeros(T, dtype=torch.int32, device="cuda")
    none = torch.tensor([all(j in low for j in range(p + 1)) for p in range(T)], device="cuda")
    for sink in (torch.full((nh,), float("-inf"), device="cuda"), torch.zeros(nh, device="cuda")):
        got = ops.paged_attention_generic(q, cache, table, seq, pos, nh, nkv, hd, hd ** -0.5, sink=sink)
        assert torch.isnan(got[none]).all() if sink[0] < 0 else (got[none] == 0).all()
        want = reference(q, cache, table, seq, pos, nh, nkv, hd, hd ** -0.5, None, 0, sink)
        err = (got.double() - want).abs()[~none]
        assert (err <= (2e-6 if dtype == torch.float32 else 2.0 ** -8 * want.abs()[~none] + 1e-5)).all(), float(err.max())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,hd", [(2, 2, 16), (6, 2, 48), (7, 1, 128), (5, 5, 128), (3, 1, 144), (8, 4, 256)])
@pytest.mark.parametrize("most", [16, 32, 33, 64, 65, 128, 129, 256])
@pytest.mark.parametrize("tokens", ["decoded", "few", "many"])
def test_attention_of_short_tables(ops, dtype, nh, nkv, hd, most, tokens):
    """A table that holds one to eight chunks of keys lets fewer warps share a row; one token, or hundreds of short sequences: the bits are
    those that a wide table gives, and near an evaluation in 64 bits."""
    g = torch.Generator(device="cuda").manual_seed(nh + hd + most)
    page, n_seqs = 16, 1 if tokens == "decoded" else 3 if tokens == "few" else 300
    width = -(-most // page)
    table = torch.randint(0, 40, (n_seqs, width), generator=torch.Generator().manual_seed(most)).to(torch.int32).cuda()
    wide = torch.cat([table, torch.full((n_seqs, 30), -1, dtype=torch.int32, device="cuda")], 1)
    cache = torch.randn(40, 2, nkv, page, hd, device="cuda", generator=g).to(dtype)
    seq = torch.arange(n_seqs, dtype=torch.int32, device="cuda")
    pos = torch.randint(0, most, (n_seqs,), device="cuda", generator=g).to(torch.int32)
    pos[0] = most - 1
    if tokens == "few":      # a portion beside decoded tokens
        seq = torch.cat([seq, torch.full((min(most, 50),), 2, dtype=torch.int32, device="cuda")])
        pos = torch.cat([pos, torch.arange(min(most, 50), dtype=torch.int32, device="cuda")])
    q = torch.randn(len(seq), nh * hd, device="cuda", generator=g).to(dtype)
    sink = torch.randn(nh, device="cuda", generator=g)
    for window, keep in ((None, 0), (20, 3)):
        got = ops.paged_attention_generic(q, cache, table, seq, pos, nh, nkv, hd, hd ** -0.5, window, sink=sink, keep_first=keep)
        assert torch.equal(got, ops.paged_attention_generic(q, cache, wide, seq, pos, nh, nkv, hd, hd ** -0.5, window, sink=sink, keep_first=keep))
        some = slice(0, 60)
        want = reference(q[some], cache, table, seq[some], pos[some], nh, nkv, hd, hd ** -0.5, window, keep, sink)
        err = (got[some].double() - want).abs()
        assert (err <= (2e-6 if dtype == torch.float32 else 2.0 ** -8 * want.abs() + 1e-5)).all(), float(err.max())


@pytest.mark.parametrize("K", [3, 4])
def test_product_of_very_many_rows(ops, K):
    """More tiles of rows than the second dimension of a grid holds, from rows on and off 16-byte boundaries."""
    M, N = 64 * 65535 + 70, 3
    g = torch.Generator(device="cuda").manual_seed(K)
    a, w = torch.randn(M, K, device="cuda", generator=g), torch.randn(N, K, device="cuda", generator=g)
    got = ops.sgemm_nt(a, w)
    want, size = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
    assert ((got.double() - want).abs() <= 4 * EPS * size).all()      # two additions of each of two chains, one of the chains


@pytest.mark.parametrize("nh,nkv", [(65541, 65541), (65537 * 3, 1)])
def test_attention_of_very_many_heads(ops, nh, nkv):
    """More groups of heads than the second dimension of a grid holds."""
    g = torch.Generator(device="cuda").manual_seed(nkv)
    hd, page = 16, 4
    cache = torch.randn(2, 2, nkv, page, hd, device="cuda", generator=g)
    table = torch.tensor([[1, 0], [0, 1]], dtype=torch.int32, device="cuda")
    seq, pos = (torch.tensor(v, dtype=torch.int32, device="cuda") for v in ([0, 1], [6, 2]))
    q, sink = torch.randn(2, nh * hd, device="cuda", generator=g), torch.randn(nh, device="cuda", generator=g)
    got = ops.paged_attention_generic(q, cache, table, seq, pos, nh, nkv, hd, 0.25, sink=sink)
    want = reference(q, cache, table, seq, pos, nh, nkv, hd, 0.25, None, 0, sink)
    assert ((got.double() - want).abs() <= 2e-6).all()
