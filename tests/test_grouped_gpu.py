"""Products with one weight matrix per group, bfloat16, at the edges of their two tensor-core kernels (groups of few rows, groups
of about a hundred and more), against 64-bit products of the same operands."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from pyre_b200.kernels import build, ops
    build.ensure_built(["grouped"])
    return ops


def agree(got, x, w, what):
    """x, w: 64-bit rows and weights of one group.  fp32 sums of K exact products, a rounding per 16 of them and one per addition of such a
    group of 16 (the tensor core may cut instead of round: one more bit), then the result's own rounding."""
    want, size = x @ w.T, x.abs() @ w.abs().T
    bound = (x.shape[1] / 16 + 16) * 2.0 ** -23 * size
    if got.dtype == torch.bfloat16:
        bound = bound + 2.0 ** -8 * want.abs()
    bad = (got.double() - want).abs() > bound
    assert not bad.any(), f"{what}: {int(bad.sum())} of {bad.numel()} entries, the first at {bad.nonzero()[0].tolist()}"


# rows per group: none, one, the ends of the 16-row pieces and 64-row tiles; and of the 128-row tiles.  33 and 70 groups: more than the
# lanes that look for a tile's group
FEW = [[0, 1, 16, 17], [3], [0] * 31 + [2, 65], [1, 0, 0, 48, 64, 33], [(7 * i) % 5 for i in range(70)]]
MANY = [[128, 129, 0, 200], [96], [1, 300], [127, 255, 256]]


@pytest.mark.parametrize("rows", FEW + MANY, ids=lambda r: f"{len(r)}g{sum(r)}")
@pytest.mark.parametrize("N,K", [(8, 8), (130, 72), (63, 64), (129, 200), (256, 520)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_product_per_expert(ops, rows, N, K, out_dtype):
    g = torch.Generator(device="cuda").manual_seed(N + K + len(rows))
    G, places = len(rows), sum(rows)
    offsets = torch.tensor([0] + rows).cumsum(0).to(torch.int32).cuda()
    x = torch.randn(40, K, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(G, N, K, device="cuda", generator=g).to(torch.bfloat16)
    src = torch.randint(0, 40, (places + 5,), device="cuda", generator=g).to(torch.int32)
    got = ops.expert_linear(x, w, offsets, src, places, out_dtype)
    own = torch.randn(places + 3, K, device="cuda", generator=g).to(torch.bfloat16)
    got_own = ops.expert_linear(own, w, offsets, None, places, out_dtype)
    ops.check_device_errors()
    lo = 0
    for e, n in enumerate(rows):
        agree(got[lo:lo + n], x[src[lo:lo + n].long()].double(), w[e].double(), f"gathered, group {e}")
        agree(got_own[lo:lo + n], own[lo:lo + n].double(), w[e].double(), f"in place, group {e}")
        lo += n


@pytest.mark.parametrize("T", [1, 17, 64, 65, 95, 96, 129, 260])
@pytest.mark.parametrize("H,N,K", [(3, 256, 128), (2, 128, 256), (5, 40, 24), (1, 130, 136)])
def test_product_per_head(ops, T, H, N, K):
    g = torch.Generator(device="cuda").manual_seed(T + N)
    wide = torch.randn(T, H * (K + 16) + 8, device="cuda", generator=g).to(torch.bfloat16)
    x = wide[:, 8:].view(T, H, K + 16)[:, :, :K]
    w = torch.randn(H, N, K, device="cuda", generator=g).to(torch.bfloat16)
    out = torch.full((T, H, N + 8), float("nan"), device="cuda", dtype=torch.bfloat16)
    ops.headwise_linear(x, w, out=out)
    ops.check_device_errors()
    assert torch.isnan(out[:, :, N:]).all(), "columns beyond a head's result stay"
    for h in range(H):
        agree(out[:, h, :N], x[:, h].double(), w[h].double(), f"head {h}")


@pytest.mark.parametrize("G,per", [(4, 2), (4, 3), (5, 16), (5, 17), (3, 95), (3, 96)])
def test_where_the_kernels_take_over(ops, G, per):
    """The rows per group at which another kernel takes a product, all of them in one group, so that it takes many tiles."""
    g = torch.Generator(device="cuda").manual_seed(G * per)
    places, N, K = G * per, 70, 136
    offsets = torch.tensor([0] + [0] * (G - 1) + [places], dtype=torch.int32, device="cuda")
    x = torch.randn(places, K, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(G, N, K, device="cuda", generator=g).to(torch.bfloat16)
    got = ops.expert_linear(x, w, offsets, None, places, torch.float32)
    ops.check_device_errors()
    agree(got, x.double(), w[G - 1].double(), "the last group")
