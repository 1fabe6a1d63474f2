"""The fixed-point product of float32 operands against an evaluation in 64 bits: tile edges in every dimension, every tile
width and split of K with the same bits, rows of any scale, rows that hold infinities or NaNs."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from pyre_b200.kernels import build, ops
    build.ensure_built(["gemm_fixed", "gemm_f32"])
    return ops


def bound(a, w, c):
    """One rounding to float; half a unit of 2^-29 of a row's leading power of two per factor; the products of byte planes 2 x 3, 3 x 2 and
    3 x 3 that are left out (K terms of at most 2^15 2^8 and 2^14 units of 2^-58)."""
    a, w = a.double(), w.double()
    ta, tw = a.abs().amax(1, keepdim=True), w.abs().amax(1, keepdim=True).t()
    steps = 2.0 ** -30 * (ta * w.abs().sum(1)[None] + a.abs().sum(1, keepdim=True) * tw)
    return 2.0 ** -24 * c.abs() + steps + 2.0 ** -34 * a.shape[1] * ta * tw + 2.0 ** -149


@pytest.mark.parametrize("M,N,K", [(1, 128, 512), (7, 129, 516), (8, 1000, 640), (9, 300, 2052), (17, 128, 3584), (33, 255, 544), (65, 384, 1000),
                                   (130, 777, 900), (200, 256, 18944), (3, 3584, 40960)])
def test_against_64_bits(ops, M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn(M, K, device="cuda", generator=g) * torch.exp2(torch.randint(-30, 30, (M, 1), device="cuda", generator=g))
    w = torch.randn(N, K, device="cuda", generator=g) * torch.exp2(torch.randint(-20, 20, (N, 1), device="cuda", generator=g))
    a[M // 2, :] = 0
    w[N // 2, ::3] *= 1e-3
    W = ops.FixedWeight(w)
    got = ops.fixed_linear(a, W)
    ops.check_device_errors()
    want = a.double() @ w.double().t()
    assert ((got.double() - want).abs() <= bound(a, w, want)).all()
    # whatever the tile, the split of K and the rows beside it: the same bits; rows off 16-byte boundaries too
    for tn, shares in [(8, 1), (16, 2), (32, 3), (48, 1), (64, 4)]:
        steps = -(-K // 32)
        if (shares - 1) * (-(-(-(-steps // shares)) // 4) * 4) >= steps:
            continue      # fewer shares than that: none may be empty
        assert torch.equal(ops.fixed_linear(a, W, (tn, shares)), got), (tn, shares)
    odd = torch.empty(M, K + 1, device="cuda")
    odd[:, :K] = a
    assert torch.equal(ops.fixed_linear(odd[:, :K], W), got)
    for r in {0, M // 2, M - 1}:
        assert torch.equal(ops.fixed_linear(a[r:r + 1], W), got[r:r + 1])
    ops.check_device_errors()


def test_rows_of_any_scale(ops):
    """Outliers, the smallest and the largest numbers: within the bound, and infinite where the result is."""
    g = torch.Generator(device="cuda").manual_seed(1)
    a, w = torch.randn(12, 1024, device="cuda", generator=g), torch.randn(256, 1024, device="cuda", generator=g)
    a[0, 5] = 3e3
    a[1] *= 1e-38
    a[2] *= 1e-44
    a[3] *= 1e37
    a[4, ::2] *= 1e-6
    w[0] *= 1e-38
    w[1] *= 1e30
    w[2, 7] = 1e6
    w[3] = 0
    got, want = ops.fixed_linear(a, ops.FixedWeight(w)).double(), a.double() @ w.double().t()
    fits = want.abs() < 3.4e38
    assert (((got - want).abs() <= bound(a, w, want)) | ~fits).all()
    assert torch.isinf(got[~fits]).all()


def test_infinities_and_nans(ops):
    """Rows without a scale give what an IEEE sum gives; the rows and features beside them keep their bits."""
    g = torch.Generator(device="cuda").manual_seed(2)
    a, w = torch.randn(20, 700, device="cuda", generator=g), torch.randn(256, 700, device="cuda", generator=g)
    clean = ops.fixed_linear(a, ops.FixedWeight(w))
    inf = float("inf")
    a[3, 5], a[4, 6], a[5, 7], a[5, 9], a[6, 11] = inf, float("nan"), -inf, inf, inf
    w[10, 11], w[12, 13], w[20, 5] = inf, float("nan"), 0
    for plan in [(0, 0), (32, 2)]:
        got, want = ops.fixed_linear(a, ops.FixedWeight(w), plan), ops.sgemm_nt(a, w)
        assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
        assert torch.equal(got[torch.isinf(got)], want[torch.isinf(want)])
        rows = [r for r in range(20) if r not in (3, 4, 5, 6)]
        cols = [c for c in range(256) if c not in (10, 12, 20)]
        assert torch.equal(got[rows][:, cols], clean[rows][:, cols])


@pytest.mark.parametrize("M,N,K,plan", [(64, 300, 40960, (0, 0)), (130, 256, 4100, (64, 1)), (40, 384, 2048, (48, 2)), (5, 700, 1024, (8, 1))])
def test_whole_tiles_without_a_scale(ops, M, N, K, plan):
    """Nothing waits for rows and features that have no scale, however long their sums take; in double precision they are nearer
    to 64 bits than any sum in 32."""
    g = torch.Generator(device="cuda").manual_seed(M)
    a, w = torch.randn(M, K, device="cuda", generator=g), torch.randn(N, K, device="cuda", generator=g)
    a[:, 3::17] = 0
    a[torch.arange(M), torch.randint(0, K // 17, (M,)) * 17 + 3] = float("inf")      # one in every row
    a[M // 2, 8] = -float("inf")
    w[N // 3, 5], w[N - 1, 3::17] = float("nan"), 0
    W = ops.FixedWeight(w)
    for x in (a, a[::3]):
        got, want = ops.fixed_linear(x, W, plan), x.double() @ w.double().t()
        ops.check_device_errors()
        assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
        assert torch.equal(got[torch.isinf(got)].double(), want[torch.isinf(want)])
    w[N // 3, 5] = 0
    w[::50, 7] = float("inf")
    a = torch.randn(M, K, device="cuda", generator=g).abs()
    got, want = ops.fixed_linear(a, ops.FixedWeight(w), plan), a.double() @ w.double().t()
    assert torch.equal(torch.isinf(got), torch.isinf(want)) and not torch.isnan(got).any()
    assert torch.equal(got[:, ::50].double(), want[:, ::50])
    ops.check_device_errors()


def digits(x):
    """The signed bytes of a 31-bit integer, the largest first."""
    out = []
    for _ in range(3):
        d = (x + 128) % 256 - 128
        out.insert(0, d)
        x = (x - d) // 256
    return [x] + out


@pytest.mark.parametrize("K", [512, 40960])
def test_the_largest_sums_of_bytes(ops, K):
    """Rows whose lower three bytes are all -128: the sums of 32 bits reach 3 K 2^14, 6 % below their limit at the longest K.  Compared with
    exact integers."""
    import numpy as np

    one, rest = 1 << 29, -0x808080
    assert digits(rest) == [0, -128, -128, -128] and digits(one) == [32, 0, 0, 0]
    a, w = torch.full((3, K), rest * 2.0 ** -29, device="cuda"), torch.full((256, K), rest * 2.0 ** -29, device="cuda")
    a[:, 5] = 1.0
    w[:, 9] = 1.0
    w[7] = -w[7]
    w[7, 9] = 1.0

    def total(rows):
        s = [0] * 5
        for x, y, times in rows:
            for i, dx in enumerate(digits(x)):
                for j, dy in enumerate(digits(y)):
                    if i + j <= 4:
                        s[i + j] += dx * dy * times
        assert max(map(abs, s)) < 1 << 31
        return sum(v << 8 * (4 - q) for q, v in enumerate(s))

    want = [float(np.float32(total([(one, x, 1), (rest, one, 1), (rest, x, K - 2)]) * 2.0 ** -42)) for x in (rest, -rest)]
    W = ops.FixedWeight(w)
    assert not (W.exponents >= ops.FIXED_NO_SCALE).any()
    for plan in [(0, 0), (64, 1)]:
        got = ops.fixed_linear(a, W, plan)
        assert (got[:, 7] == want[1]).all() and (got[:, torch.arange(256) != 7] == want[0]).all()
    ops.check_device_errors()


@pytest.mark.parametrize("K", [512, 3584, 18944])
def test_error_of_normal_operands(ops, K):
    """2-norm against 64 bits: 2.5e-8 is what the kernel's comment states, a quarter and less of what the sums in 32 bits have."""
    g = torch.Generator(device="cuda").manual_seed(K)
    a, w = torch.randn(64, K, device="cuda", generator=g), torch.randn(512, K, device="cuda", generator=g)
    want = a.double() @ w.double().t()
    got = error(ops.fixed_linear(a, ops.FixedWeight(w)), want)
    assert got < 2.7e-8 and got < 0.3 * error(ops.sgemm_nt(a, w), want)


def error(x, want):
    return float((x.double() - want).norm() / want.norm())


@pytest.mark.parametrize("r", [1.0, 30.0, 300.0, 1e3, 1e4, 1e6, 1e25])
@pytest.mark.parametrize("columns", [1, 40])
def test_outliers_cost_no_bits(ops, r, columns):
    """Columns of the activations r times the others, those columns of the weights by as much less: the error of the sums in 32 bits bounds
    it, whatever r and however many (as many as a row lists, and more); a row's bits depend on neither plan nor batch."""
    g = torch.Generator(device="cuda").manual_seed(3)
    a, w = torch.randn(70, 3584, device="cuda", generator=g), torch.randn(512, 3584, device="cuda", generator=g)
    a[:, 7:7 + columns] *= r
    w[:, 7:7 + columns] /= r
    W, want = ops.FixedWeight(w), a.double() @ w.double().t()
    got, sums = ops.fixed_linear(a, W), ops.sgemm_nt(a, w)
    assert error(got, want) <= error(sums, want)
    assert max(error(x, y) for x, y in zip(got, want)) <= max(error(x, y) for x, y in zip(sums, want))
    for plan in [(8, 1), (16, 3), (32, 1), (48, 2), (64, 7)]:
        assert torch.equal(ops.fixed_linear(a, W, plan), got), plan
    assert torch.equal(ops.fixed_linear(a[33:34], W), got[33:34])
    ops.check_device_errors()


def test_rows_of_wide_range(ops):
    """Outliers of several magnitudes in one row, as many as a row's list holds and one more, rows of few elements, features with an
    outlier of their own: each row within the error of the sums in 32 bits."""
    g = torch.Generator(device="cuda").manual_seed(4)
    K = 2052
    a, w = torch.randn(12, K, device="cuda", generator=g), torch.randn(384, K, device="cuda", generator=g)
    a[0, [5, 1700, 2051]] = torch.tensor([1e12, -1e3, 1e6], device="cuda")      # they never reach the result
    w[:, [5, 1700, 2051]] *= torch.tensor([1e-12, 1e-3, 1e-6], device="cuda")
    a[1, :16] = 1e9
    a[2, :17] = 1e9
    w[:, :17] *= 1e-9
    a[3] = torch.where(torch.rand(K, device="cuda", generator=g) < 0.995, 0.0, a[3])
    a[4] = 0
    a[4, [40, 2000]] = torch.tensor([1.0, 1e-10], device="cuda")
    a[5] = 0
    a[5, 100] = 7.5
    a[6] *= torch.exp(3 * torch.randn(K, device="cuda", generator=g))
    a[7] *= torch.exp2(torch.randint(-30, 30, (K,), device="cuda", generator=g).float())
    a[8, 1000:1010] *= 1e-30
    w[200, 99], w[201, 1001] = 1e5, 1e-5
    a[9, 99] = 1e-5
    W, want = ops.FixedWeight(w), a.double() @ w.double().t()
    assert int((W.exponents >= 1000).sum()) >= 1      # the feature with an outlier
    got, sums = ops.fixed_linear(a, W), ops.sgemm_nt(a, w)
    ops.check_device_errors()
    for t in range(12):
        assert error(got[t], want[t]) <= max(error(sums[t], want[t]), 4e-8), t
    assert torch.equal(ops.fixed_linear(a, W, (16, 4)), got)
    for t in range(12):
        assert torch.equal(ops.fixed_linear(a[t:t + 1], W)[0], got[t]), t


def test_weights_of_wide_range_stay_on_the_cuda_cores(ops):
    """A few features without a scale are the kernel's to see to; a weight with more of them is not taken."""
    w = torch.randn(16384, 512, device="cuda")
    w[:256, 3] = 1e3
    assert isinstance(ops.linear_weight(w), ops.FixedWeight)
    w[256, 3] = 1e3
    assert ops.linear_weight(w) is w


def test_a_weight_changed_in_place(ops):
    """The exponents follow the weight: elements that outgrow them, rows that get an infinity or lose their outlier, through a view too; a
    tensor without a version counter is not taken."""
    g = torch.Generator(device="cuda").manual_seed(6)
    a, w = torch.randn(9, 1024, device="cuda", generator=g), torch.randn(8192, 1024, device="cuda", generator=g)
    w[3, 4] = 1e4
    W = ops.linear_weight(w)
    ops.linear(a, W)
    for change in (lambda: w[5].mul_(1e6), lambda: w.mul_(1e-5), lambda: w[7, 7].fill_(float("inf")), lambda: w[3, 4].zero_(), lambda: w.view(-1)[9].fill_(1e9)):
        change()
        assert torch.equal(ops.linear(a, W), ops.fixed_linear(a, ops.FixedWeight(w.clone())))
    ops.check_device_errors()
    with torch.inference_mode():
        plain = torch.zeros(8192, 1024, device="cuda")
    assert ops.linear_weight(plain) is plain


def test_a_captured_step_follows_a_weight_changed_in_place(ops):
    """Decode steps replayed from a graph against the same steps launched one by one, with weights edited between them."""
    from pyre_b200 import Engine
    from pyre_b200.config import config_from_dict
    from pyre_b200.engine.step import StepEntry
    raw = dict(architectures=["Qwen2ForCausalLM"], tie_word_embeddings=False, hidden_size=512, intermediate_size=16384, num_hidden_layers=1,
               num_attention_heads=8, num_key_value_heads=2, head_dim=64, vocab_size=512, rope_theta=10000.0, rms_norm_eps=1e-6,
               max_position_embeddings=256)
    got = {}
    for graphs in (True, False):
        engine = Engine(config=config_from_dict(raw), seed=1, dtype="float32", max_cache_tokens=256, max_num_seqs=2, cuda_graphs=graphs)
        ffn = engine.model.blocks[0].ffn
        assert isinstance(ffn.w_down, ops.FixedWeight)
        engine.cache.begin(0)
        rows = got[graphs] = []
        for k in range(6):
            rows.append(engine.stepper.step([StepEntry(0, [k], [0])]).clone())
            if k == 2:
                ffn.w_down.w[:100].mul_(1e4)
            if k == 4:
                ffn.w_gate_up.w.mul_(0.01)
        engine.stepper.check_device_errors()
        assert (engine.stepper.graph_replays > 3) == graphs
    assert all(torch.equal(x, y) for x, y in zip(got[True], got[False]))


def test_many_rows_go_in_portions(ops, monkeypatch):
    """Scratch memory is bounded whatever the number of rows: portions give the same bits, of rows off 16-byte boundaries too."""
    a, W = torch.randn(330, 1027, device="cuda")[:, 3:], ops.FixedWeight(torch.randn(300, 1024, device="cuda"))
    whole = ops.fixed_linear(a, W)
    for portion in (64, 128, 320):
        monkeypatch.setattr(ops, "FIXED_SCRATCH", portion * 4 * 1024)
        assert torch.equal(ops.fixed_linear(a, W), whole)
    ops.check_device_errors()


def test_which_weights_take_it(ops):
    """The rule knows the weight alone: small ones, short and overlong rows, rows off 16-byte boundaries and rows that overlap stay with the
    CUDA cores' product."""
    def weight(N, K, ld=0):
        return torch.zeros(N, ld or K, device="cuda")[:, :K]
    assert isinstance(ops.linear_weight(weight(16384, 512)), ops.FixedWeight)
    assert isinstance(ops.linear_weight(weight(205, 40960)), ops.FixedWeight)
    for w in (weight(16383, 512), weight(16600, 508), weight(16384, 600, 601), weight(16384, 512).to(torch.bfloat16), weight(300, 40964),
              weight(1, 1024).expand(8192, 1024)):
        assert ops.linear_weight(w) is w
    W = ops.FixedWeight(weight(128, 512))
    with pytest.raises(ValueError):
        ops.fixed_linear(torch.zeros(2, 516, device="cuda"), W)
    assert ops.linear(torch.zeros(2, 512, device="cuda"), W).shape == (2, 128)
