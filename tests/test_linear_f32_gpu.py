"""The float32 product on the tensor cores (csrc/linear_f32.cu) against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from vapi_b200 import ops as o
    o.strict_fp32()
    return o


def _bound(a, w):
    """Elementwise: a piece of 64 k is 6 x 4 tensor-core additions of 16 products, each of which may drop what lies below the
    last of 24 bits (2^-23 of the sum so far), the pieces are K / 64 float additions, the split leaves out 2^-24, and
    the bias is one more rounding; all against the sum of the magnitudes."""
    K = a.shape[1]
    return (2 * 24 + -(-K // 64) + 8 + 2) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t()) + 1e-30


# one row and one tile; edges of the 64 / 128 token and 128 feature tiles; K below a stage, ragged, not a multiple of 8; K shared by
# two to eight blocks; more tiles than multiprocessors
@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (17, 6, 12), (33, 129, 60), (64, 128, 64), (65, 127, 68), (128, 256, 516), (129, 300, 1028),
                                   (31, 130, 4160), (200, 1536, 2052), (64, 2048, 8192), (513, 5000, 130 * 4)])
def test_float32_product_is_no_further_from_the_exact_one_than_its_bound(ops, M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N)
    a = torch.randn(M, K, generator=g, device="cuda") * torch.exp(2 * torch.randn(M, K, generator=g, device="cuda"))
    w = torch.randn(N, K, generator=g, device="cuda")
    b = torch.randn(N, generator=g, device="cuda")
    want = a.double() @ w.double().t()
    got = ops.linear_f32(a, w, b)
    assert ((got.double() - want - b.double()).abs() <= _bound(a, w) + 2.0 ** -23 * b.double().abs()).all()
    assert torch.equal(ops.linear_f32(a, w), ops.linear_f32(a, w))
    before = ops.launch_count
    via = ops.linear(a, w, b)
    assert M <= 16 or N * K < 1 << 20 or (ops.launch_count == before + 2 and torch.equal(via, got))


def test_float32_product_of_more_rows_than_its_scratch_holds(ops, monkeypatch):
    g = torch.Generator(device="cuda").manual_seed(8)
    a, w, b = (torch.randn(*s, generator=g, device="cuda") for s in ((301, 260), (140, 260), (140,)))
    monkeypatch.setattr(ops, "LINEAR_F32_ROWS", 128)
    got = ops.linear_f32(a, w, b)
    assert ((got.double() - a.double() @ w.double().t() - b.double()).abs() <= _bound(a, w) + 2.0 ** -23 * b.double().abs()).all()


@pytest.mark.parametrize("M,N,K", [(70, 300, 256), (40, 130, 2048), (300, 20000, 68)])
def test_float32_product_of_what_cannot_be_split(ops, M, N, K):
    """Infinities, NaN and magnitudes next to the largest float, in tokens and in weights, in the first and the last row, in tiles of one
    block and of several: what plain FMAs give, and nothing else changes."""
    g = torch.Generator(device="cuda").manual_seed(3)
    a, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    a2, w2 = a.clone(), w.clone()
    a2[0, 0], a2[3, K - 1], a2[M - 1, K // 2], a2[5, 1] = float("inf"), float("nan"), -float("inf"), 3.0e38
    w2[0, 2], w2[N - 1, K - 1], w2[N // 2, 0], w2[7, 9] = float("inf"), float("nan"), 2.0e38, 0.0
    # the huge finite ones never meet in one sum, and the huge weight does not overflow beside the other sign's infinity: what a
    # float sum makes of that depends on its order, and the float64 product below does not show it
    a2[5, 0], w2[N // 2, 1], a2[M - 1, 0] = 0.0, 0.0, 0.5
    clean = ops.linear_f32(a, w)
    got, want = ops.linear_f32(a2, w2), a2.double() @ w2.double().t()
    big = want.abs() >= 2.0 ** 128 * (1 - 2.0 ** -25)         # (what rounds to a float's infinity)
    want = torch.where(big, want.sign() * float("inf"), want)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(torch.isinf(got), torch.isinf(want))
    fin = torch.isfinite(want)
    err = torch.where(fin, (got.double() - want).abs(), torch.zeros_like(want))
    scale = torch.where(fin, (torch.nan_to_num(a2, 0, 0, 0).double().abs() @ torch.nan_to_num(w2, 0, 0, 0).double().abs().t()), torch.ones_like(want))
    assert (err <= (K + 60) * 2.0 ** -24 * scale).all()       # (a plain sum of K products is K roundings)
    rows = torch.ones(M, dtype=torch.bool, device="cuda")
    rows[[0, 3, 5, M - 1]] = False
    cols = torch.ones(N, dtype=torch.bool, device="cuda")
    cols[[0, 7, N // 2, N - 1]] = False
    assert torch.equal(got[rows][:, cols], clean[rows][:, cols])


# a tile of one block, and one shared by several
@pytest.mark.parametrize("M,N,K", [(70, 300, 256), (40, 130, 2048)])
def test_float32_product_whose_terms_overflow_though_no_operand_is_huge(ops, M, N, K):
    """Products beyond the largest float from operands of 1e25 to 1e35, with every combination of signs of the second planes (a mantissa just above
    or below one of eight bits): infinities of the product's sign, as float FMAs give, and no NaN; nothing else changes."""
    g = torch.Generator(device="cuda").manual_seed(5)
    a, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    clean = ops.linear_f32(a, w)
    a2, w2 = a.clone(), w.clone()
    mantissas = torch.tensor([1.0 + 2.0 ** -9, 1.0 - 2.0 ** -10, -1.5 - 2.0 ** -9, -1.5 + 2.0 ** -9], device="cuda")
    a2[:4, K - 3], w2[:4, K - 3] = mantissas * 2.0 ** 83, mantissas * 2.0 ** 117
    a2[M - 1, 5], w2[N - 1, 5] = 1.1e35, -1.1e25
    a2[4:M - 1, [5, K - 3]], w2[4:N - 1, [5, K - 3]] = 0.0, 0.0      # (one huge term a sum: what more give depends on their order)
    a2[:4, 5], w2[:4, 5], a2[M - 1, K - 3], w2[N - 1, K - 3] = 0.0, 0.0, 0.0, 0.0
    got, want = ops.linear_f32(a2, w2), (a2.double() @ w2.double().t()).float()
    assert int(torch.isinf(want).sum()) == 17 and torch.equal(torch.isinf(got), torch.isinf(want)) and not torch.isnan(got).any()
    assert torch.equal(got[torch.isinf(got)], want[torch.isinf(want)])
    fin = torch.isfinite(want)
    assert ((got.double() - a2.double() @ w2.double().t()).abs() <= _bound(a2, w2))[fin].all()
    assert torch.equal(ops.linear_f32(a, w), clean)


def test_float32_product_of_tiny_and_exact_numbers(ops):
    """Numbers of eight bits have empty lower planes; small whole numbers come out exactly; small magnitudes keep their bits."""
    g = torch.Generator(device="cuda").manual_seed(4)
    a = torch.randint(-9, 10, (90, 200), generator=g, device="cuda").float()
    w = torch.randint(-9, 10, (150, 200), generator=g, device="cuda").float()
    assert torch.equal(ops.linear_f32(a, w).double(), a.double() @ w.double().t())
    assert torch.equal(ops.linear_f32(a * 2.0 ** -60, w).double(), (a.double() @ w.double().t()) * 2.0 ** -60)


# one tile a block, tiles in turn, a tile shared by two to eight blocks
@pytest.mark.parametrize("M,N,K", [(70, 300, 60), (300, 20000, 132), (64, 2048, 520), (40, 130, 4160)])
def test_a_float32_product_that_gives_up_a_wait_writes_nothing_and_says_so(ops, M, N, K):
    """Waits that give up without a poll, or after one (what then is complete is written, the rest is not); the next call is unaffected."""
    g = torch.Generator(device="cuda").manual_seed(9)
    a, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    want = ops.linear_f32(a, w)
    lib, kp = ops._lib("linear_f32"), -(-K // 8) * 8
    planes, bad = torch.empty(3 * M * kp, dtype=torch.bfloat16, device="cuda"), torch.empty(M, dtype=torch.int32, device="cuda")
    for polls in (0, 1):
        out, status = torch.full((M, N), float("nan"), device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        rc = lib.vapi_linear_f32(w.data_ptr(), N, K, M, a.data_ptr(), planes.data_ptr(), bad.data_ptr(), None, out.data_ptr(), N, polls,
                                 status.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        left = torch.isnan(out)
        assert int(status) == (16 if bool(left.any()) else 0) and torch.equal(out[~left], want[~left])
        assert polls > 0 or bool(left.all())
        assert torch.equal(ops.linear_f32(a, w, status=status.zero_()), want) and int(status) == 0


# both sides of every line of the dispatch: shared K or whole rows at 3,072, 6,144 and 8,192 rows and a K of 1,024, 1,536 and 2,048; whole rows
# with and without the staged tokens (K of 128; up to eight tokens, and above twelve where rounds of blocks are not filled)
@pytest.mark.parametrize("N,K", [(3071, 1024), (3073, 1024), (3072, 1028), (8191, 2048), (8193, 2048), (6143, 1536), (6145, 1536),
                                 (6147, 1540), (6150, 2052), (3075, 4), (4099, 128), (4099, 132), (3077, 256),
                                 (3077, 260), (12289, 512), (12287, 512), (12290, 2048), (12290, 2052), (8200, 4100)])
def test_decode_product_of_wide_weights(ops, N, K):
    """Against float64 within the bound of K float FMAs, and a token's result is the same bits whatever the batch."""
    g = torch.Generator(device="cuda").manual_seed(N + K)
    a, w, b = (torch.randn(*s, generator=g, device="cuda") for s in ((16, K), (N, K), (N,)))
    want = a.double() @ w.double().t() + b.double()
    bound = (K + 2) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t() + b.double().abs())
    whole = ops.skinny_linear_f32(w, a, b)
    assert ((whole.double() - want).abs() <= bound).all()
    for M in (1, 2, 4, 5, 8, 9, 13):
        assert torch.equal(ops.skinny_linear_f32(w, a[16 - M:].contiguous(), b), whole[16 - M:]), M


# each form of the gated product (staged, whole rows, shared K), odd features, one and many pieces of K
@pytest.mark.parametrize("N,K", [(16384, 512), (8198, 1540), (8194, 128), (3074, 1024), (1034, 2048), (6, 4)])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh"])
def test_gated_decode_product_is_the_product_and_its_gate(ops, N, K, act):
    """The gate in the product's epilogue gives the bits of the two launches it stands for."""
    g = torch.Generator(device="cuda").manual_seed(N + K)
    a, w = (torch.randn(*s, generator=g, device="cuda") for s in ((16, K), (N, K)))
    for M in (1, 3, 8, 9, 16):
        x = a[:M].contiguous()
        want = ops.swiglu(ops.skinny_linear_f32(w, x), act)
        assert torch.equal(ops.linear_swiglu(x, w, act), want), M


# shared K, staged rows, whole rows with a short and a long K: one launch but for the last, above eight tokens
@pytest.mark.parametrize("N,K,M,launches", [(2048, 2048, 16, 1), (14336, 1024, 16, 1), (14336, 512, 9, 1), (14336, 516, 9, 2), (14336, 2048, 8, 1), (12288, 2048, 16, 2)])
def test_where_the_gate_rides_on_the_product(ops, N, K, M, launches):
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = (torch.randn(*s, generator=g, device="cuda") for s in ((M, K), (N, K)))
    before = ops.launch_count
    got = ops.linear_swiglu(x, w)
    assert ops.launch_count == before + launches
    assert torch.equal(got, ops.skinny_linear_f32(w, x, glu="silu")) and torch.equal(got, ops.swiglu(ops.skinny_linear_f32(w, x)))
