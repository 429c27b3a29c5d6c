"""The float32 prompt attention on the tensor cores (csrc/attention_f32.cuh) beside the general kernel and the plain form."""
import pytest
import torch

from test_kernels_gpu import _attention_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from vapi_b200 import ops as o
    o.strict_fp32()
    return o


# tiles of 64 rows and 64 keys and their edges, decode tokens beside portions, rows that no whole token fills, split keys, windows
@pytest.mark.parametrize("nh,nkv,page", [(8, 2, 64), (32, 8, 128), (3, 1, 64), (40, 1, 192)])
@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("window", [0, 1, 70])
def test_float_attention_of_portions(ops, nh, nkv, page, splits, window):
    _attention_case(ops, torch.float32, nh, nkv, 64, page, [(17, 17), (1, 130), (64, 64), (65, 129), (1, 1), (30, 400), (128, 128), (2, 63)],
                    window=window, splits=splits)
    _attention_case(ops, torch.float32, nh, nkv, 64, page, [(70, 300)] + [(1, 5 + i) for i in range(40)], window=window, splits=splits, planted=True)


# decode steps: one token a sequence, up to four q heads a kv head; slices that end inside 32 and 128 keys, empty slices, windows that begin inside
# a tile, pages of 32 to 192
@pytest.mark.parametrize("nh,nkv,page", [(8, 2, 64), (3, 1, 32), (4, 4, 96), (32, 8, 192)])
@pytest.mark.parametrize("splits", [1, 2, 7])
@pytest.mark.parametrize("window", [0, 1, 33, 200])
def test_float_attention_of_decode_tokens(ops, nh, nkv, page, splits, window):
    lens = [(1, 1), (1, 31), (1, 32), (1, 33), (1, 127), (1, 128), (1, 129), (1, 500), (1, 1000)]
    _attention_case(ops, torch.float32, nh, nkv, 64, page, lens, window=window, splits=splits)
    _attention_case(ops, torch.float32, nh, nkv, 64, page, lens, window=window, splits=splits, planted=window == 0)


def _random_case(seed, n, klen, nh, nkv):
    g = torch.Generator(device="cuda").manual_seed(seed)
    pages = -(-klen // 64)
    q = torch.randn(n, nh * 64, generator=g, device="cuda")
    cache = torch.randn(pages, 2, nkv, 64, 64, generator=g, device="cuda")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    return q, cache, (torch.arange(pages, device="cuda").int()[None], i32([0, n]), i32([klen]), n, 1, n, klen, nh, nkv, 64, 0.125)


def test_float_attention_is_no_further_from_the_exact_one(ops):
    q, cache, args = _random_case(1, 200, 700, 4, 2)
    got, general = (ops.paged_attention(q, 256, cache, *args, splits=1, impl=impl).double() for impl in ("auto", "general"))
    k, v = (cache.double()[:, i].transpose(0, 1).reshape(2, -1, 64)[:, :700].repeat_interleave(2, 0) for i in (0, 1))
    s = torch.einsum("nhd,hkd->hnk", q.double().view(200, 4, 64), k) * 0.125
    s = s.masked_fill(torch.arange(700, device="cuda")[None, :] > 500 + torch.arange(200, device="cuda")[:, None], float("-inf"))
    want = torch.einsum("hnk,hkd->nhd", s.softmax(-1), v).reshape(200, 256)
    err, before = ((t - want).norm() / want.norm() for t in (got, general))
    assert err < 3e-7 and err <= 1.05 * before, (err, before)


def test_float_attention_of_what_cannot_be_split(ops):
    """Infinities, NaN and magnitudes next to the largest float in queries, keys and values give what the general kernel gives, but for
    one element of the tokens 32 to 36: those share a tile of that kernel with token 37, whose value has the infinity, and it
    multiplies what they may not see by zero."""
    q, cache, args = _random_case(2, 100, 260, 4, 2)
    q[3, 5], q[50, 70] = float("inf"), float("nan")
    cache[1, 0, 0, 7, 3], cache[2, 0, 1, 9, 60], cache[3, 1, 0, 5, 0] = -float("inf"), 3.0e38, float("inf")
    got, want = (ops.paged_attention(q, 256, cache, *args, splits=1, impl=impl) for impl in ("auto", "general"))
    for at in (0, 64):                                     # (the first kv head's two heads)
        assert torch.equal(torch.isnan(got[32:37, at]), torch.isnan(want[32:37, at + 1])) and not torch.isinf(got[32:37, at]).any()
        got[32:37, at] = want[32:37, at]
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    fin = torch.isfinite(want)
    torch.testing.assert_close(got[fin], want[fin], atol=2e-5, rtol=2e-5)


# planted at the first, a middle and the last token of a group of 32, of a tile of 64 rows and of the portion; with and without a window
@pytest.mark.parametrize("window", [0, 40])
@pytest.mark.parametrize("token", [0, 15, 31, 32, 44, 63, 64, 99])
def test_a_value_that_a_row_may_not_see_does_not_come_into_it(ops, window, token):
    """An infinity and a NaN in one key's value: only rows that see the key, and only those two elements of them."""
    q, cache, args = _random_case(3, 100, 260, 4, 2)
    clean = ops.paged_attention(q, 256, cache, *args, window, 1).view(100, 4, 64)
    at = 160 + token
    cache[at // 64, 1, :, at % 64, 3], cache[at // 64, 1, :, at % 64, 60] = float("inf"), float("nan")
    got = ops.paged_attention(q, 256, cache, *args, window, 1).view(100, 4, 64)
    rows = torch.arange(100, device="cuda")
    sees = (rows >= token) & ((rows < token + window) if window else torch.ones_like(rows, dtype=torch.bool))
    hit = torch.zeros(100, 4, 64, dtype=torch.bool, device="cuda")
    hit[sees] = torch.zeros(64, dtype=torch.bool, device="cuda").index_fill_(0, torch.tensor([3, 60], device="cuda"), True)
    assert torch.equal(~torch.isfinite(got), hit)
    torch.testing.assert_close(got[~hit], clean[~hit], atol=2e-5, rtol=2e-5)


# signs and mantissas just above and below one of eight bits: the partial products of a score overflow together or against each other
@pytest.mark.parametrize("impl", ["auto", "general"])
@pytest.mark.parametrize("mq", [1.0 + 2.0 ** -9, 1.0 - 2.0 ** -10, 1.5 + 2.0 ** -9, 1.5 - 2.0 ** -9])
@pytest.mark.parametrize("mk", [1.0 + 2.0 ** -9, 1.5 - 2.0 ** -9])
def test_a_score_beyond_the_largest_float_is_what_float_products_make_of_it(ops, impl, mq, mk):
    """Queries and keys of 1e28 to 1e32: a score of minus infinity has no weight, one of infinity makes the row NaN; other rows stay."""
    q, cache, args = _random_case(6, 100, 260, 4, 2)
    q.view(100, 4, 64)[:, :, 9] = 0.0
    cache[:, 0, :, :, 9] = 0.0
    clean = ops.paged_attention(q, 256, cache, *args, splits=1, impl=impl).view(100, 4, 64)
    q.view(100, 4, 64)[[20, 70], :, 9] = mq * 2.0 ** 95
    cache[1, 0, 0, 30, 9] = -mk * 2.0 ** 104               # key 94, seen by all
    cache[3, 0, 1, 40, 9] = mk * 2.0 ** 104                # key 232, seen by the tokens from 72 on: by neither of the two
    got = ops.paged_attention(q, 256, cache, *args, splits=1, impl=impl).view(100, 4, 64)
    assert torch.isfinite(got).all()
    k, v = (cache.double()[:, i].transpose(0, 1).reshape(2, -1, 64)[:, :260] for i in (0, 1))
    for t in (20, 70):
        keep = [j for j in range(161 + t) if j != 94]
        for h in (0, 1):                                   # the heads of the first kv head: as if the key were not there
            s = (q.double().view(100, 4, 64)[t, h] * (torch.arange(64, device="cuda") != 9)) @ k[0, keep].t() * 0.125
            torch.testing.assert_close(got[t, h].double(), s.softmax(-1) @ v[0, keep], atol=2e-5, rtol=2e-5)
    rows = [t for t in range(100) if t not in (20, 70)]
    torch.testing.assert_close(got[rows], clean[rows], atol=2e-5, rtol=2e-5)
    cache[1, 0, 0, 30, 9] = mk * 2.0 ** 104                # now infinity
    got = ops.paged_attention(q, 256, cache, *args, splits=1, impl=impl).view(100, 4, 64)
    nan = torch.zeros_like(got, dtype=torch.bool)
    nan[[20, 70], :2] = True
    assert torch.equal(torch.isnan(got), nan)
