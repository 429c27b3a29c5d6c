"""The recurrences over long portions (csrc/recurrent_chunks.cu) against float64, token by token."""
import itertools

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from vapi_b200 import ops as o
    return o


def _step(qlens, starts):
    cu = torch.tensor([0] + list(itertools.accumulate(qlens)), dtype=torch.int32)
    pos = torch.cat([torch.arange(a, a + q) for q, a in zip(qlens, starts)]).int()
    slots = torch.randperm(len(qlens) + 2, generator=torch.Generator().manual_seed(1))[:len(qlens)].int()
    return cu, pos, slots


def _delta(qkv, ab, A, dtb, S, nh, nkv, dk, dv, eps):
    """One sequence: qkv [n, *], S [nh, dk, dv] (in place)."""
    n = qkv.shape[0]
    unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + eps)
    q, k = (unit(t.view(n, nkv, dk)).repeat_interleave(nh // nkv, 1) for t in (qkv[:, :nkv * dk], qkv[:, nkv * dk:2 * nkv * dk]))
    v, beta = qkv[:, 2 * nkv * dk:].view(n, nh, dv), torch.sigmoid(ab[:, nh:])
    g = torch.exp(-torch.exp(A) * torch.nn.functional.softplus(ab[:, :nh] + dtb))
    out = []
    for t in range(n):
        S *= g[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S += k[t][:, :, None] * u[:, None, :]
        out.append(torch.einsum("hkv,hk->hv", S, q[t]) * dk ** -0.5)
    return torch.stack(out).view(n, -1)


def _space(xbc, dt, A, dtb, D, S, nh, groups, N, P):
    n = xbc.shape[0]
    x = xbc[:, :nh * P].view(n, nh, P)
    B, C = (t.view(n, groups, N).repeat_interleave(nh // groups, 1) for t in xbc[:, nh * P:].chunk(2, -1))
    step = torch.nn.functional.softplus(dt + dtb)
    out = []
    for t in range(n):
        S *= torch.exp(-torch.exp(A) * step[t])[:, None, None]
        S += B[t][:, :, None] * (step[t][:, None] * x[t])[:, None, :]
        out.append(torch.einsum("hkv,hk->hv", S, C[t]) + D[:, None] * x[t])
    return torch.stack(out).view(n, -1)


# portions at the edges of a chunk and of the rule, walked ones among them, one alone, one alone whose rows go on behind it
@pytest.mark.parametrize("qlens,starts,extra", [([19, 20, 48, 1, 47, 64, 2, 65], [0, 5, 9, 0, 3, 0, 0, 4], 0), ([128], [0], 0), ([193], [7], 0), ([10], [3], 30)])
@pytest.mark.parametrize("rates", [(-1.0, 1.0), (3.0, 6.0), (-9.0, -7.0)])        # ordinary decays, next to none left, next to none lost
def test_chunks_give_the_recurrence(ops, qlens, starts, extra, rates):
    gen = torch.Generator().manual_seed(sum(qlens))
    cu, pos, slots = _step(qlens, starts)
    n = sum(qlens) + extra
    pos = torch.cat([pos, torch.zeros(extra, dtype=torch.int32)])
    d = lambda t: t.cuda()

    def check(got, state, want, want_state):
        # three bfloat16 planes of a float lose 2^-25, a sum over 128 rows and 64 tokens of float accumulators some 2^-21
        m = sum(qlens)
        assert (got.cpu().double()[:m] - want).norm() <= 2e-6 * want.norm()
        assert (state.cpu().double() - want_state).norm() <= 2e-6 * want_state.norm()

    for nh, nkv, dv in ((2, 1, 16), (3, 3, 48)):
        dk = 128
        qkv = torch.randn((n, 2 * nkv * dk + nh * dv), generator=gen).bfloat16()
        ab = torch.randn((n, 2 * nh + 3), generator=gen).bfloat16()
        A, dtb = torch.rand(nh, generator=gen) * (rates[1] - rates[0]) + rates[0], torch.randn(nh, generator=gen)
        state = torch.randn((len(qlens) + 2, 9 + nh * dk * dv), generator=gen)
        want_state = state.double()
        want = []
        for s, q in enumerate(qlens):
            S = want_state[slots[s], 9:].view(nh, dk, dv)
            if starts[s] == 0:
                S.zero_()
            r = slice(int(cu[s]), int(cu[s + 1]))
            want.append(_delta(qkv[r].double(), ab[r, :2 * nh].double(), A.double(), dtb.double(), S, nh, nkv, dk, dv, 1e-6))
        mine = d(state)
        got = ops.gated_delta(d(qkv), d(ab)[:, :2 * nh], d(A), d(dtb), mine, 9, d(slots), d(cu), d(pos), nh, nkv, dk, dv)
        check(got, mine, torch.cat(want), want_state)
    for nh, groups, P in ((2, 1, 32), (4, 2, 96)):
        N = 128
        xbc = torch.randn((n, nh * P + 2 * groups * N), generator=gen).bfloat16()
        dt = torch.randn((n, nh + 5), generator=gen).bfloat16()
        A, dtb, D = torch.rand(nh, generator=gen) * (rates[1] - rates[0]) + rates[0], torch.randn(nh, generator=gen) - 2, torch.randn(nh, generator=gen)
        state = torch.randn((len(qlens) + 2, 4 + nh * N * P), generator=gen)
        want_state = state.double()
        want = []
        for s, q in enumerate(qlens):
            S = want_state[slots[s], 4:].view(nh, N, P)
            if starts[s] == 0:
                S.zero_()
            r = slice(int(cu[s]), int(cu[s + 1]))
            want.append(_space(xbc[r].double(), dt[r, 2:2 + nh].double(), A.double(), dtb.double(), D.double(), S, nh, groups, N, P))
        mine = d(state)
        got = ops.state_space(d(xbc), d(dt)[:, 2:2 + nh], d(A), d(dtb), d(D), mine, 4, d(slots), d(cu), d(pos), nh, groups, N, P)
        check(got, mine, torch.cat(want), want_state)


def test_portions_give_what_the_whole_gives(ops):
    """A prompt in portions on both sides of the rule leaves the state and the outputs of the whole prompt."""
    gen = torch.Generator(device="cuda").manual_seed(5)
    n, nh, dv = 300, 2, 32
    qkv = torch.randn((n, 2 * nh * 128 + nh * dv), generator=gen, device="cuda").bfloat16()
    ab = torch.randn((n, 2 * nh), generator=gen, device="cuda").bfloat16()
    A, dtb = torch.zeros(nh, device="cuda"), torch.zeros(nh, device="cuda")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")

    def run(cuts):
        state, out = torch.full((1, nh * 128 * dv), float("nan"), device="cuda"), []
        for a, b in zip(cuts, cuts[1:]):
            out.append(ops.gated_delta(qkv[a:b], ab[a:b], A, dtb, state, 0, i32([0]), i32([0, b - a]), torch.arange(a, b, device="cuda").int(), nh, nh, 128, dv))
        return torch.cat(out), state
    whole, s1 = run([0, n])
    parts, s2 = run([0, 100, 147, 148, 212, n])
    assert (whole - parts).norm() <= 4e-6 * whole.norm() and (s1 - s2).norm() <= 4e-6 * s1.norm()
