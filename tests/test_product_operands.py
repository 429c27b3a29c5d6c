"""What the products' wrappers accept beside a weight: the bias' shape and type, the step's status word, autograd."""
import pytest
import torch

from vapi_b200 import ops

BF16, F32 = torch.bfloat16, torch.float32


class _Calls:
    """A library in place of the kernels: keeps the arguments of every call."""

    def __init__(self):
        self.got = []

    def __getattr__(self, name):
        def call(*args):
            self.got.append((name, args))
            return 0
        return call


@pytest.fixture
def calls(monkeypatch):
    lib = _Calls()
    monkeypatch.setattr(ops, "_lib", lambda name: lib)
    monkeypatch.setattr(ops, "_cuda", lambda *t: None)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    return lib


PRODUCTS = {"skinny_linear": (BF16, lambda w, x, b: ops.skinny_linear(w, act=x, bias=b)),
            "linear_tc": (BF16, lambda w, x, b: ops.linear_tc(w, act=x, bias=b)),
            "prompt_linear": (BF16, lambda w, x, b: ops.prompt_linear(w, act=x, bias=b)),
            "skinny_linear_f32": (F32, lambda w, x, b: ops.skinny_linear_f32(w, x, b)),
            "linear_f32": (F32, lambda w, x, b: ops.linear_f32(x, w, b))}


@pytest.mark.parametrize("which", list(PRODUCTS))
def test_a_bias_has_one_number_a_feature(calls, which):
    """The kernels read N numbers of it, whatever its length."""
    dtype, product = PRODUCTS[which]
    w, x = torch.zeros(48, 32, dtype=dtype), torch.zeros(9, 32, dtype=dtype)
    for n in (0, 1, 47, 49):
        with pytest.raises(ops.KernelError, match="bias"):
            product(w, x, torch.zeros(n))
    assert not calls.got, "no kernel has been called with it"
    product(w, x, torch.zeros(48))
    assert [name for name, _ in calls.got] == ["vapi_" + which]


# rows on both sides of 16 (the weight-streaming kernel, the split product) and a weight on both sides of the split product's least size
@pytest.mark.gpu
@pytest.mark.parametrize("M", [5, 33])
@pytest.mark.parametrize("N,K", [(1024, 1024), (48, 64)])
def test_linear_takes_every_bias_that_the_library_takes(M, N, K):
    ops.strict_fp32()
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    for b in (torch.randn(N, generator=g, device="cuda"), torch.randn(N, generator=g, device="cuda").bfloat16(),
              torch.randn(1, generator=g, device="cuda"), torch.randn((), generator=g, device="cuda"),
              torch.randn(1, N, generator=g, device="cuda").double(), torch.randn(2 * N, generator=g, device="cuda")[::2],
              torch.randn(M, N, generator=g, device="cuda"), torch.randn(M, 1, generator=g, device="cuda")):
        want = x.double() @ w.double().t() + b.to(torch.float32).double()
        # (K + 1 roundings of sums no larger than the sum of the magnitudes)
        bound = (K + 2) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t() + b.double().abs())
        assert ((ops.linear(x, w, b).double() - want).abs() <= bound).all(), tuple(b.shape)
    for wrong in (N - 1, N + 1, 2):
        with pytest.raises(RuntimeError):
            ops.linear(x, w, torch.zeros(wrong, device="cuda"))
