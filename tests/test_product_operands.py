"""What the products' wrappers accept beside a weight: the bias' shape and type, the step's status word, autograd."""
import math

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


@pytest.mark.parametrize("which", ["linear_tc", "prompt_linear", "linear_f32"])
def test_a_product_of_a_step_records_into_the_steps_status_word(calls, which):
    """Those with bounded waits: the word that the step holds, unless the call brings its own; none outside of a step."""
    dtype, product = PRODUCTS[which]
    w, x = torch.zeros(48, 32, dtype=dtype), torch.zeros(20, 32, dtype=dtype)
    word, own = torch.zeros(1, dtype=torch.int32), torch.zeros(1, dtype=torch.int32)
    with ops.one_stream(word):
        product(w, x, None)
        ops.linear_f32(x.float(), w.float(), status=own)
        with ops.one_stream():
            product(w, x, None)
        product(w, x, None)
    product(w, x, None)
    held = [word.data_ptr() in args for _, args in calls.got]
    assert held == [True, False, False, True, False] and own.data_ptr() in calls.got[1][1]


@pytest.mark.gpu
def test_a_step_hands_its_status_word_to_every_product_with_a_bounded_wait(monkeypatch, tmp_path):
    """A prompt of 33 rows in float32 and in bfloat16: whatever product runs, ordinary or in the stream form of its block."""
    from vapi_b200 import LLM, SamplingParams
    from vapi_b200.weights import write_random_model
    cfg = {"architectures": ["Lfm2ForCausalLM"], "model_type": "lfm2", "vocab_size": 4096, "conv_L_cache": 3, "conv_bias": False,
           "rope_theta": 1e6, "norm_eps": 1e-5, "tie_word_embeddings": True, "max_position_embeddings": 256, "num_hidden_layers": 2,
           "layer_types": ["conv", "full_attention"], "hidden_size": 512, "intermediate_size": 3072, "num_attention_heads": 8,
           "num_key_value_heads": 2, "head_dim": 64}
    write_random_model(str(tmp_path), cfg, seed=0, std=0.02, dtype=BF16)
    for dtype, names in (("f32", {"vapi_linear_f32"}), ("bf16", {"vapi_linear_tc"})):
        llm = LLM(str(tmp_path), dtype=dtype, num_blocks=16, max_concurrent_seqs=4, max_batched_tokens=256, max_context=256)
        seen, real = [], ops._lib

        class Watched:
            def __init__(self, lib):
                self.lib = lib

            def __getattr__(self, name):
                f = getattr(self.lib, name)
                if name not in ("vapi_linear_f32", "vapi_linear_tc", "vapi_prompt_linear"):
                    return f
                return lambda *args: (seen.append((name, llm.runner.status.data_ptr() in args)), f(*args))[1]

        monkeypatch.setattr(ops, "_lib", lambda name: Watched(real(name)))
        llm.generate([list(range(33))], SamplingParams(temperature=0.0, max_tokens=1, ignore_eos=True))
        monkeypatch.setattr(ops, "_lib", real)
        assert {n for n, _ in seen} == names and all(held for _, held in seen), seen


# products that had become slower than the library's (short K, a few features), and the edges of the rule; what a model's prompt has stays
@pytest.mark.parametrize("rows,n,k,pays", [(65, 2048, 512, False), (300, 4096, 256, True), (129, 4096, 256, False), (64, 8192, 128, False), (4000, 8192, 128, False),
                                           (1024, 262144, 4, False), (17, 1024, 1024, True), (17, 1024, 1023, False), (64, 64, 16384, True),
                                           (64, 63, 20000, False), (1024, 16, 65536, False), (17, 2048, 2048, True), (57, 2048, 1536, True),
                                           (1024, 16384, 2048, True), (1000, 2052, 512, True), (500, 2200, 512, True), (499, 2200, 512, False)])
def test_the_split_product_takes_what_it_is_faster_at(rows, n, k, pays):
    assert ops.linear_f32_pays(rows, n, k) == pays


def test_the_stream_form_of_prompt_steps_ends_where_it_was_not_measured_to_pay(monkeypatch):
    """More rows than a decode step only with a prompt portion, in models of the measured sizes (LFM2's, of which the average layer is
    counted), and not where the product it rests on is switched off."""
    from conftest import serving_width_config
    from vapi_b200.config.model import resolve_architecture
    for size in ("700m", "1.2b"):
        cfg = serving_width_config(size)
        arch = resolve_architecture(cfg)
        plan = arch.plan(arch.parse(cfg))
        layer = sum(math.prod(s.shape) for b in plan.layers for s in b.tensor_specs("") if s.role == "matrix") // len(plan.layers)
        assert 30_000_000 < layer < 70_000_000 and ops.stream_max_rows(57, layer) == ops.STREAM_PROMPT_MAX_ROWS == 128
    assert ops.stream_max_rows(1, layer) == ops.TC_MAX_ROWS and ops.stream_max_rows(57, 4 * layer) == ops.TC_MAX_ROWS
    monkeypatch.setattr(ops, "TC_MAX_ROWS", 16)
    assert ops.stream_max_rows(57, layer) == 16
    monkeypatch.setattr(ops, "TC_MAX_ROWS", 200)
    assert ops.stream_max_rows(1, layer) == ops.stream_max_rows(57, layer) == 200
    monkeypatch.setattr(ops, "use_tc", False)
    assert ops.stream_max_rows(1, layer) == ops.stream_max_rows(57, layer) == 16


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


@pytest.mark.gpu
def test_large_float32_products_can_be_differentiated_and_mapped():
    """33 rows against a weight of 2^20 numbers: gradients, forward mode and vmap see the product as they see the library's."""
    ops.strict_fp32()
    g = torch.Generator(device="cuda").manual_seed(1)
    x, w, b = (torch.randn(*s, generator=g, device="cuda") for s in ((33, 1024), (1024, 1024), (1024,)))
    assert ops.linear_f32_pays(33, 1024, 1024)
    tol = dict(atol=1e-3, rtol=1e-4)
    xs, ws, bs = (t.clone().requires_grad_() for t in (x, w, b))
    ops.linear(xs, ws, bs).square().sum().backward()
    up = 2 * (x.double() @ w.double().t() + b.double())
    torch.testing.assert_close(xs.grad.double(), up @ w.double(), atol=0.1, rtol=1e-4)
    torch.testing.assert_close(ws.grad.double(), up.t() @ x.double(), atol=0.1, rtol=1e-4)
    torch.testing.assert_close(bs.grad.double(), up.sum(0), atol=0.1, rtol=1e-4)
    with torch.no_grad():
        assert not ops.linear(xs, ws, bs).requires_grad
    value, tangent = torch.func.jvp(lambda t: ops.linear(t, w, b), (x,), (x,))
    torch.testing.assert_close(tangent.double(), x.double() @ w.double().t(), **tol)
    torch.testing.assert_close(torch.vmap(lambda t: ops.linear(t, w))(x.view(1, 33, 1024).repeat(3, 1, 1)).double(),
                               (x.double() @ w.double().t()).repeat(3, 1, 1), **tol)
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(x, x)
        assert torch.autograd.forward_ad.unpack_dual(ops.linear(dual, w)).tangent is not None


def test_traces_dispatch_modes_and_tensor_classes_see_large_float32_products(monkeypatch):
    """What records or replaces the operations of a program finds the library's product, not the empty tensor that a kernel fills."""
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.utils._python_dispatch import TorchDispatchMode

    class Own(torch.Tensor):
        pass

    class Seen(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            names.append(str(func))
            return func(*args, **(kwargs or {}))

    took = []
    monkeypatch.setattr(ops, "_cuda", lambda *t: None)
    monkeypatch.setattr(ops, "skinny_f32_applies", lambda *a: False)
    monkeypatch.setattr(ops, "linear_f32_applies", lambda *a: True)
    monkeypatch.setattr(ops, "linear_f32", lambda x, w, b=None: took.append(1) or x.new_zeros(x.shape[0], w.shape[0]))
    x, y, w = torch.randn(33, 64), torch.randn(33, 64), torch.randn(48, 64)
    want = torch.mm(y, w.t())
    f = lambda t: ops.linear(t, w)
    torch.testing.assert_close(torch.jit.trace(f, (x,), check_trace=False)(y), want)
    torch.testing.assert_close(make_fx(f)(x)(y), want)
    names = []
    with Seen():
        f(x)
    assert any("mm" in n for n in names), names
    assert isinstance(f(x.as_subclass(Own)), Own)
    assert not took
    f(x)
    assert took
