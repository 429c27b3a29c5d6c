"""The native calls of a few-row step (csrc/calls.cpp) against the same steps in Python, which take what those do not."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
BF, F32 = torch.bfloat16, torch.float32


@pytest.fixture
def ops():
    from vapi_b200 import ops
    return ops


def _both(ops, monkeypatch, fn):
    """``fn`` by the native call and without it; what the native call answered goes along."""
    answers = []
    native = ops._calls()

    def counted(name):
        def call(*a):
            answers.append(getattr(native, name)(*a))
            return answers[-1]
        return call

    monkeypatch.setattr(ops, "_calls", lambda: types.SimpleNamespace(product=counted("product"), shortconv=counted("shortconv")))
    a = fn()
    monkeypatch.setattr(ops, "_calls", lambda: types.SimpleNamespace(product=lambda *a: NotImplemented, shortconv=lambda *a: NotImplemented))
    b = fn()
    monkeypatch.setattr(ops, "_calls", lambda: native)
    return a, b, [x is not NotImplemented for x in answers]


def _same(a, b):
    a, b = (x if isinstance(x, tuple) else (x,) for x in (a, b))
    return len(a) == len(b) and all((x is None and y is None) or (x.dtype == y.dtype and torch.equal(x, y)) for x, y in zip(a, b))


@pytest.mark.parametrize("which,M", [("linear_tc", 17), ("linear_tc", 57), ("prompt_linear", 300)])
@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("epilogue", ["bf16", "f32", "swiglu", "resid", "resid alone"])
def test_native_product_is_the_product(ops, monkeypatch, which, M, norm, epilogue):
    g = torch.Generator(device="cuda").manual_seed(M)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    N, K = 384, 136
    w, x, bias, nw, x0 = torch.nn.Parameter(r(N, K).to(BF), requires_grad=False), r(M, K).to(BF), r(N), r(N), r(M, N)
    kw = dict(xw=x, ss_in=r(3, M).square() * K, eps=1e-5) if norm else dict(act=x)
    kw["epilogue"] = epilogue.split()[0]
    if epilogue != "swiglu":
        kw["bias"] = bias
    streams = []

    def run():
        if kw["epilogue"] == "resid":
            streams.append(x0.clone())
            return getattr(ops, which)(w, resid=streams[-1], next_weight=None if "alone" in epilogue else nw, **kw)
        return getattr(ops, which)(w, **kw)

    before = ops.launch_count
    a, b, native = _both(ops, monkeypatch, run)
    assert native == [True] and ops.launch_count == before + 2
    assert _same(a, b) and (not streams or torch.equal(*streams))


@pytest.mark.parametrize("dtype,L,native", [(BF, 3, True), (BF, 1, True), (F32, 3, False)])
def test_native_shortconv_is_the_shortconv(ops, monkeypatch, dtype, L, native):
    g = torch.Generator(device="cuda").manual_seed(L)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    i = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    H, qlens = 40, [1, 5, 2]
    n = sum(qlens)
    h3, state = r(n, 3 * H).to(dtype), r(4, max(L - 1, 1) + 1, H).to(dtype)[:, :L - 1]
    states = []

    def run():
        states.append(state.clone(memory_format=torch.preserve_format))
        return ops.shortconv(h3, r(3 * H) * 0, r(L, H) * 0 + 0.5, None, states[-1] if L > 1 else None, i([2, 0, 3]),
                             i([0, 1, 1, 1, 1, 1, 2, 2]), i([0, 1, 6, 8]), i([4, 0, 1, 2, 3, 4, 1, 2]))

    a, b, taken = _both(ops, monkeypatch, run)
    assert taken == [native] and _same(a, b) and torch.equal(*states)


def test_what_the_native_product_does_not_take_is_refused_or_done_as_before(ops):
    w, x = torch.randn(64, 32, device="cuda").to(BF), torch.randn(20, 32, device="cuda").to(BF)
    for bad in (dict(act=x[:, :16]), dict(act=x.float()), dict(xw=x), dict(act=x, bias=torch.ones(63, device="cuda")), dict(act=x, epilogue="none"),
                dict(act=x, epilogue="resid", resid=torch.zeros(20, 63, device="cuda")), dict(act=x, glu="none"), dict(act=x.cpu())):
        with pytest.raises(ops.KernelError):
            ops.linear_tc(w, **bad)
    with pytest.raises(ops.KernelError):
        ops.linear_tc(w.t(), act=x)
    with pytest.raises(ops.KernelError, match="more than 256"):          # (the C function's own refusal)
        ops.linear_tc(w, act=torch.zeros(257, 32, device="cuda", dtype=BF))

    for n, k in ((0, 32), (64, 0)):                                      # (and products of nothing)
        with pytest.raises(ops.KernelError, match="positive"):
            ops.linear_tc(torch.zeros(n, k, device="cuda", dtype=BF), act=torch.zeros(20, k, device="cuda", dtype=BF), epilogue="resid",
                          resid=torch.zeros(20, n, device="cuda"), next_weight=torch.ones(n, device="cuda"))

    class Other(torch.Tensor):
        pass

    assert torch.equal(ops.linear_tc(w, act=x.as_subclass(Other)).as_subclass(torch.Tensor), ops.linear_tc(w, act=x))


def test_a_call_that_has_been_made_is_not_made_again(ops, tmp_path):
    """An exception out of the C function is an error: ``NotImplemented`` would send the caller through the same call once more, which
    adds to the stream, or moves a state on, twice.  (The function here launches nothing.)"""
    import ctypes
    import subprocess
    from vapi_b200.csrc import build
    src = tmp_path / "throws.cpp"
    src.write_text('#include <new>\n#include <stdexcept>\nextern "C" { int calls = 0; int plan(int, int, int, int, int* a, int* b, int* c) { *a = *b = *c = 1; return 0; }\n'
                   'int memory() { ++calls; throw std::bad_alloc(); }\nint other() { ++calls; throw 1; } }\n')
    subprocess.run([build.find_cxx(), "-shared", "-fPIC", "-o", str(tmp_path / "libthrows.so"), str(src)], check=True)
    lib = ctypes.CDLL(str(tmp_path / "libthrows.so"))
    at = lambda fn: ctypes.cast(getattr(lib, fn), ctypes.c_void_p).value
    w, x, resid = torch.zeros(64, 32, device="cuda", dtype=BF), torch.zeros(20, 32, device="cuda", dtype=BF), torch.zeros(20, 64, device="cuda")
    i = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")
    h3, state = torch.zeros(1, 24, device="cuda", dtype=BF), torch.zeros(1, 2, 8, device="cuda", dtype=BF)
    for n, (fn, text) in enumerate((("memory", "bad_alloc"), ("other", "unknown"))):
        with pytest.raises(RuntimeError, match=text):
            ops._calls().product(at(fn), at("plan"), 0, w, x, None, None, 0.0, 2, None, resid, torch.ones(64, device="cuda"), None, None, 0, None)
        with pytest.raises(RuntimeError, match=text):
            ops._calls().shortconv(at(fn), h3, None, torch.zeros(3, 8, device="cuda"), None, state, i(0), i(0), i(0, 1), i(0), None, None)
        assert ctypes.c_int.in_dll(lib, "calls").value == 2 * n + 2
    assert ops._calls().product(at("memory"), at("plan"), 0, w.float(), x, None, None, 0.0, 2, None, resid, None, None, None, 0, None) is NotImplemented
    assert ctypes.c_int.in_dll(lib, "calls").value == 4


@pytest.mark.parametrize("native", [True, False])
def test_operands_that_are_too_short_are_refused(ops, monkeypatch, native):
    """Every vector is at least as long as what the kernels read of it, by the native calls and by the same steps in Python."""
    if not native:
        monkeypatch.setattr(ops, "_calls", lambda: ops._NoCalls)
    f = lambda *s: torch.zeros(*s, device="cuda")
    i = lambda *v: torch.tensor(v, dtype=torch.int32, device="cuda")
    w, x = f(64, 32).to(BF), f(20, 32).to(BF)
    for which in (ops.linear_tc, ops.prompt_linear, lambda *a, act, resid=None, **kw: ops.skinny_linear(*a, act=act[:16], resid=None if resid is None else resid[:16], **kw)):
        with pytest.raises(ops.KernelError, match="norm weight"):
            which(w, act=x, epilogue="resid", resid=f(20, 64), next_weight=f(63))
        with pytest.raises(ops.KernelError, match="activation"):
            which(w, act=x, xielu=f(1))
    with pytest.raises(ops.KernelError, match="activation"):
        ops.xielu(x, f(1))
    good = dict(h3=f(3, 24).to(BF), in_bias=f(24), taps=f(3, 8), conv_bias=f(8), state_layer=f(2, 2, 8).to(BF), state_slots=i(0, 1),
                tok_seq=i(0, 0, 1), cu_q=i(0, 2, 3), positions=i(0, 1, 4))
    assert ops.shortconv(**good).shape == (3, 8)
    for key, short in (("in_bias", f(23)), ("conv_bias", f(7)), ("state_slots", i(0)), ("tok_seq", i(0, 0)), ("positions", i(0, 1)),
                       ("state_slots", None), ("positions", None)):
        with pytest.raises(ops.KernelError):
            ops.shortconv(**{**good, key: short})
    assert ops.shortconv(**{**good, "taps": f(1, 8), "state_layer": None, "state_slots": None, "positions": None}).shape == (3, 8)
    # (longer ones are taken, as before)
    assert ops.shortconv(**{**good, "in_bias": f(30), "positions": i(0, 1, 4, 5)}).shape == (3, 8)


def test_tensor_maps_are_kept_for_weights_and_not_for_tokens(ops):
    """Prompts at other addresses leave the table of kept maps as it is (a weight has one map for each tile that its products use)."""
    maps, counts, alive = ops._lib("linear_prompt").vapi_prompt_linear_maps, [], []
    w = torch.zeros(256, 64, device="cuda", dtype=BF)
    for _ in range(2):
        for n in (33, 130, 131, 257, 300, 301, 1000):
            alive.append(torch.zeros(n, 64, device="cuda", dtype=BF))
            assert ops.prompt_linear(w, act=alive[-1]).shape == (n, 256)
        counts.append(maps())
    assert counts[0] == counts[1] >= 1
