"""What the package does where ``csrc/calls.cpp``, the one source that it can do without, cannot be built; plans of products of nothing."""
import warnings

import pytest

from vapi_b200 import ops
from vapi_b200.csrc import build


def _failing(name):
    def fake(n, verbose=True):
        if n == name:
            raise build.BuildError(f"no headers for {n}")
        return f"lib{n}.so"
    return fake


def test_the_build_goes_on_without_the_native_calls(monkeypatch):
    monkeypatch.setattr(build, "build", _failing("calls"))
    with pytest.warns(UserWarning, match="no headers for calls"):
        built = build.build_all(verbose=False)
    assert sorted(built) == [n for n in build.sources() if n != "calls"]


def test_a_kernel_that_cannot_be_built_is_an_error(monkeypatch):
    monkeypatch.setattr(build, "build", _failing("rope"))
    with pytest.raises(build.BuildError, match="no headers for rope"):
        build.build_all(verbose=False)


def test_calls_that_cannot_be_built_are_answered_with_not_implemented(monkeypatch):
    monkeypatch.setattr(build, "build", _failing("calls"))
    monkeypatch.setattr(ops, "_calls_module", None)
    with pytest.warns(UserWarning, match="launched from Python"):
        calls = ops._calls()
    with warnings.catch_warnings():
        warnings.simplefilter("error")                       # (said once)
        assert ops._calls() is calls
    assert calls.product(*range(16)) is NotImplemented and calls.shortconv(*range(12)) is NotImplemented


@pytest.mark.parametrize("N,K,epi", [(0, 64, 2), (64, 0, 2), (0, 0, 0), (1, 8, 1)])
def test_a_product_of_nothing_has_a_plan(N, K, epi):
    """The outputs are laid out by the plan before the call refuses such a product: no division by its tiles or its K."""
    assert ops._tc_plan.__wrapped__(N, K, 20, epi)[:2] == ((N + 127) // 128 if epi != 1 else (N // 2 + 63) // 64, 1)
