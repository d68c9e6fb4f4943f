"""Where the native host side of the router operators is missing or was built for another torch, the
Python operators take every call, with one warning; no kernel is launched here."""
import sys
import types
import warnings

import pytest


@pytest.fixture
def lib(monkeypatch):
    from brainstorm_b200 import _lib, build

    build.build()
    monkeypatch.setattr(_lib, "_host", None)
    return _lib


@pytest.mark.parametrize("kind", ["missing", "another torch"])
def test_the_python_operators_take_over(lib, monkeypatch, kind):
    import brainstorm_b200

    module = None  # import raises ImportError
    if kind == "another torch":
        module = types.SimpleNamespace(torch_version="1.0.0", scan=lambda *args: 1 / 0)
    monkeypatch.setitem(sys.modules, "brainstorm_b200._host_ops", module)
    monkeypatch.delattr(brainstorm_b200, "_host_ops", raising=False)
    with pytest.warns(RuntimeWarning, match="_host_ops.so"):
        ops = lib.host_ops()
    for name in ("scan", "route_scores", "dispatch", "combine"):
        assert getattr(ops, name)(None, 1, "any") is None
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert lib.host_ops() is ops


def test_the_module_that_was_built_is_used(lib):
    import torch

    with warnings.catch_warnings():
        warnings.simplefilter("error")
        ops = lib.host_ops()
    assert ops.__name__.endswith("_host_ops")
    assert ops.torch_version == torch.__version__.split("+")[0]


def test_another_torch_makes_it_stale(lib):
    import torch
    from brainstorm_b200 import build

    assert not build._host_stale(torch.__version__)
    assert build._host_stale(torch.__version__ + ".post1")
