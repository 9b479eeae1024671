"""Without the native host side, or with one of another torch, the Python route has every layer call."""
import warnings

import pytest

from spiky_b200 import _native, lut_layer


@pytest.fixture
def fresh(monkeypatch):
    monkeypatch.setattr(lut_layer, "_layer_call", lut_layer._first_layer_call)
    monkeypatch.setattr(_native, "_layer_calls", None)
    return monkeypatch


def check_python_route():
    with pytest.warns(RuntimeWarning, match="Python route"):
        assert lut_layer._layer_call(None, None) is None
    with warnings.catch_warnings():
        warnings.simplefilter("error")   # said once
        assert lut_layer._layer_call(None, None) is None


def test_missing(fresh, tmp_path):
    fresh.setattr(_native, "LAYER_CALLS_PATH", str(tmp_path / "none.so"))
    check_python_route()


def test_not_loadable(fresh, tmp_path):
    path = tmp_path / "_layer_calls.so"
    path.write_bytes(b"not a library")
    fresh.setattr(_native, "LAYER_CALLS_PATH", str(path))
    check_python_route()


def test_of_another_torch(fresh):
    import torch

    fresh.setattr(torch, "__version__", "1.2.3")
    check_python_route()
    fresh.undo()
    assert _native.layer_calls().torch_version == torch.__version__.split("+")[0]
