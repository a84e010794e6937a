"""The native half of the wrappers is an extra: without it, or with one that does not fit, calls go through Python."""
from __future__ import annotations

import logging
import types

import pytest

from comfy_kitchen.backends import cuda as backend


class _Library:
    """A library of which one entry point may be missing."""

    def __init__(self, missing=None):
        self._missing = missing

    def __getattr__(self, name):
        if name == self._missing:
            raise AttributeError(f"undefined symbol: {name}")
        return backend.ctypes.CFUNCTYPE(None)(0)


@pytest.fixture
def built(monkeypatch, tmp_path):
    """Whatever this machine has built, a file that loads as an extension whose bind() is given; no native half is bound."""
    (tmp_path / "lib").mkdir()
    (tmp_path / "lib" / "_ck_host.so").touch()
    monkeypatch.setattr(backend, "_PKG_ROOT", str(tmp_path))
    monkeypatch.setattr(backend, "_host", None)

    def loads(bind):
        class Loader:
            def __init__(self, name, path):
                pass

            def create_module(self, spec):
                return types.SimpleNamespace(bind=bind)

            def exec_module(self, module):
                pass

        monkeypatch.setattr(backend.importlib.machinery, "ExtensionFileLoader", Loader)

    return loads


def _refused(addresses, parameter):
    raise ValueError("bind: an entry point is missing")


@pytest.mark.parametrize("library, bind", [(_Library("ck_dequantize_mxfp8"), lambda *a: None), (_Library(), _refused)])
def test_an_extension_that_does_not_fit_is_left_out(built, caplog, library, bind):
    built(bind)
    with caplog.at_level(logging.WARNING, logger="comfy_kitchen"):
        backend._load_host(library)
    assert backend._host is None and len(caplog.messages) == 1 and "Python wrappers" in caplog.messages[0]


def test_one_that_fits_is_bound(built, caplog):
    got = []
    built(lambda *a: got.append(a))
    backend._load_host(_Library())
    ((addresses, parameter),) = got
    assert backend._host is not None and set(addresses) == set(backend._HOST_NAMES) and parameter is backend.torch.nn.Parameter
    assert not caplog.messages


def test_a_file_that_is_no_extension_is_left_out(monkeypatch, tmp_path, caplog):
    (tmp_path / "lib").mkdir()
    (tmp_path / "lib" / "_ck_host.so").write_bytes(b"no ELF")
    monkeypatch.setattr(backend, "_PKG_ROOT", str(tmp_path))
    monkeypatch.setattr(backend, "_host", None)
    with caplog.at_level(logging.WARNING, logger="comfy_kitchen"):
        backend._load_host(_Library())
    assert backend._host is None and len(caplog.messages) == 1
