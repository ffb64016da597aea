"""The host extension belongs to one Python and one torch: another version of either neither finds nor loads it."""

import sys

import torch

from nano_vllm_jax_b200 import _lib, build


def test_another_torch_or_python_has_another_file(monkeypatch):
    here = build.host_path()
    monkeypatch.setattr(torch, "__version__", "0.1.2+other")
    other = build.host_path()
    monkeypatch.setattr(sys.implementation, "cache_tag", "cpython-399")
    assert len({here, other, build.host_path()}) == 3


def test_a_change_of_version_builds_instead_of_loading_the_old_file(monkeypatch, tmp_path):
    assert _lib.host_module().__file__ == str(build.host_path())
    old = build.host_path()

    class Built(Exception):
        pass

    def build_host(force=False):
        raise Built

    monkeypatch.setattr(torch, "__version__", "0.1.2+other")
    monkeypatch.setattr(build, "build_host", build_host)
    monkeypatch.setattr(_lib, "_host", None)
    try:
        _lib.host_module()
    except Built:
        pass
    else:
        raise AssertionError(f"{old.name} was loaded under another torch")
