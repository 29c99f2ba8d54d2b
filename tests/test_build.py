"""CPU: when the binding of the layer API is built again."""
import os

import torch

from hesper_b200 import build


def test_binding_is_stale_after_another_torch_or_a_change_of_its_sources(monkeypatch, tmp_path):
    so, tag = tmp_path / "_binding.so", tmp_path / "_binding.tag"
    monkeypatch.setattr(build, "BINDING", str(so))
    monkeypatch.setattr(build, "BINDING_TAG", str(tag))
    assert build.binding_stale()  # not there
    so.write_bytes(b"")
    assert build.binding_stale()  # built by something that left no tag
    tag.write_text(build._binding_tag())
    assert not build.binding_stale()
    os.utime(so, (0, 0))
    assert build.binding_stale()  # older than its sources
    os.utime(so)
    monkeypatch.setattr(torch, "__version__", "0.0.0")
    assert build.binding_stale()
