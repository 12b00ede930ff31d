"""When the native host path is built again."""
import torch

import nanochat_cpp_b200 as nc
from nanochat_cpp_b200 import build


def test_the_extension_is_stale_for_another_torch(monkeypatch):
    assert nc.engine.native.built_for == build._built_for()
    assert not build._engine_stale()
    monkeypatch.setattr(torch, "__version__", "0.0.1+none")
    assert build._engine_stale()
