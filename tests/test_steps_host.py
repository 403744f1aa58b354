"""Which native module of the generation step is loaded (no GPU: nothing of it is called)."""

import sysconfig

import pytest
import torch

from kempnerforge_b200.ops import build, cuda


def test_the_module_is_named_after_what_it_was_built_for():
    """Another PyTorch has another C++ interface: a module of an older one must not be found."""
    assert sysconfig.get_config_var("SOABI") in build.STEPS_PATH.name and torch.__version__ in build.STEPS_PATH.name


def test_without_a_module_the_step_is_left_to_python(monkeypatch, tmp_path):
    monkeypatch.setattr(cuda, "_steps", None)
    monkeypatch.setattr(cuda, "STEPS_PATH", tmp_path / "kf_steps.so")
    monkeypatch.setattr(cuda.importlib.util, "spec_from_file_location", lambda *a: pytest.fail("there is nothing to load"))
    for _ in range(2):
        assert cuda.blocks_decode([object()], [object()], torch.zeros(1, 1, 8), torch.zeros(1, 4), torch.zeros(1, 4)) is None
