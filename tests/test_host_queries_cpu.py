"""What a launch would do can be asked for without a device; switches are read from the environment as it is."""
import os

import pytest


def test_queries_without_a_device():
    from neuronx_distributed_b200.ops import _ext

    e = _ext._load()
    if e is None:
        pytest.skip("extension not built")
    assert e.gemm_2cta_workspace(1000, 5112, 2504, True, False) >= 0 and e.gemm_2cta_workspace(0, 0, 0, True, False) == 0
    assert e.flash_attn_bwd_parts(1, 128, 128, 8, 0, True) == 1 and e.flash_attn_bwd_parts(0, 0, 0, 0, 0, False) == 1
    assert 8 // 2 % e.flash_attn_bwd_parts(1, 512, 512, 8, 2, True) == 0


def test_switches_follow_the_environment(monkeypatch):
    from neuronx_distributed_b200.ops import _ext

    monkeypatch.delenv("NXD_SOME_SWITCH", raising=False)
    assert _ext.env("NXD_SOME_SWITCH") == "" and _ext.env("NXD_SOME_SWITCH", "x") == "x"
    monkeypatch.setenv("NXD_SOME_SWITCH", "1")
    assert _ext.env("NXD_SOME_SWITCH") == "1"
    monkeypatch.setattr(os, "environ", {"NXD_SOME_SWITCH": "2"})
    assert _ext.env("NXD_SOME_SWITCH") == "2" and _ext.env("NXD_OTHER", "y") == "y"
