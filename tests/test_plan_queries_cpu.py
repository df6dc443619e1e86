"""What a launch would do can be asked for without a device."""
import pytest


def test_queries_without_a_device():
    from neuronx_distributed_b200.ops import _ext

    e = _ext._load()
    if e is None:
        pytest.skip("extension not built")
    assert e.gemm_2cta_workspace(1000, 5112, 2504, True, False) >= 0 and e.gemm_2cta_workspace(0, 0, 0, True, False) == 0
    assert e.flash_attn_bwd_parts(1, 128, 128, 8, 0, True) == 1 and e.flash_attn_bwd_parts(0, 0, 0, 0, 0, False) == 1
    assert 8 // 2 % e.flash_attn_bwd_parts(1, 512, 512, 8, 2, True) == 0
