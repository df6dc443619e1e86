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


def _caches(offset=0, batch=0, row=0, head=0, heads=2, sequences=2):
    """k and v [sequences, 5, heads, 128] in one buffer, their first element, batch, row and head strides off by so many elements."""
    import torch

    sh, ss = 128 + head, heads * (128 + head) + row
    sb = 5 * ss + batch
    buffer = torch.zeros(2 * (sequences * sb + offset) + 64, dtype=torch.bfloat16)
    assert buffer.data_ptr() % 16 == 0
    return [buffer.as_strided((sequences, 5, heads, 128), (sb, ss, sh, 1), offset + i * (sequences * sb // 8 * 8)) for i in range(2)]


@pytest.mark.parametrize("group", range(1, 9))
def test_caches_that_the_token_kernel_takes(group):
    """It copies 16-byte packets: every address has to be a multiple of one, whatever the group."""
    import torch

    from neuronx_distributed_b200 import ops

    if ops._ext._load() is None:
        pytest.skip("extension not built")
    ok = ops.attention.decode_group_ok
    q = torch.zeros(2, 1, 2 * group, 128, dtype=torch.bfloat16)
    assert ok(q, *_caches()) and ok(q, *_caches(offset=8, batch=8, row=16, head=24))
    for off in ({"offset": 1}, {"offset": 4}, {"batch": 4}, {"row": 2}, {"head": 4}):
        assert not ok(q, *_caches(**off)), off
        aligned = _caches()
        assert not ok(q, aligned[0], _caches(**off)[1]) and not ok(q, _caches(**off)[0], aligned[1]), off
    one = q[:1, :, :group]
    assert ok(one, *_caches(batch=3, head=5, row=3, heads=1, sequences=1))                   # strides 128 + 5 + 3 a row; others lead nowhere
    odd = torch.zeros(q.numel() + 1, dtype=torch.bfloat16)[1:].view(q.shape)                 # queries are read in words
    assert not ok(odd, *_caches()) and not ok(torch.zeros(2, 1, 2 * group + 1, 128, dtype=torch.bfloat16), *_caches())


def test_groups_of_more_than_eight_heads_go_the_general_way():
    import torch

    from neuronx_distributed_b200 import ops

    if ops._ext._load() is None:
        pytest.skip("extension not built")
    assert not ops.attention.decode_group_ok(torch.zeros(2, 1, 18, 128, dtype=torch.bfloat16), *_caches())


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_views_of_whole_packets(dtype):
    """What the library's attention gets as it is: rows at multiples of 16 bytes; strides of dimensions of one don't count."""
    import torch

    from neuronx_distributed_b200 import ops

    ok, per = ops.attention.whole_packets, 16 // getattr(torch, dtype).itemsize
    t = torch.zeros(2 * 3 * 5 * 144 + 16, dtype=getattr(torch, dtype))
    assert t.data_ptr() % 16 == 0

    def view(shape=(2, 3, 5, 128), strides=(3 * 5 * 144, 5 * 144, 144, 1), offset=0):
        return t.as_strided(shape, strides, offset)

    assert ok(view()) and ok(view(offset=per)) and ok(view().transpose(1, 2)) and ok(view((1, 3, 1, 128), (3, 144, 7, 1)))
    assert not ok(view(offset=1)) and not ok(view(offset=per // 2)) and not ok(view(strides=(3 * 5 * 144, 5 * 144, 128 + per // 2, 1)))
    assert not ok(view(strides=(3 * 5 * 144 - 1, 5 * 144, 144, 1))) and not ok(view().transpose(2, 3))
