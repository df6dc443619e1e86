"""Loader for the in-tree sm_100a extension ``nxd_b200_C``.

The extension is built IN-TREE (``neuronx_distributed_b200/_build/nxd_b200_C.so``) by
``__graft_entry__.build()`` / ``python -m neuronx_distributed_b200.ops.build`` so that it travels
with the source snapshot to GPU boxes.  On a machine with a GPU the CUDA path is the one that
runs: if the extension cannot be loaded there, ops raise instead of silently falling back
(set ``NXD_ALLOW_EAGER_FALLBACK=1`` to override, e.g. for debugging).
"""
from __future__ import annotations

import importlib.machinery
import importlib.util
import os
import sys
from pathlib import Path
from typing import Optional

import torch
from torch.autograd import forward_ad

PKG_DIR = Path(__file__).resolve().parent.parent
BUILD_DIR = PKG_DIR / "_build"
EXT_NAME = "nxd_b200_C"

_C = None
_PLAN_PROXY = None          # set by inference.launch_plan.record(): kernel calls are recorded through it
_LOAD_ERROR: Optional[BaseException] = None
_TRIED = False


def _load():
    global _C, _LOAD_ERROR, _TRIED
    if _TRIED:
        return _C
    _TRIED = True
    so = BUILD_DIR / f"{EXT_NAME}.so"
    if not so.exists():
        _LOAD_ERROR = FileNotFoundError(f"{so} not built; run `python -m neuronx_distributed_b200.ops.build`")
        return None
    try:
        loader = importlib.machinery.ExtensionFileLoader(EXT_NAME, str(so))
        spec = importlib.util.spec_from_loader(EXT_NAME, loader)
        mod = importlib.util.module_from_spec(spec)
        loader.exec_module(mod)
        sys.modules[EXT_NAME] = mod
        _C = mod
    except BaseException as e:  # pragma: no cover - depends on box
        _LOAD_ERROR = e
        _C = None
    return _C


def ext():
    """The extension module or ``None``."""
    if _PLAN_PROXY is not None:
        return _PLAN_PROXY
    return _load()


def load_error() -> Optional[BaseException]:
    _load()
    return _LOAD_ERROR


_OS_ENVIRON = os.environ
_ENVIRON = getattr(os.environ, "_data", None)      # POSIX: the dict behind os.environ (bytes to bytes)


def env(name: str, default: str = "") -> str:
    """``os.environ.get`` for switches that are read on every call: a look into the dict behind it (a missing key costs
    ``os.environ`` an encoded copy of the name and an exception, about 1 us, a hundred times in a training step)."""
    if _ENVIRON is None or os.environ is not _OS_ENVIRON:      # another mapping has been put in its place
        return os.environ.get(name, default)
    key = _ENV_KEYS.get(name)
    if key is None:
        key = _ENV_KEYS[name] = os.environ.encodekey(name)
    v = _ENVIRON.get(key)
    return default if v is None else os.environ.decodevalue(v)


_ENV_KEYS: dict = {}


def use_cuda(*tensors: torch.Tensor) -> bool:
    """True when the hand-written kernels must handle these tensors.

    CPU tensors → False (reference math).  CUDA tensors → True if the extension loaded; if
    it did not, raise loudly unless the eager fallback is explicitly allowed."""
    if not tensors:
        return False
    for t in tensors:
        if not (isinstance(t, torch.Tensor) and t.is_cuda):
            return False
    if env("NXD_FORCE_EAGER") == "1":
        return False
    if _load() is not None:
        return True
    if os.environ.get("NXD_ALLOW_EAGER_FALLBACK", "0") == "1":
        return False
    raise RuntimeError(
        f"CUDA tensors given but the sm_100a extension is not loaded ({_LOAD_ERROR!r}). "
        "Build it with `python -m neuronx_distributed_b200.ops.build` or set NXD_ALLOW_EAGER_FALLBACK=1."
    )


_PLAIN = (torch.Tensor, torch.nn.Parameter)


def native(*tensors: torch.Tensor):
    """The autograd nodes of ``csrc/native_autograd.cpp`` where they may stand in for the Functions in Python: plain CUDA tensors, calls
    that nobody records or traces, no functorch transform, no forward-mode AD; else ``None``."""
    if _PLAN_PROXY is not None:
        return None
    for t in tensors:
        if type(t) not in _PLAIN or not t.is_cuda:
            return None
    if (_load() is None or env("NXD_FORCE_EAGER") == "1" or torch._C._are_functorch_transforms_active()
            or torch._C._get_tracing_state() is not None or forward_ad._current_level >= 0):
        return None
    return _C.native


# launch accounting — bench.py reports how many of OUR kernels ran in the timed region
_LAUNCHES = 0


def count_launch(n: int = 1) -> None:
    global _LAUNCHES
    _LAUNCHES += n


def launches() -> int:
    return _LAUNCHES + (_C.native.launches() if _C is not None else 0)


def reset_launches() -> None:
    global _LAUNCHES
    _LAUNCHES = -(_C.native.launches() if _C is not None else 0)
