"""Loads the operator library so that ``torch.ops.npu.npu_*`` resolve, and its short-cut calls (``calls()``).

No fallback exists: if a library under ``lib/`` is missing this raises and
tells how to build it.
"""
from __future__ import annotations

import importlib.util
from importlib.machinery import ExtensionFileLoader
from pathlib import Path

import torch

_PKG = Path(__file__).resolve().parent
PLUGIN_PATH = _PKG / "lib" / "libop_plugin_b200.so"
CALLS_PATH = _PKG / "lib" / "_op_plugin_calls.so"
_loaded = False
_calls = None


def _require(path):
    if not path.exists():
        raise RuntimeError(f"{path} is not built; run `python {_PKG / 'build.py'}` "
                           "(there is no fallback implementation)")


def load():
    global _loaded
    if not _loaded:
        _require(PLUGIN_PATH)
        from . import capi

        capi.lib()  # RTLD_GLOBAL: the plugin resolves qmm_* from it
        torch.ops.load_library(str(PLUGIN_PATH))
        _loaded = True
    return torch.ops.npu


def calls():
    """A Python module beside the library: operators called by position, without schema matching.  A call that it leaves to
    ``torch.ops`` returns ``NotImplemented``."""
    global _calls
    if _calls is None:
        load()
        _require(CALLS_PATH)
        loader = ExtensionFileLoader("_op_plugin_calls", str(CALLS_PATH))
        spec = importlib.util.spec_from_file_location("_op_plugin_calls", CALLS_PATH, loader=loader)
        module = importlib.util.module_from_spec(spec)
        loader.exec_module(module)
        _calls = module
    return _calls
