"""Loads the operator library so that ``torch.ops.npu.npu_*`` resolve, and its short-cut calls (``calls()``).

No fallback exists: if ``lib/libop_plugin_b200.so`` is missing this raises and
tells how to build it.
"""
from __future__ import annotations

import importlib.util
from importlib.machinery import ExtensionFileLoader
from pathlib import Path

import torch

_PKG = Path(__file__).resolve().parent
PLUGIN_PATH = _PKG / "lib" / "libop_plugin_b200.so"
_loaded = False
_calls = None


def load():
    global _loaded
    if not _loaded:
        if not PLUGIN_PATH.exists():
            raise RuntimeError(f"{PLUGIN_PATH} is not built; run `python {_PKG / 'build.py'}` "
                               "(there is no fallback implementation)")
        from . import capi

        capi.lib()  # RTLD_GLOBAL: the plugin resolves qmm_* from it
        torch.ops.load_library(str(PLUGIN_PATH))
        _loaded = True
    return torch.ops.npu


def calls():
    """The library as a Python module: operators called by position, without schema matching.  A call that it leaves to
    ``torch.ops`` returns ``NotImplemented``."""
    global _calls
    if _calls is None:
        load()
        loader = ExtensionFileLoader("libop_plugin_b200", str(PLUGIN_PATH))
        spec = importlib.util.spec_from_file_location("libop_plugin_b200", PLUGIN_PATH, loader=loader)
        module = importlib.util.module_from_spec(spec)
        loader.exec_module(module)
        _calls = module
    return _calls
