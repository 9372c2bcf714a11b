"""Loader of ``_ccl_ops.so``: the host code of ``oneccl_b200.ops`` in C++ (autograd functions, allocation of outputs and
scratch, calls into ``libccl_b200.so``), built in-tree by ``oneccl_b200._build``."""
from __future__ import annotations

import importlib.util
import sys
from pathlib import Path

_EXT = None


def native():
    """The extension module; raises if it cannot be built (there is no Python fallback of it)."""
    global _EXT
    if _EXT is None:
        import torch  # noqa: F401  (its libraries must be loaded first)

        from .. import _lib

        _lib.load()  # libccl_b200.so: the extension links against it
        path = Path(__file__).resolve().parent.parent / "lib" / "_ccl_ops.so"
        if not path.exists():
            from .. import _build

            _build.build_torch_ops()
        spec = importlib.util.spec_from_file_location("_ccl_ops", str(path))
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
        sys.modules["_ccl_ops"] = mod
        _EXT = mod
    return _EXT
