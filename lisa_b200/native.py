"""``lib/_lisa_torch.so``, the compiled host side of ``lisa_b200.ops`` (csrc/torch_ops.cpp), loaded at the first call: the
package can be imported, and its build run, before the library exists or while an older one lies in its place."""
from __future__ import annotations

import importlib.machinery
import importlib.util
import os

import torch  # noqa: F401  (the module links against its libraries)

from . import _cabi

PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), "lib", "_lisa_torch.so")


def _load():
    if not os.path.exists(PATH):
        raise RuntimeError(f"{PATH} is missing: build the CUDA library with `python -m lisa_b200.build` (there is no CPU fallback)")
    _cabi.lib()  # liblisa_cuda.so first: both use the same copy of it
    loader = importlib.machinery.ExtensionFileLoader("_lisa_torch", PATH)
    module = importlib.util.module_from_spec(importlib.util.spec_from_loader("_lisa_torch", loader))
    loader.exec_module(module)
    module.set_error_class(_cabi.LisaError)
    return module


class _Extension:
    """The module's functions as attributes; the first access loads it and keeps all of them."""

    def __getattr__(self, name):
        if name.startswith("__"):
            raise AttributeError(name)
        module = _load()
        self.__dict__.update((k, v) for k, v in vars(module).items() if not k.startswith("__"))
        return getattr(module, name)


ext = _Extension()
