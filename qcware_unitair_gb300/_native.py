"""The native host path (csrc/host/host.cpp): the ordinary call of the
functions that circuit loops are made of, with its checks, allocation, launch
and autograd node in C++.  Each function returns None for a call it leaves to
the Python function of the same name.

The module is built beside libgbsv.so and loaded at the first call with a
CUDA tensor; a call with CPU tensors alone never needs it (the Python
functions reject those)."""
from __future__ import annotations

import importlib.util
import threading

from . import build_lib

NAMES = ("apply_operator", "apply_layer", "apply_phase", "norm_squared",
         "abs_squared", "inner_product", "diag_expectation_value",
         "rotation")

_lock = threading.Lock()


def load():
    """Load the module and bind its functions here; raises if it is not
    built."""
    with _lock:
        path = build_lib.host_path()
        if not path.exists():
            raise RuntimeError(
                f"{path.name} is not built ({path}); run `python -c 'import "
                "__graft_entry__ as g; g.build()'` or `python -m "
                "qcware_unitair_gb300.build_lib`.  The engine has no CPU "
                "fallback.")
        spec = importlib.util.spec_from_file_location(
            build_lib.HOST_MODULE, path)
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
        for name in NAMES:
            globals()[name] = getattr(mod, name)
        return mod


def _unloaded(name):
    def call(*args):
        if any(getattr(a, "is_cuda", False) for a in args):
            return getattr(load(), name)(*args)
        return None
    return call


for _name in NAMES:
    globals()[_name] = _unloaded(_name)
