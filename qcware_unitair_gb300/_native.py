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
import warnings

from . import build_lib

NAMES = ("apply_operator", "apply_layer", "apply_phase", "norm_squared",
         "abs_squared", "inner_product", "diag_expectation_value",
         "rotation", "dense")

_lock = threading.Lock()


def load():
    """Load the module and bind its functions here; raises if it is not
    built, or not for this torch and interpreter."""
    with _lock:
        path, tag = build_lib.host_path(), build_lib.host_tag_path()
        again = ("run `python -c 'import __graft_entry__ as g; g.build()'` or "
                 "`python -m qcware_unitair_gb300.build_lib`.")
        if not path.exists():
            raise RuntimeError(f"{path.name} is not built ({path}); {again}")
        built = tag.read_text() if tag.exists() else "an earlier version"
        if built != build_lib.host_tag():
            raise RuntimeError(f"{path.name} was built for {built}, this is "
                               f"{build_lib.host_tag()}; {again}")
        spec = importlib.util.spec_from_file_location(
            build_lib.HOST_MODULE, path)
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
        for name in NAMES:
            globals()[name] = getattr(mod, name)
        return mod


def _nothing(*args):
    return None


def _load_or_leave():
    """Load the module; where that fails, leave every call to the Python
    functions, which launch the same kernels (libgbsv.so does not depend on
    torch), and say so once."""
    try:
        load()
    except (RuntimeError, ImportError, OSError) as e:
        warnings.warn(f"the native host path is off, calls take longer on the "
                      f"host: {e}", RuntimeWarning, stacklevel=4)
        for name in NAMES:
            globals()[name] = _nothing


def _unloaded(name):
    def call(*args):
        if any(getattr(a, "is_cuda", False) for a in args):
            _load_or_leave()
            return globals()[name](*args)
        return None
    return call


for _name in NAMES:
    globals()[_name] = _unloaded(_name)
