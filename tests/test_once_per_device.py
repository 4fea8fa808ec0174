"""A kernel's shared-memory permission is asked for on every device, and again
after a failure (once.h, compiled for the host); no launch keeps it in a
static of its own, which one device's success would satisfy for all."""
import ctypes
import re
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "qcware_unitair_gb300" / "csrc"


def test_devices_and_failures(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    out = tmp_path / "libonce.so"
    subprocess.run([cxx, "-O2", "-std=c++17", "-shared", "-fPIC",
                    f"-I{CSRC}", str(HERE / "native" / "once_host.cpp"),
                    "-o", str(out)], check=True)
    lib = ctypes.CDLL(str(out))
    for dev in (0, 1, 63):
        assert lib.once_run(dev, 0) == 0 and lib.once_run(dev, 0) == 0
        assert lib.once_calls(dev) == 1
    assert lib.once_run(2, 7) == 7 and lib.once_run(2, 0) == 0
    assert lib.once_run(2, 0) == 0 and lib.once_calls(2) == 2
    # beyond the mask: every time, never another device's
    assert lib.once_run(64, 0) == 0 and lib.once_run(64, 0) == 0
    assert lib.once_calls(64) == 2 and lib.once_calls(0) == 1


def test_no_permission_in_a_plain_static():
    for path in sorted(CSRC.glob("*.cu")):
        text = path.read_text()
        for m in re.finditer(r"cudaFuncSetAttribute", text):
            before = text[max(0, m.start() - 500):m.start()]
            # per-device occupancy caches set it beside what they keep
            assert "per_sm_of[64]" in before, (path.name, m.start())
