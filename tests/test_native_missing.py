"""The native host module missing, stale or not buildable: calls go on through
the Python functions, with one warning; the kernels' library needs neither
Python's nor torch's headers."""
import importlib
import warnings

import pytest

from qcware_unitair_gb300 import _native, build_lib


class Arg:
    is_cuda = True


@pytest.fixture
def fresh():
    """_native as at import."""
    importlib.reload(_native)
    yield _native
    importlib.reload(_native)


def check_left_to_python(mod, match):
    with pytest.warns(RuntimeWarning, match=match):
        assert mod.norm_squared(Arg()) is None
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert mod.norm_squared(Arg()) is None
        assert mod.apply_operator(Arg(), [0], Arg()) is None


def test_not_built(fresh, monkeypatch, tmp_path):
    monkeypatch.setattr(build_lib, "host_path", lambda: tmp_path / "no.so")
    with pytest.raises(RuntimeError, match="not built"):
        fresh.load()
    check_left_to_python(fresh, "not built")


def test_built_for_another_torch(lib_built, fresh, monkeypatch):
    monkeypatch.setattr(build_lib, "host_tag", lambda: "torch 0.0")
    with pytest.raises(RuntimeError, match="this is torch 0.0"):
        fresh.load()
    check_left_to_python(fresh, "was built for")


def test_does_not_load(fresh, monkeypatch, tmp_path):
    path = tmp_path / "bad.so"
    path.write_bytes(b"no library")
    (tmp_path / "bad.txt").write_text(build_lib.host_tag())
    monkeypatch.setattr(build_lib, "host_path", lambda: path)
    monkeypatch.setattr(build_lib, "host_tag_path",
                        lambda: tmp_path / "bad.txt")
    check_left_to_python(fresh, "native host path is off")


def test_stamp_covers_the_host_module(monkeypatch):
    want = build_lib._stamp()
    flags = build_lib._host_flags()
    monkeypatch.setattr(build_lib, "_host_flags",
                        lambda: (flags[0] + ["-O1"], flags[1]))
    assert build_lib._stamp() != want


def test_builds_without_headers(monkeypatch, tmp_path):
    """The library alone, from one small source."""
    src = tmp_path / "csrc"
    src.mkdir()
    (src / "one.cpp").write_text('extern "C" int one() { return 1; }\n')
    monkeypatch.setattr(build_lib, "CSRC", src)
    monkeypatch.setattr(build_lib, "BUILD_DIR", tmp_path / "_build")
    monkeypatch.setattr(build_lib, "host_headers", lambda: False)
    out = build_lib.build()
    assert out.exists() and not build_lib.host_path().exists()
    stamp = out.stat().st_mtime_ns
    assert build_lib.build() == out and out.stat().st_mtime_ns == stamp
