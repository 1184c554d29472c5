"""What the build takes for up to date (no compiler runs here)."""
import os

import pytest


@pytest.fixture
def build(pkg, tmp_path, monkeypatch):
    """The build recipe on a made-up source tree, everything built a minute after it was written."""
    b = pkg._build
    csrc, include = tmp_path / "csrc", tmp_path / "include"
    csrc.mkdir()
    include.mkdir()
    monkeypatch.setattr(b, "HERE", str(tmp_path))
    monkeypatch.setattr(b, "ROOT", str(tmp_path))
    monkeypatch.setattr(b, "CSRC", str(csrc))
    monkeypatch.setattr(b, "LIB", str(tmp_path / "libtcrv_cuda.so"))
    files = [csrc / n for n in ("gemv.cu", "gemv_any.cuh", "launchers.h", "torch_calls.cpp")] + [include / "tcrv_cuda.h"]
    now = os.path.getmtime(b.__file__)
    for f in files:
        f.write_text("")
        os.utime(f, (now, now))
    for out in (b.LIB, b.torch_calls_path()):
        open(out, "w").close()
        os.utime(out, (now + 60, now + 60))
    ran = []
    monkeypatch.setattr(b.subprocess, "run", lambda cmd, **kw: ran.append(cmd))
    monkeypatch.setattr(b, "_nvcc", lambda: "/usr/local/cuda/bin/nvcc")
    return b, csrc, now, ran


def test_up_to_date_files_are_kept(build):
    b, _, _, ran = build
    b.build_library()
    b.build_torch_calls()
    assert ran == []


@pytest.mark.parametrize("name,library,calls", [("gemv_any.cuh", True, False), ("gemv.cu", True, False),
                                                ("torch_calls.cpp", False, True)])
def test_a_changed_source_rebuilds_what_it_is_part_of(build, name, library, calls):
    b, csrc, now, ran = build
    os.utime(csrc / name, (now + 120, now + 120))
    b.build_library()
    assert len(ran) == int(library)
    ran.clear()
    b.build_torch_calls()
    assert len(ran) == int(calls)


def test_another_torch_or_python_does_not_get_the_old_module(build, monkeypatch):
    import torch

    b, _, _, ran = build
    old = b.torch_calls_path()
    monkeypatch.setattr(torch, "__version__", "9.9.0")
    assert b.torch_calls_path() != old
    b.build_torch_calls()
    assert len(ran) == 1 and b.torch_calls_path() in ran[0]
    monkeypatch.undo()
    monkeypatch.setattr(b.sysconfig, "get_config_var", lambda name: "cpython-399")
    assert os.path.basename(b.torch_calls_path()) != os.path.basename(old)


def test_the_c_library_builds_where_there_is_no_torch(build, pkg, monkeypatch):
    import importlib.util

    b, csrc, now, ran = build
    os.utime(csrc / "gemv.cu", (now + 120, now + 120))
    monkeypatch.setattr(b, "build_torch_calls", lambda force=False: pytest.fail("needs torch"))
    monkeypatch.setattr(importlib.util, "find_spec", lambda name: None)
    assert pkg.build_library() == b.LIB and len(ran) == 1
