"""What the build takes for up to date (no compiler runs here)."""
import os
import shutil
import subprocess
import threading
import time

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


def test_a_changed_makefile_rebuilds_the_library(build):
    # (the compiler's flags are there)
    b, csrc, now, ran = build
    makefile = csrc.parent / "Makefile"
    makefile.write_text("")
    os.utime(makefile, (now, now))
    b.build_library()
    assert ran == []
    os.utime(makefile, (now + 120, now + 120))
    b.build_library()
    assert len(ran) == 1


def test_processes_build_one_after_another(build, monkeypatch):
    b, _, now, ran = build
    os.remove(b.LIB)
    inside = []

    def slow_make(cmd, **kw):
        inside.append(len(inside))
        time.sleep(0.2)
        open(b.LIB, "w").close()
        os.utime(b.LIB, (now + 60, now + 60))
        ran.append(cmd)

    monkeypatch.setattr(b.subprocess, "run", slow_make)
    threads = [threading.Thread(target=b.build_library) for _ in range(3)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert len(ran) == 1  # the others found it built


@pytest.fixture
def tree(pkg, tmp_path):
    """The Makefile on a made-up tree, and a call that runs it with a compiler that only notes what it was asked
    to make: make(*arguments) -> the names of the files."""
    tmp_path = tmp_path / "package"
    for name in ("csrc/gemm.cu", "csrc/gemv.cu", "examples/gpu/decode_loop.cpp", "../include/tcrv_emitc_host.h"):
        (tmp_path / name).parent.mkdir(parents=True, exist_ok=True)
        (tmp_path / name).write_text("")
    shutil.copy(os.path.join(os.path.dirname(pkg._build.__file__), "Makefile"), tmp_path)
    asked = tmp_path / "asked"
    for name in ("nvcc", "other"):
        (tmp_path / name).write_text(f"""#!/bin/sh
while [ $# -gt 0 ]; do [ "$1" = -o ] && {{ touch "$2"; basename "$2" >> {asked}; }}; shift; done
""")
        os.chmod(tmp_path / name, 0o755)

    def make(*args):
        asked.write_text("")
        subprocess.run(["make", "-s", "-C", tmp_path, *args], check=True)
        return sorted(asked.read_text().split())

    return tmp_path, make


def test_objects_follow_the_makefile_the_compiler_and_its_flags(tree):
    path, make = tree
    everything = ["gemm.o", "gemv.o", "libtcrv_cuda.so"]
    nvcc = f"NVCC={path}/nvcc"
    assert make("library", nvcc) == everything and (path / "libtcrv_cuda.so").exists()
    os.remove(path / "libtcrv_cuda.so")
    assert make("library", nvcc) == [] and (path / "libtcrv_cuda.so").exists()
    for age, pattern in ((400, "include/*"), (400, "package/csrc/*"), (400, "package/Makefile"), (300, "package/build/obj/flags"),
                         (200, "package/build/obj/*.o"), (100, "package/build/obj/*.so")):
        for f in path.parent.glob(pattern):
            os.utime(f, (time.time() - age,) * 2)
    assert make("library", nvcc) == []
    os.utime(path / "csrc/gemv.cu")
    assert make("library", nvcc) == ["gemv.o", "libtcrv_cuda.so"]
    os.utime(path / "Makefile")
    assert make("library", nvcc) == everything and make("library", nvcc) == []
    assert make("library", nvcc, "NVCCFLAGS=-O1") == everything
    assert make("library", f"NVCC={path}/other", "NVCCFLAGS=-O1") == everything


def test_the_step_loop_links_the_library_that_is_there(tree):
    path, make = tree
    (path / "libtcrv_cuda.so").write_text("")
    assert make("decode_loop", f"NVCC={path}/nvcc", f"CXX={path}/other") == ["libtcrv_decode_loop.so"]
