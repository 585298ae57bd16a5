"""The library's host code over a CUDA runtime without a device
(tests/fake_cuda): what it issues on which stream, what it allocates and what it
reports, including results that a device rarely gives."""
from __future__ import annotations

import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

import labelpropcuda_gb300 as dlp
from labelpropcuda_gb300 import _native as N
from labelpropcuda_gb300 import build as b

FAKE = Path(__file__).resolve().parent / "fake_cuda" / "cudart.cpp"


class Runtime:
    def __init__(self, lib):
        self.lib = lib
        lib.fake_log.restype = ctypes.c_char_p
        lib.fake_used.restype = ctypes.c_size_t
        lib.fake_capacity.argtypes = [ctypes.c_size_t]

    def log(self) -> list[list[str]]:
        """The operations since the last call, as words."""
        out = [x.split() for x in self.lib.fake_log().decode().splitlines()]
        self.lib.fake_clear_log()
        return out

    def result(self, *words: int) -> None:
        self.lib.fake_result((ctypes.c_int * len(words))(*words), len(words))


@pytest.fixture(scope="module")
def linked(tmp_path_factory):
    b.build()
    so = tmp_path_factory.mktemp("fake") / "libdynlp_fake.so"
    objs = [str(b.BUILD / (Path(s).stem + (".o" if s.endswith(".cu") else ".cpp.o")))
            for s in b.CU_SOURCES + b.CXX_SOURCES]
    subprocess.run(["g++", "-shared", "-fPIC", "-std=c++17", "-Wl,-Bsymbolic", "-I/usr/local/cuda/include", str(FAKE),
                    *objs, "-fopenmp", "-o", str(so)], check=True)
    return so


@pytest.fixture
def runtime(linked, monkeypatch):
    """The package over a copy of its library linked with the fake runtime."""
    handle = ctypes.CDLL(str(linked))
    for name, (res, args) in N._SIGNATURES.items():
        fn = getattr(handle, name)
        fn.restype, fn.argtypes = res, args
    monkeypatch.setattr(N, "_lib", handle)
    rt = Runtime(handle)
    rt.lib.fake_capacity(ctypes.c_size_t(-1).value)
    rt.log()
    return rt


def written(log):
    """(operation, stream) of everything that writes device memory."""
    return [(x[0], x[-1]) for x in log if x[0] in ("clear", "launch", "cooperative") or x[:2] in (["copy", "h2d"],
                                                                                                 ["copy", "d2d"])]


def test_engine_writes_on_its_own_stream_only(runtime):
    """The engine's stream does not wait for the default stream: a clear or a
    copy issued there could come after the step that relies on it."""
    p = dlp.Problem(300, 3, 3, 1, cache_dir="")
    eng = dlp.Engine(3)
    g = eng.add_problem(p)
    eng.step([(g, 0, p.batches[0])])
    snap = eng.snapshot(g)
    eng.reset_graph(g)
    eng.restore(snap)
    for i, batch in enumerate(p.batches):
        eng.step([(g, i, batch)])
    ops = written(runtime.log())
    streams = {s for _, s in ops}
    assert len(ops) > 40 and len(streams) == 1 and "default" not in streams, ops
    eng.close()
