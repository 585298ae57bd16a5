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
        lib.fake_used.restype = lib.fake_variable_bytes.restype = ctypes.c_size_t
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


def arrays(*counts):
    return [dlp.DeviceArray(np.zeros(c, np.int32)) for c in counts]


@pytest.mark.parametrize("edges", [10, 10000])  # one block, several
@pytest.mark.parametrize("status", [N.DLP_ERR_TIMEOUT, N.DLP_ERR_INVALID_ARGUMENT])
def test_step_launchers_report_what_failed_on_the_device(runtime, edges, status):
    a = arrays(*[2 * edges] * 8)
    x, y = ctypes.c_int(0), ctypes.c_int(0)
    runtime.result(status, 5)
    with pytest.raises(dlp.DlpError, match="[a-z]{4}") as e:
        N.check(N.lib().dlp_connected_components(a[0].ptr, a[1].ptr, edges, a[2].ptr, edges, a[3].ptr, ctypes.byref(x),
                                                 edges, None))
    assert e.value.status == status
    runtime.result(status, 5)
    with pytest.raises(dlp.DlpError, match="[a-z]{4}") as e:
        N.check(N.lib().dlp_build_sparsified_subgraph(
            None, None, None, a[0].ptr, None, a[1].ptr, a[2].ptr, a[3].ptr, edges, a[4].ptr, edges, a[5].ptr, 0.5, None,
            a[6].ptr, a[7].ptr, ctypes.byref(x), ctypes.byref(y), None))
    assert e.value.status == status


@pytest.mark.parametrize("inserted", [10, 10000])
def test_label_initialisation_cannot_fail_unseen(runtime, inserted):
    """It returns without waiting for the device, so it may hold no wait of a grid
    barrier that can run out there."""
    a = arrays(*[inserted + 1] * 6)
    runtime.log()
    N.check(N.lib().dlp_label_initialization(a[0].ptr, a[1].ptr, a[2].ptr, a[3].ptr, None, a[4].ptr, inserted, a[5].ptr,
                                             inserted, a[0].ptr, inserted, None))
    ops = [x[0] for x in runtime.log()]
    assert ops and set(ops) <= {"launch", "clear"}


def graph_bytes(p):
    return dlp.Engine.graph_bytes(p.num_nodes, p.num_edges)


@pytest.mark.parametrize("spare", [0, 100, 1 << 20])
def test_engine_keeps_its_budget(runtime, spare):
    """What the frontier marks take counts: within the budget when there is room
    (8 bytes a vertex in whole tiles), given back when there is none."""
    p = dlp.Problem(1001, 3, 2, 1, cache_dir="")
    eng = dlp.Engine(3, memory_budget_bytes=2 * graph_bytes(p) + spare)
    base = runtime.lib.fake_used()
    taken = []
    for _ in range(2):
        eng.add_problem(p)
        taken.append(runtime.lib.fake_used() - base - eng.bytes_in_use)
        assert taken[-1] + eng.bytes_in_use <= 2 * graph_bytes(p) + spare
    assert taken == ([8 * 1024, 16 * 1024] if spare >= 16 * 1024 else [8 * 1024, 0])
    with pytest.raises(dlp.DlpError):
        eng.add_problem(dlp.Problem(8000, 3, 2, 1, cache_dir=""))
    eng.close()


def test_marks_give_way_to_a_graph_on_a_full_device(runtime):
    p = dlp.Problem(1001, 3, 2, 1, cache_dir="")
    eng = dlp.Engine(2)
    eng.add_problem(p)
    snap = eng.snapshot(0)
    # room for the graph and what its upload or its kept deletions take, but not
    # for the marks of the first one (8 KiB) as well
    for again, full in ((lambda: eng.restore(snap), 4096), (lambda: eng.add_problem(p), 8 * p.num_edges)):
        runtime.lib.fake_capacity(runtime.lib.fake_used() + graph_bytes(p) + full - 8192)
        g = again()
        runtime.lib.fake_capacity(ctypes.c_size_t(-1).value)
        eng.remove_graph(g)
        eng.remove_graph(0)
        assert eng.add_problem(p) == 0
    eng.close()


@pytest.mark.parametrize("grow", ["reserve", "step", "stage"])
def test_marks_give_way_to_a_batch_on_a_full_device(runtime, grow):
    p = dlp.Problem(8000, 3, 1, 1, cache_dir="")
    batch = dlp.Batch.make(inserted=[0, 1], edge_src=[0], edge_dst=[1], edge_weight=[0.5])
    eng = dlp.Engine(1)
    g = eng.add_problem(p)
    if grow == "stage":
        eng.reserve(g, 1, 1)  # leaves the copy of the batch to be allocated
    runtime.log()
    runtime.lib.fake_capacity(runtime.lib.fake_used())
    if grow == "reserve":
        eng.reserve(g, 1, 1)
    else:
        eng.step([(g, 0, batch)])
    assert ["free", str(8 * 8000)] in runtime.log()
    eng.close()


def test_server_keeps_its_budget(runtime):
    p = dlp.Problem(1001, 3, 2, 1, cache_dir="")
    eng = dlp.Engine(2)
    g = eng.add_problem(p)
    batch = p.batches[0]
    request = 24 * batch.edge_src.size + 8 * batch.deleted.size + batch.nbytes() + 256
    for room in (request, request + 8 * 1024):
        srv = dlp.Server(eng, memory_budget_bytes=eng.bytes_in_use + room)
        runtime.log()
        srv.submit(g, 0, batch)
        try:
            srv.poll()
        except dlp.DlpError:
            pass  # nothing ran
        frees = [x for x in runtime.log() if x == ["free", "8192"]]
        assert len(frees) == (1 if room == request else 0)
        srv.close()
        if room == request:
            eng.close()
            eng = dlp.Engine(2)
            g = eng.add_problem(p)
    eng.close()


def test_autotuner_times_each_setting_where_it_has_an_effect(runtime):
    """Three one-block thresholds on owned rows and three lane widths over lists, two
    batches each, and the choice among all combinations of them."""
    r = dlp.autotune([500, 300], [3, 5], batches=2, max_iterations=10)
    kernels = [x[1] for x in runtime.log() if x[0] == "cooperative"]
    owned, lists = ("engine_kernelILi8ELb1", "engine_kernelILi%dELb0")
    want = 3 * 2 * [owned] + [lists % lanes for lanes in (8, 4, 1) for _ in range(2)]
    assert len(kernels) == len(want) and all(w in k for w, k in zip(want, kernels)), kernels
    assert len({(c["narrow_lanes"], c["solo_entry"], c["subgrid_entry"]) for c in r["candidates"]}) == 27
    # a millisecond each in this runtime: nothing to choose by
    assert (r["narrow_lanes"], r["engine_kw"]) == (8, {"solo_entry": 512, "subgrid_entry": 2048})


def test_tuned_shapes_are_kept_for_the_kernels_they_were_measured_on(tmp_path, monkeypatch):
    """The cache key changes with every source that the engine's kernels include."""
    import shutil
    src = Path(dlp.__file__).resolve().parent / "csrc"
    shutil.copytree(src, tmp_path / "csrc")
    monkeypatch.setattr(dlp, "__file__", str(tmp_path / "__init__.py"))
    seen = {dlp._kernel_digest()}
    for name in ("engine_kernel.cu", "engine.cu", "owner_pass.cuh", "row_stint.cuh", "common.cuh", "tune.cu"):
        with open(tmp_path / "csrc" / name, "a") as f:
            f.write("// \n")
        assert dlp._kernel_digest() not in seen, name
        seen.add(dlp._kernel_digest())


def propagate(entry, a, n):
    used = ctypes.c_int(0)
    extra = [a[6].ptr, a[7].ptr] if entry != "dlp_irlp" else []
    ptrs = [x.ptr for x in a[:6]] if entry != "dlp_irlp" else [a[i].ptr for i in (0, 1, 2, 3, 5, 6)]
    N.check(getattr(N.lib(), entry)(*ptrs, *extra, n, ctypes.c_float(1e-4), 5, ctypes.byref(used), None))


def test_launchers_after_a_device_reset(runtime):
    """cudaDeviceReset ends the context with its pools, kernel attributes and the
    addresses of device variables; the launchers work in the next one."""
    n = 1000
    for _ in range(3):
        a = arrays(*[n + 1] * 8)
        for entry in ("dlp_iterative_propagation", "dlp_irlp", "dlp_iterative_propagation_noalloc"):
            runtime.result(5, 0)
            propagate(entry, a, n)
        N.check(N.lib().dlp_label_initialization(a[0].ptr, a[1].ptr, a[2].ptr, a[3].ptr, None, a[4].ptr, n, a[5].ptr, n,
                                                 a[0].ptr, n, None))
        for x in a:
            x.ptr = ctypes.c_void_p()
        runtime.lib.cudaDeviceReset()


def test_label_initialisation_while_a_stream_captures(runtime):
    """It waits for nothing and can be part of a graph, also as the first call of a
    context: making the pool must not spoil the capture."""
    runtime.lib.cudaDeviceReset()
    n = 100
    a = arrays(*[n + 1] * 6)
    runtime.lib.fake_begin_capture()
    N.check(N.lib().dlp_label_initialization(a[0].ptr, a[1].ptr, a[2].ptr, a[3].ptr, None, a[4].ptr, n, a[5].ptr, n,
                                             a[0].ptr, n, None))
    assert runtime.lib.fake_end_capture() == 0


def test_device_memory_held_by_loading_the_library(runtime):
    """The scratch of the allocation-free propagation: three words for each of 2^20
    vertices, and less than a KiB."""
    assert 12 << 20 <= runtime.lib.fake_variable_bytes() <= (12 << 20) + 1024


@pytest.mark.parametrize("source", ["engine.cu", "engine_kernel.cu", "launchers.cu", "tune.cu"])
def test_the_build_with_512_threads_compiles(tmp_path, source):
    """A build setting of the persistent kernels (DLP_NVCC_EXTRA=-DDLP_BLOCK=512)."""
    res = subprocess.run([b._nvcc(), "-gencode", "arch=compute_103a,code=compute_103a", "-std=c++17", "-Xcicc", "-O0",
                          f"-I{b.INCLUDE}", f"-I{b.CSRC}", "-DDLP_BLOCK=512", "-cuda", str(b.CSRC / source), "-o",
                          str(tmp_path / "out.ii")], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-2000:]


def test_allocation_free_propagation_on_a_part_of_a_gpu(runtime):
    """20 multiprocessors cannot own a million vertices: lists, in the same scratch."""
    n = 1 << 20
    a = arrays(*[n + 1] * 8)
    try:
        runtime.lib.fake_multiprocessors(20)
        runtime.lib.cudaDeviceReset()  # the next context asks the device anew
        runtime.log()
        runtime.result(7, 0, 0, 0, 0)
        used = ctypes.c_int(0)
        N.check(N.lib().dlp_iterative_propagation_noalloc(*[x.ptr for x in a], n, ctypes.c_float(1e-4), 9,
                                                          ctypes.byref(used), None))
        assert used.value == 7
        launched = [x for x in runtime.log() if x[0] == "cooperative"]
        assert len(launched) == 1 and "prop_kernel" in launched[0][1] and int(launched[0][2]) % 20 == 0
    finally:
        runtime.lib.fake_multiprocessors(152)
        runtime.lib.cudaDeviceReset()
        for x in a:
            x.ptr = ctypes.c_void_p()


@pytest.mark.parametrize("passes,slice_us,owned", [(3, 0.0, False), (4, 0.0, True), (0, 14.0, False), (0, 16.0, True),
                                                   (4, 14.0, False), (0, 0.0, True)])
def test_rows_are_loaded_for_more_than_a_few_passes(runtime, passes, slice_us, owned):
    p = dlp.Problem(1001, 3, 2, 1, cache_dir="")
    eng = dlp.Engine(1, max_iterations=50)
    g = eng.add_problem(p)
    runtime.log()
    eng.step_sliced([(g, 0, dlp.DeviceBatch(p.batches[0]))], pass_budget=passes, slice_us=slice_us)
    kernel, = [x[1] for x in runtime.log() if x[0] == "cooperative"]
    assert ("ELb1" in kernel) == owned
    eng.close()
