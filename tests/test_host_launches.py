"""What the library's host side asks of CUDA, without a GPU: the built objects
linked against tests/fake_cuda.cpp, which counts launches, captures and graph
replays and refuses what the runtime refuses (a launch with more dynamic shared
memory than the kernel's limit on that device)."""
import ctypes
import importlib.util
import os
import shutil
import subprocess
import time
from pathlib import Path

import numpy as np
import pytest

PKG = Path(__file__).resolve().parents[1] / "how-mhd-kokkos_b200"


@pytest.fixture(scope="module")
def module(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not found")
    objs = [PKG / "_build" / (f.stem + ".o") for f in (PKG / "csrc").iterdir()
            if f.suffix in (".cu", ".cpp") and f.name != "driver_main.cpp"]
    if not all(o.exists() for o in objs):
        pytest.skip("the library's objects are not built")
    so = tmp_path_factory.mktemp("fake") / "libhowfake.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-o", str(so),
                    str(Path(__file__).with_name("fake_cuda.cpp")), *map(str, objs), "-lgomp", "-ldl", "-lpthread"],
                   check=True)
    old = os.environ.get("HOW_MHD_LIB")
    os.environ["HOW_MHD_LIB"] = str(so)
    try:
        spec = importlib.util.spec_from_file_location("how_mhd_fake", PKG / "how_mhd" / "__init__.py")
        hm = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(hm)
    finally:
        if old is None:
            del os.environ["HOW_MHD_LIB"]
        else:
            os.environ["HOW_MHD_LIB"] = old
    fake = ctypes.CDLL(str(so))
    fake.fake_launches.restype = ctypes.c_char_p
    fake.fake_calls.restype = ctypes.c_long
    return hm, fake


@pytest.fixture
def lib(module):
    hm, fake = module
    fake.fake_reset(2)
    yield hm, fake
    fake.fake_reset(1)


def _params(hm, n, bc="periodic", **kw):
    return hm.make_parameters(nx=n[0], ny=n[1], nz=n[2], nt=1, tend=1.0, gam=5.0 / 3.0, cour=0.4, problem="uniform",
                              x1bc=bc, x2bc=bc, x3bc=bc, **kw)


class Launch:
    def __init__(self, row):
        captured, device, grid, block, smem, watched, self.kernel = row.split(" ", 6)
        self.captured, self.device, self.smem, self.watched = captured == "1", int(device), int(smem), int(watched)
        self.blocks = int(grid.split(",")[0])


def _launches(fake, kernel=""):
    """The launches since the last call, of the kernels with this name."""
    rows = map(Launch, fake.fake_launches().decode().splitlines())
    return [r for r in rows if kernel in r.kernel]


@pytest.mark.parametrize("kw", [{}, {"precision": "mixed"}, {"precision": "mixed", "router": "on"}],
                         ids=["fp64", "mixed", "routed"])
def test_a_second_device_gets_its_own_limits(lib, kw):
    """The sweeps' shared memory is past the default limit, which is raised per
    device: a second domain on another device, and one after a device reset."""
    hm, fake = lib
    for device in (0, 1):
        fake.fake_set_device(device)
        with hm.Domain(_params(hm, (40, 37, 35), **kw)) as d:
            _launches(fake)
            d.ssprk(1e-3)
            rows = _launches(fake, "k_sweep")
            assert len(rows) == 15 and all(r.device == device and r.smem > 49152 for r in rows)
            # persistent blocks: at most as many as this device has SMs
            assert max(r.blocks for r in rows) <= (148, 100)[device]
    fake.cudaDeviceReset()
    with hm.Domain(_params(hm, (40, 37, 35), **kw)) as d:
        d.ssprk(1e-3)


def test_a_group_over_two_devices_launches(lib):
    hm, fake = lib
    p = _params(hm, (20, 18, 16))
    with hm.Group(p, 2, devices=[0, 1]) as g:
        g.set_state(np.ones((8, 26, 24, 22)))
        _launches(fake)
        with pytest.raises(hm.HowError, match="non-positive dt"):   # (no device: no dt)
            g.run(0.0, 1)
        assert {r.device for r in _launches(fake)} == {0, 1}
    for k in (0, 1):   # the parts' own steps
        fake.fake_set_device(k)
        with hm.Domain(p) as d:
            d.ssprk(1e-3)


def test_an_ensemble_on_a_second_device_launches(lib):
    hm, fake = lib
    for device in (0, 1):
        fake.fake_set_device(device)
        with hm.Ensemble([_params(hm, (40, 1, 1)), _params(hm, (24, 20, 1))]) as e:
            e.init()
            e.set_shapes(0, 1, 0)
            _launches(fake)
            e.run(1)
            rows = _launches(fake, "k_sweep")   # x sweeps, and y sweeps of the 2-D member
            assert len(rows) == 10 and all(r.captured and r.device == device for r in rows)


def test_an_ensemble_does_not_run_without_its_sweeps(lib):
    hm, fake = lib
    with hm.Ensemble([_params(hm, (40, 1, 1)), _params(hm, (24, 20, 1))]) as e:
        e.init()
        e.set_shapes(0, 0, 0)
        fake.fake_fail(b"cudaFuncSetAttribute", 999)
        with pytest.raises(hm.HowError):
            e.run(1)
        fake.fake_fail(b"cudaFuncSetAttribute", 0)
        e.run(1)


def _step(d, n):
    for _ in range(n):
        d.ssprk(1e-3)


@pytest.mark.parametrize("n", [(48, 1, 1), (24, 20, 1), (12, 10, 9)], ids=["1d", "2d", "3d"])
def test_steps_become_a_graph_per_buffer_role(lib, n):
    hm, fake = lib
    with hm.Domain(_params(hm, n)) as d:
        _step(d, 60)
        assert fake.fake_calls(b"cudaGraphInstantiate") == 2
        assert fake.fake_calls(b"cudaGraphLaunch") == 60 - 16


def test_a_written_state_keeps_the_graphs(lib):
    """A periodic axis of one cell: the two steps after a state was written fill
    axis by axis, beside the graphs."""
    hm, fake = lib
    with hm.Domain(_params(hm, (24, 20, 1))) as d:
        q = np.ones((8, 30, 26, 7))
        _step(d, 20)
        for _ in range(5):
            d.set_state(q)
            _step(d, 20)
        assert fake.fake_calls(b"cudaGraphInstantiate") == 2 and fake.fake_calls(b"cudaGraphExecDestroy") == 0
        assert fake.fake_calls(b"cudaGraphLaunch") == 4 + 5 * 18


def test_a_change_of_precision_drops_the_graphs(lib):
    hm, fake = lib
    with hm.Domain(_params(hm, (12, 10, 9))) as d:
        _step(d, 20)
        d.set_precision("mixed")
        _launches(fake)
        _step(d, 16)
        assert len(_launches(fake, "k_sweep")) == 16 * 15
        _step(d, 4)
        assert fake.fake_calls(b"cudaGraphInstantiate") == 4 and fake.fake_calls(b"cudaGraphExecDestroy") == 2
        assert fake.fake_calls(b"cudaGraphLaunch") == 4 + 4


@pytest.mark.parametrize("call", ["cudaStreamBeginCapture", "cudaStreamEndCapture", "cudaGraphInstantiate",
                                  "cudaGraphLaunch"])
def test_a_step_that_cannot_be_a_graph_is_launched(lib, call):
    hm, fake = lib
    with hm.Domain(_params(hm, (12, 10, 9))) as d:
        _step(d, 16)
        _launches(fake)
        fake.fake_fail(call.encode(), 901)
        _step(d, 30)
        rows = [r for r in _launches(fake, "k_sweep") if not r.captured]
        assert len(rows) == 30 * 15
        assert fake.fake_calls(call.encode()) == 2   # once per buffer role, then no more


def test_a_launch_refused_in_a_capture_is_not_left_out(lib):
    hm, fake = lib
    with hm.Domain(_params(hm, (12, 10, 9))) as d:
        _step(d, 16)
        _launches(fake)
        fake.fake_fail(b"captured launch", 1)
        _step(d, 4)
        assert len(_launches(fake, "k_sweep")) == 4 * 15
        assert fake.fake_calls(b"cudaGraphLaunch") == 0
        fake.fake_fail(b"cudaLaunchKernel", 1)   # a refused launch of the step itself is its error
        with pytest.raises(hm.HowError):
            d.ssprk(1e-3)


@pytest.mark.parametrize("kw", [{}, {"precision": "mixed"}, {"router": "on"}], ids=["fp64", "mixed", "routed"])
def test_sweeps_of_few_lines_leave_no_lane_idle(lib, kw):
    """x sweeps of one, two, three, five lines a plane: a line per warp; else four."""
    hm, fake = lib
    for n, lines in (((40000, 1, 1), 1), ((300, 1, 300), 1), ((300, 3, 1), 1), ((300, 5, 20), 1), ((4096, 9, 1), 1),
                     ((5, 5, 300), 4), ((300, 4, 1), 4), ((300, 7, 1), 4), ((4096, 13, 1), 4), ((300, 300, 1), 4),
                     ((40, 40, 40), 4)):
        with hm.Domain(_params(hm, n, **kw)) as d:
            _launches(fake)
            d.ssprk(1e-3)
            x = _launches(fake, "k_sweepILi0E")
            assert len(x) == 5 and all("k_sweepILi0ELi%dE" % lines in r.kernel for r in x)


@pytest.fixture(scope="module")
def chunks_offset(tmp_path_factory):
    """Where a sweep's arguments hold the chunks of its work items."""
    d = tmp_path_factory.mktemp("offset")
    (d / "o.cpp").write_text('#include "how_internal.cuh"\n#include <cstddef>\n#include <cstdio>\n'
                             'int main() { std::printf("%d", (int)offsetof(how::SweepArgs, seg_chunks)); }\n')
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not found")
    subprocess.run(["nvcc", "-x", "cu", "-std=c++17", "-w", "-I", str(PKG / "csrc"), "-I", str(PKG.parent / "include"),
                    "-o", str(d / "o"), str(d / "o.cpp")], check=True)
    return int(subprocess.run([str(d / "o")], check=True, capture_output=True, text=True).stdout)


def test_small_ensembles_take_short_items(lib, chunks_offset):
    """Members with too few items to fill the chip take items of one chunk, others
    the shape's."""
    hm, fake = lib
    for n, members, chunks in ((200, 3, (1, 1, 1)), (200, 32, (1, 1, 1)), (64, 200, (2, 1, 1)), (20000, 16, (2, 8, 2))):
        with hm.Ensemble([_params(hm, (n, 1, 1))] * members) as e:
            e.init()
            for shape in range(3):
                e.set_shapes(shape, shape, shape)
                _launches(fake)
                fake.fake_watch(chunks_offset)
                e.run(1)
                x = _launches(fake, "k_sweep")
                assert len(x) == 5 and all(r.watched == chunks[shape] for r in x)


def test_cutting_a_long_line_takes_no_time(lib):
    """How a sweep is cut is worked out at its launch: at 2e6 cells under 1 ms
    of a step (trying every length took 11 ms here, the launches take 0.05)."""
    hm, fake = lib
    with hm.Domain(_params(hm, (2000000, 1, 1), router="on")) as d:
        took = []
        for _ in range(5):
            t = time.perf_counter()
            d.ssprk(1e-3)
            took.append(time.perf_counter() - t)
    assert min(took) < 1e-3


def test_a_refused_limit_is_an_error_and_is_asked_for_again(lib):
    hm, fake = lib
    with hm.Domain(_params(hm, (40, 37, 35))) as d:
        fake.fake_fail(b"cudaFuncSetAttribute", 999)
        with pytest.raises(hm.HowError):
            d.ssprk(1e-3)
        fake.fake_fail(b"cudaFuncSetAttribute", 0)
        d.ssprk(1e-3)
