"""What the library's host code does around its launches, on the CPU: the library runs in a
child process over a recording CUDA runtime on host memory (fake_cudart.cpp), whose
kernels do nothing, and the test reads the calls that it made.
"""
import json
import os
import subprocess
import sys

import pytest

from cube_nufluid_b200.build import ARCH, CSRC, FLAGS, NVCC

TESTS = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(TESTS)
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

CHILD = """
import ctypes as C, json, os, sys
import numpy as np
sys.path.insert(0, {root!r})
from cube_nufluid_b200 import Cube, CubeError
from cube_nufluid_b200.abi import CubeScalars, make_params
fake = C.CDLL(os.environ["LD_PRELOAD"])
fake.fake_log.restype = C.c_char_p
fake.fake_poke.argtypes = [C.c_size_t, C.c_size_t, C.c_ulonglong]

def calls():
    return [dict(zip(("call", "name", "src", "stream"), l.split())) for l in fake.fake_log().decode().splitlines()]

def empty_box():
    g = Cube(make_params(16, 2), np_capacity=64)
    g.load_state(np.zeros((0, 3), np.int16), np.zeros((0, 3), np.int16), np.zeros(0, np.int32),
                 np.zeros(16 ** 3, np.int32), np.zeros((16 ** 3, 3), np.float32))
    return g
"""


@pytest.fixture(scope="module")
def child(tmp_path_factory):
    """runs code after CHILD and returns the JSON it prints"""
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", f"-I{CUDA}/include", "-o", so, os.path.join(TESTS, "fake_cudart.cpp")],
                   check=True)

    def run(code):
        r = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT) + code], env=dict(os.environ, LD_PRELOAD=so),
                           capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stderr[-2000:]
        return json.loads(r.stdout)

    return run


def test_halofind_of_a_box_without_peaks(child):
    assert child("""
g = empty_box()
s = CubeScalars()
s.a, s.sigma_vi, s.mass_p_cdm, s.vsim2phys = 0.5, 0.01, 1.0, 1.0
halos, members, hid, npeak = g.halofind(s, hid_len=10)
print(json.dumps([len(halos), len(members), hid.tolist(), npeak]))
""") == [0, 0, [0] * 10, 0]


def test_halofind_orders_everything_on_the_context_stream(child):
    """A copy by the default stream is not ordered with the context's own: the kernels of the
    first call could read the list of shells before it is there."""
    log = child("""
g = empty_box()
fake.fake_clear()
s = CubeScalars()
s.a, s.sigma_vi, s.mass_p_cdm, s.vsim2phys = 0.5, 0.01, 1.0, 1.0
g.halofind(s)
print(json.dumps(calls()))
""")
    assert [c for c in log if c["call"] == "launch"] and [c for c in log if c["name"] == "h2d"]
    streams = {c["stream"] for c in log}
    assert len(streams) == 1 and streams != {"(nil)"}, [c for c in log if c["stream"] == "(nil)"]


@pytest.mark.parametrize("nc", [16, 40])  # 2^14 cells and fewer are added on the host, more on the device
def test_contradicting_counts_are_refused_before_the_particle_arrays_are_read(child, nc):
    """A caller whose particle count is larger than its arrays (the kernels do nothing here: the
    device's total stays 0 against 64)."""
    code, read, log = child(f"""
nc = {nc}
g = Cube(make_params(nc, 2), np_capacity=64)
xp, vp, pid = np.zeros((64, 3), np.int16), np.zeros((64, 3), np.int16), np.zeros(64, np.int32)
rhoc, vf = np.zeros(nc ** 3, np.int32), np.zeros((nc ** 3, 3), np.float32)
fake.fake_clear()
try:
    g.load_state(xp, vp, pid, rhoc, vf)
    code = 0
except CubeError as e:
    code = e.code
read = [c["src"] == hex(a.ctypes.data) for a in (xp, vp, pid, vf, rhoc) for c in calls() if c["name"] == "h2d"]
n = sum(c["name"] == "h2d" for c in calls())
print(json.dumps([code, [any(read[i * n:(i + 1) * n]) for i in range(5)], calls()]))
""")
    assert code == 1
    assert read == [False] * 4 + [nc == 40], log


@pytest.mark.parametrize("short", range(5))
def test_load_state_refuses_arrays_shorter_than_the_state(child, short):
    """nplocal is the length of xp: an array with fewer bytes than that state has is refused
    and none is read; one that is longer is taken as before."""
    code, copies = child(f"""
g = Cube(make_params(16, 2, izipx=2, izipv=2), np_capacity=64)
arrays = [np.zeros((64, 3), np.int16), np.zeros((64, 3), np.int16), np.zeros(64, np.int32),
          np.zeros(16 ** 3, np.int32), np.zeros((16 ** 3, 3), np.float32)]
short = {short}
arrays[short] = arrays[short].astype(np.int8) if short == 0 else arrays[short][:-1]
fake.fake_clear()
try:
    g.load_state(*arrays)
    code = 0
except CubeError as e:
    code = e.code
print(json.dumps([code, sum(c["name"] == "h2d" for c in calls())]))
""")
    assert (code, copies) == (1, 0)


def test_refused_launch_on_the_side_stream_still_joins_it(child, tmp_path):
    """The largest cells are sorted on a stream beside the context's.  When the second of its two
    launches is refused, the call fails, and the context's stream waits for the first."""
    names = ["n_huge", "max_huge"]
    (tmp_path / "o.cu").write_text(
        '#include "cube_internal.cuh"\n#include <cstdio>\nint main() { printf("%zu ' + "%zu " * len(names) + '", sizeof(DevScal)'
        + "".join(f", offsetof(DevScal, {n})" for n in names) + "); }\n")
    subprocess.run([NVCC, *ARCH, *FLAGS, "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-o", str(tmp_path / "o"),
                    str(tmp_path / "o.cu")], check=True)
    size, n_huge, max_huge = map(int, subprocess.run([str(tmp_path / "o")], capture_output=True, text=True).stdout.split())
    code, log = child(f"""
g = empty_box()
fake.fake_poke({size}, {n_huge}, 2)
fake.fake_poke({size}, {max_huge}, 20000)
fake.fake_refuse(b"k_rebin_hugeI")
fake.fake_clear()
s = CubeScalars()
s.dt = s.dt_old = 1.0
s.sigma_vi = 0.01
try:
    g.update_x(s)
    code = 0
except CubeError as e:
    code = e.code
print(json.dumps([code, calls()]))
""")
    assert code == 3
    at = next(i for i, c in enumerate(log) if c["call"] == "refused")
    side = log[at]["stream"]
    assert log[at - 1]["stream"] == side and "k_rebin_huge_order" in log[at - 1]["name"]
    main = log[0]["stream"]
    assert main != side
    joined = [c for i, c in enumerate(log[at:]) if c["call"] == "cudaStreamWaitEvent" and c["stream"] == main
              and any(e["call"] == "cudaEventRecord" and e["src"] == c["src"] and e["stream"] == side
                      for e in log[at:at + i])]
    assert joined or any(c["call"] == "cudaStreamSynchronize" and c["stream"] == side for c in log[at:])


def test_phase_times_are_those_of_the_last_finished_call(child):
    """A call that fails on its way leaves the times that are there (event times here: calls)."""
    before, after, again = child("""
g = empty_box()
s = CubeScalars()
s.dt = s.dt_old = 1.0
s.a = s.a_mid = 0.5
s.sigma_vi = s.sigma_vi_new = 0.01
g.update_x(s)
g.particle_mesh(s)
before = g.phase_times()
for kernel, call in ((b"k_rebin_count", g.update_x), (b"k_coarse_finalize", g.particle_mesh)):
    fake.fake_refuse(kernel)
    try:
        call(s)
        raise SystemExit("not refused")
    except CubeError as e:
        assert e.code == 3
after = g.phase_times()
fake.fake_refuse(b"")
g.update_x(s)
g.particle_mesh(s)
print(json.dumps([before, after, g.phase_times()]))
""")
    assert [t > 0 for t in before] == [True, False, True, True, True, True, False, True]
    assert after == before
    assert [t > 0 for t in again] == [t > 0 for t in before]
