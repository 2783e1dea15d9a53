"""CPU tests of the library's host code where a device call fails: its objects are
linked against a stand-in for the CUDA runtime (fake/cudart.cpp: two devices,
kernels recorded by name and not run), which refuses launches or delays events
as a test asks.  Each test runs in a process of its own."""
import os
import shutil
import subprocess
import sys

import pytest

from conftest import PKG_DIR, ROOT

FAKE = os.path.join(ROOT, "tests", "fake", "cudart.cpp")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

PRELUDE = """
import ctypes, os, sys, threading, time
import numpy as np
sys.path.insert(0, %r)
from conftest import load_dcm
dcm = load_dcm()
dcm.LIBPATH = sys.argv[1]
fake = ctypes.CDLL(sys.argv[1])
cases = __import__("dcm_b200.cases", fromlist=["cases"])

def grid(ip, jp, kp):
    return cases.make_grid(ip, jp, kp, 50.0, 50.0, 50.0, [-1.0e4, 1.0e5], [300.0, 300.0])

def field(g):
    return np.zeros((g.kp + 2, g.jp + 2, g.ip + 2), order="F")

def status(call, *args):
    try:
        call(*args)
    except dcm.DCMError as e:
        return e.status
    return 0
""" % os.path.join(ROOT, "tests")


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None or not os.path.exists(NVCC):
        pytest.skip("no compilers")
    sys.path.insert(0, PKG_DIR)
    import build
    d = tmp_path_factory.mktemp("fake")
    lib = str(d / "libdcm_fake.so")
    inc = os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include")
    subprocess.run([cxx, "-std=c++17", "-O1", "-fPIC", "-I" + inc, "-c", FAKE, "-o",
                    str(d / "cudart.o")], check=True)
    subprocess.run([cxx, "-shared", "-o", lib] + build.objects() + [str(d / "cudart.o"),
                                                                    "-lpthread"], check=True)
    return lib


def run(fake_lib, script, timeout=60):
    p = subprocess.run([sys.executable, "-c", PRELUDE + script, fake_lib], timeout=timeout,
                       stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert p.returncode == 0, p.stdout[-3000:]


def test_small_solve_on_a_second_device(fake_lib):
    """Clusters of 16 blocks are allowed per device: the small FP64 solve's
    launch is accepted on both."""
    run(fake_lib, """
g = grid(16, 1, 16)
cores = [dcm.DynamicalCore(g, device=d) for d in (0, 1)]
for d, core in enumerate(cores):
    assert status(core.bicgstab, field(g), field(g), field(g), 1e-10) == 0
    assert fake.fake_launches(b"k_bicgstab_point", d) == 1, d
assert status(cores[1].set_small_cluster, 8) == 0
assert status(cores[1].set_small_cluster, 12) == dcm.DCM_E_ARG
""")


def test_refused_small_solve_is_an_error(fake_lib):
    run(fake_lib, """
g = grid(16, 1, 16)
core = dcm.DynamicalCore(g)
fake.fake_refuse(b"k_bicgstab_point")
assert status(core.bicgstab, field(g), field(g), field(g), 1e-10) == dcm.DCM_E_CUDA
core.set_small_solver(0)
fake.fake_refuse(b"k_bicg_post")
core.solver_graphs(False)
assert status(core.bicgstab, field(g), field(g), field(g), 1e-10, 0, 3) == dcm.DCM_E_CUDA
""")


@pytest.mark.parametrize("kernel", ["k_repitch", "k_unpitch", "k_exchange"])
@pytest.mark.parametrize("shape", [(16, 12, 10), (64, 64, 64)])
def test_refused_launch_between_copies_is_an_error(fake_lib, shape, kernel):
    """A launch refused before or between the copies of a call is that call's
    error, below and above the size from which threads copy, and not the next
    call's."""
    run(fake_lib, """
g = grid(*%r)
core = dcm.DynamicalCore(g)
fake.fake_refuse(%r)
assert status(core.exchange_along_dim_wo, field(g)) == dcm.DCM_E_CUDA
fake.fake_refuse(b"")
assert status(core.exchange_along_dim_wo, field(g)) == 0
""" % (shape, kernel.encode()))


@pytest.mark.parametrize("mb", [3, 17])
def test_copies_behind_unfinished_work_cost_no_cores(fake_lib, mb):
    """A copy that waits for the device sleeps: every DMA here takes 0.2 s, and
    the process uses less than a fifth of one core meanwhile (the arrays' bytes,
    and no looking around for longer than a moment, by any thread)."""
    run(fake_lib, """
import resource
def used():
    r = resource.getrusage(resource.RUSAGE_SELF)
    return r.ru_utime + r.ru_stime
g = grid(128, 126, %d)
core = dcm.DynamicalCore(g)
a = field(g)
a[...] = 1.0
core.exchange_along_dim_wo(a)  # threads, buffers and pages are made
fake.fake_busy(200)
t, c = time.time(), used()
core.exchange_along_dim_wo(a)
t, c = time.time() - t, used() - c
assert t >= 0.4, t
assert c <= 0.2 * t, (c, t)
""" % (mb * 1000000 // (8 * 130 * 128)))


def test_copies_move_every_byte(fake_lib):
    """Arrays of every number of buffers, through threads that sleep and wake
    between the chunks (each DMA takes longer than a thread looks for work) and
    that do not.  The kernels between do nothing: an upload's bytes stay in the
    stage, from where the download returns them."""
    run(fake_lib, """
rng = np.random.default_rng(5)
for kp in (62, 14, 30, 61, 93, 130):
    g = grid(128, 252, kp)
    core = dcm.DynamicalCore(g)
    for ms in (0, 2, 0):
        fake.fake_busy(ms)
        a = field(g)
        a[...] = rng.normal(size=a.shape)
        want = a.copy(order="F")
        core.exchange_along_dim_wo(a)
        assert np.array_equal(a, want)
    core.close()
""")


def test_forked_child_gives_up_its_handle(fake_lib):
    """A child process has the handle but not the threads that copy: it can
    destroy the handle (the binding does when the object goes) and exit."""
    run(fake_lib, """
g = grid(64, 64, 64)
core = dcm.DynamicalCore(g)
assert status(core.exchange_along_dim_wo, field(g)) == 0
pid = os.fork()
if pid == 0:
    core.close()
    os._exit(7)
end = time.time() + 20
while time.time() < end:
    done, st = os.waitpid(pid, os.WNOHANG)
    if done:
        break
    time.sleep(0.05)
else:
    os.kill(pid, 9)
    os.waitpid(pid, 0)
    raise AssertionError("the child hangs")
assert os.WEXITSTATUS(st) == 7
assert status(core.exchange_along_dim_wo, field(g)) == 0
core.close()
""")


def test_column_memory_stays_with_its_context(fake_lib):
    """The device memory that a thread keeps for the sedimentation calls is used
    again in the context that it came from, and not in another on the same
    device."""
    run(fake_lib, """
ncol, kp = 7, 20
met = [np.ones(kp + 2) for _ in range(4)]
w, psi = np.zeros((ncol, kp + 2)), np.ones((ncol, 1, kp + 2))
def call():
    return status(lambda: dcm.mpdata_vec_1d_columns(1.0, 1, *met, w, psi))
for c in (1, 1, 2, 2, 1):
    fake.fake_context(ctypes.c_ulonglong(c))
    assert call() == 0, c
""")
