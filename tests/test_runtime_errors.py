"""The library's host side when the CUDA runtime fails or the process ends, on a stand-in runtime
(cpp/fake_cudart.cpp) in a process of its own: no GPU and no CUDA call is involved."""
import os
import subprocess
import sys

import pytest

from bricklib_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = """
import ctypes as C
fake = C.CDLL(None)
fake.fake_live.restype = C.c_long
from bricklib_gb300 import _abi
lib = _abi.lib()
lay = _abi.bk_layout((C.c_int * 3)(8, 8, 8), (C.c_int * 3)(1, 4, 8))
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    cuda = os.path.dirname(os.path.dirname(build.nvcc()))
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-std=c++17", "-I", os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp"), "-o", so], check=True)

    def go(body, **env):
        r = subprocess.run([sys.executable, "-c", HEAD + body], cwd=ROOT, capture_output=True, text=True, timeout=300,
                           env=dict(os.environ, LD_PRELOAD=so, **env))
        assert r.returncode == 0, (r.returncode, r.stdout[-500:], r.stderr[-1500:])
        return r.stdout

    return go


def test_a_failed_launch_leaves_no_error_behind(run):
    """A launch that the runtime refuses fails its own call, and the calls after it (whose launches
    are checked through the runtime's last error) succeed."""
    out = run("""
host = (C.c_char * (1 << 20))()
at = C.addressof(host) + 15 & ~15
field = _abi.bk_field(at, 64, 512, 0, _abi.BK_F32)
dims = (C.c_long * 3)(8, 8, 8)
none = (C.c_long * 3)(0, 0, 0)
fill = lambda: lib.bk_ghost_fill(C.c_void_p(at), 4, C.byref(field), C.byref(lay), None)
copy = lambda: lib.bk_copy_to_bricks(C.c_void_p(at), dims, none, none, C.c_void_p(at), C.byref(field), C.byref(lay), None)
assert fill() == 0 and copy() == 0
fake.fake_fail(0, 1, 0)
assert fill() == _abi.BK_ERR_CUDA
assert copy() == 0, _abi.lib().bk_last_error()
assert fake.cudaGetLastError() == 0
print("done")
""")
    assert "done" in out


def test_launch_tables_outlive_the_static_destructors(run):
    """A server's thread may still launch when the process ends without closing it: the table of
    kernels' sizes is not destroyed before it (freed memory is overwritten, so a look-up in a
    destroyed table shows)."""
    out = run("""
import sys
fit = C.cast(lib._ZN2bk10kernel_fitEPKvimPiS2_PKc, C.c_void_p)
assert fake.fake_fit_at_exit(fit) == 0
""", GLIBC_TUNABLES="glibc.malloc.tcache_count=0:glibc.malloc.perturb=165")
    assert "fit after exit: ok" in out


def test_a_server_that_cannot_be_created_holds_nothing(run):
    """Whichever of its streams and events cannot be made, and where the device has no error word,
    bk_server_create gives back what it had made by then."""
    out = run("""
create = lambda: lib.bk_server_create(C.byref(C.c_void_p()), C.c_size_t(1 << 30), C.byref(lay), 4)
fake.fake_fail(0, 0, 1)
assert create() != 0 and fake.fake_live() == 0, fake.fake_live()
made = 0
for n in range(1, 1000):
    fake.fake_fail(n, 0, 1)  # the n-th stream or event; after the last one the error word
    assert create() != 0, n
    assert fake.fake_live() == 0, (n, fake.fake_live())
    if _abi.lib().bk_last_error().decode().startswith("device error word"):
        break
    made = n
assert made >= 20, made
print("done")
""")
    assert "done" in out
