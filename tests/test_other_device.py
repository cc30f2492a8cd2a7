"""Context calls from a thread whose current device is another one, on a
pretended runtime with two devices (fake_cudart.c): no GPU is needed."""
from __future__ import annotations

import os
import subprocess
import sys
from pathlib import Path

HERE = Path(__file__).resolve().parent

SCRIPT = """
import ctypes as C, sys
sys.path.insert(0, sys.argv[1])
import wwcuda as ww
L = ww.lib()
rt = C.CDLL(sys.argv[2])
h = C.c_void_p()
ww.check(L.ww_open(1, C.byref(h)), "ww_open")
b = ww.Buffers()
ww.check(L.ww_get_buffers(h, C.byref(b)), "ww_get_buffers")
def addr(v): return v if isinstance(v, int) else C.cast(v, C.c_void_p).value
u32 = lambda v, i=0: C.c_uint32.from_address(addr(v) + 4 * i)
u64 = lambda v: C.c_uint64.from_address(addr(v))
fields = [u64(b.checksum), u64(b.total_prp_count), u32(b.result_count), u32(b.primecount, 1), u32(b.overflow)]
kept = u32(b.primecount)
for f in fields + [kept]:
    f.value = 7
rt.cudaSetDevice(0)
assert L.ww_clear_results(h) == 0, L.ww_last_error()
now = C.c_int(-1)
rt.cudaGetDevice(C.byref(now))
assert now.value == 0  # the caller's device is left alone
assert [f.value for f in fields] == [0] * 5 and kept.value == 7
assert L.ww_clear_segment(h) == 0 and kept.value == 0
L.ww_close(h)
print("ok")
"""


def test_clear_results_from_a_thread_on_another_device(tmp_path, ww):
    """Clearing a context of device 1 while the thread's device is 0 works
    (ww_test_prps_host and ww_count_prps set the device themselves, so the
    caller of clear, test, read need not), zeroes every counter but the
    segment's, and leaves the thread's device as it was."""
    so = tmp_path / "libfake.so"
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-Wall", "-o", str(so), str(HERE / "fake_cudart.c")], check=True)
    r = subprocess.run([sys.executable, "-c", SCRIPT, str(Path(ww.__file__).parent), str(so)], capture_output=True,
                       text=True, env={**os.environ, "LD_PRELOAD": str(so)}, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
