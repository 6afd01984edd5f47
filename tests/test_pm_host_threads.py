"""The photon mapper's host work (footprint radii, hash-cell size) when the
system gives no thread, or one and then no more: the calling thread takes over
the rest, with the same bits, and the process goes on. In a child process whose
default thread stack is larger than the address space, or larger than half of
the address space that it may still take."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = r"""
import array, ctypes, math, random, resource, sys, threading
lib = ctypes.CDLL(sys.argv[1])
lib.hasty_debug_pm_host.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_size_t, ctypes.c_float, ctypes.c_void_p]
w, h = int(sys.argv[2]), int(sys.argv[3])

def run():
    rnd = random.Random(5)
    d = array.array("f", [rnd.uniform(1.0, 9.0) if rnd.random() < 0.95 else -1.0 for _ in range(w * h)])
    cell = ctypes.c_float()
    assert lib.hasty_debug_pm_host(d.buffer_info()[0], w, h, 0.4, ctypes.byref(cell)) == 0
    return d.tobytes(), cell.value

want = run()
assert want[1] > 0.0 and math.isfinite(want[1]) and min(array.array("f", want[0])) >= 0.0
libc = ctypes.CDLL(None)
attr = ctypes.create_string_buffer(256)
threads = int(sys.argv[4])
stack = 1 << 30 if threads else 1 << 50
assert libc.pthread_attr_init(attr) == 0
assert libc.pthread_attr_setstacksize(attr, ctypes.c_size_t(stack)) == 0
assert libc.pthread_setattr_default_np(attr) == 0
if threads:
    size = [int(x.split()[1]) << 10 for x in open("/proc/self/status") if x.startswith("VmSize")][0]
    resource.setrlimit(resource.RLIMIT_AS, (size + stack * 3 // 2,) * 2)
started, go = [], threading.Event()
try:
    for _ in range(4):
        started.append(threading.Thread(target=go.wait))
        started[-1].start()
except RuntimeError:
    started.pop()
go.set()
for t in started:
    t.join()
assert len(started) == threads, len(started)
assert run() == want
print("same")
"""


@pytest.mark.parametrize("threads", [0, 1])
@pytest.mark.parametrize("w,h", [(17, 13), (320, 200)])   # below and above the sizes that use threads
def test_no_threads_left(w, h, threads):
    so = os.path.join(ROOT, "hastyrenderer_gb300", "lib", "libhasty_gb300.so")
    r = subprocess.run([sys.executable, "-c", CHILD, so, str(w), str(h), str(threads)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", (r.returncode, r.stderr)
