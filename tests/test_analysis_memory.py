"""An analysis that runs out of host memory ends in CULIPX_OOM and gives back
what it had taken.  In a child process: its address space is limited, a little
less each time, until the analysis fails, and is then compared with what it was
before the failing call."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes, resource, sys
import culip_b200 as cb
from culip_b200 import _capi as capi

def address_space():
    return next(int(line.split()[1]) << 10 for line in open("/proc/self/status") if line.startswith("VmSize"))

n, m = 60000, 30000
rp, ci, v = cb.kkt_generate(n, m, 6, 32, 1e-2, 1e2)
bs = cb.kkt_blocking(n, m, 32)
h = ctypes.c_void_p()
capi.call("culipx_handle_create", ctypes.byref(h), -1, None)
ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)

def analyze():
    p = ctypes.c_void_p()
    status = capi.load().culipx_pattern_analyze(h, n + m, ptr(rp), ptr(ci), len(bs) - 1, ptr(bs), 0, ctypes.c_double(1.0),
                                                cb.F64, ctypes.byref(p))
    return status, p

first = analyze()  # the worker threads and their arenas exist from here on
assert first[0] == 0
held = address_space()
second = analyze()
held = address_space() - held  # what one pattern keeps
for s in (first, second):
    capi.load().culipx_pattern_destroy(s[1])
unlimited = resource.getrlimit(resource.RLIMIT_AS)
margin = 1 << 28
while True:
    before = address_space()
    resource.setrlimit(resource.RLIMIT_AS, (before + margin, unlimited[1]))
    status, p = analyze()
    resource.setrlimit(resource.RLIMIT_AS, unlimited)
    if status != 0:
        break
    capi.load().culipx_pattern_destroy(p)
    margin = int(margin * 0.97)
print(status == capi.OOM, held, address_space() - before)
"""


@pytest.mark.skipif(not os.path.exists("/proc/self/status"), reason="needs /proc")
def test_a_failed_analysis_gives_its_memory_back():
    env = dict(os.environ, OMP_NUM_THREADS="2", MALLOC_MMAP_THRESHOLD_="65536", MALLOC_ARENA_MAX="2", PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", CHILD], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0, r.stderr
    oom, held, grown = r.stdout.split()
    assert oom == "True"
    assert int(held) > 1 << 23
    assert int(grown) < int(held) // 4
