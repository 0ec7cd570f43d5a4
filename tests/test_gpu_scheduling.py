"""Where a program has asked its waits for the GPU to block (cudaDeviceScheduleBlockingSync), a
paint call's wait for its set-up takes no core: in a process of its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
import ctypes, sys, time
sys.path[:0] = ["tests", "oracle"]
import catalogs
import matt_young_mapmaking_gb300 as p2m

lib = p2m.load_library()
assert ctypes.CDLL("libcudart.so.13").cudaSetDeviceFlags(int(sys.argv[1])) == 0
import torch
rec = torch.from_numpy(catalogs.shell(8, 4_000_000, r=(100.0, 8000.0), m=(1e13, 3e15))).cuda()
with p2m.Painter(nside=4096, maps=((0, 1), (0, 2)), zmax=6.0, max_records=len(rec)) as pt:
    pt.load_table(0, catalogs.table(nu=0.0))
    for rep in range(30):
        if rep == 5:
            wall, cpu = time.perf_counter(), time.thread_time()
        # each paint call waits for the last one's painting, about a millisecond
        pt.reset()
        pt.paint_records_device(rec.data_ptr(), len(rec), 10)
        pt.flush()
    wall, cpu = time.perf_counter() - wall, time.thread_time() - cpu
    pt.synchronize()
print("%.3f" % (cpu / wall))
"""


def share(flags):
    r = subprocess.run([sys.executable, "-c", PROGRAM, str(flags)], cwd=ROOT, stdout=subprocess.PIPE,
                       stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
    return float(r.stdout.split()[-1])


def test_a_paint_call_waits_as_the_device_flags_ask():
    """The calling thread's share of a core while it paints: near 1 where it polls; blocking, what
    the launches take of a pass of about 1.5 ms, with room for a busy machine."""
    assert share(4) < 0.5  # cudaDeviceScheduleBlockingSync
