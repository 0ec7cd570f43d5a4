"""A paint call that fails after its set-up (device memory runs out) is discarded whole: the next
calls paint what they would have painted without it.  The failure is a cudaMalloc that a preloaded
shim refuses, in a process of its own; no device memory is used up."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
int shim_refuse = 0; /* the refused call, counted from the next one; 0: none */
int shim_refused = 0;
int cudaMalloc(void **p, size_t n) {
  static int (*real)(void **, size_t);
  /* the runtime that the library has loaded */
  if (!real)
    real = (int (*)(void **, size_t))dlsym(dlopen("libcudart.so.13", RTLD_LAZY), "cudaMalloc");
  if (shim_refuse > 0 && --shim_refuse == 0) {
    shim_refused++;
    return 2; /* cudaErrorMemoryAllocation */
  }
  return real(p, n);
}
"""

PROGRAM = r"""
import ctypes, sys
import numpy as np
sys.path[:0] = ["tests", "oracle"]
import catalogs
import matt_young_mapmaking_gb300 as p2m

shim = ctypes.CDLL(sys.argv[1])
refuse = ctypes.c_int.in_dll(shim, "shim_refuse")
refused = ctypes.c_int.in_dll(shim, "shim_refused")
tab = catalogs.table(nu=0.0)
first = catalogs.shell(5, 20_000, r=(500.0, 3000.0), m=(2e13, 3e15))
other = catalogs.shell(6, 9_000, r=(500.0, 3000.0), m=(2e13, 3e15))
# the same number of records, with discs of many rings: their items need more memory
large = catalogs.shell(7, 20_000, r=(100.0, 300.0), m=(1e15, 3e15))


def painter():
    pt = p2m.Painter(nside=256, precision="fixed", maps=((0, 1), (0, 2)), zmax=6.0,
                     max_records=20_000)
    pt.load_table(0, tab)
    # halos are sorted from 608 on: nsm * 128 / 32 * 1
    pt.set_tuning(sort_halos=1, halos_grid=1, halo_batch=1, big_rings=16)
    return pt


def maps(pt):
    return [pt.healpix(m) for m in range(2)]


def paint_nothing_lost(pt, rec):
    try:
        pt.paint_records(rec)
    except p2m.P2MError as e:
        return e
    return None


with painter() as pt:
    pt.paint_records(first)
    pt.paint_records(other)
    want = maps(pt)
for reset in (False, True):
    for k in (1, 2):  # the items, their counts
        with painter() as pt:
            for _ in range(3):  # every other buffer gets its size
                pt.paint_records(first)
            pt.flush()
            pt.reset()
            if not reset:
                pt.paint_records(first)
            refuse.value, refused.value = k, 0
            assert paint_nothing_lost(pt, large) is not None and refused.value == 1
            refuse.value = 0
            if reset:
                pt.reset()
                pt.paint_records(first)
            pt.paint_records(other)
            got = maps(pt)
        for a, b in zip(got, want):
            assert np.array_equal(a, b)
print("same")
"""


def test_a_paint_call_out_of_memory_leaves_nothing(tmp_path):
    """With the failed call's halos left in the sort's counts, the next sort would place halos past
    the end of their order."""
    src, so = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", str(src), "-o", str(so), "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", PROGRAM, str(so)], cwd=ROOT, stdout=subprocess.PIPE,
                       stderr=subprocess.STDOUT, text=True, timeout=300,
                       env=dict(os.environ, LD_PRELOAD=str(so)))
    assert r.returncode == 0 and r.stdout.strip().endswith("same"), r.stdout
