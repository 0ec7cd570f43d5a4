"""The calls without a context keep working after a cudaDeviceReset, which ends the CUDA context
that their device memory came from: in a process of its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
import ctypes
import numpy as np
import matt_young_mapmaking_gb300 as p2m

def results():
    rng = np.random.default_rng(3)
    f, h = rng.standard_normal(64 * 64), rng.standard_normal(12 * 32 * 32)
    return (np.frombuffer(p2m.make_maptable(1, 0.0, 0.0, nchit=5, nmht=5, nrt=40), dtype=np.uint8),
            p2m.cl_flatsky(f, fov_rad=0.17, ell_max=4000.0, nbins=20)["aa"],
            p2m.cl_healpix(h, lmax=40)["aa"])

want = results()
cudart = ctypes.CDLL("libcudart.so.13")  # the one that the library has loaded
for _ in range(3):
    assert cudart.cudaDeviceReset() == 0
    got = results()
    assert np.array_equal(got[0], want[0])
    for a, b in zip(got[1:], want[1:]):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
print("same")
"""


def test_calls_after_a_device_reset():
    """The order of the spectra's FP64 additions can differ from run to run (atomics): 1e-12 of the
    largest value; table images are equal."""
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, stdout=subprocess.PIPE,
                       stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("same"), r.stdout
