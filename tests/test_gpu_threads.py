"""The calls without a context, from several host threads at once: each gives what it gives
alone, whatever sizes the others ask for."""
import threading

import numpy as np
import pytest

import matt_young_mapmaking_gb300 as p2m

pytestmark = pytest.mark.gpu


def sphere(nside, lmax):
    m = np.random.default_rng(nside).standard_normal(12 * nside * nside).astype(np.float32)
    return lambda: p2m.cl_healpix(m, lmax=lmax)["aa"]


def flat(npix):
    m = np.random.default_rng(npix).standard_normal(npix * npix).astype(np.float32)
    return lambda: p2m.cl_flatsky(m, fov_rad=0.17, ell_max=4000.0, nbins=20)["aa"]


def table(n):
    return lambda: np.frombuffer(p2m.make_maptable(1, 0.0, 0.0, nchit=n, nmht=n, nrt=n)[36:],
                                 dtype=np.float32)


@pytest.mark.parametrize("large,small,reps", [(sphere(1024, 4), sphere(1, 1), 300),
                                              (sphere(4096, 2), sphere(16, 20), 20),
                                              (flat(4096), flat(4), 40), (table(40), table(3), 60)],
                         ids=["sphere1024", "sphere4096", "flat4096", "table"])
def test_concurrent_calls_of_different_sizes(large, small, reps):
    """One thread repeats the large call, four the small one.  The order of the spectra's FP64
    additions can differ from run to run (atomics): 1e-12 of the largest value."""
    calls, errors, done = (large, small), [], threading.Event()
    want = [c() for c in calls]

    def work(k):
        try:
            for _ in range(reps if k == 0 else 1_000_000):
                got = calls[k]()
                assert np.abs(got - want[k]).max() <= 1e-12 * np.abs(want[k]).max()
                if k and done.is_set():
                    break
        except Exception as e:  # noqa: BLE001 -- reported by the main thread
            errors.append(e)
        finally:
            if k == 0:
                done.set()

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1, 1, 1, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
