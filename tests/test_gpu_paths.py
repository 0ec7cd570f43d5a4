"""Painting paths against each other: a faster path gives the result of the one it stands
in for, bit for bit where both carry the same sums."""
import numpy as np
import pytest

import catalogs
import matt_young_mapmaking_gb300 as p2m

pytestmark = pytest.mark.gpu

MAPS = ((0, 1), (0, 2))


def pole_cone(n=3000):
    """Halos around the poles, where a candidate's longitude offset is large."""
    return np.concatenate([catalogs.cone(71, n, (0, 0, 1), 3.0, m=(1e13, 3e15)),
                           catalogs.cone(72, n, (0, 0, -1), 0.2, m=(1e13, 3e15))])


CATALOGUES = {"edges": catalogs.edge_cases, "poles": pole_cone,
              "shell": lambda: catalogs.shell(73, 60_000, m=(1e12, 3e15))}


def paint(rec, nside, precision, flags=0, maps=MAPS, **kw):
    with p2m.Painter(nside=nside, precision=precision, maps=maps, zmax=6.0, flags=flags,
                     max_records=max(len(rec), 1024), **kw) as pt:
        pt.load_table(0, catalogs.table(nu=0.0, nchit=40, nmht=40, nrt=200))
        pt.paint_records(rec)
        return [pt.healpix(m) for m in range(len(maps))], pt.stats()


@pytest.mark.parametrize("big_rings", [None, "0"])
@pytest.mark.parametrize("which", sorted(CATALOGUES))
@pytest.mark.parametrize("nside", [1, 16, 512, 4096])
def test_fp64_fast_path_equals_exact_path(nside, which, big_rings, monkeypatch):
    """The plain FP64 painter decides most candidates in float-float arithmetic.  Its
    decisions, table indices and fractions equal the double-precision path's bit for bit
    (validation of every candidate), and so do the maps painted with every candidate sent
    through that path (a recheck band of whole table cells).  A pixel's sum of a few floats
    is exact in double precision but for the deepest overlaps: the maps agree to one float
    ulp everywhere and bit for bit where a single halo deposits."""
    if big_rings is not None:
        monkeypatch.setenv("P2M_BIG_RINGS", big_rings)
    rec = CATALOGUES[which]()
    _, st = paint(rec, nside, "fp64", flags=p2m.FLAG_VALIDATE)
    assert st["val_checked"] == st["hp_candidates"]  # none on the coarsest maps
    assert st["val_bad_set"] == 0
    assert st["val_bad_index"] == 0
    fast, s1 = paint(rec, nside, "fp64")
    monkeypatch.setenv("P2M_BAND_U", "2")
    exact, s2 = paint(rec, nside, "fp64")
    assert s1["hp_updates"] == s2["hp_updates"] == st["hp_updates"]
    for a, b in zip(fast, exact):
        ulp = np.spacing(np.maximum(np.abs(a), np.abs(b)))
        assert np.all(np.abs(a.astype(np.float64) - b) <= ulp)
        assert np.mean(a != b) < 1e-4
