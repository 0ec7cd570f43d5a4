"""The FP64 and fixed-point read-outs by painted tiles: repeated without a reset (they add to maps
that hold a read-out), into bound buffers of any alignment, for discs of every size."""
import numpy as np
import pytest

import catalogs
import matt_young_mapmaking_gb300 as p2m

pytestmark = pytest.mark.gpu


def catalogue(seed):
    """Small discs, discs of many rings and discs of tens of degrees: tiles flagged one by one and
    in long spans, around the poles and across longitude 0."""
    return np.concatenate([catalogs.shell(seed, 3000, r=(500.0, 3000.0), m=(1e13, 3e15)),
                           catalogs.shell(seed + 1, 60, r=(30.0, 300.0), m=(1e14, 3e15)),
                           catalogs.shell(seed + 2, 6, r=(8.0, 20.0), m=(1e14, 3e15)),
                           catalogs.edge_cases()[:12]])


@pytest.mark.parametrize("offset", [0, 1, 2])
@pytest.mark.parametrize("precision", ["fixed", "fp64", "mixed64"])
@pytest.mark.parametrize("nside,nmaps,cones", [(1, 2, 0), (2, 3, 5), (16, 1, 5), (256, 8, 0),
                                               (256, 2, 3), (1024, 1, 0), (1024, 2, 0), (1024, 3, 0)])
def test_repeated_readouts_add_up(nside, nmaps, cones, precision, offset):
    """A second read-out adds its catalogue's sums to the first's map, one float addition a pixel:
    equal bit for bit in fixed point, whose sums do not depend on the order.  The FP64 sums'
    order can move either map by one float ulp, and the addition rounds once more: three ulps of
    the largest of the three values.  Pixels that neither catalogue paints stay zero, and nothing
    is written beside a bound buffer."""
    import torch
    maps = tuple((0, 1 + (m & 1)) for m in range(nmaps))
    recs = [catalogue(101), catalogue(111)]
    npix = 12 * nside * nside * max(cones, 1)
    bufs = [torch.full((npix + 4,), 7.0, device="cuda") for _ in range(nmaps)]

    def paint(pt, rec):
        if cones:
            pt.paint_ensemble(rec, np.linspace(0, len(rec), cones + 1).astype(np.int64))
        else:
            pt.paint_records(rec)
        pt.flush()

    with p2m.Painter(nside=nside, precision=precision, maps=maps, zmax=6.0, ncones=cones,
                     max_records=4096) as pt:
        pt.load_table(0, catalogs.table(nu=0.0))
        alone = []
        for rec in recs:
            pt.reset()
            paint(pt, rec)
            alone.append([pt.healpix(m) for m in range(nmaps)])
        pt.reset()
        for m in range(nmaps):
            pt.bind_healpix_device(m, bufs[m][offset:].data_ptr())
        for rec in recs:
            paint(pt, rec)
        pt.synchronize()
        pt.reset()  # and nothing is left for the next catalogue
        for m in range(nmaps):
            pt.bind_healpix_device(m, 0)
        paint(pt, recs[0])
        again = [pt.healpix(m) for m in range(nmaps)]
    for m in range(nmaps):
        got = bufs[m].cpu().numpy()
        assert (got[:offset] == 7.0).all() and (got[offset + npix:] == 7.0).all()
        got, a, b = got[offset:offset + npix], alone[0][m], alone[1][m]
        assert a.any() and b.any()
        if precision == "fixed":
            assert np.array_equal(got, a + b)
            assert np.array_equal(again[m], a)
        else:
            top = np.maximum(np.maximum(np.abs(a), np.abs(b)), np.abs(got))
            assert np.all(np.abs(got - (a + b)) <= 3 * np.spacing(top))
            assert np.all(np.abs(again[m] - a) <= np.spacing(np.maximum(np.abs(a), np.abs(again[m]))))
            assert not got[(a == 0) & (b == 0)].any()
