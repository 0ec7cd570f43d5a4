"""The painting order: which catalogues are sorted by first ring, and what sorted painting gives."""
import numpy as np
import pytest

import catalogs
import matt_young_mapmaking_gb300 as p2m

pytestmark = pytest.mark.gpu

BATCH = 16  # the default halo_batch


def unsorted_most():
    """A batch for each warp of 1024 threads an SM."""
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count * 32 * BATCH


@pytest.mark.parametrize("precision,nmaps", [("mixed", 1), ("mixed", 2), ("mixed", 6),
                                             ("fp64", 2), ("fixed", 2)])
def test_sorted_from_one_halo_more_than_the_limit(precision, nmaps):
    n = unsorted_most()
    rec = catalogs.shell(61, n + 1, r=(100.0, 3000.0), m=(2e13, 3e15))
    maps = tuple((0, 1 + (m & 1)) for m in range(nmaps))
    with p2m.Painter(nside=64, precision=precision, maps=maps, zmax=6.0, flags=p2m.FLAG_TIMING,
                     max_records=len(rec)) as pt:
        pt.load_table(0, catalogs.table(nu=0.0))
        pt.paint_records(rec)
        pt.flush()
        assert pt.stats()["n_enumerated"] == len(rec)  # every record is a halo
        for k, ordered in ((n, False), (n + 1, True)):
            pt.reset()
            pt.paint_records(rec[:k])
            pt.flush()
            assert (pt.timings()["big_offsets"] > 0) == ordered, k


def paint(parts, nside, precision, maps, discarded=None, **tune):
    """Maps of a catalogue painted in parts, whether sorting is on and whether the sort ran."""
    with p2m.Painter(nside=nside, precision=precision, maps=maps, zmax=6.0, flags=p2m.FLAG_TIMING,
                     max_records=max(len(p) for p in parts)) as pt:
        pt.load_table(0, catalogs.table(nu=0.0))
        pt.set_tuning(**tune)
        for k, part in enumerate(parts):
            if k and discarded is not None:
                with pytest.raises(p2m.P2MError):
                    pt.paint_records(discarded)
            pt.paint_records(part)
        pt.flush()
        return [pt.healpix(m) for m in range(len(maps))], pt.timings()["big_offsets"] > 0


def assert_same(got, want, precision):
    """Fixed-point sums do not depend on the order.  Compensated ones keep every add's exact error:
    the low words' own rounding is 2^-24 of theirs, so the rounded sums agree to one float ulp."""
    for a, b in zip(got, want):
        if precision == "fixed":
            assert np.array_equal(a, b)
        else:
            assert np.all(np.abs(a - b) <= np.spacing(np.maximum(np.abs(a), np.abs(b))))


@pytest.mark.parametrize("split", ["one", "three", "discarded"])
@pytest.mark.parametrize("nside,precision", [(1, "fixed"), (2, "fixed"), (2, "mixed"), (64, "mixed"),
                                             (64, "fixed"), (8192, "fixed")])
def test_sorted_painting_equals_the_catalogues_order(nside, precision, split):
    """The sort of 4 Nside + 1 first-ring counts, few and many, with the counts of several paint
    calls, and with those of a call that is discarded (a disc radius above pi) between them."""
    maps = ((0, 1),) if nside == 8192 else ((0, 1), (0, 2))
    rec = catalogs.shell(62, 6000, r=(100.0, 3000.0), m=(2e13, 3e15))
    parts = [rec] if split == "one" else np.array_split(rec, 3)
    bad = None
    if split == "discarded":
        bad = catalogs.shell(63, 500, r=(100.0, 3000.0), m=(2e13, 3e15)).copy()
        bad[250, :3] = (0.5, 0.5, 0.5)  # closer than its radius
    want, ran = paint(parts, nside, precision, maps, sort_halos=0)
    assert not ran
    got, ran = paint(parts, nside, precision, maps, bad, sort_halos=1, halos_grid=1, halo_batch=1)
    assert ran
    assert_same(got, want, precision)


@pytest.mark.parametrize("precision", ["fixed", "mixed"])
@pytest.mark.parametrize("tune", [dict(halos_grid=1, halo_batch=32),
                                  dict(halos_grid=1, halo_batch=8, sort_halos=0),
                                  dict(halos_grid=1, halos_threads=256, halo_batch=16),
                                  dict(big_rings=0, full_grid=1, full_chunk=65536),
                                  dict(big_rings=0, full_grid=1, full_chunk=1000)])
def test_whole_batches_and_chunks(tune, precision):
    """Catalogues large enough that the batches and chunks are those that were asked for: more
    halos than 608 (or 1216) warps' batches of 32, and more candidates than 1216 warps' chunks."""
    maps = ((0, 1), (0, 2))
    if "big_rings" in tune:
        rec = catalogs.shell(64, 1500, r=(8.0, 12.0), m=(1e15, 3e15))
        nside, least = 512, 1216 * tune["full_chunk"]
    else:
        rec = catalogs.shell(65, 45_000, r=(100.0, 3000.0), m=(2e13, 3e15))
        nside, least = 64, 0
    with p2m.Painter(nside=nside, precision=precision, maps=maps, zmax=6.0,
                     max_records=len(rec)) as pt:
        pt.load_table(0, catalogs.table(nu=0.0))
        pt.paint_records(rec)
        want = [pt.healpix(m) for m in range(2)]
        st = pt.stats()
        assert st["n_enumerated"] == len(rec) and st["hp_candidates"] > least
    got, _ = paint([rec], nside, precision, maps, **tune)
    assert_same(got, want, precision)
