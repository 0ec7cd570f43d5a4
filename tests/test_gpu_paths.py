"""Painting paths against each other: a faster path gives the result of the one it stands
in for, bit for bit where both carry the same sums."""
import numpy as np
import pytest

import catalogs
import matt_young_mapmaking_gb300 as p2m
import oracle
from test_gpu_parity import assert_maps_close

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


def first_pixel(nside, ring):
    """(first pixel, pixels, longitude of the first) of a ring, from the RING layout."""
    n, i = nside, min(ring, 4 * nside - ring)
    npr = 4 * min(i, n)
    if ring < n:
        first, shift = 2 * ring * (ring - 1), 0.5
    elif ring <= 3 * n:
        first, shift = 2 * n * (n - 1) + (ring - n) * 4 * n, 0.5 * ((ring - n + 1) % 2)
    else:
        first, shift = 12 * n * n - 2 * i * (i + 1), 0.5
    return first, npr, 2 * np.pi * shift / npr


@pytest.mark.parametrize("two", [True, False])
@pytest.mark.parametrize("nside,lmax", [(1, 4), (2, 7), (8, 20), (128, 131), (512, 64),
                                        (2048, 66), (4096, 40), (8192, 17)])
def test_sphere_spectra_of_sparse_maps(nside, lmax, two):
    """Ring transforms of every kind (power-of-two rings, chirp convolutions in one piece and
    in halves, rings of one quarter-pixel) and several groups of rings: maps that are zero but for
    some pixels of a few rings, whose a_lm are short direct sums.  The direct sum and the
    library round differently in each of ~l steps: 1e-10 of the largest C_l."""
    import spectra
    rng = np.random.default_rng(nside + lmax)
    rings = sorted({1, 2, 3, nside - 1, nside, nside + 1, 2 * nside, 2 * nside + 1, 3 * nside + 1,
                    4 * nside - 1, 4 * nside - 3, *rng.integers(1, 4 * nside, 12).tolist()}
                   & set(range(1, 4 * nside)))
    maps = np.zeros((2, 12 * nside * nside), dtype=np.float32)
    alm = np.zeros((2, lmax + 1, lmax + 1), dtype=np.complex128)
    thetas = np.array([spectra.healpix_rings(nside)[r - 1][0] for r in rings]) if nside <= 128 \
        else np.array([np.arccos(ring_z(nside, r)) for r in rings])
    lam = spectra._ylm_theta(lmax, thetas)
    for k, ring in enumerate(rings):
        first, npr, phi0 = first_pixel(nside, ring)
        js = np.unique(rng.integers(0, npr, 5))
        for q in range(2):
            v = rng.standard_normal(js.size).astype(np.float32)
            maps[q, first + js] = v
            phase = np.exp(-1j * np.outer(np.arange(lmax + 1), phi0 + 2 * np.pi * js / npr)) @ v
            alm[q] += lam[:, :, k] * phase
    alm *= 4 * np.pi / maps.shape[1]
    want = {"aa": spectra.cl_from_alm(alm[0], alm[0])}
    if two:
        want["ab"] = spectra.cl_from_alm(alm[0], alm[1])
        want["bb"] = spectra.cl_from_alm(alm[1], alm[1])
    got = p2m.cl_healpix(maps[0], maps[1] if two else None, lmax=lmax)
    assert set(got) == set(want)
    for key in want:
        assert np.abs(got[key] - want[key]).max() <= 1e-10 * np.abs(want[key]).max()


def ring_z(nside, ring):
    i = min(ring, 4 * nside - ring)
    z = 1 - i * i / (3.0 * nside * nside) if i < nside else (2 * nside - i) / (1.5 * nside)
    return z if ring <= 2 * nside else -z


@pytest.mark.parametrize("cones", [0, 5])
@pytest.mark.parametrize("nmaps", [1, 2, 3, 8])
@pytest.mark.parametrize("nside", [1, 2, 16, 256])
def test_painted_tiles_are_read_and_cleared(nside, nmaps, cones):
    """The FP64 and fixed-point read-outs visit and clear only the tiles that were painted
    (tiles may straddle the end of the map or two cones' maps): after another catalogue,
    read or dropped by a reset, the fixed-point maps are those of a new painter bit for
    bit, and every pixel outside them is zero."""
    maps = tuple((0, 1 + (m & 1)) for m in range(nmaps))
    near = catalogs.shell(81, 4000, r=(30.0, 400.0), m=(1e14, 3e15))
    far = catalogs.shell(82, 6000, m=(1e13, 3e15))
    tab = catalogs.table(nu=0.0)
    off = np.linspace(0, len(near), 6).astype(np.int64), np.linspace(0, len(far), 6).astype(np.int64)

    def painter():
        pt = p2m.Painter(nside=nside, precision="fixed", maps=maps, zmax=6.0, ncones=cones,
                         max_records=len(far))
        pt.load_table(0, tab)
        return pt

    def paint(pt, rec, o):
        if cones:
            pt.paint_ensemble(rec, o)
        else:
            pt.paint_records(rec)

    with painter() as pt:
        paint(pt, far, off[1])
        want = [pt.healpix(m) for m in range(nmaps)]
    with painter() as pt:
        for read in (True, False):
            paint(pt, near, off[0])
            pt.flush() if read else pt.synchronize()
            pt.reset()
            paint(pt, far, off[1])
            for m in range(nmaps):
                assert np.array_equal(pt.healpix(m), want[m])
            pt.reset()
            assert all(not pt.healpix(m).any() for m in range(nmaps))


@pytest.mark.parametrize("offset", [0, 1, 2])
@pytest.mark.parametrize("nside", [1, 2, 64, 512])
def test_map_statistics_of_any_alignment(nside, offset):
    """Moments and P(<y) of maps read 16 bytes at a time or one value at a time (a bound
    buffer off its 16-byte alignment), and of flat-sky maps whose size is no multiple of
    4.  Sums: float-float per thread (2^-44) and FP64 across threads, 1e-12 of the sum of
    magnitudes; counts: equal."""
    import torch
    rec = np.concatenate([catalogs.shell(91, 20_000, m=(1e13, 3e15)),
                          catalogs.cone(92, 500, (0, 0, 1), 3.0)])
    npix = 12 * nside * nside
    buf = torch.full((npix + 4,), 7.0, dtype=torch.float32, device="cuda")
    with p2m.Painter(nside=nside, npix_fs=63, fov_deg=10.0, zmax=6.0, max_records=len(rec)) as pt:
        pt.load_table(0, catalogs.table(nu=0.0))
        pt.bind_healpix_device(0, buf[offset:].data_ptr())
        pt.paint_records(rec)
        mom, rms, dpdy = pt.map_stats(0)
        fmom, frms, _ = pt.map_stats(0, flatsky=True)
        flat = pt.flatsky(0)
        hp = pt.healpix(0)
    assert np.array_equal(hp, buf[offset:offset + npix].cpu().numpy())
    assert (buf[:offset] == 7.0).all() and (buf[offset + npix:] == 7.0).all()
    for x, m, r in ((hp, mom, rms), (flat, fmom, frms)):
        x = x.astype(np.float64)
        for k in range(3):
            assert abs(m[k] - (x ** (k + 1)).mean()) <= 1e-12 * (np.abs(x) ** (k + 1)).mean()
        var = ((x - x.mean()) ** 2).mean()
        assert abs(r * r - var) <= 1e-11 * (x * x).mean()
    dy = np.float32(1e-4) / np.float32(10000)
    q = hp / dy
    m = q[(q > -1) & (q < 10000)].astype(np.int64)
    count = np.bincount(m, minlength=10000).astype(np.float32)
    assert np.array_equal(dpdy, np.cumsum(count / np.float32(npix), dtype=np.float32))


@pytest.mark.parametrize("two", [True, False])
@pytest.mark.parametrize("npix", [4, 8, 16, 100, 512, 2048])
def test_flat_spectra_sizes(npix, two):
    """Transforms with an odd and an even number of radix-2 stages, the smallest and a large
    one, and a direct one, with bins narrower than a mode's spacing and wider.  FP64 FFTs
    of different orders: 1e-11 of the largest value."""
    import spectra
    rng = np.random.default_rng(npix)
    a = rng.standard_normal(npix * npix).astype(np.float32)
    b = (a + rng.standard_normal(npix * npix)).astype(np.float32)
    fov = float(np.float32(np.radians(10.0)))
    # no mode on a bin's edge, where the last bit of ell decides
    for ell_max, nbins in ((2 * np.pi / fov * npix * 0.4123457, 1000),
                           (2 * np.pi / fov * npix * 0.3234561, 7)):
        g = p2m.cl_flatsky(a, b if two else None, fov_rad=fov, ell_max=ell_max, nbins=nbins)
        r = spectra.cl_flatsky(a, b if two else None, fov, ell_max, nbins)
        assert np.array_equal(g["nmodes"], r["nmodes"])
        for key in ("ell", "aa") + (("ab", "bb") if two else ()):
            assert np.abs(g[key] - r[key]).max() <= 1e-11 * np.abs(r[key]).max()


@pytest.mark.parametrize("npix_fs", [1, 33, 97])
@pytest.mark.parametrize("precision", ["fp64", "mixed", "fixed"])
def test_flat_sky_readout_remainders(precision, npix_fs):
    """Flat-sky maps whose pixel count is no multiple of a block's: each map against the
    oracle, and the sum that the read-out adds up against the map's own (n FP64 additions
    on either side: n 2^-52 of the sum of magnitudes)."""
    rec = catalogs.cone(75, 20_000, (1.0, 0.0, 0.0), 8.0)
    tab = catalogs.table(nu=0.0)
    p = oracle.params(nside=0, npix_fs=npix_fs, maps=MAPS, nfloat=rec.shape[1], fov_deg=10.0)
    rfs = oracle.paint(p, [oracle.Table(tab)], rec, record_sets=False)[1]
    with p2m.Painter(nside=0, npix_fs=npix_fs, precision=precision, maps=MAPS, fov_deg=10.0,
                     max_records=len(rec)) as pt:
        pt.load_table(0, tab)
        pt.paint_records(rec)
        got = [pt.flatsky(m) for m in range(2)]
        sums = pt.stats()["fs_sum"]
    for m in range(2):
        assert_maps_close(got[m], rfs[m], rel=1e-6, what="map %d" % m)
        v = got[m].astype(np.float64)
        assert abs(sums[m] - v.sum()) <= v.size * 2.0**-52 * np.abs(v).sum()


@pytest.mark.parametrize("nchi,nm,nr", [(2, 2, 2), (3, 5, 127), (2, 3, 129), (300, 300, 2)])
@pytest.mark.parametrize("model,nu", [(1, 0.0), (2, 353.0)])
def test_table_sizes(model, nu, nchi, nm, nr):
    """Tables below a warp, at the edges of a block of radii, and of more cells than one pass
    takes: every entry is the reference's float sequence, so the image is the oracle's."""
    assert p2m.make_maptable(model, nu, 0.0, nchit=nchi, nmht=nm, nrt=nr) == \
        oracle.make_maptable(model, nu, 0.0, nchit=nchi, nmht=nm, nrt=nr)


@pytest.mark.parametrize("fn", [11, 12])
def test_table_quotients_are_rounded(fn):
    """The table maker's quotients are the IEEE ones: (m - 1) / (m + 1) at every mantissa that
    the logarithm centres, and x / x_c over random distances and core radii and over the
    mantissas next to powers of two."""
    import torch
    if fn == 11:
        x = np.arange(0x3f3504f4, 0x3fb504f4, dtype=np.uint32).view(np.float32)
        y, ref = x, (x - np.float32(1)) / (x + np.float32(1))
    else:
        rng = np.random.default_rng(76)
        x = np.exp(rng.uniform(np.log(4e-3), np.log(8.0), 1 << 22)).astype(np.float32)
        y = np.exp(rng.uniform(np.log(1e-2), np.log(10.0), 1 << 22)).astype(np.float32)
        near = (np.array([1.0], np.float32).view(np.uint32) + np.arange(-1024, 1024)).astype(np.uint32)
        y[: 1 << 20] = rng.choice(near, 1 << 20).view(np.float32)
        x[1 << 19: 1 << 21] = rng.choice(near, 3 << 19).view(np.float32)
        ref = x / y
    dx, dy = torch.from_numpy(x.copy()).cuda(), torch.from_numpy(y.copy()).cuda()
    out = torch.empty_like(dx)
    assert p2m.load_library().p2m_fmath_eval_device(0, fn, dx.data_ptr(), dy.data_ptr(),
                                                    out.data_ptr(), x.size) == 0
    got = out.cpu().numpy()
    assert np.array_equal(got, ref), "%d of %d differ" % ((got != ref).sum(), x.size)


@pytest.mark.parametrize("precision", ["mixed", "fixed", "fp64"])
def test_subnormal_radii_equal_the_exact_path(precision, monkeypatch):
    """A table whose first radii are subnormal floats: the fast logarithm is for normal ones, so
    such candidates take the exact path, and the maps are those of every candidate's exact path.
    The sums' order is the only difference: to one float ulp."""
    nchi, nm, nr = 3, 3, 60
    header = np.array([nchi, nm, nr], np.int32).tobytes() + np.array(
        [1e-37, 1e-35, 1e13, 1e16, 1e-41, 2e-37], np.float32).tobytes()
    rng = np.random.default_rng(5)
    image = header + rng.uniform(0.5, 1.5, 2 * nchi * nm * nr).astype(np.float32).tobytes()
    z = np.linspace(0.0, 6.0, 10000).astype(np.float32)
    rofz = np.linspace(0.0, 6e-36, 10000).astype(np.float32)

    def maps():
        with p2m.Painter(nside=512, precision=precision, maps=MAPS, zmax=6.0) as pt:
            pt.set_cosmology_tables(rofz, z, 6.0, 6000.0)
            pt.load_table(0, image)
            for k in range(40):
                v = np.random.default_rng(k).standard_normal(3)
                x, y, w = (1000.0 * v / np.linalg.norm(v)).tolist()
                pt.project_halo(x, y, w, 8.0, 1000.0, 1e14, 1.0, 1.0, 1 + (k & 1))
            out = [pt.healpix(m) for m in range(2)]
            return out, pt.stats()["hp_updates"]

    fast, n1 = maps()
    monkeypatch.setenv("P2M_BAND_U", "2")
    exact, n2 = maps()
    assert n1 == n2 > 10_000
    for a, b in zip(fast, exact):
        assert a.any()
        assert np.all(np.abs(a - b) <= np.spacing(np.maximum(np.abs(a), np.abs(b))))


@pytest.mark.parametrize("nchi,nm,nr", [(2, 2, 200), (3, 7, 129)])
@pytest.mark.parametrize("model,nu,alpha", [(3, 0.0, 0.0), (3, 217.0, 0.02), (2, 0.0, 0.0)])
def test_table_models_at_their_largest_exponents(model, nu, alpha, nchi, nm, nr):
    """Model 3, and model 2 without a frequency, with the smallest and the largest mass at the
    nearest and the farthest distance, where the profiles' exponents are largest: every entry is
    the reference's float sequence, so the image is the oracle's."""
    assert p2m.make_maptable(model, nu, alpha, nchit=nchi, nmht=nm, nrt=nr) == \
        oracle.make_maptable(model, nu, alpha, nchit=nchi, nmht=nm, nrt=nr)
