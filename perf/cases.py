"""The work that users of the halo painter have it do, as measured cases.

Every case goes through the package's public entry points (``Painter``, ``make_maptable``,
``cl_healpix``, ``cl_flatsky``).  The kinds:

  paint   one catalogue (or an ensemble of light-cones) resident in device memory, painted
          to HEALPix maps in the caller's device buffers: reset, paint, maps ready.  With
          npix_fs also a flat-sky map, read out to the host.
  report  the pks2map flow on host data: records in page-locked host memory, painted as
          they are copied, the report's statistics, and the maps read back to the host.
  table   make_maptable: one profile table image.
  sphere  angular power spectra of two HEALPix maps in host memory.
  flat    binned power spectra of two flat-sky maps in host memory.

``exact`` states the same results in 64-bit torch and numpy.
"""
import functools
import math

import numpy as np
import torch

import matt_young_mapmaking_gb300 as p2m

DEV = "cuda"
# map sets: one Compton-y map, y + kSZ of one table, tSZ at five frequencies + kSZ
FREQS = (148.0, 200.0, 218.0, 353.0, 545.0)
MAPS = {"y": ((0, 1),), "yk": ((0, 1), (0, 2)),
        "bands": tuple((t, 1) for t in range(len(FREQS))) + ((0, 2),)}
FOV_DEG = 10.0
ZMAX = 6.0


def _paint(name, n, nside, maps="yk", precision="mixed", nfloat=10, rmax=8000.0, mmax=3e15,
           cones=0, npix_fs=0):
    case = {"kind": "paint", "n": n, "nside": nside, "maps": maps, "precision": precision,
            "nfloat": nfloat, "rmax": rmax, "mmax": mmax, "cones": cones, "npix_fs": npix_fs}
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # a quick look: a small catalogue on a coarse map, where latency is all there is
        _paint("quick look 2e4 at 256", 20_000, 256, rmax=3000.0, mmax=1e15),
        # the precision form's catalogue with a flat-sky cut-out beside the full sky
        _paint("1e5 at 512 and flat 1024", 100_000, 512, maps="y", rmax=3000.0, mmax=1e15,
               npix_fs=1024),
        # one y map of an odd-sized catalogue in the seven-float layout
        _paint("y of 1000003 at 2048", 1_000_003, 2048, maps="y", nfloat=7, rmax=5000.0),
        # the headline workload: y + kSZ of 1e7 halos at Nside 4096
        _paint("headline 1e7 at 4096", 10_000_000, 4096),
        # the plain FP64 painter, for users who want no mixed precision
        _paint("fp64 1e6 at 2048", 1_000_000, 2048, precision="fp64"),
        # maps that are bit-identical from run to run
        _paint("fixed point 3e6 at 2048", 3_000_000, 2048, precision="fixed", rmax=6000.0),
        # component-separation input: five frequencies and kSZ in one enumeration
        _paint("six maps of 4e6 at 4096", 4_000_000, 4096, maps="bands"),
        # many small independent light-cones in one call
        _paint("64 cones at 1024", 6_400_000, 1024, maps="y", rmax=4000.0, cones=64),
        # the command line's flow on host data
        {"name": "report 3e6 at 2048", "kind": "report", "n": 3_000_000, "nside": 2048,
         "maps": "yk", "nfloat": 10, "rmax": 8000.0, "mmax": 3e15},
        # the shipped table size, at one frequency
        {"name": "table 100 x 100 x 200", "kind": "table", "model": 1, "nu": 148.0,
         "nchi": 100, "nm": 100, "nr": 200},
        # spectra of the precision report: both maps' auto and cross spectra
        {"name": "sphere spectra at 512", "kind": "sphere", "nside": 512, "lmax": 1535},
        {"name": "flat spectra at 1024", "kind": "flat", "npix": 1024, "nbins": 100},
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    u = rng.random()
    if u < 0.70:
        maps = rng.choice(["y", "yk", "yk", "bands"])
        precision = rng.choice(["mixed", "mixed", "mixed", "mixed64", "fixed", "fp64"])
        cones = int(_log(rng, 2, 100)) if rng.random() < 0.15 else 0
        most, sides = 1e7, (256, 512, 1024, 2048, 4096)
        if maps == "bands":
            most = 3e6
        if precision == "fp64":
            most, sides = min(most, 1e6), sides[:4]
        if cones:
            maps, sides = "y", sides[:3]
        nside = rng.choice(sides)
        npix_fs = 0
        if not cones and rng.random() < 0.15:
            npix_fs = int(_log(rng, 64, 1500))
        return _paint(None, max(int(_log(rng, 1e3, most)), 20 * cones), nside, maps, precision,
                      rng.choice([7, 10, 10]), round(_log(rng, 1500.0, 8000.0), 1),
                      rng.choice([1e15, 3e15]), cones, npix_fs)
    if u < 0.80:
        return {"kind": "report", "n": int(_log(rng, 1e4, 5e6)),
                "nside": rng.choice([256, 512, 1024, 2048]), "maps": rng.choice(["y", "yk"]),
                "nfloat": rng.choice([7, 10]), "rmax": round(_log(rng, 1500.0, 8000.0), 1),
                "mmax": 3e15}
    if u < 0.86:
        return {"kind": "table", "model": rng.choice([1, 2, 3]),
                "nu": rng.choice([148.0, 353.0, 545.0]), "nchi": int(_log(rng, 20, 120)),
                "nm": int(_log(rng, 20, 120)), "nr": int(_log(rng, 40, 240))}
    if u < 0.93:
        nside = rng.choice([64, 128, 256, 512])
        return {"kind": "sphere", "nside": nside,
                "lmax": int(nside * rng.uniform(1.0, 3.0)) - 1}
    return {"kind": "flat", "npix": rng.choice([128, 256, 300, 500, 512, 1024, 1024]),
            "nbins": rng.choice([30, 64, 100])}


# ------------------------------------------------------------------------ preparation ----

def _offsets(case):
    """First record of each cone: uneven cones, the same for every seed."""
    r = np.random.default_rng(5 + case["cones"])
    w = np.exp(r.uniform(np.log(1.0), np.log(100.0), case["cones"]))
    cut = np.floor(np.cumsum(w) / w.sum() * case["n"]).astype(np.int64)
    cut[-1] = case["n"]
    return np.concatenate([[0], cut])


def _records(case, seed):
    return p2m.generate_catalogue(seed + 1, case["n"], case["nfloat"], r=(100.0, case["rmax"]),
                                  m=(1e12, case["mmax"]))


def _table_freqs(case):
    return FREQS if case["maps"] == "bands" else (0.0,)


def _painter(case, **kw):
    pt = p2m.Painter(nside=case["nside"], maps=MAPS[case["maps"]], zmax=ZMAX,
                     max_records=case["n"], **kw)
    for slot, nu in enumerate(_table_freqs(case)):
        pt.load_table(slot, p2m.make_maptable(1, nu, 0.0))
    return pt


def _host_maps(n, seed):
    """Two float32 host maps with a long-tailed y-like and a signed kSZ-like distribution."""
    g = torch.Generator(device=DEV).manual_seed(seed + 1)
    y = 1e-7 * torch.exp(1.5 * torch.randn(n, generator=g, device=DEV))
    k = 1e-7 * torch.randn(n, generator=g, device=DEV) + 0.1 * y
    return y.float().cpu().numpy(), k.float().cpu().numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "paint":
        pt = _painter(case, precision=case["precision"], npix_fs=case["npix_fs"],
                      fov_deg=FOV_DEG, ncones=case["cones"])
        npix = 12 * case["nside"] ** 2 * max(case["cones"], 1)
        out = [torch.empty(npix, dtype=torch.float32, device=DEV) for _ in MAPS[case["maps"]]]
        for m, o in enumerate(out):
            pt.bind_healpix_device(m, o.data_ptr())
        return {"case": case, "pt": pt, "out": out,
                "rec": torch.from_numpy(_records(case, seed)).to(DEV),
                "off": _offsets(case) if case["cones"] else None}
    if kind == "report":
        npix = 12 * case["nside"] ** 2
        return {"case": case, "pt": _painter(case),
                "rec": torch.from_numpy(_records(case, seed)).pin_memory(),
                "out": [torch.empty(npix, dtype=torch.float32).pin_memory()
                        for _ in MAPS[case["maps"]]]}
    if kind == "table":
        # the exponent of T_CMB's redshift dependence is the input that varies
        return {"case": case, "alpha": _alpha(seed)}
    n = 12 * case["nside"] ** 2 if kind == "sphere" else case["npix"] ** 2
    a, b = _host_maps(n, seed)
    return {"case": case, "a": a, "b": b}


def _alpha(seed):
    return (seed * 0.6180339887) % 0.2


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "paint":
        pt, rec = state["pt"], state["rec"]
        pt.reset()
        if case["cones"]:
            pt.paint_ensemble_device(rec.data_ptr(), state["off"], case["nfloat"])
        else:
            pt.paint_records_device(rec.data_ptr(), case["n"], case["nfloat"])
        for m, o in enumerate(state["out"]):
            pt.healpix_device(m, o.data_ptr())
        if not case["npix_fs"]:
            return state["out"]
        return state["out"] + [pt.flatsky(m) for m in range(pt.nmaps)]
    if kind == "report":
        pt = state["pt"]
        pt.reset()
        pt.paint_records(state["rec"].numpy())
        mom, rms, dpdy = pt.map_stats(0)
        for m, o in enumerate(state["out"]):
            pt.healpix_into(m, o.data_ptr())
        return state["out"] + [np.array(mom + [rms]), dpdy]
    if kind == "table":
        img = p2m.make_maptable(case["model"], case["nu"], state["alpha"], case["nchi"],
                                case["nm"], case["nr"])
        return np.frombuffer(img, dtype=np.float32, offset=36)
    if kind == "sphere":
        return p2m.cl_healpix(state["a"], state["b"], lmax=case["lmax"])
    return p2m.cl_flatsky(state["a"], state["b"], fov_rad=math.radians(FOV_DEG),
                          ell_max=8000.0, nbins=case["nbins"])


def work(case):
    kind = case["kind"]
    if kind in ("paint", "report"):
        nmaps = len(MAPS[case["maps"]])
        npix = 12 * case["nside"] ** 2 * max(case.get("cones", 0), 1)
        npix += case.get("npix_fs", 0) ** 2
        return {"bytes": 4.0 * (case["n"] * case["nfloat"] + nmaps * npix), "flops": 0.0}
    if kind == "table":
        n = case["nchi"] * case["nm"] * case["nr"]
        # two line-of-sight integrals of up to 401 steps, two powers (about 40 operations
        # each) a step
        return {"bytes": 8.0 * n, "flops": n * 2 * 401 * 80.0}
    if kind == "sphere":
        npix, lmax, rings = 12 * case["nside"] ** 2, case["lmax"], 2 * case["nside"]
        # an FFT per ring, then per (l, m, ring pair) the recursion and four sums
        return {"bytes": 8.0 * npix,
                "flops": 5.0 * npix * math.log2(4 * case["nside"])
                + 0.5 * (lmax + 1) * (lmax + 2) * rings * 12.0}
    n = case["npix"] ** 2
    return {"bytes": 8.0 * n, "flops": 5.0 * n * math.log2(n)}


# ------------------------------------------------------------- the results in 64 bits ----

PI = math.pi
OM, OL, H0, OB = 0.25, 0.75, 0.7, 0.043
RHO0 = 2.775e11 * OM * H0 * H0
RHOCRIT0 = 2.775e11 * H0 * H0
DELTA = (200.0, 500.0, 200.0)
NZ, ZTAB, RTAB = 10000, 6.0, 1.3e4


@functools.lru_cache(maxsize=None)
def _distances():
    """r(z) and z(r): Euler steps of dz/dr = H(z)/c over 10000 entries."""
    dzdr = lambda z: H0 * 100.0 / 2.99792458e5 * math.sqrt(OM * (1 + z) ** 3 + 1 - OM)  # noqa: E731
    dz, dr = ZTAB / (NZ - 1), RTAB / (NZ - 1)
    r, z = [0.0], [0.0]
    for i in range(1, NZ):
        r.append(r[-1] + dz / dzdr(i * dz))
        z.append(z[-1] + dr * dzdr(z[-1]))
    return (torch.tensor(r, dtype=torch.float64, device=DEV), dz,
            torch.tensor(z, dtype=torch.float64, device=DEV), dr)


def _lookup(tab, step, x):
    t = (x / step).clamp(0, NZ - 1)
    i = t.long().clamp(max=NZ - 2)
    f = t - i
    return (1 - f) * tab[i] + f * tab[i + 1]


def _rhocrit(z):
    c = (1 + z) ** 3
    return RHOCRIT0 * (OM * c + OL) / c


TABLE_BOUNDS = ((1e2, 7e3), (1e13, 1e16), (1e-2, 10.0))  # Mpc, Msun, Mpc
# P0, xc, beta of the pressure and P0, alpha, beta of the density: A, mass and (1+z) powers
BBPS = (((18.1, 0.154, -0.758), (0.497, -0.00865, 0.731), (4.35, 0.0393, 0.415),
         (1.9e-5, 0.29, -0.67), (0.88, -0.03, 0.20), (3.83, 0.044, -0.025)),
        ((7.49, 0.226, -0.957), (0.71, -0.0833, 0.853), (4.19, 0.048, 0.615),
         (9.1e-5, 0.10, -0.92), (0.69, -0.02, 0.27), (4.43, 0.0035, 0.037)),
        ((20.7, -0.074, -0.743), (0.438, 0.011, 1.01), (3.82, 0.0375, 0.535),
         (1.5e-4, 0.14, -1.32), (0.68, -0.02, 0.29), (6.4, 0.028, -0.25)))


@functools.lru_cache(maxsize=2)
def _table64(model, nchi, nm, nr):
    """Profile table [chi, M, r, (y without the spectral factor, tau)], and 1 + z of chi."""
    axes = [torch.exp(torch.linspace(math.log(a), math.log(b), n, dtype=torch.float64, device=DEV))
            for (a, b), n in zip(TABLE_BOUNDS, (nchi, nm, nr))]
    chi_c, mh, rt = axes
    rofz, dz, zofr, dr = _distances()
    z_c = _lookup(zofr, dr, chi_c)
    msun, mpc, kpc, c = 1.9891e33, 3.08567758e24, 3.08567758e21, 2.99792458e10
    ypm = 3 * 6.65246e-25 * (1e2 / 3.08567758e19) ** 2 / 8 / PI / 9.109383e-28 / c ** 2 * msun / 1.932
    tps = 6.65246e-25 / 1.136 / 1.67e-24 * msun / kpc ** 3 * mpc * 1e10
    delta = DELTA[model - 1]
    y0 = OB / OM * delta * H0 * H0 * ypm
    tau0 = tps * H0 * H0 * (0.75 / PI / delta) ** (1 / 3)
    steps = (torch.arange(1, 402, dtype=torch.float64, device=DEV) - 0.5) * 1e-2
    out = torch.empty(nchi, nm, nr, 2, dtype=torch.float64, device=DEV)
    for i in range(nchi):
        z = float(z_c[i])
        par = [a * (mh / 1e14) ** p * (1 + z) ** q for a, p, q in BBPS[model - 1]]
        par = [p[:, None, None] for p in par]
        chi = float(_lookup(rofz, dz, z_c[i]))
        rc = float(_rhocrit(z_c[i]))
        rvir = (3 * mh / 4 / PI / delta / rc) ** (1 / 3)
        b = chi * torch.sin(torch.atan(rt / chi_c[i]))[None, :] / rvir[:, None]
        inside = b <= 4.0
        x = torch.sqrt(steps ** 2 + b[..., None] ** 2)
        n2 = (torch.sqrt((16 - b * b).clamp(min=0)) / 1e-2 + 1e-9).long() + 1
        xx = x / par[1]
        pres = (par[0] * xx ** -0.3 * (1 + xx) ** -par[2]).sum(-1) * 1e-2
        xx = x / 0.5
        rho = par[3] * xx ** -0.2 * (1 + xx ** par[4]) ** (-(par[5] - 0.2) / par[4])
        k = torch.arange(1, 402, device=DEV)
        rho = (rho * (k <= n2[..., None])).sum(-1) * 2e-2
        fy = y0 * mh * (OM * (1 + z) ** 3 + OL)
        ft = tau0 * mh ** (1 / 3) / (1 + z) / rc ** (1 / 3)
        out[i, ..., 0] = torch.where(inside, fy[:, None] * pres, 0.0)
        out[i, ..., 1] = torch.where(inside, ft[:, None] * rho, 0.0)
    return out, 1 + z_c


def _full_table(model, nu, alpha, nchi=100, nm=100, nr=200):
    tab, zp1 = _table64(model, nchi, nm, nr)
    tab = tab.clone()
    if nu > 0:
        x = 0.017612 * nu * zp1 ** alpha
        g = x * (torch.exp(x) + 1) / (torch.exp(x) - 1) - 4
        tab[..., 0] *= g[:, None, None]
    return tab


def _halos(case, rec):
    """The halo loop's quantities of the records that pass the cuts, one row a halo."""
    p = rec[:, :3].double()
    chi = p.norm(dim=1)
    rofz, dz, zofr, dr = _distances()
    mass = 4.0 / 3.0 * PI * RHO0 * rec[:, 6].double() ** 3
    z = _lookup(zofr, dr, chi)
    chi_t = _lookup(rofz, dz, z)
    hi = float(_lookup(rofz, dz, torch.tensor(ZMAX, dtype=torch.float64, device=DEV)))
    keep = ((chi <= hi) & (mass >= 1e13) & (chi_t <= TABLE_BOUNDS[0][1])).nonzero()[:, 0]
    p, chi, mass, z, chi_t = p[keep], chi[keep], mass[keep], z[keep], chi_t[keep]
    omz = OM * (1 + z) ** 3 / (OM * (1 + z) ** 3 + 1 - OM) - 1
    mh = torch.sqrt((18 * PI ** 2 + 82 * omz - 39 * omz ** 2) / 200.0) * mass
    rh = (3 * mh / 4 / PI / 200 / _rhocrit(z)) ** (1 / 3)
    w2 = -(p * rec[keep, 3:6].double()).sum(1) / chi / 3e5
    return {"p": p, "chi": chi, "T": 4 * torch.asin(rh / chi), "chi_t": chi_t, "mh": mh, "w2": w2,
            "rec": keep}


def _cell(x, lo, hi, n):
    """Index (from 0) and unnormalised fraction of log x on the table's axis."""
    step = (math.log(hi) - math.log(lo)) / (n - 1)
    lx = torch.log(x)
    i = ((lx - math.log(lo)) / step).long()
    return i, lx - (math.log(lo) + i * step)


def _profile(h, sel, angle, tabs, maps):
    """Values of every map for halo indices sel at the given angles."""
    r = h["chi_t"][sel] * torch.tan(angle)
    nchi, nm, nr = tabs[0].shape[:3]
    (c0, c1), (m0, m1), (r0, r1) = TABLE_BOUNDS
    on = r <= r1
    ir, fr = _cell(r.clamp(min=r0 + 1e-5, max=r1), r0, r1, nr)
    ic, fc = _cell(h["chi_t"][sel].clamp(min=c0 + 1e-5), c0, c1, nchi)
    im, fm = _cell(h["mh"][sel].clamp(min=m0 + 1e-5, max=m1), m0, m1, nm)
    base = ir + nr * (im + nm * ic)
    # the chi step takes the mass fraction and the mass step the chi fraction, as the
    # reference's interpolation does
    terms = [(base, (1 - fc) * (1 - fm)), (base + nr, fc * (1 - fm)),
             (base + nr * nm, (1 - fc) * fm), (base + nr * nm + nr, fc * fm)]
    vals = []
    for slot, profile in maps:
        t = tabs[slot][..., profile - 1].reshape(-1)
        last = t.numel() - 1
        v = 0.0
        for off, w in terms:
            v = v + w * ((1 - fr) * t[off.clamp(max=last)] + fr * t[(off + 1).clamp(max=last)])
        vals.append(torch.where(on, v * (h["w2"][sel] if profile == 2 else 1.0), 0.0))
    return vals


def _ragged(count):
    """Owner and place within the owner of every element of a ragged list."""
    own = torch.repeat_interleave(torch.arange(count.numel(), device=DEV), count)
    start = torch.cumsum(count, 0) - count
    return own, torch.arange(own.numel(), device=DEV) - start[own]


def _rings(nside, i):
    """z, sin(theta), pixels, longitude shift and first pixel of ring i (from 1)."""
    f, n = i.double(), float(nside)
    s = 4 * nside - i
    cap = torch.minimum(i, s)
    polar = cap < nside
    c2 = cap.double() ** 2 / (3 * n * n)
    z = torch.where(polar, torch.where(i < s, 1 - c2, c2 - 1), (2 * n - f) / (1.5 * n))
    sth = torch.where(polar, torch.sqrt(c2 * (2 - c2)), torch.sqrt(((1 - z) * (1 + z)).clamp(min=0)))
    npr = 4 * cap.clamp(max=nside)
    shift = torch.where(polar | ((i + nside) % 2 == 0), 0.5, 0.0)
    belt = 2 * nside * (nside - 1) + (i - nside) * 4 * nside
    south = 12 * nside * nside - 2 * s * (s + 1)
    first = torch.where(polar, torch.where(i < s, 2 * i * (i - 1), south), belt)
    return z, sth, npr, shift, first


def _ring_of(nside, th):
    z, n = torch.cos(th), float(nside)
    a = n * math.sqrt(6) * torch.sin(th / 2)
    b = 4 * n - n * math.sqrt(6) * torch.cos(th / 2)
    return torch.where(z > 2 / 3, a, torch.where(z < -2 / 3, b, n * (2 - 1.5 * z)))


def _sky(case, h, tabs, cone):
    nside, maps = case["nside"], MAPS[case["maps"]]
    cone_pix = 12 * nside * nside
    out = [torch.zeros(cone_pix * max(case.get("cones", 0), 1), dtype=torch.float64, device=DEV)
           for _ in maps]
    p, chi, T = h["p"], h["chi"], h["T"]
    z0 = p[:, 2] / chi
    s0 = torch.sqrt(p[:, 0] ** 2 + p[:, 1] ** 2) / chi
    phi0 = torch.atan2(p[:, 1], p[:, 0]) % (2 * PI)
    th = torch.atan2(s0, z0)
    lo = torch.where(th - T > 0, _ring_of(nside, (th - T).clamp(min=0)).floor() - 1, 1.0)
    hi = torch.where(th + T < PI, _ring_of(nside, (th + T).clamp(max=PI)).ceil() + 1, 4.0 * nside)
    lo, hi = lo.long().clamp(1, 4 * nside - 1), hi.long().clamp(1, 4 * nside - 1)
    cost = torch.cumsum((hi - lo + 1) + cone_pix * T * T / 3, 0)
    C = 4 * torch.sin(T / 2) ** 2
    start, n = 0, chi.numel()
    while start < n:
        base = float(cost[start - 1]) if start else 0.0
        end = max(start + 1, int(torch.searchsorted(cost, base + 1.5e7)))
        end = min(end, n)
        own, k = _ragged(hi[start:end] - lo[start:end] + 1)
        own = own + start
        z, s, npr, shift, first = _rings(nside, lo[own] + k)
        A = (z - z0[own]) ** 2 + (s - s0[own]) ** 2
        B = 4 * s * s0[own]
        t = (C[own] - A) / B.clamp(min=1e-300)
        half = torch.asin(torch.sqrt(t.clamp(0, 1))) * npr / PI
        mid = phi0[own] * npr / (2 * PI) - shift
        j0 = (mid - half - 0.01).ceil()
        cnt = ((mid + half + 0.01).floor() - j0 + 1).clamp(min=0)
        full = (t >= 1) | (cnt >= npr)
        j0 = torch.where(full, torch.zeros_like(j0), j0).long()
        cnt = torch.where(full, npr, cnt.long())
        cnt = torch.where(t < -1e-9, torch.zeros_like(cnt), cnt)
        item, k = _ragged(cnt)
        j = j0[item] + k
        dphi = (j + shift[item]) * (2 * PI) / npr[item] - phi0[own[item]]
        c2 = A[item] + B[item] * torch.sin(dphi / 2) ** 2
        keep = (c2 < C[own[item]]).nonzero()[:, 0]
        item, j, c2 = item[keep], j[keep], c2[keep]
        sel = own[item]
        pix = first[item] + j % npr[item] + cone[sel] * cone_pix
        for o, v in zip(out, _profile(h, sel, 2 * torch.asin(torch.sqrt(c2) / 2), tabs, maps)):
            o.index_add_(0, pix, v)
        start = end
    return out


def _flat(case, h, tabs):
    npix, maps = case["npix_fs"], MAPS[case["maps"]]
    fov = math.radians(FOV_DEG)
    d = fov / npix
    out = [torch.zeros(npix * npix, dtype=torch.float64, device=DEV) for _ in maps]
    # the field's axes: theta from the record's third coordinate, phi from its second
    x, y = (torch.asin((h["p"][:, c] / h["chi"]).clamp(-1, 1)) for c in (2, 1))
    T = h["T"]
    near = (h["p"][:, 0] >= 0) & (x.abs() - 1.1 * T < fov / 2) & (y.abs() - 1.1 * T < fov / 2)
    sel0 = near.nonzero()[:, 0]
    x, y, T = x[sel0], y[sel0], T[sel0]
    at = lambda v: ((v + fov / 2) / d).floor().long().clamp(0, npix - 1)  # noqa: E731
    j0, j1, k0, k1 = at(x - T), at(x + T), at(y - T), at(y + T)
    for part in torch.arange(sel0.numel(), device=DEV).split(2000):
        own, t = _ragged(((j1 - j0 + 1) * (k1 - k0 + 1))[part])
        own = part[own]
        w = (j1 - j0 + 1)[own]
        j, k = j0[own] + t % w, k0[own] + t // w
        dx = -fov / 2 + (j + 0.5) * d - x[own]
        dy = -fov / 2 + (k + 0.5) * d - y[own]
        angle = torch.sqrt(dx * dx + dy * dy)
        keep = (angle < T[own]).nonzero()[:, 0]
        pix, sel, angle = (j + npix * k)[keep], sel0[own[keep]], angle[keep]
        for o, v in zip(out, _profile(h, sel, angle, tabs, maps)):
            o.index_add_(0, pix, v)
    return out


def _exact_maps(case, seed):
    rec = torch.from_numpy(_records(case, seed)).to(DEV)
    tabs = [_full_table(1, nu, 0.0) for nu in _table_freqs(case)]
    h = _halos(case, rec)
    cone = torch.zeros_like(h["rec"])
    if case.get("cones"):
        off = torch.from_numpy(_offsets(case)).to(DEV)
        cone = torch.searchsorted(off, h["rec"], right=True) - 1
    out = _sky(case, h, tabs, cone)
    if case.get("npix_fs"):
        out = out + _flat(case, h, tabs)
    return out


def _exact_report(case, seed):
    maps = _exact_maps(case, seed)
    y = maps[0]
    m1 = float(y.mean())
    mom = [m1, float((y ** 2).mean()), float((y ** 3).mean())]
    rms = math.sqrt(float(((y - m1) ** 2).mean()))
    bins = (y / 1e-8).trunc().long()
    bins = bins[(y / 1e-8 > -1) & (bins < 10000)]
    count = torch.bincount(bins, minlength=10000).clamp(max=1 << 24)  # as a float counter stops
    dpdy = torch.cumsum(count.double() / y.numel(), 0)
    return maps + [np.array(mom + [rms]), dpdy]


def _exact_sphere(case, a, b):
    """Pixel-area quadrature: ring FFTs, the Legendre recursion in l for all m and rings."""
    nside, lmax = case["nside"], case["lmax"]
    rings = torch.arange(1, 4 * nside, device=DEV)
    z, s, npr, shift, first = (t.cpu() for t in _rings(nside, rings))
    m = np.arange(lmax + 1)
    F = np.empty((2, rings.numel(), lmax + 1), dtype=np.complex128)
    for i in range(rings.numel()):
        n, f = int(npr[i]), int(first[i])
        phase = np.exp(-1j * m * (2 * PI * float(shift[i]) / n))
        for q, x in enumerate((a, b)):
            F[q, i] = np.fft.fft(x[f:f + n].astype(np.float64))[m % n] * phase
    F = torch.from_numpy(F).to(DEV)
    north = F[:, : 2 * nside]
    south = torch.zeros_like(north)
    south[:, : 2 * nside - 1] = F[:, 2 * nside:].flip(1)
    sums = (north + south, north - south)  # l + m even, odd
    z, s = z[: 2 * nside, None].to(DEV), s[: 2 * nside, None].to(DEV)
    md = torch.arange(lmax + 1, dtype=torch.float64, device=DEV)[None, :]
    k = torch.arange(1, lmax + 1, dtype=torch.float64, device=DEV)
    start = torch.cat([torch.zeros(1, dtype=torch.float64, device=DEV),
                       torch.cumsum(0.5 * torch.log((2 * k + 1) / (2 * k)), 0)])[None, :]
    big = 460.0  # log of the scale unit
    logl = start - 0.5 * math.log(4 * PI) + md * torch.log(s)
    unit = torch.floor(logl / big)
    cur = torch.exp(logl - unit * big) * (1 - 2 * (md % 2))
    prev = torch.zeros_like(cur)
    cl = np.zeros((3, lmax + 1))
    alm_w = (4 * PI / (12 * nside * nside)) ** 2
    scale = torch.exp(unit.clamp(min=-1.5) * big) * (unit > -1.5)
    for l in range(lmax + 1):
        # column m = l starts; the others step from l - 1
        if l:
            f1, f0 = float(l) ** 2, float(l - 1) ** 2
            c = md[:, :l]
            ra = torch.sqrt((4 * f1 - 1) / (f1 - c * c))
            rb = torch.sqrt(((f0 - c * c) / (4 * f0 - 1)).clamp(min=0)) if l > 1 else 0.0 * c
            nx = (z * cur[:, :l] - rb * prev[:, :l]) * ra
            prev[:, :l] = cur[:, :l]
            cur[:, :l] = nx
            grown = (nx.abs() > math.exp(big / 2)) & (unit[:, :l] < 0)
            if l % 32 == 0 or bool(grown.any()):
                f = torch.exp(-big * grown.double())
                cur[:, :l] *= f
                prev[:, :l] *= f
                unit[:, :l] += grown
                scale[:, :l] = torch.exp(big * unit[:, :l].clamp(min=-1.5)) * (unit[:, :l] > -1.5)
        lam = cur[:, : l + 1] * scale[:, : l + 1]
        par = (l + torch.arange(l + 1, device=DEV)) % 2
        pick = torch.where(par[None, None, :] == 0, sums[0][..., : l + 1], sums[1][..., : l + 1])
        alm = (lam * pick).sum(1)
        w = torch.full((l + 1,), 2.0, dtype=torch.float64, device=DEV)
        w[0] = 1.0
        aa, bb = alm[0], alm[1]
        for q, v in enumerate((aa * aa.conj(), aa * bb.conj(), bb * bb.conj())):
            cl[q, l] = float((w * v.real).sum()) * alm_w / (2 * l + 1)
    return {"aa": cl[0], "ab": cl[1], "bb": cl[2]}


def _exact_flat(case, a, b):
    n, nbins, fov, top = case["npix"], case["nbins"], float(np.float32(math.radians(FOV_DEG))), 8000.0
    fa, fb = (torch.fft.fft2(torch.from_numpy(x).to(DEV).double().reshape(n, n)) for x in (a, b))
    k = torch.fft.fftfreq(n, 1.0 / n, device=DEV, dtype=torch.float64)
    ell = 2 * PI / fov * torch.sqrt(k[:, None] ** 2 + k[None, :] ** 2)
    edge = n // 2 - 1
    use = (ell > 0) & (ell <= top) & (k[:, None].abs() <= edge) & (k[None, :].abs() <= edge)
    ell = ell[use]
    bins = (ell / top * nbins).long().clamp(max=nbins - 1)
    count = torch.bincount(bins, minlength=nbins)
    mean = lambda v: torch.bincount(bins, v, nbins) / count.clamp(min=1)  # noqa: E731
    centre = (torch.arange(nbins, device=DEV, dtype=torch.float64) + 0.5) * top / nbins
    norm = fov ** 2 / float(n) ** 4
    out = {"ell": torch.where(count > 0, mean(ell), centre), "nmodes": count}
    for key, v in (("aa", fa.abs() ** 2), ("ab", (fa * fb.conj()).real), ("bb", fb.abs() ** 2)):
        out[key] = norm * mean(v[use])
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "paint":
        return _exact_maps(case, seed)
    if kind == "report":
        return _exact_report(case, seed)
    if kind == "table":
        return _full_table(case["model"], case["nu"], _alpha(seed), case["nchi"], case["nm"],
                           case["nr"]).reshape(-1)
    n = 12 * case["nside"] ** 2 if kind == "sphere" else case["npix"] ** 2
    a, b = _host_maps(n, seed)
    return _exact_sphere(case, a, b) if kind == "sphere" else _exact_flat(case, a, b)
