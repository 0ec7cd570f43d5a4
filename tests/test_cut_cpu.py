"""The cut's thresholds (p2m_cut_thresholds) against the float tests they stand for, on the
CPU: the radial and mass cuts at and around every bound, and the table's chi bound against
the two table look-ups."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "p2m_scalar.h"
static long bad = 0, seen = 0;
static void check(bool a, bool b) { seen++; bad += a != b; }
static float step(float x, int n) { return p2m_u2f(p2m_f2u(x) + (uint32_t)n); }
int main(int argc, char **argv) {
  const int shape = atoi(argv[1]);
  const float zlo = (float)atof(argv[2]), zhi = (float)atof(argv[3]), chimax = (float)atof(argv[4]);
  p2m_cosmo c;
  std::vector<float> r(P2M_NZTAB), z(P2M_NZTAB);
  p2m_cosmo_build(&c, r.data(), z.data());
  if (shape == 1) for (auto &v : r) v *= 0.5f;                       /* rises */
  if (shape == 2) for (int i = 4000; i < P2M_NZTAB; i++) r[i] = r[4000]; /* flat end */
  if (shape == 3) for (int i = 0; i < P2M_NZTAB; i++) r[i] += 50.0f * (float)((i / 500) % 2); /* up and down */
  const float lo = p2m_lookup(r.data(), c.drofz, zlo), hi = p2m_lookup(r.data(), c.drofz, zhi);
  const float mf = FMUL(FMUL(4.0f / 3.0f, c.mypi), c.rho_0);
  p2m_cut t;
  p2m_cut_thresholds(&t, lo, hi, mf, &c, r.data(), z.data(), chimax);
  if (!t.fast) { printf("not fast\n"); return 2; }
  auto shell = [&](float s) {
    const float chi = FSQRT(s);
    check(s <= t.s_high && s >= t.s_low, !(chi > hi || chi < lo));
  };
  auto mass = [&](float rth) {
    check(rth >= t.rth_min, !(FMUL(mf, FMUL(FMUL(rth, rth), rth)) < 1e13f));
  };
  auto keep = [&](float s0) {
    const float zz = p2m_lookup(z.data(), c.dzofr, FSQRT(s0));
    const bool want = !(p2m_lookup(r.data(), c.drofz, zz) > chimax);
    if (s0 <= t.s_keep) check(true, want);
    else if (s0 >= t.s_drop) check(false, want);
  };
  for (int n = -2000; n <= 2000; n++) {
    shell(step(t.s_high, n));
    if (t.s_low > 0.0f) shell(step(t.s_low, n));
    mass(step(t.rth_min, n));
    if (t.s_keep > 0.0f && t.s_keep < 1e30f) keep(step(t.s_keep, n));
    if (t.s_drop < 1e30f) keep(step(t.s_drop, n));
  }
  srand48(7);
  for (int n = 0; n < 100000; n++) {
    const float chi = (float)(drand48() * 15000.0), s = FMUL(chi, chi);
    shell(s);
    keep(s);
    mass((float)(drand48() * 10.0 - 1.0));
  }
  shell(0.0f); mass(0.0f); mass(-3.0f); keep(0.0f);
  const int lookups = t.s_keep < 0.0f;
  printf("%ld %ld %d\n", seen, bad, lookups);
  return bad != 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("cut")
    src = d / "cut.cpp"
    src.write_text(PROGRAM)
    exe = d / "cut"
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off",
                    "-I" + os.path.join(ROOT, "matt_young_mapmaking_gb300", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("shape,lookups", [(0, False), (1, False), (2, False), (3, True)])
@pytest.mark.parametrize("zlo,zhi,chimax", [(0.0, 6.0, 7000.0), (0.0, 1.25, 7000.0),
                                            (0.1, 0.1003, 300.0), (0.0, 4.0, 1e6)])
def test_cut_thresholds_reproduce_the_float_tests(program, shape, lookups, zlo, zhi, chimax):
    """Tables that rise, end flat, or go up and down (where every halo is looked up)."""
    r = subprocess.run([program, str(shape), str(zlo), str(zhi), str(chimax)],
                       stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0, r.stdout
    seen, bad, looked_up = (int(x) for x in r.stdout.split())
    assert seen > 200_000 and bad == 0
    if chimax == 7000.0:
        assert bool(looked_up) == lookups
