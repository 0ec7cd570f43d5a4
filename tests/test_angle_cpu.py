"""The painting kernels' float-float angle of a candidate (p2m_angle.h), compiled for the CPU,
against extended precision: a proven bound on every error, and no larger an error than the
same steps with every pair normalised and an IEEE root, over discs of every size and place."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include "p2m_angle.h"
typedef long double ld;
struct ff { float h, l; };
static float A(float a, float b) { return a + b; }
static float S(float a, float b) { return a - b; }
static ff norm(float s, float e) { float h = A(s, e); return {h, S(e, S(h, s))}; }
static ff two_sum(float a, float b) {
  float s = A(a, b), bb = S(s, a);
  return {s, A(S(a, S(s, bb)), S(b, bb))};
}
static ff add_f(ff x, float y) { ff s = two_sum(x.h, y); return norm(s.h, A(s.l, x.l)); }
static ff add(ff x, ff y) { ff s = two_sum(x.h, y.h); return norm(s.h, A(s.l, A(x.l, y.l))); }
static ff mul(ff x, ff y) {
  float p = x.h * y.h;
  return norm(p, fmaf(x.h, y.l, fmaf(x.l, y.h, fmaf(x.h, y.h, -p))));
}
/* the same steps, every pair normalised after every operation, the root IEEE */
static ff normalised(ff a, ff b, ff f0, ff d, int n) {
  const ff y = mul(add_f(two_sum((float)n, f0.h), f0.l), d);
  const ff s = add_f(y, p2m_sin_minus_arg(y.h, y.h * y.h));
  const ff c2 = add(a, mul(b, mul(s, s)));
  const float r = sqrtf(c2.h);
  const ff ch = norm(r, A(fmaf(-r, r, c2.h), c2.l) / (2.0f * r));
  const float u = 0.5f * ch.h;
  return add_f(ch, 2.0f * p2m_asin_minus_arg(u, u * u));
}
static ff pair(ld v) { const float h = (float)v; return {h, (float)(v - (ld)h)}; }
static ld value(ff x) { return (ld)x.h + (ld)x.l; }
static std::mt19937_64 rng;
static double uni() { return std::uniform_real_distribution<double>(0, 1)(rng); }

int main(int argc, char **argv) {
  const long want = atol(argv[1]);
  const double amax[5] = {1e-3, 5e-3, 0.02, 0.1, 0.52}, ymax[7] = {1e-3, 1e-2, 0.1, 0.5, 1.0, 1.5, 9};
  static double sq[2][5][7];
  static long count[5][7];
  double worst = 0;
  rng.seed(atol(argv[2]));
  for (long seen = 0; seen < want;) {
    /* a disc of one of five sizes anywhere, half of them near a pole; a ring and a pixel in it */
    const double T = amax[(int)(uni() * 5)];
    const int ns = 1 << (int)(uni() * 14);
    double th0 = uni() < 0.5 ? acos(1 - 2 * uni()) : T * pow(10, 2 - 3 * uni());
    if (th0 > M_PI) continue;
    if (uni() < 0.5) th0 = M_PI - th0;
    const double ang = uni() < 0.2 ? T * pow(10, -4 * uni()) : T * sqrt(uni()), psi = 2 * M_PI * uni();
    const double z = fmin(1, fmax(-1, cos(th0) * cos(ang) + sin(th0) * sin(ang) * cos(psi)));
    const double th = acos(z), cap = ns * sqrt(6.0);
    const long ring = lround(fabs(z) <= 2.0 / 3 ? 2 * ns - z * 1.5 * ns
                             : z > 0 ? cap * sin(th / 2) : 4 * ns - cap * sin((M_PI - th) / 2));
    if (ring < 1 || ring > 4 * ns - 1) continue;
    const long i = ring < 2 * ns ? ring : 4 * ns - ring, npr = 4 * (i < ns ? i : ns);
    const ld t = (ld)i * i / (3.0L * ns * ns);
    ld zr = i < ns ? 1 - t : (2.0L * ns - i) * 2 / (3.0L * ns);
    const ld sr = i < ns ? sqrtl(t * (2 - t)) : sqrtl(1 - zr * zr);
    if (ring > 2 * ns) zr = -zr;
    const ld z0 = cosl(th0), s0 = sinl(th0);
    const ld av = (zr - z0) * (zr - z0) + (sr - s0) * (sr - s0), bv = 4 * sr * s0;
    if (!(bv > 1e-25L)) continue;
    ld q = (4 * powl(sinl(ang / 2), 2) - av) / bv;
    if (!(q >= 0)) q = 1e-6 * uni();
    ld off = asinl(sqrtl(q < 1 ? q : 1));
    if (uni() < 0.5) off = -off;
    const ld dv = acosl(-1.0L) / npr, f = (ld)uni() - 0.5L;
    const long n = lroundl(off / dv - f);
    if (labs(n) > npr / 2 + 1) continue;
    const ff a = pair(av), b = pair(bv), f0 = pair(f), d = pair(dv);
    const ff y0 = mul(f0, d);
    const ld y = ((ld)n + value(f0)) * value(d), sy = sinl(y);
    const ld chord2 = value(a) + value(b) * sy * sy, truth = 2 * asinl(sqrtl(chord2) / 2);
    if (chord2 > 0.2499L || chord2 < 1e-23L) continue;
    /* the kernels' approximate reciprocal root, off by up to 2^-22.9 */
    float c2l, y2, hi, lo;
    const float c2 = p2m_chord_sq(a.h, a.l, b.h, b.l, y0.h, y0.l, d.h, d.l, (int)n, &c2l, &y2);
    const float rs = (float)((1 + (2 * uni() - 1) * exp2l(-22.9L)) / sqrtl(c2));
    const float u = p2m_chord_angle(c2, c2l, rs, &hi, &lo);
    if (u > 0.25f) continue;
    seen++;
    /* Units of e = 2^-24.  sin(y) - y: 6 e relative, at most y^3 / 6; the low word of y, at
       most 3 e y, scaled by 1 - y^2/2 for cos(y): y^4/24 of it; both against sin(y); the
       series' end 1e-8 y^17 / 2.37^17; asin(u) - u: 5 e relative, at most u^3/6 (1 + ...); the
       float-float operations together 60 e^2 */
    const ld e = exp2l(-24), ay = fabsl(y), uu = (ld)u * u;
    const ld bound = (e * ay * ay + 3 * e * powl(ay, 4) / 24 + 1e-8L * powl(ay / 2.37L, 16)) *
                         (ay > 0 ? ay / sinl(ay) : 1) + 1.05L * 5 * e * uu / 6 + 60 * e * e;
    const ld err[2] = {(ld)hi + (ld)lo - truth, value(normalised(a, b, f0, d, (int)n)) - truth};
    const double r = (double)(fabsl(err[0]) / truth / bound);
    if (r > worst) worst = r;
    int ia = 0, iy = 0;
    while (ia < 4 && truth > amax[ia]) ia++;
    while (iy < 6 && ay > ymax[iy]) iy++;
    count[ia][iy]++;
    for (int k = 0; k < 2; k++) sq[k][ia][iy] += (double)(err[k] / truth * (err[k] / truth));
  }
  printf("%.4f", worst);
  for (int ia = 0; ia < 5; ia++)
    for (int iy = 0; iy < 7; iy++)
      if (count[ia][iy] >= 20000) printf(" %.4f", sqrt(sq[0][ia][iy] / sq[1][ia][iy]));
  printf("\n");
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("angle")
    src = d / "angle.cpp"
    src.write_text(PROGRAM)
    exe = d / "angle"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                    "-I" + os.path.join(ROOT, "matt_young_mapmaking_gb300", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    return str(exe)


def test_angle_error_is_bounded_and_no_larger_than_normalised(program):
    """Every error within the bound of the program's comment.  By size and longitude offset, the
    rms relative error is at most 1.02 of the normalised form's (2 % is four standard errors of
    an rms over 20,000 candidates)."""
    out = subprocess.run([program, "1000000", "1"], stdout=subprocess.PIPE, text=True,
                         check=True).stdout.split()
    worst, ratios = float(out[0]), [float(x) for x in out[1:]]
    assert worst <= 1.0
    assert len(ratios) >= 10
    assert max(ratios) <= 1.02, ratios
