/*
 * p2m_spectra.cu -- angular power spectra of painted maps, for the precision report.
 * Validation only: nothing here is on the painting path.
 *
 * HEALPix maps (RING order): the pixel-area quadrature analysis of the HEALPix library
 * that the reference vendors, map2alm without iterations and with unit ring weights
 * (src/modules/External/alm_map_dd_inc.F90:2978-3224), followed by alm2cl (:5347-5423):
 *
 *   a_lm = (4 pi / npix) sum_rings lambda_lm(theta_r) F_r(m)
 *   F_r(m) = sum_j f_rj exp(-i m phi_rj)     (ring_analysis, alm_tools.F90:1022-1097)
 *   C_l = (Re a_l0 b_l0 + 2 sum_{m>=1} Re a_lm conj(b_lm)) / (2l + 1)
 *
 * lambda_lm is the normalised associated Legendre function.  It is computed by the
 * three-term recursion in l of HEALPix: gen_mfac (alm_tools.F90:500-522) and
 * compute_lam_mm (:559-580) start it, gen_recfac (:394-416) gives its coefficients,
 * and the loop of map2alm_sc_d runs it.  Powers of 2^100 are factored out as the
 * recursion runs, so that lambda_mm ~ sin^m(theta) neither underflows nor overflows;
 * a term whose scale is below 2^-1000 counts as zero (rescale_tab, :284-307).  Terms
 * below l_min_ylm (:882-903) are skipped as HEALPix skips them.  The ring geometry is
 * get_pixel_layout (:311-349).  The equatorial symmetry lambda_lm(pi - theta) =
 * (-1)^(l+m) lambda_lm(theta) pairs each northern ring with its southern mirror.
 *
 * GPU layout:
 *   rings     A ring's sums F_r(m) for all m are one FFT of its pixels.  Ring lengths are 4 n:
 *             each ring pair (north and mirror) is split into its four interleaved quarters
 *             of n pixels, for the sums S = north + south and the differences
 *             D = north - south, with both maps in one complex sequence (a + i b).
 *             k_quarter_fft transforms the quarters in shared memory: radix 4 when n is a
 *             power of two (all belt rings), Bluestein's chirp convolution otherwise
 *             (k_chirp prepares each cap ring's chirp transform), in two halves where its
 *             length is over QF_MAX_CONV.  k_ring_combine joins the quarters for every m, separates the
 *             maps and writes S and D of each map, laid out [m][ring] so that the next
 *             kernel reads one m's rings contiguously.
 *   k_alm     one block per m: rings over the threads, see there.
 *   k_alm2cl  32 values of l by 32 slices of m per block.
 * All arithmetic is FP64: the estimator is a diagnostic, where exactness matters more
 * than speed.
 *
 * Flat-sky maps: the periodogram of the npix x npix map over fov x fov radians, binned
 * linearly in ell = 2 pi |k| / fov.  It has no counterpart in the reference.
 *
 *   C(ell) = (fov^2 / npix^4) |FFT(map)(k)|^2, averaged over the modes of a bin
 *
 * k = 0 is left out, and so is the Nyquist line.  Both maps go through one complex FFT
 * (a + i b).  The rows are transformed by a radix-4 FFT in shared memory when npix is
 * a power of two up to 8192, or by a direct DFT for other npix up to 2048.  The columns
 * are transformed the same way after a transpose.
 */
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <vector>

#include "../../include/p2m.h"
#include "../../include/p2m_tools.h"
#include "p2m_internal.h"

#include <mutex>

namespace {
std::mutex g_pool_mutex;
struct ContextPool {
  unsigned long long context;
  cudaMemPool_t pool;
};
std::vector<ContextPool> g_pools;

/* the driver's id of the current context, which no other context of this process ever has */
cudaError_t context_id(unsigned long long *id) {
  struct Entry {
    void *fn = nullptr;
    Entry(const char *name, unsigned version) {
      cudaDriverEntryPointQueryResult found;
      if (cudaGetDriverEntryPointByVersion(name, &fn, version, cudaEnableDefault, &found) !=
              cudaSuccess ||
          found != cudaDriverEntryPointSuccess)
        fn = nullptr;
    }
  };
  static const Entry get_current("cuCtxGetCurrent", 4000), get_id("cuCtxGetId", 12000);
  if (!get_current.fn || !get_id.fn) return cudaErrorNotSupported;
  CUcontext ctx = nullptr;
  if (((CUresult (*)(CUcontext *))get_current.fn)(&ctx) != CUDA_SUCCESS || !ctx ||
      ((CUresult (*)(CUcontext, unsigned long long *))get_id.fn)(ctx, id) != CUDA_SUCCESS)
    return cudaErrorInvalidDevice;
  return cudaSuccess;
}
}  // namespace

/* A pool belongs to the context that it was made in: after a cudaDeviceReset the next call makes
   another (what is kept of the old one is its entry in the list). */
cudaError_t p2m_pool_alloc(void **out, size_t bytes, cudaStream_t s) {
  unsigned long long context = 0;
  cudaError_t e = context_id(&context);
  if (e != cudaSuccess) return e;
  cudaMemPool_t pool = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    for (const ContextPool &c : g_pools)
      if (c.context == context) pool = c.pool;
    if (!pool) {
      cudaMemPoolProps props = {};
      props.allocType = cudaMemAllocationTypePinned;
      props.location.type = cudaMemLocationTypeDevice;
      e = cudaGetDevice(&props.location.id);
      if (e != cudaSuccess) return e;
      cudaMemPool_t made;
      e = cudaMemPoolCreate(&made, &props);
      if (e != cudaSuccess) return e;
      unsigned long long keep = 256ull << 20;
      e = cudaMemPoolSetAttribute(made, cudaMemPoolAttrReleaseThreshold, &keep);
      if (e != cudaSuccess) {
        cudaMemPoolDestroy(made);
        return e;
      }
      g_pools.push_back({context, made});
      pool = made;
    }
  }
  return cudaMallocFromPoolAsync(out, bytes ? bytes : 1, pool, s);
}
void p2m_pool_free(void *p, cudaStream_t s) {
  if (p) cudaFreeAsync(p, s);
}

namespace {

#define FULL_MASK 0xffffffffu

constexpr int QF_THREADS = 256;
constexpr int QF_MAX_CONV = 8192; /* longest transform in shared memory (128 KB) */
constexpr int RC_THREADS = 256;
constexpr int ALM_THREADS = 256;
constexpr int ALM_RINGS = 8; /* rings per thread */
constexpr int ALM_GROUP = ALM_THREADS * ALM_RINGS;
constexpr int ALM_LC = 64; /* values of l between rescalings */
constexpr int ALM_LB = 8;  /* values of l summed before a warp reduces them together */
constexpr int ALM_WARPS = ALM_THREADS / 32;
constexpr int FFT_THREADS = 256;
constexpr int FFT_MAX_POW2 = 8192;
constexpr int DFT_MAX = 2048;

struct RingGeom {
  double cth, sth;
  int nph, shift; /* shift 1: pixel centres at phi = pi (2j + 1) / nph */
  long long start;
};

/* get_pixel_layout (alm_tools.F90:311-349) for northern ring ith = 1 .. 2 nside */
__device__ RingGeom ring_geom(int nside, int ith) {
  RingGeom g;
  const double n = (double)nside;
  if (ith < nside) {
    g.cth = 1.0 - ((double)ith * (double)ith) * (1.0 / (3.0 * n * n));
    g.sth = sin(2.0 * asin((double)ith * (1.0 / (sqrt(6.0) * n))));
    g.nph = 4 * ith;
    g.shift = 1;
    g.start = 2LL * ith * (ith - 1);
  } else {
    g.cth = (double)(2 * nside - ith) * (2.0 / (3.0 * n));
    g.sth = sqrt((1.0 - g.cth) * (1.0 + g.cth));
    g.nph = 4 * nside;
    g.shift = (ith + 1 - nside) & 1;
    g.start = 2LL * nside * (nside - 1) + (long long)(ith - nside) * g.nph;
  }
  return g;
}

/* the same without z and sin(theta) */
__device__ __forceinline__ RingGeom ring_geom_int(int nside, int ith) {
  RingGeom g;
  g.cth = g.sth = 0.0;
  const bool cap = ith < nside;
  g.nph = 4 * (cap ? ith : nside);
  g.shift = cap ? 1 : (ith + 1 - nside) & 1;
  g.start = cap ? 2LL * ith * (ith - 1)
                : 2LL * nside * (nside - 1) + (long long)(ith - nside) * g.nph;
  return g;
}

/* 2^(100 s) for |s| <= 10, zero below (the scales that underflow) */
__device__ __forceinline__ double scale_factor(int s) {
  return (s < -10 || s > 10) ? 0.0 : ldexp(1.0, 100 * s);
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
/* exp(-i pi a / n) for 0 <= a < 2 n */
__device__ __forceinline__ double2 expi(long long a, int n) {
  double s, c;
  sincospi((double)a / (double)n, &s, &c);
  return make_double2(c, -s);
}

/* length of the convolution that carries a DFT of length n (power of two >= 2 n - 1), or 0
   when n is a power of two itself */
__host__ __device__ __forceinline__ int conv_len(int n) {
  if ((n & (n - 1)) == 0) return 0;
  int l = 1;
  while (l < 2 * n - 1) l <<= 1;
  return l;
}

/* u + w v and u - w v in six FP64 operations: u - w v as 2 u - (u + w v) */
__device__ __forceinline__ void butterfly(double2 &u, double2 &v, double2 w) {
  const double ar = fma(-v.y, w.y, fma(v.x, w.x, u.x)), ai = fma(v.y, w.x, fma(v.x, w.y, u.y));
  v = make_double2(fma(2.0, u.x, -ar), fma(2.0, u.y, -ai));
  u = make_double2(ar, ai);
}
__device__ __forceinline__ void butterfly1(double2 &u, double2 &v) { /* w = 1 */
  const double2 a = make_double2(u.x + v.x, u.y + v.y);
  v = make_double2(u.x - v.x, u.y - v.y);
  u = a;
}

/* In-place FFT of the len complex values in shared memory (len a power of two) by the whole
   block, input in bit-reversed order.  tw[k] = exp(-2 pi i k / twlen), twlen >= len.  Two
   radix-2 stages per pass (after one alone where their number is odd): a thread takes four
   values through both in registers, half the passes over shared memory and half the
   barriers.  FP64 issue bounds it: 6 operations a butterfly, 4 in the first two stages,
   whose factors are 1 and -i. */
__device__ void block_fft(double2 *sz, int len, const double2 *__restrict__ tw, int twlen) {
  int half = 1;
  if ((31 - __clz(len)) & 1) {
    for (int b = threadIdx.x; b < len / 2; b += blockDim.x) butterfly1(sz[2 * b], sz[2 * b + 1]);
    half = 2;
    __syncthreads();
  }
  for (; half < len; half <<= 2) {
    /* stages half and 2 half: values i, i + half, i + 2 half, i + 3 half */
    const int s1 = twlen / (2 * half), s2 = s1 >> 1;
    for (int b = threadIdx.x; b < len / 4; b += blockDim.x) {
      const int pos = b & (half - 1);
      double2 *z = sz + (((b - pos) << 2) + pos);
      double2 a0 = z[0], a1 = z[half], a2 = z[2 * half], a3 = z[3 * half];
      if (half == 1) {
        butterfly1(a0, a1);
        butterfly1(a2, a3);
        butterfly1(a0, a2);
        const double2 r = make_double2(a3.y, -a3.x); /* -i a3 */
        a3 = r;
        butterfly1(a1, a3);
      } else {
        const double2 w1 = tw[pos * s1], w2 = tw[pos * s2];
        butterfly(a0, a1, w1);
        butterfly(a2, a3, w1);
        butterfly(a0, a2, w2);
        butterfly(a1, a3, make_double2(w2.y, -w2.x)); /* -i w2 */
      }
      z[0] = a0;
      z[half] = a1;
      z[2 * half] = a2;
      z[3 * half] = a3;
    }
    __syncthreads();
  }
}
__device__ __forceinline__ int bitrev(int j, int log2len) {
  return log2len ? (int)(__brev((unsigned)j) >> (32 - log2len)) : 0;
}

/* A convolution longer than QF_MAX_CONV (16384, for n > 4096) goes as two transforms of half
   its length: the even outputs of a transform of x are those of x_lo + x_hi, the odd ones
   those of (x_lo - x_hi) w^j, w = exp(-2 pi i / conv); and of the inverse transform the first
   half is the even inputs' plus w^-j times the odd inputs'. */
__host__ __device__ __forceinline__ int conv_halves(int conv) { return conv > QF_MAX_CONV ? 2 : 1; }

/* Bluestein's chirp of cap ring n = blockIdx.x + 1: the transform of the circular sequence
   exp(+i pi j^2 / n), |j| < n, at chirp + off[n] (even outputs, then odd ones, where it is
   made in halves); rings whose n is a power of two have none (off < 0) */
__global__ void __launch_bounds__(QF_THREADS)
    k_chirp(const long long *__restrict__ off, const double2 *__restrict__ tw, int twlen,
            double2 *__restrict__ chirp) {
  extern __shared__ double2 sz[];
  const int n = blockIdx.x + 1;
  if (off[n] < 0) return;
  const int conv = conv_len(n), halves = conv_halves(conv), len = conv / halves;
  const int lg = 31 - __clz(len);
  auto value = [&](int j) {
    const int a = j < n ? j : conv - j; /* circular distance from 0 */
    double2 v = make_double2(0.0, 0.0);
    if (a < n) {
      v = expi(((long long)a * a) % (2 * n), n);
      v.y = -v.y;
    }
    return v;
  };
  for (int h = 0; h < halves; h++) {
    for (int j = threadIdx.x; j < len; j += blockDim.x) {
      double2 v = value(j);
      if (halves == 2) {
        const double2 u = value(j + len);
        v = h ? cmul(make_double2(v.x - u.x, v.y - u.y), tw[j * (twlen / conv)])
              : make_double2(v.x + u.x, v.y + u.y);
      }
      sz[bitrev(j, lg)] = v;
    }
    __syncthreads();
    block_fft(sz, len, tw, twlen);
    for (int j = threadIdx.x; j < len; j += blockDim.x) chirp[off[n] + h * len + j] = sz[j];
    __syncthreads();
  }
}

/* Transform of one quarter: blockIdx.y = 2 q + type (type 0: S, 1: D), northern ring
   blockIdx.x + 1 with its mirror, pixels 4 j + q, j < n:
   G(k) = sum_j z_j exp(-2 pi i j k / n) at g + 8 start + (2 q + type) n, where start is the
   first quarter-pixel of the ring (sum of the n of the rings before).  Latency of the
   log2(n) passes and of the pixel loads bounds it: 8 blocks per ring keep every SM busy.  The
   FP64 work is 5 n log2(n) against the 8 n (lmax + 1) of summing every m by itself.  Two maps
   at Nside 512, lmax 1535: 0.84 ms, with k_chirp 0.08 and k_ring_combine 0.44, against 48.8 ms. */
__global__ void __launch_bounds__(QF_THREADS)
    k_quarter_fft(const float *__restrict__ ma, const float *__restrict__ mb, int nside,
                  const long long *__restrict__ off, const double2 *__restrict__ chirp,
                  const double2 *__restrict__ tw, int twlen, double2 *__restrict__ g) {
  extern __shared__ double2 sz[];
  const int ith = blockIdx.x + 1, q = blockIdx.y >> 1;
  const double sgn = (blockIdx.y & 1) ? -1.0 : 1.0;
  const RingGeom rg = ring_geom_int(nside, ith);
  const int n = rg.nph >> 2;
  const long long npix = 12LL * nside * nside;
  const long long sn = rg.start + q, ss = npix - rg.start - rg.nph + q;
  const bool south = ith < 2 * nside; /* the equator has no mirror */
  double2 *out = g + (rg.start >> 2) * 8 + (long long)blockIdx.y * n;
  auto pixel = [&](int j) {
    double2 z = make_double2((double)ma[sn + 4 * j], mb ? (double)mb[sn + 4 * j] : 0.0);
    if (south) {
      z.x = fma(sgn, (double)ma[ss + 4 * j], z.x);
      if (mb) z.y = fma(sgn, (double)mb[ss + 4 * j], z.y);
    }
    return z;
  };
  const int conv = conv_len(n);
  if (conv == 0) {
    const int lg = 31 - __clz(n);
    for (int j = threadIdx.x; j < n; j += blockDim.x) sz[bitrev(j, lg)] = pixel(j);
    __syncthreads();
    block_fft(sz, n, tw, twlen);
    for (int j = threadIdx.x; j < n; j += blockDim.x) out[j] = sz[j];
    return;
  }
  /* DFT(k) = c_k sum_j (z_j c_j) conj(c_{k-j}), c_j = exp(-i pi j^2 / n): a circular
     convolution; its inverse transform as the conjugate of a forward one */
  const int halves = conv_halves(conv), len = conv / halves, lg = 31 - __clz(len);
  const double inv = 1.0 / (double)conv;
  for (int h = 0; h < halves; h++) {
    for (int j = threadIdx.x; j < len; j += blockDim.x) {
      double2 v = make_double2(0.0, 0.0);
      if (j < n) v = cmul(pixel(j), expi(((long long)j * j) % (2 * n), n));
      if (h) v = cmul(v, tw[j * (twlen / conv)]);
      sz[bitrev(j, lg)] = v;
    }
    __syncthreads();
    block_fft(sz, len, tw, twlen);
    const double2 *ch = chirp + off[n] + h * len;
    /* product, conjugated, into bit-reversed order (pairs swapped in place) */
    for (int j = threadIdx.x; j < len; j += blockDim.x) {
      const int r = bitrev(j, lg);
      if (r < j) continue;
      double2 a = cmul(sz[j], ch[j]);
      a.y = -a.y;
      if (r != j) {
        double2 b = cmul(sz[r], ch[r]);
        b.y = -b.y;
        sz[j] = b;
      }
      sz[r] = a;
    }
    __syncthreads();
    block_fft(sz, len, tw, twlen);
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
      double2 v = make_double2(sz[j].x * inv, -sz[j].y * inv);
      if (h) {
        const double2 w = tw[j * (twlen / conv)];
        v = cmul(v, make_double2(w.x, -w.y));
      }
      v = cmul(v, expi(((long long)j * j) % (2 * n), n));
      out[j] = h ? make_double2(out[j].x + v.x, out[j].y + v.y) : v;
    }
    __syncthreads();
  }
}

/* F_r(m), m = blockIdx.y * RC_THREADS + thread, of northern ring blockIdx.x + 1 with its mirror:
   Z(k) = sum_q w^(k q) G_q(k mod n) with w = exp(-2 pi i / 4n), k = m mod 4n, times the ring's
   half-pixel phase; the maps a and b of z = a + i b come apart as (Z(k) +- conj Z(-k)) / 2.
   ph[m][ring] = S and D of map a, then of map b. */
__global__ void __launch_bounds__(RC_THREADS)
    k_ring_combine(const double2 *__restrict__ g, int nside, int lmax, double *__restrict__ ph) {
  const int ith = blockIdx.x + 1, m = blockIdx.y * RC_THREADS + threadIdx.x;
  if (m > lmax) return;
  const RingGeom rg = ring_geom_int(nside, ith);
  const int nph = rg.nph, n = nph >> 2;
  const double2 half = expi(m % (2 * nph), nph); /* exp(-i pi m / nph) */
  const double2 w1 = cmul(half, half), w2 = cmul(w1, w1), w3 = cmul(w2, w1);
  const int kp = m % n, km = kp ? n - kp : 0;
  const double2 *src = g + (rg.start >> 2) * 8;
  double o[8];
#pragma unroll
  for (int type = 0; type < 2; type++) {
    double2 zp = src[type * n + kp], zm = src[type * n + km];
#pragma unroll
    for (int q = 1; q < 4; q++) {
      const double2 w = q == 1 ? w1 : q == 2 ? w2 : w3;
      const double2 a = cmul(src[(2 * q + type) * n + kp], w);
      const double2 b = cmul(src[(2 * q + type) * n + km], make_double2(w.x, -w.y));
      zp.x += a.x;
      zp.y += a.y;
      zm.x += b.x;
      zm.y += b.y;
    }
    double2 fa = make_double2(0.5 * (zp.x + zm.x), 0.5 * (zp.y - zm.y));
    double2 fb = make_double2(0.5 * (zp.y + zm.y), 0.5 * (zm.x - zp.x));
    if (rg.shift) {
      fa = cmul(fa, half);
      fb = cmul(fb, half);
    }
    o[2 * type] = fa.x;
    o[2 * type + 1] = fa.y;
    o[4 + 2 * type] = fb.x;
    o[4 + 2 * type + 1] = fb.y;
  }
  double2 *dst = (double2 *)(ph + ((size_t)m * (2 * nside) + (ith - 1)) * 8);
#pragma unroll
  for (int c = 0; c < 4; c++) dst[c] = make_double2(o[2 * c], o[2 * c + 1]);
}

/* row offset of m in the packed a_lm array (l = m .. lmax) */
__host__ __device__ __forceinline__ size_t alm_row(int m, int lmax) {
  return (size_t)m * (size_t)(lmax + 1) - (size_t)m * (size_t)(m - 1) / 2;
}

/* sums of v[32] over the warp's lanes: lane i returns the sum of the lanes' v[i].  Each step
   halves the values a lane holds, so 32 values take 31 additions, not 160. */
__device__ __forceinline__ double warp_sum32(double (&v)[32]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < o; i++) {
      const double mine = up ? v[i + o] : v[i], other = up ? v[i] : v[i + o];
      v[i] = mine + __shfl_xor_sync(FULL_MASK, other, o);
    }
  }
  return v[0];
}

/* a_lm / omega_pix of both maps for m = blockIdx.x, in alm[(row + l - m) * 4 + c],
   c = (Re a, Im a, Re b, Im b), which starts at zero.
   TWO: there is a map b (its c stay zero otherwise).

   FP64 issue bounds it (2 operations per clock and SM).  The recursion is carried without the
   normalising factors: lambda_l = C_l q_l with q_{l+1} = cos(theta) q_l - beta_l q_{l-1},
   beta_l = (l^2 - m^2) / (4 l^2 - 1) and C_l the product of rf(j) = 1 / sqrt(beta_{j+1}),
   j < l, which is applied once per l to the sum over the rings.  A ring's scale (the powers of
   2^100 and lambda_mm) is applied to its phases, and q is looked over for rescaling, every 64
   values of l, over which it changes by less than 2^310.  So a ring and l cost 2 operations of
   recursion and 2 per map for the sums.  Rings that l_min_ylm leaves out for every l are
   skipped a warp at a time, and the sums of 64 values of l below it too.  Nside 512, lmax
   1535, two maps: 14.3 ms (6 operations for each of 1.2e9 rings and l are 11.9 ms), against
   48.8 ms with every factor and test at every l. */
template <bool TWO>
__global__ void __launch_bounds__(ALM_THREADS)
    k_alm(const double *__restrict__ ph, const double *__restrict__ mfac, int nside, int lmax,
          int group, double *__restrict__ alm) {
  extern __shared__ double smem[];
  constexpr int NC = TWO ? 4 : 2;     /* sums per l */
  double *sph = smem;                 /* [component 8][group] phases, times the ring's scale */
  double *beta = sph + group * 8;     /* beta_l, l = l0 .. l0 + LC - 1 */
  double *cl = beta + ALM_LC;         /* C_l / C_l0 */
  double *red = cl + ALM_LC;          /* [warp][LC][4] */
  const int m = blockIdx.x;
  const int nrings = 2 * nside;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const double dm2 = (double)m * (double)m;
  const size_t row = alm_row(m, lmax);
  const double mf = mfac[m];
  for (int g0 = 0; g0 < nrings; g0 += group) {
    const int ng = min(group, nrings - g0);
    const int nk = (ng + ALM_THREADS - 1) / ALM_THREADS;
    double cth[ALM_RINGS], qp[ALM_RINGS], qc[ALM_RINGS], lmm[ALM_RINGS];
    int sc[ALM_RINGS], lmin[ALM_RINGS];
    unsigned alive = 0; /* bit k: some ring of this warp's k-th 32 is used */
#pragma unroll
    for (int k = 0; k < ALM_RINGS; k++) {
      const int r = k * ALM_THREADS + t;
      cth[k] = qp[k] = qc[k] = lmm[k] = 0.0;
      sc[k] = 0;
      lmin[k] = INT_MAX;
      if (r < ng) {
        const RingGeom gg = ring_geom(nside, g0 + r + 1);
        /* l_min_ylm: int((m - 40) / (1.35 sin theta)), at least m */
        const double v = (double)(m - 40) / (1.35 * gg.sth);
        const int lm = v > (double)lmax ? lmax + 1 : max(m, (int)v);
        if (lm <= lmax) {
          const double log2val = mf + (double)m * log(gg.sth) * (1.0 / log(2.0));
          const int s = (int)(log2val / 100.0);
          double lam_mm = exp2(log2val - 100.0 * (double)s);
          if (m & 1) lam_mm = -lam_mm;
          cth[k] = gg.cth;
          qc[k] = 1.0; /* lambda_m / (lambda_mm scale) */
          lmm[k] = lam_mm;
          sc[k] = s;
          lmin[k] = lm;
        }
      }
      if (__any_sync(FULL_MASK, lmin[k] <= lmax)) alive |= 1u << k;
    }
    if (!__syncthreads_or(alive != 0)) continue;
    double c_run = 1.0; /* C_l0, its power of two moved into q */
    bool first = true;
    for (int l0 = m; l0 <= lmax; l0 += ALM_LC) {
      const int nl = min(ALM_LC, lmax - l0 + 1);
      /* beta_l, and the factors 1 / sqrt(beta_{l+1}) of C */
      if (t < ALM_LC) {
        const int l = l0 + t;
        const double f0 = (double)l * (double)l, f1 = (double)(l + 1) * (double)(l + 1);
        beta[t] = l > m ? (f0 - dm2) / (4.0 * f0 - 1.0) : 0.0;
        double p = sqrt((4.0 * f1 - 1.0) / (f1 - dm2)); /* rf(l): C_{l+1} / C_l */
        /* inclusive product over the 32 lanes, then the second warp takes the first's */
        for (int o = 1; o < 32; o <<= 1) {
          const double y = __shfl_up_sync(FULL_MASK, p, o);
          if (lane >= o) p *= y;
        }
        cl[t] = p;
      }
      /* the rings' scales and rescaling */
      int lcut = INT_MAX; /* smallest l_min of this lane's rings */
#pragma unroll
      for (int k = 0; k < ALM_RINGS; k++) {
        if (k >= nk || !((alive >> k) & 1u)) continue;
        double a = fmax(fabs(qc[k]), fabs(qp[k]));
        bool moved = first;
        while (a > 0x1p100) {
          qp[k] *= 0x1p-100;
          qc[k] *= 0x1p-100;
          a *= 0x1p-100;
          sc[k] += 1;
          moved = true;
        }
        while (a < 0x1p-100 && a != 0.0) {
          qp[k] *= 0x1p100;
          qc[k] *= 0x1p100;
          a *= 0x1p100;
          sc[k] -= 1;
          moved = true;
        }
        lcut = min(lcut, lmin[k]);
        const int r = k * ALM_THREADS + t;
        if (r < ng && moved) {
          const double cm = scale_factor(sc[k]) * lmm[k];
          const double2 *src = (const double2 *)(ph + ((size_t)m * nrings + g0 + r) * 8);
#pragma unroll
          for (int c = 0; c < (TWO ? 4 : 2); c++) {
            const double2 f = cm != 0.0 ? src[c] : make_double2(0.0, 0.0);
            sph[(2 * c) * group + r] = f.x * cm;
            sph[(2 * c + 1) * group + r] = f.y * cm;
          }
        }
      }
      first = false;
      const bool sums = __any_sync(FULL_MASK, lcut < l0 + nl);
      __syncthreads();
      if (t >= 32 && t < ALM_LC) cl[t] *= cl[31];
      __syncthreads();
      for (int i0 = 0; i0 < nl; i0 += ALM_LB) {
        double acc[32];
#pragma unroll
        for (int i = 0; i < 32; i++) acc[i] = 0.0;
        const int par = (l0 + i0 + m) & 1; /* S for even l + m, D for odd */
        double b[ALM_LB];
#pragma unroll
        for (int i = 0; i < ALM_LB; i++) b[i] = beta[i0 + i];
#pragma unroll
        for (int k = 0; k < ALM_RINGS; k++) {
          if (k >= nk || !((alive >> k) & 1u)) continue;
          const int r = k * ALM_THREADS + t;
          double f[2][NC];
          if (sums) {
#pragma unroll
            for (int c = 0; c < NC; c++) {
              const int comp = (c >> 1) * 4 + (c & 1);
              f[0][c] = r < ng ? sph[(comp + 2 * par) * group + r] : 0.0;
              f[1][c] = r < ng ? sph[(comp + 2 - 2 * par) * group + r] : 0.0;
            }
          }
          double x0 = qp[k], x1 = qc[k];
#pragma unroll
          for (int i = 0; i < ALM_LB; i++) {
            if (sums) {
#pragma unroll
              for (int c = 0; c < NC; c++) acc[i * 4 + c] = fma(x1, f[i & 1][c], acc[i * 4 + c]);
            }
            /* q_{l+1}; past the last l of the chunk its values are not used */
            const double nx = fma(cth[k], x1, -b[i] * x0);
            x0 = x1;
            x1 = nx;
          }
          qp[k] = x0;
          qc[k] = x1;
        }
        const double s = sums ? warp_sum32(acc) : 0.0;
        red[(w * ALM_LC + i0) * 4 + lane] = s;
      }
      __syncthreads();
      if (t < nl * 4) {
        const int i = t >> 2, c = t & 3;
        double s = 0.0;
        for (int ww = 0; ww < ALM_WARPS; ww++) s += red[((size_t)ww * ALM_LC + i) * 4 + c];
        s *= i ? c_run * cl[i - 1] : c_run;
        alm[(row + (size_t)(l0 + i - m)) * 4 + c] += s;
      }
      /* C of the next chunk, its power of two moved into q */
      int e = 0;
      c_run = frexp(c_run * cl[ALM_LC - 1], &e);
      const double up = ldexp(1.0, e);
#pragma unroll
      for (int k = 0; k < ALM_RINGS; k++) {
        qp[k] *= up;
        qc[k] *= up;
      }
      __syncthreads();
    }
  }
}

/* alm2cl: cl[0] a x a, cl[1] a x b, cl[2] b x b, each [lmax + 1].  32 values of l (one per
   lane: their a_lm are contiguous) by 32 slices of m, summed in a fixed order */
__global__ void __launch_bounds__(1024)
    k_alm2cl(const double *__restrict__ alm, int lmax, double omega2, double *__restrict__ cl) {
  __shared__ double part[3][32][33];
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
  const int l = blockIdx.x * 32 + lane;
  double aa = 0.0, ab = 0.0, bb = 0.0;
  if (l <= lmax)
    for (int m = 1 + slice; m <= l; m += 32) {
      const double2 *a = (const double2 *)(alm + (alm_row(m, lmax) + (size_t)(l - m)) * 4);
      const double2 x = a[0], y = a[1];
      aa += x.x * x.x + x.y * x.y;
      ab += x.x * y.x + x.y * y.y;
      bb += y.x * y.x + y.y * y.y;
    }
  part[0][slice][lane] = aa;
  part[1][slice][lane] = ab;
  part[2][slice][lane] = bb;
  __syncthreads();
  if (slice >= 3 || l > lmax) return;
  double s = 0.0;
  for (int i = 0; i < 32; i++) s += part[slice][i][lane];
  const double *a0 = alm + (size_t)l * 4; /* m = 0 */
  const double z = slice == 0   ? a0[0] * a0[0] - a0[1] * a0[1]
                   : slice == 1 ? a0[0] * a0[2] - a0[1] * a0[3]
                                : a0[2] * a0[2] - a0[3] * a0[3];
  cl[(size_t)slice * (lmax + 1) + l] = (2.0 * s + z) * (omega2 / (2.0 * (double)l + 1.0));
}

/* ------------------------------------------------------------------ flat sky ---- */

__global__ void k_fs_pack(const float *__restrict__ a, const float *__restrict__ b, long long n,
                          double2 *__restrict__ z) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    z[i] = make_double2((double)a[i], b ? (double)b[i] : 0.0);
}

/* tw[k] = exp(-2 pi i k / n), k < n / 2 */
__global__ void k_twiddles(double2 *tw, int n) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n / 2) return;
  double s, c;
  sincospi(2.0 * (double)k / (double)n, &s, &c);
  tw[k] = make_double2(c, -s);
}

/* in-place FFT of each row (n a power of two, n >= 4), one block per row; FIRST: the rows are
   made from the maps (a + i b) */
template <int FIRST>
__global__ void __launch_bounds__(FFT_THREADS)
    k_fft_rows(double2 *__restrict__ z, const float *__restrict__ a, const float *__restrict__ b,
               int n, int logn, const double2 *__restrict__ tw) {
  extern __shared__ double2 sz[];
  const size_t at = (size_t)blockIdx.x * n;
  for (int j = threadIdx.x; j < n; j += FFT_THREADS)
    sz[bitrev(j, logn)] = FIRST ? make_double2((double)a[at + j], b ? (double)b[at + j] : 0.0) : z[at + j];
  __syncthreads();
  block_fft(sz, n, tw, n);
  for (int j = threadIdx.x; j < n; j += FFT_THREADS) z[at + j] = sz[j];
}

/* direct DFT of each row into out (any n <= DFT_MAX), one block per row */
__global__ void __launch_bounds__(256)
    k_dft_rows(const double2 *__restrict__ z, double2 *__restrict__ out, int n) {
  extern __shared__ double2 sr[];
  const double2 *row = z + (size_t)blockIdx.x * n;
  for (int j = threadIdx.x; j < n; j += blockDim.x) sr[j] = row[j];
  __syncthreads();
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    double s, c;
    sincospi(2.0 * (double)k / (double)n, &s, &c);
    const double step_r = c, step_i = -s;
    double accr = 0.0, acci = 0.0, wr = 1.0, wi = 0.0;
    for (int j = 0; j < n; j++) {
      if ((j & 63) == 0) { /* exact twiddle every 64 terms */
        sincospi(2.0 * (double)(((long long)k * j) % n) / (double)n, &s, &c);
        wr = c;
        wi = -s;
      }
      const double2 x = sr[j];
      accr += x.x * wr - x.y * wi;
      acci += x.x * wi + x.y * wr;
      const double nr = wr * step_r - wi * step_i;
      wi = wr * step_i + wi * step_r;
      wr = nr;
    }
    out[(size_t)blockIdx.x * n + k] = make_double2(accr, acci);
  }
}

__global__ void k_transpose(const double2 *__restrict__ in, double2 *__restrict__ out, int n) {
  __shared__ double2 tile[32][33];
  const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
  for (int dy = threadIdx.y; dy < 32; dy += blockDim.y) {
    const int x = x0 + threadIdx.x, y = y0 + dy;
    if (x < n && y < n) tile[dy][threadIdx.x] = in[(size_t)y * n + x];
  }
  __syncthreads();
  for (int dy = threadIdx.y; dy < 32; dy += blockDim.y) {
    const int x = y0 + threadIdx.x, y = x0 + dy;
    if (x < n && y < n) out[(size_t)y * n + x] = tile[threadIdx.x][dy];
  }
}

/* Per bin: modes, sum ell, |F_a|^2, Re F_a conj F_b, |F_b|^2 over |k1|, |k2| <= kmax.  The maps
   are real, so k and -k contribute alike: only k1 > 0, or k1 = 0 with k2 > 0, is visited and
   counted twice.  A thread takes a run of consecutive k2 and adds to the block's bins in shared
   memory when its bin changes. */
#define FS_RUN 4
__global__ void __launch_bounds__(256)
    k_fs_bins(const double2 *__restrict__ z, int n, double ell_fund, double ell_max, int nbins,
              int kmax, double *__restrict__ acc) {
  extern __shared__ double sb[];
  for (int i = threadIdx.x; i < nbins * 5; i += blockDim.x) sb[i] = 0.0;
  __syncthreads();
  const int side = 2 * kmax + 1, runs = (side + FS_RUN - 1) / FS_RUN;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < (kmax + 1) * runs;
       idx += gridDim.x * blockDim.x) {
    const int k1 = idx / runs, first = (idx - k1 * runs) * FS_RUN - kmax;
    const int last = min(first + FS_RUN - 1, kmax);
    const int i1 = k1, j1 = k1 ? n - k1 : 0;
    int bin = -1;
    double s[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (int k2 = k1 ? first : max(first, 1); k2 <= last; k2++) {
      const double ell = ell_fund * sqrt((double)k1 * k1 + (double)k2 * k2);
      if (ell > ell_max) continue;
      const int b = min((int)(ell / ell_max * nbins), nbins - 1);
      if (b != bin && bin >= 0) {
        for (int c = 0; c < 5; c++) {
          atomicAdd(&sb[bin * 5 + c], 2.0 * s[c]);
          s[c] = 0.0;
        }
      }
      bin = b;
      const int i2 = k2 < 0 ? k2 + n : k2, j2 = k2 > 0 ? n - k2 : -k2;
      const double2 zk = z[(size_t)i1 * n + i2], zm = z[(size_t)j1 * n + j2];
      /* F_a = (Z(k) + conj Z(-k)) / 2, F_b = (Z(k) - conj Z(-k)) / 2i */
      const double far = 0.5 * (zk.x + zm.x), fai = 0.5 * (zk.y - zm.y);
      const double fbr = 0.5 * (zk.y + zm.y), fbi = -0.5 * (zk.x - zm.x);
      s[0] += 1.0;
      s[1] += ell;
      s[2] += far * far + fai * fai;
      s[3] += far * fbr + fai * fbi;
      s[4] += fbr * fbr + fbi * fbi;
    }
    if (bin >= 0)
      for (int c = 0; c < 5; c++) atomicAdd(&sb[bin * 5 + c], 2.0 * s[c]);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nbins * 5; i += blockDim.x)
    if (sb[i] != 0.0) atomicAdd(&acc[i], sb[i]);
}

/* device buffers of one call, used on its stream only and released on every return path */
struct DevBufs {
  cudaStream_t s;
  std::vector<void *> p;
  explicit DevBufs(cudaStream_t stream) : s(stream) {}
  ~DevBufs() {
    for (void *q : p) p2m_pool_free(q, s);
  }
  template <class T>
  cudaError_t get(T **out, size_t bytes) {
    void *q = nullptr;
    cudaError_t e = p2m_pool_alloc(&q, bytes, s);
    if (e == cudaSuccess) p.push_back(q);
    *out = (T *)q;
    return e;
  }
};

struct DeviceScope {
  int prev = -1;
  bool ok = false;
  explicit DeviceScope(int dev) {
    if (cudaGetDevice(&prev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess) ok = true;
  }
  ~DeviceScope() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

struct Stream {
  cudaStream_t s = nullptr;
  Stream() { cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking); }
  ~Stream() {
    if (s) cudaStreamDestroy(s);
  }
};

#define SP_CK(x)                                                   \
  do {                                                             \
    cudaError_t e_ = (x);                                          \
    if (e_ != cudaSuccess) {                                       \
      cudaGetLastError();                                          \
      return e_ == cudaErrorMemoryAllocation ? P2M_ERR_NOMEM : P2M_ERR_CUDA; \
    }                                                              \
  } while (0)

/* allows a kernel the most dynamic shared memory that any call asks of it.  The limit belongs to
   the kernel, not to the launch: set to what one call needs, it could be lowered by another
   thread's smaller call before the launch, which would then be refused. */
template <class K>
cudaError_t allow_smem(K kernel, size_t most) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}
constexpr size_t QF_SMEM = sizeof(double2) * QF_MAX_CONV;
constexpr size_t FFT_SMEM = sizeof(double2) * FFT_MAX_POW2;
constexpr size_t alm_smem(int group) {
  return sizeof(double) * ((size_t)group * 8 + 2 * ALM_LC + (size_t)ALM_WARPS * ALM_LC * 4);
}

bool is_pow2(int n) { return n > 0 && (n & (n - 1)) == 0; }
int ilog2(int n) {
  int l = 0;
  while ((1 << l) < n) l++;
  return l;
}

}  // namespace

extern "C" {

int32_t p2m_cl_healpix(int32_t device, const float *map_a, const float *map_b, int32_t nside,
                       int32_t lmax, double *cl_aa, double *cl_ab, double *cl_bb) {
  if (!map_a || !cl_aa || !is_pow2(nside) || nside > 8192 || lmax < 0 ||
      lmax > 4 * nside || lmax > P2M_CL_LMAX_MAX)
    return P2M_ERR_BADARG;
  if (map_b && (!cl_ab || !cl_bb)) return P2M_ERR_BADARG;
  DeviceScope scope(device);
  if (!scope.ok) return P2M_ERR_CUDA;
  Stream st;
  if (!st.s) return P2M_ERR_CUDA;
  DevBufs B(st.s);
  const long long npix = 12LL * nside * nside;
  const int nrings = 2 * nside;
  const size_t nalm = alm_row(lmax + 1, lmax); /* (lmax + 1)(lmax + 2) / 2 */
  float *d_a = nullptr, *d_b = nullptr;
  double *d_ph = nullptr, *d_alm = nullptr, *d_mfac = nullptr, *d_cl = nullptr;
  SP_CK(B.get(&d_a, sizeof(float) * (size_t)npix));
  if (map_b) SP_CK(B.get(&d_b, sizeof(float) * (size_t)npix));
  SP_CK(B.get(&d_ph, sizeof(double) * 8 * (size_t)nrings * (size_t)(lmax + 1)));
  SP_CK(B.get(&d_alm, sizeof(double) * 4 * nalm));
  SP_CK(B.get(&d_mfac, sizeof(double) * (size_t)(lmax + 1)));
  SP_CK(B.get(&d_cl, sizeof(double) * 3 * (size_t)(lmax + 1)));
  /* gen_mfac: log2(prod_{k<=m} sqrt((2k+1)/(2k)) / sqrt(4 pi)) */
  std::vector<double> mfac((size_t)lmax + 1);
  {
    double f = 1.0;
    const double sq4pi_inv = 1.0 / std::sqrt(4.0 * M_PI), aln2_inv = 1.0 / std::log(2.0);
    for (int m = 0; m <= lmax; m++) {
      if (m > 0) f *= std::sqrt((double)(2 * m + 1) / (double)(2 * m));
      mfac[(size_t)m] = std::log(sq4pi_inv * f) * aln2_inv;
    }
  }
  SP_CK(cudaMemcpyAsync(d_a, map_a, sizeof(float) * (size_t)npix, cudaMemcpyHostToDevice, st.s));
  if (map_b)
    SP_CK(cudaMemcpyAsync(d_b, map_b, sizeof(float) * (size_t)npix, cudaMemcpyHostToDevice, st.s));
  SP_CK(cudaMemcpyAsync(d_mfac, mfac.data(), sizeof(double) * mfac.size(), cudaMemcpyHostToDevice,
                        st.s));
  /* the cap rings' chirps: offsets by n = 1 .. nside - 1, -1 where none is used */
  std::vector<long long> off((size_t)nside + 1, -1);
  long long nchirp = 0;
  int twlen = nside, longest = nside; /* longest transform; longest piece in shared memory */
  for (int n = 1; n < nside; n++) {
    const int len = conv_len(n);
    if (len == 0) continue;
    off[(size_t)n] = nchirp;
    nchirp += len;
    twlen = std::max(twlen, len);
    longest = std::max(longest, len / conv_halves(len));
  }
  double2 *d_tw = nullptr, *d_chirp = nullptr, *d_g = nullptr;
  long long *d_off = nullptr;
  SP_CK(B.get(&d_tw, sizeof(double2) * (size_t)(twlen / 2 + 1)));
  SP_CK(B.get(&d_chirp, sizeof(double2) * (size_t)nchirp));
  SP_CK(B.get(&d_off, sizeof(long long) * off.size()));
  /* quarters of all northern rings (2 nside (nside - 1) + 4 nside (nside + 1) pixels), S and D */
  const long long north = 2LL * nside * (nside - 1) + 4LL * nside * (nside + 1);
  SP_CK(B.get(&d_g, sizeof(double2) * 2 * (size_t)north));
  SP_CK(cudaMemcpyAsync(d_off, off.data(), sizeof(long long) * off.size(), cudaMemcpyHostToDevice,
                        st.s));
  k_twiddles<<<(twlen / 2 + 256) / 256, 256, 0, st.s>>>(d_tw, twlen);
  SP_CK(cudaGetLastError());
  const size_t fsmem = sizeof(double2) * (size_t)longest;
  SP_CK(allow_smem(k_chirp, QF_SMEM));
  SP_CK(allow_smem(k_quarter_fft, QF_SMEM));
  if (nside > 1) {
    k_chirp<<<nside - 1, QF_THREADS, fsmem, st.s>>>(d_off, d_tw, twlen, d_chirp);
    SP_CK(cudaGetLastError());
  }
  k_quarter_fft<<<dim3(nrings, 8), QF_THREADS, fsmem, st.s>>>(d_a, d_b, nside, d_off, d_chirp, d_tw,
                                                              twlen, d_g);
  SP_CK(cudaGetLastError());
  k_ring_combine<<<dim3(nrings, (lmax + RC_THREADS) / RC_THREADS), RC_THREADS, 0, st.s>>>(
      d_g, nside, lmax, d_ph);
  SP_CK(cudaGetLastError());
  SP_CK(cudaMemsetAsync(d_alm, 0, sizeof(double) * 4 * nalm, st.s));
  const int group = std::min(ALM_GROUP, (nrings + ALM_THREADS - 1) / ALM_THREADS * ALM_THREADS);
  const size_t smem = alm_smem(group);
  if (map_b) {
    SP_CK(allow_smem(k_alm<true>, alm_smem(ALM_GROUP)));
    k_alm<true><<<lmax + 1, ALM_THREADS, smem, st.s>>>(d_ph, d_mfac, nside, lmax, group, d_alm);
  } else {
    SP_CK(allow_smem(k_alm<false>, alm_smem(ALM_GROUP)));
    k_alm<false><<<lmax + 1, ALM_THREADS, smem, st.s>>>(d_ph, d_mfac, nside, lmax, group, d_alm);
  }
  SP_CK(cudaGetLastError());
  const double omega = 4.0 * M_PI / (double)npix;
  k_alm2cl<<<(lmax + 32) / 32, 1024, 0, st.s>>>(d_alm, lmax, omega * omega, d_cl);
  SP_CK(cudaGetLastError());
  std::vector<double> cl(3 * (size_t)(lmax + 1));
  SP_CK(cudaMemcpyAsync(cl.data(), d_cl, sizeof(double) * cl.size(), cudaMemcpyDeviceToHost, st.s));
  SP_CK(cudaStreamSynchronize(st.s));
  const size_t nl = (size_t)lmax + 1;
  for (size_t l = 0; l < nl; l++) {
    cl_aa[l] = cl[l];
    if (map_b) {
      cl_ab[l] = cl[nl + l];
      cl_bb[l] = cl[2 * nl + l];
    }
  }
  return P2M_OK;
}

int32_t p2m_cl_flatsky(int32_t device, const float *map_a, const float *map_b, int32_t npix,
                       float fov_rad, double ell_max, int32_t nbins, double *ell_mean,
                       double *cl_aa, double *cl_ab, double *cl_bb, int64_t *nmodes) {
  if (!map_a || !ell_mean || !cl_aa || !nmodes || npix < 2 || !(fov_rad > 0.0f) ||
      !(ell_max > 0.0) || nbins < 1 || nbins > P2M_CL_MAXBINS)
    return P2M_ERR_BADARG;
  if (map_b && (!cl_ab || !cl_bb)) return P2M_ERR_BADARG;
  const bool pow2 = is_pow2(npix) && npix >= 4;
  if (pow2 ? npix > FFT_MAX_POW2 : npix > DFT_MAX) return P2M_ERR_BADARG;
  DeviceScope scope(device);
  if (!scope.ok) return P2M_ERR_CUDA;
  Stream st;
  if (!st.s) return P2M_ERR_CUDA;
  DevBufs B(st.s);
  const long long n2 = (long long)npix * npix;
  float *d_a = nullptr, *d_b = nullptr;
  double2 *z = nullptr, *z2 = nullptr, *tw = nullptr;
  double *d_acc = nullptr;
  SP_CK(B.get(&d_a, sizeof(float) * (size_t)n2));
  if (map_b) SP_CK(B.get(&d_b, sizeof(float) * (size_t)n2));
  SP_CK(B.get(&z, sizeof(double2) * (size_t)n2));
  SP_CK(B.get(&z2, sizeof(double2) * (size_t)n2));
  SP_CK(B.get(&tw, sizeof(double2) * (size_t)(npix / 2 + 1)));
  SP_CK(B.get(&d_acc, sizeof(double) * 5 * (size_t)nbins));
  SP_CK(cudaMemcpyAsync(d_a, map_a, sizeof(float) * (size_t)n2, cudaMemcpyHostToDevice, st.s));
  if (map_b)
    SP_CK(cudaMemcpyAsync(d_b, map_b, sizeof(float) * (size_t)n2, cudaMemcpyHostToDevice, st.s));
  SP_CK(cudaMemsetAsync(d_acc, 0, sizeof(double) * 5 * (size_t)nbins, st.s));
  const dim3 tb(32, 8), tg((npix + 31) / 32, (npix + 31) / 32);
  if (pow2) {
    const int logn = ilog2(npix);
    const size_t smem = sizeof(double2) * (size_t)npix;
    SP_CK(allow_smem(k_fft_rows<1>, FFT_SMEM));
    SP_CK(allow_smem(k_fft_rows<0>, FFT_SMEM));
    k_twiddles<<<(npix / 2 + 255) / 256, 256, 0, st.s>>>(tw, npix);
    k_fft_rows<1><<<npix, FFT_THREADS, smem, st.s>>>(z, d_a, d_b, npix, logn, tw);
    k_transpose<<<tg, tb, 0, st.s>>>(z, z2, npix);
    k_fft_rows<0><<<npix, FFT_THREADS, smem, st.s>>>(z2, nullptr, nullptr, npix, logn, tw);
  } else {
    const size_t smem = sizeof(double2) * (size_t)npix;
    k_fs_pack<<<(int)std::min<long long>((n2 + 255) / 256, 4096), 256, 0, st.s>>>(d_a, d_b, n2, z);
    k_dft_rows<<<npix, 256, smem, st.s>>>(z, z2, npix);
    k_transpose<<<tg, tb, 0, st.s>>>(z2, z, npix);
    k_dft_rows<<<npix, 256, smem, st.s>>>(z, z2, npix);
  }
  SP_CK(cudaGetLastError());
  const double ell_fund = 2.0 * M_PI / (double)fov_rad;
  int kmax = (int)std::ceil(ell_max / ell_fund);
  kmax = std::min(kmax, npix / 2 - 1); /* the Nyquist line is left out */
  if (kmax >= 1) {
    const long long total = (kmax + 1LL) * ((2LL * kmax + FS_RUN) / FS_RUN);
    const int grid = (int)std::min<long long>((total + 255) / 256, 1024);
    k_fs_bins<<<grid, 256, sizeof(double) * 5 * (size_t)nbins, st.s>>>(
        z2, npix, ell_fund, ell_max, nbins, kmax, d_acc);
    SP_CK(cudaGetLastError());
  }
  std::vector<double> acc(5 * (size_t)nbins);
  SP_CK(cudaMemcpyAsync(acc.data(), d_acc, sizeof(double) * acc.size(), cudaMemcpyDeviceToHost,
                        st.s));
  SP_CK(cudaStreamSynchronize(st.s));
  const double fov = (double)fov_rad, n4 = (double)n2 * (double)n2;
  const double norm = fov * fov / n4;
  for (int b = 0; b < nbins; b++) {
    const double *q = &acc[5 * (size_t)b];
    const double cnt = q[0];
    nmodes[b] = (int64_t)cnt;
    ell_mean[b] = cnt > 0 ? q[1] / cnt : (b + 0.5) * ell_max / nbins;
    cl_aa[b] = cnt > 0 ? norm * q[2] / cnt : 0.0;
    if (map_b) {
      cl_ab[b] = cnt > 0 ? norm * q[3] / cnt : 0.0;
      cl_bb[b] = cnt > 0 ? norm * q[4] / cnt : 0.0;
    }
  }
  return P2M_OK;
}

}  // extern "C"
