// Periodic boundary conditions (3dp/): the far images beyond the first
// layer, the dipole correction and the Ewald summation used to check them.
//
// periodic (3dp/traverse_eager.h:46-93): with the source root's multipole
// Mp at the domain centre and cyc = cycle, for each of images-1 sublevels
//   L_root += sum over the 26 x 27 offsets iX = 3*(ix,iy,iz) + (cx,cy,cz),
//             (ix,iy,iz) != 0, of M2L(Mp at offset iX*cyc)       (702 M2L)
//   Mp     += sum over the 26 offsets (ix,iy,iz) != 0 of M2M(Mp from ...)
//   cyc    *= 3.
// M2L and M2M are linear in the offset harmonics, so each sum is one
// translation with the harmonics summed over the offsets; the sums depend
// only on P, the period and the number of images and are kept between
// evaluations.  FP64 in every precision form; the per-thread partial sums are
// reduced in a fixed order, so the result is deterministic.
//
// Dipole correction (3dp/fmm.cxx:63-75): d = sum q X over all bodies,
// coef = 4 pi / (3 cycle^3); p -= coef |d|^2 / N / q, F -= coef d.
//
// Ewald (3dp/ewald.h): wave part by DFT over all sources and inverse DFT at
// the targets (waves with integer k, 0 < |k| <= ksize, in the half space of
// initWaves), real part with erfc over all sources within the cutoff at the
// nearest image per axis, self term -2/sqrt(pi) q alpha.
#include <algorithm>
#include <cmath>
#include <vector>

#include "fmm.cuh"
#include "harmonics.cuh"
#include "translations.cuh"

namespace fmm {

namespace {

constexpr int PT = 256;  // threads of the harmonic sums' CTA

// The harmonic sums of the far images, per sublevel l (period cycle * 3^l):
// H[2l] the irregular harmonics summed over the 702 M2L offsets, H[2l + 1]
// the regular harmonics summed over the 26 M2M offsets (rows of nt).  They
// depend only on P, the period and the number of images, so they are made
// once per parameter set and kept.  One CTA; T threads sum the offsets,
// then the partial sums are reduced in thread order (deterministic).
__global__ void __launch_bounds__(PT) k_periodic_harm(int P, int images, double cycle, int T, double2 *H) {
  extern __shared__ double2 sp[];  // partial[T][nt]
  const int nt = tri(P);
  double2 *part = sp;
  const int tid = threadIdx.x;
  double cyc = cycle;
  for (int level = 0; level < images - 1; level++) {
    // irregular harmonics summed over the 702 M2L offsets
    for (int e = tid; e < T * nt; e += PT) part[e] = make_double2(0, 0);
    __syncthreads();
    if (tid < T) {
      double2 *mine = part + (size_t)tid * nt;
      for (int off = tid; off < 702; off += T) {
        const int outer = off / 27, inner = off % 27;
        const int oc = outer < 13 ? outer : outer + 1;  // skip the centre (ix,iy,iz) = 0
        const int ix = oc / 9 - 1, iy = (oc / 3) % 3 - 1, iz = oc % 3 - 1;
        const int cx = inner / 9 - 1, cy = (inner / 3) % 3 - 1, cz = inner % 3 - 1;
        const Sph g = sph_of(-(ix * 3 + cx) * cyc, -(iy * 3 + cy) * cyc, -(iz * 3 + cz) * cyc);
        for (int m = 0; m < P; m++)
          irregular_column(m, P, g.r, g, [&](int n, double2 z) {
            double2 &d = mine[tri(n) + m];
            d.x += z.x;
            d.y += z.y;
          });
      }
    }
    __syncthreads();
    for (int o = tid; o < nt; o += PT) {
      double2 v = make_double2(0, 0);
      for (int t = 0; t < T; t++) {
        v.x += part[(size_t)t * nt + o].x;
        v.y += part[(size_t)t * nt + o].y;
      }
      H[(size_t)(2 * level) * nt + o] = v;
    }
    __syncthreads();
    // regular harmonics summed over the 26 M2M offsets (parent - child)
    for (int e = tid; e < T * nt; e += PT) part[e] = make_double2(0, 0);
    __syncthreads();
    if (tid < 26 && tid < T) {
      double2 *mine = part + (size_t)tid * nt;
      for (int off = tid; off < 26; off += T) {
        const int oc = off < 13 ? off : off + 1;
        const int ix = oc / 9 - 1, iy = (oc / 3) % 3 - 1, iz = oc % 3 - 1;
        const Sph g = sph_of(-ix * cyc, -iy * cyc, -iz * cyc);
        for (int m = 0; m < P; m++)
          regular_column(m, P, g.r, g, g.e, [&](int n, double2 y, double2) {
            double2 &d = mine[tri(n) + m];
            d.x += y.x;
            d.y += y.y;
          });
      }
    }
    __syncthreads();
    for (int o = tid; o < nt; o += PT) {
      double2 v = make_double2(0, 0);
      for (int t = 0; t < T; t++) {
        v.x += part[(size_t)t * nt + o].x;
        v.y += part[(size_t)t * nt + o].y;
      }
      H[(size_t)(2 * level + 1) * nt + o] = v;
    }
    __syncthreads();
    cyc *= 3;
  }
}

// Per evaluation: the root's multipole through the sublevels with the kept
// harmonic sums -- L_root += M2L(Mp, H[2l]), Mp += M2M(Mp, H[2l + 1]).  One
// CTA, a chain of images - 1 levels, so latency is all: PS lanes share an
// output, each taking every PS-th input degree (a lane's chain is about 20
// products instead of 100 at P = 10), the level's two translations run side
// by side, and the harmonic sums and the running L are in shared memory
// (P = 10, three images: 34.9 -> 11.2 us).
constexpr int PPT = 512, PS = 8;

__global__ void __launch_bounds__(PPT) k_periodic(const double2 *M, double2 *L, int P, int images, const double2 *H) {
  extern __shared__ double2 sp[];  // Mp[nt], Mn[nt], Lr[nt], H1[nt], H2[nt]
  const int nt = tri(P);
  double2 *Mp = sp, *Mn = Mp + nt, *Lr = Mn + nt, *H1 = Lr + nt, *H2 = H1 + nt;
  const int tid = threadIdx.x, sl = tid & (PS - 1);
  const unsigned grp = 0xffu << (tid & 24);  // the PS lanes of an output
  for (int o = tid; o < nt; o += PPT) {
    Mp[o] = M[o];  // the root is cell 0
    Lr[o] = L[o];
  }
  for (int level = 0; level < images - 1; level++) {
    for (int o = tid; o < 2 * nt; o += PPT) H1[o] = H[(size_t)(2 * level) * nt + o];
    __syncthreads();
    for (int g = tid / PS; g < 2 * nt; g += PPT / PS) {
      const bool up = g >= nt;  // outputs of the M2M after those of the M2L
      const int o = up ? g - nt : g, j = order_of(o), k = o - tri(j);
      double2 v = make_double2(0, 0);
      if (up) {
        for (int n = sl; n <= j; n += PS)
          m2m_terms_of(j, k, n, [&](int ia, bool ca, int nn, int oo, int f) {
            const double2 a = cmul(ca ? cconj(Mp[ia]) : Mp[ia], ylook(H2, nn, oo));
            v.x += a.x * (double)f;
            v.y += a.y * (double)f;
          });
      } else {
        for (int n = sl; n <= P - 1 - j; n += PS) m2l_add(j, k, n, Mp, H1, v.x, v.y);
      }
#pragma unroll
      for (int s = PS / 2; s > 0; s >>= 1) {
        v.x += __shfl_xor_sync(grp, v.x, s);
        v.y += __shfl_xor_sync(grp, v.y, s);
      }
      if (sl == 0) {
        if (up) Mn[o] = make_double2(Mp[o].x + v.x, Mp[o].y + v.y);
        else Lr[o] = make_double2(Lr[o].x + v.x, Lr[o].y + v.y);
      }
    }
    __syncthreads();
    for (int o = tid; o < nt; o += PPT) Mp[o] = Mn[o];
  }
  __syncthreads();
  for (int o = tid; o < nt; o += PPT) L[o] = Lr[o];
}

int periodic_threads(int P) {
  const int nt = tri(P);
  int T = 160 * 1024 / (nt * (int)sizeof(double2)) - 3;
  if (T > 64) T = 64;
  if (T < 1) T = 1;
  return T;
}

// ---- dipole correction
constexpr int DB = 256;

// The root's monopole for the far images of the mixed form: the total
// charge, summed in FP64 in a fixed order (block partial sums, then one block
// over the partials in block order).  The mixed upward pass forms it from
// FP32 products, and the far images' lattice sums multiply a spurious net
// charge by their growing image shells: at 60,000 neutral bodies, P = 10,
// the potentials then drifted from the FP64 form's by 5.9e-7, 7.9e-6 and
// 7.0e-4 with 1, 2 and 4 image layers (forces unaffected: the shift is
// nearly constant).
__global__ void k_charge_partial(const double4 *src, long n, double *part) {
  __shared__ double red[DB];
  double q = 0;
  for (long i = (long)blockIdx.x * DB + threadIdx.x; i < n; i += (long)gridDim.x * DB) q += src[i].w;
  red[threadIdx.x] = q;
  __syncthreads();
  for (int s = DB / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

__global__ void k_root_monopole(const double *part, int nblk, double2 *M) {
  if (threadIdx.x == 0) {
    double q = 0;
    for (int b = 0; b < nblk; b++) q += part[b];
    M[0] = make_double2(q, 0.0);  // M_0^0 of the root (cell 0): the total charge
  }
}

__global__ void k_dipole_partial(const double4 *src, long n, double *part) {
  __shared__ double red[3][DB];
  double d[3] = {0, 0, 0};
  for (long i = (long)blockIdx.x * DB + threadIdx.x; i < n; i += (long)gridDim.x * DB) {
    const double4 b = src[i];
    d[0] += b.x * b.w;
    d[1] += b.y * b.w;
    d[2] += b.z * b.w;
  }
  for (int q = 0; q < 3; q++) red[q][threadIdx.x] = d[q];
  __syncthreads();
  for (int s = DB / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s)
      for (int q = 0; q < 3; q++) red[q][threadIdx.x] += red[q][threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int q = 0; q < 3; q++) part[blockIdx.x * 3 + q] = red[q][0];
}

__global__ void k_dipole_apply(const double4 *src, double4 *out, long n, const double *part, int nblk,
                               double cycle) {
  double d[3] = {0, 0, 0};
  for (int b = 0; b < nblk; b++)
    for (int q = 0; q < 3; q++) d[q] += part[b * 3 + q];
  const double coef = 4 * M_PI / (3 * cycle * cycle * cycle);
  const double dn = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    double4 o = out[i];
    o.x -= coef * dn / (double)n / src[i].w;
    o.y -= coef * d[0];
    o.z -= coef * d[1];
    o.w -= coef * d[2];
    out[i] = o;
  }
}

// ---- Ewald
constexpr int EB = 256;

// ---- structure factors (3dp/ewald.h:22-34, :128-141): for every wave k of
// the list, sum_b q_b e^{i th}, th = k.x scale.
//
// e^{i th} factorises over the axes, so a body needs one sincos per axis and
// its powers e^{i l X}, l <= ksize (products of halves: l's powers carry
// about log2(l) roundings, fewer than the rounding of l X itself), and a
// wave is a product of three table entries.  A unit is (l, m, n0), l, m >= 0:
// with a+ = q ex_l ey_m and a- = q ex_l conj(ey_m), the four real sums over
// the bodies of re/im(a) cos/sin(n Z), n0 <= n < n0 + DFT_N, give the waves
// (l, m, +-n) and (l, -m, +-n): 2 x 16 FMAs and 8 products per body for up to
// 16 waves.  A thread keeps one unit's sums in registers; the block's bodies
// pass through shared tables, DFT_B at a time.  1M bodies, ksize 11 (2,787
// waves): 8600 us with a sincos per wave and body.
constexpr int DFT_T = 256, DFT_B = 32, DFT_N = 4;

// One unit; base[s] (s = 0: +m, 1: -m): where the wave (l, +-m, 0) is, or would
// be, in the list (its neighbours in n are contiguous), NO_WAVE if (l, +-m) is
// not in it.
struct DftUnit {
  int l, m, n0, nmax;
  int base[2];
  int half;  // (0, 0): only n > 0, and no negative n
  int pad;
};

constexpr int NO_WAVE = -(1 << 30);

inline size_t dft_smem(int ksize) { return ((size_t)DFT_B * 3 * (ksize + 1) + DFT_N) * sizeof(double2); }

__global__ void __launch_bounds__(DFT_T, 2) k_ewald_dft(const DftUnit *units, int nunits, const double4 *src, long n,
                                                       long chunk, int ksize, double scale, double2 *part, int nw) {
  extern __shared__ double2 tab[];  // [DFT_B][3][ksize + 1]: q e^{i l X}, e^{i m Y}, e^{i n Z}
  const int K1 = ksize + 1, row = 3 * K1;
  const int u = blockIdx.x * DFT_T + threadIdx.x;
  const bool act = u < nunits;
  const DftUnit un = units[act ? u : 0];
  double sp[DFT_N][4], sm[DFT_N][4];  // sums of (ar c, ai s, ar s, ai c) for a+ and a-
#pragma unroll
  for (int j = 0; j < DFT_N; j++)
#pragma unroll
    for (int q = 0; q < 4; q++) sp[j][q] = sm[j][q] = 0;
  const long s0 = (long)blockIdx.y * chunk, s1 = min(n, s0 + chunk);
  for (long b = s0; b < s1; b += DFT_B) {
    const int m = (int)min((long)DFT_B, s1 - b);
    __syncthreads();
    for (int e = threadIdx.x; e < 3 * m; e += DFT_T) {  // thread per (body, axis)
      const int ax = e / m, k = e - ax * m;
      const double4 B = src[b + k];
      double2 *t = tab + k * row + ax * K1;
      double2 e1;
      sincos((ax == 0 ? B.x : ax == 1 ? B.y : B.z) * scale, &e1.y, &e1.x);
      t[0] = make_double2(1, 0);
      t[1] = e1;
      for (int l = 2; l <= ksize; l++) t[l] = cmul(t[l >> 1], t[l - (l >> 1)]);
      if (ax == 0)
        for (int l = 0; l <= ksize; l++) t[l] = make_double2(B.w * t[l].x, B.w * t[l].y);
    }
    __syncthreads();
    if (act) {
      const double2 *px = tab + un.l, *py = tab + K1 + un.m, *pz = tab + 2 * K1 + un.n0;
#pragma unroll 2
      for (int k = 0; k < m; k++) {
        const double2 x = px[k * row], y = py[k * row];
        const double rr = x.x * y.x, ii = x.y * y.y, ri = x.x * y.y, ir = x.y * y.x;
        const double2 ap = make_double2(rr - ii, ri + ir), am = make_double2(rr + ii, ir - ri);
#pragma unroll
        for (int j = 0; j < DFT_N; j++) {
          // past nmax the entry belongs to the next axis or body, or (the
          // last body's) lies in the pad: read, but never stored
          const double2 z = pz[k * row + j];
          sp[j][0] += ap.x * z.x;
          sp[j][1] += ap.y * z.y;
          sp[j][2] += ap.x * z.y;
          sp[j][3] += ap.y * z.x;
          sm[j][0] += am.x * z.x;
          sm[j][1] += am.y * z.y;
          sm[j][2] += am.x * z.y;
          sm[j][3] += am.y * z.x;
        }
      }
    }
  }
  if (!act) return;
  double2 *out = part + (size_t)blockIdx.y * nw;
#pragma unroll
  for (int j = 0; j < DFT_N; j++) {
    const int nn = un.n0 + j;
    if (nn > un.nmax || (un.half && nn == 0)) continue;
#pragma unroll
    for (int sgn = 0; sgn < 2; sgn++) {
      if (un.base[sgn] == NO_WAVE) continue;
      const double(&v)[4] = sgn ? sm[j] : sp[j];
      out[un.base[sgn] + nn] = make_double2(v[0] - v[1], v[2] + v[3]);
      if (nn > 0 && !un.half) out[un.base[sgn] - nn] = make_double2(v[0] + v[1], v[3] - v[2]);
    }
  }
}

// The chunks' sums added (32 waves per block, 8 threads per wave over the
// chunks, then in thread order: deterministic) and scaled by
// coef exp(-|K|^2 coef2) / |K|^2.
__global__ void __launch_bounds__(256) k_ewald_amp(const int4 *waves, const double2 *part, int nw, int nchunk,
                                                   double scale, double coef, double coef2, double2 *amp) {
  __shared__ double2 red[8][32];
  const int w = blockIdx.x * 32 + (threadIdx.x & 31), g = threadIdx.x >> 5;
  double2 s = make_double2(0, 0);
  if (w < nw)
#pragma unroll 4
    for (int c = g; c < nchunk; c += 8) {
      const double2 v = part[(size_t)c * nw + w];
      s.x += v.x;
      s.y += v.y;
    }
  red[g][threadIdx.x & 31] = s;
  __syncthreads();
  if (g > 0 || w >= nw) return;
  for (int q = 1; q < 8; q++) {
    s.x += red[q][threadIdx.x].x;
    s.y += red[q][threadIdx.x].y;
  }
  const int4 k = waves[w];
  const double kx = k.x * scale, ky = k.y * scale, kz = k.z * scale;
  const double k2 = kx * kx + ky * ky + kz * kz;
  const double f = coef * exp(-k2 * coef2) / k2;
  amp[w] = make_double2(s.x * f, s.y * f);
}

// erfcx(x) = exp(x^2) erfc(x) for 0 <= x <= ERFCX_MAX: (x + 3) erfcx(x) as a
// polynomial in t = (x - 3) / (x + 3) (the variable of Shepherd and
// Laframboise, Math. Comp. 36, 1981), here the Chebyshev interpolant of
// degree 18 on the interval's image in t, computed in 60 digits and written
// in powers of t; relative error below 6e-16 (mean 1.2e-16), the rounding of
// the evaluation.
constexpr double ERFCX_MAX = 6.5;
__constant__ double c_erfcx[19] = {
    1.0740069070883398, -0.8833944531698829, 0.5902283571041055, -0.31046726190069107,
    0.11952776128690286, -0.026827234618913183, -0.0012124166089395308, 0.0030340619011204662,
    -0.000548310106357097, -0.00027677719242548155, 0.00010756610129636827, 3.0399762259269947e-05,
    -1.749347841768703e-05, -4.786830389538246e-06, 2.789618347258467e-06, 1.1232517707098393e-06,
    -2.9310736596525035e-07, -2.466455224073059e-07, -4.3340585473038216e-08};

__device__ __forceinline__ double erfcx_near(double x) {
  const double d = x + 3.0;
  double r;  // 1 / d: the hardware's estimate and one third-order Newton step
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  const double e = fma(-d, r, 1.0);
  r = fma(r, fma(e, e, e), r);
  const double t = (x - 3.0) * r;
  double v = c_erfcx[18];
#pragma unroll
  for (int k = 17; k >= 0; k--) v = fma(v, t, c_erfcx[k]);
  return v * r;
}

__device__ __forceinline__ double nearest_image(double d, double half, double cycle) {
  return fabs(d) > half ? d - copysign(cycle, d) : d;
}

// Real-space term of one source at the nearest image per axis, inside the
// cutoff (3dp/ewald.h:82-102 realP2P): with g = exp(-(alpha r)^2) and
// erfc(alpha r) = g erfcx(alpha r), one exponential serves both terms.
// 1/r as in pair_normal (pair64.cuh); a distance outside its range makes
// alpha r infinite or NaN, and that or alpha r > ERFCX_MAX takes CUDA's
// functions.  (Those alone: 7460 us against 5400 for 1M sources on 1,000
// targets, of whose pairs about 60% are computed; their roughly 75 FP64
// instructions take 2900 us at the FP64 peak.)
__device__ __forceinline__ void ewald_real_pair(double tx, double ty, double tz, const double4 &b, double c2,
                                                double alpha, double half, double cycle, double &p, double &fx,
                                                double &fy, double &fz) {
  const double dx = nearest_image(tx - b.x, half, cycle), dy = nearest_image(ty - b.y, half, cycle),
               dz = nearest_image(tz - b.z, half, cycle);
  const double R2 = dx * dx + dy * dy + dz * dz;
  if (0 < R2 && R2 < c2) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(R2));
    const double e = fma(-(R2 * y), y, 1.0);
    double ir = fma(y * e, fma(0.375, e, 0.5), y);
    double Rs = alpha * (R2 * ir), ex;
    if (Rs <= ERFCX_MAX) {
      ex = erfcx_near(Rs);
    } else {
      ir = rsqrt(R2);
      Rs = alpha * (R2 * ir);
      ex = erfcx(Rs);
    }
    const double g = exp(-(R2 * alpha) * alpha);
    const double pot = b.w * (g * ex) * ir;
    const double dtmp = (b.w * (M_2_SQRTPI * alpha) * g + pot) * ir * ir;
    p += pot;
    fx -= dx * dtmp;
    fy -= dy * dtmp;
    fz -= dz * dtmp;
  }
}

// Inverse DFT term of one wave at a target (3dp/ewald.h:36-51 idft).
__device__ __forceinline__ void ewald_wave_term(double tx, double ty, double tz, const int4 &k, const double2 &a,
                                                double scale, double &p, double &fx, double &fy, double &fz) {
  const double th = k.x * tx * scale + k.y * ty * scale + k.z * tz * scale;
  double s, c;
  sincos(th, &s, &c);
  const double dtmp = a.x * s - a.y * c;
  p += a.x * c + a.y * s;
  fx -= dtmp * k.x * scale;
  fy -= dtmp * k.y * scale;
  fz -= dtmp * k.z * scale;
}

// Few targets, many sources.  k_ewald_real: the real part of RT targets over
// one chunk of the sources; each source is read once for the RT targets, and
// as the sources lie in tree order the 32 of a warp are mostly all inside or
// all outside a target's cutoff, so warps skip the outside ones.  RT = 2
// leaves registers for three blocks per SM (4367 us at 1M sources, 1,000
// targets; RT = 4: 4586-4826); about 16 waves of blocks, as a last wave of
// few costs more than the chunks' sums (4 waves: 4833).  The chunks'
// sums go to `part`, which k_ewald_finish adds in order to the target record
// with the inverse DFT over all waves and the self term: a block per target.
constexpr int RT = 2;

__global__ void __launch_bounds__(EB) k_ewald_real(const double4 *src, long n, long chunk, double alpha,
                                                   double cutoff, double cycle, const double *rec, long nt,
                                                   double *part) {
  __shared__ double red[EB / 32][RT * 4];
  const long t0 = (long)blockIdx.x * RT;
  double tx[RT], ty[RT], tz[RT], acc[RT][4];
#pragma unroll
  for (int u = 0; u < RT; u++) {
    const double *r = rec + 8 * min(t0 + u, nt - 1);
    tx[u] = r[0];
    ty[u] = r[1];
    tz[u] = r[2];
#pragma unroll
    for (int q = 0; q < 4; q++) acc[u][q] = 0;
  }
  const double c2 = cutoff * cutoff, half = cycle / 2;
  const long s0 = (long)blockIdx.y * chunk, s1 = min(n, s0 + chunk);
  for (long i = s0 + threadIdx.x; i < s1; i += EB) {
    const double4 b = src[i];
#pragma unroll
    for (int u = 0; u < RT; u++)
      ewald_real_pair(tx[u], ty[u], tz[u], b, c2, alpha, half, cycle, acc[u][0], acc[u][1], acc[u][2], acc[u][3]);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int u = 0; u < RT; u++)
#pragma unroll
    for (int q = 0; q < 4; q++) {
      double v = acc[u][q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) red[warp][u * 4 + q] = v;
    }
  __syncthreads();
  if (threadIdx.x < RT * 4 && t0 + threadIdx.x / 4 < nt) {
    double v = 0;
    for (int w = 0; w < EB / 32; w++) v += red[w][threadIdx.x];
    part[((size_t)blockIdx.y * nt + t0) * 4 + threadIdx.x] = v;
  }
}

__global__ void __launch_bounds__(EB) k_ewald_finish(const int4 *waves, const double2 *amp, int nw, double scale,
                                                     double alpha, int parts, const double *part, int nchunk, long nt,
                                                     double *rec) {
  __shared__ double red[4][EB];
  double *r = rec + 8 * (long)blockIdx.x;
  const double tx = r[0], ty = r[1], tz = r[2], tq = r[3];
  double p = 0, fx = 0, fy = 0, fz = 0;
  if (parts & EXAFMM_EWALD_WAVE)
    for (int w = threadIdx.x; w < nw; w += EB) ewald_wave_term(tx, ty, tz, waves[w], amp[w], scale, p, fx, fy, fz);
  if (parts & EXAFMM_EWALD_REAL)
    for (int c = threadIdx.x; c < nchunk; c += EB) {
      const double *v = part + ((size_t)c * nt + blockIdx.x) * 4;
      p += v[0];
      fx += v[1];
      fy += v[2];
      fz += v[3];
    }
  red[0][threadIdx.x] = p;
  red[1][threadIdx.x] = fx;
  red[2][threadIdx.x] = fy;
  red[3][threadIdx.x] = fz;
  __syncthreads();
  for (int s = EB / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s)
      for (int q = 0; q < 4; q++) red[q][threadIdx.x] += red[q][threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    r[4] += red[0][0] - ((parts & EXAFMM_EWALD_SELF) ? M_2_SQRTPI * tq * alpha : 0.0);
    r[5] += red[1][0];
    r[6] += red[2][0];
    r[7] += red[3][0];
  }
}

// One thread per target (many targets): sources and waves pass through
// shared memory in tiles of EB, every thread sums its own target.
__global__ void __launch_bounds__(EB) k_ewald_targets(const double4 *src, long n, const int4 *waves,
                                                      const double2 *amp, int nw, double scale, double alpha,
                                                      double cutoff, double cycle, int parts, double *rec, long nt) {
  __shared__ double4 tile[EB];
  __shared__ int4 wtile[EB];
  __shared__ double2 atile[EB];
  const long t = (long)blockIdx.x * EB + threadIdx.x;
  double tx = 0, ty = 0, tz = 0, tq = 0;
  if (t < nt) {
    const double *r = rec + 8 * t;
    tx = r[0]; ty = r[1]; tz = r[2]; tq = r[3];
  }
  double p = 0, fx = 0, fy = 0, fz = 0;
  const double c2 = cutoff * cutoff, half = cycle / 2;
  if (parts & EXAFMM_EWALD_REAL)
    for (long b = 0; b < n; b += EB) {
      __syncthreads();
      if (b + threadIdx.x < n) tile[threadIdx.x] = src[b + threadIdx.x];
      __syncthreads();
      const int m = (int)min((long)EB, n - b);
      for (int k = 0; k < m; k++) ewald_real_pair(tx, ty, tz, tile[k], c2, alpha, half, cycle, p, fx, fy, fz);
    }
  if (parts & EXAFMM_EWALD_WAVE)
    for (int w0 = 0; w0 < nw; w0 += EB) {
      __syncthreads();
      if (w0 + (int)threadIdx.x < nw) {
        wtile[threadIdx.x] = waves[w0 + threadIdx.x];
        atile[threadIdx.x] = amp[w0 + threadIdx.x];
      }
      __syncthreads();
      const int m = min(EB, nw - w0);
      for (int k = 0; k < m; k++) ewald_wave_term(tx, ty, tz, wtile[k], atile[k], scale, p, fx, fy, fz);
    }
  if (t < nt) {
    double *r = rec + 8 * t;
    r[4] += p - ((parts & EXAFMM_EWALD_SELF) ? M_2_SQRTPI * tq * alpha : 0.0);
    r[5] += fx;
    r[6] += fy;
    r[7] += fz;
  }
}

}  // namespace

void periodic_set_attributes() {
  cudaFuncSetAttribute(k_periodic_harm, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  cudaFuncSetAttribute(k_ewald_dft, cudaFuncAttributeMaxDynamicSharedMemorySize, 110 * 1024);
}

void periodic_pass(Handle &h) {
  if (h.prm.dim == 2) return periodic_pass_2d(h);
  if (h.prm.images < 2) return;
  const int P = h.prm.P, nt = tri(P), T = periodic_threads(P), images = h.prm.images;
  const double cycle = h.prm.cycle;
  if (!(h.per_P == P && h.per_images == images && h.per_cycle == cycle)) {
    h.per_harm.need((size_t)2 * (images - 1) * nt * sizeof(double2));
    k_periodic_harm<<<1, PT, (size_t)T * nt * sizeof(double2), h.stream>>>(P, images, cycle, T,
                                                                           h.per_harm.as<double2>());
    h.launches++;
    FMM_LAUNCH();
    h.per_P = P;
    h.per_images = images;
    h.per_cycle = cycle;
  }
  if (h.prm.precision == EXAFMM_MIXED) {  // the root's monopole in FP64 (see k_charge_partial)
    const int nblk = 148;
    h.per_part.need(nblk * sizeof(double));
    k_charge_partial<<<nblk, DB, 0, h.stream>>>(h.src.as<double4>(), h.n, h.per_part.as<double>());
    k_root_monopole<<<1, 32, 0, h.stream>>>(h.per_part.as<double>(), nblk, h.M.as<double2>());
    h.launches += 2;
  }
  k_periodic<<<1, PPT, (size_t)5 * nt * sizeof(double2), h.stream>>>(h.M.as<double2>(), h.L.as<double2>(), P, images,
                                                                    h.per_harm.as<double2>());
  h.launches++;
  FMM_LAUNCH();
}

void dipole_correction(Handle &h) {
  const int nblk = 148;
  Buf part;
  part.need(nblk * 3 * sizeof(double));
  k_dipole_partial<<<nblk, DB, 0, h.stream>>>(h.src.as<double4>(), h.n, part.as<double>());
  k_dipole_apply<<<grid_for(h.n, 256) < 4096 ? grid_for(h.n, 256) : 4096, 256, 0, h.stream>>>(
      h.src.as<double4>(), h.out.as<double4>(), h.n, part.as<double>(), nblk, h.prm.cycle);
  h.launches += 2;
  FMM_LAUNCH();
  FMM_CUDA(cudaStreamSynchronize(h.stream));
  part.release();
}

// The wave list of initWaves (3dp/ewald.h:53-80) and the units of
// k_ewald_dft for ksize, kept in the handle until another ksize is asked for.
static void ewald_plan(Handle &h, int ksize) {
  if (h.ew_ksize == ksize) return;
  std::vector<int4> w;
  std::vector<DftUnit> units;
  for (int l = 0; l <= ksize; l++) {
    std::vector<int> zero(2 * ksize + 1, NO_WAVE);  // index of wave (l, m, 0)
    const int mmin = l == 0 ? 0 : -ksize;
    for (int m = mmin; m <= ksize; m++) {
      const int nmin = (l == 0 && m == 0) ? 1 : -ksize;
      bool first = true;
      for (int n = nmin; n <= ksize; n++)
        if (l * l + m * m + n * n <= ksize * ksize) {
          if (first) zero[m + ksize] = (int)w.size() - n;
          first = false;
          w.push_back(make_int4(l, m, n, 0));
        }
    }
    for (int m = 0; m <= ksize; m++) {
      if (zero[m + ksize] == NO_WAVE) continue;
      int nmax = 0;
      while (l * l + m * m + (nmax + 1) * (nmax + 1) <= ksize * ksize) nmax++;
      for (int n0 = 0; n0 <= nmax; n0 += DFT_N)
        units.push_back({l, m, n0, nmax, {zero[m + ksize], m > 0 ? zero[ksize - m] : NO_WAVE}, l == 0 && m == 0, 0});
    }
  }
  // a warp's units share n0 (its z entries are then one address)
  std::stable_sort(units.begin(), units.end(), [](const DftUnit &a, const DftUnit &b) { return a.n0 < b.n0; });
  h.ew_ksize = 0;  // until both tables are in place
  h.ew_nw = (int)w.size();
  h.ew_nunits = (int)units.size();
  h.ew_waves.need(w.size() * sizeof(int4));
  h.ew_units.need(units.size() * sizeof(DftUnit));
  FMM_CUDA(cudaMemcpyAsync(h.ew_waves.p, w.data(), w.size() * sizeof(int4), cudaMemcpyHostToDevice, h.stream));
  FMM_CUDA(cudaMemcpyAsync(h.ew_units.p, units.data(), units.size() * sizeof(DftUnit), cudaMemcpyHostToDevice,
                           h.stream));
  FMM_CUDA(cudaStreamSynchronize(h.stream));
  h.ew_ksize = ksize;
}

void ewald(Handle &h, int parts, int ksize, double alpha, double sigma, double cutoff, double cycle, double *rec_dev,
           long nt) {
  ewald_plan(h, ksize);
  const int nw = h.ew_nw;
  const int4 *waves = h.ew_waves.as<int4>();
  h.ew_amp.need(nw * sizeof(double2));
  double2 *amp = h.ew_amp.as<double2>();
  const double scale = 2 * M_PI / cycle;
  const double coef = 2 / sigma / cycle / cycle / cycle, coef2 = 1 / (4 * alpha * alpha);
  if (parts & EXAFMM_EWALD_WAVE) {
    // two resident blocks per SM, each a chunk of the bodies (whole tiles)
    const int gx = grid_for(h.ew_nunits, DFT_T);
    const long want = std::max(1, 2 * h.nsm / gx);
    const long chunk = ((h.n + want - 1) / want + DFT_B - 1) / DFT_B * DFT_B;
    const int gy = (int)((h.n + chunk - 1) / chunk);
    h.ew_part.need((size_t)gy * nw * sizeof(double2));
    k_ewald_dft<<<dim3(gx, gy), DFT_T, dft_smem(ksize), h.stream>>>(h.ew_units.as<DftUnit>(), h.ew_nunits,
                                                                    h.src.as<double4>(), h.n, chunk, ksize, scale,
                                                                    h.ew_part.as<double2>(), nw);
    k_ewald_amp<<<grid_for(nw, 32), 256, 0, h.stream>>>(waves, h.ew_part.as<double2>(), nw, gy, scale, coef, coef2,
                                                       amp);
    h.launches += 2;
    FMM_LAUNCH();
  }
  // while the targets cannot fill the GPU as threads: chunks of the sources
  // for RT targets each
  if (nt < 148L * 4 * EB) {
    int gy = 0;
    if (parts & EXAFMM_EWALD_REAL) {
      int occ = 1;
      FMM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_ewald_real, EB, 0));
      const long gx = (nt + RT - 1) / RT, want = std::max<long>(1, 16L * h.nsm * std::max(occ, 1) / gx);
      const long chunk = std::max<long>(4 * EB, ((h.n + want - 1) / want + EB - 1) / EB * EB);
      gy = (int)((h.n + chunk - 1) / chunk);
      h.ew_part.need((size_t)gy * nt * 4 * sizeof(double));
      k_ewald_real<<<dim3((unsigned)gx, gy), EB, 0, h.stream>>>(h.src.as<double4>(), h.n, chunk, alpha, cutoff, cycle,
                                                               rec_dev, nt, h.ew_part.as<double>());
      h.launches++;
    }
    k_ewald_finish<<<(unsigned)nt, EB, 0, h.stream>>>(waves, amp, nw, scale, alpha, parts, h.ew_part.as<double>(), gy,
                                                      nt, rec_dev);
  } else {
    const long n = (parts & (EXAFMM_EWALD_REAL | EXAFMM_EWALD_WAVE)) ? h.n : 0;
    k_ewald_targets<<<grid_for(nt, EB), EB, 0, h.stream>>>(h.src.as<double4>(), n, waves, amp, nw, scale, alpha,
                                                           cutoff, cycle, parts, rec_dev, nt);
  }
  h.launches++;
  FMM_LAUNCH();
}

}  // namespace fmm
