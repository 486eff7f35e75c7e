// The 2D variants (2d/, 2dp/): Laplace FMM in the plane with the log kernel
// and complex power-series expansions of P terms (2d/kernel.h:12-126), FP64.
//
// Bodies sit at z = 0 in the handle's double4 arrays (x, y, 0, q) and the
// tree and the interaction lists come from the 3D machinery: on bodies in one
// plane the octree's z digit is the same for every body of a level, so the
// octree is the reference's quadtree cell for cell (2d/build_tree.h: quadrant
// (x > X) + ((y > Y) << 1), the same centre recurrence and leaf rule); with
// the cells' z centres set to zero the dual walk's distance test and branch
// rules are the 2D ones (2d/traverse_lazy.h:27-44), and a 2dp system seeds
// the nine in-plane images (2dp/traverse_lazy.h:124-141).  What is new here
// is the arithmetic:
//   P2M, L2P   a few lanes per leaf, the leaf's coefficients in registers;
//   M2M, L2L   per level, a lane per child cell, coefficients in registers;
//   M2L        4 lanes per target cell (16 in small trees) over its ordered
//              M2L list, lane per entry (2d/kernel.h:61-90; the 2dp image
//              shift :63);
// these for orders up to 16, as compile-time constants; above, warps per leaf,
// threads per coefficient and a warp per M2L entry;
//   P2P        warp per target leaf over its ordered P2P list, the sources
//              staged, q log(1/R) and q dX / R^2 (2d/kernel.h:12-31);
//   periodic   one warp: the 72 root M2Ls and the 8-copy M2M per image level
//              (2dp/traverse_eager.h:46-93).
#include <type_traits>

#include "fmm.cuh"
#include "harmonics.cuh"

namespace fmm {

namespace {

constexpr int W2 = 4;  // warps per block
constexpr int IMG_SHIFT = 26;
constexpr u32 IDX_MASK = (1u << IMG_SHIFT) - 1;

__device__ __forceinline__ double2 cdivr(double2 a, double r) { return make_double2(a.x / r, a.y / r); }
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmulr(double2 a, double r) { return make_double2(a.x * r, a.y * r); }

// a += b c, a -= b c
__device__ __forceinline__ void cadd_mul(double2 &a, double2 b, double2 c) {
  a.x = fma(b.x, c.x, fma(-b.y, c.y, a.x));
  a.y = fma(b.x, c.y, fma(b.y, c.x, a.y));
}
__device__ __forceinline__ void csub_mul(double2 &a, double2 b, double2 c) {
  a.x = fma(-b.x, c.x, fma(b.y, c.y, a.x));
  a.y = fma(-b.x, c.y, fma(-b.y, c.x, a.y));
}

// 1/z with Smith's scaling (no overflow for large or small |z|).
__device__ __forceinline__ double2 crecip(double2 z) {
  if (fabs(z.x) >= fabs(z.y)) {
    const double r = z.y / z.x, d = z.x + z.y * r;
    return make_double2(1.0 / d, -r / d);
  }
  const double r = z.x / z.y, d = z.x * r + z.y;
  return make_double2(r / d, -1.0 / d);
}

__device__ __forceinline__ double2 clog2(double2 z) { return make_double2(log(hypot(z.x, z.y)), atan2(z.y, z.x)); }

// 1/z and log z of one offset from |z|^2 where that is well inside the range
// (one division, no hypot), else by crecip and clog2.
__device__ __forceinline__ void crecip_log(double2 z, double2 &iz, double2 &lz) {
  const double r2 = z.x * z.x + z.y * z.y;
  if (r2 > 1e-280 && r2 < 1e280) {
    const double inv = 1.0 / r2;
    iz = make_double2(z.x * inv, -z.y * inv);
    lz = make_double2(0.5 * log(r2), atan2(z.y, z.x));
  } else {
    iz = crecip(z);
    lz = clog2(z);
  }
}

// Image shift of a list entry: periodic1D of the 3D walk with z = 0.
__device__ __forceinline__ void img_shift(u32 img, double cycle, double &sx, double &sy) {
  const int ix = (int)(img % 3) - 1, iy = (int)((img / 3) % 3) - 1;
  sx = ix * cycle;
  sy = iy * cycle;
}

// P2M (2d/kernel.h:34-45): M[n] += q z^n / n!, z = X_body - X_cell.
__global__ void __launch_bounds__(W2 * 32) k2_p2m(const int *leaves, int nleaves, const int *begin, const int *count,
                                                  const double4 *xr, const double4 *src, double2 *M, int P) {
  extern __shared__ double2 sh[];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * W2 + wid;
  if (w >= nleaves) return;
  double2 *acc = sh + wid * P;
  for (int k = lane; k < P; k += 32) acc[k] = make_double2(0, 0);
  __syncwarp();
  const int c = leaves[w];
  const double4 C = xr[c];
  const int b0 = begin[c], nb = count[c];
  for (int t = 0; t < nb; t += 32) {
    const bool ok = t + lane < nb;
    const double4 B = ok ? src[b0 + t + lane] : make_double4(C.x, C.y, 0, 0.0);
    const double2 Z = make_double2(B.x - C.x, B.y - C.y);
    double2 pz = make_double2(1, 0);
    for (int n = 0; n < P; n++) {
      if (n > 0) pz = cmul(pz, cdivr(Z, (double)n));
      double x = n == 0 ? B.w : pz.x * B.w, y = n == 0 ? 0.0 : pz.y * B.w;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        x += __shfl_xor_sync(0xffffffffu, x, o);
        y += __shfl_xor_sync(0xffffffffu, y, o);
      }
      if (lane == 0) {
        acc[n].x += x;
        acc[n].y += y;
      }
    }
  }
  __syncwarp();
  for (int k = lane; k < P; k += 32) M[(long)c * P + k] = acc[k];
}

// M2M (2d/kernel.h:48-59) for the parents of one level: thread per
// (parent, k); M[k] = sum over children of M_c[k] + sum_n M_c[k-n] z^n/n!,
// z = X_child - X_parent.  Leaves keep their P2M.
__global__ void k2_m2m(int c0, int ncell, const int *child, const int *nchild, const double4 *xr, double2 *M, int P) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long)ncell * P) return;
  const int c = c0 + (int)(i / P), k = (int)(i % P);
  const int nc = nchild[c];
  if (nc == 0) return;
  const double4 X = xr[c];
  double2 s = make_double2(0, 0);
  for (int j = child[c]; j < child[c] + nc; j++) {
    const double4 Y = xr[j];
    const double2 Z = make_double2(Y.x - X.x, Y.y - X.y);
    const double2 *Mc = M + (long)j * P;
    double2 pz = make_double2(1, 0);
    s = cadd(s, Mc[k]);
    for (int n = 1; n <= k; n++) {
      pz = cmul(pz, cdivr(Z, (double)n));
      s = cadd(s, cmul(Mc[k - n], pz));
    }
  }
  M[(long)c * P + k] = s;
}

// One M2L (2d/kernel.h:61-90) of source multipole M (lane k holds M[k]) into
// lane n's coefficient L[n], offset Z = X_target - X_source - shift.
__device__ __forceinline__ double2 m2l_term(double2 Z, double2 Mk, int lane, int P) {
  const double2 invZ = crecip(Z);
  const double2 M0 = make_double2(__shfl_sync(0xffffffffu, Mk.x, 0), __shfl_sync(0xffffffffu, Mk.y, 0));
  double2 acc = make_double2(0, 0);
  if (lane == 0) {
    acc = csub(acc, cmul(M0, clog2(Z)));
  } else if (lane == 1) {
    acc = csub(acc, cmul(M0, invZ));
  }
  // lane 0: + M1/z + sum_{k>=2} M_k (k-1)!/z^k; lane 1: - sum_{k>=1} M_k k!/z^(k+1);
  // lane n >= 2: sum_{k>=0} M_k (-1)^n (n+k-1)!/z^(n+k)
  double2 pw;
  if (lane == 0 || lane == 1) {
    pw = invZ;
  } else {
    double2 pnk = make_double2(1, 0);  // (n-2)!/z^(n-1), as the reference builds it over n
    for (int m = 2; m <= lane; m++) {
      pnk = cmul(pnk, invZ);
      if (m < lane) pnk = cmulr(pnk, (double)(m - 1));
    }
    pw = cmulr(pnk, (lane & 1) ? -1.0 : 1.0);
  }
  for (int k = 0; k < P; k++) {
    const double2 m = make_double2(__shfl_sync(0xffffffffu, Mk.x, k), __shfl_sync(0xffffffffu, Mk.y, k));
    if (lane == 0) {
      if (k == 1) acc = cadd(acc, cmul(m, invZ));
      if (k >= 2) {
        pw = cmul(cmulr(invZ, (double)(k - 1)), pw);
        acc = cadd(acc, cmul(m, pw));
      }
    } else if (lane == 1) {
      if (k >= 1) {
        pw = cmul(cmulr(invZ, (double)k), pw);
        acc = csub(acc, cmul(m, pw));
      }
    } else if (lane < P) {
      pw = cmul(cmulr(invZ, (double)(lane + k - 1)), pw);
      acc = cadd(acc, cmul(m, pw));
    }
  }
  return acc;
}

// M2L over the ordered lists: warp per target cell; L[t] = the sum of its
// entries (the first writer of L).
__global__ void __launch_bounds__(W2 * 32) k2_m2l(int ncells, const int *off, const u32 *ent, const double4 *xr,
                                                  const double2 *M, double2 *L, int P, double cycle) {
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * W2 + wid;
  if (t >= ncells) return;
  const double4 X = xr[t];
  double2 acc = make_double2(0, 0);
  for (int e = off[t]; e < off[t + 1]; e++) {
    const u32 en = ent[e];
    const int s = (int)(en & IDX_MASK);
    double sx, sy;
    img_shift(en >> IMG_SHIFT, cycle, sx, sy);
    const double4 Y = xr[s];
    const double2 Z = make_double2(X.x - Y.x - sx, X.y - Y.y - sy);
    const double2 Mk = lane < P ? M[(long)s * P + lane] : make_double2(0, 0);
    acc = cadd(acc, m2l_term(Z, Mk, lane, P));
  }
  if (lane < P) L[(long)t * P + lane] = acc;
}

// The same M2L with a lane per list entry (orders P <= 16): with
// q_m = (m-1)!/z^m, the terms of m2l_term are L[n] += (-1)^n M_k q_(n+k) for
// n + k >= 1 and L[0] -= M_0 log z, so one lane evaluates a whole entry --
// one reciprocal, one logarithm, the q_m by the recurrence
// q_(m+1) = q_m m / z and P^2 complex products, summed along n + k = m --
// with every coefficient in registers (P is a compile-time constant), while
// M2L_G lanes take a target's entries in turn.  The lanes' sums are then added
// in a fixed butterfly order (deterministic).  Lists hold about 30 entries
// (33 to 35 inside a uniform tree), so a warp per target had 60% of its lanes
// busy (1M bodies, P = 10: 1100 us; 16, 8 and 4 lanes: 823, 689 and 654); trees
// too small to fill the GPU with 4 lanes per target take 16.  The operations
// are those of m2l_term in another order: the expansions agree with it, and
// with the reference, to rounding.
template <int P, int M2L_G>
__global__ void __launch_bounds__(W2 * 32) k2_m2l_lane(int ncells, const int *off, const u32 *ent, const double4 *xr,
                                                       const double2 *M, double2 *L, double cycle) {
  const int g = threadIdx.x % M2L_G, tt = (blockIdx.x * W2 * 32 + threadIdx.x) / M2L_G, t = min(tt, ncells - 1);
  const double4 X = xr[t];
  double2 acc[P];
#pragma unroll
  for (int n = 0; n < P; n++) acc[n] = make_double2(0, 0);
  for (int e = off[t] + g; e < off[t + 1]; e += M2L_G) {
    const u32 en = ent[e];
    const int s = (int)(en & IDX_MASK);
    double sx, sy;
    img_shift(en >> IMG_SHIFT, cycle, sx, sy);
    const double4 Y = xr[s];
    const double2 Z = make_double2(X.x - Y.x - sx, X.y - Y.y - sy);
    double2 Mk[P];
#pragma unroll
    for (int k = 0; k < P; k++) Mk[k] = M[(long)s * P + k];
    double2 iz, lz;
    crecip_log(Z, iz, lz);
    csub_mul(acc[0], Mk[0], lz);
    double2 q = iz;  // q_1
#pragma unroll
    for (int m = 1; m <= 2 * P - 2; m++) {
#pragma unroll
      for (int n = 0; n < P; n++) {
        const int k = m - n;
        if (k < 0 || k >= P) continue;
        if (n & 1) csub_mul(acc[n], Mk[k], q);
        else cadd_mul(acc[n], Mk[k], q);
      }
      if (m < 2 * P - 2) q = cmulr(cmul(q, iz), (double)m);
    }
  }
#pragma unroll
  for (int n = 0; n < P; n++) {
#pragma unroll
    for (int o = M2L_G / 2; o > 0; o >>= 1) {
      acc[n].x += __shfl_xor_sync(0xffffffffu, acc[n].x, o);
      acc[n].y += __shfl_xor_sync(0xffffffffu, acc[n].y, o);
    }
    if (g == n % M2L_G && tt < ncells) L[(long)t * P + n] = acc[n];
  }
}

// Far periodic images of a 2dp system (2dp/traverse_eager.h:46-93): per
// image level, the 72 M2Ls from the super-cell (the root's multipole, at the
// root's centre) shifted by (3 ix + cx, 3 iy + cy) cycles into the root's L,
// then the super-cell's multipole gathers its 8 copies (M2M), and the cycle
// triples.  One warp.
__global__ void k2_periodic(const double4 *xr, const double2 *M, double2 *L, int P, int images, double cycle) {
  __shared__ double2 Ms[32];
  const int lane = threadIdx.x;
  const double4 X = xr[0];
  if (lane < P) Ms[lane] = M[lane];
  __syncwarp();
  double2 acc = make_double2(0, 0);
  double cyc = cycle;
  for (int level = 0; level < images - 1; level++) {
    const double2 Mk = lane < P ? Ms[lane] : make_double2(0, 0);
    for (int ix = -1; ix <= 1; ix++)
      for (int iy = -1; iy <= 1; iy++) {
        if (ix == 0 && iy == 0) continue;
        for (int cx = -1; cx <= 1; cx++)
          for (int cy = -1; cy <= 1; cy++) {
            const double sx = (3 * ix + cx) * cyc, sy = (3 * iy + cy) * cyc;
            const double2 Z = make_double2(X.x - X.x - sx, X.y - X.y - sy);
            acc = cadd(acc, m2l_term(Z, Mk, lane, P));
          }
      }
    // M2M of the 8 copies at the super-cell's centre +- cycle into Ms
    double2 s = make_double2(0, 0);
    if (lane < P) {
      s = Mk;
      for (int ix = -1; ix <= 1; ix++)
        for (int iy = -1; iy <= 1; iy++) {
          if (ix == 0 && iy == 0) continue;
          const double2 Z = make_double2((X.x + ix * cyc) - X.x, (X.y + iy * cyc) - X.y);
          double2 pz = make_double2(1, 0);
          s = cadd(s, Ms[lane]);
          for (int n = 1; n <= lane; n++) {
            pz = cmul(pz, cdivr(Z, (double)n));
            s = cadd(s, cmul(Ms[lane - n], pz));
          }
        }
    }
    __syncwarp();
    if (lane < P) Ms[lane] = s;
    __syncwarp();
    cyc *= 3;
  }
  if (lane < P) L[lane] = cadd(L[lane], acc);
}

// L2L (2d/kernel.h:93-106) from the parents of one level to their children:
// thread per (child, l); L_c[l] += L_p[l] + sum_k L_p[l+k] z^k/k!,
// z = X_child - X_parent.
__global__ void k2_l2l(int c0, int ncell, const int *child, const int *nchild, const double4 *xr, double2 *L, int P) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long)ncell * 8 * P) return;  // up to 4 children (8 octants) per parent
  const int c = c0 + (int)(i / (8 * P)), r = (int)(i % (8 * P)), q = r / P, l = r % P;
  if (q >= nchild[c]) return;
  const int j = child[c] + q;
  const double4 X = xr[c], Y = xr[j];
  const double2 Z = make_double2(Y.x - X.x, Y.y - X.y);
  const double2 *Lp = L + (long)c * P;
  double2 s = cadd(L[(long)j * P + l], Lp[l]), pz = make_double2(1, 0);
  for (int k = 1; k < P - l; k++) {
    pz = cmul(pz, cdivr(Z, (double)k));
    s = cadd(s, cmul(Lp[l + k], pz));
  }
  L[(long)j * P + l] = s;
}

// L2P (2d/kernel.h:109-126): p += Re sum L[n] z^n/n!, F += (Re, -Im) of
// sum L[n+1] z^n/n!.  Adds into the near-field sums.
__global__ void __launch_bounds__(W2 * 32) k2_l2p(const int *leaves, int nleaves, const int *begin, const int *count,
                                                  const double4 *xr, const double4 *src, const double2 *L,
                                                  double4 *out, int P) {
  extern __shared__ double2 sh[];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * W2 + wid;
  if (w >= nleaves) return;
  const int c = leaves[w];
  double2 *Lc = sh + wid * P;
  for (int k = lane; k < P; k += 32) Lc[k] = L[(long)c * P + k];
  __syncwarp();
  const double4 C = xr[c];
  const int b0 = begin[c], nb = count[c];
  for (int t = lane; t < nb; t += 32) {
    const double4 B = src[b0 + t];
    const double2 Z = make_double2(B.x - C.x, B.y - C.y);
    double p = Lc[0].x, fx = P > 1 ? Lc[1].x : 0.0, fy = P > 1 ? -Lc[1].y : 0.0;
    double2 pz = make_double2(1, 0);
    for (int n = 1; n < P; n++) {
      pz = cmul(pz, cdivr(Z, (double)n));
      p += cmul(Lc[n], pz).x;
      if (n < P - 1) {
        const double2 f = cmul(Lc[n + 1], pz);
        fx += f.x;
        fy -= f.y;
      }
    }
    double4 &o = out[b0 + t];
    o.x += p;
    o.y += fx;
    o.z += fy;
  }
}

// ---- orders up to 16: the same operators with every coefficient in
// registers (P a compile-time constant) and z^n/n! built with the reciprocals
// 1/n as constants.  With a warp per leaf of about 4 bodies and a division
// per term, the four took 650, 318, 316 and 355 us at 1M bodies, P = 10,
// ncrit = 8, where they now take 28, 42, 82 and 77 us (their reads and writes, 60-130 MB
// each, take 10-20 us; the rest is latency of short leaves and levels).
template <int P>
__device__ __forceinline__ double2 next_power(double2 pz, double2 Z, int n) {
  return cmul(pz, cmulr(Z, 1.0 / n));  // n is a constant of the unrolled loop
}

// P2M: G lanes per leaf (a power of two), each summing every G-th body; the
// lanes' sums are added in butterfly order.
template <int P, int G>
__global__ void __launch_bounds__(128) k2_p2m_r(const int *leaves, int nleaves, const int *begin, const int *count,
                                                const double4 *xr, const double4 *src, double2 *M) {
  const int t = blockIdx.x * 128 + threadIdx.x, w = min(t / G, nleaves - 1), g = t % G;
  const int c = leaves[w], b0 = begin[c], nb = count[c];
  const double4 C = xr[c];
  double2 acc[P];
#pragma unroll
  for (int n = 0; n < P; n++) acc[n] = make_double2(0, 0);
  for (int b = g; b < nb; b += G) {
    const double4 B = src[b0 + b];
    const double2 Z = make_double2(B.x - C.x, B.y - C.y);
    double2 pz = make_double2(1, 0);
    acc[0].x += B.w;
#pragma unroll
    for (int n = 1; n < P; n++) {
      pz = next_power<P>(pz, Z, n);
      acc[n].x = fma(pz.x, B.w, acc[n].x);
      acc[n].y = fma(pz.y, B.w, acc[n].y);
    }
  }
#pragma unroll
  for (int n = 0; n < P; n++)
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      acc[n].x += __shfl_xor_sync(0xffffffffu, acc[n].x, o);
      acc[n].y += __shfl_xor_sync(0xffffffffu, acc[n].y, o);
    }
  if (t / G >= nleaves) return;
#pragma unroll
  for (int n = 0; n < P; n++)
    if (n % G == g) M[(long)c * P + n] = acc[n];
}

// M2M for the parents of one level: four lanes per parent, a lane per child
// (a quadtree cell has at most four), added in butterfly order.
template <int P>
__global__ void __launch_bounds__(128) k2_m2m_r(int c0, int ncell, const int *child, const int *nchild,
                                                const double4 *xr, double2 *M) {
  const int t = blockIdx.x * 128 + threadIdx.x, q = t & 3;
  const int c = c0 + min(t >> 2, ncell - 1), nc = nchild[c];
  double2 acc[P];
#pragma unroll
  for (int n = 0; n < P; n++) acc[n] = make_double2(0, 0);
  if (q < nc) {
    const int j = child[c] + q;
    const double4 X = xr[c], Y = xr[j];
    const double2 Z = make_double2(Y.x - X.x, Y.y - X.y);
    double2 Mc[P], pz = make_double2(1, 0);
#pragma unroll
    for (int n = 0; n < P; n++) acc[n] = Mc[n] = M[(long)j * P + n];
#pragma unroll
    for (int n = 1; n < P; n++) {
      pz = next_power<P>(pz, Z, n);
#pragma unroll
      for (int k = n; k < P; k++) cadd_mul(acc[k], Mc[k - n], pz);
    }
  }
#pragma unroll
  for (int n = 0; n < P; n++)
#pragma unroll
    for (int o = 2; o > 0; o >>= 1) {
      acc[n].x += __shfl_xor_sync(0xffffffffu, acc[n].x, o);
      acc[n].y += __shfl_xor_sync(0xffffffffu, acc[n].y, o);
    }
  if ((t >> 2) >= ncell || nc == 0) return;  // a leaf keeps its P2M
#pragma unroll
  for (int n = 0; n < P; n++)
    if ((n & 3) == q) M[(long)c * P + n] = acc[n];
}

// L2L into the cells [c0, c0 + ncell) of one level: a thread per cell.
template <int P>
__global__ void __launch_bounds__(128) k2_l2l_r(int c0, int ncell, const int *parent, const double4 *xr, double2 *L) {
  const int t = blockIdx.x * 128 + threadIdx.x;
  if (t >= ncell) return;
  const int j = c0 + t, c = parent[j];
  if (c < 0) return;
  const double4 X = xr[c], Y = xr[j];
  const double2 Z = make_double2(Y.x - X.x, Y.y - X.y);
  double2 Lp[P], acc[P], pz = make_double2(1, 0);
#pragma unroll
  for (int n = 0; n < P; n++) {
    Lp[n] = L[(long)c * P + n];
    acc[n] = cadd(L[(long)j * P + n], Lp[n]);
  }
#pragma unroll
  for (int k = 1; k < P; k++) {
    pz = next_power<P>(pz, Z, k);
#pragma unroll
    for (int l = 0; l + k < P; l++) cadd_mul(acc[l], Lp[l + k], pz);
  }
#pragma unroll
  for (int n = 0; n < P; n++) L[(long)j * P + n] = acc[n];
}

// L2P: G lanes per leaf, each taking every G-th body; Horner's scheme for the
// potential and the force: sum L_n z^n/n! = L_0 + z/1 (L_1 + z/2 (L_2 + ...)).
template <int P, int G>
__global__ void __launch_bounds__(128) k2_l2p_r(const int *leaves, int nleaves, const int *begin, const int *count,
                                                const double4 *xr, const double4 *src, const double2 *L,
                                                double4 *out) {
  const int t = blockIdx.x * 128 + threadIdx.x, w = t / G, g = t % G;
  if (w >= nleaves) return;
  const int c = leaves[w], b0 = begin[c], nb = count[c];
  const double4 C = xr[c];
  double2 Lc[P];
#pragma unroll
  for (int n = 0; n < P; n++) Lc[n] = L[(long)c * P + n];
  for (int b = b0 + g; b < b0 + nb; b += G) {
    const double4 B = src[b];
    const double2 Z = make_double2(B.x - C.x, B.y - C.y);
    double2 h = Lc[P - 1], f = Lc[P - 1];
#pragma unroll
    for (int n = P - 1; n > 0; n--) {
      const double2 zn = cmulr(Z, 1.0 / n);
      if (n < P - 1) {
        double2 v = Lc[n];
        cadd_mul(v, f, zn);
        f = v;
      }
      double2 v = Lc[n - 1];
      cadd_mul(v, h, zn);
      h = v;
    }
    double4 o = out[b];
    o.x += h.x;
    o.y += f.x;
    o.z -= f.y;
    out[b] = o;
  }
}

// P2P (2d/kernel.h:12-31; 2dp: the image shift of each list entry):
// p += q log(1/r), F -= q (dx, dy) / r^2 over the target leaf's ordered near
// list; writes out (the first writer).  A warp per target leaf.  The bodies of
// the list's leaves are staged S2 at a time in shared memory (PERIODIC: with
// their image's shift, subtracted after the positions as the reference does:
// whether two bodies a period apart coincide depends on it), and the lanes are (target i, part g): every lane takes every
// G-th staged body, G = floor(32 / targets), so the lanes are busy whatever
// the sizes of the source leaves (with the entries dealt to the parts, 884 us
// at 1M bodies, ncrit = 8; now 650).  The parts' sums are added in part
// order at the end (deterministic).  log(1/r) is -log(r^2) / 2; pairs at
// distance zero count nothing.
constexpr int S2 = 128;

// 1/x for a normal x far from the ends of the range: the hardware's estimate
// and one third-order Newton step.
__device__ __forceinline__ double recip_normal(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

template <bool PERIODIC>
__global__ void __launch_bounds__(W2 * 32) k2_p2p(const int *leaves, int nleaves, const int *begin, const int *count,
                                                  const int *off, const u32 *ent, const double4 *src, double4 *out,
                                                  double cycle) {
  __shared__ double2 sxy[W2][S2];
  __shared__ double sq[W2][S2];
  __shared__ double2 ssh[W2][PERIODIC ? S2 : 1];
  constexpr unsigned FULL = 0xffffffffu;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * W2 + wid;
  if (w >= nleaves) return;  // warp-uniform
  const int c = leaves[w], b0 = begin[c], nb = count[c];
  const int e0 = off[c], e1 = off[c + 1];
  const int span = min(nb, 32), G = 32 / span;  // targets per pass, parts
  const int i = lane % span, g = lane / span;
  for (int tb = 0; tb < nb; tb += span) {
    const int t = tb + i;
    const bool ok = g < G && t < nb;
    const double4 T = ok ? src[b0 + t] : make_double4(0, 0, 0, 0);
    double lp = 0, fx = 0, fy = 0;  // sums of q log r^2, q dx / r^2, q dy / r^2
    for (int e = e0; e < e1; e += 32) {
      // lane k: the k-th of up to 32 source leaves
      int n = 0, base = 0;
      double sx = 0, sy = 0;
      if (e + lane < e1) {
        const u32 en = ent[e + lane];
        const int s = (int)(en & IDX_MASK);
        n = count[s];
        base = begin[s];
        img_shift(en >> IMG_SHIFT, cycle, sx, sy);
      }
      int inc = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(FULL, inc, o);
        if (lane >= o) inc += v;
      }
      const int total = __shfl_sync(FULL, inc, 31);
      base -= inc - n;  // body of slot j of this leaf: base + j
      for (int w0 = 0; w0 < total; w0 += S2) {
        const int m = min(S2, total - w0);
        __syncwarp();
        for (int k = lane; k - lane < m; k += 32) {
          const int j = w0 + k;
          int lo = 0;  // the leaves that end at or before slot j
#pragma unroll
          for (int step = 16; step > 0; step >>= 1)
            if (__shfl_sync(FULL, inc, lo + step - 1) <= j) lo += step;
          const int bk = __shfl_sync(FULL, base, lo & 31);
          double2 sh;
          if (PERIODIC) sh = make_double2(__shfl_sync(FULL, sx, lo & 31), __shfl_sync(FULL, sy, lo & 31));
          if (k < m) {
            const double4 B = src[bk + j];
            sxy[wid][k] = make_double2(B.x, B.y);
            sq[wid][k] = B.w;
            if (PERIODIC) ssh[wid][k] = sh;
          }
        }
        __syncwarp();
        if (ok) {
#pragma unroll 2
          for (int k = g; k < m; k += G) {
            const double2 S = sxy[wid][k];
            double q = sq[wid][k];
            double dx = T.x - S.x, dy = T.y - S.y;
            if (PERIODIC) {
              dx -= ssh[wid][k].x;
              dy -= ssh[wid][k].y;
            }
            double r2 = dx * dx + dy * dy;
            if (r2 == 0) {
              r2 = 1;
              q = 0;
            }
            const double inv = r2 > 1e-280 && r2 < 1e280 ? recip_normal(r2) : 1.0 / r2;
            const double qi = q * inv;
            lp = fma(q, log(r2), lp);
            fx = fma(dx, qi, fx);
            fy = fma(dy, qi, fy);
          }
        }
      }
    }
    // part 0 adds the other parts' sums in part order
    for (int gg = 1; gg < G; gg++) {
      const int from = (gg * span + i) & 31;
      const double vp = __shfl_sync(FULL, lp, from), vx = __shfl_sync(FULL, fx, from), vy = __shfl_sync(FULL, fy, from);
      if (g == 0) {
        lp += vp;
        fx += vx;
        fy += vy;
      }
    }
    if (ok && g == 0) out[b0 + t] = make_double4(-0.5 * lp, -fx, -fy, 0.0);
  }
}

// Direct summation (2d/traverse_eager.h:69-80 direct; 2dp with the
// (2 prange + 1)^2 images, 2dp/traverse_eager.h:124-143): one thread per
// target, sources in shared tiles; p, F add into out.
constexpr int DT2 = 256;
__global__ void __launch_bounds__(DT2) k2_direct(const double4 *tgt, long nt, const double4 *src, long ns,
                                                 double4 *out, int prange, double cycle) {
  __shared__ double4 tile[DT2];
  const long i = (long)blockIdx.x * DT2 + threadIdx.x;
  const double4 T = i < nt ? tgt[i] : make_double4(0, 0, 0, 0);
  double p = 0, fx = 0, fy = 0;
  for (long b = 0; b < ns; b += DT2) {
    __syncthreads();
    if (b + threadIdx.x < ns) tile[threadIdx.x] = src[b + threadIdx.x];
    __syncthreads();
    const int m = (int)min((long)DT2, ns - b);
    for (int ix = -prange; ix <= prange; ix++)
      for (int iy = -prange; iy <= prange; iy++) {
        const double sx = ix * cycle, sy = iy * cycle;
        for (int k = 0; k < m; k++) {
          const double4 S = tile[k];
          const double dx = T.x - S.x - sx, dy = T.y - S.y - sy;
          const double R2 = dx * dx + dy * dy;
          if (R2 != 0) {
            const double invR = 1 / sqrt(R2);
            p += S.w * log(invR);
            fx += dx * S.w / R2;
            fy += dy * S.w / R2;
          }
        }
      }
  }
  if (i < nt) {
    out[i].x += p;
    out[i].y -= fx;
    out[i].z -= fy;
  }
}

// Cells of a 2D tree lie in the plane z = 0.
__global__ void k2_flatten(double4 *xr, int ncells) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < ncells) xr[c].z = 0.0;
}

}  // namespace

void flatten_tree_2d(Handle &h) {
  k2_flatten<<<grid_for(h.ncells, 256), 256, 0, h.stream>>>(h.c_xr.as<double4>(), h.ncells);
  h.launches++;
  FMM_LAUNCH();
}

// f(P as a constant) for the orders with register kernels; false for others.
template <class F>
bool with_order(int P, F f) {
  switch (P) {
#define EXAFMM_2D_ORDER(p) \
  case p:                  \
    f(std::integral_constant<int, p>{}); \
    return true;
    EXAFMM_2D_ORDER(2) EXAFMM_2D_ORDER(3) EXAFMM_2D_ORDER(4) EXAFMM_2D_ORDER(5) EXAFMM_2D_ORDER(6)
    EXAFMM_2D_ORDER(7) EXAFMM_2D_ORDER(8) EXAFMM_2D_ORDER(9) EXAFMM_2D_ORDER(10) EXAFMM_2D_ORDER(11)
    EXAFMM_2D_ORDER(12) EXAFMM_2D_ORDER(13) EXAFMM_2D_ORDER(14) EXAFMM_2D_ORDER(15) EXAFMM_2D_ORDER(16)
#undef EXAFMM_2D_ORDER
  }
  return false;
}

// Lanes per leaf of P2M and L2P: one while the leaves are short on average,
// else eight.
constexpr int LEAF_LANES = 8, LONG_LEAF = 12;
bool long_leaves(const Handle &h) { return h.n > (int64_t)LONG_LEAF * h.nleaves; }

void upward_pass_2d(Handle &h, cudaStream_t s) {
  const int P = h.prm.P;
  const size_t expansions = (size_t)h.ncells * P * sizeof(double2);
  h.exp_mem.need({{&h.M, expansions}, {&h.L, expansions}});
  const bool done = with_order(P, [&](auto pc) {
    constexpr int PP = decltype(pc)::value;
    auto p2m = [&](auto gc) {
      constexpr int G = decltype(gc)::value;
      k2_p2m_r<PP, G><<<grid_for((long)h.nleaves * G, 128), 128, 0, s>>>(
          h.leaves.as<int>(), h.nleaves, h.c_begin.as<int>(), h.c_count.as<int>(), h.c_xr.as<double4>(),
          h.src.as<double4>(), h.M.as<double2>());
    };
    if (long_leaves(h)) p2m(std::integral_constant<int, LEAF_LANES>{});
    else p2m(std::integral_constant<int, 1>{});
    h.launches++;
    for (int l = h.depth - 1; l >= 0; l--) {
      const int c0 = h.level_base[l], c1 = h.level_base[l + 1];
      if (c1 <= c0) continue;
      k2_m2m_r<PP><<<grid_for((long)(c1 - c0) * 4, 128), 128, 0, s>>>(c0, c1 - c0, h.c_child.as<int>(),
                                                                     h.c_nchild.as<int>(), h.c_xr.as<double4>(),
                                                                     h.M.as<double2>());
      h.launches++;
    }
    FMM_LAUNCH();
  });
  if (done) return;
  k2_p2m<<<grid_for(h.nleaves, W2), W2 * 32, W2 * P * sizeof(double2), s>>>(
      h.leaves.as<int>(), h.nleaves, h.c_begin.as<int>(), h.c_count.as<int>(), h.c_xr.as<double4>(),
      h.src.as<double4>(), h.M.as<double2>(), P);
  h.launches++;
  FMM_LAUNCH();
  for (int l = h.depth - 1; l >= 0; l--) {
    const int c0 = h.level_base[l], c1 = h.level_base[l + 1];
    if (c1 <= c0) continue;
    k2_m2m<<<grid_for((long)(c1 - c0) * P, 256), 256, 0, s>>>(c0, c1 - c0, h.c_child.as<int>(), h.c_nchild.as<int>(),
                                                             h.c_xr.as<double4>(), h.M.as<double2>(), P);
    h.launches++;
    FMM_LAUNCH();
  }
}

constexpr int M2L_MANY = 20000;  // cells: about 16 warps per SM at 4 lanes per target

void m2l_pass_2d(Handle &h) {
  const int P = h.prm.P;
  h.L.need((size_t)h.ncells * P * sizeof(double2));
  order_m2l_lists(h);
  const double cyc = h.prm.images ? h.prm.cycle : 0.0;
  const int g = grid_for(h.ncells, W2);
  const bool done = with_order(P, [&](auto pc) {
    constexpr int PP = decltype(pc)::value;
    auto lanes = [&](auto gc) {
      constexpr int G = decltype(gc)::value;
      k2_m2l_lane<PP, G><<<grid_for((long)h.ncells * G, W2 * 32), W2 * 32, 0, h.stream>>>(
          h.ncells, h.m2l_off.as<int>(), h.m2l_ent.as<u32>(), h.c_xr.as<double4>(), h.M.as<double2>(),
          h.L.as<double2>(), cyc);
    };
    if (h.ncells >= M2L_MANY) lanes(std::integral_constant<int, 4>{});
    else lanes(std::integral_constant<int, 16>{});
  });
  if (!done)  // larger orders: a warp per entry, a lane per coefficient
    k2_m2l<<<g, W2 * 32, 0, h.stream>>>(h.ncells, h.m2l_off.as<int>(), h.m2l_ent.as<u32>(), h.c_xr.as<double4>(),
                                        h.M.as<double2>(), h.L.as<double2>(), P, cyc);
  h.launches++;
  FMM_LAUNCH();
}

void periodic_pass_2d(Handle &h) {
  if (h.prm.images < 2) return;
  k2_periodic<<<1, 32, 0, h.stream>>>(h.c_xr.as<double4>(), h.M.as<double2>(), h.L.as<double2>(), h.prm.P,
                                      h.prm.images, h.prm.cycle);
  h.launches++;
  FMM_LAUNCH();
}

void p2p_pass_2d(Handle &h, cudaStream_t s) {
  h.out.need((size_t)h.n * sizeof(double4));
  auto kern = h.prm.images ? k2_p2p<true> : k2_p2p<false>;
  kern<<<grid_for(h.nleaves, W2), W2 * 32, 0, s>>>(h.leaves.as<int>(), h.nleaves, h.c_begin.as<int>(),
                                                     h.c_count.as<int>(), h.p2p_off.as<int>(), h.p2p_ent.as<u32>(),
                                                     h.src.as<double4>(), h.out.as<double4>(),
                                                     h.prm.images ? h.prm.cycle : 0.0);
  h.launches++;
  FMM_LAUNCH();
}

void downward_pass_2d(Handle &h, cudaStream_t s, cudaEvent_t before_l2p) {
  const int P = h.prm.P;
  const bool done = with_order(P, [&](auto pc) {
    constexpr int PP = decltype(pc)::value;
    for (int l = 1; l <= h.depth; l++) {
      const int c0 = h.level_base[l], c1 = h.level_base[l + 1];
      if (c1 <= c0) continue;
      k2_l2l_r<PP><<<grid_for(c1 - c0, 128), 128, 0, s>>>(c0, c1 - c0, h.c_parent.as<int>(), h.c_xr.as<double4>(),
                                                          h.L.as<double2>());
      h.launches++;
    }
    if (before_l2p) FMM_CUDA(cudaStreamWaitEvent(s, before_l2p, 0));
    auto l2p = [&](auto gc) {
      constexpr int G = decltype(gc)::value;
      k2_l2p_r<PP, G><<<grid_for((long)h.nleaves * G, 128), 128, 0, s>>>(
          h.leaves.as<int>(), h.nleaves, h.c_begin.as<int>(), h.c_count.as<int>(), h.c_xr.as<double4>(),
          h.src.as<double4>(), h.L.as<double2>(), h.out.as<double4>());
    };
    if (long_leaves(h)) l2p(std::integral_constant<int, LEAF_LANES>{});
    else l2p(std::integral_constant<int, 1>{});
    h.launches++;
    FMM_LAUNCH();
  });
  if (done) return;
  for (int l = 0; l < h.depth; l++) {
    const int c0 = h.level_base[l], c1 = h.level_base[l + 1];
    if (c1 <= c0) continue;
    k2_l2l<<<grid_for((long)(c1 - c0) * 8 * P, 256), 256, 0, s>>>(c0, c1 - c0, h.c_child.as<int>(),
                                                                  h.c_nchild.as<int>(), h.c_xr.as<double4>(),
                                                                  h.L.as<double2>(), P);
    h.launches++;
    FMM_LAUNCH();
  }
  if (before_l2p) FMM_CUDA(cudaStreamWaitEvent(s, before_l2p, 0));
  k2_l2p<<<grid_for(h.nleaves, W2), W2 * 32, W2 * P * sizeof(double2), s>>>(
      h.leaves.as<int>(), h.nleaves, h.c_begin.as<int>(), h.c_count.as<int>(), h.c_xr.as<double4>(),
      h.src.as<double4>(), h.L.as<double2>(), h.out.as<double4>(), P);
  h.launches++;
  FMM_LAUNCH();
}

void direct_sum_2d(Handle &h, double4 *targets, double4 *out, long nt) {
  int prange = 0;  // r = sum_{i < images} 3^i (2dp/traverse_eager.h:131-134)
  for (int i = 0, p3 = 1; i < h.prm.images; i++, p3 *= 3) prange += p3;
  k2_direct<<<grid_for(nt, DT2), DT2, 0, h.stream>>>(targets, nt, h.src.as<double4>(), h.n, out, prange,
                                                     h.prm.images ? h.prm.cycle : 0.0);
  h.launches++;
  FMM_LAUNCH();
}

}  // namespace fmm
