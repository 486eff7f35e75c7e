// GPU octree build, bit-exact against the reference's recursive build
// (3d/build_tree.h:24-96, identical in 3dp/).
//
// The reference splits a cell by comparing each body with a centre that is
// produced by rounded FP64 additions, Xchild = X +/- R0/2^(level+1)
// (:116-126), leaf when NBODY <= ncrit (:81), children in octant order, bodies
// stably partitioned (:91-114).  Here:
//   1. bounds: min/max reduction, then X0, R0 exactly as getBounds (:7-21);
//   2. keys: per body, the octant digit of every level, each computed against
//      the centre of the body's own cell at that level by the same rounded
//      recurrence (__dadd_rn, no FMA contraction) -> a 3-bit-per-level key;
//   3. a stable LSD radix sort of (key, input index) on the key bits;
//   4. cells straight from the sorted keys: body i starts the cell of level l
//      that contains it iff the level-l key prefix changes at i and the parent
//      run holds more than ncrit bodies; run lengths come from binary searches
//      on the sorted keys.  Counting those cells per body and scanning gives
//      every cell its depth-first pre-order rank (cells sorted by first body,
//      then level) without any recursion;
//   5. a stable sort of the pre-order table by level gives the BFS layout the
//      level-synchronous passes use (children stay contiguous), and the
//      reference's own cell numbering (children appended as one block per
//      parent in pre-order) follows from a scan of child counts;
//   6. bodies inside each leaf are put back into input order (the reference's
//      stable partition never reorders bodies of one leaf).
// The key holds 3 bits per level for the first `key_levels` levels; if a cell
// at that depth still needs splitting the build is repeated with all 21.
//
// Batches of independent systems build one forest: every system gets its own
// bounds and root geometry, the system index sits above the octant digits in
// the sort key (so it is the level-0 prefix), each system's root always exists,
// and nothing else changes -- every system's cells and body order come out as
// if it were built alone, one after the other.
#include <cmath>

#include "fmm.cuh"
#include "srcf.cuh"

namespace fmm {

namespace {

constexpr int TB = 256;

__device__ __forceinline__ double dmin(double a, double b) { return fmin(a, b); }
__device__ __forceinline__ double dmax(double a, double b) { return fmax(a, b); }

// Min/max of the block's threads into thread 0 (exact operations: the
// reduction order cannot change the result).
__device__ void block_minmax(double lo[3], double hi[3]) {
  __shared__ double s[TB / 32][6];
  for (int o = 16; o > 0; o >>= 1)
    for (int d = 0; d < 3; d++) {
      lo[d] = dmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
      hi[d] = dmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
    }
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0)
    for (int d = 0; d < 3; d++) { s[w][d] = lo[d]; s[w][3 + d] = hi[d]; }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int k = 1; k < TB / 32; k++)
      for (int d = 0; d < 3; d++) { lo[d] = dmin(s[k][d], lo[d]); hi[d] = dmax(s[k][3 + d], hi[d]); }
}

// getBounds (3d/build_tree.h:7-21): centre = (max+min)/2, R0 = largest
// half-extent about that centre, times 1.00001.
__device__ __forceinline__ void set_root(RootGeom *g, const double lo[3], const double hi[3]) {
  double R0 = 0;
  for (int d = 0; d < 3; d++) {
    g->X0[d] = __ddiv_rn(__dadd_rn(hi[d], lo[d]), 2.0);
    R0 = dmax(__dadd_rn(g->X0[d], -lo[d]), R0);
    R0 = dmax(__dadd_rn(hi[d], -g->X0[d]), R0);
  }
  g->R0 = __dmul_rn(R0, 1.00001);
}

// Bounds of one system.  The blocks' bounds go to `part`; the last block to
// finish combines them and zeroes the counters for the build (one launch where
// the combination and the zeroing took two more).
__global__ void __launch_bounds__(TB) k_bounds(const double4 *in, long n, double *part, RootGeom *g, DevCounters *ctr) {
  double lo[3] = {in[0].x, in[0].y, in[0].z}, hi[3] = {lo[0], lo[1], lo[2]};
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const double4 b = in[i];
    lo[0] = dmin(b.x, lo[0]); lo[1] = dmin(b.y, lo[1]); lo[2] = dmin(b.z, lo[2]);
    hi[0] = dmax(b.x, hi[0]); hi[1] = dmax(b.y, hi[1]); hi[2] = dmax(b.z, hi[2]);
  }
  block_minmax(lo, hi);
  __shared__ bool last;
  if (threadIdx.x == 0) {
    for (int d = 0; d < 3; d++) {
      part[blockIdx.x * 6 + d] = lo[d];
      part[blockIdx.x * 6 + 3 + d] = hi[d];
    }
    __threadfence();
    last = atomicAdd(&ctr->bounds_ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int d = 0; d < 3; d++) {
    lo[d] = __ldcg(&part[d]);
    hi[d] = __ldcg(&part[3 + d]);
  }
  for (int k = threadIdx.x; k < (int)gridDim.x; k += TB)
    for (int d = 0; d < 3; d++) {
      lo[d] = dmin(__ldcg(&part[6 * k + d]), lo[d]);
      hi[d] = dmax(__ldcg(&part[6 * k + 3 + d]), hi[d]);
    }
  block_minmax(lo, hi);
  for (int k = threadIdx.x; k < (int)(sizeof(DevCounters) / sizeof(int)); k += TB) ((int *)ctr)[k] = 0;
  if (threadIdx.x != 0) return;
  set_root(g, lo, hi);
}

// Bounds of every system of a batch, the same getBounds arithmetic.  A system
// is cut into pieces of `piece` bodies, a block each (blocks by the largest
// system's pieces, idle past their own system's end); the piece that finishes
// last combines them.  With one block per system the launch waited for the
// largest: 87 us for 256 systems of up to 65,536 bodies, now 30.  Pieces of at
// least BPIECE bodies, and in all at most about BPIECES of them, however
// uneven the systems.
constexpr long BPIECE = 8192, BPIECES = 65536;

__global__ void __launch_bounds__(TB) k_bounds_systems(const double4 *in, const long long *off, long piece,
                                                       double *part, unsigned *ticket, RootGeom *geom) {
  const int sys = blockIdx.y;
  const long b0 = off[sys], b1 = off[sys + 1];
  const int pieces = (int)((b1 - b0 + piece - 1) / piece), k = blockIdx.x;
  if (k >= pieces) return;
  const long s0 = b0 + k * piece, s1 = min(b1, s0 + piece);
  double lo[3] = {in[s0].x, in[s0].y, in[s0].z}, hi[3] = {lo[0], lo[1], lo[2]};
  for (long i = s0 + threadIdx.x; i < s1; i += TB) {
    const double4 b = in[i];
    lo[0] = dmin(b.x, lo[0]); lo[1] = dmin(b.y, lo[1]); lo[2] = dmin(b.z, lo[2]);
    hi[0] = dmax(b.x, hi[0]); hi[1] = dmax(b.y, hi[1]); hi[2] = dmax(b.z, hi[2]);
  }
  block_minmax(lo, hi);
  __shared__ bool last;
  double *mine = part + ((size_t)sys * gridDim.x) * 6;
  if (threadIdx.x == 0) {
    last = pieces == 1;
    if (pieces > 1) {
      for (int d = 0; d < 3; d++) {
        mine[6 * k + d] = lo[d];
        mine[6 * k + 3 + d] = hi[d];
      }
      __threadfence();
      last = atomicAdd(&ticket[sys], 1u) == pieces - 1;
    }
  }
  __syncthreads();
  if (!last) return;
  if (pieces > 1) {
    __threadfence();
    for (int d = 0; d < 3; d++) {
      lo[d] = __ldcg(&mine[d]);
      hi[d] = __ldcg(&mine[3 + d]);
    }
    for (int q = threadIdx.x; q < pieces; q += TB)
      for (int d = 0; d < 3; d++) {
        lo[d] = dmin(__ldcg(&mine[6 * q + d]), lo[d]);
        hi[d] = dmax(__ldcg(&mine[6 * q + 3 + d]), hi[d]);
      }
    block_minmax(lo, hi);
  }
  if (threadIdx.x != 0) return;
  set_root(geom + sys, lo, hi);
}

// System of body i: the last s with off[s] <= i (off: nsys+1 offsets).
__device__ __forceinline__ int system_of(const long long *off, int nsys, long i) {
  int lo = 0, hi = nsys - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= i) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Octant digits of each body, level by level, against the exact centres of
// its system's cells; the system index above them.
__global__ void k_keys(const double4 *in, long n, const RootGeom *geom, const long long *sys_off, int nsys, int D,
                       u64 *keys, u32 *vals) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double4 b = in[i];
  const int sys = nsys > 1 ? system_of(sys_off, nsys, i) : 0;
  const RootGeom *g = geom + sys;
  double cx = g->X0[0], cy = g->X0[1], cz = g->X0[2];
  const double R0 = g->R0;
  u64 key = (u64)sys;
  double r = R0;
  for (int l = 0; l < D; l++) {
    const int ox = b.x > cx, oy = b.y > cy, oz = b.z > cz;
    key = (key << 3) | (u64)(ox | (oy << 1) | (oz << 2));
    r = __dmul_rn(r, 0.5);  // R0 / 2^(l+1): halving is the correctly rounded quotient
    cx = __dadd_rn(cx, ox ? r : -r);
    cy = __dadd_rn(cy, oy ? r : -r);
    cz = __dadd_rn(cz, oz ? r : -r);
  }
  keys[i] = key;
  vals[i] = (u32)i;
}

// Level-l prefix of a key: the system index and the first l octant digits.
__device__ __forceinline__ u64 prefix_of(u64 key, int D, int l) { return key >> (3 * (D - l)); }

// First index in [lo, hi) whose level-l prefix exceeds p (keys sorted, and
// keys[lo] has a prefix <= p): a galloping search up from lo, then a binary
// search in the last step -- runs near the leaves are short, so this takes
// about twice the log of the run length instead of the log of the range.
__device__ long upper_run(const u64 *keys, long lo, long hi, int D, int l, u64 p) {
  long a = lo, step = 1;
  while (a + step < hi && prefix_of(keys[a + step], D, l) <= p) {
    a += step;
    step <<= 1;
  }
  long L = a + 1, H = a + step < hi ? a + step : hi;  // the answer is in [L, H]
  while (L < H) {
    const long mid = (L + H) >> 1;
    if (prefix_of(keys[mid], D, l) > p) H = mid; else L = mid + 1;
  }
  return L;
}
// First index in [lo, hi) whose level-l prefix is >= p (keys[hi], when it
// exists, has a prefix >= p): galloping down from hi.
__device__ long lower_run(const u64 *keys, long lo, long hi, int D, int l, u64 p) {
  long b = hi, step = 1;
  while (b - step >= lo && prefix_of(keys[b - step], D, l) >= p) {
    b -= step;
    step <<= 1;
  }
  long L = b - step < lo ? lo : b - step + 1, H = b;  // the answer is in [L, H]
  while (L < H) {
    const long mid = (L + H) >> 1;
    if (prefix_of(keys[mid], D, l) >= p) H = mid; else L = mid + 1;
  }
  return L;
}

// Shallowest level whose key prefix at i differs from i-1 (D+1: same key).
__device__ __forceinline__ int first_level(const u64 *keys, long i, int D) {
  if (i == 0) return 0;
  const u64 x = keys[i] ^ keys[i - 1];
  if (x == 0) return D + 1;
  const int h = 63 - __clzll((long long)x);
  if (h >= 3 * D) return 0;  // another system: its root starts here
  return D - h / 3;
}

// Shallowest level whose key prefixes of x and y differ (D+1: none).
__device__ __forceinline__ int diff_level(u64 x, u64 y, int D) {
  const u64 d = x ^ y;
  if (d == 0) return D + 1;
  const int h = 63 - __clzll((long long)d);
  if (h >= 3 * D) return 0;  // another system
  return D - h / 3;
}

// Bodies from i on (i included) in i's level-l run, counted up to cap.
__device__ long run_ahead(const u64 *keys, long i, long n, int D, int l, u64 p, long cap) {
  const long last = i + cap < n ? i + cap : n;
  if (last == i + cap && prefix_of(keys[last - 1], D, l) == p) return cap;
  long L = i + 1, H = last;  // the run ends in [L, H]
  while (L < H) {
    const long mid = (L + H) >> 1;
    if (prefix_of(keys[mid], D, l) > p) H = mid; else L = mid + 1;
  }
  return L - i;
}

// Number of cells whose first body is sorted position i (a chain of nested
// first-children), plus the depth overflow check.  A run that starts at i
// holds more than ncrit bodies iff body i + ncrit shares its prefix, so the
// chain length follows from one comparison of keys; the parent test counts
// at most ncrit + 1 bodies on either side of i.  A chain's cells lie on
// consecutive levels and its last one is a leaf, so the cells per level and
// the leaves are counted here too: one read of the counts tells the host all
// that the launches up to the lists need.
__global__ void __launch_bounds__(TB) k_chain(const u64 *keys, long n, int D, int ncrit, int *lfirst, int *chain,
                                              DevCounters *ctr) {
  __shared__ int lc[EXAFMM_MAX_LEVEL + 2];  // cells per level that start in this block
  if (threadIdx.x < EXAFMM_MAX_LEVEL + 2) lc[threadIdx.x] = 0;
  __syncthreads();
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  int len = 0;
  const int lf = i < n ? first_level(keys, i, D) : D + 1;
  if (i < n) lfirst[i] = lf;
  if (lf <= D) {
    const u64 key = keys[i];
    bool parent_splits = true;  // a system's root is always a cell
    if (lf > 0) {
      const u64 pp = prefix_of(key, D, lf - 1);
      const long R = run_ahead(keys, i, n, D, lf - 1, pp, (long)ncrit + 1);
      const long need = (long)ncrit + 1 - R;  // parent bodies wanted before i
      parent_splits = need <= 0 || (i - need >= 0 && prefix_of(keys[i - need], D, lf - 1) == pp);
    }
    if (parent_splits) {
      // levels lf, lf+1, ... while the run from i exceeds ncrit, then the leaf
      int last = i + ncrit < n ? diff_level(key, keys[i + ncrit], D) : lf;
      if (last < lf) last = lf;
      if (last > D) {
        ctr->overflow = 1;
        last = D;
      }
      len = last - lf + 1;
    }
  }
  if (i < n) chain[i] = len;
  for (int k = 0; k < len; k++) atomicAdd_block(&lc[lf + k], 1);
  const int leaves = __syncthreads_count(len > 0);
  if (threadIdx.x == 0 && leaves) atomicAdd(&ctr->nleaves, leaves);
  if (threadIdx.x < EXAFMM_MAX_LEVEL + 2 && lc[threadIdx.x]) atomicAdd(&ctr->level_count[threadIdx.x], lc[threadIdx.x]);
}

struct PreTables {
  int *begin, *count, *level, *parent, *nchild, *face;
  double4 *xr;
};

// The body that starts each cell (pre-order rank -> sorted body position).
__global__ void k_cell_owner(long n, const int *chain, const int *prebase, int *owner) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int len = chain[i];
  for (int k = 0; k < len; k++) owner[prebase[i] + k] = (int)i;
}

// One thread per cell (pre-order rank p): the k-th cell of the chain that
// starts at body i = owner[p] is at level lfirst[i] + k.
__global__ void k_cells(const u64 *keys, long n, long C, int D, const int *lfirst, const int *owner,
                        const int *prebase, const RootGeom *g, PreTables t) {
  const long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p < C) {
    const long i = owner[p];
    const int k = (int)(p - prebase[i]), lf = lfirst[i], l = lf + k;
    const u64 key = keys[i];
    const RootGeom *gs = g + (long)(key >> (3 * D));  // the body's system
    double cx = gs->X0[0], cy = gs->X0[1], cz = gs->X0[2];
    double r = gs->R0;  // R0 / 2^l, halved exactly level by level
    int any = 0, all = l > 1 ? 7 : 0;  // octant bits on the way to the parent
    for (int q = 0; q < l; q++) {  // centre of the level-l cell holding body i
      const int o = (int)((key >> (3 * (D - 1 - q))) & 7);
      if (q < l - 1) {
        any |= o;
        all &= o;
      }
      r = __dmul_rn(r, 0.5);
      cx = __dadd_rn(cx, (o & 1) ? r : -r);
      cy = __dadd_rn(cy, (o & 2) ? r : -r);
      cz = __dadd_rn(cz, (o & 4) ? r : -r);
    }
    int parent = (int)p - 1;  // the chain's previous cell
    if (k == 0) {
      parent = -1;
      if (lf > 0) {
        const long b0 = lower_run(keys, 0, i, D, lf - 1, prefix_of(key, D, lf - 1));
        parent = prebase[b0] + (lf - 1 - lfirst[b0]);
      }
    }
    const long e = upper_run(keys, i, n, D, l, prefix_of(key, D, l));
    t.begin[p] = (int)i;
    t.count[p] = (int)(e - i);
    t.level[p] = l;
    t.parent[p] = parent;
    t.xr[p] = make_double4(cx, cy, cz, r);
    // per axis 0, 1 or 2: the parent lies at the root's low face, inside, at
    // its high face
    int face = 0;
    for (int d = 2; d >= 0; d--) face = 3 * face + ((any >> d & 1) ? 1 + (all >> d & 1) : 0);
    t.face[p] = face;
    if (parent >= 0) atomicAdd(&t.nchild[parent], 1);
  }
}

__global__ void k_level_keys(const int *level, long c, u64 *k, u32 *v) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= c) return;
  k[i] = (u64)level[i];
  v[i] = (u32)i;
}

__global__ void k_invert(const u32 *pre_of_bfs, long c, int *bfs_of_pre) {
  const long b = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (b < c) bfs_of_pre[pre_of_bfs[b]] = (int)b;
}

struct BfsCells {
  int *begin, *count, *child, *nchild, *parent, *level, *pre, *face;
  double4 *xr;
};

__global__ void k_gather_cells(const u32 *pre_of_bfs, const int *bfs_of_pre, long c, PreTables t, BfsCells o,
                               int *is_leaf) {
  const long b = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= c) return;
  const int p = (int)pre_of_bfs[b];
  o.begin[b] = t.begin[p];
  o.count[b] = t.count[p];
  o.level[b] = t.level[p];
  o.face[b] = t.face[p];
  o.xr[b] = t.xr[p];
  o.parent[b] = t.parent[p] >= 0 ? bfs_of_pre[t.parent[p]] : -1;
  const int nc = t.nchild[p];
  o.nchild[b] = nc;
  o.child[b] = nc ? bfs_of_pre[p + 1] : -1;
  o.pre[b] = p;
  is_leaf[b] = nc == 0;
}

// Reference cell number: 1 + (children allocated by parents earlier in
// pre-order) + rank among siblings (3d/build_tree.h:69-84); and the leaves in
// BFS order.
__global__ void k_ref_leaves(BfsCells o, long c, const int *blockstart_pre, int *ref, const int *is_leaf,
                             const int *leafpos, int *leaves) {
  const long b = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= c) return;
  const int par = o.parent[b];
  ref[b] = par < 0 ? 0 : 1 + blockstart_pre[o.pre[par]] + (int)(b - o.child[par]);
  if (is_leaf[b]) leaves[leafpos[b]] = (int)b;
}

// Bodies of each leaf back to input order (a warp per leaf; a body's slot is
// the rank of its input index among the leaf's), gathered into src, and (3D) the body's leaf.
// With srcf (3D mixed form) also the FP32 copy of each body as an offset from
// its leaf centre (FP64 subtraction, one rounding), alone and in pairs, as
// k_make_srcf makes them: one pass over the bodies instead of three.
__global__ void k_leaf_order(const int *leaves, int nleaves, const int *begin, const int *count, const double4 *xr,
                             const u32 *vals, const double4 *in, int *perm, double4 *src, float4 *srcf,
                             float4 *pairs, int *body_leaf) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= nleaves) return;
  const int c = leaves[w], b0 = begin[c], nb = count[c];
  const double4 C = xr[c];
  for (int a = lane; a < nb; a += 32) {
    const u32 v = vals[b0 + a];
    int r = 0;
    for (int k = 0; k < nb; k++) r += vals[b0 + k] < v;
    const int b = b0 + r;
    perm[b] = (int)v;
    const double4 B = in[v];
    src[b] = B;
    if (srcf) {
      const float4 f = make_float4((float)(B.x - C.x), (float)(B.y - C.y), (float)(B.z - C.z), (float)B.w);
      srcf[b] = f;
      put_pair(pairs, b0, r, nb, f);
    }
    if (body_leaf) body_leaf[b] = w;
  }
}


}  // namespace

void build_tree(Handle &h) {
  const long n = h.n;
  cudaStream_t s = h.stream;
  h.srcf_ready = false;  // set again once the new tree's FP32 sources are made
  const int nsys = h.nsys;
  h.geom.need((size_t)nsys * sizeof(RootGeom));
  h.counters.need(sizeof(DevCounters));
  DevCounters *ctr = h.counters.as<DevCounters>();
  RootGeom *g = h.geom.as<RootGeom>();
  const long long *sys_off = nsys > 1 ? h.sys_off.as<long long>() : nullptr;

  // 1. bounds
  if (nsys > 1) {
    long most = 0;  // bodies of the largest system
    for (int q = 0; q < nsys; q++) most = std::max<long>(most, (long)(h.sys_off_host[q + 1] - h.sys_off_host[q]));
    const long per = std::max<long>(1, BPIECES / nsys), piece = std::max(BPIECE, (most + per - 1) / per);
    const unsigned pieces = (unsigned)((most + piece - 1) / piece);
    const size_t bytes = (size_t)nsys * pieces * 6 * sizeof(double);
    h.hist.need(bytes + nsys * sizeof(unsigned));
    unsigned *ticket = (unsigned *)((char *)h.hist.p + bytes);
    FMM_CUDA(cudaMemsetAsync(ticket, 0, nsys * sizeof(unsigned), s));
    for (int q0 = 0; q0 < nsys; q0 += 65535) {  // grid.y limit
      const int nq = std::min(nsys - q0, 65535);
      k_bounds_systems<<<dim3(pieces, nq), TB, 0, s>>>(h.in.as<double4>(), sys_off + q0, piece,
                                                       h.hist.as<double>() + (size_t)q0 * pieces * 6, ticket + q0,
                                                       g + q0);
      h.launches++;
    }
  } else {
    const int nbp = (int)std::min<long>(4 * 148, (n + TB - 1) / TB);
    h.hist.need((size_t)nbp * 6 * sizeof(double));
    k_bounds<<<nbp, TB, 0, s>>>(h.in.as<double4>(), n, h.hist.as<double>(), g, ctr);
    h.launches++;
  }
  FMM_LAUNCH();

  // the system index takes the key bits above the octant digits
  int sys_bits = 0;
  while ((1ll << sys_bits) < nsys) sys_bits++;
  const int max_levels = std::min(EXAFMM_MAX_LEVEL, (64 - sys_bits) / 3);
  int D = h.key_levels;
  if (D <= 0) {
    long nmax = n;
    if (nsys > 1) {
      nmax = 0;
      for (int q = 0; q < nsys; q++) nmax = std::max<long>(nmax, (long)(h.sys_off_host[q + 1] - h.sys_off_host[q]));
    }
    double ratio = (double)nmax / (double)(h.prm.ncrit > 0 ? h.prm.ncrit : 1);
    D = (int)std::ceil(std::log(std::max(ratio, 1.0)) / std::log(8.0)) + 3;
    D = std::min(std::max(D, 2), max_levels);
  }
  D = std::min(D, max_levels);
  bool zeroed = nsys == 1;  // by k_bounds
  const bool srcf = h.prm.precision == EXAFMM_MIXED && h.prm.dim != 2;
  const size_t nb = (size_t)n;
  h.body_mem.need({{&h.keys[0], nb * 8}, {&h.keys[1], nb * 8}, {&h.vals[0], nb * 4}, {&h.vals[1], nb * 4},
                   {&h.lfirst, nb * 4}, {&h.chain, nb * 4}, {&h.prebase, (nb + 1) * 4}, {&h.perm, nb * 4},
                   {&h.src, nb * sizeof(double4)}, {&h.out, nb * sizeof(double4)},
                   {&h.srcf, srcf ? nb * sizeof(float4) : 0}, {&h.srcp, srcf ? 2 * nb * sizeof(float4) : 0},
                   {&h.body_leaf, h.prm.dim != 2 ? nb * sizeof(int) : 0}});
  for (;;) {
    if (!zeroed) FMM_CUDA(cudaMemsetAsync(ctr, 0, sizeof(DevCounters), s));
    zeroed = false;
    u64 *k = h.keys[0].as<u64>(), *k2 = h.keys[1].as<u64>();
    u32 *v = h.vals[0].as<u32>(), *v2 = h.vals[1].as<u32>();
    k_keys<<<grid_for(n, TB), TB, 0, s>>>(h.in.as<double4>(), n, g, sys_off, nsys, D, k, v);
    h.launches++;
    FMM_LAUNCH();
    radix_sort_pairs(h, k, v, k2, v2, n, 0, 3 * D + sys_bits);
    k_chain<<<grid_for(n, TB), TB, 0, s>>>(k, n, D, h.prm.ncrit, h.lfirst.as<int>(), h.chain.as<int>(), ctr);
    h.launches++;
    FMM_LAUNCH();
    scan_exclusive_int(h, h.chain.as<int>(), h.prebase.as<int>(), n, &ctr->ncells);
    if (h.prm.images > 0)  // the root radius, for the M2L operators of image keys
      FMM_CUDA(cudaMemcpyAsync(&h.root_R0, &g->R0, sizeof(double), cudaMemcpyDeviceToHost, s));
    read_counters(h);
    if (h.hc->overflow) {
      if (D == max_levels)
        throw Error{EXAFMM_ERR_DEPTH, "more than ncrit bodies share a cell at the deepest level (" +
                                          std::to_string(max_levels) + "): coincident bodies?"};
      D = max_levels;
      continue;
    }
    const long C = h.hc->ncells;
    h.ncells = (int)C;
    h.key_levels = D;
    h.nleaves = h.hc->nleaves;
    h.depth = 0;
    h.level_base[0] = 0;
    for (int l = 0; l <= EXAFMM_MAX_LEVEL; l++) {
      h.level_base[l + 1] = h.level_base[l] + h.hc->level_count[l];
      if (h.hc->level_count[l]) h.depth = l;
    }
    // pre-order tables (reuse the idle sort buffers' siblings)
    const long Cp = (C + 3) & ~3L;  // every table starts 16-byte aligned (vector loads in the scans)
    const size_t cb = (size_t)C * sizeof(int);
    h.cell_mem.need({{&h.pre_tmp, Cp * (7 * sizeof(int) + sizeof(double4)) + 256},
                     {&h.ctmp, Cp * (2 * sizeof(u64) + 2 * sizeof(u32) + 4 * sizeof(int)) + 256},
                     {&h.c_begin, cb}, {&h.c_count, cb}, {&h.c_child, cb}, {&h.c_nchild, cb}, {&h.c_parent, cb},
                     {&h.c_level, cb}, {&h.c_pre, cb}, {&h.c_ref, cb}, {&h.c_face, cb}, {&h.leaves, cb},
                     {&h.c_xr, (size_t)C * sizeof(double4)}});
    PreTables t;
    t.xr = h.pre_tmp.as<double4>();
    t.begin = (int *)(t.xr + Cp);
    t.count = t.begin + Cp;
    t.level = t.count + Cp;
    t.parent = t.level + Cp;
    t.nchild = t.parent + Cp;
    t.face = t.nchild + Cp;
    int *owner = t.face + Cp;
    FMM_CUDA(cudaMemsetAsync(t.nchild, 0, C * sizeof(int), s));
    k_cell_owner<<<grid_for(n, TB), TB, 0, s>>>(n, h.chain.as<int>(), h.prebase.as<int>(), owner);
    k_cells<<<grid_for(C, TB), TB, 0, s>>>(k, n, C, D, h.lfirst.as<int>(), owner, h.prebase.as<int>(), g, t);
    h.launches += 2;
    FMM_LAUNCH();

    // 5. BFS order = stable sort of pre-order cells by level
    u64 *lk = h.ctmp.as<u64>(), *lk2 = lk + Cp;
    u32 *lv = (u32 *)(lk2 + Cp), *lv2 = lv + Cp;
    int *bfs_of_pre = (int *)(lv2 + Cp), *is_leaf = bfs_of_pre + Cp, *blockstart = is_leaf + Cp,
        *leafpos = blockstart + Cp;
    k_level_keys<<<grid_for(C, TB), TB, 0, s>>>(t.level, C, lk, lv);
    h.launches++;
    FMM_LAUNCH();
    radix_sort_pairs(h, lk, lv, lk2, lv2, C, 0, 5);
    k_invert<<<grid_for(C, TB), TB, 0, s>>>(lv, C, bfs_of_pre);
    h.launches++;
    BfsCells o{h.c_begin.as<int>(), h.c_count.as<int>(), h.c_child.as<int>(), h.c_nchild.as<int>(),
               h.c_parent.as<int>(), h.c_level.as<int>(), h.c_pre.as<int>(), h.c_face.as<int>(), h.c_xr.as<double4>()};
    k_gather_cells<<<grid_for(C, TB), TB, 0, s>>>(lv, bfs_of_pre, C, t, o, is_leaf);
    h.launches++;
    FMM_LAUNCH();
    // reference numbering, and the leaves
    scan_exclusive_pair(h, t.nchild, blockstart, nullptr, is_leaf, leafpos, nullptr, C);
    k_ref_leaves<<<grid_for(C, TB), TB, 0, s>>>(o, C, blockstart, h.c_ref.as<int>(), is_leaf, leafpos,
                                                h.leaves.as<int>());
    h.launches++;
    FMM_LAUNCH();
    // 6. bodies of each leaf back to input order and gathered (the mixed
    // form's FP32 sources with them)
    k_leaf_order<<<grid_for((long)h.nleaves * 32, TB), TB, 0, s>>>(
        h.leaves.as<int>(), h.nleaves, o.begin, o.count, o.xr, v, h.in.as<double4>(), h.perm.as<int>(),
        h.src.as<double4>(), srcf ? h.srcf.as<float4>() : nullptr, h.srcp.as<float4>(),
        h.prm.dim != 2 ? h.body_leaf.as<int>() : nullptr);
    h.launches++;
    FMM_LAUNCH();
    h.srcf_ready = srcf;
    break;
  }
  // 2D bodies lie at z = 0: the octree is the quadtree (the z digit is the
  // same for every body of a level); its cells go to the plane z = 0
  if (h.prm.dim == 2) flatten_tree_2d(h);
}

}  // namespace fmm
