// Internal definitions of the exafmm_b200 library: the handle, device buffer
// management, error plumbing and the launchers each .cu file provides.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <functional>
#include <initializer_list>
#include <string>
#include <vector>

#include "../../include/exafmm_b200.h"

namespace fmm {

typedef unsigned long long u64;
typedef unsigned int u32;

struct Error {
  int code;
  std::string msg;
};

#define FMM_CUDA(call)                                                                                     \
  do {                                                                                                     \
    cudaError_t e_ = (call);                                                                               \
    if (e_ != cudaSuccess)                                                                                 \
      throw ::fmm::Error{EXAFMM_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_) + " at " +   \
                                              __FILE__ + ":" + std::to_string(__LINE__)};                  \
  } while (0)

#define FMM_LAUNCH()                                                                                       \
  do {                                                                                                     \
    cudaError_t e_ = cudaGetLastError();                                                                   \
    if (e_ != cudaSuccess)                                                                                 \
      throw ::fmm::Error{EXAFMM_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e_) + " at " + \
                                              __FILE__ + ":" + std::to_string(__LINE__)};                  \
  } while (0)

// A device allocation that grows on demand and is kept between evaluations,
// or a piece of a Slab.
struct Buf {
  void *p = nullptr;
  size_t bytes = 0;
  bool piece = false;  // p belongs to a Slab
  template <class T>
  T *as() const { return (T *)p; }
  void need(size_t b) {
    if (b <= bytes) return;
    release();
    allocate(b + b / 4 + 256);
  }
  void allocate(size_t nb) {  // exactly nb bytes, into an empty Buf
    if (cudaMalloc(&p, nb) != cudaSuccess) {
      cudaGetLastError();
      p = nullptr;
      throw Error{EXAFMM_ERR_NOMEM, "cudaMalloc of " + std::to_string(nb) + " bytes failed"};
    }
    bytes = nb;
  }
  void release() {
    if (p && !piece) cudaFree(p);
    p = nullptr;
    bytes = 0;
    piece = false;
  }
};

// One allocation for buffers of one life, which grow together: an allocation
// that the CUDA allocator cannot serve from memory it has mapped costs 0.35 ms
// (tens of ms on a busy host), and the first evaluation of a handle made ten.
struct Slab {
  Buf mem;
  struct Part {
    Buf *buf;
    size_t bytes;
  };
  // Every part with room for its bytes; where one has not, all of them are
  // allocated anew and lose their contents (true).
  bool need(std::initializer_list<Part> parts) {
    bool fits = true;
    size_t total = 0;
    for (const Part &q : parts) {
      fits = fits && q.bytes <= q.buf->bytes;
      total += room(q);
    }
    if (fits) return false;
    size_t size[32];
    int k = 0;
    for (const Part &q : parts) size[k++] = room(q);
    for (const Part &q : parts) q.buf->release();
    mem.release();
    mem.allocate(total);
    char *at = (char *)mem.p;
    k = 0;
    for (const Part &q : parts) {
      q.buf->p = at;
      q.buf->bytes = size[k];
      q.buf->piece = true;
      at += size[k++];
    }
    return true;
  }

 private:
  // a part that is large enough keeps its size, another gets a quarter more
  // than it asks for; whole multiples of 256 bytes
  static size_t room(const Part &q) {
    const size_t b = q.bytes <= q.buf->bytes ? q.buf->bytes : q.bytes + q.bytes / 4;
    return (b + 255) / 256 * 256;
  }
};

// Geometry of the root cell, computed on the device (bounds kernel).
struct RootGeom {
  double X0[3];
  double R0;
};

// Counters written by device code and read once per phase by the host.
struct DevCounters {
  int ncells;          // cells in the tree
  int level_count[EXAFMM_MAX_LEVEL + 2];
  int overflow;        // a cell at the deepest key level still had > ncrit bodies
  int nleaves;
  unsigned long long n_m2l, n_p2p;  // emitted list entries (may exceed capacity)
  unsigned long long frontier[3];   // BFS pair frontier sizes (rotating over the steps)
  int list_overflow;   // an emission or the frontier exceeded its capacity
  int walk_resid;      // M2L entries the walk found without a group key
  int max_m2l_seg, max_p2p_seg;
  int gcounts[4];      // grouped M2L: residual entries, flagged targets, groups, segments
  unsigned long long gfill;
  // largest |scaled multipole| over the possible M2L sources, as the bits of
  // a non-negative double (the FP16 split's power-of-two normalisation)
  unsigned long long m16_max;
  int nghost;  // ghost sources of image entries (mixed form, periodic)
  int op_new;  // group keys without a cached M2L operator
  unsigned bounds_ticket;  // blocks of the bounds kernel that are done (0 between launches)
};

// Per-phase timing slots (CUDA events on the handle stream).
enum Phase { PH_TREE = 0, PH_LISTS, PH_UP, PH_M2L, PH_P2P, PH_DOWN, PH_COUNT };

struct Handle {
  exafmm_params prm{};
  int nterm = 0;
  std::string err;
  cudaStream_t stream = nullptr;
  // a whole evaluation runs the near field on `side` (lower priority), from
  // the lists until the downward pass, beside the far field on `stream`
  cudaStream_t side = nullptr;
  // ... and the upward pass on `aux` (top priority) or `aux_lo` (one level
  // below the list build), beside the dual-tree walk
  cudaStream_t aux = nullptr, aux_lo = nullptr;
  cudaEvent_t fork_ev = nullptr, up_ev = nullptr, lists_ev = nullptr, join_ev = nullptr;
  int64_t launches = 0;

  // bodies; a batch holds nsys independent systems, system q owning input
  // bodies [sys_off[q], sys_off[q+1])
  int64_t n = 0;
  int nsys = 1;
  Buf sys_off;                        // long long [nsys + 1] (device)
  std::vector<int64_t> sys_off_host;
  Buf in;      // double4 (x,y,z,q), caller order
  Slab body_mem;  // the arrays by body that a tree build makes: sort buffers, src, out and the like
  Buf src;     // double4 (x,y,z,q), tree order
  Buf out;     // double4 (p,Fx,Fy,Fz), tree order
  Buf perm;    // int, tree position -> input index
  Buf srcf;    // float4 (x,y,z rel. to leaf centre, q), tree order (mixed form)
  Buf srcp;    // the same in pairs for the near field (srcf.cuh)
  Buf body_leaf;  // int, tree order: the leaf slot (index into `leaves`) of each body (mixed form)
  Buf l2p_f;      // mixed-form L2P: FP32 local expansions of the leaves in leaf units, then their scales
  bool srcf_ready = false;  // srcf matches the current tree
  Buf stage;   // staging for Body records crossing the boundary

  // tree build scratch
  Buf keys[2], vals[2];  // radix sort ping-pong (u64 keys, u32 values)
  Buf lfirst, chain, prebase, scan_tmp, hist;
  int key_levels = 0;

  // tree (BFS order: by level, then first body)
  int ncells = 0, nleaves = 0, depth = 0;
  int level_base[EXAFMM_MAX_LEVEL + 3] = {0};
  Slab cell_mem;  // the tables by cell (c_*, leaves, pre_tmp, ctmp)
  Buf c_begin, c_count, c_child, c_nchild, c_parent, c_level, c_xr, c_pre, c_ref;
  Buf c_face;  // which faces of the root a cell's parent touches (k_cells)
  Buf leaves;  // BFS indices of leaves
  Buf pre_tmp; // preorder tables
  Buf ctmp;    // cell-count scratch (level sort, index maps)
  Buf geom;    // RootGeom
  Buf counters;  // DevCounters
  DevCounters *hc = nullptr;  // host copy (pinned)
  double root_R0 = 0;  // radius of the root cell (one system)

  // lists (CSR by target, BFS indices)
  // what a list build makes, the raw and ordered lists and the group tables,
  // and the operator table
  Slab list_mem;
  Buf frontier[2];
  size_t frontier_cap = 0;
  Buf m2l_raw, p2p_raw;  // emitted (tgt, src|img) pairs
  Buf m2l_key;           // group key of each raw M2L entry (-1: none)
  size_t m2l_cap = 0, p2p_cap = 0;
  Buf m2l_off, m2l_ent, p2p_off, p2p_ent, fill;
  int64_t n_m2l = 0, n_p2p = 0;
  bool m2l_ordered = false;  // m2l_off/m2l_ent built: per-target CSR in the reference's recording order

  // expansions
  Slab exp_mem;  // M and L
  Buf M, L;      // double2 [ncells][nterm]
  Buf shift_ops;   // M2M / L2L harmonics of the unit child offsets (expansions.cu)
  Buf shift_terms; // M2M / L2L term tables (expansions.cu)
  size_t shift_at[4] = {0, 0, 0, 0};  // offsets of the four term tables
  int shift_P = -1;

  // grouped M2L (m2l_group.cu)
  Buf g_mt, g_ekey, g_occ, g_cnt, g_ops, g_tk, g_tile, g_seg, g_tg, g_m16, g_pairs;
  Buf g_gmark;      // ghost slots: marks, their scan, the slot of every ghost
  int g_nghost = 0;  // ghost multipole rows after the cells' in g_m16
  // operator cache: g_optab[group key] is the operator's slot in g_ops (-1:
  // not built), op_count slots built for order op_P, layout op_layout (0:
  // FP64 row blocks, 1: tensor-core FP16 images) and key space op_ks
  Buf g_optab;
  Buf g_new;         // operator slot of each group of the lists, then the keys whose operators are to be built
  long g_groups = 0;  // room for groups in each
  int op_P = -1, op_layout = -1, op_count = 0;
  long op_ks = 0;
  double op_cycle = 0, op_R0 = 0;  // image-key operators: the geometry they were built for
  int op_depth = -1;
  double op_theta = 0;  // tensor-core operators: the acceptance test their scaling is for (TcScale)
  bool g_grouped = false;  // the group tables belong to the current lists
  int g_ntiles = 0, g_ngroups = 0, g_nseg = 0;
  // the grouping of the last grouped M2L (tiles, segments, operator slots),
  // valid for the same lists, P and form: a reevaluation contracts directly
  struct {
    bool valid = false, tcore = false, ordered = false;
    int P = 0, nres = 0;
  } g_plan;
  bool force_direct_m2l = false;  // diagnostic: per-pair direct-form M2L only
  Buf op_scratch;  // single-operator entry points (ops.cu): staged arrays
  // far-image harmonic sums (periodic.cu), kept for the (P, images, cycle)
  // they were made for
  Buf per_harm;
  Buf per_part;  // partial charge sums (the mixed form's root monopole)
  Buf g_gharm;  // harmonics of the ghost shifts, per (image, finer level)
  Buf g_part;   // tensor-core M2L: partial local expansions of tiles split between CTAs
  int nsm = 0;  // streaming multiprocessors of the device
  int per_P = 0, per_images = 0;
  // Ewald: wave list and DFT units of ew_ksize, amplitudes, partial sums
  Buf ew_waves, ew_units, ew_amp, ew_part;
  int ew_ksize = 0, ew_nw = 0, ew_nunits = 0;
  double per_cycle = 0;
  // tile shapes chosen at run time (exafmm_b200_set_tile; the autotuner)
  int tile_m2l_flush = 0;  // tensor-core M2L groups per FP32 accumulator window (0: default)
  int tile_p2p_stage = 0;  // near-field source tile: bodies staged per chunk (0: default)
  // test hook (exafmm_b200_test_stall_tc): the next tensor-core M2L launch
  // waits this long on a barrier nothing arrives at, then times out
  long tc_stall_ns = 0;

  // phase state
  bool have_tree = false, have_lists = false, have_up = false, have_horiz = false, have_down = false;

  // error flags in pinned host memory, set by kernels and checked after each
  // synchronisation: [0] a bounded tensor-core wait ran out, [1] a body or
  // charge handed in is not finite; after the counters' host copy
  int *flags_host = nullptr;

  cudaEvent_t ev[PH_COUNT + 1][2];
  float ms[PH_COUNT + 1] = {0};
  bool ev_ok = false;
};

// ---- launchers (each .cu file) ----
// sort.cu
void scan_exclusive_int(Handle &h, const int *in, int *out, long n, int *total_dev);
void scan_exclusive_pair(Handle &h, const int *in0, int *out0, int *total0, const int *in1, int *out1, int *total1,
                         long n);
void radix_sort_pairs(Handle &h, u64 *&k, u32 *&v, u64 *&k2, u32 *&v2, long n, int lo_bit, int hi_bit);
// tree.cu
void build_tree(Handle &h);
// lists.cu
// near_field (or empty): queues the near field on h.side; called once the P2P
// lists are queued on h.stream, before the host waits for their counts (again
// if the lists overflowed their buffers and are made again)
void build_lists(Handle &h, const std::function<void()> &near_field);
void export_lists(Handle &h, int *m2l_off, int *m2l_src, int *m2l_img, int *p2p_off, int *p2p_src, int *p2p_img);
void order_m2l_lists(Handle &h);
// expansions.cu
void upward_pass(Handle &h, cudaStream_t s);
// before_l2p: an event the stream waits for before L2P (or nullptr)
void downward_pass(Handle &h, cudaStream_t s, cudaEvent_t before_l2p);
// m2l.cu
void m2l_pass(Handle &h);
// m2l_group.cu: group tables from the key and target marks of the lists.
// m2l_group_launch() queues the kernels; once the counters have been read,
// m2l_group_commit() builds the operators of the keys not seen before.
bool m2l_keyed(const Handle &h);       // the M2L is the grouped one: the walk computes and marks keys
bool m2l_groups_raw(const Handle &h);  // the walk's own marks are what the grouped M2L contracts
void m2l_group_launch(Handle &h, long max_groups);
void m2l_group_commit(Handle &h);
void read_counters(Handle &h);  // DevCounters to h.hc, and waits for them (api.cu)
// p2p.cu
void p2p_pass(Handle &h, cudaStream_t s);  // s: h.stream, or h.side once the FP32 sources are made
void make_srcf(Handle &h);
void direct_sum(Handle &h, double4 *targets_pq /*x,y,z,q*/, double4 *out, long nt);
// periodic.cu
void periodic_set_attributes();
void periodic_pass(Handle &h);
void dipole_correction(Handle &h);
// fmm2d.cu: the 2D variants (dim = 2) of the passes above
void flatten_tree_2d(Handle &h);
void upward_pass_2d(Handle &h, cudaStream_t s);
void m2l_pass_2d(Handle &h);
void periodic_pass_2d(Handle &h);
void p2p_pass_2d(Handle &h, cudaStream_t s);
void downward_pass_2d(Handle &h, cudaStream_t s, cudaEvent_t before_l2p);
void direct_sum_2d(Handle &h, double4 *targets, double4 *out, long nt);
void ewald(Handle &h, int parts, int ksize, double alpha, double sigma, double cutoff, double cycle, double *rec_dev,
           long nt);

inline int nterm_of(int P) { return P * (P + 1) / 2; }
inline unsigned grid_for(long n, int block) { return (unsigned)((n + block - 1) / block); }

}  // namespace fmm
