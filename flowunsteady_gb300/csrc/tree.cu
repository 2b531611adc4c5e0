// tree.cu — GPU treecode for U and ∇U (the role of FLOWVPM's UJ_fmm with
// vpm.FMM(p, ncrit, theta), src/FLOWUnsteady_simulation.jl:38,43).
//
// One evaluation runs entirely on the device, in this order:
//   1. bounding cube and 63-bit Morton codes of the particles; radix sort of
//      (code, index) pairs; gather of the state into Morton order and the
//      packed FP32 source records of that order;
//   2. octree built generation by generation: a cell with more than ncrit
//      particles whose codes differ is split at the first 3-bit Morton digit
//      where they differ (so no single-child chains), children are appended
//      with an atomic counter; cells are contiguous ranges of sorted particles;
//   3. upward pass: leaves take their bounding box, largest core and moments
//      (order P) from their particles, then, deepest generation first, parents
//      from their children (box union; moments shifted to the parent centre);
//   4. targets are taken in groups of 64 consecutive particles of the Morton
//      order (compact boxes).  The walk for a group is split over the subtrees of a
//      frontier of at most 73 cells (the leaves of generations 0-1 and generation
//      2), one thread per (subtree, group):
//      a cell s is far for group t when (R_t + R_s) < θ·d and
//      d - R_t - R_s >= sigma_factor·σmax_s (d = distance of the centres, FP32
//      boxes), then it is evaluated from its moments; otherwise its leaves are
//      summed directly, consecutive leaves merged into one range of particles
//      (two passes: count, fill); with local expansions, far cells at least
//      as large as the group go to a list for them;
//   5. local expansions (FP32, P = 4): that list's moments turned into
//      one local expansion of ψ per group (M2L, tree.cuh);
//   6. the direct near field: runs of tiles of a group's near ranges, with the
//      regularised kernels of the direct sum (FP32 pair routines on positions
//      relative to the group's first particle, or FP64);
//   7. the far field: one or two targets per thread over the far list of their
//      group (M2P, tree.cuh); 5 and 7 run beside 6 on streams of their own;
//   8. near field, far field and the local expansion at every target (L2P)
//      added, in the original order.
// The far field uses the singular kernel, as FLOWVPM's nonzero_sigma=false;
// sigma_factor keeps regularised pairs out of it (Gaussian-erf: beyond 7.1 σ
// the kernels agree to FP32 rounding).
#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "capi_internal.h"
#include "tree.cuh"
#include "vpm_device.cuh"

namespace vpm {

constexpr int kMaxGen = 23;        // root + at most 21 Morton digits (+1 spare)
// Device counters: cells, leaves, error flags, finished blocks of the running split, then the first
// cell of every generation (generation g starts at counters[kGenBase + g]).
constexpr int kCntCells = 0, kCntLeaves = 1, kCntFlags = 2, kCntDone = 3, kGenBase = 4;
constexpr int kNumCounters = kGenBase + kMaxGen + 2;
// Target group size (consecutive particles of the Morton order).  32-particle
// groups were measured at N = 1M too: at θ = 0.4 they take 0.131 s instead of
// 0.142 s but lose accuracy (rel-L2 U 5.3e-5, J 1.46e-5 against 4.4e-5, 1.15e-5),
// and at equal accuracy (θ ≈ 0.39) the two sizes take the same time.
constexpr int kTreeBlock = 64;     // threads of the far CTAs = group size
constexpr int kMaxFront = 1 + 8 + 64;   // walk roots: leaves of generations 0-1, generation 2

// ------------------------------------------------------------- workspace --
// Interaction lists of a target group: far cells (M2P), near source ranges, cells of
// its local expansion.
enum ListKind { LIST_FAR = 0, LIST_NEAR = 1, LIST_LOC = 2, kListKinds = 3 };

struct FmmWork {
  int64_t cap = 0;            // particles
  int64_t cell_cap = 0;       // cells (2·cap + 8 bounds any octree of cap points)
  int64_t mom_cells = 0;      // cells the moment buffers hold
  int mom_p = -1;
  int64_t far_cap = 0, near_cap = 0, loc_cap_list = 0;   // interaction list entries
  // particles in Morton order
  uint64_t *codes = nullptr, *codes_alt = nullptr;
  int *idx = nullptr, *perm = nullptr;
  double* sorted = nullptr;   // X 3, Γ 3, σ 1 rows of length cap
  float4* rec = nullptr;      // packed FP32 source records of the sorted particles
  // raw near-field sums, kTreeBlock targets per row, NV rows per near item
  double* near_raw = nullptr;
  size_t near_raw_cap = 0;    // doubles
  double* pot = nullptr;      // far-field U 3, J 9 per sorted particle (FP32 or FP64 rows)
  float* vw = nullptr;        // v_q, w_q rows of the ζ passes in Morton order, FP32
  // cells
  int *lo = nullptr, *hi = nullptr, *child = nullptr, *nchild = nullptr;
  int* skip = nullptr;        // the cell after this one's subtree in Morton order (-1: none)
  double* geom = nullptr;     // per cell: box min x y z, box max x y z, σmax, unused
  double* mom = nullptr;      // per cell: 3·ncoef(P) FP64 moments
  float* momf = nullptr;      // FP32 copy
  int* leaves = nullptr;      // leaf cell ids
  int* counters = nullptr;    // see kCntCells .. kGenBase
  int64_t meta_cap = 0;       // (group, frontier cell) walk slots
  float4* ggeom = nullptr;    // target-group boxes (centre, radius), FP32
  float4* cgeom = nullptr;    // walk records, two per cell (see write_cell_geom)
  int* front = nullptr;       // frontier cells (walk roots)
  unsigned long long* pairs = nullptr;   // [0] near source pairs, [1] far (target, cell) pairs
  double* box = nullptr;      // bounding cube: min x y z, size
  double* box_part = nullptr; // per-block min/max partials
  // interaction lists, one per target group, group g's at gbase[q][g] .. + gtot[q][g]
  int* wcnt = nullptr;        // per (frontier cell, group): kListKinds counts, then offsets in the group
  int* gtot = nullptr;        // kListKinds + 1 rows: list lengths; near sources
  int* gbase = nullptr;       // kListKinds + 1 rows: list starts; first near item
  int* gorder = nullptr;      // groups by decreasing far list
  long long* totals = nullptr;   // see group_scan_kernel
  int* far_list = nullptr;    // far cell ids per target group (M2P at every target)
  int2* near_list = nullptr;  // near source ranges [x, y) per target group
  int* loc_list = nullptr;    // far cell ids per target group taken by its local expansion
  // far field [0] and local expansions [1], beside the near field
  cudaStream_t aux[2] = {nullptr, nullptr};
  cudaEvent_t fork = nullptr, join[2] = {nullptr, nullptr};
  void* cub_tmp = nullptr;
  size_t cub_bytes = 0;
  int h_counters[kNumCounters];
  // statistics of the last evaluation
  int64_t last_cells = 0, last_leaves = 0, last_groups = 0, last_far = 0, last_near = 0;
  int64_t last_n = -1;
  int64_t last_items = 0;    // near items
  unsigned long long h_pairs[3] = {0, 0, 0};
  float* loc = nullptr;       // per target group: 3·ncoef(Q) local coefficients
  int64_t loc_cap = 0;
};

void fmm_free(FmmWork* w) {
  if (!w) return;
  void* ptrs[] = {w->codes, w->codes_alt, w->idx, w->perm, w->sorted, w->rec, w->near_raw, w->pot,
                  w->vw, w->lo, w->hi, w->child, w->nchild, w->skip, w->geom, w->mom, w->momf,
                  w->leaves, w->ggeom, w->cgeom, w->front, w->pairs, w->counters, w->box,
                  w->box_part, w->wcnt, w->gtot, w->gbase, w->gorder, w->totals, w->far_list,
                  w->near_list, w->cub_tmp, w->loc, w->loc_list};
  if (w->fork) cudaEventDestroy(w->fork);
  for (int k = 0; k < 2; ++k) {
    if (w->aux[k]) cudaStreamDestroy(w->aux[k]);
    if (w->join[k]) cudaEventDestroy(w->join[k]);
  }
  for (void* p : ptrs) cudaFree(p);
  delete w;
}

// ------------------------------------------------------ bounding cube, codes --
constexpr int kBoxBlocks = 256;

__global__ void box_partial_kernel(int64_t n, const double* __restrict__ X, int64_t ld,
                                   double* part) {
  __shared__ double s[6][256];
  double v[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double x = X[d * ld + i];
      v[d] = fmin(v[d], x);
      v[3 + d] = fmax(v[3 + d], x);
    }
  }
#pragma unroll
  for (int d = 0; d < 6; ++d) s[d][threadIdx.x] = v[d];
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        s[d][threadIdx.x] = fmin(s[d][threadIdx.x], s[d][threadIdx.x + o]);
        s[3 + d][threadIdx.x] = fmax(s[3 + d][threadIdx.x], s[3 + d][threadIdx.x + o]);
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int d = 0; d < 6; ++d) part[blockIdx.x * 6 + d] = s[d][0];
}

// One block of kBoxBlocks threads, one per partial box.
__global__ void box_final_kernel(const double* part, int nblocks, double* box) {
  __shared__ double s[6][kBoxBlocks];
  const int t = threadIdx.x;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    s[d][t] = t < nblocks ? part[t * 6 + d] : INFINITY;
    s[3 + d][t] = t < nblocks ? part[t * 6 + 3 + d] : -INFINITY;
  }
  __syncthreads();
  for (int o = kBoxBlocks / 2; o > 0; o >>= 1) {
    if (t < o) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        s[d][t] = fmin(s[d][t], s[d][t + o]);
        s[3 + d][t] = fmax(s[3 + d][t], s[3 + d][t + o]);
      }
    }
    __syncthreads();
  }
  if (t == 0) {
    const double size = fmax(fmax(s[3][0] - s[0][0], s[4][0] - s[1][0]), s[5][0] - s[2][0]);
    box[0] = s[0][0];
    box[1] = s[1][0];
    box[2] = s[2][0];
    box[3] = size > 0 ? size * (1.0 + 1e-9) : 1.0;
  }
}

// Spread the low 21 bits of v to every third bit (Morton interleaving).
__device__ __forceinline__ uint64_t spread3(uint64_t x) {
  x &= 0x1fffffull;
  x = (x | x << 32) & 0x1f00000000ffffull;
  x = (x | x << 16) & 0x1f0000ff0000ffull;
  x = (x | x << 8) & 0x100f00f00f00f00full;
  x = (x | x << 4) & 0x10c30c30c30c30c3ull;
  x = (x | x << 2) & 0x1249249249249249ull;
  return x;
}

__global__ void morton_kernel(int64_t n, const double* __restrict__ X, int64_t ld,
                              const double* __restrict__ box, uint64_t* codes, int* idx) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double scale = double(1 << 21) / box[3];
  uint64_t q[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double t = floor((X[d * ld + i] - box[d]) * scale);
    q[d] = uint64_t(fmin(fmax(t, 0.0), double((1 << 21) - 1)));
  }
  codes[i] = spread3(q[0]) << 2 | spread3(q[1]) << 1 | spread3(q[2]);
  idx[i] = int(i);
}

// Sorted FP64 state (X 3, Γ 3, σ 1 rows of length ldw) in Morton order.
__global__ void gather_kernel(int64_t n, const int* __restrict__ perm, const double* __restrict__ X,
                              const double* __restrict__ G, const double* __restrict__ S,
                              int64_t ld, double* sorted, int64_t ldw) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t j = perm[i];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    sorted[d * ldw + i] = X[d * ld + j];
    sorted[(3 + d) * ldw + i] = G[d * ld + j];
  }
  sorted[6 * ldw + i] = S[j];
}

// ------------------------------------------------------------- tree build --
__global__ void tree_init_kernel(int64_t n, int* lo, int* hi, int* skip, int* counters) {
  lo[0] = 0;
  hi[0] = int(n);
  skip[0] = -1;
  counters[kCntCells] = 1;
  counters[kCntLeaves] = 0;
  counters[kCntFlags] = 0;
  counters[kCntDone] = 0;
  counters[kGenBase + 0] = 0;   // generation 0 is the root
  counters[kGenBase + 1] = 1;
}

__device__ __forceinline__ int lower_bound_code(const uint64_t* codes, int lo, int hi,
                                                uint64_t key) {
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (codes[mid] < key) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Split or close the cells of generation g, eight lanes per cell: lane v finds
// where Morton digit v begins, so that the seven binary searches of a cell (16
// to 20 dependent loads each) run side by side.  One thread per cell walked them
// one after another: 38 µs a generation at N = 60,000 against 12 µs.  The last
// block to finish closes generation g + 1, which ends where the cells appended
// here end (a launch of its own before).
__global__ void tree_split_kernel(int g, int ncrit, int64_t cell_cap, const uint64_t* __restrict__ codes,
                                  int* lo, int* hi, int* child, int* nchild, int* skip, int* leaves,
                                  int* counters) {
  const int begin = counters[kGenBase + g], end = counters[kGenBase + g + 1];
  const int lane = threadIdx.x & 31, v = lane & 7, base = lane & ~7;
  const int per = int(blockDim.x) / 8;
  for (int c0 = begin + int(blockIdx.x) * per; c0 < end; c0 += int(gridDim.x) * per) {
    const int cell = c0 + int(threadIdx.x) / 8;
    const bool valid = cell < end;
    int a = 0, b = 0;
    uint64_t first = 0, last = 0;
    if (valid) {
      a = lo[cell];
      b = hi[cell];
      first = codes[a];
      last = codes[b - 1];
    }
    const bool split = valid && b - a > ncrit && first != last;
    int bound = a;
    if (split && v > 0) {
      const int bit = 63 - __clzll((long long)(first ^ last));   // highest differing bit
      const int shift = (bit / 3) * 3;                            // its Morton digit
      const uint64_t prefix = first & ~((uint64_t(8) << shift) - 1);
      bound = lower_bound_code(codes, a, b, prefix | (uint64_t(v) << shift));
    }
    int next = __shfl_down_sync(0xffffffffu, bound, 1);
    if (v == 7) next = b;
    const bool some = split && next > bound;
    const unsigned mask = (__ballot_sync(0xffffffffu, some) >> base) & 0xffu;
    const int nc = __popc(mask);
    int first_child = 0;
    if (valid && v == 0) {
      if (split) first_child = atomicAdd(&counters[kCntCells], nc);
      else leaves[atomicAdd(&counters[kCntLeaves], 1)] = cell;
    }
    first_child = __shfl_sync(0xffffffffu, first_child, base);
    const bool fits = split && first_child + nc <= cell_cap;
    if (some && fits) {
      const int k = first_child + __popc(mask & ((1u << v) - 1u));
      lo[k] = bound;
      hi[k] = next;
      skip[k] = k + 1 < first_child + nc ? k + 1 : skip[cell];
    }
    if (valid && v == 0) {
      child[cell] = fits ? first_child : -1;
      nchild[cell] = fits ? nc : 0;
      if (split && !fits) atomicOr(&counters[kCntFlags], 1);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&counters[kCntDone], 1) == int(gridDim.x) - 1) {
      counters[kGenBase + g + 2] = atomicAdd(&counters[kCntCells], 0);
      counters[kCntDone] = 0;
    }
  }
}

// ------------------------------------------------------------ upward pass --
// Cell geometry record (8 doubles): box min x y z, box max x y z, σmax, unused.
constexpr int kGeom = 8;

__device__ __forceinline__ void cell_centre(const double* g, double& cx, double& cy, double& cz,
                                            double& r) {
  cx = 0.5 * (g[0] + g[3]);
  cy = 0.5 * (g[1] + g[4]);
  cz = 0.5 * (g[2] + g[5]);
  const double ex = 0.5 * (g[3] - g[0]), ey = 0.5 * (g[4] - g[1]), ez = 0.5 * (g[5] - g[2]);
  r = sqrt(ex * ex + ey * ey + ez * ez);
}

// Smallest and largest of a double over the warp, on the order-preserving integer
// image of its bits: FP64 comparisons would queue on GB300's FP64 pipe (about two
// operations per SM and cycle).
__device__ __forceinline__ long long order_key(double x) {
  const long long b = __double_as_longlong(x);
  return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ double order_value(long long k) {
  return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffll));
}
__device__ __forceinline__ bool is_nan(double x) {
  return (__double_as_longlong(x) & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
}
__device__ __forceinline__ long long warp_min_key(long long k) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) k = min(k, __shfl_xor_sync(0xffffffffu, k, o));
  return k;
}
__device__ __forceinline__ long long warp_max_key(long long k) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) k = max(k, __shfl_xor_sync(0xffffffffu, k, o));
  return k;
}

// Bounding box of the particles [lo, hi) of the sorted rows, by one warp; every
// lane gets it in g[0..5], and the largest core (sorted row 6) in g[6].
__device__ __forceinline__ void warp_box(const double* __restrict__ sorted, int64_t ldw, int64_t lo,
                                         int64_t hi, double (&g)[8]) {
  long long mn[3], mx[3], ms = order_key(0.0);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    mn[d] = order_key(INFINITY);
    mx[d] = order_key(-INFINITY);
  }
  for (int64_t i = lo + (threadIdx.x & 31); i < hi; i += 32) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double x = sorted[d * ldw + i];
      if (is_nan(x)) continue;   // a diverged particle does not widen the box
      const long long k = order_key(x);
      mn[d] = min(mn[d], k);
      mx[d] = max(mx[d], k);
    }
    const double sg = sorted[6 * ldw + i];
    if (!is_nan(sg)) ms = max(ms, order_key(sg));
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    g[d] = order_value(warp_min_key(mn[d]));
    g[3 + d] = order_value(warp_max_key(mx[d]));
  }
  g[6] = order_value(warp_max_key(ms));
  g[7] = 0.0;
}

// Exponents (a, b, c) of every multi-index |k| <= 6 in graded order, packed as
// a | b << 4 | c << 8 (computed at compile time).
struct MidxTable {
  short v[ncoef(6)];
};
constexpr MidxTable make_midx_table() {
  MidxTable t{};
  for (int n = 0; n <= 6; ++n)
    for (int a = n; a >= 0; --a)
      for (int b = n - a; b >= 0; --b) t.v[midx(a, b, n - a - b)] = short(a | b << 4 | (n - a - b) << 8);
  return t;
}
__constant__ MidxTable c_midx = make_midx_table();
__constant__ double c_fact[7] = {1, 1, 2, 6, 24, 120, 720};
__constant__ double c_ifact[7] = {1, 1, 0.5, 1.0 / 6, 1.0 / 24, 1.0 / 120, 1.0 / 720};

// What the upward kernels write for a cell: its box, FP64 moments, their FP32 copy
// (momf, where given) and its walk record.
struct CellOut {
  double* geom;
  double* mom;
  float* momf;
  float4* walk;
  const int* skip;
};

// Walk record of a cell, two float4 read together by the traversal:
//   rec[2c]     = centre x, y, z and radius (FP32, inflated by 1e-6 of the
//                 coordinates' magnitude so that rounding cannot shrink it);
//   rec[2c + 1] = largest core (FP32), then as integer bits: the first child
//                 (or the first particle of a leaf), the end of a leaf's
//                 particle range (-1: not a leaf), and the cell after this one's
//                 subtree in Morton order (-1: none).
__device__ __forceinline__ void write_cell_geom(const CellOut& o, int cell, const double (&g)[8],
                                                int first, int end) {
  double* gc = o.geom + int64_t(cell) * kGeom;
#pragma unroll
  for (int d = 0; d < 8; ++d) gc[d] = g[d];
  double cx, cy, cz, r;
  cell_centre(g, cx, cy, cz, r);
  const double pad = 1e-6 * (fabs(cx) + fabs(cy) + fabs(cz) + r);
  o.walk[2 * int64_t(cell)] = make_float4(float(cx), float(cy), float(cz), float(r + pad));
  o.walk[2 * int64_t(cell) + 1] = make_float4(float(g[6]), __int_as_float(first),
                                              __int_as_float(end), __int_as_float(o.skip[cell]));
}

// The upward pass is FP64 sums of a few thousand terms per cell, on a pipe that
// retires about two of them per SM and cycle: what matters is that a cell's sums
// run side by side and not as one thread's chain.  One thread per (cell, component)
// took 1.66 ms of a treecode evaluation at N = 60,000 (eight launches of 160 to
// 300 µs, each the length of one chain); these two kernels take 0.26 ms (leaves
// 51 µs, a generation of parents 22 to 61 µs).
//
// Leaves, one warp each: lane = particle forms the box and the monomials
// (y - c)^k, then lane = (component, k) sums Γ^m (y - c)^k over the particles in
// their order.
constexpr int kLeafWarps = 4;
template <int P>
__global__ void __launch_bounds__(32 * kLeafWarps) tree_leaf_kernel(
    int nleaves, const int* __restrict__ leaves, const int* __restrict__ lo,
    const int* __restrict__ hi, const double* __restrict__ sorted, int64_t ldw, CellOut out) {
  constexpr int NC = ncoef(P), ROUNDS = (3 * NC + 31) / 32;
  constexpr int CH = P > 4 ? 16 : 32;   // particles staged at a time
  __shared__ double s_pw[kLeafWarps][CH][NC], s_g[kLeafWarps][CH][3];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int l = int(blockIdx.x) * kLeafWarps + wid;
  if (l >= nleaves) return;
  const int cell = leaves[l], a = lo[cell], b = hi[cell];
  double g[8];
  warp_box(sorted, ldw, a, b, g);
  if (lane == 0) write_cell_geom(out, cell, g, a, b);
  double cx, cy, cz, rad;
  cell_centre(g, cx, cy, cz, rad);
  double acc[ROUNDS];
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) acc[r] = 0.0;
  for (int i0 = a; i0 < b; i0 += CH) {
    const int cnt = min(CH, b - i0);
    __syncwarp();
    if (lane < cnt) {
      const int i = i0 + lane;
      double pw[NC];
      monomials<P, double>(sorted[i] - cx, sorted[ldw + i] - cy, sorted[2 * ldw + i] - cz, pw);
#pragma unroll
      for (int k = 0; k < NC; ++k) s_pw[wid][lane][k] = pw[k];
#pragma unroll
      for (int m = 0; m < 3; ++m) s_g[wid][lane][m] = sorted[(3 + m) * ldw + i];
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
      const int e = lane + 32 * r;
      if (e < 3 * NC) {
        const int m = e / NC, k = e - m * NC;
        for (int i = 0; i < cnt; ++i) acc[r] += s_g[wid][i][m] * s_pw[wid][i][k];
      }
    }
  }
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    const int e = lane + 32 * r;
    if (e < 3 * NC) {
      out.mom[int64_t(cell) * 3 * NC + e] = acc[r];
      if (out.momf) out.momf[int64_t(cell) * 3 * NC + e] = float(acc[r]);
    }
  }
}

// Parents of generation g from their children (of later generations, already
// done), one CTA per cell.  The moment shift
//   M_k/k! = Σ_{children q} Σ_{j<=k} (M_j^q/j!) (c_q - c)^{k-j}/(k-j)!
// runs with one thread per (coefficient slot, child slot); kUpSlots child slots
// are summed in order at the end.
constexpr int kUpSlots = 4, kUpThreads = 128;
template <int P>
__global__ void __launch_bounds__(kUpThreads * kUpSlots) tree_upward_kernel(
    int g, int* counters, const int* __restrict__ child, const int* __restrict__ nchild,
    CellOut out) {
  constexpr int NC = ncoef(P), NE = 3 * NC;
  __shared__ double s_m[8][NE], s_t[8][NC], s_box[8][8], s_geom[8];
  __shared__ double s_sum[kUpSlots - 1][NE];
  const int tid = threadIdx.x, slot = tid / kUpThreads, tl = tid - slot * kUpThreads;
  const int begin = counters[kGenBase + g], end = counters[kGenBase + g + 1];
  const int total = counters[kCntCells];
  for (int cell = begin + int(blockIdx.x); cell < end; cell += int(gridDim.x)) {
    int nc = nchild[cell];
    const int ch = child[cell];
    if (nc == 0) continue;   // a leaf: done by tree_leaf_kernel
    if (nc > 8 || ch < 0 || ch + nc > total) {   // outside the tree: record, skip
      if (tid == 0) atomicOr(&counters[kCntFlags], 32);
      continue;
    }
    __syncthreads();   // the previous cell is done with shared memory
    if (tid < 8 * nc) s_box[tid >> 3][tid & 7] = out.geom[int64_t(ch + (tid >> 3)) * kGeom + (tid & 7)];
    for (int e = tid; e < nc * NE; e += blockDim.x) {
      const int q = e / NE, r = e - q * NE;
      const int x = c_midx.v[r % NC];
      s_m[q][r] = out.mom[int64_t(ch) * NE + e] *
                  (c_ifact[x & 15] * c_ifact[(x >> 4) & 15] * c_ifact[x >> 8]);
    }
    __syncthreads();
    if (tid < 7) {
      double v = s_box[0][tid];
      for (int q = 1; q < nc; ++q) {
        const double u = s_box[q][tid];
        v = (tid < 3 ? order_key(u) < order_key(v) : order_key(u) > order_key(v)) ? u : v;
      }
      s_geom[tid] = v;
    }
    if (tid == 7) s_geom[7] = 0.0;
    __syncthreads();
    // (c_q - c)^k / k!
    for (int e = tid; e < nc * NC; e += blockDim.x) {
      const int q = e / NC, k = e - q * NC, x = c_midx.v[k];
      double f = 1.0;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const int ex = (x >> (4 * d)) & 15;
        const double dd = 0.5 * (s_box[q][d] + s_box[q][3 + d]) - 0.5 * (s_geom[d] + s_geom[3 + d]);
        double w = c_ifact[ex];
        for (int i = 0; i < ex; ++i) w *= dd;
        f *= w;
      }
      s_t[q][k] = f;
    }
    if (tid == 0) {
      double gg[8];
#pragma unroll
      for (int d = 0; d < 8; ++d) gg[d] = s_geom[d];
      write_cell_geom(out, cell, gg, ch, -1);
    }
    __syncthreads();
    for (int e0 = 0; e0 < NE; e0 += kUpThreads) {
      const int e = e0 + tl;
      double acc = 0.0;
      int x = 0;
      if (e < NE) {
        const int m = e / NC;
        x = c_midx.v[e - m * NC];
        const int a = x & 15, b = (x >> 4) & 15, c = x >> 8;
        for (int q = slot; q < nc; q += kUpSlots) {
          const double* mq = s_m[q] + m * NC;
          const double* tq = s_t[q];
          for (int ja = 0; ja <= a; ++ja)
            for (int jb = 0; jb <= b; ++jb)
              for (int jc = 0; jc <= c; ++jc)
                acc += tq[midx(a - ja, b - jb, c - jc)] * mq[midx(ja, jb, jc)];
        }
        if (slot > 0) s_sum[slot - 1][e] = acc;
      }
      __syncthreads();
      if (slot == 0 && e < NE) {
#pragma unroll
        for (int q = 0; q < kUpSlots - 1; ++q) acc += s_sum[q][e];
        acc *= c_fact[x & 15] * c_fact[(x >> 4) & 15] * c_fact[x >> 8];
        out.mom[int64_t(cell) * NE + e] = acc;
        if (out.momf) out.momf[int64_t(cell) * NE + e] = float(acc);
      }
    }
  }
}

// -------------------------------------------------------------- traversal --
// Targets are taken in groups of kTreeBlock consecutive particles of the Morton
// order (the last one shorter): compact boxes, full CTAs.  Each group's box
// (centre, radius) goes to an FP32 record for the walk, by one warp per group;
// radii are inflated by 1e-6 of the coordinates' magnitude so that rounding
// cannot shrink them.
__global__ void group_geom_kernel(int64_t n, const double* __restrict__ sorted, int64_t ldw,
                                  float4* ggeom) {
  const int64_t g = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32;
  const int64_t a = g * kTreeBlock;
  if (a >= n) return;
  double bx[8];
  warp_box(sorted, ldw, a, a + kTreeBlock < n ? a + kTreeBlock : n, bx);
  double cx, cy, cz, r;
  cell_centre(bx, cx, cy, cz, r);
  const double pad = 1e-6 * (fabs(cx) + fabs(cy) + fabs(cz) + r);
  if ((threadIdx.x & 31) == 0) ggeom[g] = make_float4(float(cx), float(cy), float(cz), float(r + pad));
}

// One thread per (frontier cell j, target group g), t = j·ngroups + g: the walk of
// the subtree below frontier cell j for group g, in Morton order.  A warp holds 32
// neighbouring groups on one subtree, so its lanes visit nearly the same cells, and
// each cell's record leads to both the cell inside it and the one after it (no
// stack).  FILL = false counts the far cells, near source ranges, local-expansion
// cells and near sources; FILL = true writes them at the scanned offsets (same
// order); a group's lists are the concatenation over j.  Near leaves that continue
// the previous near range in Morton order extend it.
// With one lane per subtree of one group and a stack of cells in local memory the
// two passes took 205 + 209 µs at N = 60,000; this form takes 133 + 144 µs.
template <bool FILL>
__global__ void traverse_kernel(int ngroups, int nfront, const int* __restrict__ front,
                                const float4* __restrict__ ggeom, const float4* __restrict__ walk,
                                float theta, float sfac, int mark_local, int* wcnt, int* nsrc,
                                const int* __restrict__ gbase, int* far_list, int2* near_list,
                                int* loc_list, int* counters, int ncells) {
  const int64_t nwalk = int64_t(ngroups) * nfront;
  const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= nwalk) return;
  const int g = int(t % ngroups);
  const float4 tg = ggeom[g];
  int cf = 0, cn = 0, cl = 0, cs = 0, last_hi = -1;
  int of = 0, on = 0, ol = 0;
  if (FILL) {
    of = gbase[g] + wcnt[t];
    on = gbase[ngroups + g] + wcnt[nwalk + t];
    if (mark_local) ol = gbase[2 * ngroups + g] + wcnt[2 * nwalk + t];
  }
  int s = front[t / ngroups];
  int stop = -1;
  for (int visits = 0; s != stop || visits == 0; ++visits) {
    if (s < 0 || s >= ncells || visits >= ncells) {   // cannot happen: the walk left the tree
      atomicOr(&counters[kCntFlags], 16);
      break;
    }
    const float4 cs4 = walk[2 * s], ck = walk[2 * s + 1];
    const int first = __float_as_int(ck.y), end = __float_as_int(ck.z), next = __float_as_int(ck.w);
    if (visits == 0) stop = next;
    const float dx = tg.x - cs4.x, dy = tg.y - cs4.y, dz = tg.z - cs4.z;
    const float d = sqrtf(dx * dx + dy * dy + dz * dz);
    if (tg.w + cs4.w < theta * d && d - tg.w - cs4.w >= sfac * ck.x) {
      // Cells at least as large as the group go to its local expansion.
      if (mark_local && cs4.w >= tg.w) {
        if (FILL) loc_list[ol + cl] = s;
        ++cl;
      } else {
        if (FILL) far_list[of + cf] = s;
        ++cf;
      }
    } else if (end >= 0) {   // a leaf
      if (cn > 0 && first == last_hi) {
        if (FILL) near_list[on + cn - 1].y = end;
      } else {
        if (FILL) near_list[on + cn] = make_int2(first, end);
        ++cn;
      }
      cs += end - first;
      last_hi = end;
    } else {
      s = first;
      continue;
    }
    s = next;
  }
  if (!FILL) {
    wcnt[t] = cf;
    wcnt[nwalk + t] = cn;
    wcnt[2 * nwalk + t] = cl;
    nsrc[t] = cs;
  }
}

// Lengths of group g's lists and its near sources (gtot rows), and in wcnt the
// offset of every subtree's part in the group's list: one warp per group, lane =
// frontier cell.
__global__ void group_lists_kernel(int ngroups, int nfront, int* wcnt, const int* __restrict__ nsrc,
                                   int* gtot) {
  const int g = int((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32), lane = threadIdx.x & 31;
  if (g >= ngroups) return;
  const int64_t nwalk = int64_t(ngroups) * nfront;
  for (int q = 0; q <= kListKinds; ++q) {
    int carry = 0;
    for (int j0 = 0; j0 < nfront; j0 += 32) {
      const int j = j0 + lane;
      const int64_t t = int64_t(j) * ngroups + g;
      const int v = j >= nfront ? 0 : q < kListKinds ? wcnt[q * nwalk + t] : nsrc[t];
      int incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
      }
      if (j < nfront && q < kListKinds) wcnt[q * nwalk + t] = carry + incl - v;
      carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) gtot[int64_t(q) * ngroups + g] = carry;
  }
}

// Starts of the groups' lists and of their near items, and the groups by decreasing
// far list (within 64 steps of the longest), by one block.
//   totals[0..2]  list lengths;  totals[3]  near items;  totals[4]  tiles of an item;
//   totals[5]     near sources over all groups.
// Near items are runs of whole fold groups (kItemTiles tiles) of one group's near
// tiles, of equal length: the shortest for which the field has about kNearItems of
// them beside one per group.  gbase row 3 holds each group's first item.
constexpr int kScanThreads = 1024;
constexpr int kItemTiles = 16;               // tiles between two folds (near_tile_kernel)
constexpr long long kNearItems = 16 * 3 * 152;   // about 16 waves of near CTAs

__device__ __forceinline__ int near_tiles(int sources, int ranges) {
  return sources / 128 + (ranges + 127) / 128;   // at most: every 128 ranges end a tile
}

__global__ void __launch_bounds__(kScanThreads) group_scan_kernel(int ngroups, const int* __restrict__ gtot,
                                                                 int* gbase, int* gorder,
                                                                 int whole_groups, long long* totals) {
  __shared__ long long s_part[32], s_carry[4];
  __shared__ int s_max, s_hist[64];
  __shared__ long long s_tiles;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (tid == 0) s_max = 0;
  if (tid < 64) s_hist[tid] = 0;
  if (tid < 4) s_carry[tid] = 0;
  __syncthreads();
  long long tiles = 0, srcs = 0;
  int fmax_ = 0;
  for (int g = tid; g < ngroups; g += kScanThreads) {
    const int n = gtot[int64_t(kListKinds) * ngroups + g];
    srcs += n;
    tiles += near_tiles(n, gtot[int64_t(LIST_NEAR) * ngroups + g]);
    fmax_ = max(fmax_, gtot[g]);
  }
  auto block_sum = [&](long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) s_part[wid] = v;
    __syncthreads();
    long long r = 0;
    for (int w = 0; w < kScanThreads / 32; ++w) r += s_part[w];
    return r;
  };
  tiles = block_sum(tiles);
  srcs = block_sum(srcs);
  atomicMax(&s_max, fmax_);
  if (tid == 0) {
    const long long want = (tiles + kNearItems - 1) / kNearItems;
    s_tiles = whole_groups ? (1ll << 40) : max(1ll, (want + kItemTiles - 1) / kItemTiles) * kItemTiles;
    totals[4] = s_tiles;
    totals[5] = srcs;
  }
  __syncthreads();
  const long long per = s_tiles;
  const int fmx = s_max;
  for (int g0 = 0; g0 < ngroups; g0 += kScanThreads) {
    const int g = g0 + tid;
    const bool live = g < ngroups;
    const int far = live ? gtot[g] : 0;
    const int rng = live ? gtot[int64_t(LIST_NEAR) * ngroups + g] : 0;
    const int loc = live ? gtot[int64_t(LIST_LOC) * ngroups + g] : 0;
    const int src = live ? gtot[int64_t(kListKinds) * ngroups + g] : 0;
    const long long nt = near_tiles(src, rng);
    const long long vals[4] = {far, rng, loc, live ? max(1ll, (nt + per - 1) / per) : 0ll};
    if (live) atomicAdd(&s_hist[63 - int(int64_t(far) * 63 / max(fmx, 1))], 1);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      long long incl = vals[q];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const long long u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
      }
      __syncthreads();
      if (lane == 31) s_part[wid] = incl;
      __syncthreads();
      long long before = s_carry[q], all = 0;
      for (int w = 0; w < kScanThreads / 32; ++w) {
        if (w < wid) before += s_part[w];
        all += s_part[w];
      }
      if (live) gbase[int64_t(q) * ngroups + g] = int(before + incl - vals[q]);
      __syncthreads();
      if (tid == 0) s_carry[q] += all;
    }
  }
  __syncthreads();
  if (tid < 4) totals[tid] = s_carry[tid];
  if (tid == 0) {   // starts of the order's steps
    int at = 0;
    for (int b = 0; b < 64; ++b) {
      const int n = s_hist[b];
      s_hist[b] = at;
      at += n;
    }
  }
  __syncthreads();
  for (int g = tid; g < ngroups; g += kScanThreads)
    gorder[atomicAdd(&s_hist[63 - int(int64_t(gtot[g]) * 63 / max(fmx, 1))], 1)] = g;
}

// --------------------------------------------------------------- near field --
// Groups' near fields differ a hundredfold (a group that straddles a jump of the
// Morton curve has a box as large as the wake and nearly every particle near it), so
// the work is dealt in items of equal length (group_scan_kernel) and not in groups:
// with one CTA per group the longest one, 60,000 sources at N = 60,000 against
// 11,000 on average, set the launch's 2.0 ms; items take 1.11 ms.  One CTA of kNearThreads threads per
// item: its run of the tiles of the group's near source ranges, with the pair
// routines of the direct sum (vpm_device.cuh) on T targets per thread:
//   - the group's kTreeBlock targets are held as TQ = kTreeBlock/T target sets of T targets
//     (target t = tq + TQ·k), each set by SL = kNearThreads/TQ threads, one per
//     source slice;
//   - the concatenated near ranges are staged kNearThreads sources at a time
//     (positions relative to the group's first particle, from the packed
//     records); slice s takes the staged sources s, s + SL, s + 2·SL, ..., so
//     every thread reads each of its sources with broadcast 16-byte loads and
//     applies it to T targets (packed FP32 pairs for T even);
//   - a tile is always full: slots past the sources hold a padding source at
//     1e18 with zero strength, which adds exactly 0 (its q and p underflow),
//     so the warp votes of the pair routines see the same trip count on every
//     lane;
//   - FP32 sums are folded into (hi, lo) pairs (Knuth's TwoSum) every
//     kNearFoldSources sources of a thread; the epilogue forms every target's raw
//     sums in FP64 as the slices' (hi + lo) in slice order.
// Raw sums of target t of item i go to raw[(i·NV + k)·kTreeBlock + t]; the reader adds
// a group's items in order.  An item starts at a fold, so that the FP32 sums are
// those of one CTA that walks the whole group:
//   PASS_UJ    U 3, A 9, W 3 (Gaussian-erf A sums hold p/(-3), as the direct
//              pass's do);
//   PASS_UJD   those plus DA 9, DW 3 (Gaussian-erf: Dq, Dp vanish beyond the
//              near field's 7.1σ to FP32 significance);
//   PASS_ZETA  Ω 3, V 3; PASS_ZETAD also DΩ 3, DV 3 (Gaussian-erf: ζ likewise),
//              with v_q (and w_q) taken from vw rows of the Morton order.
// Coincident pairs are dropped: the Winckelmans and ζ routines run masked,
// and the Gaussian-erf U/J routines drop them in their series branch.
constexpr int kNearThreads = 128;
constexpr float kNearPadX = 1e18f;
constexpr int kNearFoldSources = 256;   // sources a thread sums in FP32 between folds

template <int PASS>
struct NearShape {
  // Targets per thread.  U/J: four, at three CTAs per SM (168 registers, of
  // which the pass spills 192 bytes; measured at N = 1M it is still 4 % faster
  // than two targets at four CTAs).  U/J + DJ holds 27 sums per target: two.
  // The ζ passes (6 or 12 sums): four.
  static constexpr int T = PASS == PASS_UJD ? 2 : 4;
  static constexpr int TQ = kTreeBlock / T;
  static constexpr int SL = kNearThreads / TQ;
  static constexpr int NV = nval_of(PASS);
  static constexpr bool UJ = PASS == PASS_UJ || PASS == PASS_UJD;
  static constexpr int QUADS = UJ ? 2 : (PASS == PASS_ZETA ? 3 : 4);
  static constexpr size_t kQuadBytes = size_t(kNearThreads) * QUADS * sizeof(float4);
  static constexpr size_t kFoldBytes = size_t(kNearThreads) * T * NV * 2 * sizeof(float);
  static constexpr size_t kSmem = kQuadBytes + kFoldBytes;
  static constexpr int kMinBlocks = PASS == PASS_ZETA ? 4 : 3;
};

template <int KERNEL, int PASS>
__global__ void __launch_bounds__(kNearThreads, NearShape<PASS>::kMinBlocks) near_tile_kernel(
    int ngroups, const int* __restrict__ gbase, const int* __restrict__ gtot,
    const long long* __restrict__ totals, const int2* __restrict__ near_list,
    const float4* __restrict__ rec, const float* __restrict__ vw, int64_t ldv, double* raw,
    int64_t n, int* counters, unsigned long long* pairs) {
  using Sh = NearShape<PASS>;
  constexpr int T = Sh::T, TQ = Sh::TQ, SL = Sh::SL, NV = Sh::NV;
  constexpr bool UJ = Sh::UJ;
  constexpr bool D = PASS == PASS_UJD || PASS == PASS_ZETAD;
  constexpr int PER = kNearThreads / SL;              // staged sources per thread and tile
  constexpr int FOLD_TILES = kNearFoldSources / PER;  // tiles between two folds
  static_assert(kItemTiles % FOLD_TILES == 0, "items start at folds");
  static_assert(kNearThreads == 128 && kNearThreads % TQ == 0 && kTreeBlock <= kNearThreads,
                "four-warp scan below; whole target sets");
  extern __shared__ __align__(16) unsigned char near_smem[];
  float4* tA = reinterpret_cast<float4*>(near_smem);
  float4* tB = tA + kNearThreads;
  float4* tC = tB + kNearThreads;
  float4* tD = tC + kNearThreads;
  float* fold_hi = reinterpret_cast<float*>(near_smem + Sh::kQuadBytes);
  float* fold_lo = fold_hi + size_t(kNearThreads) * T * NV;
  __shared__ int s_start[kNearThreads], s_pref[kNearThreads + 1], s_wsum[4];

  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int tq = tid % TQ, sl = tid / TQ;
  const int item = int(blockIdx.x);
  if (item >= totals[3]) return;
  int grp = 0;   // the last group whose first item is <= item
  {
    const int* first = gbase + int64_t(kListKinds) * ngroups;
    int hi_g = ngroups - 1;
    while (grp < hi_g) {
      const int mid = (grp + hi_g + 1) >> 1;
      if (first[mid] <= item) grp = mid;
      else hi_g = mid - 1;
    }
  }
  const long long w0 = (item - gbase[int64_t(kListKinds) * ngroups + grp]) * totals[4],
                  w1 = w0 + totals[4];   // its tiles
  const int a = grp * kTreeBlock, b = int(min(int64_t(a) + kTreeBlock, n));
  const float4 o0 = rec[3 * int64_t(a)], o1 = rec[3 * int64_t(a) + 1];
  const int l0 = gbase[int64_t(LIST_NEAR) * ngroups + grp], ln = gtot[int64_t(LIST_NEAR) * ngroups + grp];

  float tx[T], ty[T], tz[T];
#pragma unroll
  for (int k = 0; k < T; ++k) {
    const int i = a + tq + TQ * k;
    tx[k] = ty[k] = tz[k] = 0.f;
    if (i < b) {
      const float4 r0 = rec[3 * int64_t(i)], r1 = rec[3 * int64_t(i) + 1];
      tx[k] = rel_f32(r0.x, r1.x, o0.x, o1.x);
      ty[k] = rel_f32(r0.y, r1.y, o0.y, o1.y);
      tz[k] = rel_f32(r0.z, r1.z, o0.z, o1.z);
    }
  }
  float acc[T][NV];
#pragma unroll
  for (int k = 0; k < T; ++k)
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      acc[k][v] = 0.f;
      fold_hi[(v * T + k) * kNearThreads + tid] = 0.f;
      fold_lo[(v * T + k) * kNearThreads + tid] = 0.f;
    }
  auto fold = [&]() {
#pragma unroll
    for (int k = 0; k < T; ++k)
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const int o = (v * T + k) * kNearThreads + tid;
        float s, e;
        two_sum(fold_hi[o], acc[k][v], s, e);
        fold_hi[o] = s;
        fold_lo[o] += e;
        acc[k][v] = 0.f;
      }
  };

  int tiles = 0;
  long long tile0 = 0;   // first tile of the chunk of ranges
  // The near ranges, kNearThreads at a time: their lengths' prefix sums in
  // shared memory; the concatenated sources are then staged in full tiles, each
  // slot finding its range by binary search.
  for (int rc0 = 0; rc0 < ln && tile0 < w1; rc0 += kNearThreads) {
    const int nr = min(kNearThreads, ln - rc0);
    int len = 0;
    __syncthreads();   // previous chunk's tiles consumed
    if (tid < nr) {
      const int2 rg = near_list[l0 + rc0 + tid];
      if (rg.x < 0 || rg.y > n || rg.x > rg.y) {
        atomicOr(&counters[kCntFlags], 8);
      } else {
        len = rg.y - rg.x;
      }
      s_start[tid] = rg.x;
    }
    int incl = len;   // inclusive scan over the 128 threads
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) s_wsum[wid] = incl;
    __syncthreads();
    for (int w = 0; w < wid; ++w) incl += s_wsum[w];
    s_pref[tid + 1] = incl;
    if (tid == 0) s_pref[0] = 0;
    __syncthreads();
    const int total = s_pref[nr];
    const int chunk_tiles = (total + kNearThreads - 1) / kNearThreads;
    const int q_begin = int(min((long long)chunk_tiles, max(0ll, w0 - tile0))) * kNearThreads;
    const int q_end = int(min((long long)total, max(0ll, w1 - tile0) * kNearThreads));
    tile0 += chunk_tiles;
    if (tid == 0 && pairs && q_end > q_begin)
      atomicAdd(&pairs[0], (unsigned long long)(q_end - q_begin) * (unsigned long long)(b - a));
    for (int q0 = q_begin; q0 < q_end; q0 += kNearThreads) {
      const int q = q0 + tid;
      float4 qa = make_float4(kNearPadX, kNearPadX, kNearPadX, 0.f);
      float4 qb = make_float4(0.f, 0.f, 0.f, 0.f);
      float4 qc = make_float4(0.f, 0.f, 0.f, 0.f), qd = qc;
      // Padding constants: a unit core.
      if (UJ && KERNEL == VPM_KERNEL_WINCKELMANS) {
        qa.w = 1.f; qb.w = 1.5f;
      } else {
        qa.w = float(-0.5 * kLog2e);
        qb.w = UJ ? 1.f : float(kZeta0Gauss);
      }
      if (q < total) {
        int lo_r = 0, hi_r = nr - 1;   // last range r with s_pref[r] <= q
        while (lo_r < hi_r) {
          const int mid = (lo_r + hi_r + 1) >> 1;
          if (s_pref[mid] <= q) lo_r = mid;
          else hi_r = mid - 1;
        }
        const int64_t j = s_start[lo_r] + (q - s_pref[lo_r]);
        const float4 r0 = rec[3 * j], r1 = rec[3 * j + 1], r2 = rec[3 * j + 2];
        qa = make_float4(rel_f32(r0.x, r1.x, o0.x, o1.x), rel_f32(r0.y, r1.y, o0.y, o1.y),
                         rel_f32(r0.z, r1.z, o0.z, o1.z), r0.w);
        if (UJ) {
          qb = make_float4(r2.x, r2.y, r2.z, r1.w);
        } else {
          // Gaussian-erf ζ constants: a = -log2(e)/(2σ²) (as for U/J), b = ζ(0)/σ³.
          const float is1 = r1.w;
          qb = make_float4(r2.x, r2.y, r2.z, float(kZeta0Gauss) * is1 * is1 * is1);
          qc = make_float4(vw[j], vw[ldv + j], vw[2 * ldv + j], 0.f);
          if (D) qd = make_float4(vw[3 * ldv + j], vw[4 * ldv + j], vw[5 * ldv + j], 0.f);
        }
      }
      __syncthreads();   // previous tile consumed
      tA[tid] = qa;
      tB[tid] = qb;
      if (!UJ) {
        tC[tid] = qc;
        if (D) tD[tid] = qd;
      }
      __syncthreads();
#pragma unroll 1
      for (int m = 0; m < PER; ++m) {
        const int js = sl + SL * m;
        if constexpr (PASS == PASS_UJ) {
          if (KERNEL == VPM_KERNEL_WINCKELMANS) uj_source_winck<T, true>(tA[js], tB[js], tx, ty, tz, acc);
          else uj_source_gauss<T, true>(tA[js], tB[js], tx, ty, tz, acc);
        } else if constexpr (PASS == PASS_UJD) {
          if (KERNEL == VPM_KERNEL_WINCKELMANS) ujd_source_winck<T, true>(tA[js], tB[js], tx, ty, tz, acc);
          else ujd_source_gauss<T, true>(tA[js], tB[js], tx, ty, tz, acc);
        } else {
          zeta_source<KERNEL, T, true, D, true>(tA[js], tB[js], tC[js], D ? tD[js] : tC[js], tx,
                                                ty, tz, acc);
        }
      }
      if (++tiles % FOLD_TILES == 0) fold();
    }
  }
  fold();
  __syncthreads();
  if (tid < kTreeBlock) {
    const int i = a + tid;
    if (i < b) {
      const int k = tid / TQ, s0 = tid % TQ;
      // One value at a time (a fully unrolled epilogue would hold every slice's
      // pairs of every value in registers at once).
      double a00 = 0.0, a11 = 0.0, d00 = 0.0, d11 = 0.0;
#pragma unroll 1
      for (int w = 0; w < NV; ++w) {
        double v = 0.0;
#pragma unroll
        for (int l = 0; l < SL; ++l) {
          const int o = (w * T + k) * kNearThreads + l * TQ + s0;
          v += double(fold_hi[o]) + double(fold_lo[o]);
        }
        if (UJ && KERNEL == VPM_KERNEL_GAUSSIANERF && w >= 3 && w < 11)
          v *= kGaussAScale;   // A holds p/(-3) sums
        if (UJ) {   // A22: the FP32 forms keep J trace-free
          if (w == 3) a00 = v;
          if (w == 7) a11 = v;
          if (w == 11) v = -(a00 + a11);
        }
        if (PASS == PASS_UJD) {
          if (w == 15) d00 = v;
          if (w == 19) d11 = v;
          if (w == 23) v = -(d00 + d11);
        }
        raw[(int64_t(item) * NV + w) * kTreeBlock + tid] = v;
      }
    }
  }
}

template <int KERNEL, int PASS>
cudaError_t launch_near(int ngroups, int64_t items, const FmmWork* w, const float* vw, int64_t ldv,
                        int64_t n, unsigned long long* pairs, cudaStream_t st) {
  static PerContext done;
  const cudaError_t e = allow_smem(done, near_tile_kernel<KERNEL, PASS>, NearShape<PASS>::kSmem);
  if (e != cudaSuccess) return e;
  near_tile_kernel<KERNEL, PASS><<<int(items), kNearThreads, NearShape<PASS>::kSmem, st>>>(
      ngroups, w->gbase, w->gtot, w->totals, w->near_list, w->rec, vw, ldv, w->near_raw, n,
      w->counters, pairs);
  return cudaSuccess;   // (a failed launch is the caller's cudaGetLastError)
}

// Raw sums [K0, K0 + K) of target t of a group: its near items in order, all K loads
// of an item in flight together (a group has up to 30 items).
template <int NV, int K0, int K>
__device__ __forceinline__ void near_sums(const double* __restrict__ raw, int item0, int item1, int t,
                                          double (&v)[K]) {
#pragma unroll
  for (int k = 0; k < K; ++k) v[k] = 0.0;
  for (int i = item0; i < item1; ++i) {
    const double* r = raw + (int64_t(i) * NV + K0) * kTreeBlock + t;
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] += r[k * kTreeBlock];
  }
}
__device__ __forceinline__ void group_items(const int* __restrict__ gbase,
                                            const long long* __restrict__ totals, int ngroups, int g,
                                            int& item0, int& item1) {
  const int* first = gbase + int64_t(kListKinds) * ngroups;
  item0 = first[g];
  item1 = g + 1 < ngroups ? first[g + 1] : int(totals[3]);
}

// ζ sums of the near items to the original order.
template <int NV>
__global__ void __launch_bounds__(kTreeBlock) zeta_scatter_kernel(
    int64_t n, int ngroups, const int* __restrict__ gbase, const long long* __restrict__ totals,
    const double* __restrict__ raw, const int* __restrict__ perm, double* dst, int64_t ldd) {
  const int64_t i = int64_t(blockIdx.x) * kTreeBlock + threadIdx.x;
  if (i >= n) return;
  int item0, item1;
  group_items(gbase, totals, ngroups, int(blockIdx.x), item0, item1);
  const int64_t o = perm[i];
  double v[NV];
  near_sums<NV, 0, NV>(raw, item0, item1, threadIdx.x, v);
#pragma unroll
  for (int k = 0; k < NV; ++k) dst[k * ldd + o] = v[k];
}

// Rows of a Morton-ordered array back to the original order.
__global__ void scatter_rows_kernel(int64_t n, int rows, const int* __restrict__ perm,
                                    const double* __restrict__ src, int64_t lds, double* dst,
                                    int64_t ldd) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t o = perm[i];
  for (int r = 0; r < rows; ++r) dst[r * ldd + o] = src[r * lds + i];
}

// Rows of an array in the original order into the Morton order.
__global__ void gather_rows_kernel(int64_t n, int rows, const int* __restrict__ perm,
                                   const double* __restrict__ src, int64_t lds, double* dst,
                                   int64_t ldd) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t o = perm[i];
  for (int r = 0; r < rows; ++r) dst[r * ldd + i] = src[r * lds + o];
}

// Rows of an FP64 array in the original order into FP32 rows of the Morton
// order: the ζ passes' v_q and w_q, converted once per pass rather than once
// per staged source in the near field (GB300 converts FP64 at its FP64 rate).
__global__ void gather_rows_f32_kernel(int64_t n, int rows, const int* __restrict__ perm,
                                       const double* __restrict__ src, int64_t lds, float* dst,
                                       int64_t ldd) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t o = perm[i];
  for (int r = 0; r < rows; ++r) dst[r * ldd + i] = float(src[r * lds + o]);
}

// FP64 near field on the sorted FP64 state (positions relative to the leaf's
// first particle; pairs with r = 0 skipped as in the direct FP64 sum).
template <int KERNEL>
__global__ void __launch_bounds__(kTreeBlock) near_f64_kernel(
    int ngroups, const int* __restrict__ gbase, const int* __restrict__ gtot,
    const int2* __restrict__ near_list, const double* __restrict__ sorted, int64_t ldw, double* raw,
    int64_t n, int* counters) {
  __shared__ double sx[kTreeBlock], sy[kTreeBlock], sz[kTreeBlock], sa_[kTreeBlock];
  __shared__ double sg0[kTreeBlock], sg1[kTreeBlock], sg2[kTreeBlock], sb_[kTreeBlock];
  const int tid = threadIdx.x;
  const int a = int(blockIdx.x) * kTreeBlock, b = int(min(int64_t(a) + kTreeBlock, n));
  const double cx = sorted[a], cy = sorted[ldw + a], cz = sorted[2 * ldw + a];
  const int l0 = gbase[int64_t(LIST_NEAR) * ngroups + blockIdx.x];
  const int ln = gtot[int64_t(LIST_NEAR) * ngroups + blockIdx.x];
  for (int t0 = a; t0 < b; t0 += kTreeBlock) {
    const int i = t0 + tid;
    double tx = 0.0, ty = 0.0, tz = 0.0;
    if (i < b) {
      tx = sorted[i] - cx;
      ty = sorted[ldw + i] - cy;
      tz = sorted[2 * ldw + i] - cz;
    }
    double acc[15];
#pragma unroll
    for (int v = 0; v < 15; ++v) acc[v] = 0.0;
    for (int l = 0; l < ln; ++l) {
      const int2 rg = near_list[l0 + l];
      const int s_lo = rg.x, s_hi = rg.y;
      if (s_lo < 0 || s_hi > n || s_lo > s_hi) {
        if (tid == 0) atomicOr(&counters[kCntFlags], 8);
        continue;
      }
      for (int s0 = s_lo; s0 < s_hi; s0 += kTreeBlock) {
        __syncthreads();
        const int j = s0 + tid;
        if (j < s_hi) {
          sx[tid] = sorted[j] - cx;
          sy[tid] = sorted[ldw + j] - cy;
          sz[tid] = sorted[2 * ldw + j] - cz;
          sg0[tid] = sorted[3 * ldw + j];
          sg1[tid] = sorted[4 * ldw + j];
          sg2[tid] = sorted[5 * ldw + j];
          double ka, kb;
          source_consts<KERNEL, double>(sorted[6 * ldw + j], ka, kb);
          sa_[tid] = ka;
          sb_[tid] = kb;
        }
        __syncthreads();
        const int cnt = min(kTreeBlock, s_hi - s0);
        for (int js = 0; js < cnt; ++js) {
          const double dx = tx - sx[js], dy = ty - sy[js], dz = tz - sz[js];
          const double r2 = dx * dx + dy * dy + dz * dz;
          double q, p;
          pair_qp<KERNEL>(r2, sa_[js], sb_[js], q, p);
          if (r2 == 0.0) q = p = 0.0;
          const double gx = sg0[js], gy = sg1[js], gz = sg2[js];
          const double c0 = dy * gz - dz * gy, c1 = dz * gx - dx * gz, c2 = dx * gy - dy * gx;
          acc[0] += q * c0; acc[1] += q * c1; acc[2] += q * c2;
          const double p0 = p * c0, p1 = p * c1, p2 = p * c2;
          acc[3] += p0 * dx; acc[4] += p0 * dy; acc[5] += p0 * dz;
          acc[6] += p1 * dx; acc[7] += p1 * dy; acc[8] += p1 * dz;
          acc[9] += p2 * dx; acc[10] += p2 * dy; acc[11] += p2 * dz;
          acc[12] += q * gx; acc[13] += q * gy; acc[14] += q * gz;
        }
      }
    }
    if (i < b) {
#pragma unroll
      for (int k = 0; k < 15; ++k) raw[(int64_t(blockIdx.x) * 15 + k) * kTreeBlock + tid] = acc[k];
    }
  }
}

// ------------------------------------------------------------ local expansions --
// With local expansions on, far cells at least as large as their target group go to a
// list of their own (LIST_LOC): m2l_kernel turns them into the group's local expansion
// (tree.cuh), which finish_kernel evaluates at each target (L2P).
constexpr int kLocalOrder = 7;   // Q for P = 4: L2P within a few per cent of M2P in J (tree.cuh)

// Two warps per target group.  The group's local-expansion cells are taken
// kM2lChunk at a time; then
//   1. one lane per cell forms its ρ, s and powers;
//   2. four lanes per cell form B̃_j for |j| <= P + Q, order by order (one
//      shared-memory row per cell);
//   3. the moments are loaded coalesced and scaled by ρ^{|k|}/k!;
//   4. lane l of warp v accumulates the local coefficients n = l + 32·(2q + v),
//      q = 0, 1, over the chunk's cells, Σ_k M̃_k B̃_{k+n} times ρ(-s)^{|n|}/n!, two
//      coefficients per packed FP32 instruction.
// The group's coefficients go to loc[g·3·NQ + m·NQ + n].  Bound by shared-memory
// loads: 35 moments (one broadcast each) and 35·4 gathers of B̃ (2.1 wavefronts on
// average) a cell, beside the 120·35·3 FMAs, which take a quarter of that.  The
// chunk's 33 KB leave six groups on an SM.  With one warp a group and one lane a
// cell in step 2 those were six warps with half their lanes idle a third of the
// time: 11.1 ms at N = 500,000, now 8.4 ms.
constexpr int kM2lChunk = 16, kM2lThreads = 64;

template <int P, int Q>
struct M2lShape {
  static constexpr int NC = ncoef(P), NQ = ncoef(Q), NB = ncoef(P + Q);
  static constexpr int ROW = NB % 2 ? NB : NB + 1;        // odd stride: lanes' rows hit distinct banks
  static constexpr int NPOW = (P + 1) + (Q + 1);          // ρ^0..ρ^P, then ρ(-s)^0..ρ(-s)^Q
  static constexpr int SLOTS = (NQ + 63) / 64;            // coefficients per lane
  static constexpr size_t kSmem = size_t(kM2lChunk) * ROW * sizeof(float) +
                                  size_t(kM2lChunk) * NC * sizeof(float4) +
                                  size_t(kM2lChunk) * NPOW * sizeof(float);
  static_assert(SLOTS % 2 == 0, "coefficient slots are packed in pairs");
};

__device__ __forceinline__ void decode_midx(int j, int& a, int& b, int& c) {
  int n = 0;
  while (ncoef(n) <= j) ++n;
  int r = j - (n > 0 ? ncoef(n - 1) : 0);
  a = n;
  while (r >= n - a + 1) {
    r -= n - a + 1;
    --a;
  }
  b = n - a - r;
  c = n - a - b;
}

__device__ __forceinline__ float inv_fact3(int a, int b, int c) {
  float f = 1.f;
  for (int i = 2; i <= a; ++i) f *= float(i);
  for (int i = 2; i <= b; ++i) f *= float(i);
  for (int i = 2; i <= c; ++i) f *= float(i);
  return 1.f / f;
}

template <int P, int Q>
__global__ void __launch_bounds__(kM2lThreads) m2l_kernel(int ngroups, const int* __restrict__ gbase,
                                                 const int* __restrict__ gtot,
                                                 const int* __restrict__ loc_list,
                                                 const double* __restrict__ geom,
                                                 const float* __restrict__ momf,
                                                 const float4* __restrict__ ggeom, int ncells,
                                                 float* __restrict__ loc, int* counters) {
  using Sh = M2lShape<P, Q>;
  constexpr int NC = Sh::NC, NQ = Sh::NQ, ROW = Sh::ROW, NPOW = Sh::NPOW, SLOTS = Sh::SLOTS;
  constexpr int CH = kM2lChunk, H = SLOTS / 2;
  extern __shared__ __align__(16) unsigned char m2l_smem[];
  float4* sM = reinterpret_cast<float4*>(m2l_smem);                            // [cell][k]
  float* sB = reinterpret_cast<float*>(m2l_smem + size_t(CH) * NC * sizeof(float4));   // [cell][j]
  float* sP = sB + CH * ROW;                                                     // [cell][NPOW]
  __shared__ int ids[CH];
  __shared__ float4 dir[CH];
  const int tid = threadIdx.x, lane = tid & 31, wv = tid >> 5;
  const int g = blockIdx.x;
  const float4 tg = ggeom[g];
  const double zx = tg.x, zy = tg.y, zz = tg.z;
  const double h = tg.w;

  // This lane's local coefficients n = lane + 32·(2q + warp): index tables of k + n.
  int t3[SLOTS][P + 1], t2[SLOTS][P + 1], ncs[SLOTS], nord[SLOTS];
  float invf[SLOTS];
#pragma unroll
  for (int q = 0; q < SLOTS; ++q) {
    const int n = lane + 32 * (2 * q + wv);
    int na = 0, nb = 0, nc = 0;
    if (n < NQ) decode_midx(n, na, nb, nc);
    const int nn = na + nb + nc;
    ncs[q] = nc;
    nord[q] = nn;
    invf[q] = n < NQ ? inv_fact3(na, nb, nc) : 0.f;
#pragma unroll
    for (int K = 0; K <= P; ++K) {
      const int N = K + nn;
      t3[q][K] = N * (N + 1) * (N + 2) / 6;
      const int M = K + nb + nc;
      t2[q][K] = M * (M + 1) / 2;
    }
  }
  // The moment elements e = tid + 64·i of a cell row this thread scales.
  constexpr int NE = (3 * NC + kM2lThreads - 1) / kM2lThreads;
  int eord[NE];
  float efac[NE];
#pragma unroll
  for (int i = 0; i < NE; ++i) {
    const int e = tid + kM2lThreads * i;
    int a = 0, b = 0, c = 0;
    if (e < 3 * NC) decode_midx(e % NC, a, b, c);
    eord[i] = a + b + c;
    efac[i] = inv_fact3(a, b, c);
  }

  float Lacc[SLOTS][3];
#pragma unroll
  for (int q = 0; q < SLOTS; ++q) Lacc[q][0] = Lacc[q][1] = Lacc[q][2] = 0.f;

  const int f0 = gbase[int64_t(LIST_LOC) * ngroups + g], fn = gtot[int64_t(LIST_LOC) * ngroups + g];
  for (int base = 0; base < fn; base += CH) {
    const int cnt = min(CH, fn - base);
    // 1. scale factors of cell tid, and its direction for the lanes of step 2.
    if (tid < CH) {
      int cell = -1;
      if (tid < cnt) {
        cell = loc_list[f0 + base + tid];
        if (cell < 0 || cell >= ncells) {   // a list entry outside the tree: record, skip
          atomicOr(&counters[kCntFlags], 4);
          cell = -1;
        }
      }
      ids[tid] = cell;
      double rho = 0.0;
      float rx = 1.f, ry = 0.f, rz = 0.f;
      if (cell >= 0) {
        double cx, cy, cz, cr;
        cell_centre(geom + int64_t(cell) * kGeom, cx, cy, cz, cr);
        const double dx = zx - cx, dy = zy - cy, dz = zz - cz;
        rho = 1.0 / sqrt(dx * dx + dy * dy + dz * dz);
        rx = float(dx * rho); ry = float(dy * rho); rz = float(dz * rho);
      }
      dir[tid] = make_float4(rx, ry, rz, 0.f);
      float* pw = sP + tid * NPOW;
      float v = 1.f;
#pragma unroll
      for (int j = 0; j <= P; ++j) {
        pw[j] = v;
        v *= float(rho);
      }
      const float ns = -float(h * rho);
      v = float(rho);
#pragma unroll
      for (int j = 0; j <= Q; ++j) {
        pw[P + 1 + j] = v;
        v *= ns;
      }
    }
    __syncthreads();
    // 2. B̃ rows: lanes 4c .. 4c + 3 of the block for cell c.
    {
      const float4 r = dir[tid >> 2];
      scaled_taylor_unit4<P + Q>(r.x, r.y, r.z, tid & 3, sB + (tid >> 2) * ROW);
    }
    // 3. moments of the chunk's cells, coalesced, scaled by ρ^{|k|}/k!.
    for (int c = 0; c < cnt; ++c) {
      const int cell = ids[c];
      const float* row = momf + int64_t(cell < 0 ? 0 : cell) * 3 * NC;
      const float* pw = sP + c * NPOW;
#pragma unroll
      for (int i = 0; i < NE; ++i) {
        const int e = tid + kM2lThreads * i;
        if (e < 3 * NC) {
          const int m = e / NC, k = e % NC;
          reinterpret_cast<float*>(&sM[c * NC + k])[m] =
              cell < 0 ? 0.f : row[e] * pw[eord[i]] * efac[i];
        }
      }
    }
    __syncthreads();
    // 4. local coefficients, slots (2h, 2h + 1) packed.
    for (int c = 0; c < cnt; ++c) {
      const float* brow = sB + c * ROW;
      const float4* mrow = sM + c * NC;
      float2 acc[H][3];
#pragma unroll
      for (int q = 0; q < H; ++q) acc[q][0] = acc[q][1] = acc[q][2] = bc2(0.f);
#pragma unroll
      for (int n = 0; n <= P; ++n)
#pragma unroll
        for (int a = n; a >= 0; --a)
#pragma unroll
          for (int b = n - a; b >= 0; --b) {
            const int cc = n - a - b;
            const float4 mk = mrow[midx(a, b, cc)];
            const float2 m0 = bc2(mk.x), m1 = bc2(mk.y), m2 = bc2(mk.z);
#pragma unroll
            for (int q = 0; q < H; ++q) {
              const float2 bv =
                  make_float2(brow[t3[2 * q][n] + t2[2 * q][b + cc] + cc + ncs[2 * q]],
                              brow[t3[2 * q + 1][n] + t2[2 * q + 1][b + cc] + cc + ncs[2 * q + 1]]);
              acc[q][0] = fma2(m0, bv, acc[q][0]);
              acc[q][1] = fma2(m1, bv, acc[q][1]);
              acc[q][2] = fma2(m2, bv, acc[q][2]);
            }
          }
      const float* pw = sP + c * NPOW + P + 1;
#pragma unroll
      for (int q = 0; q < H; ++q) {
        const float fa = pw[nord[2 * q]] * invf[2 * q], fb2 = pw[nord[2 * q + 1]] * invf[2 * q + 1];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          Lacc[2 * q][m] = fmaf(fa, acc[q][m].x, Lacc[2 * q][m]);
          Lacc[2 * q + 1][m] = fmaf(fb2, acc[q][m].y, Lacc[2 * q + 1][m]);
        }
      }
    }
    __syncthreads();
  }
  float* out = loc + int64_t(g) * 3 * NQ;
#pragma unroll
  for (int q = 0; q < SLOTS; ++q) {
    const int n = lane + 32 * (2 * q + wv);
    if (n < NQ) {
      out[n] = Lacc[q][0];
      out[NQ + n] = Lacc[q][1];
      out[2 * NQ + n] = Lacc[q][2];
    }
  }
}

// ---------------------------------------------------------------- far field --
// One CTA per target group, one thread per target or two, the longest far lists first (they
// are ten times the average, and one that starts last runs alone): the moments of
// the group's far cells at the target (M2P; the cells of the group's local expansion
// are on their own list).  U and J of the far field, without the 1/(4π), go to rows
// of pot in Morton order; finish_kernel adds the other parts.
// The group's far cells are taken kFarChunk at a time: the CTA stages their
// moments and centres in shared memory with coalesced loads, then every thread
// reads them from there (broadcast) for its target.
template <int P, typename M>
__host__ __device__ constexpr int far_chunk() {
  return 12288 / int(ncoef(P) * sizeof(M4<M>)) > 0 ? 12288 / int(ncoef(P) * sizeof(M4<M>)) : 1;
}

// PAIR (FP32, P <= 4): two targets per thread (m2p2), one warp a group.  Half the issue
// slots, so the better form where the SMs are full: N = 500,009 (7,813 groups) 14.5 ->
// 12.6 ms.  A field of one wave of groups ends with its longest list, which one warp
// with every target walks slower than two (938 groups: 1.5 -> 1.9 ms); two waves of its
// eight groups per SM is where the line lies.
constexpr int kFarPairGroups = 2 * 8 * 152;

template <int P, typename R, typename M, bool PAIR>
__global__ void __launch_bounds__(PAIR ? kTreeBlock / 2 : kTreeBlock) far_kernel(
    int64_t n, int ngroups, const int* __restrict__ gorder, const int* __restrict__ gbase,
    const int* __restrict__ gtot, const int* __restrict__ far_list,
    const double* __restrict__ geom, const M* __restrict__ mom, const double* __restrict__ sorted,
    int64_t ldw, R* __restrict__ pot, int64_t ldp, int ncells, int* counters,
    unsigned long long* pairs) {
  constexpr int NC = ncoef(P), ROWM = 3 * NC, FCH = far_chunk<P, M>();
  // The three components of a moment together: one broadcast load, where a row of
  // each took three (a third of the kernel's shared-memory instructions remain).
  __shared__ M4<M> smom[FCH * NC];
  __shared__ R sctr[FCH][3];
  const int g = gorder[blockIdx.x];
  const int a = g * kTreeBlock, b = int(min(int64_t(a) + kTreeBlock, n));
  // Targets and cell centres relative to the group's first target, formed in
  // FP64 once per target and once per staged cell, so that the evaluations
  // subtract in R (GB300's FP64 pipe retires about two operations per SM and
  // cycle; three FP64 differences and conversions per evaluation cost more
  // than the FP32 work they feed).
  const double ox = sorted[a], oy = sorted[ldw + a], oz = sorted[2 * ldw + a];
  const int f0 = gbase[g], fn = gtot[g];
  if (threadIdx.x == 0) atomicAdd(&pairs[1], (unsigned long long)fn * (unsigned long long)(b - a));
  constexpr int THREADS = PAIR ? kTreeBlock / 2 : kTreeBlock;
  using V = typename std::conditional<PAIR, float2, R>::type;   // a value of the thread's targets
  const int i = a + int(threadIdx.x);
  {
    // Target i, and with PAIR target i + 32 beside it.
    auto coordinate = [&](int d, double o) {
      const int i0 = i < b ? i : a;
      const R x0 = R(sorted[d * ldw + i0] - o);
      if constexpr (PAIR) {
        const int i1 = i + THREADS < b ? i + THREADS : a;
        return make_float2(x0, R(sorted[d * ldw + i1] - o));
      } else {
        return x0;
      }
    };
    const V x = coordinate(0, ox), y = coordinate(1, oy), z = coordinate(2, oz);
    V dp[9] = {}, dd[18] = {};
    for (int c0 = 0; c0 < fn; c0 += FCH) {
      const int cnt = min(FCH, fn - c0);
      __syncthreads();   // previous chunk consumed
      for (int e = int(threadIdx.x); e < cnt * ROWM; e += THREADS) {
        const int c = e / ROWM, k = e - c * ROWM;
        const int s = far_list[f0 + c0 + c];
        const int m = k / NC;
        reinterpret_cast<M*>(&smom[c * NC + (k - m * NC)])[m] =
            (s < 0 || s >= ncells) ? M(0) : mom[int64_t(s) * ROWM + k];
      }
      for (int c = int(threadIdx.x); c < cnt; c += THREADS) {
        const int s = far_list[f0 + c0 + c];
        double sx = 1e18, sy = 0.0, sz = 0.0, sr;   // far away: finite, negligible terms
        if (s < 0 || s >= ncells) {   // a list entry outside the tree: record, skip (zero moments)
          atomicOr(&counters[kCntFlags], 4);
        } else {
          cell_centre(geom + int64_t(s) * kGeom, sx, sy, sz, sr);
        }
        sctr[c][0] = R(sx - ox); sctr[c][1] = R(sy - oy); sctr[c][2] = R(sz - oz);
      }
      __syncthreads();
      for (int c = 0; c < cnt; ++c) {
        if constexpr (PAIR) {
          const float cx = sctr[c][0], cy = sctr[c][1], cz = sctr[c][2];
          m2p2<P>(add2(x, bc2(-cx)), add2(y, bc2(-cy)), add2(z, bc2(-cz)), smom + c * NC, dp, dd);
        } else {
          R bk[ncoef(P + 2)];
          taylor_coefficients<P + 2, R>(x - sctr[c][0], y - sctr[c][1], z - sctr[c][2], bk);
          m2p_accumulate<P, R, M>(bk, smom + c * NC, dp, dd);
        }
      }
    }
    auto store = [&](int t, const R (&p1)[9], const R (&p2)[18]) {
      if (t >= b) return;
      R uf[3], jf[9];
      curl_from_potential<R>(p1, p2, uf, jf);
#pragma unroll
      for (int k = 0; k < 3; ++k) pot[k * ldp + t] = uf[k];
#pragma unroll
      for (int k = 0; k < 9; ++k) pot[(3 + k) * ldp + t] = jf[k];
    };
    if constexpr (PAIR) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        R p1[9], p2[18];
#pragma unroll
        for (int k = 0; k < 9; ++k) p1[k] = h ? dp[k].y : dp[k].x;
#pragma unroll
        for (int k = 0; k < 18; ++k) p2[k] = h ? dd[k].y : dd[k].x;
        store(i + h * THREADS, p1, p2);
      }
    } else {
      store(i, dp, dd);
    }
  }
}

// Final values of a group's targets, at their original indices: the near items'
// raw sums, the far field of far_kernel and, with Q > 0, the group's local expansion
// (L2P).  One CTA per group, thread = target.
template <int KERNEL, typename R, bool D, int Q>
__global__ void __launch_bounds__(kTreeBlock) finish_kernel(
    int64_t n, int ngroups, const int* __restrict__ gbase, const long long* __restrict__ totals,
    const double* __restrict__ raw, const R* __restrict__ pot, int64_t ldp,
    const float4* __restrict__ ggeom, const float* __restrict__ loc,
    const double* __restrict__ sorted, int64_t ldw, const int* __restrict__ perm, double* U,
    double* J, double* DJ, int64_t ldo) {
  constexpr int NV = D ? 27 : 15;
  const int64_t i = int64_t(blockIdx.x) * kTreeBlock + threadIdx.x;
  if (i >= n) return;
  int item0, item1;
  group_items(gbase, totals, ngroups, int(blockIdx.x), item0, item1);
  float lu[3], lj[9];
  if constexpr (Q > 0) {
    const float4 tg = ggeom[blockIdx.x];
    const double ih = 1.0 / double(tg.w);
    float dp[9], dd[18];
#pragma unroll
    for (int k = 0; k < 9; ++k) dp[k] = 0.f;
#pragma unroll
    for (int k = 0; k < 18; ++k) dd[k] = 0.f;
    l2p_accumulate<Q, float>(loc + int64_t(blockIdx.x) * 3 * ncoef(Q),
                             float((sorted[i] - double(tg.x)) * ih),
                             float((sorted[ldw + i] - double(tg.y)) * ih),
                             float((sorted[2 * ldw + i] - double(tg.z)) * ih), float(ih), dp, dd);
    curl_from_potential<float>(dp, dd, lu, lj);
  }
  const double w = kInv4Pi, kp = kp_to_qr<KERNEL>();
  const int64_t o = perm[i];
  double v15[15];
  near_sums<NV, 0, 15>(raw, item0, item1, threadIdx.x, v15);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    double u = -w * v15[k] + w * double(pot[k * ldp + i]);
    if constexpr (Q > 0) u += w * double(lu[k]);
    U[k * ldo + o] = u;
  }
  // J_ab = -(kp A_ab + ε_abc W_c)/(4π)
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int a = k / 3, b = k % 3;
    double v = kp * v15[3 + k];
    if (a != b) v = (b - a + 3) % 3 == 1 ? v + v15[15 - a - b] : v - v15[15 - a - b];
    double j = -w * v + w * double(pot[(3 + k) * ldp + i]);
    if constexpr (Q > 0) j += w * double(lj[k]);
    J[k * ldo + o] = j;
  }
  if constexpr (D) {   // α-derivative: near field only (see near_tile_kernel)
    double d12[12];
    near_sums<NV, 15, 12>(raw, item0, item1, threadIdx.x, d12);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const int a = k / 3, b = k % 3;
      double v = kp * d12[k];
      if (a != b) v = (b - a + 3) % 3 == 1 ? v + d12[12 - a - b] : v - d12[12 - a - b];
      DJ[k * ldo + o] = -w * v;
    }
  }
}

// ------------------------------------------------------------------- host --
namespace {

cudaError_t reserve_particles(FmmWork* w, int64_t n) {
  if (n <= w->cap) return cudaSuccess;
  const int64_t cap = std::max<int64_t>(n, 1024);
  const int64_t cells = 2 * cap + 8;
  void* ptrs[] = {w->codes, w->codes_alt, w->idx, w->perm, w->sorted, w->rec, w->pot, w->vw,
                  w->lo, w->hi, w->child, w->nchild, w->skip, w->geom, w->leaves, w->ggeom,
                  w->cgeom, w->front, w->pairs, w->counters, w->box, w->box_part, w->wcnt,
                  w->gtot, w->gbase, w->gorder, w->totals, w->cub_tmp};
  for (void* p : ptrs) cudaFree(p);
  cudaError_t e = cudaSuccess;
  auto al = [&](auto*& p, size_t count) {
    if (e == cudaSuccess) e = cudaMalloc(&p, count * sizeof(*p));
  };
  al(w->codes, cap); al(w->codes_alt, cap); al(w->idx, cap); al(w->perm, cap);
  al(w->sorted, 7 * size_t(cap)); al(w->rec, 3 * size_t(cap)); al(w->pot, 12 * size_t(cap));
  al(w->vw, 6 * size_t(cap));
  al(w->lo, cells); al(w->hi, cells); al(w->child, cells); al(w->nchild, cells);
  al(w->skip, cells);
  const int64_t groups = cap / kTreeBlock + 2, meta = groups * kMaxFront;
  al(w->geom, size_t(cells) * kGeom); al(w->leaves, cells);
  al(w->ggeom, cap / kTreeBlock + 2); al(w->cgeom, 2 * size_t(cells));
  al(w->front, kMaxFront); al(w->pairs, 3);
  al(w->counters, kNumCounters); al(w->box, 4); al(w->box_part, kBoxBlocks * 6);
  al(w->wcnt, (kListKinds + 1) * size_t(meta)); al(w->gtot, (kListKinds + 1) * size_t(groups));
  al(w->gbase, (kListKinds + 1) * size_t(groups)); al(w->gorder, groups); al(w->totals, 6);
  if (e != cudaSuccess) {
    w->cap = 0;
    return e;
  }
  if (!w->fork) e = cudaEventCreateWithFlags(&w->fork, cudaEventDisableTiming);
  for (int k = 0; k < 2; ++k) {
    if (e == cudaSuccess && !w->aux[k])
      e = cudaStreamCreateWithFlags(&w->aux[k], cudaStreamNonBlocking);
    if (e == cudaSuccess && !w->join[k])
      e = cudaEventCreateWithFlags(&w->join[k], cudaEventDisableTiming);
  }
  if (e != cudaSuccess) {
    w->cap = 0;
    return e;
  }
  e = cub::DeviceRadixSort::SortPairs(nullptr, w->cub_bytes, w->codes, w->codes_alt, w->idx, w->perm,
                                      int(cap), 0, 63);
  if (e == cudaSuccess) e = cudaMalloc(&w->cub_tmp, w->cub_bytes);
  if (e != cudaSuccess) {
    w->cap = 0;
    return e;
  }
  w->cap = cap;
  w->cell_cap = cells;
  w->meta_cap = meta;
  return cudaSuccess;
}

// Leaves, then the parents generation by generation, the deepest first; returns
// the launches.
template <int P>
int launch_upward(FmmWork* w, int nleaves, int last_gen, bool f64, int64_t ldw, cudaStream_t st) {
  const CellOut out = {w->geom, w->mom, f64 ? nullptr : w->momf, w->cgeom, w->skip};
  tree_leaf_kernel<P><<<(nleaves + kLeafWarps - 1) / kLeafWarps, 32 * kLeafWarps, 0, st>>>(
      nleaves, w->leaves, w->lo, w->hi, w->sorted, ldw, out);
  int launches = 1;
  for (int g = last_gen - 1; g >= 0; --g, ++launches) {
    const int ncells_in_gen = w->h_counters[kGenBase + g + 1] - w->h_counters[kGenBase + g];
    tree_upward_kernel<P><<<std::min(ncells_in_gen, 4096), kUpThreads * kUpSlots, 0, st>>>(
        g, w->counters, w->child, w->nchild, out);
  }
  return launches;
}

template <int P, int Q>
cudaError_t launch_m2l(FmmWork* w, int ngroups, int ncells, cudaStream_t st) {
  static PerContext done;
  const cudaError_t e = allow_smem(done, m2l_kernel<P, Q>, M2lShape<P, Q>::kSmem);
  if (e != cudaSuccess) return e;
  m2l_kernel<P, Q><<<ngroups, kM2lThreads, M2lShape<P, Q>::kSmem, st>>>(
      ngroups, w->gbase, w->gtot, w->loc_list, w->geom, w->momf, w->ggeom, ncells, w->loc,
      w->counters);
  return cudaSuccess;   // (a failed launch is the caller's cudaGetLastError)
}

template <int P>
void launch_far(FmmWork* w, bool f64, int64_t n, int ngroups, int ncells, int64_t ldw,
                cudaStream_t st) {
  auto go = [&](auto kernel, int threads, auto* mom, auto* pot) {
    kernel<<<ngroups, threads, 0, st>>>(n, ngroups, w->gorder, w->gbase, w->gtot, w->far_list, w->geom,
                                        mom, w->sorted, ldw, pot, ldw, ncells, w->counters, w->pairs);
  };
  if (f64) {
    go(far_kernel<P, double, double, false>, kTreeBlock, w->mom, w->pot);
    return;
  }
  float* pot = reinterpret_cast<float*>(w->pot);
  if constexpr (P <= 4) {
    if (ngroups >= kFarPairGroups) {
      go(far_kernel<P, float, float, true>, kTreeBlock / 2, w->momf, pot);
      return;
    }
  }
  go(far_kernel<P, float, float, false>, kTreeBlock, w->momf, pot);
}

template <int KERNEL, typename R, bool D, int Q>
void launch_finish(FmmWork* w, int64_t n, int ngroups, int64_t ldw, double* U, double* J, double* DJ,
                   int64_t ldo, cudaStream_t st) {
  finish_kernel<KERNEL, R, D, Q><<<ngroups, kTreeBlock, 0, st>>>(
      n, ngroups, w->gbase, w->totals, w->near_raw, reinterpret_cast<const R*>(w->pot), ldw, w->ggeom,
      w->loc, w->sorted, ldw, w->perm, U, J, DJ, ldo);
}

// FP64, or FP32 without and with local expansions; the α-derivative is FP32
// Gaussian-erf only (checked by the caller).
template <int KERNEL>
void finish(FmmWork* w, bool f64, bool local, int64_t n, int ngroups, int64_t ldw, double* U, double* J,
            double* DJ, int64_t ldo, cudaStream_t st) {
  constexpr int Q = kLocalOrder, G = VPM_KERNEL_GAUSSIANERF;
  if (DJ && local) launch_finish<G, float, true, Q>(w, n, ngroups, ldw, U, J, DJ, ldo, st);
  else if (DJ) launch_finish<G, float, true, 0>(w, n, ngroups, ldw, U, J, DJ, ldo, st);
  else if (f64) launch_finish<KERNEL, double, false, 0>(w, n, ngroups, ldw, U, J, nullptr, ldo, st);
  else if (local) launch_finish<KERNEL, float, false, Q>(w, n, ngroups, ldw, U, J, nullptr, ldo, st);
  else launch_finish<KERNEL, float, false, 0>(w, n, ngroups, ldw, U, J, nullptr, ldo, st);
}

// Room for the raw sums of the near items of a pass.
cudaError_t reserve_raw(FmmWork* w, int64_t items, int nv) {
  const size_t need = size_t(items) * nv * kTreeBlock;
  if (need <= w->near_raw_cap) return cudaSuccess;
  cudaFree(w->near_raw);
  w->near_raw = nullptr;
  w->near_raw_cap = 0;
  const cudaError_t e = cudaMalloc(&w->near_raw, need * sizeof(double));
  if (e == cudaSuccess) w->near_raw_cap = need;
  return e;
}

// Room for `need` entries of a list.
template <typename T>
cudaError_t reserve_list(T*& p, int64_t& have, int64_t need) {
  need = std::max<int64_t>(need, 1);
  if (need <= have) return cudaSuccess;
  cudaFree(p);
  p = nullptr;
  have = 0;
  const cudaError_t e = cudaMalloc(&p, need * sizeof(T));
  if (e == cudaSuccess) have = need;
  return e;
}

}  // namespace

bool fmm_order_supported(int p) { return p == 2 || p == 4 || p == 6; }
bool fmm_local_order_supported(int q) { return q == 0 || q == kLocalOrder; }

void fmm_stats(const FmmWork* w, int64_t* out) {
  out[0] = w ? w->last_cells : 0;
  out[1] = w ? w->last_leaves : 0;
  out[2] = w ? w->last_groups : 0;
  out[3] = w ? w->last_far : 0;
  out[4] = w ? w->last_near : 0;
  out[5] = w ? int64_t(w->h_pairs[0]) : 0;
  out[6] = w ? int64_t(w->h_pairs[1]) : 0;
  out[7] = w ? int64_t(w->h_pairs[2]) : 0;
}

// U and J of every particle of the context by the treecode (see the header).
// Returns a CUDA error, or cudaErrorInvalidValue with *why set for a tree that
// outgrew its bounds (cannot happen for the 2n + 8 cells reserved).
cudaError_t fmm_eval(vpm_ctx* c, int kernel, int prec, int p, int ncrit, double theta,
                     double sfac, int local_order, double* dj, const char** why) {
  *why = nullptr;
  const int64_t n = c->n;
  if (n == 0) return cudaSuccess;
  if (!c->fmm) c->fmm = new FmmWork();
  FmmWork* w = c->fmm;
  cudaError_t e = reserve_particles(w, n);
  if (e != cudaSuccess) return e;
  cudaStream_t st = c->st;
  const int64_t ldw = w->cap;
  const bool f64 = prec == VPM_PREC_FP64;
  // Local expansions: FP32 far fields of order-4 moments.
  const int local = local_order > 0 && p == 4 && !f64;
  // VPM_FMM_SYNC=1: synchronise after every stage so that an error names it.
  static const bool stage_sync = [] {
    const char* v = std::getenv("VPM_FMM_SYNC");
    return v && v[0] && v[0] != '0';
  }();
  const char* stage = "codes";
  auto launched = [&](int k) {
    c->launches += k;
    cudaError_t le = cudaGetLastError();
    if (le == cudaSuccess && stage_sync) le = cudaStreamSynchronize(st);
    if (le != cudaSuccess) *why = stage;
    return le;
  };

  // 1. codes, sort, gather
  box_partial_kernel<<<kBoxBlocks, 256, 0, st>>>(n, c->X, c->ld, w->box_part);
  box_final_kernel<<<1, kBoxBlocks, 0, st>>>(w->box_part, kBoxBlocks, w->box);
  morton_kernel<<<int((n + 255) / 256), 256, 0, st>>>(n, c->X, c->ld, w->box, w->codes, w->idx);
  if ((e = launched(3)) != cudaSuccess) return e;
  size_t bytes = w->cub_bytes;
  e = cub::DeviceRadixSort::SortPairs(w->cub_tmp, bytes, w->codes, w->codes_alt, w->idx, w->perm,
                                      int(n), 0, 63, st);
  if (e != cudaSuccess) return e;
  c->launches += 4;   // the radix sort's passes (counted approximately)
  const uint64_t* codes = w->codes_alt;
  gather_kernel<<<int((n + 255) / 256), 256, 0, st>>>(n, w->perm, c->X, c->G, c->S, c->ld,
                                                     w->sorted, ldw);
  if ((e = launched(1)) != cudaSuccess) return e;
  if (!f64) {
    e = launch_pack_sources(kernel, n, w->sorted, w->sorted + 3 * ldw, w->sorted + 6 * ldw, ldw,
                            1.0, w->rec, st);
    if ((e = e == cudaSuccess ? launched(1) : e) != cudaSuccess) return e;
  }

  // 2. tree, generation by generation
  stage = "tree build";
  tree_init_kernel<<<1, 1, 0, st>>>(n, w->lo, w->hi, w->skip, w->counters);
  // (32 cells a block; most of the launches find an empty generation.)
  const int split_grid = int(std::min<int64_t>((w->cell_cap + 31) / 32, 152));
  for (int g = 0; g < kMaxGen - 1; ++g) {
    tree_split_kernel<<<split_grid, 256, 0, st>>>(g, ncrit, w->cell_cap, codes, w->lo, w->hi,
                                                  w->child, w->nchild, w->skip, w->leaves, w->counters);
  }
  if ((e = launched(1 + (kMaxGen - 1))) != cudaSuccess) return e;
  int* hc = w->h_counters;
  e = cudaMemcpyAsync(hc, w->counters, sizeof(int) * kNumCounters, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return e;
  if (hc[kCntFlags] != 0) {
    *why = "tree outgrew its cell bounds";
    return cudaErrorInvalidValue;
  }
  const int ncells = hc[kCntCells], nleaves = hc[kCntLeaves];
  const int ngroups = int((n + kTreeBlock - 1) / kTreeBlock);
  // Walk roots: the leaves among generations 0 and 1, and generation 2.
  int nfront = 0;
  {
    const int g2 = hc[kGenBase + 2], g3 = hc[kGenBase + 3];
    std::vector<int> nch(g2), first(g3);
    e = cudaMemcpy(nch.data(), w->nchild, sizeof(int) * g2, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess)
      e = cudaMemcpy(first.data(), w->lo, sizeof(int) * g3, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return e;
    int hf[kMaxFront];
    for (int cidx = 0; cidx < g2 && nfront < kMaxFront; ++cidx)
      if (nch[cidx] == 0) hf[nfront++] = cidx;
    const int leaves01 = nfront;
    for (int cidx = g2; cidx < g3 && nfront < kMaxFront; ++cidx) hf[nfront++] = cidx;
    // Cells of a generation are numbered as the atomic counter handed them out;
    // the roots go in Morton order, so that the lists (and the order of every
    // sum over them) are the same in every evaluation.
    auto morton = [&](int x, int y) { return first[x] < first[y]; };
    std::sort(hf, hf + leaves01, morton);
    std::sort(hf + leaves01, hf + nfront, morton);
    if (nfront == 0 || nfront != leaves01 + (g3 - g2)) {   // at most 9 + 64 by construction
      *why = "tree frontier larger than expected";
      return cudaErrorInvalidValue;
    }
    e = cudaMemcpyAsync(w->front, hf, sizeof(int) * nfront, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
  }
  const int64_t nwalk = int64_t(ngroups) * nfront;
  if (nwalk > w->meta_cap) {
    *why = "treecode walk table too small";
    return cudaErrorInvalidValue;
  }

  // 3. upward pass (deepest generation first)
  const int NC = p == 2 ? ncoef(2) : p == 4 ? ncoef(4) : ncoef(6);
  if (w->mom_cells < ncells || w->mom_p != p) {
    cudaFree(w->mom);
    cudaFree(w->momf);
    w->mom = nullptr;
    w->momf = nullptr;
    w->mom_cells = 0;
    e = cudaMalloc(&w->mom, size_t(ncells) * 3 * NC * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&w->momf, size_t(ncells) * 3 * NC * sizeof(float));
    if (e != cudaSuccess) return e;
    w->mom_cells = ncells;
    w->mom_p = p;
  }
  stage = "upward pass";
  int last_gen = 0;
  for (int g = 0; g < kMaxGen; ++g)
    if (hc[kGenBase + g + 1] > hc[kGenBase + g]) last_gen = g;
  // (The deepest generation holds only leaves.)
  if (p == 2) e = launched(launch_upward<2>(w, nleaves, last_gen, f64, ldw, st));
  else if (p == 4) e = launched(launch_upward<4>(w, nleaves, last_gen, f64, ldw, st));
  else e = launched(launch_upward<6>(w, nleaves, last_gen, f64, ldw, st));
  if (e != cudaSuccess) return e;
  group_geom_kernel<<<(ngroups + 7) / 8, 256, 0, st>>>(n, w->sorted, ldw, w->ggeom);
  if ((e = launched(1)) != cudaSuccess) return e;

  // 4. interaction lists: count, scan, fill
  stage = "traversal";
  const int tgrid = int((nwalk + 127) / 128);
  int* nsrc = w->wcnt + kListKinds * nwalk;
  traverse_kernel<false><<<tgrid, 128, 0, st>>>(ngroups, nfront, w->front, w->ggeom, w->cgeom,
                                                float(theta), float(sfac), local, w->wcnt, nsrc,
                                                nullptr, nullptr, nullptr, nullptr, w->counters,
                                                ncells);
  group_lists_kernel<<<(ngroups + 3) / 4, 128, 0, st>>>(ngroups, nfront, w->wcnt, nsrc, w->gtot);
  group_scan_kernel<<<1, kScanThreads, 0, st>>>(ngroups, w->gtot, w->gbase, w->gorder, f64, w->totals);
  if ((e = launched(3)) != cudaSuccess) return e;
  long long totals[6];
  e = cudaMemcpyAsync(totals, w->totals, sizeof(totals), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return e;
  const int64_t nf = totals[LIST_FAR], nn = totals[LIST_NEAR], nl = totals[LIST_LOC], items = totals[3];
  if (nf > INT32_MAX || nn > INT32_MAX || nl > INT32_MAX) {
    *why = "treecode interaction lists exceed 2^31 entries";
    return cudaErrorInvalidValue;
  }
  e = reserve_list(w->far_list, w->far_cap, nf);
  if (e == cudaSuccess) e = reserve_list(w->near_list, w->near_cap, nn);
  if (e == cudaSuccess && local) e = reserve_list(w->loc_list, w->loc_cap_list, nl);
  if (e == cudaSuccess) e = reserve_raw(w, items, dj ? 27 : 15);
  if (e == cudaSuccess && local)
    e = reserve_list(w->loc, w->loc_cap, int64_t(ngroups) * 3 * ncoef(kLocalOrder));
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(w->pairs, 0, 2 * sizeof(unsigned long long), st);
  if (e != cudaSuccess) return e;
  traverse_kernel<true><<<tgrid, 128, 0, st>>>(ngroups, nfront, w->front, w->ggeom, w->cgeom,
                                               float(theta), float(sfac), local, w->wcnt, nsrc,
                                               w->gbase, w->far_list, w->near_list, w->loc_list,
                                               w->counters, ncells);
  if ((e = launched(1)) != cudaSuccess) return e;

  // 5.-7. far field (M2P) and local expansions (M2L) on streams of their own, the near
  // field on the context's: they share nothing that is written.  The far field goes
  // first: its CTAs leave room for M2L's (96 registers of 64 threads, bound by shared
  // memory) but not for the near field's (168 of 128), which fill the SMs as the far
  // field's shorter lists end.
  e = cudaEventRecord(w->fork, st);
  for (int k = 0; k < 2; ++k)
    if (e == cudaSuccess) e = cudaStreamWaitEvent(w->aux[k], w->fork, 0);
  if (e != cudaSuccess) return e;
  stage = "far field";
  cudaError_t le = cudaSuccess, ne = cudaSuccess;   // of the launches; the streams rejoin in any case
  if (p == 2) launch_far<2>(w, f64, n, ngroups, ncells, ldw, w->aux[0]);
  else if (p == 4) launch_far<4>(w, f64, n, ngroups, ncells, ldw, w->aux[0]);
  else launch_far<6>(w, f64, n, ngroups, ncells, ldw, w->aux[0]);
  if (local) le = launch_m2l<4, kLocalOrder>(w, ngroups, ncells, w->aux[1]);
  if (f64) {
    if (kernel == VPM_KERNEL_WINCKELMANS)
      near_f64_kernel<VPM_KERNEL_WINCKELMANS><<<ngroups, kTreeBlock, 0, st>>>(
          ngroups, w->gbase, w->gtot, w->near_list, w->sorted, ldw, w->near_raw, n, w->counters);
    else
      near_f64_kernel<VPM_KERNEL_GAUSSIANERF><<<ngroups, kTreeBlock, 0, st>>>(
          ngroups, w->gbase, w->gtot, w->near_list, w->sorted, ldw, w->near_raw, n, w->counters);
  } else if (dj) {
    ne = launch_near<VPM_KERNEL_GAUSSIANERF, PASS_UJD>(ngroups, items, w, nullptr, 0, n, w->pairs, st);
  } else if (kernel == VPM_KERNEL_WINCKELMANS) {
    ne = launch_near<VPM_KERNEL_WINCKELMANS, PASS_UJ>(ngroups, items, w, nullptr, 0, n, w->pairs, st);
  } else {
    ne = launch_near<VPM_KERNEL_GAUSSIANERF, PASS_UJ>(ngroups, items, w, nullptr, 0, n, w->pairs, st);
  }
  if (le == cudaSuccess) le = ne;
  if ((ne = launched(2 + local)) != cudaSuccess) le = ne;
  else if (le != cudaSuccess) *why = stage;
  // The other streams always rejoin, whatever failed.
  for (int k = 0; k < 2; ++k) {
    cudaError_t je = cudaEventRecord(w->join[k], w->aux[k]);
    if (je == cudaSuccess) je = cudaStreamWaitEvent(st, w->join[k], 0);
    if (je != cudaSuccess) cudaStreamSynchronize(w->aux[k]);
    if (e == cudaSuccess) e = je;
  }
  if (le != cudaSuccess) return le;
  if (e != cudaSuccess) return e;

  // 8. final values
  stage = "output";
  if (kernel == VPM_KERNEL_WINCKELMANS)
    finish<VPM_KERNEL_WINCKELMANS>(w, f64, local, n, ngroups, ldw, c->U, c->J, dj, c->ld, st);
  else
    finish<VPM_KERNEL_GAUSSIANERF>(w, f64, local, n, ngroups, ldw, c->U, c->J, dj, c->ld, st);
  if ((e = launched(1)) != cudaSuccess) return e;
  e = cudaMemcpyAsync(hc, w->counters, sizeof(int) * kGenBase, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(w->h_pairs, w->pairs, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return e;
  if (hc[kCntFlags] != 0) {
    *why = "treecode index out of range (checked, skipped)";
    return cudaErrorInvalidValue;
  }
  w->last_cells = ncells;
  w->last_leaves = nleaves;
  w->last_groups = ngroups;
  w->last_items = items;
  w->last_far = nf + nl;
  w->h_pairs[2] = (unsigned long long)nl;
  w->last_near = nn;
  w->last_n = n;
  return cudaSuccess;
}

// The ζ sums of a pair pass (PASS_ZETA: Ω, V; PASS_ZETAD: also DΩ, DV; raw
// rows as the direct pass writes them) over the near lists of the last
// treecode evaluation, which must be of the same particle positions and cores
// (Gaussian-erf: ζ beyond the near field's 7.1σ is below FP32 significance).
cudaError_t fmm_zeta(vpm_ctx* c, bool d, const double* vs, const double* ws, double* out,
                     const char** why) {
  *why = nullptr;
  FmmWork* w = c->fmm;
  const int64_t n = c->n;
  if (!w || w->last_n != n || n == 0) {
    *why = "the treecode ζ pass needs a treecode U/J evaluation of the same field";
    return cudaErrorInvalidValue;
  }
  cudaStream_t st = c->st;
  const int64_t ldw = w->cap;
  const int ngroups = int(w->last_groups);
  const int64_t items = w->last_items;
  const int grid = int((n + 255) / 256);
  const cudaError_t re = reserve_raw(w, items, d ? 12 : 6);
  if (re != cudaSuccess) return re;
  gather_rows_f32_kernel<<<grid, 256, 0, st>>>(n, 3, w->perm, vs, c->ld, w->vw, ldw);
  if (d)
    gather_rows_f32_kernel<<<grid, 256, 0, st>>>(n, 3, w->perm, ws, c->ld, w->vw + 3 * ldw, ldw);
  cudaError_t ne;
  if (d) {
    ne = launch_near<VPM_KERNEL_GAUSSIANERF, PASS_ZETAD>(ngroups, items, w, w->vw, ldw, n, nullptr, st);
    zeta_scatter_kernel<12><<<ngroups, kTreeBlock, 0, st>>>(n, ngroups, w->gbase, w->totals,
                                                            w->near_raw, w->perm, out, c->ld);
  } else {
    ne = launch_near<VPM_KERNEL_GAUSSIANERF, PASS_ZETA>(ngroups, items, w, w->vw, ldw, n, nullptr, st);
    zeta_scatter_kernel<6><<<ngroups, kTreeBlock, 0, st>>>(n, ngroups, w->gbase, w->totals,
                                                           w->near_raw, w->perm, out, c->ld);
  }
  c->launches += d ? 4 : 3;
  const cudaError_t e = cudaGetLastError();
  return ne != cudaSuccess ? ne : e;
}

}  // namespace vpm

// ------------------------------------------------------ Morton order of a pass --
namespace vpm {

// Buffers of the Morton order used by the direct pair passes (csrc/capi.cu):
// codes, the permutation and CUB scratch, apart from the treecode's own.
struct SortWork {
  int64_t cap = 0;
  int fcap = 0;                          // fields the per-field boxes hold
  uint64_t *codes = nullptr, *codes_alt = nullptr;
  int *idx = nullptr, *perm = nullptr;
  double *box = nullptr, *box_part = nullptr;
  double* fbox = nullptr;                // 4 per field: corner, cube edge
  void* cub_tmp = nullptr;
  size_t cub_bytes = 0;
};

void sort_free(SortWork* s) {
  if (!s) return;
  void* ptrs[] = {s->codes, s->codes_alt, s->idx, s->perm, s->box, s->box_part, s->fbox, s->cub_tmp};
  for (void* p : ptrs) cudaFree(p);
  delete s;
}

cudaError_t sort_reserve(SortWork*& s, int64_t n, int nfields) {
  if (!s) s = new SortWork();
  if (n <= s->cap && nfields <= s->fcap) return cudaSuccess;
  n = std::max(n, s->cap);
  nfields = std::max(nfields, std::max(s->fcap, 1));
  void* ptrs[] = {s->codes, s->codes_alt, s->idx, s->perm, s->box, s->box_part, s->fbox, s->cub_tmp};
  for (void* p : ptrs) cudaFree(p);
  *s = SortWork();
  cudaError_t e = cudaSuccess;
  auto al = [&](auto*& p, size_t count) {
    if (e == cudaSuccess) e = cudaMalloc(&p, count * sizeof(*p));
  };
  al(s->codes, n); al(s->codes_alt, n); al(s->idx, n); al(s->perm, n);
  al(s->box, 4); al(s->box_part, kBoxBlocks * 6); al(s->fbox, 4 * size_t(nfields));
  if (e == cudaSuccess)
    e = cub::DeviceRadixSort::SortPairs(nullptr, s->cub_bytes, s->codes, s->codes_alt, s->idx,
                                        s->perm, int(n), 0, 64);
  if (e == cudaSuccess) e = cudaMalloc(&s->cub_tmp, s->cub_bytes);
  if (e != cudaSuccess) return e;
  s->cap = n;
  s->fcap = nfields;
  return cudaSuccess;
}

// perm = the particles of X (rows of leading dimension ld) along a Morton curve
// of their bounding cube, to 2^10 cells per axis (the top 30 bits of the code;
// ties keep their index order); 3 launches plus the radix sort's, no host sync.
cudaError_t sort_order(SortWork* s, int64_t n, const double* X, int64_t ld, cudaStream_t st,
                       const int** perm) {
  box_partial_kernel<<<kBoxBlocks, 256, 0, st>>>(n, X, ld, s->box_part);
  box_final_kernel<<<1, kBoxBlocks, 0, st>>>(s->box_part, kBoxBlocks, s->box);
  morton_kernel<<<int((n + 255) / 256), 256, 0, st>>>(n, X, ld, s->box, s->codes, s->idx);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  size_t bytes = s->cub_bytes;
  e = cub::DeviceRadixSort::SortPairs(s->cub_tmp, bytes, s->codes, s->codes_alt, s->idx, s->perm,
                                      int(n), 33, 63, st);
  *perm = s->perm;
  return e;
}

// Bounding cube of field f (particles [foff[f], foff[f+1]) or [foff[f], n)),
// one block per field.  Minima and maxima on the integer images (order_key): FP64
// comparisons of 16,384 particles on one SM's FP64 pipe took 44 µs.
constexpr int kFieldBoxThreads = 1024;
__global__ void __launch_bounds__(kFieldBoxThreads) field_box_kernel(
    int64_t n, const int64_t* __restrict__ foff, int nfields, const double* __restrict__ X,
    int64_t ld, double* fbox) {
  __shared__ long long s[6][32];
  const int f = blockIdx.x, t = threadIdx.x;
  const int64_t i0 = foff[f], i1 = f + 1 < nfields ? foff[f + 1] : n;
  long long v[6];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    v[d] = order_key(INFINITY);
    v[3 + d] = order_key(-INFINITY);
  }
  for (int64_t i = i0 + t; i < i1; i += blockDim.x)
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double x = X[d * ld + i];
      if (is_nan(x)) continue;
      const long long k = order_key(x);
      v[d] = min(v[d], k);
      v[3 + d] = max(v[3 + d], k);
    }
#pragma unroll
  for (int d = 0; d < 6; ++d) {
    v[d] = d < 3 ? warp_min_key(v[d]) : warp_max_key(v[d]);
    if ((t & 31) == 0) s[d][t >> 5] = v[d];
  }
  __syncthreads();
  if (t < 32) {
    double b[6];
#pragma unroll
    for (int d = 0; d < 6; ++d)
      b[d] = order_value(d < 3 ? warp_min_key(s[d][t]) : warp_max_key(s[d][t]));
    if (t == 0) {
      const double size = fmax(fmax(b[3] - b[0], b[4] - b[1]), b[5] - b[2]);
      const bool any = i1 > i0;
      fbox[4 * f + 0] = any ? b[0] : 0.0;
      fbox[4 * f + 1] = any ? b[1] : 0.0;
      fbox[4 * f + 2] = any ? b[2] : 0.0;
      fbox[4 * f + 3] = any && size > 0 ? size * (1.0 + 1e-9) : 1.0;
    }
  }
}

// Key of particle i: its field in the high bits, then the top 30 bits of its
// Morton code in the field's own cube.
__global__ void morton_fields_kernel(int64_t n, const double* __restrict__ X, int64_t ld,
                                     const int64_t* __restrict__ foff, int nfields,
                                     const double* __restrict__ fbox, uint64_t* codes, int* idx) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int lo = 0, hi = nfields - 1;   // the last field whose offset is <= i
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (foff[mid] <= i) lo = mid;
    else hi = mid - 1;
  }
  const double* b = fbox + 4 * lo;
  const double scale = double(1 << 10) / b[3];
  uint64_t q[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double t = floor((X[d * ld + i] - b[d]) * scale);
    q[d] = uint64_t(fmin(fmax(t, 0.0), double((1 << 10) - 1)));
  }
  codes[i] = uint64_t(lo) << 30 | spread3(q[0]) << 2 | spread3(q[1]) << 1 | spread3(q[2]);
  idx[i] = int(i);
}

// perm for a batch of fields laid out one after another: each field's
// particles along the Morton curve of its own cube, within its own range.
cudaError_t sort_order_fields(SortWork* s, int64_t n, const double* X, int64_t ld,
                              const int64_t* foff, int nfields, cudaStream_t st, const int** perm) {
  if (nfields > s->fcap || n > s->cap) return cudaErrorInvalidValue;
  field_box_kernel<<<nfields, kFieldBoxThreads, 0, st>>>(n, foff, nfields, X, ld, s->fbox);
  morton_fields_kernel<<<int((n + 255) / 256), 256, 0, st>>>(n, X, ld, foff, nfields, s->fbox,
                                                            s->codes, s->idx);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  int bits = 30;
  while (bits < 64 && (uint64_t(nfields - 1) >> (bits - 30)) != 0) ++bits;
  size_t bytes = s->cub_bytes;
  e = cub::DeviceRadixSort::SortPairs(s->cub_tmp, bytes, s->codes, s->codes_alt, s->idx, s->perm,
                                      int(n), 0, bits, st);
  *perm = s->perm;
  return e;
}

cudaError_t launch_gather_rows(int64_t n, int rows, const int* perm, const double* src,
                               int64_t lds, double* dst, int64_t ldd, cudaStream_t st) {
  if (n <= 0 || rows <= 0) return cudaSuccess;
  gather_rows_kernel<<<int((n + 255) / 256), 256, 0, st>>>(n, rows, perm, src, lds, dst, ldd);
  return cudaGetLastError();
}

cudaError_t launch_scatter_rows(int64_t n, int rows, const int* perm, const double* src,
                                int64_t lds, double* dst, int64_t ldd, cudaStream_t st) {
  if (n <= 0 || rows <= 0) return cudaSuccess;
  scatter_rows_kernel<<<int((n + 255) / 256), 256, 0, st>>>(n, rows, perm, src, lds, dst, ldd);
  return cudaGetLastError();
}

}  // namespace vpm
