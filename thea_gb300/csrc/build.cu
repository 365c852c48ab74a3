// LBVH build of a forest: one BVH per segment of elements (one segment for a single mesh or point set; one per mesh
// for a batch), all built together in one pass: element boxes -> per-segment 3D Morton codes with the segment id in the
// top bits -> one stable radix sort -> Karras binary radix trees that never cross a segment boundary -> bottom-up box
// refit -> top-down collapse into W-wide trees whose leaves are contiguous runs of sorted elements -> element records in
// leaf order.
//
// Replaces BvhN::init / initTree / createKdTree (Code/Source/Algorithms/BvhN.hpp:705-794, 1366-1525). The reference
// builds a median-split kd-tree with leaves of at most 5 elements and pads every node box by 5%; this build produces a
// different tree over the same elements. Query results do not depend on the tree: every query returns the element with
// the smallest distance or hit time, ties to the lowest index, and node boxes are padded so that no element at the best
// distance can be pruned by rounding.
//
// Index conventions: elements are addressed by their global sorted position; a leaf stores its first element relative to
// its segment's first sorted position (so one segment may hold up to 2^27 - 1 elements while a forest may hold more),
// and element records store the element's index within its segment (the face index within its mesh).
#include "bvh.hpp"
#include "device_util.cuh"
#include "query.hpp"
#include "slab_range.cuh"
#include "traverse_ops.cuh"

#include <algorithm>
#include <vector>

namespace thea {
namespace {

constexpr int BUILD_THREADS = 256;

__device__ __forceinline__ int f2ord(float f) {
  int i = __float_as_int(f);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
__host__ __device__ __forceinline__ float ord2f(int i) {
#ifdef __CUDA_ARCH__
  return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff);
#else
  int j = i >= 0 ? i : i ^ 0x7fffffff;
  float f;
  memcpy(&f, &j, 4);
  return f;
#endif
}

// Segment of element i: largest s with start[s] <= i (start has M + 1 entries, start[0] = 0)
__device__ __forceinline__ int segment_of(int64_t const * __restrict__ start, int M, int64_t i) {
  int lo = 0, hi = M - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (start[mid] <= i) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// A face index outside [0, nv) sets *bad and reads vertex 0 in its place (nv > 0); the host refuses the build when it next
// synchronizes.
__device__ __forceinline__ int64_t face_vertex(int32_t const * __restrict__ F, int64_t k, int64_t nv, bool & out) {
  int64_t f = F[k];
  if (f >= 0 && f < nv) return f;
  out = true;
  return 0;
}

// Per-segment bounds, 12 ordered ints per segment: [0..2] min of box centres, [3..5] max of box centres,
// [6..8] min of box lo, [9..11] max of box hi. A warp whose lanes share one segment reduces before its atomics, and a
// block whose warps all share one segment reduces once more, so a single large segment takes 12 atomics per block
// rather than per warp (the per-warp form spent 0.5 ms of contended atomics on 2 M triangles).
__global__ void elem_box_kernel(float const * __restrict__ V, int64_t nv, int32_t const * __restrict__ F, int64_t n,
                                int is_mesh, int64_t const * __restrict__ seg_start, int M, float4 * __restrict__ elo,
                                float4 * __restrict__ ehi, int * __restrict__ bounds, int * __restrict__ bad) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool ok = i < n;
  int v[12];
  int seg = 0;
  if (ok) {
    V3 lo, hi;
    if (is_mesh) {
      bool out = false;
      V3 a = load_v3(V + 3 * face_vertex(F, 3 * i, nv, out));
      V3 b = load_v3(V + 3 * face_vertex(F, 3 * i + 1, nv, out));
      V3 c = load_v3(V + 3 * face_vertex(F, 3 * i + 2, nv, out));
      if (out) *bad = 1;
      lo = V3{fminf(a.x, fminf(b.x, c.x)), fminf(a.y, fminf(b.y, c.y)), fminf(a.z, fminf(b.z, c.z))};
      hi = V3{fmaxf(a.x, fmaxf(b.x, c.x)), fmaxf(a.y, fmaxf(b.y, c.y)), fmaxf(a.z, fmaxf(b.z, c.z))};
    } else {
      lo = hi = load_v3(V + 3 * i);
    }
    elo[i] = make_float4(lo.x, lo.y, lo.z, 0.f);
    ehi[i] = make_float4(hi.x, hi.y, hi.z, 0.f);
    V3 c = 0.5f * (hi + lo);
    v[0] = v[3] = f2ord(c.x); v[1] = v[4] = f2ord(c.y); v[2] = v[5] = f2ord(c.z);
    v[6] = f2ord(lo.x); v[7] = f2ord(lo.y); v[8] = f2ord(lo.z);
    v[9] = f2ord(hi.x); v[10] = f2ord(hi.y); v[11] = f2ord(hi.z);
    seg = M > 1 ? segment_of(seg_start, M, i) : 0;
  } else {
#pragma unroll
    for (int t = 0; t < 12; ++t) v[t] = ((t < 3) || (t >= 6 && t < 9)) ? INT_MAX : INT_MIN;
    seg = -1;
  }
  int seg0 = __shfl_sync(0xffffffffu, seg, 0);
  bool uniform = __all_sync(0xffffffffu, seg == seg0 || seg < 0) && seg0 >= 0;
  if (uniform) {
#pragma unroll
    for (int t = 0; t < 12; ++t) {
      bool is_min = (t < 3) || (t >= 6 && t < 9);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        int u = __shfl_xor_sync(0xffffffffu, v[t], o);
        v[t] = is_min ? min(v[t], u) : max(v[t], u);
      }
    }
  }
  // block level: warps that reduced for the same segment combine in shared memory
  __shared__ int s_v[BUILD_THREADS / 32][12];
  __shared__ int s_seg[BUILD_THREADS / 32];
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) s_seg[warp] = uniform ? seg0 : -1;
  if (uniform && lane < 12) s_v[warp][lane] = v[lane];
  __syncthreads();
  int bseg = s_seg[0];
  bool block_uniform = bseg >= 0;
  for (int w = 1; w < BUILD_THREADS / 32; ++w) block_uniform = block_uniform && s_seg[w] == bseg;
  if (block_uniform) {
    if (threadIdx.x < 12) {
      int t = threadIdx.x;
      bool is_min = (t < 3) || (t >= 6 && t < 9);
      int r = s_v[0][t];
      for (int w = 1; w < BUILD_THREADS / 32; ++w) r = is_min ? min(r, s_v[w][t]) : max(r, s_v[w][t]);
      if (is_min) atomicMin(&bounds[12 * bseg + t], r);
      else atomicMax(&bounds[12 * bseg + t], r);
    }
    return;
  }
  if (uniform) {
    if (lane == 0) {
#pragma unroll
      for (int t = 0; t < 12; ++t) {
        bool is_min = (t < 3) || (t >= 6 && t < 9);
        if (is_min) atomicMin(&bounds[12 * seg0 + t], v[t]);
        else atomicMax(&bounds[12 * seg0 + t], v[t]);
      }
    }
  } else if (ok) {
#pragma unroll
    for (int t = 0; t < 12; ++t) {
      bool is_min = (t < 3) || (t >= 6 && t < 9);
      if (is_min) atomicMin(&bounds[12 * seg + t], v[t]);
      else atomicMax(&bounds[12 * seg + t], v[t]);
    }
  }
}

// Start values: bounds, the error words and, for one segment, its start (single_root_kernel and segment_roots_kernel write the
// roots and the collapse's first level)
__global__ void build_init_kernel(int * __restrict__ bounds, int M, int * __restrict__ bad, unsigned * __restrict__ err,
                                  int64_t * __restrict__ seg_start, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) {
    *bad = 0;
    *err = 0;
    if (M == 1) {
      seg_start[0] = 0;
      seg_start[1] = n;
    }
  }
  if (i >= 12 * (int64_t)M) return;
  int t = (int)(i % 12);
  bounds[i] = ((t < 3) || (t >= 6 && t < 9)) ? INT_MAX : INT_MIN;
}

__device__ __forceinline__ uint64_t expand21(uint32_t v) {
  uint64_t x = v & 0x1fffffull;
  x = (x | x << 32) & 0x1f00000000ffffull;
  x = (x | x << 16) & 0x1f0000ff0000ffull;
  x = (x | x << 8) & 0x100f00f00f00f00full;
  x = (x | x << 4) & 0x10c30c30c30c30c3ull;
  x = (x | x << 2) & 0x1249249249249249ull;
  return x;
}

// key = (segment << 3 bpa) | Morton code with bpa bits per axis of the box centre within its segment's centre bounds
__global__ void morton_kernel(float4 const * __restrict__ elo, float4 const * __restrict__ ehi, int64_t n,
                              int64_t const * __restrict__ seg_start, int M, int const * __restrict__ bounds, int bpa,
                              uint64_t * __restrict__ keys, uint32_t * __restrict__ vals) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int seg = M > 1 ? segment_of(seg_start, M, i) : 0;
  float4 l = elo[i], h = ehi[i];
  float c[3] = {0.5f * (h.x + l.x), 0.5f * (h.y + l.y), 0.5f * (h.z + l.z)};
  float cells = (float)(1u << bpa);
  uint32_t q[3];
  // One scale for all axes (the largest extent), so that the implicit split planes are spatial medians of a cube: a
  // flat or elongated segment gets few splits across its thin axes. (Per-axis scaling gave the 2 M-triangle heightfield,
  // 0.3 units thick over 1 x 1, as many splits in z as in x and y, whose children overlap in x and y: 12 % slower rays.)
  float ext = 0.f;
#pragma unroll
  for (int a = 0; a < 3; ++a) ext = fmaxf(ext, ord2f(bounds[12 * seg + 3 + a]) - ord2f(bounds[12 * seg + a]));
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float lo = ord2f(bounds[12 * seg + a]);
    float t = ext > 0.f ? (c[a] - lo) / ext : 0.f;
    t = fminf(fmaxf(t, 0.f), 1.f);
    q[a] = min((uint32_t)(t * cells), (1u << bpa) - 1u);
  }
  uint64_t code = (expand21(q[0]) << 2) | (expand21(q[1]) << 1) | expand21(q[2]);
  keys[i] = ((uint64_t)seg << (3 * bpa)) | code;
  vals[i] = (uint32_t)i;
}

// Common-prefix length of sorted keys i and j inside [a, b), extended by the positions when the keys are equal
// (Karras 2012); -1 outside the segment.
__device__ __forceinline__ int kdelta(uint64_t const * __restrict__ codes, int64_t a, int64_t b, int64_t i, int64_t j) {
  if (j < a || j >= b) return -1;
  uint64_t x = codes[i], y = codes[j];
  if (x == y) return 64 + __clzll((long long)(i ^ j));
  return __clzll((long long)(x ^ y));
}

// Binary radix trees, one per segment. The internal node at sorted position i of segment s lives in slot i - s.
// Child codes: >= 0 an internal slot, < 0 a leaf at sorted position ~code.
__global__ void karras_kernel(uint64_t const * __restrict__ codes, int64_t n, int64_t const * __restrict__ seg_start,
                              int M, int mbits, int * __restrict__ left, int * __restrict__ right,
                              int * __restrict__ first, int * __restrict__ last, int * __restrict__ parent,
                              int * __restrict__ leaf_parent, unsigned * __restrict__ visits) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int s = M > 1 ? (int)(codes[i] >> mbits) : 0;
  int64_t a = M > 1 ? seg_start[s] : 0, b = M > 1 ? seg_start[s + 1] : n;
  if (b - a == 1) leaf_parent[i] = -1;  // no internal node
  if (i >= b - 1) return;  // a segment of m elements has m - 1 internal nodes, at positions a .. b - 2
  visits[i - s] = 0;
  if (i == a) parent[i - s] = -1;  // the segment's root
  int d = (kdelta(codes, a, b, i, i + 1) - kdelta(codes, a, b, i, i - 1)) >= 0 ? 1 : -1;
  int dmin = kdelta(codes, a, b, i, i - d);
  int64_t lmax = 2;
  while (kdelta(codes, a, b, i, i + lmax * d) > dmin) lmax <<= 1;
  int64_t l = 0;
  for (int64_t t = lmax >> 1; t >= 1; t >>= 1)
    if (kdelta(codes, a, b, i, i + (l + t) * d) > dmin) l += t;
  int64_t j = i + l * d;
  int dnode = kdelta(codes, a, b, i, j);
  int64_t sp = 0, t = l;
  do {
    t = (t + 1) >> 1;
    if (kdelta(codes, a, b, i, i + (sp + t) * d) > dnode) sp += t;
  } while (t > 1);
  int64_t gamma = i + sp * d + (d < 0 ? -1 : 0);
  int64_t lo = i < j ? i : j, hi = i < j ? j : i;
  int slot = (int)(i - s);
  int lc = (lo == gamma) ? ~(int)gamma : (int)(gamma - s);
  int rc = (hi == gamma + 1) ? ~(int)(gamma + 1) : (int)(gamma + 1 - s);
  left[slot] = lc;
  right[slot] = rc;
  first[slot] = (int)lo;
  last[slot] = (int)hi;
  if (lc < 0) leaf_parent[~lc] = slot; else parent[lc] = slot;
  if (rc < 0) leaf_parent[~rc] = slot; else parent[rc] = slot;
}

__device__ __forceinline__ void child_box(int code, float4 const * __restrict__ elo, float4 const * __restrict__ ehi,
                                          uint32_t const * __restrict__ sorted, float4 const * ilo, float4 const * ihi,
                                          float4 & lo, float4 & hi) {
  if (code < 0) {
    uint32_t e = sorted[~code];
    lo = elo[e];
    hi = ehi[e];
  } else {
    lo = __ldcg(ilo + code);
    hi = __ldcg(ihi + code);
  }
}

__device__ __forceinline__ float half_area(float4 lo, float4 hi) {
  float x = hi.x - lo.x, y = hi.y - lo.y, z = hi.z - lo.z;
  return x * y + y * z + z * x;
}

// Bottom-up refit: the second thread to reach a node merges its two children and continues upwards.
__global__ void refit_kernel(int64_t n, int const * __restrict__ left, int const * __restrict__ right,
                             int const * __restrict__ first, int const * __restrict__ last,
                             int const * __restrict__ parent, int const * __restrict__ leaf_parent,
                             float4 const * __restrict__ elo, float4 const * __restrict__ ehi,
                             uint32_t const * __restrict__ sorted, float4 * ilo, float4 * ihi,
                             unsigned * __restrict__ visits) {
  int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  int p = leaf_parent[s];
  while (p >= 0) {
    __threadfence();
    unsigned old = atomicAdd(&visits[p], 1u);
    if (old == 0) return;
    float4 al, ah, bl, bh;
    child_box(left[p], elo, ehi, sorted, ilo, ihi, al, ah);
    child_box(right[p], elo, ehi, sorted, ilo, ihi, bl, bh);
    // the box, with its half area in lo.w and the number of elements in hi.w
    float4 lo = make_float4(fminf(al.x, bl.x), fminf(al.y, bl.y), fminf(al.z, bl.z), 0.f);
    float4 hi = make_float4(fmaxf(ah.x, bh.x), fmaxf(ah.y, bh.y), fmaxf(ah.z, bh.z), 0.f);
    lo.w = half_area(lo, hi);
    hi.w = __int_as_float(last[p] - first[p] + 1);
    __stcg(ilo + p, lo);
    __stcg(ihi + p, hi);
    p = parent[p];
  }
}

struct CollapseArgs {
  int const * left;
  int const * right;
  int const * first;
  int const * last;
  float4 const * elo;
  float4 const * ehi;
  uint32_t const * sorted;
  float4 const * ilo;
  float4 const * ihi;
  int64_t const * seg_start;  // sorted position where each segment starts (nullptr: one segment)
  int M;
  int leaf_size;
};

__device__ __forceinline__ int code_count(CollapseArgs const & a, int code) {
  return code < 0 ? 1 : __float_as_int(a.ihi[code].w);
}
__device__ __forceinline__ int code_first(CollapseArgs const & a, int code) { return code < 0 ? ~code : a.first[code]; }

// The level being collapsed, kept on the device so that all levels run between two host synchronisations: its frontier
// size, the wide index of its first node, and the number of levels emitted so far.
struct CollapseLevel {
  int64_t fsize;
  int64_t base;
  int64_t levels;
  int64_t overflow;  // set if a node would have landed past the node bound (never, by the bound's construction)
};

// The W binary subtrees that become the children of frontier node f's wide node: starting from its two children,
// repeatedly open the subtree with the largest surface area among those too big to be a leaf. Returns how many are
// internal.
template <int W>
__device__ __forceinline__ int collapse_decide_one(CollapseArgs const & a, int const * __restrict__ frontier, int64_t f,
                                                   int * __restrict__ chosen) {
  int b = frontier[f];
  int codes[W];
  float area[W];  // of the subtrees too big to be a leaf; negative otherwise
  auto put = [&](int e, int code) {
    codes[e] = code;
    bool big = code >= 0 && __float_as_int(a.ihi[code].w) > a.leaf_size;
    area[e] = big ? a.ilo[code].w : -1.f;
    if (big && !(area[e] >= 0.f)) area[e] = 0.f;  // (a NaN or negative area still opens, last)
  };
#pragma unroll
  for (int e = 0; e < W; ++e) codes[e] = CHILD_EMPTY, area[e] = -1.f;
  put(0, a.left[b]);
  put(1, a.right[b]);
#pragma unroll
  for (int ne = 2; ne < W; ++ne) {
    int best = -1, code = CHILD_EMPTY;
    float best_sa = -1.f;
#pragma unroll
    for (int e = 0; e < W; ++e)
      if (e < ne && area[e] > best_sa) best_sa = area[e], best = e, code = codes[e];
    if (best < 0) break;
    int l = a.left[code], r = a.right[code];
#pragma unroll
    for (int e = 0; e < W; ++e)
      if (e == best) put(e, l);
    put(ne, r);
  }
  int nint = 0;
#pragma unroll
  for (int e = 0; e < W; ++e) {
    chosen[f * W + e] = codes[e];
    nint += area[e] >= 0.f ? 1 : 0;
  }
  return nint;
}

// A level takes two launches: every frontier node's children decided, with the internal ones counted per block (offs: the
// node's place among its block's, tot: the block's count); then the wide nodes written, the internal children placed
// after those of the blocks before (summed here from tot, or read from `scanned` when there are too many blocks). The
// numbering is the frontier's order, whatever order the blocks run in. The state for the next level goes to `next`.
template <int W>
__global__ void __launch_bounds__(BUILD_THREADS)
collapse_decide_kernel(CollapseArgs a, int const * __restrict__ frontier, CollapseLevel const * __restrict__ lv,
                       int * __restrict__ chosen, int * __restrict__ offs, int * __restrict__ tot) {
  int64_t fsize = lv->fsize;
  int64_t f0 = (int64_t)blockIdx.x * BUILD_THREADS;
  if (f0 >= fsize) {
    if (threadIdx.x == 0) tot[blockIdx.x] = 0;
    return;
  }
  int64_t f = f0 + threadIdx.x;
  int nint = f < fsize ? collapse_decide_one<W>(a, frontier, f, chosen) : 0;
  int total;
  int off = block_exclusive_scan<int>(nint, total);
  if (f < fsize) offs[f] = off;
  if (threadIdx.x == 0) tot[blockIdx.x] = total;
}

// Pad a box outwards by a relative margin of its coordinates' magnitude, so that rounding in element distances and hit
// times can never make an element that lies inside the box look closer than the box.
__device__ __forceinline__ void pad_box(float4 & lo, float4 & hi) {
  float const R = 1.0f / 1048576.0f;  // 2^-20
  float px = (fabsf(lo.x) + fabsf(hi.x)) * R, py = (fabsf(lo.y) + fabsf(hi.y)) * R, pz = (fabsf(lo.z) + fabsf(hi.z)) * R;
  lo.x -= px; lo.y -= py; lo.z -= pz;
  hi.x += px; hi.y += py; hi.z += pz;
}

template <int W> __device__ __forceinline__ void clear_node(WideNode<W> & node) {
#pragma unroll
  for (int e = 0; e < W; ++e) {
    node.lox[e] = node.loy[e] = node.loz[e] = INFINITY;
    node.hix[e] = node.hiy[e] = node.hiz[e] = -INFINITY;
    node.child[e] = CHILD_EMPTY;
  }
#pragma unroll
  for (int e = 0; e < (W == 4 ? 4 : 8); ++e) node.pad[e] = 0;
}

// Writes frontier node f's wide node (level_base + f) and appends its internal children to the next frontier at
// offset `off` (their wide indices next_base + off + k); false if a node would land past the node bound
template <int W>
__device__ __forceinline__ bool collapse_emit_one(CollapseArgs const & a, int const * __restrict__ frontier, int64_t f,
                                                  int const * __restrict__ chosen, int off, int64_t level_base,
                                                  int64_t next_base, int64_t cap, WideNode<W> * __restrict__ nodes,
                                                  int * __restrict__ next_frontier) {
  if (level_base + f >= cap) return false;
  WideNode<W> node;
  clear_node(node);
  int k = 0;
  // leaves store their first element relative to the segment's first sorted position
  int64_t seg_base = 0;
  if (a.M > 1) {
    int64_t pos = a.first[frontier[f]];
    seg_base = a.seg_start[segment_of(a.seg_start, a.M, pos)];
  }
#pragma unroll
  for (int e = 0; e < W; ++e) {
    int code = chosen[f * W + e];
    if (code == CHILD_EMPTY) continue;
    float4 lo, hi;
    child_box(code, a.elo, a.ehi, a.sorted, a.ilo, a.ihi, lo, hi);
    pad_box(lo, hi);
    node.lox[e] = lo.x; node.loy[e] = lo.y; node.loz[e] = lo.z;
    node.hix[e] = hi.x; node.hiy[e] = hi.y; node.hiz[e] = hi.z;
    int cnt = code_count(a, code);
    if (cnt <= a.leaf_size) {
      node.child[e] = encode_leaf((int)(code_first(a, code) - seg_base), cnt);
    } else {
      if (next_base + off + k >= cap) return false;
      node.child[e] = (int)(next_base + off + k);
      next_frontier[off + k] = code;
      ++k;
    }
  }
  nodes[level_base + f] = node;
  return true;
}

template <int W>
__global__ void __launch_bounds__(BUILD_THREADS)
collapse_emit_kernel(CollapseArgs a, int const * __restrict__ frontier, int * __restrict__ next_frontier,
                     CollapseLevel const * __restrict__ lv, CollapseLevel * __restrict__ next,
                     int const * __restrict__ chosen, int const * __restrict__ offs, int const * __restrict__ tot,
                     int const * __restrict__ scanned, int64_t cap, WideNode<W> * __restrict__ nodes) {
  __shared__ int s_sum[BUILD_THREADS / 32];
  int64_t fsize = lv->fsize;
  int64_t f0 = (int64_t)blockIdx.x * BUILD_THREADS;
  if (f0 >= fsize && blockIdx.x > 0) return;
  int64_t level_base = lv->base;
  int nb = (int)ceil_div(fsize, BUILD_THREADS);
  // internal children of the blocks before this one; block 0 sums all of them instead, for the next level's size
  int sum = 0;
  if (scanned) {
    if (threadIdx.x == 0) sum = blockIdx.x > 0 ? scanned[blockIdx.x] : (nb > 0 ? scanned[nb - 1] + tot[nb - 1] : 0);
  } else {
    int upto = blockIdx.x > 0 ? (int)blockIdx.x : nb;
    for (int i = threadIdx.x; i < upto; i += BUILD_THREADS) sum += tot[i];
  }
  sum = __reduce_add_sync(0xffffffffu, sum);
  if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = sum;
  __syncthreads();
  sum = 0;
#pragma unroll
  for (int w = 0; w < BUILD_THREADS / 32; ++w) sum += s_sum[w];
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) {
      next->fsize = sum;
      next->base = level_base + fsize;
      next->levels = lv->levels + (fsize > 0 ? 1 : 0);
      if (lv->overflow) atomicOr((unsigned long long *)&next->overflow, 1ull);
    }
    sum = 0;
  }
  int64_t f = f0 + threadIdx.x;
  if (f >= fsize) return;
  if (!collapse_emit_one<W>(a, frontier, f, chosen, sum + offs[f], level_base, level_base + fsize, cap, nodes,
                            next_frontier))
    atomicOr((unsigned long long *)&next->overflow, 1ull);
}

// Segment roots: big segments (more elements than a leaf) become level-0 frontier entries; small non-empty segments get
// a single-leaf root node. Small roots take wide indices [0, num_small), big roots [num_small, num_small + num_big).
__global__ void segment_flags_kernel(int64_t const * __restrict__ seg_start, int M, int64_t n, int leaf_size,
                                     int * __restrict__ is_small, int * __restrict__ is_big) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= M) return;
  int64_t a = seg_start ? seg_start[s] : 0, b = seg_start ? seg_start[s + 1] : n;
  int64_t cnt = b - a;
  is_small[s] = (cnt >= 1 && cnt <= leaf_size) ? 1 : 0;
  is_big[s] = cnt > leaf_size ? 1 : 0;
}

template <int W>
__device__ __forceinline__ void write_leaf_root(WideNode<W> & out, int const * __restrict__ bounds, int count) {
  WideNode<W> node;
  clear_node(node);
  float4 lo = make_float4(ord2f(bounds[6]), ord2f(bounds[7]), ord2f(bounds[8]), 0.f);
  float4 hi = make_float4(ord2f(bounds[9]), ord2f(bounds[10]), ord2f(bounds[11]), 0.f);
  pad_box(lo, hi);
  node.lox[0] = lo.x; node.loy[0] = lo.y; node.loz[0] = lo.z;
  node.hix[0] = hi.x; node.hiy[0] = hi.y; node.hiz[0] = hi.z;
  node.child[0] = encode_leaf(0, count);
  out = node;
}

// Level 0 of one segment: its root, or the only node when everything fits in a leaf
template <int W>
__global__ void single_root_kernel(int64_t n, int leaf_size, int const * __restrict__ bounds,
                                   WideNode<W> * __restrict__ nodes, int * __restrict__ frontier,
                                   int * __restrict__ seg_root, CollapseLevel * __restrict__ lv) {
  bool big = n > leaf_size;
  if (!big) write_leaf_root<W>(nodes[0], bounds, (int)n);
  frontier[0] = 0;  // the binary root
  seg_root[0] = 0;
  lv[0] = CollapseLevel{big ? 1 : 0, big ? 0 : 1, 0, 0};
  lv[1].overflow = 0;
}

template <int W>
__global__ void segment_roots_kernel(CollapseArgs a, int64_t n, int const * __restrict__ is_small,
                                     int const * __restrict__ small_rank, int const * __restrict__ is_big,
                                     int const * __restrict__ big_rank, int const * __restrict__ bounds,
                                     WideNode<W> * __restrict__ nodes, int * __restrict__ frontier,
                                     int * __restrict__ seg_root, CollapseLevel * __restrict__ lv) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= a.M) return;
  int num_small = small_rank[a.M - 1] + is_small[a.M - 1];
  if (s == 0) {
    lv[0] = CollapseLevel{big_rank[a.M - 1] + is_big[a.M - 1], num_small, 0, 0};
    lv[1].overflow = 0;
  }
  int64_t sa = a.seg_start[s], sb = a.seg_start[s + 1];
  if (is_big[s]) {
    // the Karras root of the segment is the internal node at its first position, slot sa - s
    frontier[big_rank[s]] = (int)(sa - s);
    seg_root[s] = num_small + big_rank[s];
  } else if (is_small[s]) {
    write_leaf_root<W>(nodes[small_rank[s]], bounds + 12 * (int64_t)s, (int)(sb - sa));
    seg_root[s] = small_rank[s];
  } else {
    seg_root[s] = -1;  // empty segment
  }
}

__global__ void count_big_kernel(int const * __restrict__ first, int const * __restrict__ last, int64_t m, int leaf_size,
                                 unsigned long long * __restrict__ out) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool big = i < m && (last[i] - first[i] + 1) > leaf_size;
  unsigned b = __ballot_sync(0xffffffffu, big);
  if ((threadIdx.x & 31) == 0 && b) atomicAdd(out, (unsigned long long)__popc(b));
}

// Element records in sorted order; the stored index is the element's index within its segment.
__global__ void mesh_records_kernel(float const * __restrict__ V, int64_t nv, int32_t const * __restrict__ F, int64_t n,
                                    int64_t const * __restrict__ seg_start, int M, uint32_t const * __restrict__ sorted,
                                    float4 * __restrict__ cp_rec, float4 * __restrict__ ray_rec,
                                    int32_t * __restrict__ leaf_to_elem) {
  int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  int64_t ge = (int64_t)sorted[s];
  int e = (int)(M > 1 ? ge - seg_start[segment_of(seg_start, M, ge)] : ge);
  leaf_to_elem[s] = e;
  bool out = false;  // (reported by elem_box_kernel)
  V3 v0 = load_v3(V + 3 * face_vertex(F, 3 * ge, nv, out));
  V3 v1 = load_v3(V + 3 * face_vertex(F, 3 * ge + 1, nv, out));
  V3 v2 = load_v3(V + 3 * face_vertex(F, 3 * ge + 2, nv, out));
  if (cp_rec) {
    TriPlane pl = tri_plane(v0, v1, v2);
    V3 d0, d1, d2;
    float l0, l1, l2;
    edge_dir(v0, v1, d0, l0);
    edge_dir(v1, v2, d1, l1);
    edge_dir(v2, v0, d2, l2);
    float4 * r = cp_rec + s * CP_REC_F4;
    r[0] = make_float4(v0.x, v0.y, v0.z, pl.dist);
    r[1] = make_float4(v1.x, v1.y, v1.z, l0);
    r[2] = make_float4(v2.x, v2.y, v2.z, l1);
    r[3] = make_float4(pl.normal.x, pl.normal.y, pl.normal.z, __int_as_float(pl.axis));
    r[4] = make_float4(d0.x, d0.y, d0.z, l2);
    r[5] = make_float4(d1.x, d1.y, d1.z, __int_as_float(e));
    r[6] = make_float4(d2.x, d2.y, d2.z, pl.area);
    r[7] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (ray_rec) {
    V3 e01 = v1 - v0, e02 = v2 - v0;
    float4 * r = ray_rec + s * RAY_REC_F4;
    r[0] = make_float4(v0.x, v0.y, v0.z, __int_as_float(e));
    r[1] = make_float4(e01.x, e01.y, e01.z, 0.f);
    r[2] = make_float4(e02.x, e02.y, e02.z, 0.f);
  }
}

__global__ void point_records_kernel(float const * __restrict__ P, int64_t n, int64_t const * __restrict__ seg_start,
                                     int M, uint32_t const * __restrict__ sorted, float4 * __restrict__ pt_rec,
                                     int32_t * __restrict__ leaf_to_elem) {
  int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  int64_t ge = (int64_t)sorted[s];
  int e = (int)(M > 1 ? ge - seg_start[segment_of(seg_start, M, ge)] : ge);
  leaf_to_elem[s] = e;
  V3 p = load_v3(P + 3 * ge);
  pt_rec[s] = make_float4(p.x, p.y, p.z, __int_as_float(e));
}

// Blocks of a level up to which the emitting kernel sums the counts of the blocks before it by itself
constexpr int64_t COLLAPSE_SUM_BLOCKS = 1024;
// Elements up to which the node array is first sized by the worst case and the nodes copied out; larger builds count their
// nodes first, at the price of one more synchronisation and of a larger array in the handle (the count bounds them too, but
// less tightly). The worst case takes 107 bytes an element at width 4 and 165 at width 8 (leaves of one): 224 and 346 MB of
// scratch at this line, which the scratch pool keeps mapped (with a line at 4,194,304 elements 447 and 690). Counted, the
// array of a 2,093,058-triangle mesh made its build 7.6 ms instead of 6.9.
constexpr int64_t COLLAPSE_BOUND_MAX = 1 << 21;

// What the build reads back, in one copy: the collapse's two alternating levels, whether a face index was out of range,
// and the bounds of every segment (12 ordered ints each, see elem_box_kernel)
struct BuildState {
  CollapseLevel level[2];
  int bad;
  int pad[3];
  __host__ __device__ int * bounds() { return reinterpret_cast<int *>(this + 1); }
  static size_t bytes(int M) { return sizeof(BuildState) + (size_t)12 * M * sizeof(int); }
};

template <int W>
void collapse(thea_bvh * b, CollapseArgs const & a, int64_t n, BuildState * state, std::vector<char> & h_state,
              cudaStream_t stream) {
  int M = a.M;
  // Wide nodes: every one but a small segment's root stands for a binary node with more elements than a leaf holds. At
  // most one per leaf + 1 elements has fewer than W children, all of them leaves; the others have W, so there are at most
  // (n - 1) / (W - 1) of them.
  int64_t cap = (n - 1) / (W - 1) + n / (a.leaf_size + 1) + M + 1;
  bool exact = n > COLLAPSE_BOUND_MAX;
  if (exact) {
    int64_t m = n - M;  // binary internal nodes in the forest (segments are non-empty)
    Scratch cnt(sizeof(unsigned long long), stream);
    THEA_CUDA_CHECK(cudaMemsetAsync(cnt.ptr, 0, cnt.bytes, stream));
    if (m > 0)
      THEA_LAUNCH(count_big_kernel, (unsigned)ceil_div(m, BUILD_THREADS), BUILD_THREADS, 0, stream, a.first, a.last, m,
                  a.leaf_size, cnt.as<unsigned long long>());
    unsigned long long nbig = 0;
    THEA_CUDA_CHECK(cudaMemcpyAsync(&nbig, cnt.ptr, sizeof(nbig), cudaMemcpyDeviceToHost, stream));
    THEA_CUDA_CHECK(cudaStreamSynchronize(stream));
    cap = std::min<int64_t>(cap, (int64_t)nbig + M);
  }
  Scratch bound_nodes;
  WideNode<W> * nodes = nullptr;
  if (exact) {
    THEA_CUDA_CHECK(thea_malloc_async((void **)&nodes, (size_t)cap * sizeof(WideNode<W>), stream));
    b->nodes = nodes;
  } else {
    bound_nodes = Scratch((size_t)cap * sizeof(WideNode<W>), stream);
    nodes = bound_nodes.as<WideNode<W>>();
  }
  THEA_CUDA_CHECK(thea_malloc_async((void **)&b->seg_root, (size_t)M * sizeof(int32_t), stream));
  int64_t blocks_cap = ceil_div(cap, BUILD_THREADS);
  Scratch fr((size_t)cap * 2 * sizeof(int), stream), chosen((size_t)cap * W * sizeof(int), stream);
  Scratch offs((size_t)cap * sizeof(int), stream), tot((size_t)blocks_cap * 2 * sizeof(int), stream);
  int * frontier[2] = {fr.as<int>(), fr.as<int>() + cap};
  CollapseLevel * level = state->level;  // (device addresses)
  int const * d_bounds = state->bounds();
  if (M == 1) {
    THEA_LAUNCH(single_root_kernel<W>, 1, 1, 0, stream, n, a.leaf_size, d_bounds, nodes, frontier[0], b->seg_root, level);
  } else {
    Scratch is_small((size_t)M * sizeof(int), stream), is_big((size_t)M * sizeof(int), stream);
    Scratch small_rank((size_t)M * sizeof(int), stream), big_rank((size_t)M * sizeof(int), stream);
    THEA_LAUNCH(segment_flags_kernel, (unsigned)ceil_div(M, BUILD_THREADS), BUILD_THREADS, 0, stream, a.seg_start, M, n,
                a.leaf_size, is_small.as<int>(), is_big.as<int>());
    exclusive_scan<int>(is_small.as<int>(), small_rank.as<int>(), M, stream);
    exclusive_scan<int>(is_big.as<int>(), big_rank.as<int>(), M, stream);
    THEA_LAUNCH((segment_roots_kernel<W>), (unsigned)ceil_div(M, BUILD_THREADS), BUILD_THREADS, 0, stream, a, n,
                is_small.as<int>(), small_rank.as<int>(), is_big.as<int>(), big_rank.as<int>(), d_bounds, nodes,
                frontier[0], b->seg_root, level);
  }
  // As many levels as a balanced tree and a few more, then the state is read; a deeper tree takes further rounds. Levels
  // past the last one find an empty frontier and do nothing.
  int64_t bound = M;
  int run = 4;
  for (int64_t m = n / M; m > a.leaf_size; m /= W) ++run;
  CollapseLevel h{0, 0, 0, 0};
  int par = 0;
  do {
    for (int l = 0; l < run; ++l) {
      unsigned grid = (unsigned)ceil_div(bound, BUILD_THREADS);
      int * scanned = grid > COLLAPSE_SUM_BLOCKS ? tot.as<int>() + blocks_cap : nullptr;
      THEA_LAUNCH(collapse_decide_kernel<W>, grid, BUILD_THREADS, 0, stream, a, frontier[par], level + par,
                  chosen.as<int>(), offs.as<int>(), tot.as<int>());
      if (scanned) exclusive_scan<int>(tot.as<int>(), scanned, grid, stream);
      THEA_LAUNCH(collapse_emit_kernel<W>, grid, BUILD_THREADS, 0, stream, a, frontier[par], frontier[par ^ 1],
                  level + par, level + (par ^ 1), chosen.as<int>(), offs.as<int>(), tot.as<int>(), scanned, cap, nodes);
      bound = std::min<int64_t>(bound * W, cap);
      par ^= 1;
    }
    THEA_CUDA_CHECK(cudaMemcpyAsync(h_state.data(), state, h_state.size(), cudaMemcpyDeviceToHost, stream));
    THEA_CUDA_CHECK(cudaStreamSynchronize(stream));
    BuildState hs;
    memcpy(&hs, h_state.data(), sizeof(hs));
    h = hs.level[par];
    THEA_REQUIRE(!hs.bad, "build: a face index lies outside [0, num_vertices)");
    THEA_REQUIRE(!h.overflow, "BVH collapse exceeded its node bound");
    run = 8;
  } while (h.fsize > 0);
  if (!exact) {
    THEA_CUDA_CHECK(thea_malloc_async(&b->nodes, (size_t)h.base * sizeof(WideNode<W>), stream));
    THEA_CUDA_CHECK(cudaMemcpyAsync(b->nodes, nodes, (size_t)h.base * sizeof(WideNode<W>), cudaMemcpyDeviceToDevice,
                                    stream));
  }
  b->num_nodes = h.base;
  b->depth = (int)std::max<int64_t>(1, h.levels);
}

}  // namespace

thea_bvh * build_forest(bool is_mesh, float const * V, int64_t nv, int32_t const * F, int64_t n_elems,
                        int64_t const * seg_start_host, int M, thea_build_config const & cfg, cudaStream_t stream) {
  int64_t n = is_mesh ? n_elems : nv;
  THEA_REQUIRE(M >= 1, "build: at least one segment is required");
  THEA_REQUIRE(n >= 1, "build: at least one element is required");
  THEA_REQUIRE(n < (int64_t(1) << 31) - 1, "build: at most 2^31 - 2 elements per forest");
  int width = cfg.width == 0 ? 4 : cfg.width;
  THEA_REQUIRE(width == 4 || width == 8, "build: width must be 4 or 8");
  int leaf = cfg.max_leaf_size == 0 ? (is_mesh ? 2 : 1) : cfg.max_leaf_size;
  THEA_REQUIRE(leaf >= 1 && leaf <= MAX_LEAF_SIZE, "build: max_leaf_size must be in 1..16");
  uint32_t layouts = is_mesh ? (cfg.layouts == 0 ? (THEA_LAYOUT_CLOSEST | THEA_LAYOUT_RAY) : cfg.layouts) : 0u;
  THEA_REQUIRE((layouts & ~3u) == 0, "build: unknown layout bits");
  std::vector<int64_t> starts;
  if (M > 1) {
    THEA_REQUIRE(seg_start_host, "build: segment starts are required for more than one segment");
    starts.assign(seg_start_host, seg_start_host + M + 1);
    THEA_REQUIRE(starts[0] == 0 && starts[M] == n, "build: segment starts must run from 0 to the element count");
    for (int s = 0; s < M; ++s) {
      THEA_REQUIRE(starts[s + 1] > starts[s], "build: every segment must hold at least one element");
      THEA_REQUIRE(starts[s + 1] - starts[s] < (int64_t(1) << 27), "build: at most 2^27 - 1 elements per segment");
    }
  } else {
    THEA_REQUIRE(n < (int64_t(1) << 27), "build: at most 2^27 - 1 elements per BVH");
    starts = {0, n};
  }

  THEA_REQUIRE(!is_mesh || nv > 0, "build: a face index lies outside [0, num_vertices)");

  thea_bvh * b = new thea_bvh;
  try {
    THEA_CUDA_CHECK(cudaGetDevice(&b->device));
    b->is_mesh = is_mesh ? 1 : 0;
    b->width = width;
    b->leaf_size = leaf;
    b->layouts = layouts;
    b->query_order = cfg.query_order;
    b->n = n;
    b->num_segments = M;
    b->seg_start_host = starts;

    THEA_CUDA_CHECK(thea_malloc_async((void **)&b->seg_start, (size_t)(M + 1) * sizeof(int64_t), stream));
    THEA_CUDA_CHECK(thea_malloc_async((void **)&b->err, sizeof(unsigned), stream));
    b->err_host = take_host_word();
    if (M > 1)
      THEA_CUDA_CHECK(cudaMemcpyAsync(b->seg_start, starts.data(), (size_t)(M + 1) * sizeof(int64_t),
                                      cudaMemcpyHostToDevice, stream));
    int64_t const * seg = b->seg_start;

    Scratch elo((size_t)n * sizeof(float4), stream), ehi((size_t)n * sizeof(float4), stream);
    Scratch state_buf(BuildState::bytes(M), stream);
    BuildState * state = state_buf.as<BuildState>();
    int * bounds = state->bounds();
    THEA_LAUNCH(build_init_kernel, (unsigned)ceil_div(12 * (int64_t)M, BUILD_THREADS), BUILD_THREADS, 0, stream,
                bounds, M, &state->bad, b->err, b->seg_start, n);
    unsigned grid = (unsigned)ceil_div(n, BUILD_THREADS);
    THEA_LAUNCH(elem_box_kernel, grid, BUILD_THREADS, 0, stream, V, nv, F, n, is_mesh ? 1 : 0, seg, M, elo.as<float4>(),
                ehi.as<float4>(), bounds, &state->bad);

    int segbits = 0;
    while ((int64_t(1) << segbits) < M) ++segbits;
    int bpa = std::min(21, (63 - segbits) / 3);
    int mbits = 3 * bpa;
    Scratch keys((size_t)n * sizeof(uint64_t), stream), vals((size_t)n * sizeof(uint32_t), stream);
    THEA_LAUNCH(morton_kernel, grid, BUILD_THREADS, 0, stream, elo.as<float4>(), ehi.as<float4>(), n, seg, M,
                bounds, bpa, keys.as<uint64_t>(), vals.as<uint32_t>());
    radix_sort_pairs(keys.as<uint64_t>(), vals.as<uint32_t>(), n, mbits + segbits, stream, /*probe_passes=*/false);

    int64_t m = n - M;  // binary internal nodes
    size_t mm = (size_t)std::max<int64_t>(m, 1);
    Scratch left(mm * sizeof(int), stream), right(mm * sizeof(int), stream);
    Scratch first(mm * sizeof(int), stream), last(mm * sizeof(int), stream);
    Scratch parent(mm * sizeof(int), stream), leaf_parent((size_t)n * sizeof(int), stream);
    Scratch ilo(mm * sizeof(float4), stream), ihi(mm * sizeof(float4), stream);
    Scratch visits(mm * sizeof(unsigned), stream);
    if (m >= 1) {
      THEA_LAUNCH(karras_kernel, grid, BUILD_THREADS, 0, stream, keys.as<uint64_t>(), n, seg, M, mbits,
                  left.as<int>(), right.as<int>(), first.as<int>(), last.as<int>(), parent.as<int>(),
                  leaf_parent.as<int>(), visits.as<unsigned>());
      THEA_LAUNCH(refit_kernel, grid, BUILD_THREADS, 0, stream, n, left.as<int>(), right.as<int>(), first.as<int>(),
                  last.as<int>(), parent.as<int>(), leaf_parent.as<int>(), elo.as<float4>(), ehi.as<float4>(), vals.as<uint32_t>(), ilo.as<float4>(),
                  ihi.as<float4>(), visits.as<unsigned>());
    }
    CollapseArgs a{left.as<int>(), right.as<int>(), first.as<int>(), last.as<int>(), elo.as<float4>(),
                   ehi.as<float4>(), vals.as<uint32_t>(), ilo.as<float4>(), ihi.as<float4>(),
                   M > 1 ? seg : nullptr, M, leaf};
    std::vector<char> h_state(BuildState::bytes(M));
    if (width == 4) collapse<4>(b, a, n, state, h_state, stream);
    else collapse<8>(b, a, n, state, h_state, stream);
    std::vector<int> hb((size_t)12 * M);
    memcpy(hb.data(), h_state.data() + sizeof(BuildState), hb.size() * sizeof(int));
    int64_t node_bytes = b->num_nodes * (width == 4 ? (int64_t)sizeof(WideNode<4>) : (int64_t)sizeof(WideNode<8>));

    int need = b->depth * (width - 1) + 1;
    if (need > (width == 4 ? 256 : 512))
      throw Error(THEA_ERR_NOT_SUPPORTED, "build: tree too deep for the traversal stack (depth " +
                                              std::to_string(b->depth) + ")");
    THEA_CUDA_CHECK(thea_malloc_async((void **)&b->leaf_to_elem, (size_t)n * sizeof(int32_t), stream));
    int64_t rec_bytes = n * (int64_t)sizeof(int32_t);
    if (is_mesh) {
      if (layouts & THEA_LAYOUT_CLOSEST) {
        THEA_CUDA_CHECK(thea_malloc_async((void **)&b->cp_rec, (size_t)n * CP_REC_F4 * sizeof(float4), stream));
        rec_bytes += n * CP_REC_F4 * (int64_t)sizeof(float4);
      }
      if (layouts & THEA_LAYOUT_RAY) {
        THEA_CUDA_CHECK(thea_malloc_async((void **)&b->ray_rec, (size_t)n * RAY_REC_F4 * sizeof(float4) + RAY_REC_PAD,
                                          stream));
        rec_bytes += n * RAY_REC_F4 * (int64_t)sizeof(float4);
      }
      THEA_LAUNCH(mesh_records_kernel, grid, BUILD_THREADS, 0, stream, V, nv, F, n, seg, M, vals.as<uint32_t>(),
                  b->cp_rec, b->ray_rec, b->leaf_to_elem);
    } else {
      THEA_CUDA_CHECK(thea_malloc_async((void **)&b->pt_rec, (size_t)n * sizeof(float4), stream));
      rec_bytes += n * (int64_t)sizeof(float4);
      THEA_LAUNCH(point_records_kernel, grid, BUILD_THREADS, 0, stream, V, n, seg, M, vals.as<uint32_t>(), b->pt_rec,
                  b->leaf_to_elem);
    }
    b->seg_lo.resize((size_t)3 * M);
    b->seg_hi.resize((size_t)3 * M);
    for (int s = 0; s < M; ++s)
      for (int t = 0; t < 3; ++t) {
        b->seg_lo[3 * s + t] = ord2f(hb[12 * s + 6 + t]);
        b->seg_hi[3 * s + t] = ord2f(hb[12 * s + 9 + t]);
      }
    for (int t = 0; t < 3; ++t) {
      b->lo[t] = b->seg_lo[t];
      b->hi[t] = b->seg_hi[t];
      for (int s = 1; s < M; ++s) {
        b->lo[t] = std::min(b->lo[t], b->seg_lo[3 * s + t]);
        b->hi[t] = std::max(b->hi[t], b->seg_hi[3 * s + t]);
      }
    }
    b->device_bytes = node_bytes + rec_bytes;
    init_segment_roots(b, stream);
    init_slabs(b, stream);
    THEA_CUDA_CHECK(cudaStreamSynchronize(stream));
    if (b->slabs) b->device_bytes += b->num_nodes * width * (int64_t)sizeof(float4);
    return b;
  } catch (...) {
    cudaStreamSynchronize(stream);
    destroy_bvh(b);
    throw;
  }
}

//============================================================================================================================
// Oriented slabs of the child slots (slab_normal / slab_lower_bound in traverse_ops.cuh): n = the area-weighted mean of
// the slot's triangle normals (triangles with a non-finite normal or area left out; +z if the mean vanishes), encoded and
// decoded as the searches decode it, and the range of n . v over the slot's vertices, rounded outwards to float
// (slab_project, slab_range.cuh: the values of an FP64 evaluation at 19 us a pass for 81,920 triangles; FP64 itself took
// 64, most of it on the FP64 pipe). Slots with no elements get an empty slab. The sums of the normals are added in the order
// the lanes arrive, so a slab may differ from one build to the next, within its own rules; answers do not depend on it.
//
// Every element contributes to the slot of each of its ancestors, so both passes (normals, then ranges) run one thread
// per element, which climbs from its leaf's slot to the root. A warp's elements are neighbours in leaf order, hence
// share nearly all of their ancestors: the lanes climb level by level together, the lanes under one slot (a contiguous
// run) reduce with shuffles, and one lane per run issues the atomics. Work is n x depth spread evenly over the GPU.
// (One block per slot over the slot's whole run left the four slots of the root, a quarter of the mesh each, to four
// blocks: 646 us for 81,920 triangles, and 12 passes and three host synchronisations to find the runs; this form takes 54
// in all, six launches. A rebuild of that mesh with 16,384 queries: 2.67 -> 1.96 ms.)
//============================================================================================================================

constexpr int SLAB_MAX_LEVEL = 254;

// parent[i]: the slot (node * W + child) under which wide node i hangs; -2 - s for the root of segment s; -1 if none.
// A node array that does not follow the build's layout (a child before its parent, or under two slots) sets *bad.
template <int W>
__global__ void slab_parent_kernel(WideNode<W> const * __restrict__ nodes, int64_t num_nodes, int * __restrict__ parent,
                                   int * __restrict__ bad) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= num_nodes * W) return;
  int code = nodes[k / W].child[k % W];
  if (code < 0) return;  // a leaf or empty
  if ((int64_t)code >= num_nodes || (int64_t)code <= k / W || atomicCAS(&parent[code], -1, (int)k) != -1)
    atomicOr(bad, 1);
}

__global__ void slab_roots_kernel(int32_t const * __restrict__ seg_root, int M, int64_t num_nodes,
                                  int * __restrict__ parent, int * __restrict__ bad) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= M) return;
  int r = seg_root[s];
  if (r < 0 || (int64_t)r >= num_nodes || atomicCAS(&parent[r], -1, -2 - s) != -1) atomicOr(bad, 1);
}

// leaf_slot[k] / leaf_level[k]: the slot whose leaf holds the element at sorted position k, and its distance from the
// root (the root's own slots are level 0). The climb to the root gives the segment, to which leaf codes are relative.
template <int W>
__global__ void slab_leaf_kernel(WideNode<W> const * __restrict__ nodes, int64_t num_nodes,
                                 int const * __restrict__ parent, int64_t const * __restrict__ seg_start, int M,
                                 int64_t n, int * __restrict__ leaf_slot, uint8_t * __restrict__ leaf_level,
                                 int * __restrict__ bad) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= num_nodes * W) return;
  int code = nodes[k / W].child[k % W];
  if (code >= 0 || code == CHILD_EMPTY) return;
  int level = 0;
  int up = parent[k / W];
  while (up >= 0 && level < SLAB_MAX_LEVEL) {
    up = parent[up / W];
    ++level;
  }
  if (up > -2 || -2 - up >= M) {
    atomicOr(bad, 1);
    return;
  }
  int64_t a = seg_start[-2 - up], b = seg_start[-1 - up];
  int first, count;
  decode_leaf(code, first, count);
  if (a < 0 || b > n || first < 0 || a + first + count > b) {
    atomicOr(bad, 1);
    return;
  }
  for (int64_t e = a + first; e < a + first + count; ++e) {
    if (atomicCAS(&leaf_slot[e], -1, (int)k) != -1) atomicOr(bad, 1);
    leaf_level[e] = (uint8_t)level;
  }
}

// Adds (or takes the minimum and maximum of) a float at x without a return value; fmin/fmax of floats of either sign
// through their integer encodings, with *x starting at +inf (minimum) or -inf (maximum). A negative zero, which the
// encodings would order below every negative float, counts as zero.
__device__ __forceinline__ void atomic_min_float(float * x, float v) {
  v += 0.f;
  if (v >= 0.f) atomicMin(reinterpret_cast<int *>(x), __float_as_int(v));
  else atomicMax(reinterpret_cast<unsigned *>(x), __float_as_uint(v));
}
__device__ __forceinline__ void atomic_max_float(float * x, float v) {
  v += 0.f;
  if (v >= 0.f) atomicMax(reinterpret_cast<int *>(x), __float_as_int(v));
  else atomicMin(reinterpret_cast<unsigned *>(x), __float_as_uint(v));
}

// RANGE = false: sums of (normal * area) into slabs[slot].xyz. RANGE = true: the range of n . v into slabs[slot].zw.
template <int W, bool RANGE>
__global__ void __launch_bounds__(BUILD_THREADS)
slab_climb_kernel(int64_t n, int const * __restrict__ leaf_slot, uint8_t const * __restrict__ leaf_level,
                  int const * __restrict__ parent, float4 const * __restrict__ rec, float4 * slabs,
                  int * __restrict__ bad) {
  unsigned const FULL = 0xffffffffu;
  int lane = threadIdx.x & 31;
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int slot = k < n ? leaf_slot[k] : -1;
  if (k < n && slot < 0) atomicOr(bad, 1);  // an element under no leaf
  int level = slot >= 0 ? leaf_level[k] : -1;
  V3 v0 = V3{0.f, 0.f, 0.f}, v1 = v0, v2 = v0;  // RANGE: the vertices; else v0 = normal * area
  if (slot >= 0) {
    float4 const * r = rec + k * CP_REC_F4;
    if constexpr (RANGE) {
      v0 = xyz(__ldg(r));
      v1 = xyz(__ldg(r + 1));
      v2 = xyz(__ldg(r + 2));
    } else {
      V3 nn = xyz(__ldg(r + 3));
      float area = __ldg(r + 6).w;
      if (isfinite(nn.x) && isfinite(nn.y) && isfinite(nn.z) && isfinite(area)) v0 = nn * area;
    }
  }
  int top = __reduce_max_sync(FULL, level);
  for (int l = top; l >= 0; --l) {
    bool on = slot >= 0 && level >= l;  // this lane's slot at level l
    int run = on ? slot : -1 - lane;    // equal only among the lanes under one slot
    float a = 0.f, b = 0.f, c = 0.f;
    if constexpr (RANGE) {
      a = INFINITY;
      b = -INFINITY;
      if (on) {
        float2 enc = *reinterpret_cast<float2 const *>(slabs + slot);
        V3 nv = slab_normal(make_float4(enc.x, enc.y, 0.f, 0.f));
        V3 v[3] = {v0, v1, v2};
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          float lo, hi;
          slab_project(nv.x, nv.y, nv.z, v[j].x, v[j].y, v[j].z, lo, hi);
          a = fminf(a, lo);
          b = fmaxf(b, hi);
        }
      }
    } else if (on) {
      a = v0.x;
      b = v0.y;
      c = v0.z;
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int ro = __shfl_down_sync(FULL, run, o);
      float ao = __shfl_down_sync(FULL, a, o), bo = __shfl_down_sync(FULL, b, o);
      float co = RANGE ? 0.f : __shfl_down_sync(FULL, c, o);
      if (lane + o < 32 && ro == run) {
        if constexpr (RANGE) {
          a = fminf(a, ao);
          b = fmaxf(b, bo);
        } else {
          a += ao;
          b += bo;
          c += co;
        }
      }
    }
    int before = __shfl_up_sync(FULL, run, 1);
    if (on && (lane == 0 || before != run)) {
      float * out = reinterpret_cast<float *>(slabs + slot);
      if constexpr (RANGE) {
        atomic_min_float(out + 2, a);
        atomic_max_float(out + 3, b);
      } else {
        atomicAdd(out, a);
        atomicAdd(out + 1, b);
        atomicAdd(out + 2, c);
      }
    }
    if (on && l > 0) slot = parent[slot / W];
  }
}

// Summed normals -> encoded unit normal with an empty range
__global__ void slab_normal_kernel(int64_t slots, float4 * __restrict__ slabs) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= slots) return;
  float4 s = slabs[k];
  float x = s.x, y = s.y, z = s.z;
  float l = sqrtf(x * x + y * y + z * z);
  if (!(l > 0.f) || !isfinite(l)) x = 0.f, y = 0.f, z = 1.f, l = 1.f;
  float4 e = slab_encode(V3{x / l, y / l, z / l});
  slabs[k] = make_float4(e.x, e.y, INFINITY, -INFINITY);
}

template <int W>
static void build_slabs(thea_bvh * b, cudaStream_t stream) {
  WideNode<W> const * nodes = (WideNode<W> const *)b->nodes;
  int64_t nn = b->num_nodes, slots = nn * W, n = b->n;
  int M = b->num_segments;
  Scratch parent((size_t)nn * sizeof(int), stream), leaf_slot((size_t)n * sizeof(int), stream);
  Scratch leaf_level((size_t)n, stream), bad(sizeof(int), stream);
  THEA_CUDA_CHECK(cudaMemsetAsync(parent.ptr, 0xff, parent.bytes, stream));
  THEA_CUDA_CHECK(cudaMemsetAsync(leaf_slot.ptr, 0xff, leaf_slot.bytes, stream));
  THEA_CUDA_CHECK(cudaMemsetAsync(bad.ptr, 0, sizeof(int), stream));
  THEA_CUDA_CHECK(thea_malloc_async((void **)&b->slabs, (size_t)slots * sizeof(float4), stream));
  THEA_CUDA_CHECK(cudaMemsetAsync(b->slabs, 0, (size_t)slots * sizeof(float4), stream));
  unsigned sgrid = (unsigned)ceil_div(slots, BUILD_THREADS), egrid = (unsigned)ceil_div(n, BUILD_THREADS);
  THEA_LAUNCH(slab_roots_kernel, (unsigned)ceil_div(M, BUILD_THREADS), BUILD_THREADS, 0, stream, b->seg_root, M, nn,
              parent.as<int>(), bad.as<int>());
  THEA_LAUNCH(slab_parent_kernel<W>, sgrid, BUILD_THREADS, 0, stream, nodes, nn, parent.as<int>(), bad.as<int>());
  THEA_LAUNCH(slab_leaf_kernel<W>, sgrid, BUILD_THREADS, 0, stream, nodes, nn, parent.as<int>(), b->seg_start, M, n,
              leaf_slot.as<int>(), leaf_level.as<uint8_t>(), bad.as<int>());
  THEA_LAUNCH((slab_climb_kernel<W, false>), egrid, BUILD_THREADS, 0, stream, n, leaf_slot.as<int>(),
              leaf_level.as<uint8_t>(), parent.as<int>(), b->cp_rec, b->slabs, bad.as<int>());
  THEA_LAUNCH(slab_normal_kernel, sgrid, BUILD_THREADS, 0, stream, slots, b->slabs);
  THEA_LAUNCH((slab_climb_kernel<W, true>), egrid, BUILD_THREADS, 0, stream, n, leaf_slot.as<int>(),
              leaf_level.as<uint8_t>(), parent.as<int>(), b->cp_rec, b->slabs, bad.as<int>());
  int h = 0;
  THEA_CUDA_CHECK(cudaMemcpyAsync(&h, bad.ptr, sizeof(int), cudaMemcpyDeviceToHost, stream));
  THEA_CUDA_CHECK(cudaStreamSynchronize(stream));
  if (h) {
    cudaFreeAsync(b->slabs, stream);
    b->slabs = nullptr;  // searches use boxes alone
  }
}

// Oriented slabs go with single-mesh BVHs that have the closest layout: they shorten the longest searches of the
// one-query-per-thread kernels (small batches, serving), whose warps wait for their slowest lane, and of the
// warp-per-query kernel. The persistent batched kernels, which refill a lane as soon as its query ends, ran faster with
// boxes alone, so forests have none (with them in the second phase alone, 256 meshes of 320 to 327,680 triangles with
// 5.2 M queries: 12.4 -> 12.0 ms, for a build of 25 -> 29 ms).
void init_slabs(thea_bvh * b, cudaStream_t stream) {
  if (!b->is_mesh || b->num_segments != 1 || !b->cp_rec || b->slabs) return;
  if (b->num_nodes * b->width >= (int64_t(1) << 31)) return;  // slots are addressed with 31 bits
  if (b->width == 4) build_slabs<4>(b, stream);
  else build_slabs<8>(b, stream);
}

void init_segment_roots(thea_bvh * b, cudaStream_t stream) {
  int M = b->num_segments;
  std::vector<RootCut> & h = b->seg_roots_host;
  h.resize((size_t)M);
  for (int s = 0; s < M; ++s) h[(size_t)s] = root_cut_of(&b->seg_lo[3 * (size_t)s], &b->seg_hi[3 * (size_t)s], nullptr);
  if (!b->seg_roots) THEA_CUDA_CHECK(thea_malloc_async(&b->seg_roots, (size_t)M * sizeof(RootCut), stream));
  // (the handle keeps h: an asynchronous copy from pageable memory may read it late)
  THEA_CUDA_CHECK(cudaMemcpyAsync(b->seg_roots, h.data(), (size_t)M * sizeof(RootCut), cudaMemcpyHostToDevice, stream));
}

thea_bvh * build_bvh(bool is_mesh, float const * V, int64_t nv, int32_t const * F, int64_t nf,
                     thea_build_config const & cfg, cudaStream_t stream) {
  return build_forest(is_mesh, V, nv, F, nf, nullptr, 1, cfg, stream);
}

void destroy_bvh(thea_bvh * b) {
  if (!b) return;
  if (b->world) {
    b->world->err = nullptr;  // shared with b
    destroy_bvh(b->world);
    b->world = nullptr;
  }
  int prev = -1;
  cudaGetDevice(&prev);
  cudaSetDevice(b->device);
  cudaDeviceSynchronize();
  // the device is idle: the arrays go back to the library's pool for the next handle
  for (void * p : {b->nodes, (void *)b->cp_rec, (void *)b->slabs, (void *)b->ray_rec, (void *)b->pt_rec,
                   (void *)b->leaf_to_elem, (void *)b->err, (void *)b->seg_start, (void *)b->seg_root,
                   (void *)b->seg_roots})
    if (p) cudaFreeAsync(p, (cudaStream_t)0);
  if (b->err_host) release_host_word(b->err_host);
  if (prev >= 0) cudaSetDevice(prev);
  delete b;
}

}  // namespace thea
