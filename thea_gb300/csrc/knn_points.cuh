// k nearest points of one query (BvhN::kClosestPairs + KClosestPairsFunctor + BoundedSortedArrayN; BvhN.hpp:474-500,
// 1139-1146; BoundedSortedArrayN.hpp:137-214): the list of the best so far, and the search.
//
// An entry is one 64-bit key, (bits of the squared distance) << 32 | element index: distances are not negative, so keys
// order as (distance, index), the contract's order. An empty entry is (threshold, INT_MAX), which every element at or
// below the threshold precedes. A list of capacity K that is to hold k < K entries starts with K - k zero keys, which no
// element evicts: the bound is then the k-th distance, not the K-th.
#pragma once

#include "traverse_ops.cuh"

namespace thea {

__device__ __forceinline__ uint64_t knn_key(float d2, int idx) {
  return ((uint64_t)__float_as_uint(d2) << 32) | (uint32_t)idx;
}
__device__ __forceinline__ float knn_key_d2(uint64_t key) { return __uint_as_float((uint32_t)(key >> 32)); }
__device__ __forceinline__ int knn_key_index(uint64_t key) { return (int)(uint32_t)key; }

// Kernels over points keep their K best in shared memory from K = 16 on (width-8 trees, whose 256-byte nodes leave fewer
// registers, from K = 8 on), and in registers below. Shared memory against registers, 262,144 queries: K = 8, width 4,
// 0.266 / 0.251 ms; K = 8, width 8, 0.408 / 0.420; K = 16, width 4, 0.403 / 0.454 (five resident blocks). The register
// allocator is asked for eight resident blocks of 128 threads (four for K = 32, whose lists take 32 KB). The lists of
// triangles (knn_mesh_kernel) are in shared memory from K = 8 on.
template <int W, int K> __host__ __device__ constexpr bool knn_lists_shared() { return K >= 16 || (W == 8 && K >= 8); }
template <int K> constexpr int knn_point_min_blocks() { return K <= 16 ? 8 : 4; }

// Compare-exchange network sorting K keys ascending (bitonic; every thread the same instructions)
template <int K> __device__ __forceinline__ void sort_keys(uint64_t (&r)[K]) {
#pragma unroll
  for (int k = 2; k <= K; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
#pragma unroll
      for (int i = 0; i < K; ++i) {
        int l = i ^ j;
        if (l > i) {
          bool sw = (r[i] > r[l]) == ((i & k) == 0);
          uint64_t a = sw ? r[l] : r[i], b = sw ? r[i] : r[l];
          r[i] = a;
          r[l] = b;
        }
      }
    }
  }
}

// Small lists: sorted in registers, an insertion bubbles through
template <int K> struct RegisterKnnList {
  uint64_t r[K];
  // entry(j): the j-th initial key (of any order)
  template <class Entry> __device__ __forceinline__ void init(Entry entry) {
#pragma unroll
    for (int j = 0; j < K; ++j) r[j] = ~0ull;
#pragma unroll
    for (int j = 0; j < K; ++j) insert(entry(j));
  }
  __device__ __forceinline__ uint64_t kth() const { return r[K - 1]; }
  __device__ __forceinline__ void insert(uint64_t key) {
#pragma unroll
    for (int j = 0; j < K; ++j) {
      bool lt = key < r[j];
      uint64_t t = r[j];
      r[j] = lt ? key : t;
      key = lt ? t : key;
    }
  }
  __device__ __forceinline__ void finish(uint64_t (&out)[K]) const {
#pragma unroll
    for (int j = 0; j < K; ++j) out[j] = r[j];
  }
};

// Larger lists (knn_lists_shared): unsorted in shared memory ([K][B], entry j of thread t at [j][t]: no bank conflicts), in groups of
// four with each group's largest key in a register. An insertion replaces the largest key of all and looks at its group
// alone: one store, three loads and a fixed sequence of selects, where a sorted list shifts K / 2 entries on average and
// a warp waits for the longest shift of its lanes. The row is sorted once, at the end, by a network all lanes run
// together.
template <int K, int B> struct SharedKnnList {
  static constexpr int G = K / 4;
  uint64_t (*s)[B];
  uint64_t top[G];
  uint64_t worst;
  __device__ __forceinline__ explicit SharedKnnList(uint64_t (*list)[B]) : s(list) {}
  __device__ __forceinline__ void settle() {
    worst = top[0];
#pragma unroll
    for (int g = 1; g < G; ++g) worst = top[g] > worst ? top[g] : worst;
  }
  template <class Entry> __device__ __forceinline__ void init(Entry entry) {
#pragma unroll
    for (int g = 0; g < G; ++g) {
      top[g] = 0;
#pragma unroll
      for (int j = 4 * g; j < 4 * g + 4; ++j) {
        uint64_t e = entry(j);
        s[j][threadIdx.x] = e;
        top[g] = e > top[g] ? e : top[g];
      }
    }
    settle();
  }
  __device__ __forceinline__ uint64_t kth() const { return worst; }
  __device__ __forceinline__ void insert(uint64_t key) {
    int g = 0;
#pragma unroll
    for (int u = 1; u < G; ++u) g = top[u] == worst ? u : g;
    uint64_t(*e)[B] = s + 4 * g;
    uint64_t e0 = e[0][threadIdx.x], e1 = e[1][threadIdx.x], e2 = e[2][threadIdx.x], e3 = e[3][threadIdx.x];
    // one entry of the group equals `worst`
    int j = e0 == worst ? 0 : (e1 == worst ? 1 : (e2 == worst ? 2 : 3));
    e[j][threadIdx.x] = key;
    e0 = j == 0 ? key : e0;
    e1 = j == 1 ? key : e1;
    e2 = j == 2 ? key : e2;
    e3 = j == 3 ? key : e3;
    uint64_t a = e0 > e1 ? e0 : e1, b = e2 > e3 ? e2 : e3;
    a = a > b ? a : b;
#pragma unroll
    for (int u = 0; u < G; ++u) top[u] = u == g ? a : top[u];
    settle();
  }
  __device__ __forceinline__ void finish(uint64_t (&out)[K]) const {
#pragma unroll
    for (int j = 0; j < K; ++j) out[j] = s[j][threadIdx.x];
    sort_keys<K>(out);
  }
};

// The search, nearest child first. Elements at leaf positions in [skip_lo, skip_hi) are left out: the list has them
// already. What bounds it: the L1 data pipe (86 % busy with the sorted lists, 40 % of it their shifting) and instruction
// issue. With the lists above and the self mode's start (knn_kernel): 1,048,576 points, their 16 nearest each 1.62 ->
// 1.29 ms, 32 nearest 4.08 -> 2.69; 262,144 queries of 262,144 points, 16 nearest 0.52 -> 0.40, 8 nearest 0.31 -> 0.27.
// (Offering the points of a node's leaf children at once instead of pushing them: 2-10 % slower for lists up to 16,
// 3 % to 8 % faster for most sizes with lists of 32.)
template <int W, int STACK, class List>
__device__ __forceinline__ void knn_points_search(WideNode<W> const * __restrict__ nodes,
                                                  float4 const * __restrict__ pts, int root, int64_t elem_base, V3 p,
                                                  int excl, int64_t skip_lo, int64_t skip_hi, List & list,
                                                  unsigned * err) {
  LocalStack<STACK> stk;
  int sp = 0;
  int next = root;  // nearest child of the last node, visited without a stack round trip
  while (next != CHILD_EMPTY || sp > 0) {
    int code = next;
    float lim = knn_key_d2(list.kth()) * PRUNE_SLACK;
    if (code == CHILD_EMPTY) {
      --sp;
      int2 e = stk.get(sp);
      code = e.x;
      if (__int_as_float(e.y) > lim) continue;
    }
    next = CHILD_EMPTY;
    if (code >= 0) {
      NodeRegs<W> nd;
      load_node(nodes, code, nd);
      float lb[W];
      point_child_bounds<W>(nd, p, lb);
      push_children_next<W>(nd, lb, lim, stk, sp, next, err);
    } else {
      int first, count;
      decode_leaf(code, first, count);
      int64_t k0 = elem_base + first;
      for (int64_t k = k0; k < k0 + count; ++k) {
        float4 a = __ldg(pts + k);
        int idx = __float_as_int(a.w);
        if (idx == excl || (k >= skip_lo && k < skip_hi)) continue;
        // MetricL2Impl<point, point>::closestPoints: (element - query).squaredNorm(). A NaN's key passes no bound.
        uint64_t key = knn_key(squared_norm(xyz(a) - p), idx);
        if (key < list.kth()) list.insert(key);
      }
    }
  }
}

// Row `row` of the k-NN outputs from K ascending keys whose first K - k_out are fillers: -1 for empty entries. Rows of a
// multiple of four entries go out as 16-byte stores when they can: rows land at scattered element indices (self mode),
// and full-sector writes keep the L2 from sending partial sectors to DRAM.
template <int K>
__device__ __forceinline__ void write_knn_keys(int32_t * __restrict__ out_index, float * __restrict__ out_d2, int64_t row,
                                               int k_out, uint64_t const (&r)[K]) {
  int pad = K - k_out;
  uintptr_t outs = reinterpret_cast<uintptr_t>(out_index) | reinterpret_cast<uintptr_t>(out_d2);
  int32_t * oi = out_index + row * k_out - pad;
  float * od = out_d2 + row * k_out - pad;
  if (K % 4 == 0 && k_out % 4 == 0 && (outs & 15) == 0) {
#pragma unroll
    for (int j = 0; j < K; j += 4) {
      if (j < pad) continue;
      int i[4];
      float d[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        i[u] = knn_key_index(r[(j + u) % K]);
        d[u] = i[u] != INT_MAX ? knn_key_d2(r[(j + u) % K]) : -1.f;
        if (i[u] == INT_MAX) i[u] = -1;
      }
      *reinterpret_cast<int4 *>(oi + j) = make_int4(i[0], i[1], i[2], i[3]);
      *reinterpret_cast<float4 *>(od + j) = make_float4(d[0], d[1], d[2], d[3]);
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < K; ++j) {
    if (j < pad) continue;
    int i = knn_key_index(r[j]);
    oi[j] = i != INT_MAX ? i : -1;
    od[j] = i != INT_MAX ? knn_key_d2(r[j]) : -1.f;
  }
}

}  // namespace thea
