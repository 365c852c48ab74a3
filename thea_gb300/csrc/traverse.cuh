// Wide-node access and the per-query traversal stack shared by the query kernels.
#pragma once

#include "common.cuh"

namespace thea {

template <int W> struct NodeRegs {
  float lox[W], hix[W], loy[W], hiy[W], loz[W], hiz[W];
  int child[W];
};

// 32-byte read-only load (two float4s), 32-byte aligned. In the per-lane searches every lane reads its own 128-byte line,
// and each load instruction then costs the L1 data pipe one wavefront per lane whatever its width: that pipe, not memory,
// bounds the search kernels (72-88 % of its peak with 16-byte loads), and 32-byte loads halve what a line costs it.
__device__ __forceinline__ void ldg8(float4 const * p, float4 & a, float4 & b) {
  asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
               : "l"(p));
}

// A node is W*6 box floats followed by W child codes.
__device__ __forceinline__ void node_from_line(float4 const (&f)[8], NodeRegs<4> & r) {
  r.lox[0] = f[0].x; r.lox[1] = f[0].y; r.lox[2] = f[0].z; r.lox[3] = f[0].w;
  r.hix[0] = f[1].x; r.hix[1] = f[1].y; r.hix[2] = f[1].z; r.hix[3] = f[1].w;
  r.loy[0] = f[2].x; r.loy[1] = f[2].y; r.loy[2] = f[2].z; r.loy[3] = f[2].w;
  r.hiy[0] = f[3].x; r.hiy[1] = f[3].y; r.hiy[2] = f[3].z; r.hiy[3] = f[3].w;
  r.loz[0] = f[4].x; r.loz[1] = f[4].y; r.loz[2] = f[4].z; r.loz[3] = f[4].w;
  r.hiz[0] = f[5].x; r.hiz[1] = f[5].y; r.hiz[2] = f[5].z; r.hiz[3] = f[5].w;
  r.child[0] = __float_as_int(f[6].x); r.child[1] = __float_as_int(f[6].y);
  r.child[2] = __float_as_int(f[6].z); r.child[3] = __float_as_int(f[6].w);
}

// 128 bytes (a width-4 node or a closest-point record)
__device__ __forceinline__ void load_line(float4 const * p, float4 (&r)[8]) {
#pragma unroll
  for (int j = 0; j < 8; j += 2) ldg8(p + j, r[j], r[j + 1]);
}

// The same node through 16-byte loads, which the compiler may place where their values are used: fewer registers at width 8,
// where a node is 256 bytes, for kernels that need the resident warps more than the data pipe
template <int W> __device__ __forceinline__ void load_node_16(WideNode<W> const * __restrict__ nodes, int idx,
                                                              NodeRegs<W> & r) {
  float4 const * p = reinterpret_cast<float4 const *>(nodes + idx);
  constexpr int Q = W / 4;
  float * const rows[6] = {r.lox, r.hix, r.loy, r.hiy, r.loz, r.hiz};
#pragma unroll
  for (int q = 0; q < Q; ++q) {
#pragma unroll
    for (int a = 0; a < 6; ++a) {
      float4 u = __ldg(p + a * Q + q);
      rows[a][4 * q] = u.x; rows[a][4 * q + 1] = u.y; rows[a][4 * q + 2] = u.z; rows[a][4 * q + 3] = u.w;
    }
    int4 c = __ldg(reinterpret_cast<int4 const *>(p + 6 * Q + q));
    r.child[4 * q] = c.x; r.child[4 * q + 1] = c.y; r.child[4 * q + 2] = c.z; r.child[4 * q + 3] = c.w;
  }
}

template <int W> __device__ __forceinline__ void load_node(WideNode<W> const * __restrict__ nodes, int idx,
                                                           NodeRegs<W> & r) {
  float4 const * p = reinterpret_cast<float4 const *>(nodes + idx);
  if constexpr (W == 4) {
    float4 f[8];
    load_line(p, f);
    node_from_line(f, r);
  } else {
    float * const rows[6] = {r.lox, r.hix, r.loy, r.hiy, r.loz, r.hiz};
#pragma unroll
    for (int a = 0; a < 7; ++a) {
      float4 u, v;
      ldg8(p + 2 * a, u, v);
      if (a < 6) {
        rows[a][0] = u.x; rows[a][1] = u.y; rows[a][2] = u.z; rows[a][3] = u.w;
        rows[a][4] = v.x; rows[a][5] = v.y; rows[a][6] = v.z; rows[a][7] = v.w;
      } else {
        r.child[0] = __float_as_int(u.x); r.child[1] = __float_as_int(u.y);
        r.child[2] = __float_as_int(u.z); r.child[3] = __float_as_int(u.w);
        r.child[4] = __float_as_int(v.x); r.child[5] = __float_as_int(v.y);
        r.child[6] = __float_as_int(v.z); r.child[7] = __float_as_int(v.w);
      }
    }
  }
}

// Ascending odd-even transposition sort of W (key, code) pairs held in registers. Keys are non-negative float bit
// patterns or 0xFFFFFFFF for "do not visit".
template <int W> __device__ __forceinline__ void sort_children(uint32_t (&key)[W], int (&code)[W]) {
#pragma unroll
  for (int pass = 0; pass < W; ++pass) {
#pragma unroll
    for (int i = pass & 1; i + 1 < W; i += 2) {
      bool sw = key[i + 1] < key[i];
      uint32_t k0 = sw ? key[i + 1] : key[i], k1 = sw ? key[i] : key[i + 1];
      int c0 = sw ? code[i + 1] : code[i], c1 = sw ? code[i] : code[i + 1];
      key[i] = k0; key[i + 1] = k1;
      code[i] = c0; code[i + 1] = c1;
    }
  }
}

// Squared distance from a point to a box (any order of evaluation gives a valid bound thanks to the box padding)
__device__ __forceinline__ float point_box_d2(float px, float py, float pz, float lx, float ly, float lz, float hx,
                                              float hy, float hz) {
  float dx = fmaxf(fmaxf(lx - px, px - hx), 0.f);
  float dy = fmaxf(fmaxf(ly - py, py - hy), 0.f);
  float dz = fmaxf(fmaxf(lz - pz, pz - hz), 0.f);
  return __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz));
}

// Stack depth bound: a W-wide tree of depth D needs at most D * (W - 1) + 1 entries
template <int W> struct StackSize { static constexpr int value = W == 4 ? 64 : 128; };

// Traversal stacks of (child code, bound bits) entries. LocalStack keeps them in local memory. SharedStack keeps the
// first S entries of each of a block's B threads in shared memory and the rest in local memory: lanes of a warp stand at
// different depths, so every push and pop of a local-memory stack touches up to 32 separate sectors, which the search's
// own node traffic evicts from L1 before they are popped, while the [S][B] layout in shared memory has no bank conflicts
// at any mix of depths. S: a closest-point search pushes three entries a level on its first descent (nothing bounds it
// yet) and fits 24 (262,144 queries on 81,920 triangles: 1.19 / 1.18 / 1.13 / 1.33 ms at 0 / 16 / 24 / 32 entries, the
// last for want of resident blocks; 256 meshes, 5.2 M queries: 10.66 / 10.34 / 9.85 / 10.76); a ray's children mostly
// miss, 16 do (4.2 M rays on 2.1 M triangles: 0.94 / 0.91 / 0.92 / 1.01). The k-NN kernels, whose lists fill the shared
// memory, and the any-hit kernel ran slower with one.
template <int STACK> struct LocalStack {
  static constexpr int SIZE = STACK, FAST = STACK;
  int2 e[STACK];
  __device__ __forceinline__ int2 get(int i) const { return e[i]; }
  __device__ __forceinline__ void set(int i, int2 v) { e[i] = v; }
  __device__ __forceinline__ void set_fast(int i, int2 v) { e[i] = v; }  // i < FAST
};
constexpr int CLOSEST_SHARED_STACK = 24, RAY_SHARED_STACK = 16;
template <int STACK, int S, int B> struct SharedStack {
  static constexpr int SIZE = STACK, FAST = S;
  int2 (*sh)[B];
  int2 e[STACK - S];
  __device__ __forceinline__ explicit SharedStack(int2 (*s)[B]) : sh(s) {}
  __device__ __forceinline__ int2 get(int i) const { return i < S ? sh[i][threadIdx.x] : e[i - S]; }
  __device__ __forceinline__ void set(int i, int2 v) {
    if (i < S) sh[i][threadIdx.x] = v;
    else e[i - S] = v;
  }
  __device__ __forceinline__ void set_fast(int i, int2 v) { sh[i][threadIdx.x] = v; }  // i < FAST
};

// Device-side error bits reported through the handle's error word
constexpr unsigned ERR_STACK_OVERFLOW = 1u;
// a bounded wait of the tensor-core k-NN candidate kernel gave up (its queries fell back to the plain search)
constexpr unsigned ERR_GRAM_TIMEOUT = 2u;

}  // namespace thea
