// The any-hit ray loop (BvhN::rayIntersects) as a template over where rays come from and where verdicts go, shared by
// the occlusion query, Visibility and the sample graph's reachability test. Instantiated per translation unit.
#pragma once

#include "device_util.cuh"
#include "query.hpp"
#include "transform.hpp"
#include "traverse_ops.cuh"

#include <algorithm>
#include <cstring>

namespace thea {
namespace {

constexpr int ANY_THREADS = 128;
constexpr int ANY_WARP_BLOCK = 64;
// lanes without a ray that a refill waits for (see ray_persistent_kernel): 4.2 M occlusion rays 0.802 -> 0.722 ms, 6.6 M
// visibility rays with their stream 3.48 -> 3.04
constexpr int ANY_REFILL_AT = 8;

struct Inverse {
  float m[12];
  int on;
};

// rays given as arrays (optionally mapped into object space)
struct RayArrays {
  float const * o;
  float const * d;
  Inverse inv;
  __device__ __forceinline__ void get(int64_t r, V3 & ro, V3 & rd) const {
    ro = load_v3(o + 3 * r);
    rd = load_v3(d + 3 * r);
    if (inv.on) {
      ro = affine_point(inv.m, ro);
      rd = affine_vector(inv.m, rd);
    }
  }
};

struct HitFlags {
  uint8_t * out;
  __device__ __forceinline__ void put(int64_t r, bool hit) const { out[r] = hit ? 1 : 0; }
};

template <int W, int STACK, class Src, class Sink>
__global__ void __launch_bounds__(ANY_THREADS)
any_hit_kernel(WideNode<W> const * __restrict__ nodes, float4 const * __restrict__ rec, Src src, Sink sink, int64_t n,
               float max_time, unsigned * __restrict__ err, unsigned long long * __restrict__ counter) {
  unsigned const FULL = 0xffffffffu;
  int lane = threadIdx.x & 31;
  int64_t qb = 0, qe = 0;  // warp-local block of ray ids, warp-uniform
  bool exhausted = false;  // warp-uniform
  int64_t q = -1;          // this lane's ray (-1: idle)
  RayState ray;
  ray_setup(ray, V3{0.f, 0.f, 0.f}, V3{0.f, 0.f, 1.f});
  float const bound = max_time >= 0.f ? max_time : INFINITY;
  // the first-hit step; any element it accepts ends the search (TriangleN<3>::rayIntersection: a hit at t >= 0, and
  // t <= max_time when bounded)
  float best = 0.f;
  int best_idx = INT_MAX;
  int64_t best_slot = -1;
  LocalStack<STACK> stk;
  int sp = 0;
  int next = CHILD_EMPTY;
  while (true) {
    // lanes whose ray is done, or that have none
    bool done = best_idx != INT_MAX || (next == CHILD_EMPTY && sp == 0);
    unsigned idle = __ballot_sync(FULL, done);
    if (__popc(idle) >= ANY_REFILL_AT || idle == FULL) {
      if (done && q >= 0) {
        sink.put(q, best_idx != INT_MAX);
        q = -1;
      }
      if (!exhausted && qb >= qe) {
        unsigned long long b = 0;
        if (lane == 0) b = atomicAdd(counter, (unsigned long long)ANY_WARP_BLOCK);
        b = __shfl_sync(FULL, b, 0);
        qb = (int64_t)b;
        qe = qb + ANY_WARP_BLOCK < n ? qb + ANY_WARP_BLOCK : n;
        if (qb >= n) exhausted = true;
      }
      if (!exhausted) {
        int rank = __popc(idle & ((1u << lane) - 1));
        int take = __popc(idle);
        int64_t avail = qe - qb;
        if (done && rank < avail) {
          q = qb + rank;
          V3 o, d;
          src.get(q, o, d);
          ray_setup(ray, o, d);
          best = bound;
          best_idx = INT_MAX;
          sp = 0;
          next = 0;
          done = false;
        }
        qb += take < avail ? take : avail;
      } else if (idle == FULL) {
        break;
      }
    }
    if (done) continue;
    int code = next;
    if (code == CHILD_EMPTY) code = stk.get(--sp).x;  // entries were pushed within the fixed bound
    ray_step<W>(nodes, rec, 0, code, ray, best, best_idx, best_slot, stk, sp, next, err);
  }
}

template <int W, int STACK, class Src, class Sink>
void launch_any(thea_bvh const * b, Src const & src, Sink const & sink, int64_t n, float max_time, cudaStream_t s) {
  auto k = any_hit_kernel<W, STACK, Src, Sink>;
  int per_sm = 0;
  THEA_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, ANY_THREADS, 0));
  int64_t need = ceil_div(ceil_div(n, ANY_WARP_BLOCK) * 32, ANY_THREADS);
  unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>((int64_t)std::max(1, per_sm) * sm_count(), need));
  Scratch counter(sizeof(unsigned long long), s);
  THEA_CUDA_CHECK(cudaMemsetAsync(counter.ptr, 0, sizeof(unsigned long long), s));
  THEA_LAUNCH_NAMED("any_hit_kernel", k, grid, ANY_THREADS, 0, s, (WideNode<W> const *)b->nodes, b->ray_rec, src, sink,
                    n, max_time, b->err, counter.as<unsigned long long>());
}

template <class Src, class Sink>
void dispatch_any(thea_bvh const * b, Src const & src, Sink const & sink, int64_t n, float max_time, cudaStream_t s) {
  bool sm = small_stack_ok(b);
  if (b->width == 4) sm ? launch_any<4, 64>(b, src, sink, n, max_time, s) : launch_any<4, 256>(b, src, sink, n, max_time, s);
  else sm ? launch_any<8, 128>(b, src, sink, n, max_time, s) : launch_any<8, 512>(b, src, sink, n, max_time, s);
}

Inverse inverse_of(thea_bvh const * b) {
  Inverse v;
  std::memcpy(v.m, b->xf_inv, sizeof(v.m));
  v.on = b->has_transform;
  return v;
}

}  // namespace
}  // namespace thea
