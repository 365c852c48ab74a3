// Batched queries over a forest of BVHs (one per mesh or point set).
#pragma once

#include "bvh.hpp"
#include "query.hpp"

namespace thea {

// Device view of a forest passed by value to the persistent kernels
struct BatchForest {
  void const * nodes;
  float4 const * cp_rec;
  float4 const * ray_rec;
  float4 const * pt_rec;
  float4 const * slabs;  // oriented slabs of the child slots (single-mesh BVHs; nullptr otherwise)
  int64_t const * seg_start;
  int32_t const * seg_root;
  int M;
  unsigned * err;
};

BatchForest forest_view(thea_bvh const * b);

// Step budget of a batched closest-point search whose caller names none. A query past its budget is finished by a whole
// warp, which shortens the launch's longest chains but costs the GPU about five times a thread's search, so a batch that
// fills the GPU hands over only its longest queries, while a small one is bound by its longest chain. Times over those at 32
// (each in the kernels of before, the best and the worst of near the surface, in the box, in [-1, 1]^3 and all deep inside;
// 64 meshes of 1,280 triangles, 16 of 20,480 and 153 of 320 to 81,920; FP32) at budgets of 128 / 256 and, width 8, 64 / 128 / 256:
//  * width 4, leaves of one to four: 98,304 queries 0.26 - 1.21 / 0.26 - 1.53; 196,608 up to 1.01 / up to 0.87 (leaves of
//    four 1.04); 262,144 up to 1.03 / 0.99; 393,216 0.17 - 1.03 / 0.17 - 0.84; 1,048,576 0.15 - 0.66 / 0.15 - 0.63.
//    Leaves of eight: 393,216 0.31 - 0.91 / 0.31 - 1.05; 1,048,576 0.29 - 0.66 / 0.29 - 0.80.
//  * width 8, whose steps test twice as many boxes and whole leaves, leaves of one to four: 98,304 queries up to 1.16 / 1.14 /
//    1.47; 196,608 1.06 / 1.01 / 1.27 (leaves up to two 1.04 / 1.01 / 1.02); 393,216 1.07 / 1.00 / 1.04 (1.06 / 1.00 / 0.86).
//    Leaves of eight: 393,216 0.39 - 1.08 / 1.10 / 1.32; 1,048,576 0.37 - 0.95 / 0.99 / 1.10.
constexpr int64_t BATCH_BUDGET_MIN = 98304, BATCH_BUDGET_LARGE = 786432;
inline int batch_closest_budget(int64_t nq, int width, int leaf) {
  if (nq < BATCH_BUDGET_MIN) return 32;
  if (width == 4) return nq < (leaf <= 4 ? BATCH_BUDGET_LARGE / 3 : BATCH_BUDGET_LARGE) ? 128 : 256;
  if (leaf <= 2 && nq >= BATCH_BUDGET_LARGE / 2) return 256;
  return nq < (leaf <= 4 ? BATCH_BUDGET_LARGE / 4 : BATCH_BUDGET_LARGE) ? 64 : 128;
}

// qoff: device array of M + 1 query offsets (queries of segment m are [qoff[m], qoff[m+1])), or null for one segment, whose
// queries are all of them. chunk: queries a warp takes per fetch (a multiple of 32).
void run_batch_closest(thea_bvh const * b, float const * q, int64_t const * qoff, int64_t nq, ClosestParams const & cp,
                       int chunk, int32_t * idx, float * dist, float * cpt, float * err, cudaStream_t s);
// FP32 closest point of a small batch on one BVH (num_segments == 1, small_stack_ok), a whole warp per query below
// CLOSEST_WHOLE_WARP_MAX queries and half a warp from there.
constexpr int64_t CLOSEST_WHOLE_WARP_MAX = 3072;
void run_closest_teams(thea_bvh const * b, float const * q, int64_t nq, ClosestParams const & cp, int32_t * idx,
                       float * dist, float * cpt, cudaStream_t s);
// FP64 re-check of a small batch on one BVH (num_segments == 1, small_stack_ok), a warp per query.
void run_closest_warps_f64(thea_bvh const * b, float const * q, int64_t nq, ClosestParams const & cp, int32_t * idx,
                           float * dist, float * cpt, float * err, cudaStream_t s);
// FP32 closest point of one BVH with queries and results in pinned host memory accessed by the kernels in place
// (device-usable pointers); cp.budget > 0 enables the warp-per-query second phase.
void run_closest_stream(thea_bvh const * b, float const * q, int64_t nq, ClosestParams const & cp, int32_t * idx,
                        float * dist, float * cpt, cudaStream_t s);
void run_batch_ray(thea_bvh const * b, float const * o, float const * d, int64_t const * qoff, int64_t nq,
                   float max_time, int chunk, float * t, int32_t * idx, cudaStream_t s);
void run_batch_knn(thea_bvh const * b, float const * q, int64_t const * qoff, int64_t nq, int k, float thresh,
                   int chunk, int32_t * idx, float * d2, cudaStream_t s);

}  // namespace thea
