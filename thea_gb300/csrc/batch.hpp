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
// 64 meshes of 1,280 triangles and 16 of 20,480; FP32): width 4, 98,304 queries 0.26 - 1.09 at 128 and 0.26 - 1.53 at 256;
// 393,216 0.17 - 1.04 and 0.17 - 1.05; 1,048,576 0.15 - 0.66 and 0.15 - 0.80. Width 8, whose steps test twice as many boxes
// and whole leaves: 98,304 queries 0.40 - 1.11 at 64 and 0.38 - 1.58 at 256; 393,216 0.35 - 1.08 and 0.35 - 1.32; 1,048,576
// 0.32 - 0.99 at 128 and 0.32 - 1.10 at 256.
constexpr int64_t BATCH_BUDGET_MIN = 98304, BATCH_BUDGET_LARGE = 786432;
inline int batch_closest_budget(int64_t nq, int width) {
  if (nq < BATCH_BUDGET_MIN) return 32;
  int budget = nq < BATCH_BUDGET_LARGE ? 128 : 256;
  return width == 4 ? budget : budget / 2;
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
