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
// fills the GPU hands over only its longest queries. 256 meshes of 320 to 327,680 triangles with 5.2 M queries: FP32 9.0 /
// 8.6 ms at budgets of 256 / 384 (with the searches as they were before: 33.3 / 17.7 / 12.4 / 12.3 at 32 / 128 / 256 / 384),
// FP64 re-check 35.1 / 23.6 / 20.3 / 19.5 at 128 / 192 / 256 / 384; 64 meshes with 210,677 queries: FP32 1.28 / 0.80 / 0.80
// / 0.89 at 32 / 160 / 256 / 384, FP64 1.60 / 1.42 / 1.40 / 1.48 at 128 / 192 / 256 / 384. A small batch is bound by its
// longest chain instead (81,920 triangles, two kernels: 32,768 queries 0.44 ms at 16 steps, 0.89 at 256).
inline int batch_closest_budget(int64_t nq) { return nq >= 98304 ? 256 : 32; }

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
