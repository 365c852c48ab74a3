// Single-BVH query kernels: closest element of a mesh, first ray hit, k nearest points. One thread per query; the
// traversal routines live in traverse_ops.cuh and are shared with the batched kernels.
#include "bvh.hpp"
#include "device_util.cuh"
#include "query.hpp"
#include "transform.hpp"
#include "traverse_ops.cuh"
#include "warp_traverse.cuh"
#include "batch.hpp"
#include "knn_points.cuh"

#include <algorithm>

namespace thea {
namespace {

constexpr int QUERY_THREADS = 128;

// Queries a warp of the one-query-per-thread kernels takes: all its lanes once that gives every SM `warps_per_sm` warps, fewer
// below. The lanes of a warp wait for one another's branches and for the slowest of them, and a small batch packed 32 to a
// warp leaves most of the GPU idle meanwhile. Call times at 8 / 16 / 24 / 32 / 64 warps per SM, and always packed: 1,000 rays
// on 32,768 triangles 55 / 60 / 49 / 64 / 50, 64 us; 10,000 rays on 178,802 78 / 72 / 64 / 66 / 75, 78 us; the 8 nearest of
// 262,144 points, 1,000 queries of 65,536: 70 / 71 / 66 / 70 / 73, 105 us; 10,000: 118 / 108 / 108 / 114 / 137, 124 us.
constexpr int SPARSE_WARPS_PER_SM = 24;
int queries_per_warp(int64_t n, int most = 8, int warps_per_sm = SPARSE_WARPS_PER_SM) {
  int64_t warps = (int64_t)sm_count() * warps_per_sm;
  int per = 1;
  while ((int64_t)per * warps < n) per *= 2;
  return per <= most ? per : 32;
}
// For k-NN searches (K: the list's capacity). An insertion costs a warp the same whichever of its lanes make it, so spread lists
// spend the GPU faster than they gain, the longer the list the more: fewer warps an SM, up to 16 queries each. Spread over 24
// warps an SM, calls of 16,384 queries on six streams at once took 1.5 times as long as the packed sorted lists of before for the
// 16 nearest of 262,144 points at width 4, and 2.1 times for the 32 nearest at width 8. As below, calls of 4,000 to 16,384
// queries for 8, 16 and 32 nearest take 0.71 - 0.99 of it on six streams and 0.51 - 0.90 on one.
// Triangles (the sorted lists of before): likewise, with 8 and 16 nearest spread as far as 16 points and 32 less.
int knn_queries_per_warp(int64_t n, int width, int K, bool triangles, bool self) {
  int warps_per_sm = width == 4 ? (K <= 4 ? SPARSE_WARPS_PER_SM : K <= 8 ? 12 : 7) : (K <= 2 ? SPARSE_WARPS_PER_SM : K <= 4 ? 12 : 4);
  if (triangles) warps_per_sm = K <= 4 ? 12 : K <= 16 && width == 4 ? 7 : 4;
  int most = warps_per_sm < SPARSE_WARPS_PER_SM ? 16 : 8;
  return queries_per_warp(n, self ? most / 2 : most, warps_per_sm);
}
unsigned sparse_grid(int64_t n, int per) { return (unsigned)ceil_div(ceil_div(n, per) * 32, QUERY_THREADS); }
// This thread's query, or n where it has none
__device__ __forceinline__ int64_t sparse_query(int64_t n, int per) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int lane = threadIdx.x & 31;
  int64_t q = (t >> 5) * per + lane;
  return lane < per && q < n ? q : n;
}

//============================================================================================================================
// Closest element (BvhN::closestPair -> processNeighbors -> TriangleN<3>::closestPoint; BvhN.hpp:1082-1114, 1868-1893,
// 2038-2089; Triangle3.hpp:294-304)
//============================================================================================================================

template <int W, int STACK, int PREC>
__global__ void __launch_bounds__(QUERY_THREADS)
closest_kernel(WideNode<W> const * __restrict__ nodes, float4 const * __restrict__ rec, float const * __restrict__ queries,
               int64_t n, float thresh, double bound2, float scene_scale, int32_t * __restrict__ out_index,
               float * __restrict__ out_dist, float * __restrict__ out_cp, float * __restrict__ out_err,
               unsigned * __restrict__ err, uint32_t const * __restrict__ order, float4 const * __restrict__ slabs) {
  // no early exit: the FP64 step and the error estimate run with the warp's lanes together
  int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool active = q < n;
  if (active && order) q = order[q];
  V3 p = active ? load_v3(queries + 3 * q) : V3{0.f, 0.f, 0.f};
  ClosestOut r;
  r.idx = INT_MAX;
  r.d2 = 0.f;
  r.d2_64 = 0.0;
  r.slot = -1;
  float dist = 0.f;
  if constexpr (PREC == THEA_PRECISION_FP64_RECHECK) {
    __shared__ F64WarpBuf buf[QUERY_THREADS / 32];
    float scale = fmaxf(scene_scale, fmaxf(fabsf(p.x), fmaxf(fabsf(p.y), fabsf(p.z))));
    F64Search s;
    if (active) closest_search_f64<W, STACK>(nodes, rec, 0, 0, p, bound2, scale, err, s, 0, slabs);
    else f64_search_init(s);
    f64_resolve_warp(s, active, rec, 0, p, bound2, buf[threadIdx.x >> 5]);
    r = f64_result(s);
    dist = (float)sqrt(r.d2_64);
  } else {
    if (active) r = closest_query<W, STACK>(nodes, rec, 0, 0, p, thresh, err, 0, slabs);
    dist = sqrtf(r.d2);
  }
  bool found = r.idx != INT_MAX;
  double d64 = r.d2_64;
  if (PREC != THEA_PRECISION_FP64_RECHECK && out_err) {
    // FP64 distance of the returned element, evaluated with the warp's lanes together
    __syncwarp();
    if (active && found) {
      D3 cp64;
      cp_record_f64(rec, r.slot, p, cp64, d64);
    }
  }
  if (!active) return;
  out_index[q] = found ? r.idx : -1;
  if (out_dist) out_dist[q] = found ? dist : -1.f;
  if (out_cp) {
    out_cp[3 * q] = found ? r.cp.x : 0.f;
    out_cp[3 * q + 1] = found ? r.cp.y : 0.f;
    out_cp[3 * q + 2] = found ? r.cp.z : 0.f;
  }
  // |returned distance - FP64 distance of the returned element|
  if (out_err) out_err[q] = found ? (float)fabs((double)dist - sqrt(d64)) : -1.f;
}

//============================================================================================================================
// First ray hit (BvhN::rayStructureIntersection, BvhN.hpp:1292-1316, 2241-2291; TriangleN<3>::rayIntersection,
// Triangle3.hpp:542-552 -> rayTriangleIntersectionTime, Triangle3.hpp:1466-1524)
//============================================================================================================================

template <int W, int STACK, bool RECHECK>
__device__ __forceinline__ void ray_body(WideNode<W> const * __restrict__ nodes, float4 const * __restrict__ rec, float const * __restrict__ origins,
           float const * __restrict__ dirs, int64_t n, float max_time, float * __restrict__ out_time,
           int32_t * __restrict__ out_index, float * __restrict__ out_normal, float * __restrict__ out_time64,
           int32_t * __restrict__ out_index64, int32_t * __restrict__ out_flags, unsigned * __restrict__ err,
           uint32_t const * __restrict__ order, int per_warp) {
  int64_t q = sparse_query(n, per_warp);
  float t;
  int idx;
  int64_t slot;
  double t64 = 0.0;
  int idx64 = INT_MAX;
  if constexpr (RECHECK) {
    // no early exit: the FP64 step runs with the warp's lanes together
    __shared__ RayWarpBuf buf[QUERY_THREADS / 32];
    bool active = q < n;
    if (active && order) q = order[q];
    V3 o = active ? load_v3(origins + 3 * q) : V3{0.f, 0.f, 1.f};
    V3 d = active ? load_v3(dirs + 3 * q) : V3{0.f, 0.f, 1.f};
    RaySearch64 s;
    if (active) ray_search_f64<W, STACK>(nodes, rec, 0, 0, o, d, max_time, err, s);
    else ray_search_init(s, max_time);
    ray_resolve_warp(s, active, rec, 0, o, d, max_time, buf[threadIdx.x >> 5]);
    if (!active) return;
    t = s.t;
    idx = s.idx;
    slot = s.slot;
    t64 = s.best64;
    idx64 = s.idx64;
  } else {
    if (q >= n) return;
    if (order) q = order[q];
    RayOut r = ray_query<W, STACK, false>(nodes, rec, 0, 0, load_v3(origins + 3 * q), load_v3(dirs + 3 * q), max_time,
                                          err);
    t = r.t;
    idx = r.idx;
    slot = r.slot;
  }
  bool found = idx != INT_MAX;
  out_time[q] = found ? t : -1.f;
  if (out_index) out_index[q] = found ? idx : -1;
  if (out_normal) {
    V3 nn = V3{0.f, 0.f, 0.f};
    if (found) {
      float4 const * rr = rec + slot * RAY_REC_F4;
      nn = normalized(cross(xyz(__ldg(rr + 1)), xyz(__ldg(rr + 2))));
    }
    out_normal[3 * q] = nn.x;
    out_normal[3 * q + 1] = nn.y;
    out_normal[3 * q + 2] = nn.z;
  }
  if (RECHECK) {
    bool f64 = idx64 != INT_MAX;
    if (out_time64) out_time64[q] = f64 ? (float)t64 : -1.f;
    if (out_index64) out_index64[q] = f64 ? idx64 : -1;
    if (out_flags) out_flags[q] = (found != f64 ? THEA_RAY_FLAG_HIT_DIFFERS : 0) |
                                  (found && f64 && idx != idx64 ? THEA_RAY_FLAG_ELEMENT_DIFFERS : 0);
  }
}

template <int W, int STACK, bool RECHECK>
__global__ void __launch_bounds__(QUERY_THREADS)
ray_kernel(WideNode<W> const * __restrict__ nodes, float4 const * __restrict__ rec, float const * __restrict__ origins,
           float const * __restrict__ dirs, int64_t n, float max_time, float * __restrict__ out_time,
           int32_t * __restrict__ out_index, float * __restrict__ out_normal, float * __restrict__ out_time64,
           int32_t * __restrict__ out_index64, int32_t * __restrict__ out_flags, unsigned * __restrict__ err,
           uint32_t const * __restrict__ order, int per_warp) {
  ray_body<W, STACK, false>(nodes, rec, origins, dirs, n, max_time, out_time, out_index, out_normal, out_time64,
                            out_index64, out_flags, err, order, per_warp);
}

// The FP64 re-check form: register use capped so that five blocks of 128 threads fit on an SM
template <int W, int STACK>
__global__ void __launch_bounds__(QUERY_THREADS, 5)
ray_recheck_kernel(WideNode<W> const * __restrict__ nodes, float4 const * __restrict__ rec,
                   float const * __restrict__ origins, float const * __restrict__ dirs, int64_t n, float max_time,
                   float * __restrict__ out_time, int32_t * __restrict__ out_index, float * __restrict__ out_normal,
                   float * __restrict__ out_time64, int32_t * __restrict__ out_index64, int32_t * __restrict__ out_flags,
                   unsigned * __restrict__ err, uint32_t const * __restrict__ order, int per_warp) {
  ray_body<W, STACK, true>(nodes, rec, origins, dirs, n, max_time, out_time, out_index, out_normal, out_time64,
                           out_index64, out_flags, err, order, per_warp);
}

// Persistent form of ray_kernel for large batches (FP32 verdict only). Rays that leave the mesh after a few nodes and
// rays that traverse deep share warps; with one ray per thread the finished lanes idle until their warp's last ray is
// done. Here lanes take new rays as theirs finish: every loop iteration advances each busy lane by one stack entry, and
// idle lanes are refilled from a warp-local block of 64 rays (one atomic per block). Results are the
// same as ray_kernel's: each ray's traversal is the same sequence of steps. (Measured on the 2 M-triangle heightfield:
// skipping pruned entries in an inner loop, or postponing leaves so that node steps run converged, were both slower,
// since a lane's extra steps then stall its whole warp; keeping the nearest child in a register and packing stack
// entries into 8 bytes gained 4.5 %.) What bounds it: the L1 data pipe (81 % of its peak with 16-byte loads inside the
// node and leaf branches, each lane's line a wavefront per load; 78 % now) and the latency of those loads. Node or leaf
// read through one set of 32-byte loads (ray_step) and the first 16 stack entries in shared memory: 4.2 M rays on 2.1 M
// triangles 1.011 -> 0.871 ms, 0.771 with the refill below; from pinned host arrays (ray_stream_kernel, seven blocks per
// SM: eight would spill) 1.130 -> 1.006 ms. Lines fetched by eight lanes together into shared memory: 0.790 ms, not taken.
constexpr int RAY_WARP_BLOCK = 64;
// Lanes without a ray wait until this many of their warp's do (or all of them): writing a ray's results, fetching the next
// and its three divisions then run for eight or more lanes together instead of one or two. 4.2 M rays on 2.1 M triangles
// (half of them done after two steps), refilled at 1 / 4 / 8 / 12 / 16 / 24 lanes: 0.817 / 0.789 / 0.771 / 0.781 / 0.821 /
// 0.997 ms (0.869 with the results written as each ray ends).
constexpr int RAY_REFILL_AT = 8;
constexpr int64_t RAY_PERSISTENT_MIN = 1 << 16;

template <int W, int STACK>
__global__ void __launch_bounds__(QUERY_THREADS)
ray_persistent_kernel(WideNode<W> const * __restrict__ nodes, float4 const * __restrict__ rec,
                      float const * __restrict__ origins, float const * __restrict__ dirs, int64_t n, float max_time,
                      float * __restrict__ out_time, int32_t * __restrict__ out_index, float * __restrict__ out_normal,
                      unsigned * __restrict__ err, uint32_t const * __restrict__ order,
                      unsigned long long * __restrict__ counter) {
  unsigned const FULL = 0xffffffffu;
  int lane = threadIdx.x & 31;
  int64_t qb = 0, qe = 0;  // warp-local block of ray ids [qb, qe), warp-uniform
  bool exhausted = false;  // warp-uniform
  int64_t q = -1;          // this lane's ray (-1: idle)
  RayState ray;
  ray_setup(ray, V3{0.f, 0.f, 0.f}, V3{0.f, 0.f, 1.f});
  float best = 0.f;
  int best_idx = INT_MAX;
  int64_t best_slot = -1;
  __shared__ int2 s_stk[RAY_SHARED_STACK][QUERY_THREADS];
  SharedStack<STACK, RAY_SHARED_STACK, QUERY_THREADS> stk(s_stk);
  int sp = 0;
  int next = CHILD_EMPTY;  // the nearest child of the last node: visited next without a stack round trip
  while (true) {
    // lanes whose ray is done, or that have none
    bool done = next == CHILD_EMPTY && sp == 0;
    unsigned idle = __ballot_sync(FULL, done);
    if (__popc(idle) >= RAY_REFILL_AT || idle == FULL) {
      if (done && q >= 0) {
        // the same outputs as ray_kernel
        bool found = best_idx != INT_MAX;
        out_time[q] = found ? best : -1.f;
        if (out_index) out_index[q] = found ? best_idx : -1;
        if (out_normal) {
          V3 nn = V3{0.f, 0.f, 0.f};
          if (found) {
            float4 const * rr = rec + best_slot * RAY_REC_F4;
            nn = normalized(cross(xyz(__ldg(rr + 1)), xyz(__ldg(rr + 2))));
          }
          out_normal[3 * q] = nn.x;
          out_normal[3 * q + 1] = nn.y;
          out_normal[3 * q + 2] = nn.z;
        }
        q = -1;
      }
      if (!exhausted && qb >= qe) {
        unsigned long long b = 0;
        if (lane == 0) b = atomicAdd(counter, (unsigned long long)RAY_WARP_BLOCK);
        b = __shfl_sync(FULL, b, 0);
        qb = (int64_t)b;
        qe = qb + RAY_WARP_BLOCK < n ? qb + RAY_WARP_BLOCK : n;
        if (qb >= n) exhausted = true;
      }
      if (!exhausted) {
        int rank = __popc(idle & ((1u << lane) - 1));
        int take = __popc(idle);
        int64_t avail = qe - qb;
        if (done && rank < avail) {
          q = qb + rank;
          if (order) q = (int64_t)order[q];
          ray_setup(ray, load_v3(origins + 3 * q), load_v3(dirs + 3 * q));
          best = max_time >= 0.f ? max_time : INFINITY;
          best_idx = INT_MAX;
          best_slot = -1;
          next = 0;  // the root
          done = false;
        }
        qb += take < avail ? take : avail;
      } else if (idle == FULL) {
        break;
      }
    }
    if (done) continue;
    int code = next;
    if (code == CHILD_EMPTY) {
      --sp;
      int2 top = stk.get(sp);
      code = top.x;
      if (__int_as_float(top.y) > best * PRUNE_SLACK) continue;
    }
    ray_step<W>(nodes, rec, 0, code, ray, best, best_idx, best_slot, stk, sp, next, err);
  }
}

// Host-resident form of ray_persistent_kernel, for rays and results in pinned host memory read and written by the
// kernel itself (Grace-Blackwell reaches host memory coherently over NVLink-C2C). Instead of staging the batch through
// device buffers in chunks (each launch then ends with its own tail of long rays), one launch covers the batch: a warp
// copies each 64-ray block into shared memory once when it takes the block (one wait per block instead of one per ray),
// and results go to a per-warp ring of block buffers in shared memory that are written out, in ray order and with
// coalesced stores, once every ray of the block is done. A warp takes a new block only when a ring slot is free; the
// lanes then idle until their warp's oldest block completes, which always happens because its rays are in flight on
// lanes of the same warp. Time and index only (the normal variant keeps the staged path).
constexpr int STREAM_RING = 4;
constexpr int STREAM_WARPS = QUERY_THREADS / 32;

template <int W, int STACK>
__global__ void __launch_bounds__(QUERY_THREADS, 7)
ray_stream_kernel(WideNode<W> const * __restrict__ nodes, float4 const * __restrict__ rec,
                  float const * __restrict__ origins, float const * __restrict__ dirs, int64_t n, float max_time,
                  float * __restrict__ out_time, int32_t * __restrict__ out_index, unsigned * __restrict__ err,
                  unsigned long long * __restrict__ counter) {
  __shared__ float s_in[STREAM_WARPS][RAY_WARP_BLOCK * 6];
  __shared__ float s_t[STREAM_WARPS][STREAM_RING][RAY_WARP_BLOCK];
  __shared__ int s_i[STREAM_WARPS][STREAM_RING][RAY_WARP_BLOCK];
  __shared__ int s_left[STREAM_WARPS][STREAM_RING];
  __shared__ long long s_base[STREAM_WARPS][STREAM_RING];
  __shared__ int s_cnt[STREAM_WARPS][STREAM_RING];
  unsigned const FULL = 0xffffffffu;
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float * in = s_in[warp];
  int64_t qb = 0, qe = 0;   // rays of the current block not yet handed out, warp-uniform
  bool exhausted = false;   // warp-uniform
  long long taken = 0;      // blocks taken by this warp, warp-uniform
  long long oldest = 0;     // oldest block not written out yet, warp-uniform
  int64_t q = -1;           // this lane's ray (-1: idle)
  int slot = 0;             // ring slot of this lane's ray
  int64_t qbase = 0;        // first ray of that slot's block
  RayState ray;
  ray_setup(ray, V3{0.f, 0.f, 0.f}, V3{0.f, 0.f, 1.f});
  float best = 0.f;
  int best_idx = INT_MAX;
  int64_t best_slot = -1;  // (not an output here)
  __shared__ int2 s_stk[RAY_SHARED_STACK][QUERY_THREADS];
  SharedStack<STACK, RAY_SHARED_STACK, QUERY_THREADS> stk(s_stk);
  int sp = 0;
  int next = CHILD_EMPTY;
  while (true) {
    __syncwarp();
    // write out completed blocks, oldest first
    while (oldest < taken && s_left[warp][oldest % STREAM_RING] == 0) {
      int sl = (int)(oldest % STREAM_RING);
      long long base = s_base[warp][sl];
      int cnt = s_cnt[warp][sl];
      for (int j = lane; j < cnt; j += 32) {
        out_time[base + j] = s_t[warp][sl][j];
        if (out_index) out_index[base + j] = s_i[warp][sl][j];
      }
      ++oldest;
    }
    __syncwarp();
    unsigned idle = __ballot_sync(FULL, q < 0);
    if ((__popc(idle) >= RAY_REFILL_AT || idle == FULL) && !exhausted) {
      if (qb >= qe && taken - oldest < STREAM_RING) {
        unsigned long long b = 0;
        if (lane == 0) b = atomicAdd(counter, (unsigned long long)RAY_WARP_BLOCK);
        b = __shfl_sync(FULL, b, 0);
        if ((int64_t)b >= n) {
          exhausted = true;
        } else {
          qb = (int64_t)b;
          qe = qb + RAY_WARP_BLOCK < n ? qb + RAY_WARP_BLOCK : n;
          int cnt = (int)(qe - qb);
          // one coalesced copy of the block's origins and directions
          for (int k = lane; k < 3 * cnt; k += 32) {
            in[(k / 3) * 6 + k % 3] = origins[3 * qb + k];
            in[(k / 3) * 6 + 3 + k % 3] = dirs[3 * qb + k];
          }
          int sl = (int)(taken % STREAM_RING);
          if (lane == 0) {
            s_base[warp][sl] = qb;
            s_cnt[warp][sl] = cnt;
            s_left[warp][sl] = cnt;
          }
          ++taken;
          __syncwarp();
        }
      }
      if (!exhausted && qb < qe) {
        int rank = __popc(idle & ((1u << lane) - 1));
        int take = __popc(idle);
        int64_t avail = qe - qb;
        if (q < 0 && rank < avail) {
          q = qb + rank;
          slot = (int)((taken - 1) % STREAM_RING);
          qbase = s_base[warp][slot];
          float const * r = in + (q - qbase) * 6;
          ray_setup(ray, V3{r[0], r[1], r[2]}, V3{r[3], r[4], r[5]});
          best = max_time >= 0.f ? max_time : INFINITY;
          best_idx = INT_MAX;
          sp = 0;
          next = 0;
        }
        qb += take < avail ? take : avail;
      }
    }
    bool busy = __ballot_sync(FULL, q >= 0) != 0;
    if (!busy && oldest == taken && (exhausted || qb >= qe)) {
      if (exhausted) break;
      continue;  // every block written out and no ray in flight: take the next block
    }
    if (q < 0) continue;
    int code = next;
    if (code == CHILD_EMPTY) {
      if (sp == 0) {
        bool found = best_idx != INT_MAX;
        int j = (int)(q - qbase);
        s_t[warp][slot][j] = found ? best : -1.f;
        s_i[warp][slot][j] = found ? best_idx : -1;
        atomicSub(&s_left[warp][slot], 1);
        q = -1;
        continue;
      }
      --sp;
      int2 top = stk.get(sp);
      code = top.x;
      if (__int_as_float(top.y) > best * PRUNE_SLACK) continue;
    }
    ray_step<W>(nodes, rec, 0, code, ray, best, best_idx, best_slot, stk, sp, next, err);
  }
}

template <int W, int STACK>
void launch_ray_stream(thea_bvh const * b, float const * o, float const * d, int64_t n, float max_time, float * t,
                       int32_t * idx, unsigned * err, cudaStream_t s) {
  auto k = ray_stream_kernel<W, STACK>;
  int per_sm = 0;
  THEA_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, QUERY_THREADS, 0));
  int64_t need = ceil_div(ceil_div(n, RAY_WARP_BLOCK) * 32, QUERY_THREADS);
  unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>((int64_t)std::max(1, per_sm) * sm_count(), need));
  Scratch counter(sizeof(unsigned long long), s);
  THEA_CUDA_CHECK(cudaMemsetAsync(counter.ptr, 0, sizeof(unsigned long long), s));
  THEA_LAUNCH_NAMED("ray_stream_kernel", k, grid, QUERY_THREADS, 0, s, (WideNode<W> const *)b->nodes, b->ray_rec, o, d,
                    n, max_time, t, idx, err, counter.as<unsigned long long>());
}

//============================================================================================================================
// k nearest points (BvhN::kClosestPairs + KClosestPairsFunctor + BoundedSortedArrayN; BvhN.hpp:474-500, 1139-1146;
// BoundedSortedArrayN.hpp:137-214)
//============================================================================================================================

// Row `row` of the k-NN outputs from a K-entry list read through gd(j) / gi(j) (registers or shared memory): -1 for
// empty entries. Whole rows go out as 16-byte stores when they can: rows land at scattered element indices (self
// mode), and full-sector writes keep the L2 from sending partial sectors to DRAM.
template <int K, class GD, class GI>
__device__ __forceinline__ void write_knn_row(int32_t * __restrict__ out_index, float * __restrict__ out_d2, int64_t row,
                                              int k_out, GD gd, GI gi) {
  uintptr_t outs = reinterpret_cast<uintptr_t>(out_index) | reinterpret_cast<uintptr_t>(out_d2);
  if (K % 4 == 0 && k_out == K && (outs & 15) == 0) {
    int4 * oi = reinterpret_cast<int4 *>(out_index + row * K);
    float4 * od = reinterpret_cast<float4 *>(out_d2 + row * K);
#pragma unroll
    for (int j = 0; j < K; j += 4) {
      int i0 = gi(j), i1 = gi(j + 1), i2 = gi(j + 2), i3 = gi(j + 3);
      i0 = i0 != INT_MAX ? i0 : -1;
      i1 = i1 != INT_MAX ? i1 : -1;
      i2 = i2 != INT_MAX ? i2 : -1;
      i3 = i3 != INT_MAX ? i3 : -1;
      oi[j / 4] = make_int4(i0, i1, i2, i3);
      od[j / 4] = make_float4(i0 >= 0 ? gd(j) : -1.f, i1 >= 0 ? gd(j + 1) : -1.f, i2 >= 0 ? gd(j + 2) : -1.f,
                              i3 >= 0 ? gd(j + 3) : -1.f);
    }
    return;
  }
  for (int j = 0; j < k_out; ++j) {
    int i = gi(j);
    bool v = i != INT_MAX;
    out_index[row * k_out + j] = v ? i : -1;
    out_d2[row * k_out + j] = v ? gd(j) : -1.f;
  }
}

template <int W, int K, int STACK>
__global__ void __launch_bounds__(QUERY_THREADS, knn_point_min_blocks<K>())
knn_kernel(WideNode<W> const * __restrict__ nodes, float4 const * __restrict__ pts, float const * __restrict__ queries,
           int64_t n, int k_out, float thresh, int32_t const * __restrict__ exclude, int32_t * __restrict__ out_index,
           float * __restrict__ out_d2, unsigned * __restrict__ err, uint32_t const * __restrict__ order,
           float const * __restrict__ init_bound, int per_warp) {
  int64_t q = sparse_query(n, per_warp);
  if (q >= n) return;
  if (order) q = order[q];
  V3 p;
  int excl;
  int64_t row;
  if (queries) {
    p = load_v3(queries + 3 * q);
    excl = exclude ? exclude[q] : -1;
    row = q;
  } else {
    // self mode: query q is the point at leaf position q, excluding itself; its row is its element index
    float4 a = __ldg(pts + q);
    p = xyz(a);
    excl = __float_as_int(a.w);
    row = excl;
  }
  // init_bound (self mode, per leaf position): an upper bound on the k-th neighbour's squared distance, inclusive, from
  // actual points; the search keeps every point within it, so the result is the same as without it
  float start = (init_bound ? fminf(thresh, init_bound[q]) : thresh) + 0.0f;  // (no negative zero)
  bool any = start >= 0.f;  // a negative threshold admits nothing
  // self mode starts from the points around its own in leaf order: a bound from the first step on, for a few loads that a
  // warp shares
  int pad = K - k_out;
  int64_t lo = 0, hi = 0;
  if (!queries && any) {
    hi = q + 1 + k_out / 2 < n ? q + 1 + k_out / 2 : n;
    lo = hi - (k_out + 1) > 0 ? hi - (k_out + 1) : 0;
    hi = lo + k_out + 1 < n ? lo + k_out + 1 : n;
  }
  uint64_t none = knn_key(any ? start : 0.f, INT_MAX);
  auto entry = [&](int j) {  // initial entry j
    if (j < pad) return (uint64_t)0;
    int64_t k = lo + (j - pad);
    if (k >= q) ++k;  // past the query's own point
    if (k >= hi) return none;
    float4 a = __ldg(pts + k);
    uint64_t key = knn_key(squared_norm(xyz(a) - p), __float_as_int(a.w));
    return key < none ? key : none;
  };
  uint64_t keys[K];
  if constexpr (knn_lists_shared<W, K>()) {
    __shared__ uint64_t s_list[K][QUERY_THREADS];
    SharedKnnList<K, QUERY_THREADS> list(s_list);
    list.init(entry);
    if (any) knn_points_search<W, STACK>(nodes, pts, 0, 0, p, excl, lo, hi, list, err);
    list.finish(keys);
  } else {
    RegisterKnnList<K> list;
    list.init(entry);
    if (any) knn_points_search<W, STACK>(nodes, pts, 0, 0, p, excl, lo, hi, list, err);
    list.finish(keys);
  }
  write_knn_keys<K>(out_index, out_d2, row, k_out, keys);
}

// k nearest triangles of a mesh BVH to each query point (kClosestPairs on a MeshBvh)
template <int W, int K, int STACK>
__global__ void __launch_bounds__(QUERY_THREADS, knn_point_min_blocks<K>())
knn_mesh_kernel(WideNode<W> const * __restrict__ nodes, float4 const * __restrict__ rec,
                float const * __restrict__ queries, int64_t n, int k_out, float thresh,
                int32_t const * __restrict__ exclude, int32_t * __restrict__ out_index, float * __restrict__ out_d2,
                unsigned * __restrict__ err, uint32_t const * __restrict__ order, int per_warp) {
  int64_t q = sparse_query(n, per_warp);
  if (q >= n) return;
  if (order) q = order[q];
  V3 p = load_v3(queries + 3 * q);
  int excl = exclude ? exclude[q] : -1;
  if constexpr (K >= 8) {
    __shared__ float s_d[K][QUERY_THREADS];
    __shared__ int s_i[K][QUERY_THREADS];
    int t = threadIdx.x;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      s_d[j][t] = thresh;
      s_i[j][t] = INT_MAX;
    }
    float kth = thresh;
    int kth_i = INT_MAX;
    knn_mesh_query_shared<W, K, STACK, QUERY_THREADS>(nodes, rec, 0, 0, p, excl, s_d, s_i, kth, kth_i, err);
    write_knn_row<K>(out_index, out_d2, q, k_out, [&](int j) { return s_d[j][t]; }, [&](int j) { return s_i[j][t]; });
  } else {
    float bd[K];
    int bi[K];
#pragma unroll
    for (int j = 0; j < K; ++j) { bd[j] = thresh; bi[j] = INT_MAX; }
    knn_mesh_query<W, K, STACK>(nodes, rec, 0, 0, p, excl, bd, bi, err);
    write_knn_row<K>(out_index, out_d2, q, k_out, [&](int j) { return bd[j]; }, [&](int j) { return bi[j]; });
  }
}

// FP32 calls on one BVH by size. Call times in ms on 81,920 triangles, queries near the surface / uniform in its box grown
// by half (a seventh of them deep inside, ten times the steps of the others):
//  * fewer than CLOSEST_WARP_MAX queries: 32 or 16 lanes per query (run_closest_teams). 1,000 queries: 0.047 / 0.088 with
//    32 lanes, 0.041 / 0.113 with 16; 4,000: 0.078 / 0.119 and 0.043 / 0.137; 16,000: 0.189 / 0.287 and 0.091 / 0.240;
//    57,000: 0.616 / 0.882 and 0.260 / 0.617; with 8 lanes 0.175 / 0.764. (Two kernels, a 16-step budget on one thread and
//    then a warp: 0.059 / 0.093, 0.077 / 0.118, 0.146 / 0.233, 0.374 / 0.608; that form stays for trees too deep for the
//    teams' stacks.)
//  * up to CLOSEST_TWO_PHASE_MIN: one query per thread (65,536 queries in the box: 0.71 ms; 0.72 with a 16-step budget);
//  * from there: two kernels with a 256-step budget (persistent lanes, then a warp per query past it; 262,144 queries in
//    the box: 1.06 ms against 1.84 one per thread).
//  * at width 8, where a step of 16 lanes expands two nodes, the teams end at CLOSEST_TEAM_MAX_W8: 81,920 triangles, leaves of
//    four, 32,768 queries in the box 0.63 ms with 16 lanes, 0.51 in two kernels (six streams at once 2.98 and 2.41).
constexpr int64_t CLOSEST_WARP_MAX = 57344;
constexpr int64_t CLOSEST_TEAM_MAX_W8 = 16384;
constexpr int CLOSEST_WARP_BUDGET = 16;
constexpr int64_t CLOSEST_TWO_PHASE_MIN = 98304;
constexpr int CLOSEST_TWO_PHASE_BUDGET = 256;

// FP64 re-check calls on one BVH: fewer than F64_WARP_MAX queries (F64_WARP_MAX_SMALL on small meshes) run as a warp per
// query; the others through the collecting and resolving kernels with a step budget, or one query per thread, in Morton
// order, with slabs. 1,000 queries on 20,480 triangles, near the surface / uniform in the box grown by half: a warp per query
// 0.066 / 0.075 ms, one per thread 0.143 / 0.491.
constexpr int64_t F64_WARP_MAX = 3072;
constexpr int64_t F64_WARP_MAX_SMALL = 2048;
constexpr int64_t F64_SMALL_MESH = 2048;
constexpr int64_t F64_SMALL_LARGE_BATCH = 65536;

bool f64_small_mesh(thea_bvh const * b, int64_t n) {
  return b->n <= F64_SMALL_MESH || (b->n <= 4 * F64_SMALL_MESH && n >= F64_SMALL_LARGE_BATCH);
}

// Step budget of the collecting kernel, or 0 for one query per thread. The collected form is taken where no kind of query
// (near the surface, in the box grown by half, in [-1, 1]^3, all deep inside, far outside) is slower in it. Its time over that
// of one query per thread, the best kind and the worst, on 20,480, 81,920 and 327,680 triangles (budget):
//  * width 4, leaves of one and two: 3,500 queries 0.22 - 0.88 (64), 8,192 0.40 - 0.81 (128), 16,384 0.54 - 0.87 (192), 32,768
//    0.57 - 0.82 (256), 65,536 0.63 - 1.09 (256), 100,003 0.56 - 1.01 (256) and 0.58 - 1.03 (224; half the kinds 3 to 5 %
//    faster), 131,072 0.59 - 1.16 (256) and 0.61 - 1.01 (384), 163,840 0.63 - 1.04 (384), 262,144 0.70 - 1.33 (384): the slow
//    ones are the queries deep inside, which the slabs of the one-per-thread form shorten tenfold. 5,120 triangles: 16,384
//    0.75 - 0.88 (128) and 0.75 - 1.22 (256).
//  * width 4, larger leaves: 3,500 0.24 - 0.79 (64), 16,384 0.57 - 0.82 (128), 32,768 0.65 - 0.98 (256), 65,536 0.70 - 1.12
//    (256), 262,144 0.74 - 1.60.
//  * width 8, leaves of one and two: 3,500 0.25 - 0.73 (64), 16,384 0.61 - 0.85 (128), 32,768 0.58 - 0.95 (256), 131,072 0.46
//    - 1.00 (256), 262,144 0.57 - 1.26. Leaves of four: 16,384 0.74 - 1.02 (128), 65,536 0.73 - 1.09 (256). Leaves of eight
//    and sixteen: 8,192 0.56 - 1.19 (128), 65,536 0.74 - 1.73 (256).
//  * small meshes: nodes and records stay in L1 or nearly, and a warp of neighbours reads them together. 1,280 triangles,
//    100,000 queries in the box: 0.511 ms one per thread, 0.670 collected.
// Calls of several streams at once pay for the warps that finish the queries over budget: six streams with 16,384 queries
// each took 0.97 - 1.28 times as long as one per thread with these budgets (192; 1.01 - 1.50 with 128, 0.81 - 1.33 with 256),
// at 0.54 - 0.87 of its time on one stream.
int f64_collect_budget(thea_bvh const * b, int64_t n) {
  if (f64_small_mesh(b, n)) return 0;
  if (b->width == 4) {
    if (n < 6144) return 64;
    if (n < 12288 || (b->n <= 4 * F64_SMALL_MESH && n < 65536)) return 128;
    if (b->leaf_size <= 2) return n < 24576 ? 192 : n < 81920 ? 256 : n < 114688 ? 224 : n < 163840 ? 384 : 0;
    return n < 32768 ? 128 : n < 65536 ? 256 : 0;
  }
  if (b->leaf_size <= 2) return n < 6144 ? 64 : n < 32768 ? 128 : n < 131072 ? 256 : 0;
  return b->leaf_size < 8 && n < 32768 ? (n < 6144 ? 64 : 128) : 0;
}

//============================================================================================================================
// Points within a radius (BvhN::rangeQueryIndices with a Ball3 range, BvhN.hpp:1208-1219, 2118-2171; BallN::contains,
// BallN.hpp:83: (p - center).squaredNorm() <= radius * radius, inclusive, FP32). Counting pass, then a filling pass into
// each query's slice of a CSR list; the slices are then put in ascending element order.
//============================================================================================================================

// Calls visit(leaf position, record) for every point under a node child whose box reaches within `lim` of p. Every such
// child is visited whatever the order, so internal children go on the stack unsorted (the first stays in a register) and
// the points of a node's leaf children are read at once, together, instead of one stack round trip and one memory wait
// each: with one point to a leaf they are most of the children a search meets.
template <int W, int STACK, class Visit>
__device__ __forceinline__ void range_search(WideNode<W> const * __restrict__ nodes, float4 const * __restrict__ pts, V3 p,
                                             float lim, unsigned * err, Visit visit) {
  int stk[STACK];
  int sp = 0;
  int next = 0;
  while (true) {
    int code = next;
    if (code == CHILD_EMPTY) {
      if (sp == 0) break;
      code = stk[--sp];
    }
    next = CHILD_EMPTY;
    NodeRegs<W> nd;
    load_node(nodes, code, nd);
    float lb[W];
    point_child_bounds<W>(nd, p, lb);
    float4 a[W];
    bool leaf[W];
#pragma unroll
    for (int c = 0; c < W; ++c) {
      leaf[c] = nd.child[c] < 0 && nd.child[c] != CHILD_EMPTY && lb[c] <= lim;
      if (leaf[c]) a[c] = __ldg(pts + (~nd.child[c] >> LEAF_COUNT_BITS));
    }
#pragma unroll
    for (int c = 0; c < W; ++c) {
      if (nd.child[c] >= 0 && lb[c] <= lim) {
        if (next == CHILD_EMPTY) next = nd.child[c];
        else if (sp < STACK) stk[sp++] = nd.child[c];
        else atomicOr(err, ERR_STACK_OVERFLOW);
      }
    }
#pragma unroll
    for (int c = 0; c < W; ++c) {
      if (leaf[c]) {
        int first, count;
        decode_leaf(nd.child[c], first, count);
        visit(first, a[c]);
        for (int k = first + 1; k < first + count; ++k) visit(k, __ldg(pts + k));
      }
    }
  }
}

// MODE 0: count each query's neighbours; 1: write (query, element) keys and squared distances at the query's offset,
// for the global sort into ascending element order; 2: write the elements (and squared distances, if asked) directly, in
// traversal order; 3: count, and write the first row_cap elements into row q of out_idx.
template <int W, int STACK, int MODE>
__global__ void __launch_bounds__(QUERY_THREADS)
range_kernel(WideNode<W> const * __restrict__ nodes, float4 const * __restrict__ pts, float const * __restrict__ queries,
             int64_t n, int per_warp, float r2, int32_t const * __restrict__ exclude, int64_t * __restrict__ count_or_offset,
             uint64_t * __restrict__ keys, float * __restrict__ out_d2, unsigned * __restrict__ err,
             int32_t * __restrict__ out_idx = nullptr, int row_cap = 0, unsigned * __restrict__ overflow = nullptr) {
  constexpr bool FILL = MODE == 1 || MODE == 2;
  int64_t q = sparse_query(n, per_warp);
  if (q >= n) return;
  V3 p = load_v3(queries + 3 * q);
  int ex = exclude ? exclude[q] : -1;
  int64_t w = FILL ? count_or_offset[q] : 0;
  int64_t c = 0;
  range_search<W, STACK>(nodes, pts, p, r2 * PRUNE_SLACK, err, [&](int, float4 a) {
    int idx = __float_as_int(a.w);
    if (idx == ex) return;
    float d2 = squared_norm(xyz(a) - p);
    if (d2 <= r2) {
      if (MODE == 1) {
        keys[w + c] = ((uint64_t)q << 32) | (uint32_t)idx;
        out_d2[w + c] = d2;
      } else if (MODE == 2) {
        out_idx[w + c] = idx;
        if (out_d2) out_d2[w + c] = d2;
      } else if (MODE == 3) {
        if (c < row_cap) out_idx[q * row_cap + c] = idx;
      }
      ++c;
    }
  });
  if (!FILL) count_or_offset[q] = c;
  if (MODE == 3 && c > row_cap) atomicOr(overflow, 1u);
}

// Total number of neighbours and the longest row, for the host's choice of sort
__global__ void range_extent_kernel(int64_t const * __restrict__ offsets, int64_t n, unsigned long long * __restrict__ out) {
  unsigned long long m = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    unsigned long long c = (unsigned long long)(offsets[i + 1] - offsets[i]);
    m = c > m ? c : m;
  }
  for (int o = 16; o; o >>= 1) {
    unsigned long long u = __shfl_xor_sync(0xffffffffu, m, o);
    m = u > m ? u : m;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(out + 1, m);
  if (blockIdx.x == 0 && threadIdx.x == 0) out[0] = (unsigned long long)offsets[n];
}

// Puts each row of a CSR list in ascending element order, in place, one warp per row: up to 32 entries by a bitonic
// network across the lanes, up to ROW_SORT_MAX in shared memory. Elements of a row are distinct. Reading and writing the
// list once is what bounds it; a radix sort of (query, element) keys moved every entry six times (200,003 points, 24
// neighbours each: 0.49 of the call's 0.96 ms; this takes 0.065 and the call 0.52), and stays for longer rows.
constexpr int ROW_SORT_MAX = 512;
constexpr int ROW_SORT_WARPS = 4;

__global__ void __launch_bounds__(ROW_SORT_WARPS * 32)
range_sort_rows_kernel(int64_t const * __restrict__ offsets, int64_t n, int32_t * __restrict__ idx,
                       float * __restrict__ d2) {
  __shared__ uint64_t s_e[ROW_SORT_WARPS][ROW_SORT_MAX];
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int64_t q = (int64_t)blockIdx.x * ROW_SORT_WARPS + warp;
  if (q >= n) return;  // the whole warp
  int64_t o = offsets[q];
  int m = (int)(offsets[q + 1] - o);
  if (m <= 1) return;
  if (m <= 32) {
    uint32_t key = lane < m ? (uint32_t)idx[o + lane] : 0xffffffffu;
    int val = lane < m && d2 ? __float_as_int(d2[o + lane]) : 0;
    warp_sort_pairs(key, val);
    if (lane < m) {
      idx[o + lane] = (int32_t)key;
      if (d2) d2[o + lane] = __int_as_float(val);
    }
    return;
  }
  int size = 64;
  while (size < m) size <<= 1;
  uint64_t * e = s_e[warp];
  for (int i = lane; i < size; i += 32)
    e[i] = i < m ? ((uint64_t)(uint32_t)idx[o + i] << 32) | (d2 ? __float_as_uint(d2[o + i]) : 0u) : ~0ull;
  __syncwarp();
  for (int k = 2; k <= size; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int t = lane; t < size / 2; t += 32) {
        int lo = ((t & ~(j - 1)) << 1) | (t & (j - 1)), hi = lo | j;
        uint64_t u = e[lo], v = e[hi];
        if ((u > v) == ((lo & k) == 0)) {
          e[lo] = v;
          e[hi] = u;
        }
      }
      __syncwarp();
    }
  }
  for (int i = lane; i < m; i += 32) {
    idx[o + i] = (int32_t)(uint32_t)(e[i] >> 32);
    if (d2) d2[o + i] = __uint_as_float((uint32_t)e[i]);
  }
}

__global__ void range_total_kernel(int64_t const * __restrict__ counts, int64_t n, int64_t * __restrict__ offsets) {
  offsets[n] = offsets[n - 1] + counts[n - 1];
}

__global__ void range_iota_kernel(int64_t total, uint32_t * __restrict__ v) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < total) v[i] = (uint32_t)i;
}

// After the key sort: element index from the low key bits, squared distance gathered through the permutation
__global__ void range_emit_kernel(uint64_t const * __restrict__ keys, uint32_t const * __restrict__ perm,
                                  float const * __restrict__ d2_unsorted, int64_t total, int32_t * __restrict__ out_idx,
                                  float * __restrict__ out_d2) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  out_idx[i] = (int32_t)(uint32_t)(keys[i] & 0xffffffffu);
  if (out_d2) out_d2[i] = d2_unsorted[perm[i]];
}

template <int W, int STACK>
void launch_range(thea_bvh const * b, float const * q, int64_t n, float r2, int32_t const * ex, int64_t * offsets,
                  int32_t * out_idx, float * out_d2, unsigned * err, bool sorted, cudaStream_t s) {
  int per = queries_per_warp(n);
  unsigned grid = sparse_grid(n, per);
  if (out_idx && !sorted) {
    THEA_LAUNCH((range_kernel<W, STACK, 2>), grid, QUERY_THREADS, 0, s, (WideNode<W> const *)b->nodes, b->pt_rec, q,
                n, per, r2, ex, offsets, (uint64_t *)nullptr, out_d2, err, out_idx);
    return;
  }
  if (!out_idx) {
    Scratch counts((size_t)n * sizeof(int64_t), s);
    THEA_LAUNCH((range_kernel<W, STACK, 0>), grid, QUERY_THREADS, 0, s, (WideNode<W> const *)b->nodes, b->pt_rec,
                q, n, per, r2, ex, counts.as<int64_t>(), (uint64_t *)nullptr, (float *)nullptr, err);
    exclusive_scan<int64_t>(counts.as<int64_t>(), offsets, n, s);
    THEA_LAUNCH(range_total_kernel, 1, 1, 0, s, counts.as<int64_t>(), n, offsets);
    return;
  }
  unsigned long long extent[2] = {0, 0};  // neighbours in all, longest row
  {
    Scratch ext(sizeof(extent), s);
    THEA_CUDA_CHECK(cudaMemsetAsync(ext.ptr, 0, sizeof(extent), s));
    THEA_LAUNCH(range_extent_kernel, (unsigned)std::min<int64_t>(ceil_div(n, 256), 256), 256, 0, s, offsets, n,
                ext.as<unsigned long long>());
    THEA_CUDA_CHECK(cudaMemcpyAsync(extent, ext.ptr, sizeof(extent), cudaMemcpyDeviceToHost, s));
    THEA_CUDA_CHECK(cudaStreamSynchronize(s));
  }
  int64_t total = (int64_t)extent[0];
  if (total <= 0) return;
  THEA_REQUIRE(total < (int64_t(1) << 32), "radius_neighbors: more than 2^32 neighbours in one call");
  if (extent[1] <= (unsigned long long)ROW_SORT_MAX) {
    THEA_LAUNCH((range_kernel<W, STACK, 2>), grid, QUERY_THREADS, 0, s, (WideNode<W> const *)b->nodes, b->pt_rec, q,
                n, per, r2, ex, offsets, (uint64_t *)nullptr, out_d2, err, out_idx);
    THEA_LAUNCH(range_sort_rows_kernel, (unsigned)ceil_div(n, ROW_SORT_WARPS), ROW_SORT_WARPS * 32, 0, s, offsets, n,
                out_idx, out_d2);
    return;
  }
  Scratch keys((size_t)total * sizeof(uint64_t), s), d2((size_t)total * sizeof(float), s);
  Scratch perm((size_t)total * sizeof(uint32_t), s);
  THEA_LAUNCH((range_kernel<W, STACK, 1>), grid, QUERY_THREADS, 0, s, (WideNode<W> const *)b->nodes, b->pt_rec, q,
              n, per, r2, ex, offsets, keys.as<uint64_t>(), d2.as<float>(), err);
  THEA_LAUNCH(range_iota_kernel, (unsigned)ceil_div(total, 256), 256, 0, s, total, perm.as<uint32_t>());
  int qbits = 1;
  while ((int64_t(1) << qbits) < n) ++qbits;
  radix_sort_pairs(keys.as<uint64_t>(), perm.as<uint32_t>(), total, 32 + qbits, s);
  THEA_LAUNCH(range_emit_kernel, (unsigned)ceil_div(total, 256), 256, 0, s, keys.as<uint64_t>(), perm.as<uint32_t>(),
              d2.as<float>(), total, out_idx, out_d2);
}

template <int W, int STACK>
void launch_range_rows(thea_bvh const * b, float const * q, int64_t n, float r2, int32_t const * ex, int64_t * offsets,
                       int32_t * rows, int row_cap, unsigned * overflow, unsigned * err, cudaStream_t s) {
  int per = queries_per_warp(n);
  unsigned grid = sparse_grid(n, per);
  Scratch counts((size_t)n * sizeof(int64_t), s);
  THEA_LAUNCH((range_kernel<W, STACK, 3>), grid, QUERY_THREADS, 0, s, (WideNode<W> const *)b->nodes, b->pt_rec, q, n, per,
              r2, ex, counts.as<int64_t>(), (uint64_t *)nullptr, (float *)nullptr, err, rows, row_cap, overflow);
  exclusive_scan<int64_t>(counts.as<int64_t>(), offsets, n, s);
  THEA_LAUNCH(range_total_kernel, 1, 1, 0, s, counts.as<int64_t>(), n, offsets);
}

//============================================================================================================================
// Distance bounds of closest-element queries (BoundCut in query.hpp)
//============================================================================================================================

}  // namespace

RootCut root_cut_of(float const * elem_lo, float const * elem_hi, float const * xf) {
  RootCut r;
  float lo[3], hi[3];
  for (int a = 0; a < 3; ++a) {
    // scaleCentered(1.05f): centre = 0.5 (hi + lo); lo = 1.05 (lo - centre) + centre, hi likewise
    float ctr = 0.5f * (elem_hi[a] + elem_lo[a]);
    lo[a] = 1.05f * (elem_lo[a] - ctr) + ctr;
    hi[a] = 1.05f * (elem_hi[a] - ctr) + ctr;
  }
  if (xf) {
    // transformAndBound: the box of the eight mapped corners
    float wlo[3] = {INFINITY, INFINITY, INFINITY}, whi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int k = 0; k < 8; ++k) {
      V3 w = affine_point(xf, V3{(k & 1) ? hi[0] : lo[0], (k & 2) ? hi[1] : lo[1], (k & 4) ? hi[2] : lo[2]});
      float wc[3] = {w.x, w.y, w.z};
      for (int a = 0; a < 3; ++a) {
        wlo[a] = std::min(wlo[a], wc[a]);
        whi[a] = std::max(whi[a], wc[a]);
      }
    }
    for (int a = 0; a < 3; ++a) lo[a] = wlo[a], hi[a] = whi[a];
  }
  for (int a = 0; a < 3; ++a) r.lo[a] = lo[a], r.hi[a] = hi[a];
  V3 ext = V3{hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2]};
  float nrm = std::sqrt(squared_norm(ext));
  r.fudge = std::max(0.001 * (double)nrm, (double)(100.0f * 1.1920928955078125e-07f));
  return r;
}

namespace {

__global__ void closest_cut_kernel(float const * __restrict__ q, int64_t n, int64_t const * __restrict__ qoff, int M,
                                   BoundCut one, BoundCut const * __restrict__ cuts, int32_t * __restrict__ idx,
                                   float * __restrict__ dist, float * __restrict__ cpt, float * __restrict__ errout) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  BoundCut c = one;
  if (cuts) {
    int lo = 0, hi = M - 1;
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (__ldg(qoff + mid) <= i) lo = mid;
      else hi = mid - 1;
    }
    c = cuts[lo];
  }
  if (!bound_cut_out(c, load_v3(q + 3 * i))) return;
  idx[i] = -1;
  if (dist) dist[i] = -1.f;
  if (cpt) cpt[3 * i] = cpt[3 * i + 1] = cpt[3 * i + 2] = 0.f;
  if (errout) errout[i] = -1.f;
}

}  // namespace

namespace {
__global__ void segment_cuts_kernel(RootCut const * __restrict__ roots, int M, float dist_bound,
                                    BoundCut * __restrict__ out) {
  int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m < M) out[m] = make_bound_cut(roots[m], dist_bound);
}
}  // namespace

void run_segment_cuts(thea_bvh const * b, float dist_bound, BoundCut * out, cudaStream_t s) {
  THEA_REQUIRE(b->seg_roots, "segment cuts: the forest has no per-segment root boxes");
  THEA_LAUNCH(segment_cuts_kernel, (unsigned)ceil_div(b->num_segments, 256), 256, 0, s, b->seg_roots,
              b->num_segments, dist_bound, out);
}

void run_closest_cut(float const * q, int64_t n, BoundCut const & one, int64_t const * qoff, int M,
                     BoundCut const * cuts, int32_t * idx, float * dist, float * cpt, float * errout, cudaStream_t s) {
  if (n <= 0 || (!cuts && one.b2 < 0.0)) return;
  THEA_LAUNCH(closest_cut_kernel, (unsigned)ceil_div(n, 256), 256, 0, s, q, n, qoff, M, one, cuts, idx, dist, cpt,
              errout);
}

namespace {

//============================================================================================================================
// Query ordering: large batches can be traversed in the order of a Morton code of the query point (rays: of the
// origin, with the direction octant as the top bits). Results are written to each query's own slot.
//============================================================================================================================

constexpr int64_t ORDER_MIN_QUERIES = 1 << 15;

__device__ __forceinline__ uint32_t expand10(uint32_t x) {
  x &= 0x3ffu;
  x = (x | x << 16) & 0x030000FFu;
  x = (x | x << 8) & 0x0300F00Fu;
  x = (x | x << 4) & 0x030C30C3u;
  x = (x | x << 2) & 0x09249249u;
  return x;
}

__global__ void query_key_kernel(float const * __restrict__ p, float const * __restrict__ dir, int64_t n, float lx,
                                 float ly, float lz, float sx, float sy, float sz, uint64_t * __restrict__ keys,
                                 uint32_t * __restrict__ vals) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int bits = dir ? 9 : 10;
  float cells = (float)(1 << bits);
  float c[3] = {(p[3 * i] - lx) * sx, (p[3 * i + 1] - ly) * sy, (p[3 * i + 2] - lz) * sz};
  uint32_t q[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float t = fminf(fmaxf(c[a], 0.f), 1.f);  // NaN-safe: fminf/fmaxf drop a NaN operand
    q[a] = min((uint32_t)(t * cells), (uint32_t)(1 << bits) - 1u);
  }
  uint32_t key = (expand10(q[0]) << 2) | (expand10(q[1]) << 1) | expand10(q[2]);
  if (dir) {
    uint32_t oct = (dir[3 * i] < 0.f ? 4u : 0u) | (dir[3 * i + 1] < 0.f ? 2u : 0u) | (dir[3 * i + 2] < 0.f ? 1u : 0u);
    key |= oct << 27;
  }
  keys[i] = key;
  vals[i] = (uint32_t)i;
}

struct QueryOrder {
  Scratch keys, vals;
  uint32_t const * order = nullptr;
  QueryOrder(thea_bvh const * b, float const * p, float const * dir, int64_t n, cudaStream_t s, bool always = false) {
    if ((!b->query_order && !always) || n < ORDER_MIN_QUERIES) return;
    keys = Scratch((size_t)n * sizeof(uint64_t), s);
    vals = Scratch((size_t)n * sizeof(uint32_t), s);
    float sc[3];
    for (int a = 0; a < 3; ++a) {
      float ext = b->hi[a] - b->lo[a];
      sc[a] = ext > 0.f ? 1.0f / ext : 0.f;
    }
    THEA_LAUNCH(query_key_kernel, (unsigned)ceil_div(n, 256), 256, 0, s, p, dir, n, b->lo[0], b->lo[1], b->lo[2],
                sc[0], sc[1], sc[2], keys.as<uint64_t>(), vals.as<uint32_t>());
    radix_sort_pairs(keys.as<uint64_t>(), vals.as<uint32_t>(), n, 30, s, /*probe_passes=*/false);
    order = vals.as<uint32_t>();
  }
};

template <int W, int STACK>
void launch_closest(thea_bvh const * b, float const * q, int64_t n, ClosestParams const & cp, int32_t * idx,
                    float * dist, float * cpt, float * errout, unsigned * err, uint32_t const * order, cudaStream_t s) {
  unsigned grid = (unsigned)ceil_div(n, QUERY_THREADS);
  if (cp.precision == THEA_PRECISION_FP64_RECHECK)
    THEA_LAUNCH((closest_kernel<W, STACK, THEA_PRECISION_FP64_RECHECK>), grid, QUERY_THREADS, 0, s,
                (WideNode<W> const *)b->nodes, b->cp_rec, q, n, cp.thresh, cp.bound2, cp.scene_scale, idx, dist, cpt,
                errout, err, order, b->slabs);
  else
    THEA_LAUNCH((closest_kernel<W, STACK, THEA_PRECISION_FP32_REFERENCE>), grid, QUERY_THREADS, 0, s,
                (WideNode<W> const *)b->nodes, b->cp_rec, q, n, cp.thresh, cp.bound2, cp.scene_scale, idx, dist, cpt,
                errout, err, order, b->slabs);
}

template <int W, int STACK>
void launch_ray(thea_bvh const * b, float const * o, float const * d, int64_t n, RayParams const & rp, float * t,
                int32_t * idx, float * nrm, float * t64, int32_t * idx64, int32_t * flags, unsigned * err,
                uint32_t const * order, cudaStream_t s) {
  unsigned grid = (unsigned)ceil_div(n, QUERY_THREADS);
  if (!rp.recheck && n >= RAY_PERSISTENT_MIN) {
    auto k = ray_persistent_kernel<W, STACK>;
    int sms = sm_count();
    int per_sm = 0;
    THEA_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, QUERY_THREADS, 0));
    unsigned pgrid = (unsigned)std::min<int64_t>((int64_t)std::max(1, per_sm) * sms, grid);
    Scratch counter(sizeof(unsigned long long), s);
    THEA_CUDA_CHECK(cudaMemsetAsync(counter.ptr, 0, sizeof(unsigned long long), s));
    THEA_LAUNCH_NAMED("ray_kernel_persistent", k, pgrid, QUERY_THREADS, 0, s, (WideNode<W> const *)b->nodes,
                      b->ray_rec, o, d, n, rp.max_time, t, idx, nrm, err, order, counter.as<unsigned long long>());
    return;
  }
  int per = queries_per_warp(n);
  grid = sparse_grid(n, per);
  if (rp.recheck)
    THEA_LAUNCH((ray_recheck_kernel<W, STACK>), grid, QUERY_THREADS, 0, s, (WideNode<W> const *)b->nodes, b->ray_rec,
                o, d, n, rp.max_time, t, idx, nrm, t64, idx64, flags, err, order, per);
  else
    THEA_LAUNCH((ray_kernel<W, STACK, false>), grid, QUERY_THREADS, 0, s, (WideNode<W> const *)b->nodes, b->ray_rec, o,
                d, n, rp.max_time, t, idx, nrm, t64, idx64, flags, err, order, per);
}

template <int W, int K, int STACK>
void launch_knn_k(thea_bvh const * b, float const * q, int64_t n, int k, float thresh, int32_t const * ex,
                  int32_t * idx, float * d2, unsigned * err, uint32_t const * order, float const * ib, cudaStream_t s) {
  int per = knn_queries_per_warp(n, W, K, /*triangles=*/false, /*self=*/!q);
  THEA_LAUNCH((knn_kernel<W, K, STACK>), sparse_grid(n, per), QUERY_THREADS, 0, s, (WideNode<W> const *)b->nodes,
              b->pt_rec, q, n, k, thresh, ex, idx, d2, err, order, ib, per);
}

constexpr int64_t KNN_MESH_PACKED = 2048;

template <int W, int K, int STACK>
void launch_knn_mesh_k(thea_bvh const * b, float const * q, int64_t n, int k, float thresh, int32_t const * ex,
                       int32_t * idx, float * d2, unsigned * err, uint32_t const * order, cudaStream_t s) {
  // (a small mesh's queries share its records in L1: 1,000 queries around 1,280 triangles, their nearest, 0.38 ms packed and
  // 0.52 spread)
  int per = b->n <= KNN_MESH_PACKED ? 32 : knn_queries_per_warp(n, W, K, /*triangles=*/true, /*self=*/false);
  THEA_LAUNCH((knn_mesh_kernel<W, K, STACK>), sparse_grid(n, per), QUERY_THREADS, 0, s, (WideNode<W> const *)b->nodes,
              b->cp_rec, q, n, k, thresh, ex, idx, d2, err, order, per);
}

template <int W, int STACK>
void launch_knn_mesh(thea_bvh const * b, float const * q, int64_t n, int k, float thresh, int32_t const * ex,
                     int32_t * idx, float * d2, unsigned * err, uint32_t const * order, cudaStream_t s) {
  if (k <= 1) launch_knn_mesh_k<W, 1, STACK>(b, q, n, k, thresh, ex, idx, d2, err, order, s);
  else if (k <= 4) launch_knn_mesh_k<W, 4, STACK>(b, q, n, k, thresh, ex, idx, d2, err, order, s);
  else if (k <= 8) launch_knn_mesh_k<W, 8, STACK>(b, q, n, k, thresh, ex, idx, d2, err, order, s);
  else if (k <= 16) launch_knn_mesh_k<W, 16, STACK>(b, q, n, k, thresh, ex, idx, d2, err, order, s);
  else launch_knn_mesh_k<W, 32, STACK>(b, q, n, k, thresh, ex, idx, d2, err, order, s);
}

template <int W, int STACK>
void launch_knn(thea_bvh const * b, float const * q, int64_t n, int k, float thresh, int32_t const * ex, int32_t * idx,
                float * d2, unsigned * err, uint32_t const * order, float const * ib, cudaStream_t s) {
  if (b->is_mesh) {
    launch_knn_mesh<W, STACK>(b, q, n, k, thresh, ex, idx, d2, err, order, s);
    return;
  }
  if (k <= 1) launch_knn_k<W, 1, STACK>(b, q, n, k, thresh, ex, idx, d2, err, order, ib, s);
  else if (k <= 2) launch_knn_k<W, 2, STACK>(b, q, n, k, thresh, ex, idx, d2, err, order, ib, s);
  else if (k <= 4) launch_knn_k<W, 4, STACK>(b, q, n, k, thresh, ex, idx, d2, err, order, ib, s);
  else if (k <= 8) launch_knn_k<W, 8, STACK>(b, q, n, k, thresh, ex, idx, d2, err, order, ib, s);
  else if (k <= 16) launch_knn_k<W, 16, STACK>(b, q, n, k, thresh, ex, idx, d2, err, order, ib, s);
  else launch_knn_k<W, 32, STACK>(b, q, n, k, thresh, ex, idx, d2, err, order, ib, s);
}

}  // namespace

bool small_stack_ok(thea_bvh const * b) {
  int need = b->depth * (b->width - 1) + 1;
  return need <= (b->width == 4 ? 64 : 128);
}

void run_closest(thea_bvh const * b, float const * q, int64_t n, ClosestParams const & cp, int32_t * idx, float * dist,
                 float * cpt, float * errout, unsigned * err, cudaStream_t s) {
  if (n <= 0) return;
  if (cp.precision == THEA_PRECISION_FP64_RECHECK) {
    if (n < (f64_small_mesh(b, n) ? F64_WARP_MAX_SMALL : F64_WARP_MAX) && small_stack_ok(b)) {
      run_closest_warps_f64(b, q, n, cp, idx, dist, cpt, errout, s);
      return;
    }
    ClosestParams c2 = cp;
    c2.budget = f64_collect_budget(b, n);
    if (c2.budget > 0) {
      run_batch_closest(b, q, nullptr, n, c2, 64, idx, dist, cpt, errout, s);
      return;
    }
  }
  if (cp.precision == THEA_PRECISION_FP32_REFERENCE && !errout && !b->query_order &&
      (n < CLOSEST_WARP_MAX || n >= CLOSEST_TWO_PHASE_MIN)) {
    if (n < (b->width == 4 ? CLOSEST_WARP_MAX : CLOSEST_TEAM_MAX_W8) && small_stack_ok(b)) {
      run_closest_teams(b, q, n, cp, idx, dist, cpt, s);
      return;
    }
    // Persistent lanes with a step budget, then one warp per query over budget (the BVH is a one-mesh forest). The
    // same searches, so the same results.
    ClosestParams c2 = cp;
    c2.budget = n < CLOSEST_WARP_MAX ? CLOSEST_WARP_BUDGET : CLOSEST_TWO_PHASE_BUDGET;
    run_batch_closest(b, q, nullptr, n, c2, 64, idx, dist, cpt, nullptr, s);
    return;
  }
  // FP64 re-check: warps of Morton-ordered queries share band candidates (config 0: 2.64 -> 2.26 ms), so the order is
  // taken whatever the BVH's query_order option says
  QueryOrder ord(b, q, nullptr, n, s, cp.precision == THEA_PRECISION_FP64_RECHECK);
  uint32_t const * o = ord.order;
  bool sm = small_stack_ok(b);
  if (b->width == 4) sm ? launch_closest<4, 64>(b, q, n, cp, idx, dist, cpt, errout, err, o, s)
                        : launch_closest<4, 256>(b, q, n, cp, idx, dist, cpt, errout, err, o, s);
  else sm ? launch_closest<8, 128>(b, q, n, cp, idx, dist, cpt, errout, err, o, s)
          : launch_closest<8, 512>(b, q, n, cp, idx, dist, cpt, errout, err, o, s);
}

void run_ray(thea_bvh const * b, float const * o, float const * d, int64_t n, RayParams const & rp, float * t,
             int32_t * idx, float * nrm, float * t64, int32_t * idx64, int32_t * flags, unsigned * err, cudaStream_t s) {
  if (n <= 0) return;
  QueryOrder ord(b, o, d, n, s);
  uint32_t const * od = ord.order;
  bool sm = small_stack_ok(b);
  if (b->width == 4) sm ? launch_ray<4, 64>(b, o, d, n, rp, t, idx, nrm, t64, idx64, flags, err, od, s)
                        : launch_ray<4, 256>(b, o, d, n, rp, t, idx, nrm, t64, idx64, flags, err, od, s);
  else sm ? launch_ray<8, 128>(b, o, d, n, rp, t, idx, nrm, t64, idx64, flags, err, od, s)
          : launch_ray<8, 512>(b, o, d, n, rp, t, idx, nrm, t64, idx64, flags, err, od, s);
}

void run_ray_stream(thea_bvh const * b, float const * o, float const * d, int64_t n, float max_time, float * t,
                    int32_t * idx, unsigned * err, cudaStream_t s) {
  if (n <= 0) return;
  bool sm = small_stack_ok(b);
  if (b->width == 4) sm ? launch_ray_stream<4, 64>(b, o, d, n, max_time, t, idx, err, s)
                        : launch_ray_stream<4, 256>(b, o, d, n, max_time, t, idx, err, s);
  else sm ? launch_ray_stream<8, 128>(b, o, d, n, max_time, t, idx, err, s)
          : launch_ray_stream<8, 512>(b, o, d, n, max_time, t, idx, err, s);
}

void run_range(thea_bvh const * b, float const * q, int64_t n, float radius, int32_t const * ex, int64_t * offsets,
               int32_t * idx, float * d2, unsigned * err, cudaStream_t s, bool sorted) {
  if (n <= 0) return;
  float r2 = radius * radius;  // BallN::contains compares with radius * radius in FP32
  bool sm = small_stack_ok(b);
  if (b->width == 4) sm ? launch_range<4, 64>(b, q, n, r2, ex, offsets, idx, d2, err, sorted, s)
                        : launch_range<4, 256>(b, q, n, r2, ex, offsets, idx, d2, err, sorted, s);
  else sm ? launch_range<8, 128>(b, q, n, r2, ex, offsets, idx, d2, err, sorted, s)
          : launch_range<8, 512>(b, q, n, r2, ex, offsets, idx, d2, err, sorted, s);
}

void run_range_rows(thea_bvh const * b, float const * q, int64_t n, float radius, int32_t const * ex,
                    int64_t * offsets, int32_t * rows, int row_cap, unsigned * overflow, unsigned * err, cudaStream_t s) {
  if (n <= 0) return;
  float r2 = radius * radius;
  bool sm = small_stack_ok(b);
  if (b->width == 4) sm ? launch_range_rows<4, 64>(b, q, n, r2, ex, offsets, rows, row_cap, overflow, err, s)
                        : launch_range_rows<4, 256>(b, q, n, r2, ex, offsets, rows, row_cap, overflow, err, s);
  else sm ? launch_range_rows<8, 128>(b, q, n, r2, ex, offsets, rows, row_cap, overflow, err, s)
          : launch_range_rows<8, 512>(b, q, n, r2, ex, offsets, rows, row_cap, overflow, err, s);
}

void run_knn(thea_bvh const * b, float const * q, int64_t n, int k, float thresh, int32_t const * ex, int32_t * idx,
             float * d2, unsigned * err, cudaStream_t s, float const * init_bound) {
  if (n <= 0) return;
  // self mode already runs in leaf order
  QueryOrder ord(b, q, nullptr, q ? n : 0, s);
  uint32_t const * o = ord.order;
  float const * ib = q ? nullptr : init_bound;
  bool sm = small_stack_ok(b);
  if (b->width == 4) sm ? launch_knn<4, 64>(b, q, n, k, thresh, ex, idx, d2, err, o, ib, s)
                        : launch_knn<4, 256>(b, q, n, k, thresh, ex, idx, d2, err, o, ib, s);
  else sm ? launch_knn<8, 128>(b, q, n, k, thresh, ex, idx, d2, err, o, ib, s)
          : launch_knn<8, 512>(b, q, n, k, thresh, ex, idx, d2, err, o, ib, s);
}

}  // namespace thea
