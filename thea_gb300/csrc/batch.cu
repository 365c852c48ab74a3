// Batched queries over a forest (one BVH per mesh or point set, built together by build_forest).
//
// One persistent launch serves every mesh: the grid is sized to fill the GPU once (blocks per SM x SMs), and each warp
// repeatedly takes the next chunk of queries from a global counter, so meshes with 1k or 100k queries and 320 or
// 327,680 triangles share the SMs without a tail of idle blocks. Queries are grouped by mesh (query_offsets, M + 1
// entries); a lane finds its query's mesh by binary search and starts from that mesh's root node. The whole call is
// asynchronous and allocation-stable, so it can be captured once into a CUDA graph and replayed.
#include "batch.hpp"
#include "device_util.cuh"
#include "knn_points.cuh"
#include "traverse_ops.cuh"
#include "warp_traverse.cuh"

#include <algorithm>
#include <chrono>
#include <vector>

namespace thea {
namespace {

constexpr int BATCH_THREADS = 128;

__device__ __forceinline__ int mesh_of_query(int64_t const * __restrict__ qoff, int M, int64_t q) {
  int lo = 0, hi = M - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (__ldg(qoff + mid) <= q) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Each warp takes `chunk` consecutive queries per fetch; lanes stride through them.
__device__ __forceinline__ bool next_chunk(unsigned long long * counter, int chunk, int64_t nq, int64_t & base) {
  unsigned long long b = 0;
  if ((threadIdx.x & 31) == 0) b = atomicAdd(counter, (unsigned long long)chunk);
  b = __shfl_sync(0xffffffffu, b, 0);
  base = (int64_t)b;
  return base < nq;
}

//============================================================================================================================
// Closest element. With error estimates (batch_closest_kernel) each warp works in rounds of 32 queries, one per lane; every
// lane of the warp takes part in every round (lanes past the end of the chunk carry no query), so the FP64 error estimate
// runs with all lanes together. Without, and in the mixed-precision mode, lanes take new queries as theirs end.
//
// Two-phase form: with budget > 0, phase 1 stops a query after that many steps (nodes and leaves) and queues it with the best
// element found so far (a valid upper bound); phase 2 finishes the queued queries with one warp per query.
//============================================================================================================================

struct HardQueue {
  int64_t * q;
  float * bound;  // FP32 squared distance of the best element found so far (+inf if none)
  int32_t * idx;
  int64_t * slot;
  unsigned long long * count;
};

// d64: FP64 squared distance of the returned element (for the error estimate)
__device__ __forceinline__ void write_closest(int64_t q, bool found, float dist, V3 cp, int idx, double d64,
                                              int32_t * out_index, float * out_dist, float * out_cp, float * out_err) {
  out_index[q] = found ? idx : -1;
  if (out_dist) out_dist[q] = found ? dist : -1.f;
  if (out_cp) {
    out_cp[3 * q] = found ? cp.x : 0.f;
    out_cp[3 * q + 1] = found ? cp.y : 0.f;
    out_cp[3 * q + 2] = found ? cp.z : 0.f;
  }
  if (out_err) out_err[q] = found ? (float)fabs((double)dist - sqrt(d64)) : -1.f;
}

struct ClosestArgs {
  float const * queries;
  int64_t const * qoff;
  float thresh;
  double bound2;
  float scene_scale;
  int32_t * out_index;
  float * out_dist;
  float * out_cp;
  float * out_err;
  BoundCut const * seg_cut = nullptr;  // per mesh: thresh and bound2 of that mesh (nullptr: the scalars for all)
};

__device__ __forceinline__ float thresh_of(ClosestArgs const & a, int m) {
  return a.seg_cut ? a.seg_cut[m].thresh : a.thresh;
}
__device__ __forceinline__ double bound2_of(ClosestArgs const & a, int m) {
  return a.seg_cut ? a.seg_cut[m].bound2 : a.bound2;
}

// One round: lane query q when active. Called by all 32 lanes of the warp together.
template <int W, int STACK>
__device__ __forceinline__ void closest_round(BatchForest const & f, ClosestArgs const & a, int64_t q, bool active,
                                              int budget, HardQueue const & hq) {
  WideNode<W> const * nodes = (WideNode<W> const *)f.nodes;
  V3 p = V3{0.f, 0.f, 0.f};
  ClosestOut r;
  r.idx = INT_MAX;
  r.d2 = 0.f;
  r.slot = -1;
  r.best32 = INFINITY;
  r.done = true;
  if (active) {
    int m = mesh_of_query(a.qoff, f.M, q);
    p = load_v3(a.queries + 3 * q);
    r = closest_query<W, STACK>(nodes, f.cp_rec, __ldg(f.seg_root + m), __ldg(f.seg_start + m), p, thresh_of(a, m), f.err,
                                budget);
  }
  float dist = sqrtf(r.d2);
  if (active && !r.done) {
    unsigned long long pos = atomicAdd(hq.count, 1ull);
    hq.q[pos] = q;
    hq.bound[pos] = r.best32;
    hq.idx[pos] = r.idx;
    hq.slot[pos] = r.slot;
  }
  bool fin = active && r.done;
  bool found = r.idx != INT_MAX;
  double d64 = 0.0;
  if (a.out_err) {
    __syncwarp();
    if (fin && found) {
      D3 cp64;
      cp_record_f64(f.cp_rec, r.slot, p, cp64, d64);
    }
  }
  if (fin) write_closest(q, found, dist, r.cp, r.idx, d64, a.out_index, a.out_dist, a.out_cp, a.out_err);
}

template <int W, int STACK>
__global__ void __launch_bounds__(BATCH_THREADS)
batch_closest_kernel(BatchForest f, ClosestArgs a, int64_t nq, unsigned long long * counter, int chunk, int budget,
                     HardQueue hq) {
  int lane = threadIdx.x & 31;
  int64_t base;
  while (next_chunk(counter, chunk, nq, base)) {
    int64_t end = base + chunk < nq ? base + chunk : nq;
    for (int64_t r0 = base; r0 < end; r0 += 32)
      closest_round<W, STACK>(f, a, r0 + lane, r0 + lane < end, budget, hq);
  }
}

// Persistent-lane form of batch_closest_kernel: lanes take new queries as theirs end, instead of idling until the slowest
// query of its warp's round (the queries deep inside a mesh take ten times the steps of the others). Every loop iteration
// advances each busy lane by one stack entry; idle lanes are refilled from a warp-local block of query indices (`block`).
// FP32 search only; closest_collect_kernel below is the mixed-precision form. Results are the round-based kernel's: each
// query's search is the same sequence of steps.
//
// What bounds it: the L1 data pipe (68 % busy), the issue slots (65 %) and the latency of the node and record loads, with
// a third of the lanes active (a warp mixes lanes at nodes, at leaves and between queries). One 128-byte line per lane and
// step through 32-byte loads, issued before node and leaf lanes part ways (closest_step), and the first 24 stack entries
// in shared memory (SharedStack): 262,144 queries on 81,920 triangles 1.41 -> 1.13 ms, 256 meshes with 5.2 M queries 12.4
// -> 9.85 ms; 1.04 and 9.01 with the refill below. Measured and not taken: blocks of 16 or 32 indices (within 3 %); a
// lower step budget once the indices run out (1.27 -> 1.74 ms at 128); queries in Morton order (1.18 -> 1.21 ms before the
// sort's own time); a line fetched by eight lanes with 16-byte asynchronous copies into shared memory (1.04 -> 1.47 ms:
// fewer wavefronts, but every step waits for the copies and reads the line once more).
//
// Lanes without a query wait until this many of their warp's do (or all of them), so that results are written and queries
// fetched for several lanes at a time. FP32, refilled at 1 / 2 / 4 / 8 lanes: 262,144 queries near 81,920 triangles 0.270 /
// 0.270 / 0.270 / 0.289 ms (0.296 with each result written as it ends), 256 meshes with 5.2 M queries 9.62 / 9.25 / 9.01 /
// 8.99 (9.81). The collecting kernel, whose lanes also pack their band entries: 100,003 queries 0.934 / 0.934 / 0.933 /
// 0.783 (0.951); 12 and 16 lanes as 8.
constexpr int CLOSEST_REFILL_AT = 4, COLLECT_REFILL_AT = 8;
constexpr int REFILL_BLOCK = 64;

template <int W, int STACK>
__global__ void __launch_bounds__(BATCH_THREADS)
batch_closest_refill_kernel(BatchForest f, ClosestArgs a, int64_t nq, unsigned long long * counter, int budget,
                            HardQueue hq, int block) {
  unsigned const FULL = 0xffffffffu;
  int lane = threadIdx.x & 31;
  WideNode<W> const * nodes = (WideNode<W> const *)f.nodes;
  int64_t qb = 0, qe = 0;  // warp-local block of query indices, warp-uniform
  bool exhausted = false;  // warp-uniform
  int64_t q = -1;          // this lane's query (-1: idle)
  int64_t ebase = 0;
  V3 p = V3{0.f, 0.f, 0.f};
  __shared__ int2 s_stk[CLOSEST_SHARED_STACK][BATCH_THREADS];
  SharedStack<STACK, CLOSEST_SHARED_STACK, BATCH_THREADS> stk(s_stk);
  int sp = 0;
  int next = CHILD_EMPTY;  // nearest child of the last node, visited next without a stack round trip
  float best = 0.f;  // best squared distance
  int best_idx = INT_MAX;
  int64_t best_slot = -1;
  V3 best_cp = V3{0.f, 0.f, 0.f};
  int pops = 0;  // stack entries taken by this lane's query (two-phase form: budget > 0)
  while (true) {
    // lanes whose query is done, or that have none
    bool done = next == CHILD_EMPTY && sp == 0;
    unsigned idle = __ballot_sync(FULL, done);
    if (__popc(idle) >= CLOSEST_REFILL_AT || idle == FULL) {
      if (done && q >= 0) {
        write_closest(q, best_idx != INT_MAX, sqrtf(best), best_cp, best_idx, 0.0, a.out_index, a.out_dist, a.out_cp,
                      nullptr);
        q = -1;
      }
      if (exhausted && idle == FULL) break;
    }
    if ((__popc(idle) >= CLOSEST_REFILL_AT || idle == FULL) && !exhausted) {
      if (qb >= qe) {
        unsigned long long b = 0;
        if (lane == 0) b = atomicAdd(counter, (unsigned long long)block);
        b = __shfl_sync(FULL, b, 0);
        qb = (int64_t)b;
        qe = qb + block < nq ? qb + block : nq;
        if (qb >= nq) exhausted = true;
      }
      if (!exhausted) {
        int rank = __popc(idle & ((1u << lane) - 1));
        int64_t avail = qe - qb;
        int64_t take = __popc(idle);
        if (done && rank < avail) {
          done = false;
          q = qb + rank;
          int m = mesh_of_query(a.qoff, f.M, q);
          ebase = __ldg(f.seg_start + m);
          p = load_v3(a.queries + 3 * q);
          sp = 0;
          next = __ldg(f.seg_root + m);
          pops = 0;
          best = thresh_of(a, m);
          best_idx = INT_MAX;
          best_slot = -1;
        }
        qb += take < avail ? take : avail;
      }
    }
    if (done) continue;
    if (budget > 0 && ++pops > budget) {
      // over budget (steps taken, the register-held child included): queued with the best element so far, finished
      // by a warp of its own in the second kernel
      unsigned long long pos = atomicAdd(hq.count, 1ull);
      hq.q[pos] = q;
      hq.bound[pos] = best;
      hq.idx[pos] = best_idx;
      hq.slot[pos] = best_slot;
      q = -1;
      next = CHILD_EMPTY;
      sp = 0;
      continue;
    }
    int code = next;
    if (code == CHILD_EMPTY) {
      --sp;
      int2 top = stk.get(sp);
      code = top.x;
      if (__int_as_float(top.y) > best * PRUNE_SLACK) continue;
    }
    closest_step<W>(nodes, f.cp_rec, ebase, code, p, best, best_idx, best_slot, best_cp, stk, sp, next, f.err, nullptr,
                    0.f);
    pops -= leaf_rest(code, next);
  }
}

// The mixed-precision search in two kernels. closest_collect_kernel is the persistent-lane FP32 traversal above with the
// band rule of closest_search_f64: it keeps the elements whose FP32 distance lies within the band of the best (in shared
// memory, F64_CAND a lane) and leaves each query's final band entries in `cand`, -1 past the last. closest_resolve_kernel
// evaluates them in FP64, 32 queries to a warp in full-warp rounds (f64_resolve_warp). Apart, the traversal runs at the
// FP32 search's registers and refills its lanes, and the FP64 pipe sees nothing but full rounds; one kernel that does both
// needs 128 registers, or idles lanes until their warp's next round. A query over the step budget, or with more band
// entries than fit (rare), goes to the warp-per-query kernel with the FP32 best as its bound. Results do not depend on who
// finishes a query.
constexpr int F64_HARD = -2;  // cand[0] of a query left to the warp-per-query kernel

template <int W, int STACK>
__global__ void __launch_bounds__(BATCH_THREADS)
closest_collect_kernel(BatchForest f, ClosestArgs a, int64_t nq, unsigned long long * counter, int budget, HardQueue hq,
                       int block, int32_t * __restrict__ cand) {
  __shared__ int2 s_stk[CLOSEST_SHARED_STACK][BATCH_THREADS];
  __shared__ float s_cd[F64_CAND][BATCH_THREADS];
  __shared__ int s_ck[F64_CAND][BATCH_THREADS];
  unsigned const FULL = 0xffffffffu;
  float const REL = 1.0f + 1.0f / 16384.0f;
  int lane = threadIdx.x & 31, t = threadIdx.x;
  WideNode<W> const * nodes = (WideNode<W> const *)f.nodes;
  int64_t qb = 0, qe = 0;  // warp-local block of query indices, warp-uniform
  bool exhausted = false;  // warp-uniform
  int64_t q = -1;          // this lane's query (-1: idle)
  int64_t ebase = 0;
  V3 p = V3{0.f, 0.f, 0.f};
  SharedStack<STACK, CLOSEST_SHARED_STACK, BATCH_THREADS> stk(s_stk);
  int sp = 0;
  int next = CHILD_EMPTY;  // nearest child of the last node, visited next without a stack round trip
  float lim = 0.f;         // band limit on FP32 squared distances
  float best32 = INFINITY, abs_tol = 0.f;
  int nc = 0;     // entries kept, some of them outside the band by now
  int steps = 0;  // (two-phase form: budget > 0)
  while (true) {
    // lanes whose query is done, or that have none
    bool done = next == CHILD_EMPTY && sp == 0;
    unsigned idle = __ballot_sync(FULL, done);
    if (__popc(idle) >= COLLECT_REFILL_AT || idle == FULL) {
      if (done && q >= 0) {
        // finished: the entries still in the band
        int out[F64_CAND];
        int c = 0;
  #pragma unroll
        for (int j = 0; j < F64_CAND; ++j) out[j] = -1;
        for (int j = 0; j < nc; ++j) {
          if (s_cd[j][t] <= lim) {
            int k = s_ck[j][t];
  #pragma unroll
            for (int u = 0; u < F64_CAND; ++u) out[u] = u == c ? k : out[u];
            ++c;
          }
        }
        int4 * o = reinterpret_cast<int4 *>(cand + q * F64_CAND);
  #pragma unroll
        for (int j = 0; j < F64_CAND; j += 4) o[j / 4] = make_int4(out[j], out[j + 1], out[j + 2], out[j + 3]);
        q = -1;
      }
      if (exhausted && idle == FULL) break;
    }
    if ((__popc(idle) >= COLLECT_REFILL_AT || idle == FULL) && !exhausted) {
      if (qb >= qe) {
        unsigned long long b = 0;
        if (lane == 0) b = atomicAdd(counter, (unsigned long long)block);
        b = __shfl_sync(FULL, b, 0);
        qb = (int64_t)b;
        qe = qb + block < nq ? qb + block : nq;
        if (qb >= nq) exhausted = true;
      }
      if (!exhausted) {
        int rank = __popc(idle & ((1u << lane) - 1));
        int64_t avail = qe - qb;
        int64_t take = __popc(idle);
        if (done && rank < avail) {
          done = false;
          q = qb + rank;
          int m = mesh_of_query(a.qoff, f.M, q);
          ebase = __ldg(f.seg_start + m);
          p = load_v3(a.queries + 3 * q);
          sp = 0;
          next = __ldg(f.seg_root + m);
          steps = 0;
          nc = 0;
          float scale = fmaxf(a.scene_scale, fmaxf(fabsf(p.x), fmaxf(fabsf(p.y), fabsf(p.z))));
          lim = f64_band_start(bound2_of(a, m), scale, abs_tol);
          best32 = INFINITY;
        }
        qb += take < avail ? take : avail;
      }
    }
    if (done) continue;
    bool hard = budget > 0 && ++steps > budget;
    if (!hard) {
      int code = next;
      if (code == CHILD_EMPTY) {
        --sp;
        int2 top = stk.get(sp);
        code = top.x;
        if (__int_as_float(top.y) > lim * PRUNE_SLACK) continue;
      }
      next = CHILD_EMPTY;
      int first = 0, count = 0;
      if (code < 0) decode_leaf(code, first, count);
      auto children = [&](NodeRegs<W> const & nd) {
        float lb[W];
        point_child_bounds<W>(nd, p, lb);
        push_children_next<W>(nd, lb, lim * PRUNE_SLACK, stk, sp, next, f.err);
      };
      auto take = [&](float d2, int kr) {
        if (!(d2 <= lim)) return;
        if (d2 < best32) {
          best32 = d2;
          float lb1 = sqrtf(best32) * REL + abs_tol;
          lim = fminf(lim, lb1 * lb1);
        }
        if (nc == F64_CAND) {
          // drop the entries that have left the band
          int m = 0;
          for (int j = 0; j < F64_CAND; ++j) {
            float d = s_cd[j][t];
            int k = s_ck[j][t];
            if (d <= lim) {
              s_cd[m][t] = d;
              s_ck[m][t] = k;
              ++m;
            }
          }
          nc = m;
        }
        if (nc < F64_CAND) {
          s_cd[nc][t] = d2;
          s_ck[nc][t] = kr;
          ++nc;
        } else {
          hard = true;  // more entries in the band than fit
        }
      };
      if constexpr (W == 4) {
        int64_t k = ebase + first;
        float4 r[8];
        load_line(code >= 0 ? reinterpret_cast<float4 const *>(nodes + code) : f.cp_rec + k * CP_REC_F4, r);
        if (code >= 0) {
          NodeRegs<W> nd;
          node_from_line(r, nd);
          children(nd);
        } else {
          V3 cp;
          take(cp_record_eval(r, p, cp), first);
          if (count > 1) next = encode_leaf(first + 1, count - 1);
          steps -= leaf_rest(code, next);
        }
      } else {
        if (code >= 0) {
          NodeRegs<W> nd;
          load_node(nodes, code, nd);
          children(nd);
        } else {
          V3 cp;
          take(cp_record_test(f.cp_rec, ebase + first, p, cp), first);
          if (count > 1) next = encode_leaf(first + 1, count - 1);
          steps -= leaf_rest(code, next);
        }
      }
    }
    if (hard) {
      unsigned long long pos = atomicAdd(hq.count, 1ull);
      hq.q[pos] = q;
      hq.bound[pos] = best32;
      hq.idx[pos] = INT_MAX;
      hq.slot[pos] = -1;
      cand[q * F64_CAND] = F64_HARD;
      q = -1;
      next = CHILD_EMPTY;
      sp = 0;
    }
  }
}

__global__ void __launch_bounds__(BATCH_THREADS)
closest_resolve_kernel(BatchForest f, ClosestArgs a, int64_t q0, int64_t nq, int32_t const * __restrict__ cand) {
  __shared__ F64WarpBuf s_buf[BATCH_THREADS / 32];
  int64_t q = q0 + (int64_t)blockIdx.x * BATCH_THREADS + threadIdx.x;
  bool active = q < nq;
  F64Search s;
  f64_search_init(s);
  int64_t ebase = 0;
  double bound2 = -1.0;
  V3 p = V3{0.f, 0.f, 0.f};
  if (active) {
    int4 const * c = reinterpret_cast<int4 const *>(cand + q * F64_CAND);
#pragma unroll
    for (int j = 0; j < F64_CAND; j += 4) {
      int4 v = __ldg(c + j / 4);
      s.cand_k[j] = v.x;
      s.cand_k[j + 1] = v.y;
      s.cand_k[j + 2] = v.z;
      s.cand_k[j + 3] = v.w;
    }
    if (s.cand_k[0] == F64_HARD) {
      active = false;
    } else {
#pragma unroll
      for (int j = 0; j < F64_CAND; ++j) s.cand_d[j] = 0.f;  // all of them lie in the band
      int m = mesh_of_query(a.qoff, f.M, q);
      ebase = __ldg(f.seg_start + m);
      bound2 = bound2_of(a, m);
      p = load_v3(a.queries + 3 * q);
    }
  }
  f64_resolve_warp(s, active, f.cp_rec, ebase, p, bound2, s_buf[threadIdx.x >> 5]);
  if (!active) return;
  ClosestOut r = f64_result(s);
  write_closest(q, r.idx != INT_MAX, (float)sqrt(r.d2_64), r.cp, r.idx, r.d2_64, a.out_index, a.out_dist, a.out_cp,
                a.out_err);
}

constexpr int PHASE2_WARPS = BATCH_THREADS / 32;

template <int W, int PREC>
__global__ void __launch_bounds__(BATCH_THREADS)
batch_closest_phase2_kernel(BatchForest f, ClosestArgs a, HardQueue hq, unsigned long long * counter) {
  __shared__ int s_code[PHASE2_WARPS][WARP_STACK];
  __shared__ float s_lb[PHASE2_WARPS][WARP_STACK];
  __shared__ float s_cd[PHASE2_WARPS][PREC == THEA_PRECISION_FP64_RECHECK ? WARP_CAND : 1];
  __shared__ int64_t s_ck[PHASE2_WARPS][PREC == THEA_PRECISION_FP64_RECHECK ? WARP_CAND : 1];
  WideNode<W> const * nodes = (WideNode<W> const *)f.nodes;
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned long long total = *hq.count;
  while (true) {
    unsigned long long j = 0;
    if (lane == 0) j = atomicAdd(counter, 1ull);
    j = __shfl_sync(0xffffffffu, j, 0);
    if (j >= total) break;
    int64_t q = hq.q[j];
    int m = mesh_of_query(a.qoff, f.M, q);
    int root = __ldg(f.seg_root + m);
    int64_t ebase = __ldg(f.seg_start + m);
    V3 p = load_v3(a.queries + 3 * q);
    if (PREC == THEA_PRECISION_FP64_RECHECK) {
      float scale = fmaxf(a.scene_scale, fmaxf(fabsf(p.x), fmaxf(fabsf(p.y), fabsf(p.z))));
      WarpBest64 b = closest_warp_query_f64<W>(nodes, f.cp_rec, root, ebase, p, bound2_of(a, m), scale, hq.bound[j],
                                               s_code[warp], s_lb[warp], s_cd[warp], s_ck[warp], f.err, f.slabs);
      if (lane == 0) {
        bool found = b.idx != INT_MAX;
        V3 cp = V3{0.f, 0.f, 0.f};
        if (found) {
          D3 cp64;
          double d64;
          cp_record_f64(f.cp_rec, b.slot, p, cp64, d64);
          cp = V3{(float)cp64.x, (float)cp64.y, (float)cp64.z};
        }
        write_closest(q, found, (float)sqrt(b.d2), cp, b.idx, b.d2, a.out_index, a.out_dist, a.out_cp, a.out_err);
      }
    } else {
      WarpBest init;
      init.idx = hq.idx[j];
      init.d2 = init.idx != INT_MAX ? hq.bound[j] : thresh_of(a, m);
      init.slot = hq.slot[j];
      // the queries over budget are the long searches (deep inside closed surfaces), which the slabs cut most
      WarpBest b = closest_warp_query<W>(nodes, f.cp_rec, root, ebase, p, init, s_code[warp], s_lb[warp], f.err,
                                         f.slabs);
      if (lane == 0) {
        bool found = b.idx != INT_MAX;
        V3 cp = V3{0.f, 0.f, 0.f};
        double d64 = 0.0;
        if (found) {
          cp_record_test(f.cp_rec, b.slot, p, cp);
          if (a.out_err) {
            D3 cp64;
            cp_record_f64(f.cp_rec, b.slot, p, cp64, d64);
          }
        }
        write_closest(q, found, sqrtf(b.d2), cp, b.idx, d64, a.out_index, a.out_dist, a.out_cp, a.out_err);
      }
    }
    __syncwarp();
  }
}

// A warp per query from the root, FP64 re-check, one BVH: the small-batch form of the mixed-precision search
template <int W>
__global__ void __launch_bounds__(BATCH_THREADS)
closest_warp_f64_kernel(BatchForest f, ClosestArgs a, int64_t nq) {
  __shared__ int s_code[PHASE2_WARPS][WARP_STACK];
  __shared__ float s_lb[PHASE2_WARPS][WARP_STACK];
  __shared__ float s_cd[PHASE2_WARPS][WARP_CAND];
  __shared__ int64_t s_ck[PHASE2_WARPS][WARP_CAND];
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int64_t q = (int64_t)blockIdx.x * PHASE2_WARPS + warp;
  if (q >= nq) return;  // the whole warp
  V3 p = load_v3(a.queries + 3 * q);
  float scale = fmaxf(a.scene_scale, fmaxf(fabsf(p.x), fmaxf(fabsf(p.y), fabsf(p.z))));
  WarpBest64 b = closest_warp_query_f64<W>((WideNode<W> const *)f.nodes, f.cp_rec, 0, 0, p, a.bound2, scale, INFINITY,
                                           s_code[warp], s_lb[warp], s_cd[warp], s_ck[warp], f.err, f.slabs);
  if (lane == 0) {
    bool found = b.idx != INT_MAX;
    V3 cp = V3{0.f, 0.f, 0.f};
    if (found) {
      D3 cp64;
      double d64;
      cp_record_f64(f.cp_rec, b.slot, p, cp64, d64);
      cp = V3{(float)cp64.x, (float)cp64.y, (float)cp64.z};
    }
    write_closest(q, found, (float)sqrt(b.d2), cp, b.idx, b.d2, a.out_index, a.out_dist, a.out_cp, a.out_err);
  }
}

// TEAM lanes per query from the root, FP32, one BVH: the small-batch form, in one launch. What bounds it is the longest
// query's chain of dependent steps; a search on one thread takes four to ten times as many.
template <int W, int TEAM>
__global__ void __launch_bounds__(BATCH_THREADS)
closest_team_kernel(BatchForest f, ClosestArgs a, int64_t nq) {
  constexpr int TEAMS = BATCH_THREADS / TEAM;
  constexpr int CAP = TEAM == 32 ? WARP_STACK : 256;
  __shared__ int s_code[TEAMS][CAP];
  __shared__ float s_lb[TEAMS][CAP];
  int team = threadIdx.x / TEAM;
  int64_t q = (int64_t)blockIdx.x * TEAMS + team;
  bool active = q < nq;
  V3 p = active ? load_v3(a.queries + 3 * q) : V3{0.f, 0.f, 0.f};
  WarpBest b = closest_team_query<W, TEAM>((WideNode<W> const *)f.nodes, f.cp_rec, active, p, a.thresh, s_code[team],
                                           s_lb[team], CAP, f.err, f.slabs);
  if (active && threadIdx.x % TEAM == 0) {
    bool found = b.idx != INT_MAX;
    V3 cp = V3{0.f, 0.f, 0.f};
    if (found) cp_record_test(f.cp_rec, b.slot, p, cp);
    write_closest(q, found, sqrtf(b.d2), cp, b.idx, 0.0, a.out_index, a.out_dist, a.out_cp, nullptr);
  }
}

// Closest point of one BVH with queries and results in pinned host memory, read and written by the kernel (the
// in-place form of the first phase above, FP32 reference arithmetic): a warp copies each 64-query block into shared
// memory once, results collect in a per-warp ring of block buffers and are written out in query order with coalesced
// stores once the block is done. A query over the step budget is queued as in the first phase and counts as done for
// its block; the warp-per-query kernel then writes its result over the block's placeholder.
constexpr int CP_STREAM_RING = 4;
constexpr int CP_STREAM_WARPS = BATCH_THREADS / 32;

template <int W, int STACK>
__global__ void __launch_bounds__(BATCH_THREADS)
closest_stream_kernel(BatchForest f, ClosestArgs a, int64_t nq, unsigned long long * counter, int budget,
                      HardQueue hq) {
  __shared__ float s_in[CP_STREAM_WARPS][REFILL_BLOCK * 3];
  __shared__ int s_i[CP_STREAM_WARPS][CP_STREAM_RING][REFILL_BLOCK];
  __shared__ float s_d[CP_STREAM_WARPS][CP_STREAM_RING][REFILL_BLOCK];
  __shared__ float s_c[CP_STREAM_WARPS][CP_STREAM_RING][REFILL_BLOCK * 3];
  __shared__ int s_left[CP_STREAM_WARPS][CP_STREAM_RING];
  __shared__ long long s_base[CP_STREAM_WARPS][CP_STREAM_RING];
  __shared__ int s_cnt[CP_STREAM_WARPS][CP_STREAM_RING];
  unsigned const FULL = 0xffffffffu;
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  WideNode<W> const * nodes = (WideNode<W> const *)f.nodes;
  int const root = __ldg(f.seg_root);
  float * in = s_in[warp];
  int64_t qb = 0, qe = 0;  // queries of the current block not yet handed out, warp-uniform
  bool exhausted = false;  // warp-uniform
  long long taken = 0, oldest = 0;  // blocks taken / oldest block not written out, warp-uniform
  int64_t q = -1;
  int slot = 0;
  int64_t qbase = 0;
  V3 p = V3{0.f, 0.f, 0.f};
  __shared__ int2 s_stk[CLOSEST_SHARED_STACK][BATCH_THREADS];
  SharedStack<STACK, CLOSEST_SHARED_STACK, BATCH_THREADS> stk(s_stk);
  int sp = 0;
  int next = CHILD_EMPTY;
  float best = 0.f;
  int best_idx = INT_MAX;
  int64_t best_slot = -1;
  V3 best_cp = V3{0.f, 0.f, 0.f};
  int pops = 0;
  while (true) {
    __syncwarp();
    while (oldest < taken && s_left[warp][oldest % CP_STREAM_RING] == 0) {
      int sl = (int)(oldest % CP_STREAM_RING);
      long long base = s_base[warp][sl];
      int cnt = s_cnt[warp][sl];
      for (int j = lane; j < cnt; j += 32) {
        a.out_index[base + j] = s_i[warp][sl][j];
        if (a.out_dist) a.out_dist[base + j] = s_d[warp][sl][j];
      }
      if (a.out_cp)
        for (int j = lane; j < 3 * cnt; j += 32) a.out_cp[3 * base + j] = s_c[warp][sl][j];
      ++oldest;
    }
    __syncwarp();
    unsigned idle = __ballot_sync(FULL, q < 0);
    if ((__popc(idle) >= CLOSEST_REFILL_AT || idle == FULL) && !exhausted) {
      if (qb >= qe && taken - oldest < CP_STREAM_RING) {
        unsigned long long b = 0;
        if (lane == 0) b = atomicAdd(counter, (unsigned long long)REFILL_BLOCK);
        b = __shfl_sync(FULL, b, 0);
        if ((int64_t)b >= nq) {
          exhausted = true;
        } else {
          qb = (int64_t)b;
          qe = qb + REFILL_BLOCK < nq ? qb + REFILL_BLOCK : nq;
          int cnt = (int)(qe - qb);
          for (int k = lane; k < 3 * cnt; k += 32) in[k] = a.queries[3 * qb + k];
          int sl = (int)(taken % CP_STREAM_RING);
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
          slot = (int)((taken - 1) % CP_STREAM_RING);
          qbase = s_base[warp][slot];
          float const * r = in + (q - qbase) * 3;
          p = V3{r[0], r[1], r[2]};
          best = a.thresh;
          best_idx = INT_MAX;
          best_slot = -1;
          sp = 0;
          next = root;
          pops = 0;
        }
        qb += take < avail ? take : avail;
      }
    }
    bool busy = __ballot_sync(FULL, q >= 0) != 0;
    if (!busy && oldest == taken && (exhausted || qb >= qe)) {
      if (exhausted) break;
      continue;
    }
    if (q < 0) continue;
    if (next == CHILD_EMPTY && sp == 0) {
      bool found = best_idx != INT_MAX;
      int j = (int)(q - qbase);
      s_i[warp][slot][j] = found ? best_idx : -1;
      s_d[warp][slot][j] = found ? sqrtf(best) : -1.f;
      s_c[warp][slot][3 * j] = found ? best_cp.x : 0.f;
      s_c[warp][slot][3 * j + 1] = found ? best_cp.y : 0.f;
      s_c[warp][slot][3 * j + 2] = found ? best_cp.z : 0.f;
      atomicSub(&s_left[warp][slot], 1);
      q = -1;
      continue;
    }
    if (budget > 0 && ++pops > budget) {
      // over budget: queued with its best element; the warp-per-query kernel writes its result in place later
      unsigned long long pos = atomicAdd(hq.count, 1ull);
      hq.q[pos] = q;
      hq.bound[pos] = best;
      hq.idx[pos] = best_idx;
      hq.slot[pos] = best_slot;
      atomicSub(&s_left[warp][slot], 1);
      q = -1;
      continue;
    }
    int code = next;
    if (code == CHILD_EMPTY) {
      --sp;
      int2 top = stk.get(sp);
      code = top.x;
      if (__int_as_float(top.y) > best * PRUNE_SLACK) continue;
    }
    closest_step<W>(nodes, f.cp_rec, 0, code, p, best, best_idx, best_slot, best_cp, stk, sp, next, f.err, nullptr,
                    0.f);
    pops -= leaf_rest(code, next);
  }
}

// First hit at width 8 for the batched kernel: the search of ray_query with node and leaf read where they are used, and the
// node through 16-byte loads: 61 registers and eight resident blocks instead of 80 and six. 2,097,152 rays over 16 meshes of
// 20,480 triangles: 1.06 ms, through ray_query 1.49.
template <int STACK>
__device__ __forceinline__ RayOut ray_query_w8(WideNode<8> const * __restrict__ nodes, float4 const * __restrict__ rec,
                                               int root, int64_t elem_base, V3 o, V3 d, float max_time, unsigned * err) {
  RayState ray;
  ray_setup(ray, o, d);
  RayOut out;
  out.t = max_time >= 0.f ? max_time : INFINITY;
  out.idx = INT_MAX;
  out.slot = -1;
  LocalStack<STACK> stk;
  int sp = 0;
  int next = root;
  while (next != CHILD_EMPTY || sp > 0) {
    int code = next;
    if (code == CHILD_EMPTY) {
      --sp;
      int2 top = stk.get(sp);
      code = top.x;
      if (__int_as_float(top.y) > out.t * PRUNE_SLACK) continue;
    }
    next = CHILD_EMPTY;
    if (code >= 0) {
      NodeRegs<8> nd;
      load_node_16(nodes, code, nd);
      float lb[8];
      ray_child_bounds<8>(nd, ray, lb);
      push_children_next<8, LocalStack<STACK>, false>(nd, lb, out.t * PRUNE_SLACK, stk, sp, next, err);
    } else {
      int first, count;
      decode_leaf(code, first, count);
      for (int64_t k = elem_base + first; k < elem_base + first + count; ++k) {
        float4 const * r = rec + k * RAY_REC_F4;
        float4 a = __ldg(r), b = __ldg(r + 1), c = __ldg(r + 2);
        float t = ray_triangle_time(o, d, xyz(a), xyz(b), xyz(c));
        int idx = __float_as_int(a.w);
        if (t >= 0.f && t <= out.t && (t < out.t || idx < out.idx)) {
          out.t = t;
          out.idx = idx;
          out.slot = k;
        }
      }
    }
  }
  return out;
}

template <int W, int STACK>
__global__ void __launch_bounds__(BATCH_THREADS)
batch_ray_kernel(BatchForest f, float const * __restrict__ origins, float const * __restrict__ dirs,
                 int64_t const * __restrict__ qoff, int64_t nq, float max_time, float * __restrict__ out_time,
                 int32_t * __restrict__ out_index, unsigned long long * counter, int chunk) {
  WideNode<W> const * nodes = (WideNode<W> const *)f.nodes;
  int64_t base;
  while (next_chunk(counter, chunk, nq, base)) {
    int64_t end = base + chunk < nq ? base + chunk : nq;
    for (int64_t q = base + (threadIdx.x & 31); q < end; q += 32) {
      int m = mesh_of_query(qoff, f.M, q);
      RayOut r;
      if constexpr (W == 8)
        r = ray_query_w8<STACK>(nodes, f.ray_rec, __ldg(f.seg_root + m), __ldg(f.seg_start + m), load_v3(origins + 3 * q),
                                load_v3(dirs + 3 * q), max_time, f.err);
      else
        r = ray_query<W, STACK, false>(nodes, f.ray_rec, __ldg(f.seg_root + m), __ldg(f.seg_start + m),
                                       load_v3(origins + 3 * q), load_v3(dirs + 3 * q), max_time, f.err);
      bool found = r.idx != INT_MAX;
      out_time[q] = found ? r.t : -1.f;
      if (out_index) out_index[q] = found ? r.idx : -1;
    }
  }
}

// SORTED: the K best in a sorted list in shared memory (knn_search_shared), for batches that fill the GPU (see
// knn_sorted_lists). Its insertions shift K / 2 entries, but it needs 50 registers at K = 32 where the unsorted list and its
// final sort need 88, so seven blocks of 128 threads are resident instead of five.
template <int W, int K, int STACK, bool SORTED>
__global__ void __launch_bounds__(BATCH_THREADS, SORTED ? (K == 32 ? 1 : 8) : knn_point_min_blocks<K>())
batch_knn_kernel(BatchForest f, float const * __restrict__ queries, int64_t const * __restrict__ qoff, int64_t nq,
                 int k_out, float thresh, int32_t * __restrict__ out_index, float * __restrict__ out_d2,
                 unsigned long long * counter, int chunk) {
  WideNode<W> const * nodes = (WideNode<W> const *)f.nodes;
  int64_t base;
  while (next_chunk(counter, chunk, nq, base)) {
    int64_t end = base + chunk < nq ? base + chunk : nq;
    for (int64_t q = base + (threadIdx.x & 31); q < end; q += 32) {
      int m = mesh_of_query(qoff, f.M, q);
      V3 p = load_v3(queries + 3 * q);
      int root = __ldg(f.seg_root + m);
      int64_t ebase = __ldg(f.seg_start + m);
      if constexpr (SORTED) {
        __shared__ float s_d[K][BATCH_THREADS];
        __shared__ int s_i[K][BATCH_THREADS];
        int t = threadIdx.x;
#pragma unroll
        for (int j = 0; j < K; ++j) {
          s_d[j][t] = thresh;
          s_i[j][t] = INT_MAX;
        }
        float kth = thresh;
        int kth_i = INT_MAX;
        knn_search_shared<W, K, STACK, BATCH_THREADS, W == 8>(nodes, root, ebase, p, -1, s_d, s_i, kth, kth_i, f.err,
                                                              [&](int64_t k, int & idx, float & d2) {
                                                                float4 a = __ldg(f.pt_rec + k);
                                                                idx = __float_as_int(a.w);
                                                                d2 = squared_norm(xyz(a) - p);
                                                                return true;
                                                              });
        // the row from shared memory
        for (int j = 0; j < k_out; ++j) {
          int i = s_i[j][t];
          out_index[q * k_out + j] = i != INT_MAX ? i : -1;
          out_d2[q * k_out + j] = i != INT_MAX ? s_d[j][t] : -1.f;
        }
      } else {
        int pad = K - k_out;
        float start = thresh + 0.0f;  // (no negative zero)
        bool any = start >= 0.f;      // a negative threshold admits nothing
        uint64_t none = knn_key(any ? start : 0.f, INT_MAX);
        auto entry = [&](int j) { return j < pad ? (uint64_t)0 : none; };
        uint64_t keys[K];
        // lists in shared memory as in knn_kernel (width 4, K = 8, 200,000 queries over 100 sets of 2,000 points: 0.322 ms,
        // in registers 0.237)
        if constexpr (knn_lists_shared<W, K>()) {
          __shared__ uint64_t s_list[K][BATCH_THREADS];
          SharedKnnList<K, BATCH_THREADS> list(s_list);
          list.init(entry);
          if (any) knn_points_search<W, STACK>(nodes, f.pt_rec, root, ebase, p, -1, 0, 0, list, f.err);
          list.finish(keys);
        } else {
          RegisterKnnList<K> list;
          list.init(entry);
          if (any) knn_points_search<W, STACK>(nodes, f.pt_rec, root, ebase, p, -1, 0, 0, list, f.err);
          list.finish(keys);
        }
        write_knn_keys<K>(out_index, out_d2, q, k_out, keys);
      }
    }
  }
}

int persistent_grid(void const * kernel) {
  int sms = sm_count();
  int per_sm = 0;
  THEA_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, BATCH_THREADS, 0));
  return std::max(1, per_sm) * sms;
}

// Blocks of query indices a warp takes at a time: the caller's `chunk`, but no larger than a warp's share, so that a small
// batch keeps every warp busy
int refill_block(int64_t nq, int grid, int chunk) {
  int64_t per = ceil_div(nq, (int64_t)grid * (BATCH_THREADS / 32));
  return (int)std::min<int64_t>(chunk, std::max<int64_t>(1, per));
}

// Queries of a mixed-precision batch that are collected and resolved at a time: the candidates and the queue of unfinished
// queries take 56 bytes each, 5 GB for the 90.2 million of 4,096 meshes at once, 0.94 GB in slices. Each slice ends with its
// own longest queries: 348.7 ms at 4,194,304 queries a slice, 328.1 at 16,777,216, 321.6 in one (without a step budget).
constexpr int64_t F64_SLICE = int64_t(1) << 24;

__global__ void slice_counters_kernel(unsigned long long * counters, int64_t q0) {
  counters[0] = (unsigned long long)q0;  // next query
  counters[1] = 0;                       // next queued query
  counters[2] = 0;                       // queued queries
}

// Scratch of one closest-point batch, in one allocation: the counters (zeroed on the stream), the queue of `queue` unfinished
// queries and the band candidates of `cand` queries. (Six allocations and a kernel that wrote one BVH's query range, which
// nothing reads, cost a small call 8 us of host time.)
struct ClosestScratch {
  Scratch all;
  unsigned long long * counters;  // next query, next queued query, queued queries
  HardQueue hq;
  int32_t * cand;
  ClosestScratch(int64_t queue, int64_t cands, cudaStream_t s)
      : all((size_t)(64 + queue * (int64_t)(2 * sizeof(int64_t) + sizeof(float) + sizeof(int32_t)) +
                     cands * (int64_t)(F64_CAND * sizeof(int32_t))), s) {
    char * p = all.as<char>();
    counters = reinterpret_cast<unsigned long long *>(p);
    cand = reinterpret_cast<int32_t *>(p + 64);
    p += 64 + cands * (int64_t)(F64_CAND * sizeof(int32_t));
    hq.q = reinterpret_cast<int64_t *>(p);
    hq.slot = hq.q + queue;
    hq.bound = reinterpret_cast<float *>(hq.slot + queue);
    hq.idx = reinterpret_cast<int32_t *>(hq.bound + queue);
    hq.count = counters + 2;
    THEA_CUDA_CHECK(cudaMemsetAsync(counters, 0, 3 * sizeof(unsigned long long), s));
  }
};

template <int W, int STACK>
void launch_batch_closest(BatchForest const & f, ClosestArgs const & a, int64_t nq, int prec, int budget, int chunk,
                          ClosestScratch const & w, cudaStream_t s) {
  unsigned long long * counters = w.counters;
  HardQueue const & hq = w.hq;
  int first_budget = budget > 0 ? budget : 0;
  if (prec == THEA_PRECISION_FP64_RECHECK) {
    // slice by slice, each from its first query on in the arrays of the whole batch
    auto k1 = closest_collect_kernel<W, STACK>;
    auto k2 = batch_closest_phase2_kernel<W, THEA_PRECISION_FP64_RECHECK>;
    int grid = persistent_grid((void const *)k1), grid2 = persistent_grid((void const *)k2);
    for (int64_t q0 = 0; q0 < nq; q0 += F64_SLICE) {
      int64_t end = std::min(nq, q0 + F64_SLICE);
      // (its entries are found at 8 q: as if the array began with query 0's)
      int32_t * c = reinterpret_cast<int32_t *>(reinterpret_cast<uintptr_t>(w.cand) -
                                                (uintptr_t)q0 * (F64_CAND * sizeof(int32_t)));
      if (q0 > 0) THEA_LAUNCH(slice_counters_kernel, 1, 1, 0, s, counters, q0);
      THEA_LAUNCH_NAMED("batch_closest_kernel_fp64", k1, grid, BATCH_THREADS, 0, s, f, a, end, counters, first_budget, hq,
                        refill_block(end - q0, grid, chunk), c);
      THEA_LAUNCH_NAMED("closest_resolve_kernel", closest_resolve_kernel, (unsigned)ceil_div(end - q0, BATCH_THREADS),
                        BATCH_THREADS, 0, s, f, a, q0, end, c);
      THEA_LAUNCH_NAMED("batch_closest_phase2_kernel", k2, grid2, BATCH_THREADS, 0, s, f, a, hq, counters + 1);
    }
    return;
  }
  char const * name = budget > 0 ? "batch_closest_phase1_kernel" : "batch_closest_kernel_fp32";
  // without error estimates: persistent lanes (1.5x on the 256-mesh case), also as the first phase of the two-phase form
  if (!a.out_err) {
    auto kr = batch_closest_refill_kernel<W, STACK>;
    int grid = persistent_grid((void const *)kr);
    THEA_LAUNCH_NAMED(name, kr, grid, BATCH_THREADS, 0, s, f, a, nq, counters, first_budget, hq,
                      refill_block(nq, grid, chunk));
  } else {
    auto k1 = batch_closest_kernel<W, STACK>;
    THEA_LAUNCH_NAMED(name, k1, persistent_grid((void const *)k1), BATCH_THREADS, 0, s, f, a, nq, counters, chunk,
                      first_budget, hq);
  }
  if (budget <= 0) return;
  auto k2 = batch_closest_phase2_kernel<W, THEA_PRECISION_FP32_REFERENCE>;
  THEA_LAUNCH_NAMED("batch_closest_phase2_kernel", k2, persistent_grid((void const *)k2), BATCH_THREADS, 0, s, f, a, hq,
                    counters + 1);
}

template <int W, int STACK>
void launch_batch_ray(BatchForest const & f, float const * o, float const * d, int64_t const * qoff, int64_t nq,
                      float max_time, float * t, int32_t * idx, unsigned long long * counter, int chunk,
                      cudaStream_t s) {
  auto k = batch_ray_kernel<W, STACK>;
  THEA_LAUNCH_NAMED("batch_ray_kernel", k, persistent_grid((void const *)k), BATCH_THREADS, 0, s, f, o, d, qoff, nq, max_time, t, idx, counter,
              chunk);
}

// Batches that keep the sorted lists: K = 32 (17 neighbours and more) from 98,304 queries on, and K = 16 at width 8, where the
// unsorted list shares the registers with 256-byte nodes, from 524,288. Call times in ms, sorted and unsorted, over 100 sets of
// 1,000 points, 32 nearest, width 4: 300,000 queries 1.62 / 2.05, 1,000,000 4.01 / 5.54; width 8: 1.79 / 2.20, 4.63 / 6.86; 16
// nearest, width 8: 1,000,000 2.17 / 2.34. (50,000 queries, 32 nearest: 0.94 / 0.73.)
template <int W, int K> bool knn_sorted_lists(int64_t nq) {
  if (K == 32) return nq >= 98304;
  return W == 8 && K == 16 && nq >= 524288;
}

template <int W, int K, int STACK>
void launch_batch_knn_k(BatchForest const & f, float const * q, int64_t const * qoff, int64_t nq, int k, float thresh,
                        int32_t * idx, float * d2, unsigned long long * counter, int chunk, cudaStream_t s) {
  auto kern = batch_knn_kernel<W, K, STACK, false>;
  if constexpr (K == 32 || (W == 8 && K == 16)) {
    if (knn_sorted_lists<W, K>(nq)) kern = batch_knn_kernel<W, K, STACK, true>;
  }
  THEA_LAUNCH_NAMED("batch_knn_kernel", kern, persistent_grid((void const *)kern), BATCH_THREADS, 0, s, f, q, qoff, nq, k,
                    thresh, idx, d2, counter, chunk);
}

template <int W, int STACK>
void launch_batch_knn(BatchForest const & f, float const * q, int64_t const * qoff, int64_t nq, int k, float thresh,
                      int32_t * idx, float * d2, unsigned long long * counter, int chunk, cudaStream_t s) {
  if (k <= 1) launch_batch_knn_k<W, 1, STACK>(f, q, qoff, nq, k, thresh, idx, d2, counter, chunk, s);
  else if (k <= 2) launch_batch_knn_k<W, 2, STACK>(f, q, qoff, nq, k, thresh, idx, d2, counter, chunk, s);
  else if (k <= 4) launch_batch_knn_k<W, 4, STACK>(f, q, qoff, nq, k, thresh, idx, d2, counter, chunk, s);
  else if (k <= 8) launch_batch_knn_k<W, 8, STACK>(f, q, qoff, nq, k, thresh, idx, d2, counter, chunk, s);
  else if (k <= 16) launch_batch_knn_k<W, 16, STACK>(f, q, qoff, nq, k, thresh, idx, d2, counter, chunk, s);
  else launch_batch_knn_k<W, 32, STACK>(f, q, qoff, nq, k, thresh, idx, d2, counter, chunk, s);
}

}  // namespace

BatchForest forest_view(thea_bvh const * b) {
  BatchForest f;
  f.nodes = b->nodes;
  f.cp_rec = b->cp_rec;
  f.ray_rec = b->ray_rec;
  f.pt_rec = b->pt_rec;
  f.slabs = b->slabs;
  f.seg_start = b->seg_start;
  f.seg_root = b->seg_root;
  f.M = b->num_segments;
  f.err = b->err;
  return f;
}

namespace {

// One batched closest-point search of `a` (queries, offsets, outputs) over the forest
void batch_closest_core(thea_bvh const * b, ClosestArgs const & a, int64_t nq, ClosestParams const & cp, int chunk,
                        cudaStream_t s) {
  BatchForest f = forest_view(b);
  bool sm = small_stack_ok(b);
  int budget = cp.budget > 0 ? cp.budget : 0;
  // (the mixed-precision search may hand over queries at any budget, a slice of the batch at a time)
  bool f64 = cp.precision == THEA_PRECISION_FP64_RECHECK;
  int64_t slice = std::min(nq, F64_SLICE);
  ClosestScratch w(f64 ? slice : (budget > 0 ? nq : 0), f64 ? slice : 0, s);
  if (b->width == 4) sm ? launch_batch_closest<4, 64>(f, a, nq, cp.precision, budget, chunk, w, s)
                        : launch_batch_closest<4, 256>(f, a, nq, cp.precision, budget, chunk, w, s);
  else sm ? launch_batch_closest<8, 128>(f, a, nq, cp.precision, budget, chunk, w, s)
          : launch_batch_closest<8, 512>(f, a, nq, cp.precision, budget, chunk, w, s);
}

}  // namespace

void run_batch_closest(thea_bvh const * b, float const * q, int64_t const * qoff, int64_t nq, ClosestParams const & cp,
                       int chunk, int32_t * idx, float * dist, float * cpt, float * err, cudaStream_t s) {
  if (nq <= 0) return;
  ClosestArgs a{q, qoff, cp.thresh, cp.bound2, cp.scene_scale, idx, dist, cpt, err, cp.seg_cut};
  batch_closest_core(b, a, nq, cp, chunk, s);
}

template <int W, int TEAM>
void launch_closest_team(BatchForest const & f, ClosestArgs const & a, int64_t nq, cudaStream_t s) {
  unsigned grid = (unsigned)ceil_div(nq, BATCH_THREADS / TEAM);
  THEA_LAUNCH((closest_team_kernel<W, TEAM>), grid, BATCH_THREADS, 0, s, f, a, nq);
}

void run_closest_teams(thea_bvh const * b, float const * q, int64_t nq, ClosestParams const & cp, int32_t * idx,
                       float * dist, float * cpt, cudaStream_t s) {
  if (nq <= 0) return;
  BatchForest f = forest_view(b);
  ClosestArgs a{q, nullptr, cp.thresh, cp.bound2, cp.scene_scale, idx, dist, cpt, nullptr};
  bool whole = nq < CLOSEST_WHOLE_WARP_MAX;
  if (b->width == 4) whole ? launch_closest_team<4, 32>(f, a, nq, s) : launch_closest_team<4, 16>(f, a, nq, s);
  else whole ? launch_closest_team<8, 32>(f, a, nq, s) : launch_closest_team<8, 16>(f, a, nq, s);
}

void run_closest_warps_f64(thea_bvh const * b, float const * q, int64_t nq, ClosestParams const & cp, int32_t * idx,
                           float * dist, float * cpt, float * err, cudaStream_t s) {
  if (nq <= 0) return;
  BatchForest f = forest_view(b);
  ClosestArgs a{q, nullptr, cp.thresh, cp.bound2, cp.scene_scale, idx, dist, cpt, err};
  unsigned grid = (unsigned)ceil_div(nq, PHASE2_WARPS);
  if (b->width == 4) THEA_LAUNCH(closest_warp_f64_kernel<4>, grid, BATCH_THREADS, 0, s, f, a, nq);
  else THEA_LAUNCH(closest_warp_f64_kernel<8>, grid, BATCH_THREADS, 0, s, f, a, nq);
}

template <int W, int STACK>
void launch_closest_stream(BatchForest const & f, ClosestArgs const & a, int64_t nq, int budget,
                           unsigned long long * counters, HardQueue const & hq, cudaStream_t s) {
  auto k1 = closest_stream_kernel<W, STACK>;
  int64_t need = ceil_div(ceil_div(nq, REFILL_BLOCK) * 32, BATCH_THREADS);
  unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(persistent_grid((void const *)k1), need));
  THEA_LAUNCH_NAMED("closest_stream_kernel", k1, grid, BATCH_THREADS, 0, s, f, a, nq, counters, budget, hq);
  auto k2 = batch_closest_phase2_kernel<W, THEA_PRECISION_FP32_REFERENCE>;
  THEA_LAUNCH_NAMED("batch_closest_phase2_kernel", k2, persistent_grid((void const *)k2), BATCH_THREADS, 0, s, f, a, hq,
                    counters + 1);
}

void run_closest_stream(thea_bvh const * b, float const * q, int64_t nq, ClosestParams const & cp, int32_t * idx,
                        float * dist, float * cpt, cudaStream_t s) {
  if (nq <= 0) return;
  THEA_REQUIRE(b->num_segments == 1, "closest_stream: one BVH only");
  BatchForest f = forest_view(b);
  bool sm = small_stack_ok(b);
  ClosestArgs a{q, nullptr, cp.thresh, cp.bound2, cp.scene_scale, idx, dist, cpt, nullptr};
  int budget = cp.budget > 0 ? cp.budget : 0;
  ClosestScratch w(budget > 0 ? nq : 1, 0, s);
  if (b->width == 4) sm ? launch_closest_stream<4, 64>(f, a, nq, budget, w.counters, w.hq, s)
                        : launch_closest_stream<4, 256>(f, a, nq, budget, w.counters, w.hq, s);
  else sm ? launch_closest_stream<8, 128>(f, a, nq, budget, w.counters, w.hq, s)
          : launch_closest_stream<8, 512>(f, a, nq, budget, w.counters, w.hq, s);
}

void run_batch_ray(thea_bvh const * b, float const * o, float const * d, int64_t const * qoff, int64_t nq,
                   float max_time, int chunk, float * t, int32_t * idx, cudaStream_t s) {
  if (nq <= 0) return;
  BatchForest f = forest_view(b);
  Scratch counter(sizeof(unsigned long long), s);
  THEA_CUDA_CHECK(cudaMemsetAsync(counter.ptr, 0, sizeof(unsigned long long), s));
  auto * c = counter.as<unsigned long long>();
  bool sm = small_stack_ok(b);
  if (b->width == 4) sm ? launch_batch_ray<4, 64>(f, o, d, qoff, nq, max_time, t, idx, c, chunk, s)
                        : launch_batch_ray<4, 256>(f, o, d, qoff, nq, max_time, t, idx, c, chunk, s);
  else sm ? launch_batch_ray<8, 128>(f, o, d, qoff, nq, max_time, t, idx, c, chunk, s)
          : launch_batch_ray<8, 512>(f, o, d, qoff, nq, max_time, t, idx, c, chunk, s);
}

void run_batch_knn(thea_bvh const * b, float const * q, int64_t const * qoff, int64_t nq, int k, float thresh,
                   int chunk, int32_t * idx, float * d2, cudaStream_t s) {
  if (nq <= 0) return;
  BatchForest f = forest_view(b);
  Scratch counter(sizeof(unsigned long long), s);
  THEA_CUDA_CHECK(cudaMemsetAsync(counter.ptr, 0, sizeof(unsigned long long), s));
  auto * c = counter.as<unsigned long long>();
  bool sm = small_stack_ok(b);
  if (b->width == 4) sm ? launch_batch_knn<4, 64>(f, q, qoff, nq, k, thresh, idx, d2, c, chunk, s)
                        : launch_batch_knn<4, 256>(f, q, qoff, nq, k, thresh, idx, d2, c, chunk, s);
  else sm ? launch_batch_knn<8, 128>(f, q, qoff, nq, k, thresh, idx, d2, c, chunk, s)
          : launch_batch_knn<8, 512>(f, q, qoff, nq, k, thresh, idx, d2, c, chunk, s);
}

}  // namespace thea
