// Which kernels answer a closest-point call, by precision, tree and batch size.
#include "fake_cuda.hpp"

#include "../../thea_gb300/csrc/common.cuh"
#include "../../thea_gb300/csrc/batch.hpp"
#include "../../thea_gb300/csrc/bvh.hpp"
#include "../../thea_gb300/csrc/query.hpp"

using namespace thea;

static bool check(int width, int leaf, int64_t triangles, int64_t n, int precision, char const * kernel) {
  thea_bvh b;
  b.is_mesh = 1;
  b.n = triangles;
  b.depth = 9;
  b.width = width;
  b.leaf_size = leaf;
  fake::State & s = fake::state();
  s.launches.clear();
  ClosestParams cp;
  cp.precision = precision;
  std::vector<float> q(3);
  int32_t idx;
  unsigned err = 0;
  run_closest(&b, q.data(), n, cp, &idx, nullptr, nullptr, nullptr, &err, nullptr);
  s.queue.clear();  // (its memory is only named, never reached)
  if (fake::launches_of(kernel) > 0) return true;
  std::printf("width %d, leaves of %d, %lld triangles, %lld queries, precision %d: not %s but\n", width, leaf,
              (long long)triangles, (long long)n, precision, kernel);
  for (auto const & l : s.launches) std::printf("  %s\n", l.c_str());
  return false;
}

int main() {
  int const f32 = THEA_PRECISION_FP32_REFERENCE, f64 = THEA_PRECISION_FP64_RECHECK;
  char const *warps = "closest_warp_f64_kernel", *collect = "closest_collect_kernel", *threads = "14closest_kernel",
             *teams = "closest_team_kernel", *lanes = "batch_closest_refill_kernel";
  bool ok = true;
  for (int width : {4, 8})
    for (int leaf : {1, 2, 4, 8, 16}) {
      ok = check(width, leaf, 81920, 3071, f64, warps) && ok;
      ok = check(width, leaf, 1280, 100000, f64, threads) && ok;
      ok = check(width, leaf, 81920, 262144, f64, threads) && ok;
      ok = check(width, leaf, 81920, 3072, f64, width == 8 && leaf >= 8 ? threads : collect) && ok;
    }
  // the ends of the collected form
  ok = check(4, 2, 81920, 163839, f64, collect) && check(4, 2, 81920, 163840, f64, threads) && ok;
  ok = check(4, 4, 20480, 65535, f64, collect) && check(4, 4, 20480, 65536, f64, threads) && ok;
  ok = check(8, 2, 20480, 131071, f64, collect) && check(8, 2, 20480, 131072, f64, threads) && ok;
  ok = check(8, 4, 20480, 32767, f64, collect) && check(8, 4, 20480, 32768, f64, threads) && ok;
  // and of the teams
  ok = check(4, 1, 81920, 57343, f32, teams) && check(4, 1, 81920, 57344, f32, threads) && ok;
  ok = check(8, 4, 81920, 16383, f32, teams) && check(8, 4, 81920, 16384, f32, lanes) && ok;
  // default step budgets of batches: width, leaf size, queries, budget
  int64_t const budgets[][4] = {{4, 2, 98303, 32},   {4, 2, 98304, 128},  {4, 2, 262143, 128}, {4, 4, 262144, 256},
                                {4, 8, 786431, 128}, {4, 8, 786432, 256}, {8, 2, 98303, 32},   {8, 2, 98304, 64},
                                {8, 4, 196607, 64},  {8, 4, 196608, 128}, {8, 2, 393215, 128}, {8, 2, 393216, 256},
                                {8, 4, 1 << 24, 128}, {8, 8, 786431, 64}, {8, 8, 786432, 128}};
  for (auto const & c : budgets)
    if (batch_closest_budget(c[2], (int)c[0], (int)c[1]) != c[3]) {
      std::printf("width %d, leaves of %d, %lld queries: budget %d\n", (int)c[0], (int)c[1], (long long)c[2],
                  batch_closest_budget(c[2], (int)c[0], (int)c[1]));
      ok = false;
    }
  if (!ok) return 1;
  std::printf("routes as measured\n");
  return 0;
}
