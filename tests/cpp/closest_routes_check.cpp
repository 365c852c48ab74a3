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
  // default step budgets of batches
  int64_t const at[] = {1, 98303, 98304, 786431, 786432, 16777216};
  int const w4[] = {32, 32, 128, 128, 256, 256}, w8[] = {32, 32, 64, 64, 128, 128};
  for (int i = 0; i < 6; ++i)
    if (batch_closest_budget(at[i], 4) != w4[i] || batch_closest_budget(at[i], 8) != w8[i]) {
      std::printf("%lld queries: budgets %d and %d\n", (long long)at[i], batch_closest_budget(at[i], 4),
                  batch_closest_budget(at[i], 8));
      ok = false;
    }
  if (!ok) return 1;
  std::printf("routes as measured\n");
  return 0;
}
