// What a small closest-point call asks of the runtime: one allocation and its kernels, nothing else to wait for.
#include "fake_cuda.hpp"

#include "../../thea_gb300/csrc/common.cuh"
#include "../../thea_gb300/csrc/bvh.hpp"
#include "../../thea_gb300/csrc/query.hpp"

using namespace thea;

static bool check(thea_bvh const & b, int64_t n, int precision, int allocations, size_t launches) {
  fake::State & s = fake::state();
  s.allocations = 0;
  s.launches.clear();
  ClosestParams cp;
  cp.precision = precision;
  float q[3];
  int32_t idx;
  unsigned err = 0;
  run_closest(&b, q, n, cp, &idx, nullptr, nullptr, nullptr, &err, nullptr);
  cudaStreamSynchronize(nullptr);
  if (s.allocations <= allocations && s.launches.size() <= launches) return true;
  std::printf("%lld queries, precision %d: %d allocations, %zu kernels\n", (long long)n, precision, s.allocations, s.launches.size());
  for (auto const & l : s.launches) std::printf("  %s\n", l.c_str());
  return false;
}

int main() {
  thea_bvh b;
  b.is_mesh = 1;
  b.n = 81920;
  b.depth = 9;
  b.leaf_size = 1;
  bool ok = check(b, 1000, THEA_PRECISION_FP32_REFERENCE, 0, 1);
  ok = check(b, 1000, THEA_PRECISION_FP64_RECHECK, 0, 1) && ok;
  ok = check(b, 5000, THEA_PRECISION_FP64_RECHECK, 1, 3) && ok;     // collect, resolve, finish
  ok = check(b, 100000, THEA_PRECISION_FP32_REFERENCE, 1, 2) && ok;  // persistent lanes, finish
  if (!ok) return 1;
  std::printf("small calls are small\n");
  return 0;
}
