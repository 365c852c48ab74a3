// Batched closest-point queries fetch their work in blocks of the caller's queries_per_warp, in both precisions, and in smaller
// ones only where a warp's share of the batch is smaller.
#include "fake_cuda.hpp"

#include "../../thea_gb300/csrc/common.cuh"
#include "../../thea_gb300/csrc/bvh.hpp"
#include "../../thea_gb300/csrc/query.hpp"
#include "../../thea_gb300/csrc/batch.hpp"

int main() {
  using namespace thea;
  thea_bvh b;
  b.is_mesh = 1;
  b.n = 100;
  b.depth = 3;
  int block = -1;
  fake::state().on_launch = [&](std::string const & name, void ** args) {
    // (forest, arguments, queries, counters, budget, queue, block, ...)
    if (name.find("batch_closest_refill_kernel") != std::string::npos ||
        name.find("closest_collect_kernel") != std::string::npos)
      block = *(int *)args[6];
  };
  float q[3];
  int64_t off[2] = {0, 0};
  int32_t idx;
  for (int precision : {THEA_PRECISION_FP32_REFERENCE, THEA_PRECISION_FP64_RECHECK})
    for (int budget : {0, 32})
      for (int chunk : {32, 64, 128}) {
        ClosestParams cp;
        cp.precision = precision;
        cp.budget = budget;
        block = -1;
        run_batch_closest(&b, q, off, 4000000, cp, chunk, &idx, nullptr, nullptr, nullptr, nullptr);
        cudaStreamSynchronize(nullptr);
        if (block != chunk) {
          std::printf("precision %d, budget %d: blocks of %d where the caller asked for %d\n", precision, budget, block, chunk);
          return 1;
        }
        run_batch_closest(&b, q, off, 5000, cp, chunk, &idx, nullptr, nullptr, nullptr, nullptr);
        cudaStreamSynchronize(nullptr);
        if (block < 1 || block > 32) {
          std::printf("5,000 queries in blocks of %d\n", block);
          return 1;
        }
      }
  std::printf("fetches as asked\n");
  return 0;
}
