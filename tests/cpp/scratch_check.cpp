// Scratch memory the library asks for: a batch in the mixed-precision mode takes no more than one slice's, however large it
// is.
#include "fake_cuda.hpp"

#include "../../thea_gb300/csrc/common.cuh"
#include "../../thea_gb300/csrc/bvh.hpp"
#include "../../thea_gb300/csrc/query.hpp"
#include "../../thea_gb300/csrc/batch.hpp"

using namespace thea;

int main() {
  fake::State & s = fake::state();
  thea_bvh b;
  b.is_mesh = 1;
  b.n = 100;
  b.depth = 3;
  float q[3];
  int64_t off[2] = {0, 0};
  int32_t idx;
  for (int budget : {0, 256}) {
    ClosestParams cp;
    cp.precision = THEA_PRECISION_FP64_RECHECK;
    cp.budget = budget;
    s.peak = s.now;
    size_t before = s.now;
    run_batch_closest(&b, q, off, 90200000, cp, 64, &idx, nullptr, nullptr, nullptr, nullptr);
    size_t peak = s.peak - before;
    cudaStreamSynchronize(nullptr);
    if (peak > (size_t)300 << 20) {
      std::printf("90.2 million queries, budget %d: %zu bytes of scratch\n", budget, peak);
      return 1;
    }
    if (s.now != before) {
      std::printf("scratch kept\n");
      return 1;
    }
  }
  std::printf("batches bounded\n");
  return 0;
}
