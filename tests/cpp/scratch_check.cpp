// Scratch memory the library asks for: the node arrays of a build are bounded whatever its size, and a batch in the
// mixed-precision mode takes no more than one slice's.
#include "fake_cuda.hpp"

#include "../../thea_gb300/csrc/common.cuh"
#include "../../thea_gb300/csrc/bvh.hpp"
#include "../../thea_gb300/csrc/query.hpp"
#include "../../thea_gb300/csrc/batch.hpp"

using namespace thea;

static size_t build_peak(int64_t n, int width) {
  fake::State & s = fake::state();
  thea_build_config cfg{};
  cfg.width = width;
  cfg.max_leaf_size = 1;
  std::vector<float> p(3);  // (no kernel reads it)
  s.peak = s.now;
  size_t before = s.now;
  thea_bvh * b = build_bvh(false, p.data(), n, nullptr, 0, cfg, nullptr);
  size_t peak = s.peak - before;
  destroy_bvh(b);
  cudaDeviceSynchronize();
  return peak;
}

int main(int argc, char ** argv) {
  if (argc > 1 && std::string(argv[1]) == "build") {
    // what the sort and the binary tree take grows with the size; the node arrays beside them are bounded
    for (int width : {4, 8}) {
      double per = (double)build_peak(8 << 20, width) / (8 << 20);
      for (int64_t n : {300000, 1 << 20, 1 << 21, (1 << 21) + 1, 1 << 22, (1 << 22) + 1}) {
        double nodes = (double)build_peak(n, width) - per * (double)n;
        if (nodes > (double)((int64_t)448 << 20)) {
          std::printf("width %d, %lld elements: %.0f MB of scratch for the nodes\n", width, (long long)n, nodes / (1 << 20));
          return 1;
        }
      }
    }
    std::printf("builds bounded\n");
    return 0;
  }
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
    if (peak > (size_t)1 << 30) {
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
