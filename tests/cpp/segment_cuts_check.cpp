// The per-segment root cuts of a forest reach the device whole, however late the runtime reads the array they are copied
// from: init_segment_roots on the fake runtime, whose copies take place at the stream's next synchronisation.
#include "fake_cuda.hpp"

#include "../../thea_gb300/csrc/common.cuh"
#include "../../thea_gb300/csrc/bvh.hpp"
#include "../../thea_gb300/csrc/query.hpp"

int main() {
  using namespace thea;
  for (int M : {1, 3, 1000, 40000}) {
    thea_bvh * b = new thea_bvh;
    b->num_segments = M;
    b->seg_lo.resize(3 * (size_t)M);
    b->seg_hi.resize(3 * (size_t)M);
    for (size_t i = 0; i < 3 * (size_t)M; ++i) {
      b->seg_lo[i] = -(float)(i % 7) - 1.f;
      b->seg_hi[i] = (float)(i % 5) + 1.f;
    }
    init_segment_roots(b, nullptr);
    // what a program's next allocations do to memory that has been given back
    std::vector<std::vector<unsigned char>> other;
    for (int k = 0; k < 8; ++k) other.emplace_back((size_t)M * sizeof(RootCut), (unsigned char)0xa5);
    cudaStreamSynchronize(nullptr);
    for (int s = 0; s < M; ++s) {
      RootCut want = root_cut_of(&b->seg_lo[3 * (size_t)s], &b->seg_hi[3 * (size_t)s], nullptr);
      if (std::memcmp(&want, &b->seg_roots[s], sizeof(want)) != 0) {
        std::printf("segment %d of %d: the cut on the device is not the one computed\n", s, M);
        return 1;
      }
    }
    destroy_bvh(b);
  }
  std::printf("segment cuts whole\n");
  return 0;
}
