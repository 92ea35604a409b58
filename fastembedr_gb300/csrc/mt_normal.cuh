// Normal draws of the std::mt19937 stream on the GPU.
#pragma once

#include <cstddef>
#include <cstdint>

#include "common.cuh"
#include "normal_stream.cuh"

namespace fe {

// out[i] = scale * draw i of N(0, sd) from a freshly seeded std::mt19937, in the order of
// std::normal_distribution (Marsaglia's polar method; see normal_stream.cuh), for an even count. The words and the
// accepted points are those of the host stream (NormalStream::radius_rounding() must be known); the logarithm is CUDA's
// (within a unit in the last place). *enough is set to 1 when the words sufficed (they do but for one seed in far more than 10^9).
class MtNormalBlock {
 public:
  // max_points > 0: words for no more candidate points than that (a test of the case that they do not suffice)
  MtNormalBlock(std::uint32_t seed, std::size_t count, double sd, double scale, long long max_points = 0);
  ~MtNormalBlock();
  // whether a block of that many draws can be made: its candidate points are numbered by an int
  static bool fits(std::size_t count) { return count / 2 <= (std::size_t)800000000; }
  // Copies the draws to dst on stream s, after them; false when the words did not suffice.
  bool copy_to(double* dst, cudaStream_t s);

 private:
  Stream stream_;
  Arena arena_;
  double* out_ = nullptr;
  int* enough_ = nullptr;
  std::size_t count_;
};

}  // namespace fe
