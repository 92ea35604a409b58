// Spectral start of UMAP on the GPU: the block subspace iteration of the reference's CPU
// initialisation (the start that umap_knn uses on every backend).
#pragma once

#include <future>
#include <memory>
#include <random>
#include <vector>

#include "common.cuh"
#include "mt_normal.cuh"
#include "normal_stream.cuh"

namespace fe {

// The start's random draws for n points in the reference's stream order: the start block (n x B
// normal(0, 1e-4) x 1e4 draws) and, speculatively and on another thread, the jitter that follows it when no
// Gram-Schmidt column needs a redraw (drawn from a copy of the stream state after the block), with that state, for
// redraws. Independent of the graph, so a caller can make them while the GPU builds it. From kSpectralDeviceDraws
// points on the block is drawn on the GPU `device`: the host's engine takes 0.08 us a point, longer than the graph
// from there on (20,000 points: 1.7 ms beside 0.64; on the GPU 0.2), and only has to be through by the end of the
// rounds, for the jitter.
constexpr int kSpectralDeviceDraws = 8192;
struct SpectralTail {
  std::mt19937 rng;  // after the block
  std::vector<double> jitter;
};
struct SpectralDraws {
  int n = 0;
  std::vector<double> block;              // drawn on the host, or
  std::shared_ptr<MtNormalBlock> device;  // on the GPU
  NormalStream normal{0.0, 0.0001};       // continues after the block
  std::shared_future<SpectralTail> tail;
};
SpectralDraws spectral_draws(int n, int seed, int device, bool on_host = false);

// Start layout of the symmetric fuzzy graph (device CSR: n + 1 offsets, neighbours 0-based and
// ascending per row, no self entries, w_ij == w_ji) into out: device, column-major n x 2 doubles.
// spectral_n_iter rounds, seed for the std::mt19937 stream of the reference, init_scale > 0
// rescales every column to that standard deviation (NaN: no rescaling). Synchronises s.
// `pre` (may be null): the draws of spectral_draws(n, seed), made ahead. max_blocks > 0: no more blocks in the rounds
// than that (otherwise one per SM).
void umap_spectral_start(const int* offsets, const int* neighbors, const float* weights, int n, long long nnz,
                         int spectral_n_iter, double init_scale, int seed, double* out, cudaStream_t s,
                         SpectralDraws* pre = nullptr, int max_blocks = 0);

}  // namespace fe
