// The grid search of UMAP's curve fit (find_ab_params, src/fast_knn_umap.cpp:437-497) on the GPU.
#pragma once

#include "common.cuh"

namespace fe {

constexpr int kCurvePoints = 300;
constexpr int kCurveLogA = 41, kCurveB = 36;  // log a = -4 .. 4 by 0.2, b = 0.25 .. 2 by 0.05
constexpr int kCurveGrid = kCurveLogA * kCurveB;

// loss[ia * kCurveB + ib] = sum over the points of (1 / (1 + a x^(2b)) - y)^2, to FP64 rounding.
void curve_grid_losses(double spread, double min_dist, double* loss, cudaStream_t s);

}  // namespace fe
