// Kernels and device functions of the library launched alone: on inputs that its entry points reach at sizes too large
// for a test, and over the whole range of an argument.
#include "../fastembedr_gb300/csrc/tsne_exact.cu"
#include "../fastembedr_gb300/csrc/tsne_grid.cu"
#include "../fastembedr_gb300/csrc/umap_spectral.cu"

namespace {
constexpr long long kEntries = 1LL << 31;  // of P: one more than the largest row bound

// Fills the last `tail` of kEntries entries of a fresh device array from host values.
template <typename T>
struct Tail {
  T* d = nullptr;
  Tail(const T* host, long long tail) {
    FE_CUDA(cudaMalloc(&d, sizeof(T) * kEntries));
    FE_CUDA(cudaMemcpy(d + kEntries - tail, host, sizeof(T) * tail, cudaMemcpyHostToDevice));
  }
  ~Tail() { cudaFree(d); }
};
template <typename T>
struct Array {
  T* d = nullptr;
  Array(const T* host, long long count) {
    FE_CUDA(cudaMalloc(&d, sizeof(T) * count));
    FE_CUDA(cudaMemcpy(d, host, sizeof(T) * count, cudaMemcpyHostToDevice));
  }
  ~Array() { cudaFree(d); }
};
}  // namespace

// rows: n bounds into the kEntries entries, whose last `tail` are given; col is relabelled in place.
extern "C" int edge_relabel(const int* rows, int n, int* col, long long tail, const int* delta) {
  return fe::guarded([&] {
    Array<int2> r((const int2*)rows, n);
    Array<int> dl(delta, n);
    Tail<int> c(col, tail);
    fe::relabel_rows_kernel<<<1, 256>>>(c.d, r.d, n, dl.d);
    FE_LAUNCH("relabel_rows_kernel");
    FE_CUDA(cudaMemcpy(col, c.d + kEntries - tail, sizeof(int) * tail, cudaMemcpyDeviceToHost));
  });
}

extern "C" int edge_attractive(const int* rows, int n, const int* col, const float* val, long long tail, const float* y,
                               float* attr) {
  return fe::guarded([&] {
    Array<int2> r((const int2*)rows, n);
    Array<float2> p((const float2*)y, n), out((const float2*)attr, n);
    std::vector<unsigned> zero(2 * fe::kAttrCtrStride, 0u);
    Array<unsigned> ctr(zero.data(), zero.size());
    Tail<int> c(col, tail);
    Tail<float> v(val, tail);
    fe::attractive_kernel<<<1, fe::kAttrThreads>>>(r.d, c.d, v.d, p.d, n, 1.0f, out.d, ctr.d, 1, 1u);
    FE_LAUNCH("attractive_kernel");
    FE_CUDA(cudaMemcpy(attr, out.d, sizeof(float2) * n, cudaMemcpyDeviceToHost));
  });
}

// part[b]: the blocks' sums of p log((p + 1e-9) / (q / z + 1e-9)); bounds: n + 1 row bounds.
extern "C" int edge_kl(const int* bounds, int n, const int* col, const float* val, long long tail, const float* y, double z,
                       double* sum) {
  return fe::guarded([&] {
    Array<int> b(bounds, n + 1);
    Array<float2> p((const float2*)y, n);
    Array<double> dz(&z, 1), out(&z, 1);
    Tail<int> c(col, tail);
    Tail<float> v(val, tail);
    fe::kl_rows_kernel<<<1, 256>>>(b.d, c.d, v.d, p.d, p.d, nullptr, n, dz.d, out.d);
    FE_LAUNCH("kl_rows_kernel");
    FE_CUDA(cudaMemcpy(sum, out.d, sizeof(double), cudaMemcpyDeviceToHost));
  });
}

// w: normalised in place by the degrees; out = W x, n x columns (column-major).
extern "C" int edge_spectral(const int* bounds, int n, const int* col, float* w, long long tail, const float* degree,
                             const double* x, int columns, double* out) {
  return fe::guarded([&] {
    Array<int> b(bounds, n + 1);
    Array<float> dg(degree, n);
    Array<double> dx(x, (long long)n * columns), dy(out, (long long)n * columns);
    Tail<int> c(col, tail);
    Tail<float> v(w, tail), nw(w, tail);
    fe::sp_adjacency_kernel<<<1, fe::kSpThreads>>>(b.d, c.d, v.d, dg.d, n, nw.d);
    FE_LAUNCH("sp_adjacency_kernel");
    fe::sp_multiply_kernel<<<1, fe::kSpThreads>>>(b.d, c.d, nw.d, n, columns, dx.d, dy.d);
    FE_LAUNCH("sp_multiply_kernel");
    FE_CUDA(cudaMemcpy(w, nw.d + kEntries - tail, sizeof(float) * tail, cudaMemcpyDeviceToHost));
    FE_CUDA(cudaMemcpy(out, dy.d, sizeof(double) * n * columns, cudaMemcpyDeviceToHost));
  });
}

namespace {
__global__ void exp_kernel(const float2* x, int n, double* relative) {
  __shared__ float2 table[fe::kExpEntries];
  fe::fill_exp_table(table);
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const fe::Float2Sum v{x[i].x, x[i].y};
    const double want = exp(fe::value(v));
    relative[i] = (fe::value(fe::exp_two(v, table)) - want) / want;
  }
}
__global__ void log_kernel(const float2* x, int n, double* absolute) {
  __shared__ float4 table[fe::kLogEntries];
  fe::fill_log_table(table);
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const fe::Float2Sum v{x[i].x, x[i].y};
    absolute[i] = fe::value(fe::log_two(v, table)) - log(fe::value(v));
  }
}
__global__ void reciprocal_kernel(int exponent, unsigned long long* differ) {
  const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
  const float x = __uint_as_float((unsigned)(127 + exponent) << 23 | m);
  const float got = fe::reciprocal(x), want = __frcp_rn(x);
  if (m < (1u << 23) && !(got == want || (isnan(got) && isnan(want)))) atomicAdd(differ, 1ull);
}
}  // namespace

// error[i]: of exp(x[i]) relative to CUDA's FP64 function, or of log(x[i]) absolute; x: high and low parts.
extern "C" int edge_two_float(int logarithm, const float* x, int n, double* error) {
  return fe::guarded([&] {
    Array<float2> dx((const float2*)x, n);
    Array<double> e(error, n);
    if (logarithm) log_kernel<<<64, 256>>>(dx.d, n, e.d);
    else exp_kernel<<<64, 256>>>(dx.d, n, e.d);
    FE_LAUNCH("two-float function");
    FE_CUDA(cudaMemcpy(error, e.d, sizeof(double) * n, cudaMemcpyDeviceToHost));
  });
}

// How many of the 2^23 floats in [2^exponent, 2^(exponent + 1)) (128: infinity and the NaNs) have a reciprocal other than the correctly rounded one.
extern "C" int edge_reciprocal(int exponent, unsigned long long* differ) {
  return fe::guarded([&] {
    *differ = 0;
    Array<unsigned long long> d(differ, 1);
    reciprocal_kernel<<<(1 << 23) / 256, 256>>>(exponent, d.d);
    FE_LAUNCH("reciprocal_kernel");
    FE_CUDA(cudaMemcpy(differ, d.d, sizeof(*differ), cudaMemcpyDeviceToHost));
  });
}

// Z, the sum of q over all pairs of different points.
extern "C" int edge_z(const float* y, int n, double* z) {
  return fe::guarded([&] {
    const int tiles = (n + fe::kPairTile - 1) / fe::kPairTile, blocks = 256;
    std::vector<double> part(blocks);
    Array<float2> p((const float2*)y, n);
    Array<double> out(part.data(), blocks);
    fe::sum_q_tiles_kernel<<<blocks, 256>>>(p.d, n, tiles, out.d);
    FE_LAUNCH("sum_q_tiles_kernel");
    FE_CUDA(cudaMemcpy(part.data(), out.d, sizeof(double) * blocks, cudaMemcpyDeviceToHost));
    *z = 0.0;
    for (double v : part) *z += v;
  });
}
