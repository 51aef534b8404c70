// The two-float conversions and operations of the kernels, on arrays: reads n
// doubles a and b and n floats f from stdin, writes one record per element.
#include <cstdio>
#include <vector>

#include "../rdc-xpbd-taichi_gb300/csrc/xpbd_device.cuh"

using namespace xpbd;

struct Out {
  float2 split;                   // ff_split(a)
  double sum, prod, quot, wide;   // of ff_split(a) and ff_split(b); widen(f)
  float narrow;                   // narrow(a)
  int less;                       // ff_less(ff_split(a), ff_split(b))
};

__global__ void k_ops(const double* a, const double* b, const float* f, Out* out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float2 x = ff_split(a[i]), y = ff_split(b[i]);
  Out o;
  o.split = x;
  o.sum = ff_double(ff_add(x, y));
  o.prod = ff_double(ff_mul(x, y));
  o.quot = ff_double(ff_div(1.f, y));
  o.wide = widen(f[i]);
  o.narrow = narrow(a[i]);
  o.less = ff_less(x, y);
  out[i] = o;
}

#define CHECK(e) do { if ((e) != cudaSuccess) { std::fprintf(stderr, "%s\n", cudaGetErrorString(cudaGetLastError())); return 1; } } while (0)

int main() {
  int n = 0;
  if (std::fread(&n, sizeof(n), 1, stdin) != 1 || n <= 0 || n > (1 << 20)) return 2;
  std::vector<double> a(n), b(n);
  std::vector<float> f(n);
  std::vector<Out> out(n);
  if (std::fread(a.data(), 8, n, stdin) != (size_t)n || std::fread(b.data(), 8, n, stdin) != (size_t)n ||
      std::fread(f.data(), 4, n, stdin) != (size_t)n)
    return 2;
  double *da = nullptr, *db = nullptr;
  float* df = nullptr;
  Out* dout = nullptr;
  CHECK(cudaMalloc(&da, 8 * (size_t)n));
  CHECK(cudaMalloc(&db, 8 * (size_t)n));
  CHECK(cudaMalloc(&df, 4 * (size_t)n));
  CHECK(cudaMalloc(&dout, sizeof(Out) * (size_t)n));
  CHECK(cudaMemcpy(da, a.data(), 8 * (size_t)n, cudaMemcpyHostToDevice));
  CHECK(cudaMemcpy(db, b.data(), 8 * (size_t)n, cudaMemcpyHostToDevice));
  CHECK(cudaMemcpy(df, f.data(), 4 * (size_t)n, cudaMemcpyHostToDevice));
  k_ops<<<(n + 255) / 256, 256>>>(da, db, df, dout, n);
  CHECK(cudaGetLastError());
  CHECK(cudaMemcpy(out.data(), dout, sizeof(Out) * (size_t)n, cudaMemcpyDeviceToHost));
  return std::fwrite(out.data(), sizeof(Out), n, stdout) == (size_t)n ? 0 : 2;
}
