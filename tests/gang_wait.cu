// One grid of the cooperative form with two empty patches, which still exchange
// their residual sums: a host for tests of the exchange's waits.  Prints, per
// launch, status, milliseconds and the second CTA's count of residual exchanges.
#include <cstdio>

#include "../rdc-xpbd-taichi_gb300/csrc/xpbd_device.cuh"

#include "../rdc-xpbd-taichi_gb300/csrc/xpbd_gang.cuh"

using namespace xpbd;

struct IO {
  static constexpr bool kTapes = false;
  int* flags;    // timeout, nonfinite
  double* rows;  // [4 K]
  __device__ int body(int) const { return 0; }
  __device__ int tets(int) const { return 0; }
  __device__ int first_tet(int) const { return 0; }
  __device__ int group(int) const { return 2; }
  __device__ int first(int) const { return 0; }
  __device__ void compliance(int, int, const float (&)[9], float&, float&) const {}
  __device__ double count(int) const { return 1.0; }
  __device__ double rho(int) const { return 0.999; }
  __device__ double* row(int, int k) const { return rows + 4 * k; }
  __device__ void nonfinite() const { flags[1] = 1; }
  __device__ void timeout() const { flags[0] = 1; }
  __device__ bool timed_out() const { return *reinterpret_cast<volatile int*>(flags) != 0; }
  __device__ void substep_done(int, int, int, int) const {}
  __device__ void done(int, bool, double, int) const {}
};

#define CHECK(e) do { if ((e) != cudaSuccess) { std::printf("%s\n", cudaGetErrorString(cudaGetLastError())); return 1; } } while (0)

int main() {
  constexpr int K = 5;
  char* m = nullptr;
  CHECK(cudaMalloc(&m, 1 << 16));
  CHECK(cudaMemset(m, 0, 1 << 16));
  // empty patches: offsets of zero everywhere, no vertex, no tet
  GangDev d{};
  d.voff = d.dst_off = d.inbox = reinterpret_cast<int*>(m);
  d.corners = reinterpret_cast<uint16_t*>(m + 4096);  // [2][1024]
  d.vert_slots = reinterpret_cast<uint4*>(m + 16384);
  d.sums = reinterpret_cast<double*>(m + 20480);
  d.bar = reinterpret_cast<unsigned*>(m + 24576);
  d.state = reinterpret_cast<uint2*>(m + 28672);
  d.n_patches = 2;
  IO io{reinterpret_cast<int*>(m + 32768), reinterpret_cast<double*>(m + 36864)};
  GangRun r{};
  r.K = K;
  r.n_sub = r.cheb = 1;
  r.rec_base = -1;
  r.dt = 0.01f;
  Gang g{};
  g.d = d;
  g.smem = sizeof(GangPatch);
  g.n_ctas = 2;
  auto kernel = k_gang<IO, true, false, false, kGangPlain>;
  CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g.smem));
  cudaEvent_t a, b;
  CHECK(cudaEventCreate(&a));
  CHECK(cudaEventCreate(&b));
  for (int launch = 0; launch < 5; ++launch) {
    if (launch == 2) {  // the first CTA now waits for an exchange that nobody comes to
      uint2 st{};
      CHECK(cudaMemcpy(&st, d.state, sizeof(st), cudaMemcpyDeviceToHost));
      st.y += 1000;
      CHECK(cudaMemcpy(d.state, &st, sizeof(st), cudaMemcpyHostToDevice));
    }
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[1];
    gang_config<IO>(g, cfg, at);
    CHECK(cudaEventRecord(a));
    CHECK(cudaLaunchKernelEx(&cfg, kernel, g.d, r, io));
    CHECK(cudaEventRecord(b));
    CHECK(cudaDeviceSynchronize());
    float ms = 0.f;
    int timeout = 0;
    uint2 st[2];
    CHECK(cudaEventElapsedTime(&ms, a, b));
    CHECK(cudaMemcpy(&timeout, io.flags, sizeof(int), cudaMemcpyDeviceToHost));
    CHECK(cudaMemcpy(st, d.state, sizeof(st), cudaMemcpyDeviceToHost));
    std::printf("%d %.3f %u\n", timeout, ms, st[1].y);
  }
  return 0;
}
