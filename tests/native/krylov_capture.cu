// GMRES whose operator fails while the iteration is captured -- by an exception, or by a launch
// that the runtime refuses -- and then no longer does: the call raises, the same Krylov state
// solves afterwards, and its destruction after a failure is clean. On one thread and on four.
#include <cmath>
#include <cstdio>
#include <thread>
#include <vector>

#include "krylov.h"

using namespace prbf;

__global__ void k_scale(int n, const double* x, double* y, int inverse) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = inverse ? x[i] / (1.0 + 0.5 * (i % 3)) : x[i] * (2.0 + i % 7);
}

struct Op : Operator {
  int n = 0, how = 0;  // how it fails inside a capture: 0 not, 1 an exception, 2 a refused launch
  static bool capturing(cudaStream_t s) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    PRBF_CUDA(cudaStreamIsCapturing(s, &st));
    return st != cudaStreamCaptureStatusNone;
  }
  void apply_A(const double* x, double* y, const int*, cudaStream_t s) const override {
    k_scale<<<(n + 255) / 256, 256, 0, s>>>(n, x, y, 0);
    PRBF_CHECK_LAUNCH();
  }
  void apply_B(const double* r, double* z, const int*, cudaStream_t s) const override {
    if (how == 1 && capturing(s)) throw Error(PRBF_ERR_CAPACITY, "made to fail");
    // (more shared memory than an SM has: refused before anything runs)
    k_scale<<<(n + 255) / 256, 256, how == 2 && capturing(s) ? 300 * 1024 : 0, s>>>(n, r, z, 1);
    PRBF_CHECK_LAUNCH();
  }
};

static int run(int n) {
  int wrong = 0;
  cudaStream_t s;
  PRBF_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  DevBuf<double> b, x;
  std::vector<double> h(n), g(n);
  for (int i = 0; i < n; i++) h[i] = std::cos(0.1 * i);
  b.reserve(n + 64);
  x.reserve(n + 64);
  PRBF_CUDA(cudaMemsetAsync(b.get(), 0, sizeof(double) * (n + 64), s));
  PRBF_CUDA(cudaMemcpyAsync(b.get(), h.data(), sizeof(double) * n, cudaMemcpyHostToDevice, s));
  for (int round = 0; round < 6; round++) {
    Krylov K;
    K.init(n, 20, s);
    Op op;
    op.n = n;
    for (int how : {1, 2, 0, 2, 0, 1}) {  // (destroyed after a failure in the end)
      op.how = how;
      K.graph_op = nullptr;
      PRBF_CUDA(cudaMemsetAsync(x.get(), 0, sizeof(double) * (n + 64), s));
      bool raised = false;
      try {
        K.solve(op, b.get(), x.get(), true, 1e-12, 0.0, 1e10, 100, true, s);
      } catch (const Error&) {
        raised = true;
      }
      if (raised != (how != 0)) wrong++;
      if (raised) continue;
      PRBF_CUDA(cudaMemcpyAsync(g.data(), x.get(), sizeof(double) * n, cudaMemcpyDeviceToHost, s));
      PRBF_CUDA(cudaStreamSynchronize(s));
      for (int i = 0; i < n; i++)
        if (!(std::fabs(g[i] * (2.0 + i % 7) - h[i]) <= 1e-10)) wrong++;
    }
  }
  PRBF_CUDA(cudaStreamSynchronize(s));
  cudaStreamDestroy(s);
  return wrong;
}

int main() {
  try {
    int wrong = run(1000);
    std::vector<int> w(4, 0);
    std::vector<std::thread> t;
    for (int k = 0; k < 4; k++) t.emplace_back([&w, k] { w[k] = run(500 + 300 * k); });
    for (auto& q : t) q.join();
    for (int k : w) wrong += k;
    const cudaError_t e = cudaDeviceSynchronize();
    std::printf("wrong %d, %s\n", wrong, cudaGetErrorString(e));
    return wrong || e != cudaSuccess;
  } catch (const Error& e) {
    std::printf("%s\n", e.what());
    return 1;
  }
}
