// Basic Schwarz in FP64 with several right-hand sides: the slots of several vectors are taken
// only where they fit the budget, and the applies of four vectors are the same either way.
#include <cmath>
#include <cstdio>
#include <vector>

#include "petrbf_gb300.h"
#include "rasm.h"

using namespace prbf;

int main() {
  try {
    const int m = 40, n = m * m, nv = 4;
    std::vector<double> x(n), y(n);
    for (int i = 0; i < n; i++) {
      x[i] = (i / m + 0.2 * std::sin(7.0 * i)) / m;
      y[i] = (i % m + 0.2 * std::cos(5.0 * i)) / m;
    }
    prbf_params p;
    prbf_params_default(&p);
    p.sigma = 1.25 / m;
    p.pc_type = PRBF_PC_ASM;
    prbf_ctx* ctx = nullptr;
    if (prbf_ctx_create(&p, &ctx) || prbf_matvec_setup(ctx, n, x.data(), y.data(), nullptr)) return 2;
    Ctx& c = ctx->c;
    const long long ld = (n + 4 + 31) / 32 * 32;
    DevBuf<double> r, z;
    r.reserve(ld * nv);
    z.reserve(ld * nv);
    std::vector<double> h(ld * nv, 0.0), out[3];
    for (size_t i = 0; i < h.size(); i++) h[i] = std::sin(0.37 * i) + 0.1 * std::cos(3.1 * i);
    PRBF_CUDA(cudaMemcpy(r.get(), h.data(), sizeof(double) * h.size(), cudaMemcpyHostToDevice));
    int bad = 0;
    long long slots = 0;
    for (int k = 0; k < 3; k++) {
      RasmPlan R;
      R.max_nv = nv;
      // plenty; the slots of two vectors and a half; next to nothing
      rasm_build(R, c.mv_pts, false, c.ws, c.err.get(), c.stream, k == 0 ? 1e9 : k == 1 ? 2.5 * 8 * slots : 1.0, false,
                 true);
      rasm_set_apply_smem(R);
      slots = R.nslot;
      const int want = k == 0 ? 4 : k == 1 ? 2 : 1;
      if (R.max_nv != want || R.Y.n < (size_t)R.nslot * R.max_nv) bad |= 1 << k;
      if (k && R.Y.n >= (size_t)R.nslot * nv) bad |= 16;
      PRBF_CUDA(cudaMemset(z.get(), 0, sizeof(double) * ld * nv));
      PRBF_CUDA(cudaDeviceSynchronize());
      rasm_apply(R, c.mv_pts.cs.get(), r.get(), z.get(), c.stream, nullptr, nv, ld);
      PRBF_CUDA(cudaStreamSynchronize(c.stream));
      out[k].resize(h.size());
      PRBF_CUDA(cudaMemcpy(out[k].data(), z.get(), sizeof(double) * h.size(), cudaMemcpyDeviceToHost));
      if (out[k] != out[0]) bad |= 256 << k;
      std::printf("slots %lld, vectors %d (%d)\n", R.nslot, R.max_nv, want);
    }
    prbf_ctx_destroy(ctx);
    std::printf("bad %d\n", bad);
    return bad ? 1 : 0;
  } catch (const Error& e) {
    std::printf("%s\n", e.what());
    return 2;
  }
}
