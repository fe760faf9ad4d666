// Applies of blocks factored by LU (the fallback on a block whose Cholesky fails) to several
// vectors at once against one vector at a time, bit for bit; restricted and basic Schwarz, LU
// blocks beside Cholesky ones.
#include <cmath>
#include <cstdio>
#include <vector>

#include "petrbf_gb300.h"
#include "rasm.h"

using namespace prbf;

static int run(int pc, int nv) {
  std::vector<double> x, y;
  unsigned q = 99;
  auto uniform = [&] { return (q = q * 1664525u + 1013904223u) / 4294967296.0; };
  for (int i = 0; i < 30; i++)
    for (int j = 0; j < 30; j++) {
      x.push_back(i + 0.3 * uniform());
      y.push_back(j + 0.3 * uniform());
    }
  for (int i = 0; i < 40; i++) {  // far closer than sigma: no positive pivots there
    x.push_back(3.0 + 0.1 * uniform());
    y.push_back(3.0 + 0.1 * uniform());
  }
  const int n = (int)x.size();
  prbf_params p;
  prbf_params_default(&p);
  p.sigma = 1.0;
  p.nsigma_box = 6;
  p.sigma_buffer = 14;
  p.sigma_trunc = 20;
  p.pc_type = pc;
  p.block_fallback = PRBF_FALLBACK_LU;
  prbf_ctx* ctx = nullptr;
  if (prbf_ctx_create(&p, &ctx) || prbf_matvec_setup(ctx, n, x.data(), y.data(), nullptr)) return 1000;
  Ctx& c = ctx->c;
  int bad = 0;
  {
    RasmPlan R;
    R.max_nv = nv;
    R.lu_fallback = true;
    rasm_build(R, c.mv_pts, false, c.ws, c.err.get(), c.stream, 1e9, false, pc == PRBF_PC_ASM);
    rasm_set_apply_smem(R);
    if (R.nlu < 1 || R.nlu >= R.nblocks) bad += 1;  // some, not all
    const long long ld = (n + 4 + 31) / 32 * 32;
    std::vector<double> h(ld * nv, 0.0), all(ld * nv), one(ld);
    for (int v = 0; v < nv; v++)
      for (int i = 0; i < n; i++) h[v * ld + i] = std::sin(0.1 * (v + 1) * i + v);
    DevBuf<double> r, z;
    r.reserve(ld * nv);
    z.reserve(ld * nv);
    PRBF_CUDA(cudaMemcpy(r.get(), h.data(), sizeof(double) * h.size(), cudaMemcpyHostToDevice));
    PRBF_CUDA(cudaMemset(z.get(), 0, sizeof(double) * ld * nv));
    PRBF_CUDA(cudaDeviceSynchronize());
    rasm_apply(R, c.mv_pts.cs.get(), r.get(), z.get(), c.stream, nullptr, nv, ld);
    PRBF_CUDA(cudaStreamSynchronize(c.stream));
    PRBF_CUDA(cudaMemcpy(all.data(), z.get(), sizeof(double) * all.size(), cudaMemcpyDeviceToHost));
    for (int v = 0; v < nv; v++) {
      rasm_apply(R, c.mv_pts.cs.get(), r.get() + v * ld, z.get(), c.stream);
      PRBF_CUDA(cudaStreamSynchronize(c.stream));
      PRBF_CUDA(cudaMemcpy(one.data(), z.get(), sizeof(double) * n, cudaMemcpyDeviceToHost));
      for (int i = 0; i < n; i++) bad += one[i] != all[v * ld + i] || !std::isfinite(one[i]) ? 2 : 0;
    }
    std::printf("pc %d, %d vectors: %d of %d blocks by LU, bad %d\n", pc, nv, R.nlu, R.nblocks, bad);
  }
  prbf_ctx_destroy(ctx);
  return bad;
}

int main() {
  try {
    int bad = 0;
    for (int pc : {PRBF_PC_RASM, PRBF_PC_ASM})
      for (int nv : {2, 3, 4}) bad += run(pc, nv);
    return bad ? 1 : 0;
  } catch (const Error& e) {
    std::printf("%s\n", e.what());
    return 2;
  }
}
