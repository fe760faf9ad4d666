// The batched sums with items of 32, 64 and 128 targets: an item computes its own targets and no
// others, and the targets' sums do not depend on the tile. One problem of three cells; the
// fixed-point, the FP64 pipe's and the FP32 kernels.
#include <cmath>
#include <cstdio>
#include <vector>

#include "context.h"

using namespace prbf;

static int run(int dim, int forms, bool fp32) {
  const int per[3] = {100, 40, 128};
  const double sigma = 0.01;
  std::vector<double> xyz[3];
  std::vector<int> hcs = {0};
  unsigned r = 12345;
  auto uniform = [&] { return (r = r * 1664525u + 1013904223u) / 4294967296.0; };
  double bb[6] = {1e9, -1e9, 1e9, -1e9, 1e9, -1e9};
  for (int c = 0; c < 3; c++) {
    for (int i = 0; i < per[c]; i++)
      for (int d = 0; d < 3; d++) {
        const double u = (0.05 + 0.9 * uniform()) * 0.04 + (d == 1 ? 0.04 * c : 0.0);
        xyz[d].push_back(u);
        bb[2 * d] = std::fmin(bb[2 * d], u);
        bb[2 * d + 1] = std::fmax(bb[2 * d + 1], u);
      }
    hcs.push_back(hcs.back() + per[c]);
  }
  bb[0] = bb[2] = bb[4] = 0.0;  // the grid's corner, so that cells are where the points are
  const int n = hcs.back();
  Grid g = make_grid(dim, bb, sigma, 4, 12, 20);
  if (g.nx != 1 || g.nz != 1 || g.ny != 3) return 100;
  cudaStream_t s;
  PRBF_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  DevBuf<double> p[3], gv, w;
  DevBuf<int> cs;
  DevBuf<unsigned> err;
  std::vector<double> hg(n + 4, 0.0), hw(n);
  for (int i = 0; i < n; i++) hg[i] = uniform() - 0.5;
  auto up = [&](auto& b, const auto& h, size_t pad) {
    b.reserve(h.size() + pad);
    PRBF_CUDA(cudaMemset(b.get(), 0, sizeof(h[0]) * (h.size() + pad)));
    PRBF_CUDA(cudaMemcpy(b.get(), h.data(), sizeof(h[0]) * h.size(), cudaMemcpyHostToDevice));
  };
  for (int d = 0; d < 3; d++) up(p[d], xyz[d], 4);
  up(gv, hg, 4);
  up(cs, hcs, 1);
  w.reserve(n + 4);
  err.reserve(4);
  PRBF_CUDA(cudaMemset(err.get(), 0, 16));
  exp_table_dev(s);
  const PointsView v{n, p[0].get(), p[1].get(), dim == 3 ? p[2].get() : nullptr, cs.get()};
  GaussPlan P;
  P.g = g;
  P.batched = true;
  up(P.grids, std::vector<Grid>{g}, 0);
  up(P.cprob, std::vector<int>(3, 0), 0);
  PRBF_CUDA(cudaDeviceSynchronize());
  gauss_plan_forms_batch(P, {g}, v, forms, s);
  int wrong = 0;
  std::vector<double> ref;
  for (int tile : {128, 64, 32}) {
    std::vector<int2> items;
    for (int c = 0; c < 3; c++)
      for (int t = hcs[c]; t < hcs[c + 1]; t += tile) items.push_back(make_int2(c, t));
    P.max_tile = tile;
    for (int pass = 0; pass < 2; pass++) {  // the first item alone, then all
      P.nitems = pass ? (int)items.size() : 1;
      up(P.items, items, 0);
      std::vector<double> seven(n + 4, 7.0);
      PRBF_CUDA(cudaMemcpy(w.get(), seven.data(), sizeof(double) * (n + 4), cudaMemcpyHostToDevice));
      PRBF_CUDA(cudaDeviceSynchronize());
      gauss_sum_dev(P, v, v, gv.get(), w.get(), fp32, err.get(), s);
      PRBF_CUDA(cudaStreamSynchronize(s));
      PRBF_CUDA(cudaMemcpy(hw.data(), w.get(), sizeof(double) * n, cudaMemcpyDeviceToHost));
      if (!pass) {
        for (int i = 0; i < n; i++) wrong += (hw[i] != 7.0) != (i < std::min(tile, per[0]));
      } else if (ref.empty()) {
        ref = hw;
        for (double q : ref) wrong += !(std::isfinite(q) && q != 7.0);
      } else {
        for (int i = 0; i < n; i++) wrong += hw[i] != ref[i];
      }
    }
  }
  unsigned he = 0;
  PRBF_CUDA(cudaMemcpy(&he, err.get(), sizeof(he), cudaMemcpyDeviceToHost));
  cudaStreamDestroy(s);
  return wrong + (he ? 1000 : 0);
}

int main() {
  try {
    int bad = 0;
    for (int dim : {2, 3}) {
      const int k[3] = {run(dim, FORM_F64, false), run(dim, FORM_PIPE64, false), run(dim, FORM_F32, true)};
      std::printf("%dD: fixed point %d, FP64 pipe %d, FP32 %d\n", dim, k[0], k[1], k[2]);
      bad |= k[0] | k[1] | k[2];
    }
    return bad ? 1 : 0;
  } catch (const Error& e) {
    std::printf("%s\n", e.what());
    return 2;
  }
}
