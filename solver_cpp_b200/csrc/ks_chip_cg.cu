// Instantiations and launches of the CG with the matrix on chip
// (ks_chip_cg.cuh), on tiles (ks_tile_cg.cuh) and of CSR matrices (ks_csr_cg.cuh).
#include "ks_csr_cg.cuh"
#include "ks_tile_cg.cuh"

namespace ks {

// A cooperative launch of fn(args...), the kernel `name`, or with `probe` only
// the check that it can be co-resident.
template <class... KArgs, class... Args>
static cudaError_t coop_launch(ks_ctx *ctx, const char *name, void (*fn)(KArgs...), const ChipShape &sh, bool probe,
                               bool *fits, int cls, int threads, const Args &...args) {
  cudaError_t e = allow_smem(ctx, fn);
  if (e != cudaSuccess) return e;
  if (probe) {
    int b = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fn, threads, sh.smem);
    *fits = e == cudaSuccess && b >= 1;
    return e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sh.G);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = sh.smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  ctx->solve_kernel = name;
  ctx->launches++;
  ProfLaunch pl(ctx, cls);
  return cudaLaunchKernelEx(&cfg, fn, args...);
}

template <class VT, int NDG, int RJ, bool kTile>
static cudaError_t chip_launch_n(ks_ctx *ctx, const ChipArgs &a, const ChipShape &sh, bool probe, bool *fits, int cls) {
  return coop_launch(ctx, "k_cg_chip", k_cg_chip<VT, NDG, RJ, kTile>, sh, probe, fits, cls, kChipThreads, a);
}

template <class VT, int NDG, bool kTile>
static cudaError_t chip_launch_d(ks_ctx *ctx, const ChipArgs &a, const ChipShape &sh, bool probe, bool *fits, int cls) {
  if (sh.rj == 1) return chip_launch_n<VT, NDG, 1, kTile>(ctx, a, sh, probe, fits, cls);
  if (sh.rj == 2) return chip_launch_n<VT, NDG, 2, kTile>(ctx, a, sh, probe, fits, cls);
  if (sh.rj == 4) return chip_launch_n<VT, NDG, 4, kTile>(ctx, a, sh, probe, fits, cls);
  if (sh.rj == 8) return chip_launch_n<VT, NDG, 8, kTile>(ctx, a, sh, probe, fits, cls);
  if constexpr (sizeof(VT) == 4) return chip_launch_n<VT, NDG, 16, kTile>(ctx, a, sh, probe, fits, cls);
  return cudaErrorInvalidValue;
}
template <class VT>
static cudaError_t chip_launch_t(ks_ctx *ctx, const ChipArgs &a, const ChipShape &sh, bool probe, bool *fits, int cls) {
  if (sh.tile) return chip_launch_d<VT, 7, true>(ctx, a, sh, probe, fits, cls);
  if (a.nd == 7) return chip_launch_d<VT, 7, false>(ctx, a, sh, probe, fits, cls);
  if (a.nd == 5) return chip_launch_d<VT, 5, false>(ctx, a, sh, probe, fits, cls);
  return chip_launch_d<VT, 0, false>(ctx, a, sh, probe, fits, cls);
}

cudaError_t chip_launch_f64(ks_ctx *ctx, const ChipArgs &a, const ChipShape &sh, bool probe, bool *fits, int cls) {
  return chip_launch_t<double>(ctx, a, sh, probe, fits, cls);
}
cudaError_t chip_launch_f32(ks_ctx *ctx, const ChipArgs &a, const ChipShape &sh, bool probe, bool *fits, int cls) {
  return chip_launch_t<float>(ctx, a, sh, probe, fits, cls);
}

cudaError_t tile_launch(ks_ctx *ctx, const CsrDev &A, const ChipArgs &a, const ChipShape &sh, bool probe, bool *fits,
                        int cls) {
  TileDiag D{};
  for (int k = 0; k < 7; k++) D.v[k] = A.dia_cv[k];
  return coop_launch(ctx, "k_cg_tile", k_cg_tile, sh, probe, fits, cls, kChipThreads, a, D);
}

bool csr_window_fits(const ks_ctx *ctx, long long n, int lo, int hi) {
  CsrShape s;
  return csr_shape(ctx, n, lo, hi, &s);
}

cudaError_t csr_launch(ks_ctx *ctx, const CsrCgArgs &a, const CsrShape &sh, bool probe, bool *fits, int cls) {
  auto run = [&](auto kern) { return coop_launch(ctx, "k_cg_csr", kern, sh, probe, fits, cls, sh.threads, a); };
  if (sh.threads == 1024) return run(k_cg_csr<1024, 4>);  // more than 2,048 rows per CTA
  return sh.rj == 1 ? run(k_cg_csr<512, 1>) : sh.rj == 2 ? run(k_cg_csr<512, 2>) : run(k_cg_csr<512, 4>);
}

}  // namespace ks
