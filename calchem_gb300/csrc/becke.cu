// becke.cu -- the Becke weight derivative of the FP64 XC gradient, sum_g raw_w f dB/dR, as its own kernel.
//
// One warp per point (becke_point), its pair tables in shared memory up to 45 atoms and in device memory
// above.  The FP64 pipe (one warp instruction per 16 cycles and SM) bounds it, so the warps of several CTAs
// share an SM, the pairs are evaluated once each, their constants come from tables and the step takes the slope's
// factors on its way: ~500 FP64 instructions a point for 24 atoms.  Eight waters (Medium): 4.20 ms with both
// orientations of a pair, 2.55 ms with one, 2.2 ms so.  Each CTA takes a range of consecutive points and
// writes one row of per-atom sums.
#include <cuda_runtime.h>

#include <algorithm>

#include "becke_grad.cuh"
#include "common.cuh"
#include "launch.h"

namespace cxc {

namespace {

constexpr int kWarps = 4;
constexpr int kPtsPerWarp = 4;             // with tables in shared memory
constexpr int kGlobalCtas = 304;           // with tables in device memory,
constexpr size_t kGlobalBytes = (size_t)4 << 30;  // which take this much at most (and what the caller can spare)
constexpr size_t kBeckeSmem = 200 << 10;

__global__ void __launch_bounds__(32 * kWarps) becke_fp64_kernel(DevGrid G, GradArgs A, const double* __restrict__ fx,
                                                                 double* __restrict__ part, double* tables,
                                                                 int pts_per_warp) {
  extern __shared__ __align__(16) unsigned char bsm[];
  const int n = A.n_atoms, n3 = 3 * n;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t per_warp = becke::becke_scratch_doubles(n);
  double* const scr = tables ? tables + (size_t)blockIdx.x * kWarps * per_warp : reinterpret_cast<double*>(bsm);
  becke::BeckeScratch W;
  W.carve(scr + (size_t)warp * per_warp, n);
  for (int k = lane; k < n3; k += 32) W.wacc[k] = 0.0;
  __syncwarp();
  const int p0 = (blockIdx.x * kWarps + warp) * pts_per_warp;
  for (int p = p0; p < min(p0 + pts_per_warp, G.n_pts); ++p) {
    const double f = fx[p], rw = A.raw_w[p];
    if (fabs(f) < 1e-18 || rw == 0.0) continue;
    becke::becke_point(n, A.xyz, A.inv_r, A.pair_tab, A.pairs, A.n_pairs, A.host[p], G.px[p], G.py[p], G.pz[p], rw * f, W);
  }
  __syncthreads();
  double* out = part + (size_t)blockIdx.x * n3;
  for (int k = threadIdx.x; k < n3; k += 32 * kWarps) {
    double v = 0.0;
    for (int w = 0; w < kWarps; ++w) v += scr[(size_t)w * per_warp + 2 * n + k];
    out[k] = v;
  }
}

size_t smem_bytes(int n_atoms) { return kWarps * becke::becke_scratch_doubles(n_atoms) * sizeof(double); }
bool in_smem(int n_atoms) { return smem_bytes(n_atoms) <= kBeckeSmem; }

}  // namespace

int becke_fp64_ctas(int n_pts, int n_atoms, size_t budget) {
  const int c = (n_pts + kWarps * kPtsPerWarp - 1) / (kWarps * kPtsPerWarp);
  if (in_smem(n_atoms)) return c;
  return std::max<size_t>(1, std::min<size_t>({(size_t)c, (size_t)kGlobalCtas,
                                                    std::min(kGlobalBytes, budget) / smem_bytes(n_atoms)}));
}

size_t becke_fp64_table_doubles(int n_ctas, int n_atoms) {
  return in_smem(n_atoms) ? 0 : (size_t)n_ctas * kWarps * becke::becke_scratch_doubles(n_atoms);
}

cudaError_t launch_becke_fp64(const DevGrid& G, const GradArgs& A, const double* fx, double* part, double* tables,
                              int n_ctas, cudaStream_t st) {
  const bool shared = in_smem(A.n_atoms);
  const size_t smem = shared ? smem_bytes(A.n_atoms) : 0;
  if (shared) {
    const cudaError_t e = cudaFuncSetAttribute(becke_fp64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  becke_fp64_kernel<<<n_ctas, 32 * kWarps, smem, st>>>(G, A, fx, part, shared ? nullptr : tables,
                                                       (G.n_pts + n_ctas * kWarps - 1) / (n_ctas * kWarps));
  return cudaGetLastError();
}

}  // namespace cxc
