// becke.cu -- the Becke weight derivative of the FP64 XC gradient, sum_g raw_w f dB/dR, as its own kernel for
// molecules whose pair tables fit in shared memory (up to 45 atoms); larger ones run it inside the quadrature
// kernel, one warp per point with tables in its slab.
//
// One warp per point as there (becke_point), but with the tables in shared memory and 8-12 warps resident
// per SM instead of one CTA's eight sharing it with the contractions: the FP64 pipe (one warp instruction
// per 16 cycles and SM) is what bounds it.  Each warp takes kPtsPerWarp consecutive points and each CTA writes
// one row of per-atom sums.
#include <cuda_runtime.h>

#include "becke_grad.cuh"
#include "common.cuh"
#include "launch.h"

namespace cxc {

namespace {

constexpr int kWarps = 4;
constexpr int kPtsPerWarp = 4;
constexpr size_t kBeckeSmem = 200 << 10;

__global__ void __launch_bounds__(32 * kWarps) becke_fp64_kernel(DevGrid G, GradArgs A, const double* __restrict__ fx,
                                                                 double* __restrict__ part) {
  extern __shared__ __align__(16) unsigned char bsm[];
  const int n = A.n_atoms, n3 = 3 * n;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* const scr = reinterpret_cast<double*>(bsm);
  const size_t per_warp = becke::becke_scratch_doubles(n);
  becke::BeckeScratch W;
  W.dist = scr + (size_t)warp * per_warp;
  W.cell = W.dist + n;
  W.wacc = W.cell + n;
  W.s = W.wacc + n3;
  W.e = W.s + (size_t)n * n;
  W.l = W.e + (size_t)n * n;
  for (int k = lane; k < n3; k += 32) W.wacc[k] = 0.0;
  __syncwarp();
  const int p0 = (blockIdx.x * kWarps + warp) * kPtsPerWarp;
  for (int p = p0; p < min(p0 + kPtsPerWarp, G.n_pts); ++p) {
    const double f = fx[p], rw = A.raw_w[p];
    if (fabs(f) < 1e-18 || rw == 0.0) continue;
    becke::becke_point(n, A.xyz, A.inv_r, A.a_ij, A.pairs, A.n_pairs, A.host[p], G.px[p], G.py[p], G.pz[p], rw * f, W);
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

}  // namespace

bool becke_fp64_fits(int n_atoms) { return n_atoms > 1 && smem_bytes(n_atoms) <= kBeckeSmem; }

int becke_fp64_ctas(int n_pts) { return (n_pts + kWarps * kPtsPerWarp - 1) / (kWarps * kPtsPerWarp); }

cudaError_t launch_becke_fp64(const DevGrid& G, const GradArgs& A, const double* fx, double* part, cudaStream_t st) {
  const size_t smem = smem_bytes(A.n_atoms);
  const cudaError_t e = cudaFuncSetAttribute(becke_fp64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  becke_fp64_kernel<<<becke_fp64_ctas(G.n_pts), 32 * kWarps, smem, st>>>(G, A, fx, part);
  return cudaGetLastError();
}

}  // namespace cxc
