// becke.cu -- the Becke weight derivative of the FP64 XC gradient, sum_g raw_w f dB/dR, as its own kernel.
//
// One warp per point up to 32 atoms, eight above (becke_point), with the pair tables in shared memory up to 95 atoms
// and in device memory above.  The FP64 pipe (one warp instruction per 16 cycles and SM) bounds it, so the warps
// of several CTAs share an SM, the pairs are evaluated once each, their constants come from tables and the
// step takes the slope's factors on its way: 492 FP64 warp instructions a point for 24 atoms, that pipe 84 % busy.  Eight waters
// (Medium): 4.20 ms with both orientations of a pair, 2.55 ms with one, 2.2 ms so.  A warp's tables of 36 atoms
// already leave four warps per SM, so that larger molecules give a point to the whole CTA; the gradient call on
// Coarse grids, one warp per point against eight: 24 atoms 4.49 against 5.72 ms, 30: 3.57 against 4.28, 36: 7.15
// against 6.92, 45: 12.1 against 10.4, 54 (its tables in device memory with one) 21.0 against 14.5, 72: 53.9 against
// 35.9, 120 (in device memory with both) 274 against 168.  Each CTA takes a range of consecutive points and
// writes one row of per-atom sums.
#include <cuda_runtime.h>

#include <algorithm>

#include "becke_grad.cuh"
#include "common.cuh"
#include "launch.h"

namespace cxc {

namespace {

constexpr int kWarps = 4;        // points in flight per CTA with one warp per point
constexpr int kWarpAtoms = 32;   // up to here
constexpr int kTeam = 256;       // threads per point above
constexpr int kPts = 16;         // points of a CTA with tables in shared memory
constexpr int kGlobalCtas = 304;                  // with tables in device memory,
constexpr size_t kGlobalBytes = (size_t)4 << 30;  // which take this much at most (and what the caller can spare)
constexpr size_t kBeckeSmem = 220 << 10;

__host__ __device__ int teams_of(int n) { return n <= kWarpAtoms ? kWarps : 1; }
// doubles of one team: its tables, and above one warp the warps' sums
__host__ __device__ size_t team_doubles(int n) {
  return becke::becke_scratch_doubles(n) + (n <= kWarpAtoms ? 0 : 3 * kTeam / 32);
}

template <int kT>
__global__ void __launch_bounds__(kT == 32 ? 32 * kWarps : kT)
    becke_fp64_kernel(DevGrid G, GradArgs A, const double* __restrict__ fx, double* __restrict__ part, double* tables,
                      int pts_per_team) {
  extern __shared__ __align__(16) unsigned char bsm[];
  constexpr int kTeams = kT == 32 ? kWarps : 1;
  const int n = A.n_atoms, n3 = 3 * n;
  const int team = threadIdx.x / kT, tid = threadIdx.x % kT;
  const size_t per_team = team_doubles(n);
  double* const scr = tables ? tables + (size_t)blockIdx.x * per_team : reinterpret_cast<double*>(bsm);
  becke::BeckeScratch W;
  W.carve(scr + (size_t)team * per_team, n);
  double* const red = scr + becke::becke_scratch_doubles(n);
  for (int k = tid; k < n3; k += kT) W.wacc[k] = 0.0;
  __syncthreads();
  const int p0 = (blockIdx.x * kTeams + team) * pts_per_team;
  for (int p = p0; p < min(p0 + pts_per_team, G.n_pts); ++p) {
    const double f = fx[p], rw = A.raw_w[p];
    if (fabs(f) < 1e-18 || rw == 0.0) continue;
    becke::becke_point<kT>(n, A.xyz, A.inv_r, A.pair_tab, A.pairs, A.n_pairs, A.host[p], G.px[p], G.py[p], G.pz[p],
                           rw * f, W, tid, red);
  }
  __syncthreads();
  double* out = part + (size_t)blockIdx.x * n3;
  for (int k = threadIdx.x; k < n3; k += kT * kTeams) {
    double v = 0.0;
    for (int w = 0; w < kTeams; ++w) v += scr[(size_t)w * per_team + 2 * n + k];
    out[k] = v;
  }
}

size_t cta_bytes(int n) { return teams_of(n) * team_doubles(n) * sizeof(double); }
bool in_smem(int n) { return cta_bytes(n) <= kBeckeSmem; }

}  // namespace

int becke_fp64_ctas(int n_pts, int n_atoms, size_t budget) {
  const int c = (n_pts + kPts - 1) / kPts;
  if (in_smem(n_atoms)) return c;
  return (int)std::max<size_t>(
      1, std::min<size_t>({(size_t)c, (size_t)kGlobalCtas, std::min(kGlobalBytes, budget) / cta_bytes(n_atoms)}));
}

size_t becke_fp64_table_doubles(int n_ctas, int n_atoms) {
  return in_smem(n_atoms) ? 0 : (size_t)n_ctas * cta_bytes(n_atoms) / sizeof(double);
}

cudaError_t launch_becke_fp64(const DevGrid& G, const GradArgs& A, const double* fx, double* part, double* tables,
                              int n_ctas, cudaStream_t st) {
  const int n = A.n_atoms, teams = teams_of(n);
  const bool shared = in_smem(n);
  const size_t smem = shared ? cta_bytes(n) : 0;
  auto* kernel = teams > 1 ? becke_fp64_kernel<32> : becke_fp64_kernel<kTeam>;
  if (shared) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  kernel<<<n_ctas, teams > 1 ? 32 * kWarps : kTeam, smem, st>>>(G, A, fx, part, shared ? nullptr : tables,
                                                              (G.n_pts + n_ctas * teams - 1) / (n_ctas * teams));
  return cudaGetLastError();
}

}  // namespace cxc
