// xc_grad_f64tc.cu -- the FP64 XC gradient's quadrature with its contractions on the tensor cores.
//
// The work of xc_grad.cu (the AO force terms and the host atoms' terms of dExc/dR at fixed densities; the
// weight derivative is becke.cu's), with T_s = P_s Phi and Y_s = P_s Psi_s, Psi_s = (w u_s) . grad Phi, as
// exact integer-slice products (f64_gemm.cuh) in place of FP64 FMAs, two CTAs of 256 threads per SM.  The
// FP64 pipe keeps the AO values with their second derivatives, rho, the functional and the force terms.
//
// A row's force on its atom is summed per point over runs of columns of one atom, a run's sum is reduced
// over the warp's 32 points, and the runs are added to the batch's per-atom sums in a fixed order, so that
// results are deterministic.
//
// The SIMT form is bound by its 2 m^2 FMAs a point and spin on the FP64 pipe; here that pipe keeps the Hessians
// and the force terms, which run under the other CTA's copies and MMAs.  Eight waters
// B3LYP Medium: 5.50 -> 2.11 ms.
#include <cuda_runtime.h>

#include "common.cuh"
#include "f64_gemm.cuh"
#include "fp64_ao.cuh"
#include "launch.h"
#include "xc_device.cuh"

namespace cxc {

namespace {

using namespace f64s;

constexpr int kGrad = 1, kHess = 4, kPsi = 10, kTp = 11, kPlanes = 13;  // planes; phi is 0, T_s 11 and 12
constexpr int kMaxAtoms = 256;  // per-atom sums in shared memory, atom indices of one byte

constexpr int kOffCoef = kStage;                     // double [8][128]
constexpr int kOffAcc = kOffCoef + 8 * 128 * 8;      // double [3 kMaxAtoms]
constexpr int kOffRunV = kOffAcc + 3 * kMaxAtoms * 8;  // double [kT / 32][kCols][3]
constexpr int kOffRunAt = kOffRunV + kT / 32 * kCols * 24;  // int [kT / 32][kCols]
constexpr int kOffRunN = kOffRunAt + kT / 32 * kCols * 4;   // int [kT / 32]
constexpr int kOffAo = kOffRunN + 64;                // uint16 [kMaxM]
constexpr int kOffAtom = kOffAo + kMaxM * 2;         // uint8 [kMaxM]: atom of each local row
constexpr int kOffEg = kOffAtom + kMaxM;             // int [128]
constexpr int kOffEf = kOffEg + 128 * 4;             // int [2][64]
constexpr int kOffHost = kOffEf + 128 * 4;           // int [128]
constexpr int kOffMisc = kOffHost + 128 * 4;
constexpr int kSmem = kOffMisc + 96 + 1024;
static_assert(2 * (kSmem + 1024) <= 233472, "two CTAs share one SM's shared memory");
constexpr int kENanMark = 4096;  // stands for exponents that give NaN where two are added up

// The points' biased exponents of one plane's rows [0, m): s_e, through 256 words of the idle stage.
__device__ void point_exponents(const double* __restrict__ plane, int m, uint32_t* sc, int* s_e) {
  const int tid = threadIdx.x, g = tid & 127;
  uint32_t mx = 0;
  for (int i = tid >> 7; i < m; i += kT / 128)
    mx = max(mx, (uint32_t)__double2hiint(plane[(size_t)i * 128 + g]) & 0x7FFFFFFFu);
  sc[tid] = mx;
  __syncthreads();
  if (tid < 128) s_e[g] = (int)(max(sc[g], sc[128 + g]) >> 20);
  __syncthreads();
}

__global__ void __launch_bounds__(kT, 2) xc_grad_f64tc_kernel(DevGrid G, GradArgs A, int* __restrict__ status) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  double(*coef)[128] = reinterpret_cast<double(*)[128]>(base + kOffCoef);
  double(*dens)[4][128] = reinterpret_cast<double(*)[4][128]>(base);  // [2], the stage idle
  double(*hsum)[3][128] = reinterpret_cast<double(*)[3][128]>(base);  // [2], likewise
  double* acc = reinterpret_cast<double*>(base + kOffAcc);
  double(*run_v)[kCols][3] = reinterpret_cast<double(*)[kCols][3]>(base + kOffRunV);
  int(*run_at)[kCols] = reinterpret_cast<int(*)[kCols]>(base + kOffRunAt);
  int* run_n = reinterpret_cast<int*>(base + kOffRunN);
  uint16_t* s_ao = reinterpret_cast<uint16_t*>(base + kOffAo);
  uint8_t* s_atom = base + kOffAtom;
  int* s_eg = reinterpret_cast<int*>(base + kOffEg);
  int* s_ef = reinterpret_cast<int*>(base + kOffEf);
  int* s_host = reinterpret_cast<int*>(base + kOffHost);
  int* s_batch = reinterpret_cast<int*>(base + kOffMisc + kGemmBytes);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = tid & 127, h = tid >> 7;
  const int na3 = 3 * A.n_atoms;
  const bool fused = A.xc >= 0;
  const bool two = !fused || !A.closed;  // a force pass of its own for the beta spin
  Gemm gemm;
  gemm.begin(base, base + kOffMisc);
  bool failed = false;

  double* const slab = A.slab + (size_t)blockIdx.x * A.slab_stride;
  const size_t plane = up(A.max_m, 32) * 128;
  unsigned char* const apack = reinterpret_cast<unsigned char*>(slab + kPlanes * plane);
  const unsigned long long* const Y0 = reinterpret_cast<const unsigned long long*>(A.Pa);
  const int* const f0 = reinterpret_cast<const int*>(Y0 + 2 * G.nn_total);
  constexpr int kAdder = 96;  // threads kAdder .. + 2 add up the runs (not in the issuing warp)
  for (int k = tid; k < na3; k += kT) acc[k] = 0.0;

  while (!failed) {
    __syncthreads();
    if (tid == 0) *s_batch = atomicAdd(A.counter, 1);
    __syncthreads();
    const int q = *s_batch;
    if (q >= G.n_batches) break;
    const int b = G.order[q];
    const BatchDesc bd = G.batches[b];
    const int m = bd.m, m_k = (m + 31) / 32 * 32, n = G.n_ao;
    const bool live = g < bd.n_pts;
    const size_t pt = (size_t)bd.pt_start + g;
    for (int i = tid; i < m; i += kT) {
      const int ao = G.batch_ao[bd.ao_start + i];
      s_ao[i] = (uint16_t)ao;
      s_atom[i] = (uint8_t)A.ao_atom[ao];
    }
    if (h == 0) s_host[g] = live ? A.host[pt] : 0;
    eval_batch_hess<kT>(G, bd, slab, plane);
    __syncthreads();
    // the packed operand of a plane (phi, psi) relative to the points' largest entries
    auto pack = [&](const double* p) {
      point_exponents(p, m, reinterpret_cast<uint32_t*>(base), s_eg);
      pack_points(apack, p, s_eg, m, m_k);
      fence_proxy_async_global();  // read by bulk copies, and the stage written by them
      fence_proxy_async_smem();
      __syncthreads();
    };
    // the exponent to add to a sum of density row exponent ef
    auto exponent = [&](int eg, int ef) {
      return max((ef >= kENan ? kENanMark : ef) + (eg >= kENan ? kENanMark : eg) - 2096 + sum_shift(m), kScaleMin);
    };
    pack(slab);
    double rho[2] = {0, 0}, gx[2] = {0, 0}, gy[2] = {0, 0}, gz[2] = {0, 0};
    for (int s = 0; s < (A.closed ? 1 : 2) && !failed; ++s) {
      const int eg = s_eg[g];
      double* const tp = slab + (kTp + s) * plane;
      double sr = 0, sx = 0, sy = 0, sz = 0;
      failed = !gemm.rows(apack, Y0 + (s ? G.nn_total : 0), f0 + (s ? G.n_total : 0), s_ao, s_ef, m, n,
                          [&](int nc, const int* ef, long long (&V)[kCols]) {
#pragma unroll
        for (int j0 = 0; j0 < kCols; j0 += 4) {
          if (nc + h * kCols + j0 >= m) break;
          double p[4][4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const double* r = slab + (size_t)min(nc + h * kCols + j0 + j, m - 1) * 128 + g;
#pragma unroll
            for (int k = 0; k < 4; ++k) p[j][k] = r[k * plane];
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int i = nc + h * kCols + j0 + j;
            const double t = scaled_or_nan(V[j0 + j], exponent(eg, ef[h * kCols + j0 + j]));
            if (i < m) tp[(size_t)i * 128 + g] = t;
            sr = fma(p[j][0], t, sr);
            sx = fma(p[j][1], t, sx);
            sy = fma(p[j][2], t, sy);
            sz = fma(p[j][3], t, sz);
          }
        }
      });
      if (failed) break;
      __syncthreads();
      dens[h][0][g] = sr;
      dens[h][1][g] = sx;
      dens[h][2][g] = sy;
      dens[h][3][g] = sz;
      __syncthreads();
      rho[s] = dens[0][0][g] + dens[1][0][g];
      gx[s] = 2.0 * (dens[0][1][g] + dens[1][1][g]);
      gy[s] = 2.0 * (dens[0][2][g] + dens[1][2][g]);
      gz[s] = 2.0 * (dens[0][3][g] + dens[1][3][g]);
      fence_proxy_async_smem();
      __syncthreads();
    }
    if (failed) break;
    if (h == 0) {
#pragma unroll
      for (int k = 0; k < 8; ++k) coef[k][g] = fused || !live ? 0.0 : A.wxc[8 * pt + k];
      double fx = 0.0;
      if (fused) {
        const int o = A.closed ? 0 : 1;
        const double ra = rho[0] < 0.0 ? 0.0 : rho[0], rb = rho[o] < 0.0 ? 0.0 : rho[o];  // (NaN stays)
        if (live && !(ra + rb < 1e-18)) {
          const double gaa = gx[0] * gx[0] + gy[0] * gy[0] + gz[0] * gz[0];
          const double gab = gx[0] * gx[o] + gy[0] * gy[o] + gz[0] * gz[o];
          const double gbb = gx[o] * gx[o] + gy[o] * gy[o] + gz[o] * gz[o];
          const XcVal v = xc_eval(A.xc, ra, rb, gaa, gab, gbb);
          const double w = G.pw[pt];
          if (fabs(w) > 1e-24) {
            coef[0][g] = w * v.vra;
            coef[1][g] = w * (2.0 * v.vgaa * gx[0] + v.vgab * gx[o]);
            coef[2][g] = w * (2.0 * v.vgaa * gy[0] + v.vgab * gy[o]);
            coef[3][g] = w * (2.0 * v.vgaa * gz[0] + v.vgab * gz[o]);
            coef[4][g] = w * v.vrb;
            coef[5][g] = w * (2.0 * v.vgbb * gx[o] + v.vgab * gx[0]);
            coef[6][g] = w * (2.0 * v.vgbb * gy[o] + v.vgab * gy[0]);
            coef[7][g] = w * (2.0 * v.vgbb * gz[o] + v.vgab * gz[0]);
          }
          fx = v.f + (ra - ra) + (rb - rb);
        }
        if (live && A.fx_out) A.fx_out[pt] = fx;
      }
    }
    __syncthreads();

    const double scale = two ? -2.0 : -4.0;
    double hs[3] = {0, 0, 0};
    for (int s = 0; s < (two ? 2 : 1) && !failed; ++s) {
      const double c0 = coef[4 * s][g], u0 = coef[4 * s + 1][g], u1 = coef[4 * s + 2][g], u2 = coef[4 * s + 3][g];
      double* const psi = slab + kPsi * plane;
      for (int i = h; i < m; i += 2) {
        const double* p = slab + (size_t)i * 128 + g;
        psi[(size_t)i * 128 + g] = fma(u2, p[3 * plane], fma(u1, p[2 * plane], u0 * p[plane]));
      }
      __syncthreads();
      pack(psi);
      const int eg = s_eg[g], sp = s && !A.closed ? 1 : 0;
      const double* const tp = slab + (kTp + sp) * plane;
      failed = !gemm.rows(apack, Y0 + (sp ? G.nn_total : 0), f0 + (sp ? G.n_total : 0), s_ao, s_ef, m, n,
                          [&](int nc, const int* ef, long long (&V)[kCols]) {
        double r0 = 0, r1 = 0, r2 = 0;
        int cur = -1, runs = 0;
        auto flush = [&]() {  // the run's sum over the warp's points
          hs[0] += r0;
          hs[1] += r1;
          hs[2] += r2;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            r0 += __shfl_xor_sync(0xffffffffu, r0, o);
            r1 += __shfl_xor_sync(0xffffffffu, r1, o);
            r2 += __shfl_xor_sync(0xffffffffu, r2, o);
          }
          if (lane == 0) {
            run_v[warp][runs][0] = r0;
            run_v[warp][runs][1] = r1;
            run_v[warp][runs][2] = r2;
            run_at[warp][runs] = cur;
          }
          ++runs;
          r0 = r1 = r2 = 0.0;
        };
#pragma unroll
        for (int j = 0; j < kCols; ++j) {
          const int i = nc + h * kCols + j;
          if (i >= m) break;
          const double* p = slab + (size_t)i * 128 + g;
          const double t = tp[(size_t)i * 128 + g];
          const double d0 = p[kGrad * plane], d1 = p[(kGrad + 1) * plane], d2 = p[(kGrad + 2) * plane];
          const double hxx = p[kHess * plane], hxy = p[(kHess + 1) * plane], hxz = p[(kHess + 2) * plane],
                       hyy = p[(kHess + 3) * plane], hyz = p[(kHess + 4) * plane], hzz = p[(kHess + 5) * plane];
          const int at = s_atom[i];  // the same for the whole warp
          if (at != cur) {
            if (cur >= 0) flush();
            cur = at;
          }
          const double y = scaled_or_nan(V[j], exponent(eg, ef[h * kCols + j]));
          const double a0 = fma(u2, hxz, fma(u1, hxy, fma(u0, hxx, c0 * d0)));
          const double a1 = fma(u2, hyz, fma(u1, hyy, fma(u0, hxy, c0 * d1)));
          const double a2 = fma(u2, hzz, fma(u1, hyz, fma(u0, hxz, c0 * d2)));
          r0 = fma(a0, t, fma(d0, y, r0));
          r1 = fma(a1, t, fma(d1, y, r1));
          r2 = fma(a2, t, fma(d2, y, r2));
        }
        if (cur >= 0) flush();
        if (lane == 0) run_n[warp] = runs;
        __syncthreads();
        if (tid >= kAdder && tid < kAdder + 3) {
          const int k = tid - kAdder;
          for (int w = 0; w < kT / 32; w += 4)
            for (int r = 0; r < run_n[w]; ++r)
              acc[3 * run_at[w][r] + k] +=
                  scale * (run_v[w][r][k] + run_v[w + 1][r][k] + run_v[w + 2][r][k] + run_v[w + 3][r][k]);
        }
      });
      __syncthreads();
    }
    if (failed) break;
    // each point's total goes to its host atom with the opposite sign
#pragma unroll
    for (int k = 0; k < 3; ++k) hsum[h][k][g] = scale * hs[k];
    __syncthreads();
    if (tid >= kAdder && tid < kAdder + 3) {
      const int k = tid - kAdder;
      int cur = s_host[0];
      double run = 0.0;
      for (int p = 0; p < bd.n_pts; ++p) {
        if (s_host[p] != cur) {
          acc[3 * cur + k] -= run;
          cur = s_host[p];
          run = 0.0;
        }
        run += hsum[0][k][p] + hsum[1][k][p];
      }
      acc[3 * cur + k] -= run;
    }
    fence_proxy_async_smem();  // the stage is written by bulk copies next
    __syncthreads();
    for (int k = tid; k < na3; k += kT) {
      A.part[(size_t)b * na3 + k] = acc[k];
      acc[k] = 0.0;
    }
  }
  if (failed && tid == 0) atomicExch(status, 1);
  gemm.end(failed);
}

}  // namespace

bool grad_f64tc_fits(int max_m, int n_atoms) { return max_m <= kMaxM && n_atoms <= kMaxAtoms; }

size_t grad_f64tc_slab_doubles(int max_m) { return kPlanes * up(max_m, 32) * 128 + up(max_m, 32) / 32 * kABytes / 8; }

cudaError_t launch_xc_grad_f64tc(const DevGrid& G, const GradArgs& A, int n_ctas, int* status, cudaStream_t st) {
  const cudaError_t e = cudaFuncSetAttribute(xc_grad_f64tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  if (e != cudaSuccess) return e;
  xc_grad_f64tc_kernel<<<n_ctas, kT, kSmem, st>>>(G, A, status);
  return cudaGetLastError();
}

}  // namespace cxc
