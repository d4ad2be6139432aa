// fp64_ao.cuh -- FP64 AO values and gradients of one batch, and their second derivatives, shared by
// the FP64 quadrature and gradient kernels.
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"

namespace cxc {

__device__ __forceinline__ void pow_d1(double x, int l, double& p, double& d) {
  if (l == 0) { p = 1.0; d = 0.0; }
  else if (l == 1) { p = x; d = 1.0; }
  else if (l == 2) { p = x * x; d = 2.0 * x; }
  else { p = x * x * x; d = 3.0 * x * x; }
}

// AO values and gradients of the batch's candidate shells at its points into planes 0..3 (phi, d/dx,
// d/dy, d/dz) of `slab`, [row = local AO][128 points] each, `plane` doubles apart, with the reference's
// screening (ao_grid.rs:182-230).  kT threads, one point per thread of each 128.  Returns the largest
// |phi| of this thread's point as the high word of its FP64 pattern (monotonic in |phi|; infinities and
// NaN compare above every finite value).
template <int kT>
__device__ uint32_t eval_batch_aos(const DevGrid& G, const BatchDesc& bd, double* __restrict__ slab, size_t plane) {
  const int tid = threadIdx.x;
  const int g = tid & (kBlockPts - 1);
  const bool live = g < bd.n_pts;
  uint32_t vmax = 0;
  double x = 0, y = 0, z = 0;
  if (live) {
    x = G.px[bd.pt_start + g];
    y = G.py[bd.pt_start + g];
    z = G.pz[bd.pt_start + g];
  }
  for (int ci = tid >> 7; ci < bd.n_cand; ci += kT / kBlockPts) {
    const AoShellGpu sh = G.shells[G.cand_shells[bd.cand_start + ci]];
    const int loc = G.cand_loc[bd.cand_start + ci];
    double r0 = 0.0, r1 = 0.0, dx = 0, dy = 0, dz = 0;
    bool on = false;
    if (live) {
      dx = x - sh.center[0];
      dy = y - sh.center[1];
      dz = z - sh.center[2];
      const double r2 = dx * dx + dy * dy + dz * dz;
      if (!(r2 > sh.r2_cutoff)) {
        for (int p = 0; p < sh.n_prims; ++p) {
          const AoPrimGpu pr = G.prims[sh.prim_start + p];
          const double e = pr.weighted_norm * exp(-pr.exponent * r2);
          r0 += e;
          r1 -= 2.0 * pr.exponent * e;
        }
        on = !(fabs(r0) < 1e-18 && fabs(r1) < 1e-18);
      }
    }
    for (int c = 0; c < sh.n_funcs; ++c) {
      double v = 0, gx = 0, gy = 0, gz = 0;
      if (on) {
        const AoCompGpu cp = G.comps[sh.comp_start + c];
        double px, dpx, py, dpy, pz, dpz;
        pow_d1(dx, cp.lx, px, dpx);
        pow_d1(dy, cp.ly, py, dpy);
        pow_d1(dz, cp.lz, pz, dpz);
        const double mm = px * py * pz;
        v = cp.scale * mm * r0;
        gx = cp.scale * (dpx * py * pz * r0 + mm * dx * r1);
        gy = cp.scale * (px * dpy * pz * r0 + mm * dy * r1);
        gz = cp.scale * (px * py * dpz * r0 + mm * dz * r1);
        if (!(fabs(v) > 1e-16 || fabs(gx) > 1e-16 || fabs(gy) > 1e-16 || fabs(gz) > 1e-16)) v = gx = gy = gz = 0;
      }
      const size_t o = (size_t)(loc + c) * kBlockPts + g;
      vmax = max(vmax, (uint32_t)__double2hiint(v) & 0x7FFFFFFFu);
      slab[o] = v;
      slab[plane + o] = gx;
      slab[2 * plane + o] = gy;
      slab[3 * plane + o] = gz;
    }
  }
  return vmax;
}

__device__ __forceinline__ void pow012(double x, int l, double& p, double& d, double& d2) {
  if (l == 0) { p = 1.0; d = 0.0; d2 = 0.0; }
  else if (l == 1) { p = x; d = 1.0; d2 = 0.0; }
  else if (l == 2) { p = x * x; d = 2.0 * x; d2 = 2.0; }
  else { p = x * x * x; d = 3.0 * x * x; d2 = 6.0 * x; }
}

// (A) values, gradients and Hessians (xx, xy, xz, yy, yz, zz) of the batch's AOs.
template <int kT>
__device__ void eval_batch_hess(const DevGrid& G, const BatchDesc& bd, double* __restrict__ slab, size_t plane) {
  const int tid = threadIdx.x;
  const int g = tid & (kBlockPts - 1);
  const bool live = g < bd.n_pts;
  double x = 0, y = 0, z = 0;
  if (live) {
    x = G.px[bd.pt_start + g];
    y = G.py[bd.pt_start + g];
    z = G.pz[bd.pt_start + g];
  }
  for (int ci = tid >> 7; ci < bd.n_cand; ci += kT / kBlockPts) {
    const AoShellGpu sh = G.shells[G.cand_shells[bd.cand_start + ci]];
    const int loc = G.cand_loc[bd.cand_start + ci];
    double r0 = 0.0, r1 = 0.0, r2r = 0.0, dx = 0, dy = 0, dz = 0;
    bool on = false;
    if (live) {
      dx = x - sh.center[0];
      dy = y - sh.center[1];
      dz = z - sh.center[2];
      const double r2 = dx * dx + dy * dy + dz * dz;
      if (!(r2 > sh.r2_cutoff)) {
        for (int p = 0; p < sh.n_prims; ++p) {
          const AoPrimGpu pr = G.prims[sh.prim_start + p];
          const double e = pr.weighted_norm * exp(-pr.exponent * r2);
          r0 += e;
          r1 -= 2.0 * pr.exponent * e;
          r2r += 4.0 * pr.exponent * pr.exponent * e;
        }
        on = !(fabs(r0) < 1e-18 && fabs(r1) < 1e-18 && fabs(r2r) < 1e-18);
      }
    }
    for (int c = 0; c < sh.n_funcs; ++c) {
      double o[10];
#pragma unroll
      for (int k = 0; k < 10; ++k) o[k] = 0.0;
      if (on) {
        const AoCompGpu cp = G.comps[sh.comp_start + c];
        double px, dpx, d2px, py, dpy, d2py, pz, dpz, d2pz;
        pow012(dx, cp.lx, px, dpx, d2px);
        pow012(dy, cp.ly, py, dpy, d2py);
        pow012(dz, cp.lz, pz, dpz, d2pz);
        const double s = cp.scale;
        const double mm = px * py * pz;
        const double m0 = dpx * py * pz, m1 = px * dpy * pz, m2 = px * py * dpz;
        o[0] = s * mm * r0;
        o[1] = s * (m0 * r0 + mm * dx * r1);
        o[2] = s * (m1 * r0 + mm * dy * r1);
        o[3] = s * (m2 * r0 + mm * dz * r1);
        o[4] = s * (d2px * py * pz * r0 + (2.0 * m0 * dx + mm) * r1 + mm * dx * dx * r2r);
        o[5] = s * (dpx * dpy * pz * r0 + (m0 * dy + m1 * dx) * r1 + mm * dx * dy * r2r);
        o[6] = s * (dpx * py * dpz * r0 + (m0 * dz + m2 * dx) * r1 + mm * dx * dz * r2r);
        o[7] = s * (px * d2py * pz * r0 + (2.0 * m1 * dy + mm) * r1 + mm * dy * dy * r2r);
        o[8] = s * (px * dpy * dpz * r0 + (m1 * dz + m2 * dy) * r1 + mm * dy * dz * r2r);
        o[9] = s * (px * py * d2pz * r0 + (2.0 * m2 * dz + mm) * r1 + mm * dz * dz * r2r);
      }
      const size_t off = (size_t)(loc + c) * kBlockPts + g;
#pragma unroll
      for (int k = 0; k < 10; ++k) slab[k * plane + off] = o[k];
    }
  }
}

}  // namespace cxc
