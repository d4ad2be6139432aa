// fp64_ao.cuh -- FP64 AO values and gradients of one batch, shared by the FP64 quadrature kernels
// (vxc_fp64.cu, vxc_f64tc.cu).
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

}  // namespace cxc
