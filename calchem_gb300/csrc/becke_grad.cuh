// becke_grad.cuh -- derivative of the Becke partition weight of one grid point with respect to the
// nuclei (grid.rs:423-584), one team of threads per point.
#pragma once

#include <cuda_runtime.h>

namespace cxc {
namespace becke {

// v limited to [-1, 1], on the integer pipe (an FP64 comparison takes as long as an FP64 FMA)
__device__ __forceinline__ double clamp_unit(double v) {
  const int hi = __double2hiint(v);
  const bool out = (hi & 0x7FFFFFFF) >= 0x3FF00000;
  return out ? __hiloint2double((hi & (int)0x80000000) | 0x3FF00000, 0) : v;
}

// Becke step s(nu) (grid.rs:129-140): three times f(x) = x (3 - x^2) / 2 = x (1 + y / 2) with y = 1 - x^2.  d is the
// product of the three y: ds/dnu = -(3/2)^3 d / 2.
__device__ __forceinline__ void step_d(double nu, double& s, double& d) {
  double x = clamp_unit(nu);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double y = fma(-x, x, 1.0);
    d = k ? d * y : y;
    x *= fma(0.5, y, 1.0);
  }
  s = fma(-0.5, x, 0.5);
}

// Row stride of the n x n tables: odd, so that lanes on consecutive rows of a table in shared memory fall into
// different banks.
__host__ __device__ __forceinline__ int becke_ld(int n) { return n | 1; }

__host__ __device__ __forceinline__ size_t becke_scratch_doubles(int n) {
  return 5 * (size_t)n + 3 * (size_t)n * becke_ld(n);
}

// Per-point pair tables of one team (n rows of becke_ld(n)), behind dist[n], cell[n] and wacc[3 n].
struct BeckeScratch {
  double* dist;  // |r - R_c|
  double* cell;  // P_c = prod_{d != c} s_cd
  double* wacc;  // [3 n] the team's weight-derivative sums
  double* s;     // s_cd (s_dc = 1 - s_cd, both stored; 1 for coincident atoms)
  double* e;     // prod_{d != c, k} s_cd at [c][k]
  double* l;     // ds_cd/dmu_cd at [c][d], c < d
  __device__ __forceinline__ void carve(double* base, int n) {
    const size_t nn = (size_t)n * becke_ld(n);
    dist = base;
    cell = dist + n;
    wacc = cell + n;
    s = wacc + 3 * n;
    e = s + nn;
    l = e + nn;
  }
};

// raw_w f dW/dR for one point by a team of kTeam threads (a warp or more; tid within it; red: 3 doubles per warp of
// scratch for more); wacc[3a + q] is owned by thread a % kTeam.  tab, rows over the pairs (c < d):
// 1 / R_cd (0 for coincident atoms), the size adjustment a_cd, 27/8 a_cd, and (R_c - R_d) / R_cd.
//   1. lanes over the unordered pairs (c < d): s_cd from mu_cd = (r_c - r_d) / R_cd and the size
//      adjustment, and its slope (grid.rs:447-476);
//   2. lanes over atoms c: the cell function P_c (factors multiplied in increasing d, as the
//      reference accumulates them) and every "product but one" prod_{d != c, k} s_cd as a prefix
//      times a suffix product -- the reference's cell[c] / s_ck, or the explicit product when
//      s_ck <= 1e-12 (grid.rs:500-515), without a division;
//   3. lanes over the pairs: with k = ds/dmu / R_cd, m = mu_cd / R_cd and d = (E_cd - E_dc) k, the pair adds
//      d to the sum that multiplies dr_c/dR_c in dZ/dR_c and d m (R_c - R_d) to the one subtracted from it,
//      and the same with the other sign for atom d; they replace the pair's s and slope (grid.rs:517-583);
//   4. lanes over atoms a != host: dZ/dR_a from the pairs' sums, dP_host/dR_a from the pair with the host;
//      the host atom gets minus the others' sum.
template <int kTeam>
__device__ void becke_point(int n, const double* __restrict__ xyz, const double* __restrict__ inv_r,
                            const double* __restrict__ tab, const int2* __restrict__ pairs, int n_pairs, int host,
                            double x, double y, double z, double pref_in, const BeckeScratch& W, int tid, double* red) {
  const int lane = tid & 31;
  auto team_sync = [] {
    if (kTeam == 32) __syncwarp();
    else __syncthreads();
  };
  for (int c = tid; c < n; c += kTeam) {
    const double dx = x - xyz[3 * c], dy = y - xyz[3 * c + 1], dz = z - xyz[3 * c + 2];
    W.dist[c] = sqrt(dx * dx + dy * dy + dz * dz);
  }
  team_sync();
  const int ld = becke_ld(n);
  for (int p = tid; p < n_pairs; p += kTeam) {
    const int c = pairs[p].x, d = pairs[p].y;
    const double inv = tab[p];
    double sv = 1.0, sc = 1.0, sl = 0.0;
    if (inv != 0.0) {
      const double mu = clamp_unit((W.dist[c] - W.dist[d]) * inv);
      step_d(fma(tab[n_pairs + p], fma(-mu, mu, 1.0), mu), sv, sl);
      sl *= fma(tab[2 * n_pairs + p], mu, -1.6875);
      sc = 1.0 - sv;
    }
    W.s[c * ld + d] = sv;
    W.s[d * ld + c] = sc;
    W.l[c * ld + d] = sl;
  }
  team_sync();
  double zl = 0.0;
  for (int c = tid; c < n; c += kTeam) {
    const double* __restrict__ sr = W.s + c * ld;
    double* __restrict__ er = W.e + c * ld;
    double pre = 1.0;
    for (int k = 0; k < n; ++k) {
      er[k] = pre;
      if (k != c) pre *= sr[k];
    }
    W.cell[c] = pre;
    if (kTeam == 32) zl += pre;
    double suf = 1.0;
    for (int k = n - 1; k >= 0; --k) {
      er[k] *= suf;
      if (k != c) suf *= sr[k];
    }
  }
  if (kTeam > 32) {
    team_sync();
    for (int c = lane; c < n; c += 32) zl += W.cell[c];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) zl += __shfl_xor_sync(0xffffffffu, zl, o);
  if (kTeam == 32) team_sync();
  const double zs = zl;  // the same in every thread
  if (zs <= 1e-30) return;
  for (int p = tid; p < n_pairs; p += kTeam) {
    const int c = pairs[p].x, d = pairs[p].y;
    const double slope = W.l[c * ld + d];
    double q = 0.0, w0 = 0.0, w1 = 0.0, w2 = 0.0;
    if ((__double2hiint(slope) & 0x7FFFFFFF) >= 0x39B40000) {  // |slope| above ~1e-30
      const double inv = tab[p];
      const double mu = clamp_unit((W.dist[c] - W.dist[d]) * inv);
      const double k = slope * inv, ec = W.e[c * ld + d], ed = W.e[d * ld + c];
      q = (ec - ed) * k;
      const double qm = q * mu;
      w0 = qm * tab[3 * n_pairs + p];
      w1 = qm * tab[4 * n_pairs + p];
      w2 = qm * tab[5 * n_pairs + p];
      if (c == host) W.e[c * ld + d] = ec * k;  // E_{host a} k of the other atom a
      if (d == host) W.e[d * ld + c] = ed * k;
    } else {
      if (c == host) W.e[c * ld + d] = 0.0;
      if (d == host) W.e[d * ld + c] = 0.0;
    }
    W.l[c * ld + d] = q;
    W.s[c * ld + d] = w0;
    W.s[d * ld + c] = w1;
    W.l[d * ld + c] = w2;
  }
  team_sync();
  const double wn = W.cell[host] / zs, pref = pref_in / zs;
  double h0 = 0, h1 = 0, h2 = 0;
  for (int a = tid; a < n; a += kTeam) {
    if (a == host) continue;
    const double ra = W.dist[a];
    if (ra < 1e-14) continue;
    const double ax = xyz[3 * a], ay = xyz[3 * a + 1], az = xyz[3 * a + 2];
    double c = 0, zz0 = 0, zz1 = 0, zz2 = 0;
    for (int b = 0; b < n; ++b) {
      if (b == a) continue;
      const int u = (b < a ? b : a) * ld + (b < a ? a : b), v = (b < a ? a : b) * ld + (b < a ? b : a);
      const int sign = b < a ? (int)0x80000000 : 0;  // the pair (b, a) counts with the other sign
      auto flip = [sign](double t) { return __hiloint2double(__double2hiint(t) ^ sign, __double2loint(t)); };
      c += flip(W.l[u]);
      zz0 -= flip(W.s[u]);
      zz1 -= flip(W.s[v]);
      zz2 -= flip(W.l[v]);
    }
    const double ir = 1.0 / ra;
    const double dr0 = -(x - ax) * ir, dr1 = -(y - ay) * ir, dr2 = -(z - az) * ir;
    // dP_host/dR_a = -E_{host a} k (dr_a - mu_ah (R_a - R_h) / R_ah^2)
    const double inv = inv_r[(size_t)a * n + host];
    const double kb = W.e[host * ld + a], m = clamp_unit((ra - W.dist[host]) * inv) * inv;
    const double ph0 = -kb * (dr0 - m * (ax - xyz[3 * host])), ph1 = -kb * (dr1 - m * (ay - xyz[3 * host + 1])),
                 ph2 = -kb * (dr2 - m * (az - xyz[3 * host + 2]));
    zz0 += c * dr0;
    zz1 += c * dr1;
    zz2 += c * dr2;
    const double w0 = pref * (ph0 - wn * zz0), w1 = pref * (ph1 - wn * zz1), w2 = pref * (ph2 - wn * zz2);
    W.wacc[3 * a] += w0;
    W.wacc[3 * a + 1] += w1;
    W.wacc[3 * a + 2] += w2;
    h0 -= w0;
    h1 -= w1;
    h2 -= w2;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    h0 += __shfl_xor_sync(0xffffffffu, h0, o);
    h1 += __shfl_xor_sync(0xffffffffu, h1, o);
    h2 += __shfl_xor_sync(0xffffffffu, h2, o);
  }
  if (kTeam == 32) {
    __syncwarp();
    if (lane == 0) {
      W.wacc[3 * host] += h0;
      W.wacc[3 * host + 1] += h1;
      W.wacc[3 * host + 2] += h2;
    }
    __syncwarp();
  } else {
    if (lane == 0) {
      red[3 * (tid >> 5)] = h0;
      red[3 * (tid >> 5) + 1] = h1;
      red[3 * (tid >> 5) + 2] = h2;
    }
    __syncthreads();
    if (tid < 3) {
      double h = 0.0;
      for (int w = 0; w < kTeam / 32; ++w) h += red[3 * w + tid];
      W.wacc[3 * host + tid] += h;
    }
  }
}

}  // namespace becke
}  // namespace cxc
