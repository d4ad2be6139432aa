// vxc_f64tc.cu -- the FP64 XC quadrature with its contractions on the tensor cores (tcgen05).
//
// Same phases, screening and FP64 arithmetic as vxc_fp64.cu; the two contractions of a batch of m AOs
// and 128 points, T = P_sub Phi and W = Z Phi^T, run as exact integer-slice products (f64_slices.cuh)
// instead of FP64 FMAs.  Each operand vector (an AO row of P, a point's or an AO's row of Phi, an AO's
// row of Z) is cut into six 9-bit BF16 slices relative to its largest element; the 21 slice products
// i + j <= 5 go into five FP32 accumulators in TMEM (levels 0-3 exact over 64 terms, levels 4 and 5
// together), which are drained every 64 terms into 64-bit integers; rho, the functional, Z and all sums
// stay in FP64.
//
// Error, relative to the product of the two rows' largest elements and per term: 2 x 2^-53 from the operands'
// rounding, at most 20 x 2^-54 from the products left out (five of i + j = 6) and 12 x 2^-54 from the last
// accumulator's additions, so below 9 x 2^-52 in all.  Measured on whole builds, V is as far from a plain FP64
// evaluation by its largest entry as the SIMT form's.  But an FMA chain rounds relative to its own terms and this
// form relative to row maxima: an element 2^k below its row's largest keeps 53 - k bits, so that an entry of V
// between AOs that hardly meet is right to about 2^-52 of the largest products in absolute terms, not in its own
// digits.  The TD-DFT kernel's finite differences, which would turn that into 5e-12 to 4e-9 of dV, keep the SIMT
// form's densities (calchem_xc_fxc_prepare).  Rows with infinities or NaN, or of 2^957 and above, give NaN.
//
// What bounds it: GB300 has 2 FP64 FMA lanes per SM and clock, so the SIMT form spends 2 m^2 FP64 FMAs a
// point there; here the tensor cores take them and the FP64 pipe is left with ~m (4 for rho and
// grad rho, 4 for Z, 2 for the conversion of T) FMAs a point and the functional.  Two CTAs of 256
// threads share an SM (240 TMEM columns and ~109 KB of shared memory each), so that one CTA's FP64
// phases run under the other's copies and MMAs.  N = 48 columns is what five accumulators leave of
// 256 TMEM columns.
//
// Measured against the SIMT form (whole host calls, FP64): C8H18 B3LYP Fine 32.9 -> 2.38 ms, 24 waters
// B3LYP Medium 30.9 -> 2.02 ms, C6H14 PBE open shell 7.33 -> 0.77 ms, one water 0.63 -> 0.16 ms; the
// relative error of V against a plain FP64 evaluation is the same (2.6e-15 on C8H18, 2.7e-15 before).
// On C8H18 a batch takes a CTA 280 us (210 alone on its SM): 36 % in MMA rounds, whose 128 x 32-byte A
// reads bind them to shared memory (44 cycles per MMA of N = 48, 43 at N = 16), 46 % in rho, functional
// and Z on the FP64 pipe, 10 % draining accumulators, 7 % in V's reductions.  What shortened it from 2.72
// ms: A tiles reloaded one by one under the others' MMAs and B gathered under them (-4 %), MMAs issued
// from uniform registers (-3 %), rho's loads and V's reductions free of branches (-5 %).  Measured without
// effect: L2 prefetches of the operands and planes, the next Z row's loads in registers.
//
// AO values, their packed slices and exponents depend on the grid and basis only: batches with a block
// in the grid's AO cache compute them in the first launch that reaches them and read them afterwards,
// as the tensor-core form of vxc_mixed.cu does.
//
// V is accumulated as the full square sum_b Z Phi^T (transposed, so that a warp's lanes add to
// neighbouring elements) and symmetrised by launch_finish: half the MMAs of Z Phi^T + Phi Z^T on one
// triangle.  Every mbarrier wait is bounded; one that expires sets the status word, waits (bounded) for
// the CTA's own MMAs and copies, frees TMEM and returns.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "f64_gemm.cuh"
#include "f64_slices.cuh"
#include "fp64_ao.cuh"
#include "mixed_ops.cuh"
#include "tc_ptx.cuh"
#include "xc_device.cuh"

namespace cxc {

namespace {

using namespace f64s;

constexpr int kOffCoef = kABytes + 2 * kBBytes;     // double [8][128]; two B buffers before it
constexpr int kOffAo = kOffCoef + 8 * 128 * 8;      // uint16 [kMaxM]: AO (within the molecule) of each local row
constexpr int kOffEz = kOffAo + kMaxM * 2;          // uint16 [kMaxM]: biased exponents of the Z rows
constexpr int kOffEp = kOffEz + kMaxM * 2;          // uint16 [kMaxM]: of the Phi rows
constexpr int kOffEg = kOffEp + kMaxM * 2;          // int [128]: of the points
constexpr int kOffEf = kOffEg + 128 * 4;            // int [2][64]: of the chunk's density rows
constexpr int kOffRed = kOffEf + 128 * 4;           // double [3][kT / 32]
constexpr int kOffMisc = kOffRed + 3 * (kT / 32) * 8;
constexpr int kSmem = kOffMisc + 96 + 1024;
static_assert(2 * (kSmem + 1024) <= 233472, "two CTAs share one SM's shared memory");
static_assert(kLevels * kN <= (int)kTmem, "the accumulators fit the CTA's TMEM columns");
static_assert(8 * 128 * 8 <= kABytes, "the density sums live in the idle operand stage");
constexpr int kENanMark = 4096;          // and are kept as this one where two of them are added up

// A batch's block: FP64 planes [4][m_k][128], the GEMM1 operand (m_k / 32 K blocks of 48 KB), the Phi
// image (four 32-point K blocks of three tiles [m_r][128 B]), the Phi rows' exponents, the points'.
struct Block {
  size_t plane, apack, img, ep, eg, bytes;
  int m_r;
  __host__ __device__ explicit Block(int m) {
    const size_t m_k = up(m, 32);
    m_r = (int)up(m, kN);
    plane = m_k * 128;
    apack = 4 * plane * 8;
    img = apack + m_k / 32 * kABytes;
    ep = img + (size_t)12 * m_r * 128;
    eg = ep + up(4 * (size_t)m, 16);
    bytes = up(eg + 512, 1024);
  }
};

__host__ __device__ constexpr size_t z_bytes(int m) { return 12 * up(m, 128) * 128; }

// One AO row over the batch's points into an image [4 K blocks][3 tiles][m_r rows][128 B], by one warp:
// lane l holds points 4 l .. 4 l + 3.  Returns the row's exponent.
__device__ __forceinline__ int pack_row(unsigned char* __restrict__ img, int m_r, int row, const double (&x)[4]) {
  const int lane = threadIdx.x & 31;
  uint32_t mx = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) mx = max(mx, (uint32_t)__double2hiint(x[k]) & 0x7FFFFFFFu);
  mx = __reduce_max_sync(0xFFFFFFFFu, mx);
  const int E = (int)(mx >> 20);
  unsigned long long Y[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) Y[k] = to_fixed(x[k], E);
  uint32_t w0[kSlices], w1[kSlices];
  slice_pairs(Y[0], Y[1], w0);
  slice_pairs(Y[2], Y[3], w1);
  unsigned char* t = img + (size_t)(lane >> 3) * 3 * m_r * 128 + (lane & 1) * 8;
#pragma unroll
  for (int s = 0; s < kSlices; ++s)
    *reinterpret_cast<uint2*>(t + (size_t)(s >> 1) * m_r * 128 + (size_t)(row & ~7) * 128 +
                              slice_off(s, row & 7, (lane & 7) >> 1)) = make_uint2(w0[s], w1[s]);
  return E;
}

__device__ __forceinline__ void load4(const double* p, double (&x)[4]) {
  const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 2);
  x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
}

__global__ void __launch_bounds__(kT, 2) vxc_f64tc_kernel(DevGrid G, EvalArgs A) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* stage = base;
  double(*coef)[128] = reinterpret_cast<double(*)[128]>(base + kOffCoef);
  double(*dens)[4][128] = reinterpret_cast<double(*)[4][128]>(base);  // [2], the stage idle
  uint16_t* s_ao = reinterpret_cast<uint16_t*>(base + kOffAo);
  uint16_t* s_ez = reinterpret_cast<uint16_t*>(base + kOffEz);
  uint16_t* s_ep = reinterpret_cast<uint16_t*>(base + kOffEp);
  int* s_eg = reinterpret_cast<int*>(base + kOffEg);
  int* s_ef = reinterpret_cast<int*>(base + kOffEf);
  double(*red)[kT / 32] = reinterpret_cast<double(*)[kT / 32]>(base + kOffRed);
  int* s_batch = reinterpret_cast<int*>(base + kOffMisc + kGemmBytes);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = tid & 127, h = tid >> 7;
  const bool uks = A.mode == kModeUks;

  Gemm gemm;
  gemm.begin(base, base + kOffMisc);
  bool failed = false;

  unsigned char* const slab = reinterpret_cast<unsigned char*>(A.slab + (size_t)blockIdx.x * A.slab_stride);
  unsigned char* const zimg = slab;  // the Z image, then the block of a batch without a cache block
  const unsigned long long* const Y0 = reinterpret_cast<const unsigned long long*>(A.Pa);
  const int* const f0 = reinterpret_cast<const int*>(Y0 + 2 * G.nn_total);

  while (!failed) {
    if (tid == 0) *s_batch = atomicAdd(A.counter, 1);
    __syncthreads();
    const int q = *s_batch;
    __syncthreads();
    if (q >= G.n_batches) break;
    const int b = G.order[q];
    const BatchDesc bd = G.batches[b];
    const int m = bd.m, m_k = (m + 31) / 32 * 32, nkb = m_k / 32;
    const int n = mol_nao(G, bd.mol);
    const long long moff = mol_mat(G, bd.mol);
    const int roff = mol_row(G, bd.mol);
    const Block L(m);
    const int m_z = (m + 127) / 128 * 128;
    for (int i = tid; i < m; i += kT) s_ao[i] = G.batch_ao[bd.ao_start + i];
    long long off = -1;
    if (A.ao_cache) off = A.ao_cache_off[b];
    unsigned char* const blk = off >= 0 ? A.ao_cache + off : slab + z_bytes(A.max_m);
    double* const phi = reinterpret_cast<double*>(blk);
    // only this CTA writes the flag, at the end of the fill below
    const bool cached = off >= 0 && *reinterpret_cast<volatile int*>(A.ao_cache_ok + b) != 0;
    int* const blk_ep = reinterpret_cast<int*>(blk + L.ep);
    int* const blk_eg = reinterpret_cast<int*>(blk + L.eg);
    __syncthreads();
    if (cached) {
      if (h == 0) s_eg[g] = blk_eg[g];
      for (int i = tid; i < m; i += kT) s_ep[i] = (uint16_t)(blk_ep[i] >= kENan ? kENanMark : blk_ep[i]);
      __syncthreads();
    } else {
      const uint32_t vmax = eval_batch_aos<kT>(G, bd, phi, L.plane);
      uint32_t* sc = reinterpret_cast<uint32_t*>(stage);
      sc[tid] = vmax;
      __syncthreads();
      if (h == 0) {
        const int E = (int)(max(sc[g], sc[128 + g]) >> 20);
        s_eg[g] = E;
        blk_eg[g] = E;
      }
      __syncthreads();
      pack_points(blk + L.apack, phi, s_eg, m, m_k);
      for (int row = warp; row < m; row += kT / 32) {
        double x[4];
        load4(phi + (size_t)row * 128 + 4 * lane, x);
        const int E = pack_row(blk + L.img, L.m_r, row, x);
        if (lane == 0) {
          s_ep[row] = (uint16_t)(E >= kENan ? kENanMark : E);
          blk_ep[row] = E;
        }
      }
      fence_proxy_async_global();  // the packed operands are read by bulk copies, the stage written by them
      fence_proxy_async_smem();
      __syncthreads();
      if (off >= 0 && tid == 0) {
        __threadfence();
        A.ao_cache_ok[b] = 1;  // read by later launches only
      }
    }

    double rho[2] = {0, 0}, gx[2] = {0, 0}, gy[2] = {0, 0}, gz[2] = {0, 0};
    for (int s = 0; s < (A.mode == kModeAccum ? 0 : uks ? 2 : 1) && !failed; ++s) {
      const unsigned long long* Yp = Y0 + (s ? G.nn_total : 0) + moff;
      const int* fp = f0 + (s ? G.n_total : 0) + roff;
      double sr = 0, sx = 0, sy = 0, sz = 0;
      failed = !gemm.rows(blk + L.apack, Yp, fp, s_ao, s_ef, m, n, [&](int nc, const int* ef, long long (&V)[kCols]) {
        // rho = sum phi T, grad rho = 2 sum grad phi T; T = V 2^(E_f + E_g - 2096 + sh), the point's part
        // of the exponent applied to the sums
        // (columns beyond m have V = 0 and read the last row: no branches between the loads of a group)
#pragma unroll
        for (int j0 = 0; j0 < kCols; j0 += 4) {
          if (nc + h * kCols + j0 >= m) break;
          double p[4][4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const double* r = phi + (size_t)min(nc + h * kCols + j0 + j, m - 1) * 128 + g;
#pragma unroll
            for (int k = 0; k < 4; ++k) p[j][k] = r[k * L.plane];
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const double t = scaled_or_nan(V[j0 + j], ef[h * kCols + j0 + j] - 1023 + sum_shift(m));
            sr = fma(p[j][0], t, sr);
            sx = fma(p[j][1], t, sx);
            sy = fma(p[j][2], t, sy);
            sz = fma(p[j][3], t, sz);
          }
        }
      });
      if (failed) break;
      const int E = s_eg[g];
      const double seg = point_scale(E);
      __syncthreads();
      dens[h][0][g] = sr * seg;
      dens[h][1][g] = sx * seg;
      dens[h][2][g] = sy * seg;
      dens[h][3][g] = sz * seg;
      __syncthreads();
      rho[s] = dens[0][0][g] + dens[1][0][g];
      gx[s] = 2.0 * (dens[0][1][g] + dens[1][1][g]);
      gy[s] = 2.0 * (dens[0][2][g] + dens[1][2][g]);
      gz[s] = 2.0 * (dens[0][3][g] + dens[1][3][g]);
      fence_proxy_async_smem();  // the stage is written by bulk copies next
      __syncthreads();
    }
    if (failed) break;

    // the functional, one thread per point; a closed shell's exchange and VWN terms in the threads
    // h == 0, its other correlation terms in h == 1
    const bool live = g < bd.n_pts;
    const size_t pt = (size_t)bd.pt_start + g;
    double e_loc = 0, na_loc = 0, nb_loc = 0;
    if (A.mode == kModeRks) {
      XcCs part{0.0, 0.0, 0.0};
      const bool on = live && !(rho[0] < 1e-18);
      const double gam = gx[0] * gx[0] + gy[0] * gy[0] + gz[0] * gz[0];
      if (on) part = xc_eval_cs(A.xc, 0.5 * rho[0], 0.25 * gam, h ? 2 : 1);
      part.f += rho[0] - rho[0];  // (NaN where a density row holds infinities or NaN, which the functional drops)
      if (h == 1) {
        dens[1][0][g] = part.f;
        dens[1][1][g] = part.vr;
        dens[1][2][g] = part.vg;
      }
      __syncthreads();
      if (h == 0) {
        double c0 = 0, us = 0;
        if (on) {
          const double w = G.pw[pt];
          const double vr = part.vr + dens[1][1][g];
          e_loc = w * (part.f + dens[1][0][g]);
          na_loc = w * rho[0];
          us = w * (part.vg + dens[1][2][g]);
          c0 = 0.5 * w * vr;
          if (A.point_out) {
            A.point_out[2 * pt] = e_loc;
            A.point_out[2 * pt + 1] = w * vr * rho[0] + us * gam;
          }
        }
        coef[0][g] = c0;
        coef[1][g] = us * gx[0];
        coef[2][g] = us * gy[0];
        coef[3][g] = us * gz[0];
      }
    } else if (h == 0) {
#pragma unroll
      for (int k = 0; k < 8; ++k) coef[k][g] = 0.0;
      if (A.mode == kModeAccum) {
        if (live)
#pragma unroll
          for (int k = 0; k < 4; ++k) coef[k][g] = A.wv_in[4 * pt + k];
      } else if (A.mode == kModeRho) {
        if (live) {
          A.rho_out[4 * pt] = rho[0];
          A.rho_out[4 * pt + 1] = gx[0];
          A.rho_out[4 * pt + 2] = gy[0];
          A.rho_out[4 * pt + 3] = gz[0];
        }
      } else if (A.mode == kModeFxc) {
        if (live) {  // the density is the trial matrix: rho = eta, (gx, gy, gz) = xi (fxc.rs:374-645)
          const double* c = A.fxc_coef + 11 * pt;
          const double* kc = c + (A.triplet ? 7 : 3);
          const double w = G.pw[pt];
          const double sigma = c[0] * gx[0] + c[1] * gy[0] + c[2] * gz[0];
          const double dv = kc[0] * rho[0] + kc[1] * sigma;
          const double gc = kc[1] * rho[0] + kc[2] * sigma;
          coef[0][g] = 0.5 * w * dv;
          coef[1][g] = w * (kc[3] * gx[0] + gc * c[0]);
          coef[2][g] = w * (kc[3] * gy[0] + gc * c[1]);
          coef[3][g] = w * (kc[3] * gz[0] + gc * c[2]);
        }
      } else {
        const double ra = rho[0] < 0.0 ? 0.0 : rho[0], rb = rho[1] < 0.0 ? 0.0 : rho[1];  // (NaN stays)
        if (live && !(ra + rb < 1e-18)) {
          const double w = G.pw[pt];
          const double gaa = gx[0] * gx[0] + gy[0] * gy[0] + gz[0] * gz[0];
          const double gab = gx[0] * gx[1] + gy[0] * gy[1] + gz[0] * gz[1];
          const double gbb = gx[1] * gx[1] + gy[1] * gy[1] + gz[1] * gz[1];
          const XcVal o = xc_eval(A.xc, ra, rb, gaa, gab, gbb);
          e_loc = w * (o.f + (ra - ra) + (rb - rb));
          na_loc = w * ra;
          nb_loc = w * rb;
          coef[0][g] = 0.5 * w * o.vra;
          coef[1][g] = w * (2.0 * o.vgaa * gx[0] + o.vgab * gx[1]);
          coef[2][g] = w * (2.0 * o.vgaa * gy[0] + o.vgab * gy[1]);
          coef[3][g] = w * (2.0 * o.vgaa * gz[0] + o.vgab * gz[1]);
          coef[4][g] = 0.5 * w * o.vrb;
          coef[5][g] = w * (2.0 * o.vgbb * gx[1] + o.vgab * gx[0]);
          coef[6][g] = w * (2.0 * o.vgbb * gy[1] + o.vgab * gy[0]);
          coef[7][g] = w * (2.0 * o.vgbb * gz[1] + o.vgab * gz[0]);
        }
      }
    }
    if (A.mode == kModeRks || uks) {
      double v[3] = {e_loc, na_loc, nb_loc};
#pragma unroll
      for (int k = 0; k < 3; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
        if (lane == 0) red[k][warp] = v[k];
      }
    }
    __syncthreads();
    if ((A.mode == kModeRks || uks) && tid < 3) {
      double t = 0;
      for (int k = 0; k < kT / 32; ++k) t += red[tid][k];
      A.batch_red[3 * (size_t)b + tid] = t;
    }
    if (A.mode == kModeRho || A.shares_only || m == 0) {  // (m == 0: a batch that no AO reaches)
      fence_proxy_async_smem();  // the functional's halves met in the stage; the next batch's copies write it
      continue;
    }

    for (int s = 0; s < (uks ? 2 : 1) && !failed; ++s) {
      double* Vm = (s ? A.Vb : A.Va) + moff;
      if (s) __syncthreads();  // the exponents of the first spin's rows have been read
      {
        // Z = (w v_rho / 2) Phi + (w u) . grad Phi, one warp per row, four points per lane
        double c0[4], cx[4], cy[4], cz[4];
        load4(&coef[4 * s][4 * lane], c0);
        load4(&coef[4 * s + 1][4 * lane], cx);
        load4(&coef[4 * s + 2][4 * lane], cy);
        load4(&coef[4 * s + 3][4 * lane], cz);
        for (int row = warp; row < m; row += kT / 32) {
          const double* p = phi + (size_t)row * 128 + 4 * lane;
          double x[4], y[4], z[4];
          load4(p, x);
          load4(p + L.plane, y);
#pragma unroll
          for (int k = 0; k < 4; ++k) z[k] = fma(cx[k], y[k], c0[k] * x[k]);
          load4(p + 2 * L.plane, x);
          load4(p + 3 * L.plane, y);
#pragma unroll
          for (int k = 0; k < 4; ++k) z[k] = fma(cz[k], y[k], fma(cy[k], x[k], z[k]));
          const int E = pack_row(zimg, m_z, row, z);
          if (lane == 0) s_ez[row] = (uint16_t)(E >= kENan ? kENanMark : E);
        }
      }
      fence_proxy_async_global();
      fence_proxy_async_smem();
      __syncthreads();
      // operand addresses of K block kb of tile (I, J)
      auto src_a = [&](int I, int kb) { return zimg + ((size_t)kb * 3 * m_z + I) * 128; };
      auto src_b = [&](int J, int kb) { return blk + L.img + ((size_t)kb * 3 * L.m_r + J) * 128; };
      const size_t st_a = (size_t)m_z * 128, st_b = (size_t)L.m_r * 128;
      bool bad = false;
      if (gemm.issuer) {
        bad = !gemm.load_a(src_a(0, 0), st_a);
        gemm.load_b(0, src_b(0, 0), st_b);
      }
      for (int I = 0; I < m && !failed; I += 128) {
        for (int J = 0; J < m && !failed; J += kN) {
          long long V[kCols];
#pragma unroll
          for (int k = 0; k < kCols; ++k) V[k] = 0;
          const int J1 = J + kN < m ? J + kN : 0, I1 = J1 ? I : I + 128;  // the next tile
          for (int kh = 0; kh < 2; ++kh) {
            if (gemm.issuer)
              for (int kb = 2 * kh; kb < 2 * kh + 2 && !bad; ++kb) {
                const bool more = kb < 3 || I1 < m;
                const unsigned char* next = nullptr;
                if (more) {  // the other B buffer's MMAs (the K block before) are done
                  next = kb < 3 ? src_a(I, kb + 1) : src_a(I1, 0);
                  gemm.load_b((kb + 1) & 1, kb < 3 ? src_b(J, kb + 1) : src_b(J1, 0), st_b);
                }
                bad = !gemm.wait_full(3 + (kb & 1)) || !gemm.mma_round((kb & 1) == 0, kb & 1, next, st_a);
              }
            if (__syncthreads_or(bad)) { failed = true; break; }
            tc_fence_after();
            gemm.drain(V, 0);
            __syncthreads();
          }
          if (failed) break;
          // V[j][i] += W_ij = V 2^(E_z + E_p - 2096), without branches between the elements
          const int i = I + g;
          if (i < m) {
            const int ez = s_ez[i] - 2096;
            double* const col = Vm + s_ao[i];
#pragma unroll
            for (int k = 0; k < kCols; ++k) {
              if (k % 8 == 0 && J + h * kCols + k >= m) break;
              const int j = min(J + h * kCols + k, m - 1);
              const double w = scaled_or_nan(V[k], max(ez + (int)s_ep[j], kScaleMin));
              red_add_if(col + (size_t)s_ao[j] * n, w, J + h * kCols + k < m && w != 0.0);
            }
          }
        }
      }
    }
  }

  if (failed && tid == 0) atomicExch(A.counter + 2, 1);
  gemm.end(failed);
}

// One CTA per packed density row: the row's exponent and the fixed-point Y of its elements.
__global__ void __launch_bounds__(256) fixed_density_kernel(PrepareArgs A) {
  __shared__ uint32_t red[8];
  const PreparedRow r = prepared_row(A);
  const double* __restrict__ D = A.P[blockIdx.y] + r.off;
  unsigned long long* __restrict__ out = static_cast<unsigned long long*>(A.out) + blockIdx.y * A.nn + r.off;
  uint32_t mx = 0;
  for (int j = threadIdx.x; j < r.n; j += 256) mx = max(mx, (uint32_t)__double2hiint(D[j]) & 0x7FFFFFFFu);
  mx = __reduce_max_sync(0xFFFFFFFFu, mx);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 8; ++k) mx = max(mx, red[k]);
  const int E = max((int)(mx >> 20), 64);  // rows below 2^-959 count as zeros
  if (threadIdx.x == 0) A.fexp[(size_t)blockIdx.y * A.n_total + blockIdx.x] = E;
  for (int j = threadIdx.x; j < r.n; j += 256) out[j] = to_fixed(D[j], E);
  prepared_clear(A, r);
}

}  // namespace

int f64tc_max_m() { return kMaxM; }

size_t f64tc_slab_bytes(int max_m) { return z_bytes(max_m) + Block(max_m).bytes; }

size_t f64tc_cache_block_bytes(int m) { return Block(m).bytes; }

cudaError_t f64tc_set_attributes() {
  static bool attr = false;
  if (attr) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(vxc_f64tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  if (e == cudaSuccess) attr = true;
  return e;
}

cudaError_t launch_f64tc(const DevGrid& G, const EvalArgs& A, int n_ctas, cudaStream_t st) {
  if (A.max_m > kMaxM) return cudaErrorInvalidValue;
  const cudaError_t e = f64tc_set_attributes();
  if (e != cudaSuccess) return e;
  vxc_f64tc_kernel<<<n_ctas, kT, kSmem, st>>>(G, A);
  return cudaGetLastError();
}

cudaError_t launch_f64tc_prepare(const PrepareArgs& A, cudaStream_t st) {
  fixed_density_kernel<<<dim3(A.n_total, A.n_spin), 256, 0, st>>>(A);
  return cudaGetLastError();
}

}  // namespace cxc
