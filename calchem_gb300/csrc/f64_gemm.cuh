// f64_gemm.cuh -- the tensor-core contractions of the FP64 forms (vxc_f64tc.cu, xc_grad_f64tc.cu): operands as
// exact integer slices (f64_slices.cuh), 21 slice products into five FP32 accumulators, 64-bit sums.
//
// A CTA of 256 threads, two per SM: 240 of its 256 TMEM columns hold the accumulators of a 128 x 48 tile; the
// operand stage is one K block (32) of the 128-row operand A (three 16 KB tiles of 128-byte rows, two
// slices each) and two buffers of the 48-row operand B (18 KB each).
#pragma once

#include <cuda_runtime.h>

#include "f64_slices.cuh"
#include "mixed_ops.cuh"
#include "tc_ptx.cuh"

namespace cxc {
namespace f64s {

using mix::st_shared_v4;
using mix::sw128;

constexpr int kT = 256;                       // threads per CTA, two CTAs per SM
constexpr int kN = 48;                        // AO columns per accumulator
constexpr int kCols = kN / 2;                 // columns per thread (two thread groups of 128)
constexpr int kLevels = 5;
constexpr uint32_t kTmem = 256;
constexpr int kTiles = kSlices / 2;           // 128-byte rows hold two slices of 32 K values
constexpr int kABytes = kTiles * 128 * 128;   // one K block (32) of a 128-row operand
constexpr int kBTile = kN * 128;
constexpr int kBBytes = kTiles * kBTile;
constexpr int kMaxM = 2048;
constexpr uint32_t kSpin = 1u << 26;
constexpr int kStage = kABytes + 2 * kBBytes;  // bytes of the operand stage
constexpr int kGemmBytes = 72;                 // barriers and the TMEM slot, in shared memory
constexpr int kENan = kScaleNan + 1023;        // biased exponents from here on give NaN

__host__ __device__ constexpr size_t up(size_t x, size_t k) { return (x + k - 1) / k * k; }

// Contractions longer than 1024 terms drop the lowest bit of each K group's sum, to stay within 64 bits.
__device__ __forceinline__ int sum_shift(int m) { return m > 1024 ? 1 : 0; }

// 2^(E - 1073): what is left of a point's exponent after its products were scaled by 2^(E_f - 1023).
__device__ __forceinline__ double point_scale(int E) {
  return E >= kENan ? __longlong_as_double(0x7FF8000000000000ll) : (E > 51 ? __hiloint2double((E - 50) << 20, 0) : 0.0);
}

// Byte offset of slice s (even element pair words) for chunk c (8 K values) of row r in a K block's tiles.
__device__ __forceinline__ uint32_t slice_off(int s, int r, int c) { return sw128(r, (s & 1) * 4 + c); }

// Slices of 8 consecutive K values (Y[8]) stored as six 16-byte chunks: tile s >> 1 at base + (s >> 1) * tile.
template <typename Store>
__device__ __forceinline__ void store8(const unsigned long long (&Y)[8], int r, int c, Store&& store) {
  uint32_t w[4][kSlices];
#pragma unroll
  for (int k = 0; k < 4; ++k) slice_pairs(Y[2 * k], Y[2 * k + 1], w[k]);
#pragma unroll
  for (int s = 0; s < kSlices; ++s) store(s >> 1, slice_off(s, r, c), make_uint4(w[0][s], w[1][s], w[2][s], w[3][s]));
}

// The GEMM1 A operand: Phi[g][mu] for 128 points, K = AOs, relative to each point's exponent.
static __device__ void pack_points(unsigned char* __restrict__ apack, const double* __restrict__ phi, const int* s_eg, int m,
                            int m_k) {
  for (int e = threadIdx.x; e < m_k / 8 * 128; e += kT) {
    const int g = e & 127, c8 = e >> 7;
    const int E = s_eg[g];
    unsigned long long Y[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int mu = 8 * c8 + k;
      Y[k] = mu < m ? to_fixed(phi[(size_t)mu * 128 + g], E) : kBias;
    }
    unsigned char* t = apack + (size_t)(c8 >> 2) * kABytes;
    store8(Y, g, c8 & 3, [&](int tile, uint32_t off, uint4 v) {
      *reinterpret_cast<uint4*>(t + tile * 16384 + off) = v;
    });
  }
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}

// One thread of warp 0 copies the operands and issues the MMAs.  An A tile (two slices) is copied again as
// soon as the MMAs reading it are done, so that the next K block's tiles arrive under the MMAs of the others.
// The phases, the tiles whose release has not been waited for and the copies not waited for (bits 0-2 A
// tiles, 3-4 B buffers) are that thread's.
struct Gemm {
  uint64_t *full, *empty, *full_b;  // [3] A tile t has arrived, [3] the MMAs reading it are done, [2] B buffer
  uint32_t tmem, tl, sb;            // TMEM base, this thread's first column, the stage
  bool issuer;
  uint64_t pol_keep;
  uint32_t ph_full = 0, ph_empty = 0, pend = 0, inflight = 0;

  // By the whole CTA: stage 1 KB-aligned, misc kGemmBytes of shared memory.
  __device__ __forceinline__ void begin(unsigned char* stage, unsigned char* misc) {
    const int warp = threadIdx.x >> 5;
    full = reinterpret_cast<uint64_t*>(misc);
    empty = full + 3;
    full_b = full + 6;
    uint32_t* slot = reinterpret_cast<uint32_t*>(misc + 64);
    if (threadIdx.x == 0) {
      for (int k = 0; k < 8; ++k) mbar_init(full + k, 1);
      fence_mbar_init();
    }
    if (warp == 0) {
      tmem_alloc(slot, kTmem);
      tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    tmem = warp_uniform(*slot);
    tl = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)((threadIdx.x >> 7) * kCols);
    sb = warp_uniform(smem_addr(stage));
    issuer = warp_uniform(warp) == 0 && elect_one();
    pol_keep = l2_policy_evict_last();  // operands are read again per column chunk
  }
  // By the whole CTA, after its last contraction or a failed one (which waits, bounded, for what is in flight).
  __device__ __forceinline__ void end(bool failed) {
    if (failed && issuer) {
      for (int k = 0; k < 5; ++k)
        if (inflight >> k & 1u) wait_full(k);
      for (int t = 0; t < kTiles; ++t) wait_empty(t);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x < 32) tmem_dealloc(tmem, kTmem);
  }
  __device__ __forceinline__ bool wait_full(int k) {  // k: 0-2 A tiles, 3-4 B buffers
    uint64_t* bar = k < 3 ? full + k : full_b + (k - 3);
    if (!mbar_wait_bounded(bar, (ph_full >> k) & 1u, kSpin)) return false;
    ph_full ^= 1u << k;
    inflight &= ~(1u << k);
    return true;
  }
  __device__ __forceinline__ bool wait_empty(int t) {
    if (!(pend >> t & 1u)) return true;
    if (!mbar_wait_bounded(empty + t, (ph_empty >> t) & 1u, kSpin)) return false;
    ph_empty ^= 1u << t;
    pend &= ~(1u << t);
    return true;
  }
  __device__ __forceinline__ bool load_a(const unsigned char* src, size_t tile_stride) {  // the three tiles of a K block
#pragma unroll
    for (int t = 0; t < kTiles; ++t) {
      if (!wait_empty(t)) return false;
      mbar_arrive_expect_tx(full + t, 16384);
      bulk_g2s_hint(sb + t * 16384, src + t * tile_stride, 16384, full + t, pol_keep);
      inflight |= 1u << t;
    }
    return true;
  }
  __device__ __forceinline__ void load_b(int buf, const unsigned char* src, size_t tile_stride) {
    mbar_arrive_expect_tx(full_b + buf, kBBytes);
#pragma unroll
    for (int t = 0; t < kTiles; ++t)
      bulk_g2s_hint(sb + kABytes + buf * kBBytes + t * kBTile, src + t * tile_stride, kBTile, full_b + buf, pol_keep);
    inflight |= 8u << buf;
  }
  // One K block of 32 against B buffer buf: slice products i + j <= 5, level min(i + j, 4) into accumulator
  // columns 48 level; then the next K block's A copies (next != nullptr).  Returns with the MMAs done.
  __device__ __forceinline__ bool mma_round(bool first, int buf, const unsigned char* next, size_t tile_stride) {
    tc_fence_after();
    const uint32_t idesc = idesc_bf16_f32(128, kN);
    const uint64_t db = sdesc_sw128(sb + kABytes) + (uint32_t)buf * (kBBytes >> 4);
#pragma unroll
    for (int t = 0; t < kTiles; ++t) {
      if (!wait_full(t)) return false;
      const uint64_t a = sdesc_sw128(sb) + t * 1024;
#pragma unroll
      for (int ks = 0; ks < 2; ++ks)
#pragma unroll
        for (int i = 2 * t; i < 2 * t + 2; ++i)
#pragma unroll
          for (int j = 0; i + j < kSlices; ++j) {
            const int lev = i + j < kLevels ? i + j : kLevels - 1;
            // each level's first product (i = 0, levels 0..4) overwrites at the start of a K group
            const uint32_t acc = (first && ks == 0 && i == 0 && j < kLevels) ? 0u : 1u;
            mma_bf16_ss(tmem + lev * kN, a + (i & 1) * 4 + ks * 2,
                        db + (j >> 1) * (kBTile >> 4) + (j & 1) * 4 + ks * 2, idesc, acc);
          }
      mma_commit(empty + t);
      pend |= 1u << t;
    }
    if (next) {
      if (!load_a(next, tile_stride)) return false;
    } else {
#pragma unroll
      for (int t = 0; t < kTiles; ++t)
        if (!wait_empty(t)) return false;
    }
    tc_fence_before();
    return true;
  }
  // The accumulators' K group into the thread's 64-bit sums.
  __device__ __forceinline__ void drain(long long (&V)[kCols], int sh) {
#pragma unroll
    for (int c = 0; c < kCols; c += 8) {
      uint32_t r[kLevels][8];
#pragma unroll
      for (int l = 0; l < kLevels; ++l) tmem_ld8(tl + l * kN + c, r[l]);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int l = 0; l < kLevels; ++l)  // the loads' results are read after the wait
#pragma unroll
        for (int k = 0; k < 8; ++k) asm volatile("" : "+r"(r[l][k]));
#pragma unroll
      for (int k = 0; k < 8; ++k)
        V[c + k] += level_sum(__uint_as_float(r[0][k]), __uint_as_float(r[1][k]), __uint_as_float(r[2][k]),
                              __uint_as_float(r[3][k]), __uint_as_float(r[4][k])) >> sh;
    }
    tc_fence_before();
  }
  // T = P Phi^T for one batch, 48 rows of P (AOs) at a time: apack the 128-point operand (pack_points), Yp and fp
  // the fixed-point density and its rows' exponents, gathered through the AO list s_ao (warps 2-7, under the
  // MMAs of the K block before).  s_ef: int [2][64].  epi(nc, ef, V): the thread's 24 sums of chunk nc; row
  // nc + 24 h + j at point g is V[j] 2^(ef[24 h + j] + E_g - 2096 + sum_shift(m)).  False: a wait expired.
  template <typename Epi>
  __device__ __forceinline__ bool rows(const unsigned char* apack, const unsigned long long* __restrict__ Yp,
                                       const int* __restrict__ fp, const uint16_t* s_ao, int* s_ef, int m, int n, Epi&& epi) {
    if (m == 0) return true;  // no chunk would wait for the first copies
    const int tid = threadIdx.x, nkb = (m + 31) / 32, sh = sum_shift(m);
    auto gather = [&](int nc, int kb, int buf) {
      const int r = (tid - 64) >> 2, c = tid & 3;
      const int k0 = kb * 32 + c * 8;
      unsigned long long Y[8];
      const unsigned long long* row = Yp + (nc + r < m ? (size_t)s_ao[nc + r] * n : 0);
#pragma unroll
      for (int k = 0; k < 8; ++k) Y[k] = (nc + r < m && k0 + k < m) ? __ldg(row + s_ao[k0 + k]) : kBias;
      const uint32_t o = sb + kABytes + buf * kBBytes;
      store8(Y, r, c, [&](int tile, uint32_t off, uint4 v) { st_shared_v4(o + tile * kBTile + off, v); });
      fence_proxy_async_smem();
    };
    int buf = 0;
    bool bad = false;
    if (issuer) bad = !load_a(apack, 16384);
    if (tid >= 64) gather(0, 0, 0);
    __syncthreads();
    for (int nc = 0; nc < m; nc += kN) {
      // (double-buffered: slower threads may still read the previous chunk's)
      int* const ef = s_ef + (nc / kN & 1) * 64;
      if (tid < kN) ef[tid] = nc + tid < m ? fp[s_ao[nc + tid]] : 0;
      long long V[kCols];
#pragma unroll
      for (int k = 0; k < kCols; ++k) V[k] = 0;
      for (int kb = 0; kb < nkb; ++kb, buf ^= 1) {
        const bool last_k = kb == nkb - 1;
        const bool more = !last_k || nc + kN < m;
        const int kb1 = last_k ? 0 : kb + 1;
        if (issuer)
          bad = bad || !mma_round((kb & 1) == 0, buf, more ? apack + (size_t)kb1 * kABytes : nullptr, 16384);
        else if (tid >= 64 && more)
          gather(last_k ? nc + kN : nc, kb1, buf ^ 1);
        if (__syncthreads_or(bad)) return false;
        if ((kb & 1) || last_k) {
          tc_fence_after();
          drain(V, sh);
          __syncthreads();
        }
      }
      epi(nc, ef, V);
    }
    return true;
  }
};

}  // namespace f64s
}  // namespace cxc
