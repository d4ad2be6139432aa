// becke_mixed.cu -- the Becke weight derivative of the tensor-core XC gradient, sum_g raw_w f dB/dR
// (grid.rs:423-584), as its own kernel in double-float arithmetic on the FP32 pipe.
//
// A team of threads per point (team_threads).  Per point and unordered atom pair (c, d) it holds 32 bytes, in
// shared memory up to 72 atoms and in device memory above:
//   1. lanes over pairs: s_cd, 1 - s_cd (grid.rs:129-140, 447-476) and the slope ds_cd/dmu_cd;
//   2. lanes over atoms: the cell functions P_c = prod_{d != c} s_cd, 0 where a factor is at most 1e-30;
//   3. lanes over pairs: with E_cd = P_c / s_cd and k = slope / R_cd (grid.rs:500-583),
//        q = (E_cd - E_dc) k = (P_c (1 - s_cd) - P_d s_cd) k / (s_cd (1 - s_cd))
//      and q mu_cd (R_c - R_d) / R_cd take the place of the pair's entries; a pair with a factor at most 1e-30
//      adds less than 1e-24 (its slope is below 1e-26) and is left out;
//   4. lanes over atoms: the pairs' entries summed, dr_a/dR_a applied, the host atom given minus the others' sum.
// The step's polynomial p(y) = (3 y - y^3) / 2 is iterated through t = 1 - |y|, which obeys t' = t^2 (3 - t) / 2
// exactly, so that s and 1 - s keep their relative precision when one of them is tiny, and p'(y) = 3 t (2 - t) / 2.
// 1 - |nu| comes from (1 - |mu|)(1 - a (1 + |mu|)), the sign of nu turning mu and a.
//
// Instructions bound it: 13,100 a point on octane (26 atoms; 70 % of the issue slots, 20 of 32 lanes active) while
// the sums over one point's atoms were serial, the pairs' divisions were two and the orientations branched; 6,490
// (60 %, 26.7 lanes) now.  The pair passes take two pairs per thread in packed FP32 instructions, one division
// serves both E_cd and E_dc, 1 - x takes the short sum (the operand order is known), step 4 adds with a sign
// and no thread sums alone.  The whole gradient call: octane 9.22 -> 7.18 ms, 72 atoms 32.8 -> 16.2 ms, 183 atoms
// (one warp per point with its tables in device memory before) 1051 -> 140 ms.  Packed against scalar FP32: the same
// at 26 atoms, 16.2 against 17.1 ms at 72 and 141 against 174 at 183.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "dfloat.cuh"
#include "launch.h"

namespace cxc {

namespace {

constexpr int kPts = 16;              // points of a CTA with its tables in shared memory
constexpr size_t kTableSmem = 98304;  // shared memory of a CTA: two of them per SM at the least
constexpr int kTeam = 256;            // threads per point at most
constexpr int kGlobalCtas = 608;      // CTAs with their tables in device memory,
constexpr size_t kGlobalBytes = (size_t)4 << 30;  // which take this much at most (and what the caller can spare)

// ---- two FP32 values in one register pair; every operation rounds each value to nearest ----------------
struct f2 {
  unsigned long long v;
};
__device__ __forceinline__ f2 pack(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack(f2 a, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v)); }
__device__ __forceinline__ f2 add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ f2 both(float a) { return pack(a, a); }
__device__ __forceinline__ f2 sub(f2 a, f2 b) { return fma(b, both(-1.f), a); }
__device__ __forceinline__ f2 neg(f2 a) { float x, y; unpack(a, x, y); return pack(-x, -y); }

// double-floats of two pairs at once (the operations of dfloat.cuh)
struct D2 {
  f2 hi, lo;
};
__device__ __forceinline__ D2 d2(df32 a, df32 b) { return {pack(a.hi, b.hi), pack(a.lo, b.lo)}; }
__device__ __forceinline__ void split(D2 a, df32& x, df32& y) {
  unpack(a.hi, x.hi, y.hi);
  unpack(a.lo, x.lo, y.lo);
}
__device__ __forceinline__ D2 fast_sum(f2 a, f2 b) {  // |a| >= |b|
  const f2 s = add(a, b);
  return {s, sub(b, sub(s, a))};
}
__device__ __forceinline__ D2 add(D2 a, D2 b) {
  const f2 s = add(a.hi, b.hi), bb = sub(s, a.hi);
  const f2 e = add(sub(a.hi, sub(s, bb)), sub(b.hi, bb));
  return fast_sum(s, add(e, add(a.lo, b.lo)));
}
__device__ __forceinline__ D2 sub(D2 a, D2 b) { return add(a, D2{neg(b.hi), neg(b.lo)}); }
__device__ __forceinline__ D2 mul(D2 a, D2 b) {
  const f2 p = mul(a.hi, b.hi);
  const f2 e = fma(a.hi, b.hi, neg(p));
  return fast_sum(p, fma(a.hi, b.lo, fma(a.lo, b.hi, e)));
}
// x scaled by a power of two
__device__ __forceinline__ D2 scaled(D2 a, float c) { return {mul(a.hi, both(c)), mul(a.lo, both(c))}; }
// c - x for |x| <= c
__device__ __forceinline__ D2 rest_of(float c, D2 x) {
  const f2 s = sub(both(c), x.hi);
  return fast_sum(s, sub(sub(sub(both(c), s), x.hi), x.lo));
}

__device__ __forceinline__ df32 clamp_unit(df32 v) {
  return fabsf(v.hi) >= 1.f ? df32{copysignf(1.f, v.hi), 0.f} : v;
}
__device__ __forceinline__ float turn(float v, unsigned sign) { return __uint_as_float(__float_as_uint(v) ^ sign); }

// mu of two pairs, limited to [-1, 1]
__device__ __forceinline__ void mu_of(D2 ra, D2 rb, D2 inv, df32& m0, df32& m1) {
  split(mul(sub(ra, rb), inv), m0, m1);
  m0 = clamp_unit(m0);
  m1 = clamp_unit(m1);
}

// s_cd, 1 - s_cd and ds/dmu of two pairs
__device__ __forceinline__ void step(df32 m0, df32 m1, df32 a0, df32 a1, df32* s, df32* sc, df32* slope) {
  // the sign of nu = mu + a (1 - mu^2); near zero either side of the polynomial serves
  const unsigned g0 = __float_as_uint(fmaf(a0.hi, fmaf(-m0.hi, m0.hi, 1.f), m0.hi)) & 0x80000000u;
  const unsigned g1 = __float_as_uint(fmaf(a1.hi, fmaf(-m1.hi, m1.hi, 1.f), m1.hi)) & 0x80000000u;
  const D2 mu = d2(df32{turn(m0.hi, g0), turn(m0.lo, g0)}, df32{turn(m1.hi, g1), turn(m1.lo, g1)});
  const D2 a = d2(df32{turn(a0.hi, g0), turn(a0.lo, g0)}, df32{turn(a1.hi, g1), turn(a1.lo, g1)});
  const D2 op = rest_of(1.f, D2{neg(mu.hi), neg(mu.lo)});
  D2 t = mul(rest_of(1.f, mu), rest_of(1.f, mul(a, op)));
  D2 d{};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const D2 dk = mul(t, rest_of(2.f, t));
    d = k ? mul(d, dk) : dk;
    t = scaled(mul(mul(t, t), rest_of(3.f, t)), 0.5f);
  }
  const D2 half = scaled(t, 0.5f), rest = rest_of(1.f, half);
  // ds/dnu = -(3/2)^3 d / 2, dnu/dmu = 1 - 2 a mu
  const D2 sl = mul(mul(d, D2{both(-1.6875f), both(0.f)}), rest_of(1.f, scaled(mul(a, mu), 2.f)));
  df32 h0, h1, r0, r1;
  split(half, h0, h1);
  split(rest, r0, r1);
  split(sl, slope[0], slope[1]);
  s[0] = g0 ? r0 : h0;
  sc[0] = g0 ? h0 : r0;
  s[1] = g1 ? r1 : h1;
  sc[1] = g1 ? h1 : r1;
}

// ---- a team's block ------------------------------------------------------------------------------------
// ranges that a row of n atoms is dealt in: as the threads allow, of at least four atoms
__host__ __device__ __forceinline__ int parts_of(int n, int nt) {
  const int k = nt / n < n / 4 ? nt / n : n / 4;
  return k > 1 ? k : 1;
}

// xyz[3n], dist[n], cell[n], tmp[3n], wacc[3n], ph[4n], part[4 parts n] double-floats
__host__ __device__ __forceinline__ size_t atom_bytes(int n, int nt) {
  return (8 * (size_t)n * (15 + 4 * (size_t)parts_of(n, nt)) + 15) / 16 * 16;
}
__host__ __device__ __forceinline__ size_t table_bytes(int n) { return 16 * (size_t)n * (size_t)(n - 1); }

struct Team {
  df32 *xyz, *dist, *cell, *tmp, *wacc, *ph, *part;
  float4 *t1, *t2;  // (s, 1 - s) and (slope, -), then (q, w_x, their low parts) and (w_y, w_z, their low parts)
  __device__ void carve(unsigned char* base, unsigned char* tables, int n) {
    xyz = reinterpret_cast<df32*>(base);
    dist = xyz + 3 * n;
    cell = dist + n;
    tmp = cell + n;
    wacc = tmp + 3 * n;
    ph = wacc + 3 * n;  // per atom a: E_{host a} k and mu e of the pair (a, host)
    part = ph + 4 * n;
    t1 = reinterpret_cast<float4*>(tables);
    t2 = t1 + (size_t)n * (n - 1) / 2;
  }
};

__device__ __forceinline__ int pair_id(int c, int d, int n) { return c * n - c * (c + 1) / 2 + (d - c - 1); }

template <bool kWarp>
__device__ __forceinline__ void team_sync() {
  if (kWarp) __syncwarp();
  else __syncthreads();
}

__device__ __forceinline__ df32 lane_sum(df32 v, int from) {
  for (int o = from; o > 0; o >>= 1)
    v = df_add(v, df32{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)});
  return v;
}

// One point (arguments uniform over the team).  tab: per pair, in rows of n_pairs, 1 / R_cd (0 for coincident
// atoms), a_cd and (R_c - R_d) / R_cd as double-floats.
template <bool kWarp>
__device__ void point(int n, int np, const df32* __restrict__ tab, const int2* __restrict__ pairs, int host, df32 x,
                      df32 y, df32 z, df32 pref_in, const Team& T, int tid, int nt) {
  constexpr int kUnroll = kWarp ? 1 : 4;  // one-warp teams: 16 or more per SM, each at a place of its own in the code
  const df32 zero = {0.f, 0.f}, one = {1.f, 0.f};
  for (int c = tid; c < n; c += nt) {
    const df32 dx = df_sub(x, T.xyz[3 * c]), dy = df_sub(y, T.xyz[3 * c + 1]), dz = df_sub(z, T.xyz[3 * c + 2]);
    T.dist[c] = df_sqrt(df_add(df_add(df_mul(dx, dx), df_mul(dy, dy)), df_mul(dz, dz)));
  }
  team_sync<kWarp>();
  for (int p = tid; p < np; p += 2 * nt) {
    const bool two = p + nt < np;
    const int p1 = two ? p + nt : p;
    const int2 u = pairs[p], v = pairs[p1];
    const df32 i0 = tab[p], i1 = tab[p1];
    df32 m0, m1, s[2], sc[2], sl[2];
    mu_of(d2(T.dist[u.x], T.dist[v.x]), d2(T.dist[u.y], T.dist[v.y]), d2(i0, i1), m0, m1);
    step(m0, m1, tab[np + p], tab[np + p1], s, sc, sl);
    if (i0.hi == 0.f) s[0] = sc[0] = one, sl[0] = zero;
    T.t1[p] = make_float4(s[0].hi, s[0].lo, sc[0].hi, sc[0].lo);
    T.t2[p] = make_float4(sl[0].hi, sl[0].lo, 0.f, 0.f);
    if (two) {
      if (i1.hi == 0.f) s[1] = sc[1] = one, sl[1] = zero;
      T.t1[p1] = make_float4(s[1].hi, s[1].lo, sc[1].hi, sc[1].lo);
      T.t2[p1] = make_float4(sl[1].hi, sl[1].lo, 0.f, 0.f);
    }
  }
  team_sync<kWarp>();
  // teams of more threads than atoms: each row's atoms d in `parts` ranges
  const int parts = parts_of(n, nt), span = (n + parts - 1) / parts;
  const df32* const st = reinterpret_cast<const df32*>(T.t1);  // s_cd at 2 p, 1 - s_cd at 2 p + 1
  for (int k = tid; k < parts * n; k += nt) {
    const int c = k % n, d0 = k / n * span, d1 = min(n, d0 + span);
    df32 pr = one;
    bool none = false;
    int p = d0 < c ? pair_id(d0, c, n) : pair_id(c, d0, n);  // (d0 == c: the entry before the row's first)
#pragma unroll kUnroll
    for (int d = d0; d < d1; ++d) {
      if (d != c) {
        const df32 f = st[2 * p + (d < c)];
        none |= !(f.hi > 1e-30f);
        pr = df_mul(pr, f);
      }
      p += d < c - 1 ? n - d - 2 : d == c - 1 ? pair_id(c, c, n) - p : 1;
    }
    if (none) pr = zero;
    if (parts == 1) T.cell[c] = pr;
    else T.part[k] = pr;
  }
  team_sync<kWarp>();
  if (parts > 1) {
    for (int c = tid; c < n; c += nt) {
      df32 pr = T.part[c];
      for (int q = 1; q < parts; ++q) pr = df_mul(pr, T.part[q * n + c]);
      T.cell[c] = pr;
    }
    team_sync<kWarp>();
  }
  const int lane = tid & 31;
  df32 zs = zero;
  for (int c = lane; c < n; c += 32) zs = df_add(zs, T.cell[c]);
  zs = lane_sum(zs, n > 16 ? 16 : n > 8 ? 8 : n > 4 ? 4 : 2);  // (the lanes that hold a term)
  zs = df32{__shfl_sync(0xffffffffu, zs.hi, 0), __shfl_sync(0xffffffffu, zs.lo, 0)};
  if (zs.hi <= 1e-30f) return;
  const df32 ch = T.cell[host], wn = df_div(ch, zs), pref = df_div(pref_in, zs);
  for (int a = tid; a < n; a += nt) {
    df32 kb = zero, e0 = zero, e1 = zero, e2 = zero;
    if (a != host) {
      const int c = min(a, host), d = max(a, host), p = pair_id(c, d, n);
      const df32 s = st[2 * p + (host == d)], sl = {T.t2[p].x, T.t2[p].y}, inv = tab[p];
      if (s.hi > 1e-30f && st[2 * p + (host == c)].hi > 1e-30f && inv.hi != 0.f) {
        const df32 mu = clamp_unit(df_mul(df_sub(T.dist[c], T.dist[d]), inv));
        kb = df_mul(df_div(ch, s), df_mul(sl, inv));
        e0 = df_mul(mu, tab[2 * np + p]);
        e1 = df_mul(mu, tab[3 * np + p]);
        e2 = df_mul(mu, tab[4 * np + p]);
      }
    }
    T.ph[4 * a] = kb;
    T.ph[4 * a + 1] = e0;
    T.ph[4 * a + 2] = e1;
    T.ph[4 * a + 3] = e2;
  }
  team_sync<kWarp>();
  for (int p = tid; p < np; p += 2 * nt) {
    const bool two = p + nt < np;
    const int p1 = two ? p + nt : p;
    const int2 u = pairs[p], v = pairs[p1];
    const float4 a0 = T.t1[p], a1 = T.t1[p1];
    const float2 l0 = *reinterpret_cast<const float2*>(T.t2 + p), l1 = *reinterpret_cast<const float2*>(T.t2 + p1);
    const bool on0 = fminf(a0.x, a0.z) > 1e-30f, on1 = fminf(a1.x, a1.z) > 1e-30f;
    const D2 s = {pack(a0.x, a1.x), pack(a0.y, a1.y)}, sc = {pack(a0.z, a1.z), pack(a0.w, a1.w)};
    const D2 sl = {pack(l0.x, l1.x), pack(l0.y, l1.y)}, inv = d2(tab[p], tab[p1]);
    const D2 diff = sub(mul(d2(T.cell[u.x], T.cell[v.x]), sc), mul(d2(T.cell[u.y], T.cell[v.y]), s));
    // k / (s (1 - s)): an approximate quotient and its correction from the exact remainder
    const D2 num = mul(sl, inv), den = mul(s, sc);
    float y0, y1;
    unpack(den.hi, y0, y1);
    const f2 rc = pack(on0 ? __fdividef(1.f, y0) : 0.f, on1 ? __fdividef(1.f, y1) : 0.f);
    const f2 q1 = mul(num.hi, rc), nq = neg(q1);
    const D2 ratio = fast_sum(q1, mul(fma(nq, den.lo, add(fma(nq, den.hi, num.hi), num.lo)), rc));
    df32 m0, m1;
    mu_of(d2(T.dist[u.x], T.dist[v.x]), d2(T.dist[u.y], T.dist[v.y]), inv, m0, m1);
    const D2 q = mul(diff, ratio), qm = mul(q, d2(m0, m1));
    const D2 w0 = mul(qm, d2(tab[2 * np + p], tab[2 * np + p1])), w1 = mul(qm, d2(tab[3 * np + p], tab[3 * np + p1])),
             w2 = mul(qm, d2(tab[4 * np + p], tab[4 * np + p1]));
    df32 q0, qq, x0, x1, z0, z1, v0, v1;
    split(q, q0, qq);
    split(w0, x0, x1);
    split(w1, z0, z1);
    split(w2, v0, v1);
    T.t1[p] = make_float4(q0.hi, x0.hi, q0.lo, x0.lo);
    T.t2[p] = make_float4(z0.hi, v0.hi, z0.lo, v0.lo);
    if (two) {
      T.t1[p1] = make_float4(qq.hi, x1.hi, qq.lo, x1.lo);
      T.t2[p1] = make_float4(z1.hi, v1.hi, z1.lo, v1.lo);
    }
  }
  team_sync<kWarp>();
  // sums over b of the pairs (a, b), with the other sign where b < a: the high parts by error-free sums whose
  // errors collect with the low parts
  for (int k = tid; k < parts * n; k += nt) {
    const int a = k % n, b0 = k / n * span, b1 = min(n, b0 + span);
    f2 h0 = both(0.f), h1 = h0, c0 = h0, c1 = h0;
    int p = b0 < a ? pair_id(b0, a, n) : pair_id(a, b0, n);
#pragma unroll kUnroll
    for (int b = b0; b < b1; ++b) {
      if (b != a) {
        const f2 sg = both(b < a ? -1.f : 1.f);
        const float4 v = T.t1[p], w = T.t2[p];
        auto put = [&](f2& h, f2& c, f2 hi, f2 lo) {
          const f2 s = fma(hi, sg, h), bb = sub(s, h);
          const f2 e = add(sub(h, sub(s, bb)), fma(hi, sg, neg(bb)));
          c = fma(lo, sg, add(c, e));
          h = s;
        };
        put(h0, c0, pack(v.x, v.y), pack(v.z, v.w));
        put(h1, c1, pack(w.x, w.y), pack(w.z, w.w));
      }
      p += b < a - 1 ? n - b - 2 : b == a - 1 ? pair_id(a, a, n) - p : 1;
    }
    const D2 r0 = fast_sum(h0, c0), r1 = fast_sum(h1, c1);
    split(r0, T.part[4 * k], T.part[4 * k + 1]);
    split(r1, T.part[4 * k + 2], T.part[4 * k + 3]);
  }
  team_sync<kWarp>();
  for (int a = tid; a < n; a += nt) {
    df32 t0 = zero, t1 = zero, t2 = zero;
    const df32 dra = T.dist[a];
    if (a != host && dra.hi >= 1e-14f) {
      df32 cs = T.part[4 * a], w0 = T.part[4 * a + 1], w1 = T.part[4 * a + 2], w2 = T.part[4 * a + 3];
      for (int q = 1; q < parts; ++q) {
        const df32* r = T.part + 4 * (q * n + a);
        cs = df_add(cs, r[0]);
        w0 = df_add(w0, r[1]);
        w1 = df_add(w1, r[2]);
        w2 = df_add(w2, r[3]);
      }
      const df32 ir = df_div(one, dra);
      const df32 dr0 = df_mul(df_sub(T.xyz[3 * a], x), ir);
      const df32 dr1 = df_mul(df_sub(T.xyz[3 * a + 1], y), ir);
      const df32 dr2 = df_mul(df_sub(T.xyz[3 * a + 2], z), ir);
      const df32 z0 = df_sub(df_mul(dr0, cs), w0), z1 = df_sub(df_mul(dr1, cs), w1), z2 = df_sub(df_mul(dr2, cs), w2);
      // dP_host/dR_a = -E_{host a} k (dr_a - mu e); mu and e both turn with the pair's orientation
      const df32 kb = T.ph[4 * a];
      const df32 p0 = df_mul(kb, df_sub(T.ph[4 * a + 1], dr0)), p1 = df_mul(kb, df_sub(T.ph[4 * a + 2], dr1)),
                 p2 = df_mul(kb, df_sub(T.ph[4 * a + 3], dr2));
      t0 = df_mul(pref, df_sub(p0, df_mul(wn, z0)));
      t1 = df_mul(pref, df_sub(p1, df_mul(wn, z1)));
      t2 = df_mul(pref, df_sub(p2, df_mul(wn, z2)));
      T.wacc[3 * a] = df_add(T.wacc[3 * a], t0);
      T.wacc[3 * a + 1] = df_add(T.wacc[3 * a + 1], t1);
      T.wacc[3 * a + 2] = df_add(T.wacc[3 * a + 2], t2);
    }
    T.tmp[3 * a] = t0;
    T.tmp[3 * a + 1] = t1;
    T.tmp[3 * a + 2] = t2;
  }
  team_sync<kWarp>();
  if (tid < 32) {  // eight lanes per component (the last eight repeat the third)
    const int q = min(tid >> 3, 2);
    df32 h = zero;
    for (int a = tid & 7; a < n; a += 8) h = df_sub(h, T.tmp[3 * a + q]);  // (the host's own is zero)
    h = lane_sum(h, 4);
    if ((tid & 7) == 0 && tid < 24) T.wacc[3 * host + q] = df_add(T.wacc[3 * host + q], h);
  }
}

template <bool kWarp>
__global__ void __launch_bounds__(kWarp ? 32 : kTeam)
    becke_mixed_kernel(DevGrid G, GradArgs A, const double* __restrict__ fx, double* __restrict__ part,
                       unsigned char* tables, int pts) {
  extern __shared__ __align__(16) unsigned char bsm[];
  const int n = A.n_atoms, na3 = 3 * n;
  const int tid = threadIdx.x, nt = blockDim.x;
  Team T;
  T.carve(bsm, tables ? tables + (size_t)blockIdx.x * table_bytes(n) : bsm + atom_bytes(n, nt), n);
  for (int k = tid; k < na3; k += nt) {
    T.xyz[k] = df_from_double(A.xyz[k]);
    T.wacc[k] = df32{0.f, 0.f};
  }
  team_sync<kWarp>();
  const int p0 = blockIdx.x * pts;
  for (int p = p0; p < min(p0 + pts, G.n_pts); ++p) {
    const double f = fx[p], rw = A.raw_w[p];
    if (fabs(f) < 1e-18 || rw == 0.0) continue;
    point<kWarp>(n, A.n_pairs, reinterpret_cast<const df32*>(A.pair_df), A.pairs, A.host[p], df_from_double(G.px[p]),
                 df_from_double(G.py[p]), df_from_double(G.pz[p]), df_from_double(rw * f), T, tid, nt);
  }
  team_sync<kWarp>();
  double* out = part + (size_t)blockIdx.x * na3;
  for (int k = tid; k < na3; k += nt) out[k] = df_to_double(T.wacc[k]);
}

// Threads per point: one warp while it has a lane per atom and shared memory holds 16 points per SM or so (26
// atoms: 7.5 ms a call against 7.9 with two warps), then two (36 atoms: 3.4 against 4.0 ms with one), and eight from
// where a point's tables leave few points per SM (42 atoms: 4.64 against 4.79 ms with two, 72: 16.2 against 31;
// sixteen 22).
int team_threads(int n) { return n <= 32 ? 32 : n <= 40 ? 64 : kTeam; }
bool in_smem(int n) { return atom_bytes(n, team_threads(n)) + table_bytes(n) <= kTableSmem; }

}  // namespace

int becke_mixed_ctas(int n_pts, int n_atoms, size_t budget) {
  if (in_smem(n_atoms)) return (n_pts + kPts - 1) / kPts;
  return (int)std::max<size_t>(
      1, std::min<size_t>({(size_t)n_pts, (size_t)kGlobalCtas, std::min(kGlobalBytes, budget) / table_bytes(n_atoms)}));
}

size_t becke_mixed_table_doubles(int n_ctas, int n_atoms) {
  return in_smem(n_atoms) ? 0 : (size_t)n_ctas * table_bytes(n_atoms) / sizeof(double);
}

cudaError_t launch_becke_mixed(const DevGrid& G, const GradArgs& A, const double* fx, double* part, double* tables,
                               int n_ctas, cudaStream_t st) {
  const int n = A.n_atoms, nt = team_threads(n);
  const bool shared = in_smem(n);
  const size_t smem = atom_bytes(n, nt) + (shared ? table_bytes(n) : 0);
  auto* kernel = nt == 32 ? becke_mixed_kernel<true> : becke_mixed_kernel<false>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  kernel<<<n_ctas, nt, smem, st>>>(G, A, fx, part, shared ? nullptr : reinterpret_cast<unsigned char*>(tables),
                                   (G.n_pts + n_ctas - 1) / n_ctas);
  return cudaGetLastError();
}

}  // namespace cxc
