// DFT model on the tensor cores (point and Gaussian families with at most one
// spectral index or tabulated fluxes, on uniformly spaced channels).
//
// Over a uniformly spaced run the phasor of channel k = D a + n factors as
// exp(2 pi i P f_k) = H_a G_n with H_a = exp(2 pi i P D (a - a0) df) and
// G_n = exp(2 pi i P f(a0, n)), so a record's model over a grid of rows a and
// columns n is, per component, an outer product, and over the components a
// complex matrix product (rows x components) (components x columns).  A warp
// takes 16 MA rows x 8 NJ columns of one record: per component 16 MA + 8 NJ
// phasors are formed on the FP32 pipe instead of 128 MA NJ, and the products
// go to the tensor cores.  mma.sync m16n8k16 (f16 inputs, FP32 sums) takes
// both operands from registers, where the lanes form them; tcgen05.mma would
// need every operand written to shared memory per 8 components and record.
// The k dimension is (component, re / im): a register of the A fragment is one
// H_a (re, im), of the B fragments one G_n as (Gr, -Gi) (real parts of the
// model) and (Gi, Gr) (imaginary parts).
//
// FP32 accuracy from f16 inputs: each operand is split x = hi + lo, hi the
// nearest f16 and lo the f16 of the (exact) remainder, and hi hi + hi lo + lo hi
// are summed (the split of Markidis et al., "NVIDIA Tensor Core
// Programmability, Performance & Precision", 2018).  Phasors are at most 1 and
// G carries the amplitude scaled by a power of two per chunk of 32 components,
// so what is dropped is below 2^-23 of the chunk's largest amplitude.  The
// tensor cores truncate when they add, so the sums of a chunk (12 products)
// are added to FP32 totals by the lanes, and those every kMergeChunks chunks
// to compensated ones.
//
// Spectra and tapers: the exponent E(a, n) of a component's amplitude is split
// into a row part on H, a column part on G and a remainder.  For a spectral
// index alpha the remainder alpha R(a, n) is taken as alpha_t R for the chunk's
// middle index alpha_t, a factor common to the chunk (the table is ordered by
// index), and (alpha - alpha_t) R is either below the planner's bound or, in
// the kCross instances, kept to first order by one more product whose operands
// are (alpha - alpha_t) xl(a) H_a and y(n) G_n; a taper's remainder
// Q 2 D a df (f_n - f_m) is exactly of that form.
//
// What bounds it: a product issues every 8.3 cycles per scheduler and FP32
// instructions beside it add 0.65 (packed) to 0.9 cycles instead of overlapping,
// so a step of 8 components x 512 channels takes 200 cycles of products and
// about 200 of phasors, splits and prologue.  Points: 11.3, 10.8, 8.6 and 5.8 T
// evaluations/s with teams of 1024, 512, 256 and 128 channels, against 4.6 of the
// recurrence (22 GHz, 23,808 records x 512 channels x 10,000: 28.2 to 11.5 ms);
// 7.5 T with a spectral index against 4.8.  12 warps per SM at 168 registers ran
// as 16 at 128 do.
//
// Per chunk the lanes first take one component each: the split-FP32 phase, the
// accurate phasors of the steps and anchors and their first powers go to
// shared memory in the lanes' order.  T warps of one record (segments of one
// run) share that work, a chunk each.
#pragma once
#include <stdint.h>

#include "beam_common.cuh"
#include "dft_kernels.cuh"
#include "dft_tc.h"

namespace obit {

namespace {

// Exponent terms of an instance.
constexpr int kExNone = 0, kExSpec = 1, kExGauss = 2, kExBoth = 3;
constexpr int kExTab = 4;  // fluxes tabulated per coarse plane (with kExSpec)

constexpr int kEntry = 80;         // floats per table entry: 16 pairs x 4 and padding (see tc_tab)
constexpr int kEntW = 0, kEntS = 8, kEntW8 = 16, kEntExp = 17, kEntAnchor = 18;
constexpr int kMergeChunks = 16;   // chunks between additions to the compensated totals

// Table of one chunk: entry e of component pair p (components 8 (p / 4) + p % 4
// and + 4) is {re, re, im, im}; the entry stride of 320 bytes keeps the
// 128-bit reads of a quarter-warp (4 pairs x 2 entries) on distinct banks.
__host__ __device__ constexpr int tc_tab_floats(int NJ, int T) { return (kEntAnchor + NJ * T) * kEntry; }

__host__ __device__ constexpr size_t tc_smem_floats(int MA, int NJ, int T) {
  return (size_t)T * tc_tab_floats(NJ, T) + 4 * T * T + (size_t)T * 32 * MA * NJ * 8 * 2;
}

__device__ __forceinline__ f2x neg2(f2x a) { return a ^ 0x8000000080000000ull; }

// sin(2 pi y) / y and cos(2 pi y) as polynomials in y^2 for |y| <= 1/4 turn, each
// coefficient twice: minimax fits (Remez exchange on the absolute error, the
// leading coefficient held at a float), 7.4e-9 and 2.5e-10.
__constant__ float kSin2[5][2] = {{6.2831850051879883f, 6.2831850051879883f},
                                  {-41.34161819478147f, -41.34161819478147f},
                                  {81.59869857034278f, 81.59869857034278f},
                                  {-76.49729076975476f, -76.49729076975476f},
                                  {39.14351487952847f, 39.14351487952847f}};
__constant__ float kCos2[6][2] = {{1.0f, 1.0f},
                                  {-19.73920862435062f, -19.73920862435062f},
                                  {64.93935359613609f, 64.93935359613609f},
                                  {-85.45383071153066f, -85.45383071153066f},
                                  {60.14820496695489f, 60.14820496695489f},
                                  {-25.006796783287495f, -25.006796783287495f}};

__device__ __forceinline__ f2x const2(const float (&c)[2]) { return *reinterpret_cast<const f2x*>(c); }

// Two unit phasors exp(2 pi i P f) at once, f = fh + fl (each a pair): the
// split-FP32 product, the nearest integer of its high word and then the nearest
// half turn of the rest removed exactly, the low word added to what is left
// (at most 2^-27 turns of rounding), and the polynomials above.
__device__ __forceinline__ void phasors2(f2x nPh, f2x nPl, f2x Ph, f2x fh, f2x fl, f2x& c, f2x& s) {
  const f2x p = mul2(Ph, fh);
  const f2x nlo = fma2(nPh, fl, fma2(nPl, fh, fma2(nPh, fh, p)));  // minus the low word
  float p0, p1;
  up2(p, p0, p1);
  const f2x h = sub2(p, pk2(rintf(p0), rintf(p1)));
  const f2x M = pk2(6291456.0f, 6291456.0f);  // 1.5 2^22: the sum's last bit is a half turn
  const f2x t = add2(sub2(h, nlo), M);
  const f2x y = sub2(sub2(h, sub2(t, M)), nlo);
  const f2x z = mul2(y, y);
  f2x a = fma2(const2(kSin2[4]), z, const2(kSin2[3]));
  f2x b = fma2(const2(kCos2[5]), z, const2(kCos2[4]));
  a = fma2(a, z, const2(kSin2[2]));
  b = fma2(b, z, const2(kCos2[3]));
  a = fma2(a, z, const2(kSin2[1]));
  b = fma2(b, z, const2(kCos2[2]));
  a = fma2(a, z, const2(kSin2[0]));
  b = fma2(b, z, const2(kCos2[1]));
  // an odd number of half turns changes both signs
  const f2x flip = (t << 31) & 0x8000000080000000ull;
  s = mul2(a, y) ^ flip;
  c = fma2(b, z, const2(kCos2[0])) ^ flip;
}

// (re, im) -> f16 pairs hi + lo.  (volatile, as the products: the compiler keeps
// their order, in which one step's splits fill the gaps of another's products)
__device__ __forceinline__ void split16(float re, float im, uint32_t& hi, uint32_t& lo) {
  asm volatile("{\n\t.reg .f16 a, b, m;\n\t.reg .f32 lr, li;\n\t"
      "cvt.rn.f16x2.f32 %0, %3, %2;\n\t"
      "mov.b32 {a, b}, %0;\n\t"
      "mov.b16 m, 0xBC00;\n\t"  // -1
      "fma.rn.f32.f16 lr, a, m, %2;\n\t"
      "fma.rn.f32.f16 li, b, m, %3;\n\t"
      "cvt.rn.f16x2.f32 %1, li, lr;\n\t}"
      : "=&r"(hi), "=r"(lo)
      : "f"(re), "f"(im));
}

__device__ __forceinline__ uint32_t swap16(uint32_t v) { return __byte_perm(v, v, 0x1032); }
__device__ __forceinline__ uint32_t neg_im(uint32_t v) { return v ^ 0x80000000u; }
__device__ __forceinline__ uint32_t hmul2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t dup16(float x) {
  uint32_t d;
  asm("cvt.rn.f16x2.f32 %0, %1, %1;" : "=r"(d) : "f"(x));
  return d;
}

__device__ __forceinline__ void mma16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// z <- z w (packed over two components)
__device__ __forceinline__ void cmul2(f2x& zr, f2x& zi, f2x wr, f2x wi, f2x nwi) {
  const f2x nr = fma2(zr, wr, mul2(zi, nwi));
  zi = fma2(zr, wi, mul2(zi, wr));
  zr = nr;
}

__device__ __forceinline__ f2x exp2f2(f2x x) {  // packed exp
  float a, b;
  up2(x, a, b);
  return pk2(exp_fast(a), exp_fast(b));
}

// Applies one model value to the selected polarizations of a channel (the
// rules of apply_tile).
__device__ __forceinline__ void apply_channel(const KParams& p, float* v0, float sr, float si) {
  bool any = (p.op == kOpRepl);
  for (int jp = 0; jp < p.npol; jp++) any = any || (v0[jp * p.incs + 2] > 0.0f);
  if (!any) return;
  float cum = 1.0f;
  for (int jp = 0; jp < p.npol; jp++) {
    float* v = v0 + jp * p.incs;
    const float wt = v[2];
    if (wt <= 0.0f && p.op != kOpRepl) continue;
    const float fac = p.polFact[jp] * cum;
    float mr = sr * fac, mi = si * fac;
    if (p.flipMask & (1 << jp)) { const float t = mr; mr = -mi; mi = t; }
    if (p.op == kOpDiv) {
      const float a2 = mr * mr + mi * mi;
      const float dr = mr / a2, di = mi / a2;
      const float vr = v[0], vi = v[1];
      v[0] = dr * vr + di * vi;
      v[1] = dr * vi - di * vr;
      v[2] = wt * sqrtf(a2);
    } else if (p.op == kOpRepl) {
      v[0] = mr;
      v[1] = mi;
    } else {
      v[0] -= mr;
      v[1] -= mi;
    }
    if (p.cumulative) cum *= p.stokFactor;
  }
}

// Fragments of one step: rows (hi, lo and cross operands) and columns (hi, lo).
template <int MA, int NJ, bool kCross>
struct TcFrag {
  uint32_t ah[MA][4], al[MA][4], a2[kCross ? MA : 1][4];
  uint32_t h[NJ][2], l[NJ][2];
};

// The sums of one warp: totals of the chunks since the last merge, and the
// compensated (value, error) pairs in shared memory.
template <int MA, int NJ>
struct TcSums {
  f2x tot[MA][NJ][2][2];  // {column 2t, 2t + 1} at rows g and g + 8
  int chunks = 0;
  bool merged = false;
};

// Model correlation (XX, XY, YX, YY) of a beam's column group.
__host__ __device__ constexpr int tc_corr(int NJ, int j) { return NJ == 4 ? j : 3 * j; }

// One table of components (rows of p.k.cstride floats at comps), accumulated
// into S.
// kBeam: column group j is model correlation tc_corr(NJ, j) at the same eight
// channels instead of the next eight; its anchors carry the component's Jones
// coefficient for the record's antenna types ta, tc (bm: the beam's tables,
// perm: the component's index in the Jones table).
template <int MA, int NJ, int T, int EX, bool kCross, bool kBeam>
__device__ __forceinline__ void tc_pass(const TcParams& p, const TcTeamDesc& tm, const float* comps,
                                        const float* compsLo, int ncomp, int specField, float u, float v,
                                        float w, float* sTab, float2* sScale, float2* sL2,
                                        TcSums<MA, NJ>& S, const BeamKParams* bm = nullptr,
                                        const int* perm = nullptr, int ta = 0, int tc = 0) {
  static_assert(!kBeam || T == 1, "a beam's segments lie in one Jones plane each");
  constexpr bool kSpec = (EX & kExSpec) != 0, kGau = (EX & kExGauss) != 0, kTab = (EX & kExTab) != 0;
  constexpr int kTabF = tc_tab_floats(NJ, T);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const TcSeg& seg = tm.seg[warp];
  const bool mine = seg.ch0 < seg.end;
  const float* ex = p.expo + seg.expo;
  // this lane's row and column constants
  float lamR[2 * MA], xiR[2 * MA], xlR[2 * MA], xfR[2 * MA], lamC[NJ], xiC[NJ];
  uint32_t yC[NJ];
  int fieldR[kTab ? 2 * MA : 1];  // table field of the rows' plane fluxes
#pragma unroll
  for (int i = 0; i < 2 * MA; i++) {
    lamR[i] = kSpec ? ex[p.lay.lamRow + 8 * i + g] : 0.f;
    xiR[i] = kGau ? ex[p.lay.xiRow + 8 * i + g] : 0.f;
    xlR[i] = (kCross && kSpec) ? ex[p.lay.xl + 8 * i + g] : 0.f;
    xfR[i] = (kCross && kGau) ? ex[p.lay.xf + 8 * i + g] : 0.f;
    if constexpr (kTab) fieldR[i] = specField + 1 + __float_as_int(ex[p.lay.plane + 8 * i + g]);
  }
#pragma unroll
  for (int j = 0; j < NJ; j++) {
    const int n = kBeam ? g : 8 * j + g;
    lamC[j] = kSpec ? ex[p.lay.lamCol + n] : 0.f;
    xiC[j] = kGau ? ex[p.lay.xiCol + n] : 0.f;
    yC[j] = kCross ? dup16(ex[p.lay.y + n]) : 0u;
  }

  {  // power 0 of both steps: one, for every component
    float* tb = sTab + warp * kTabF + lane * 2;
    *reinterpret_cast<float2*>(tb + (kEntW + 4) * kEntry) = *reinterpret_cast<float2*>(tb + (kEntS + 4) * kEntry) =
        ((lane & 1) ^ (lane >> 4)) ? make_float2(0.f, 0.f) : make_float2(1.f, 1.f);
  }
  // the lowest squared frequency ratio of the team (a team's last segments may be empty)
  const float xiMin =
      (T > 1 && tm.seg[T - 1].ch0 < tm.seg[T - 1].end) ? fminf(tm.seg[0].xi0, tm.seg[T - 1].xi0) : tm.seg[0].xi0;
  for (int base = 0; base < ncomp; base += kTcChunk * T) {
    __syncthreads();  // the previous chunks' readers are done with the tables
    {
      // ---- one component per lane: chunk `warp` of this group of chunks ----
      const int c = base + kTcChunk * warp + lane;
      const bool have = c < ncomp;
      const float4* cp = reinterpret_cast<const float4*>(comps + (size_t)(have ? c : 0) * p.k.cstride);
      const float4 c0 = __ldg(cp);
      float A = have ? c0.x : 0.f;
      float al = 0.f, Q = 0.f;
      if constexpr (kSpec || kGau) {
        const float4 c1 = __ldg(cp + 1);
        // (a taper below e^-200 is zero in FP32 at every channel: the clamp keeps the
        // cross factors of such components finite in f16)
        if constexpr (kGau)
          Q = fmaxf(c1.x * u * u + c1.y * v * v + c1.z * u * v, -200.0f / xiMin);
        if constexpr (kSpec) al = (specField == 4) ? c1.x : c1.w;
      }
      ds P;
      if (compsLo) {  // FP64 positions
        const float4 lo = __ldg(reinterpret_cast<const float4*>(compsLo) + (have ? c : 0));
        P = ds_dot3_lo(c0.y, lo.x, u, c0.z, lo.y, v, c0.w, lo.z, w);
      } else {
        P = ds_dot3(c0.y, u, c0.z, v, c0.w, w);
      }
      // (the second half of the pairs holds {im, im, re, re}: the 32 lanes' stores
      // fall on 32 banks)
      const int half = lane >> 4;
      float* tb = sTab + warp * kTabF + ((lane >> 3) * 4 + (lane & 3)) * 4 + ((lane >> 2) & 1) + 2 * half;
      const int im0 = half ? -2 : 2;
      auto put = [&](int e, float re, float im) {
        tb[e * kEntry] = re;
        tb[e * kEntry + im0] = im;
      };
      const f2x Ph = pk2(P.hi, P.hi), nPh = neg2(Ph), nPl = pk2(-P.lo, -P.lo);
      // the row and channel steps' powers -4 .. 3 (packed; power 0 is written once)
      float s8r, s8i;  // eight channels
      {
        f2x zr, zi;
        phasors2(nPh, nPl, Ph, pk2(tm.w_hi, tm.s_hi), pk2(tm.w_lo, tm.s_lo), zr, zi);
        const f2x nzi = neg2(zi), zr2 = add2(zr, zr);
        const f2x r2 = fma2(zr, zr, mul2(zi, nzi)), i2 = mul2(zr2, zi);
        const f2x r3 = fma2(r2, zr, mul2(i2, nzi)), i3 = fma2(r2, zi, mul2(i2, zr));
        const f2x r4 = fma2(r2, r2, mul2(i2, neg2(i2))), i4 = mul2(add2(r2, r2), i2);
        float wr, wi, sr, si;
        auto both = [&](int k, f2x r, f2x i) {  // power k and, conjugated, -k
          up2(r, wr, sr);
          up2(i, wi, si);
          if (k < 4) {
            put(kEntW + 4 + k, wr, wi);
            put(kEntS + 4 + k, sr, si);
          }
          put(kEntW + 4 - k, wr, -wi);
          put(kEntS + 4 - k, sr, -si);
        };
        both(1, zr, zi);
        both(2, r2, i2);
        both(3, r3, i3);
        both(4, r4, i4);
        s8r = __fmaf_rn(sr, sr, -si * si);
        s8i = 2.0f * sr * si;
      }
      // the step of eight rows and the segments' anchors at their first group
      float ar[T], ai[T];
#pragma unroll
      for (int q = 0; q < T; q += 2) {
        f2x zr, zi;
        float x, y;
        if (q == 0) {
          phasors2(nPh, nPl, Ph, pk2(tm.w8_hi, tm.seg[0].fa_hi), pk2(tm.w8_lo, tm.seg[0].fa_lo), zr, zi);
          up2(zr, x, ar[0]);
          up2(zi, y, ai[0]);
          put(kEntW8, x, y);
        }
        if (q + 1 < T) {
          const int q2 = (q + 2 < T) ? q + 2 : q + 1;
          phasors2(nPh, nPl, Ph, pk2(tm.seg[q + 1].fa_hi, tm.seg[q2].fa_hi), pk2(tm.seg[q + 1].fa_lo, tm.seg[q2].fa_lo),
                   zr, zi);
          up2(zr, ar[q + 1], x);
          up2(zi, ai[q + 1], y);
          if (q + 2 < T) {
            ar[q2] = x;
            ai[q2] = y;
          }
        }
      }
      float at = 0.f;  // the chunk's middle index (the rows are ordered by index)
      if constexpr (kSpec) {
        const int last = min(kTcChunk, max(1, ncomp - (base + kTcChunk * warp))) - 1;
        at = 0.5f * (__shfl_sync(0xffffffffu, al, 0) + __shfl_sync(0xffffffffu, al, last));
      }
      if constexpr (kSpec || kGau) put(kEntExp, al, Q);
#pragma unroll
      for (int q = 0; q < T; q++) {
        const TcSeg& sg = tm.seg[q];
        float amp = A;
        if constexpr (kTab) {  // the rows carry the planes' fluxes; the scale is their largest
          amp = have ? 1.f : 0.f;
          A = 0.f;
          const float* sp = comps + (size_t)(have ? c : 0) * p.k.cstride + specField + 1;
          for (int pl = sg.plane0; pl <= sg.plane1; pl++) A = fmaxf(A, fabsf(__ldg(sp + pl)));
        }
        if constexpr (kSpec || kGau) {
          float e = 0.f;
          if constexpr (kSpec) e = al * sg.lam0;
          if constexpr (kGau) e = __fmaf_rn(Q, sg.xi0, e);
          amp = (kTab ? amp : A) * expf(e);
        }
        float cr[4], ci[4], big = amp;
        if constexpr (kBeam) {
          const int pc = have ? (perm ? __ldg(perm + c) : c) : 0;
          const size_t at0 = ((size_t)pc * bm->numJChan + sg.jplane) * 8, type = (size_t)bm->jonesComps * bm->numJChan * 8;
          const float4* j1 = reinterpret_cast<const float4*>(bm->jones + ta * type + at0);
          const float4* j2 = reinterpret_cast<const float4*>(bm->jones + tc * type + at0);
          const float4 a0 = __ldg(j1), a1 = __ldg(j1 + 1), b0 = __ldg(j2), b1 = __ldg(j2 + 1);
          const float J1r[4] = {a0.x, a0.z, a1.x, a1.z}, J1i[4] = {a0.y, a0.w, a1.y, a1.w};
          const float J2r[4] = {b0.x, b0.z, b1.x, b1.z}, J2i[4] = {b0.y, b0.w, b1.y, b1.w};
          beam_coeffs(*bm, J1r, J1i, J2r, J2i, cr, ci);
          float most = 0.f;
#pragma unroll
          for (int j = 0; j < NJ; j++)
            most = fmaxf(most, fmaxf(fabsf(cr[tc_corr(NJ, j)]), fabsf(ci[tc_corr(NJ, j)])));
          big = amp * most;
        }
        // the chunk's power-of-two scale: its largest amplitude goes to [1, 2)
        const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(big) & 0x7fffffffu);
        const int e2 = min(max((int)(m >> 23), 1), 253);
        const float up = __uint_as_float((uint32_t)(254 - e2) << 23);
        const float inv = __uint_as_float((uint32_t)e2 << 23);
        amp *= up;
        if constexpr (kTab) {  // the fluxes on H have a scale of their own
          const uint32_t ms = __reduce_max_sync(0xffffffffu, __float_as_uint(have ? A : 0.f));
          const int es = min(max((int)(ms >> 23), 1), 253);
          const float upS = __uint_as_float((uint32_t)(254 - es) << 23);
          if (lane == 0) sScale[T * T + warp * T + q] = make_float2(upS, __uint_as_float((uint32_t)es << 23));
        }
        if (lane == 0) sScale[warp * T + q] = make_float2(inv, at);
        float zr = amp * ar[q], zi = amp * ai[q];
#pragma unroll
        for (int j = 0; j < NJ; j++) {
          if constexpr (kBeam) {
            const float gr = cr[tc_corr(NJ, j)], gi = ci[tc_corr(NJ, j)];
            put(kEntAnchor + j, __fmaf_rn(zr, gr, -zi * gi), __fmaf_rn(zr, gi, zi * gr));
            continue;
          }
          put(kEntAnchor + q * NJ + j, zr, zi);  // the next group is eight channels on
          const float nr = __fmaf_rn(zr, s8r, -zi * s8i);
          zi = __fmaf_rn(zr, s8i, zi * s8r);
          zr = nr;
        }
      }
    }
    __syncthreads();

    for (int q = 0; q < T; q++) {
      const int nc = min(kTcChunk, ncomp - (base + kTcChunk * q));
      if (nc <= 0 || !mine) continue;
      float acc[MA][NJ][2][4];
#pragma unroll
      for (int i = 0; i < MA * NJ * 8; i++) (&acc[0][0][0][0])[i] = 0.f;
      const float2 sc = sScale[q * T + warp];
      const float at = sc.y;
      const float2 fl = kTab ? sScale[T * T + q * T + warp] : make_float2(1.f, 1.f);  // the fluxes' scale and its inverse
      const float up = fl.x;
      const int cq = base + kTcChunk * q + t;
      const float* tb = sTab + q * kTabF + t * 4;
      // ---- 4 steps of 8 components.  The fragments of the next step are formed
      // between the products of this one: stage i is a row (pair of fragment
      // registers per component) or a column group, and a group of products
      // (2 MA independent ones) follows each.
      TcFrag<MA, NJ, kCross> F[2];
      f2x E1, E2, Zr, Zi, Br, Bi, W8r, W8i;
      auto stage = [&](int ks, int i, TcFrag<MA, NJ, kCross>& f) {
        const float* te = tb + 16 * ks;
        auto entry = [&](int e, f2x& r, f2x& m) {
          const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(te + e * kEntry);
          r = (ks & 2) ? x.y : x.x;
          m = (ks & 2) ? x.x : x.y;
        };
        if (i == 0) {
          if constexpr (kSpec || kGau) entry(kEntExp, E1, E2);
          if constexpr (kSpec) E1 = sub2(E1, pk2(at, at));
          entry(kEntW + g, Br, Bi);
          entry(kEntW8, W8r, W8i);
          Zr = Br;
          Zi = Bi;
        }
        // exponent x on (zr, zi): to first order where the indices of a chunk are
        // close (the planner's bound), else exp(x)
        auto grow = [&](f2x x, f2x& zr, f2x& zi) {
          if constexpr (!kGau && !kCross) {
            zr = fma2(zr, x, zr);
            zi = fma2(zi, x, zi);
          } else {
            x = exp2f2(x);
            zr = mul2(zr, x);
            zi = mul2(zi, x);
          }
        };
        if (i < 2 * MA) {  // rows g + 8 r: MA - 1 upwards from the table's power, then below it
          const int r = (i <= MA) ? MA - 1 + i : 2 * MA - 1 - i;
          if (i > 0 && i <= MA) cmul2(Zr, Zi, W8r, W8i, neg2(W8i));
          if (i == MA + 1) {
            Zr = Br;
            Zi = Bi;
          }
          if (i > MA) cmul2(Zr, Zi, W8r, neg2(W8i), W8i);
          f2x K = 0ull;
          if constexpr (kCross) {
            if constexpr (kSpec) K = mul2(E1, pk2(xlR[r], xlR[r]));
            if constexpr (kGau) K = fma2(E2, pk2(xfR[r], xfR[r]), K);
          }
          f2x zr = Zr, zi = Zi;
          if constexpr (kTab) {
            const float* sp = comps + fieldR[kTab ? r : 0];
            const int ca = min(cq + 8 * ks, ncomp - 1), cb = min(cq + 8 * ks + 4, ncomp - 1);
            const f2x S = mul2(pk2(__ldg(sp + (size_t)ca * p.k.cstride), __ldg(sp + (size_t)cb * p.k.cstride)), pk2(up, up));
            zr = mul2(zr, S);
            zi = mul2(zi, S);
          }
          if constexpr (kSpec || kGau) {
            f2x x = 0ull;
            if constexpr (kSpec) x = mul2(E1, pk2(lamR[r], lamR[r]));
            if constexpr (kGau) x = fma2(E2, pk2(xiR[r], xiR[r]), x);
            grow(x, zr, zi);
          }
          float r0, r1, i0, i1;
          up2(zr, r0, r1);
          up2(zi, i0, i1);
          const int mi = r >> 1, h = r & 1;
          split16(r0, i0, f.ah[mi][h], f.al[mi][h]);
          split16(r1, i1, f.ah[mi][h + 2], f.al[mi][h + 2]);
          if constexpr (kCross) {
            float k0, k1;
            up2(K, k0, k1);
            f.a2[mi][h] = hmul2(f.ah[mi][h], dup16(k0));
            f.a2[mi][h + 2] = hmul2(f.ah[mi][h + 2], dup16(k1));
          }
        } else {
          const int j = i - 2 * MA;
          f2x Gr, Gi, Sr, Si;
          entry(kEntAnchor + warp * NJ + j, Gr, Gi);
          entry(kEntS + g, Sr, Si);
          cmul2(Gr, Gi, Sr, Si, neg2(Si));
          if constexpr (kSpec || kGau) {
            f2x x = 0ull;
            if constexpr (kSpec) x = mul2(E1, pk2(lamC[j], lamC[j]));
            if constexpr (kGau) x = fma2(E2, pk2(xiC[j], xiC[j]), x);
            grow(x, Gr, Gi);
          }
          float r0, r1, i0, i1;
          up2(Gr, r0, r1);
          up2(Gi, i0, i1);
          split16(r0, i0, f.h[j][0], f.l[j][0]);
          split16(r1, i1, f.h[j][1], f.l[j][1]);
        }
      };
      // product group m of a step: per column group lo hi, hi lo, (cross,) hi hi
      constexpr int kProd = kCross ? 4 : 3;
      auto products = [&](int m, const TcFrag<MA, NJ, kCross>& f) {
        const int j = m / kProd, w = m - j * kProd;
        uint32_t b0, b1;
        if (w == 1) {
          b0 = f.l[j][0];
          b1 = f.l[j][1];
        } else if (kCross && w == 2) {
          b0 = hmul2(f.h[j][0], yC[j]);
          b1 = hmul2(f.h[j][1], yC[j]);
        } else {
          b0 = f.h[j][0];
          b1 = f.h[j][1];
        }
        const uint32_t r0 = neg_im(b0), r1 = neg_im(b1), i0 = swap16(b0), i1 = swap16(b1);
#pragma unroll
        for (int mi = 0; mi < MA; mi++) {
          const uint32_t(&a)[4] = (w == 0) ? f.al[mi] : (kCross && w == 2) ? f.a2[kCross ? mi : 0] : f.ah[mi];
          mma16(acc[mi][j][0], a, r0, r1);
          mma16(acc[mi][j][1], a, i0, i1);
        }
      };
      constexpr int kStages = 2 * MA + NJ, kGroups = NJ * kProd;
#pragma unroll
      for (int i = 0; i < kStages; i++) stage(0, i, F[0]);
#pragma unroll
      for (int ks = 0; ks < 4; ks++) {
#pragma unroll
        for (int m = 0; m < kGroups; m++) {
          if (ks < 3)
#pragma unroll
            for (int i = m * kStages / kGroups; i < (m + 1) * kStages / kGroups; i++) stage(ks + 1, i, F[(ks + 1) & 1]);
          products(m, F[ks & 1]);
        }
      }
      // ---- fold: the chunk's scale and common spectral factor ----
#pragma unroll
      for (int mi = 0; mi < MA; mi++)
#pragma unroll
        for (int j = 0; j < NJ; j++) {
          const float f0 = kTab ? fl.y : 1.f;  // (two factors: their product may leave the range)
          float f[4] = {sc.x, sc.x, sc.x, sc.x};
          if constexpr (kSpec) {
            const float4 R = __ldg(reinterpret_cast<const float4*>(ex + p.lay.L) + (kBeam ? mi : mi * NJ + j) * 32 + lane);
            const float r[4] = {R.x, R.y, R.z, R.w};
#pragma unroll
            for (int e = 0; e < 4; e++) f[e] = sc.x * (kTab ? f0 * expf(at * r[e]) : expf(at * r[e]));
          }
#pragma unroll
          for (int h = 0; h < 2; h++)
#pragma unroll
            for (int x = 0; x < 2; x++)
              S.tot[mi][j][x][h] = fma2(pk2(acc[mi][j][x][2 * h], acc[mi][j][x][2 * h + 1]),
                                        pk2(f[2 * h], f[2 * h + 1]), S.tot[mi][j][x][h]);
        }
      if (++S.chunks == kMergeChunks) {  // into the compensated totals
        S.chunks = 0;
        f2x* tt = &S.tot[0][0][0][0];
#pragma unroll
        for (int e = 0; e < MA * NJ * 4; e++) {
          float x[2];
          up2(tt[e], x[0], x[1]);
#pragma unroll
          for (int h = 0; h < 2; h++) {
            float2& l = sL2[(2 * e + h) * (32 * T) + threadIdx.x];
            const float2 o = S.merged ? l : make_float2(0.f, 0.f);
            const ds s = two_sum(o.x, x[h]);
            l = make_float2(s.hi, o.y + s.lo);
          }
          tt[e] = 0ull;
        }
        S.merged = true;
      }
    }
  }
}

// kMix: a Gaussian-family model whose untapered rows come first as points
// (p.k.compsPt, p.k.ncompPt).
template <int MA, int NJ, int T, int EX, bool kCross, int kMix>
__global__ void __launch_bounds__(32 * T, 12 / T)
    dft_tc_kernel(const __grid_constant__ TcParams p) {
  extern __shared__ __align__(16) float smem[];
  float* sTab = smem;
  float2* sScale = reinterpret_cast<float2*>(sTab + T * tc_tab_floats(NJ, T));
  float2* sL2 = sScale + 2 * T * T;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const long long nItems = (long long)p.k.nvis * p.nteam;
  for (long long item = blockIdx.x; item < nItems; item += gridDim.x) {
    const int row = (int)(item / p.nteam);
    const TcTeamDesc& tm = p.teams[item - (long long)row * p.nteam];
    float* rec = p.k.vis + (size_t)(p.k.rowBase + row) * p.k.lrec;
    const float u = rec[p.k.ilocu], v = rec[p.k.ilocv], w = rec[p.k.ilocw];
    TcSums<MA, NJ> S;
#pragma unroll
    for (int i = 0; i < MA * NJ * 4; i++) (&S.tot[0][0][0][0])[i] = 0ull;
    if constexpr (kMix != 0)
      tc_pass<MA, NJ, T, kExSpec | (EX & kExTab), (kMix == 2), false>(p, tm, p.k.compsPt, nullptr, p.k.ncompPt, 4, u, v, w, sTab, sScale,
                                               sL2, S);
    tc_pass<MA, NJ, T, EX, kCross, false>(p, tm, p.k.comps, p.k.compsLo, p.k.ncomp, p.specField, u, v, w, sTab, sScale, sL2,
                                   S);
    // every warp has read u, v, w and applies its own channels
    const TcSeg& seg = tm.seg[warp];
#pragma unroll
    for (int mi = 0; mi < MA; mi++)
#pragma unroll
      for (int j = 0; j < NJ; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const int a = 16 * mi + g + 8 * (e >> 1), n = 8 * j + 2 * t + (e & 1);
          const int ch = seg.ch0 + tm.D * a + n;
          float sr, si;
          {
            float x[2], y[2];
            up2(S.tot[mi][j][0][e >> 1], x[0], x[1]);
            up2(S.tot[mi][j][1][e >> 1], y[0], y[1]);
            sr = x[e & 1];
            si = y[e & 1];
          }
          if (S.merged) {
            const int i0 = ((mi * NJ + j) * 2) * 4 + e;
            const float2 lr = sL2[i0 * (32 * T) + threadIdx.x], li = sL2[(i0 + 4) * (32 * T) + threadIdx.x];
            sr = lr.x + (lr.y + sr);
            si = li.x + (li.y + si);
          }
          if (ch < seg.end) apply_channel(p.k, rec + p.chanOff[ch], sr, si);
        }
  }
}

// Resident CTAs of a kernel across the device, its shared-memory limit raised.
inline int tc_resident(const void* fn, int threads, size_t smem, int* gridCap, std::string* err) {
  if (int rc = raise_smem_limit(fn, smem, err)) return rc;
  int perSM = 0, dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const cudaError_t ce = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, fn, threads, smem);
  if (ce != cudaSuccess || perSM < 1) {
    *err = std::string("tensor-core kernel cannot be resident: ") + cudaGetErrorString(ce);
    return 2;
  }
  *gridCap = perSM * nsm;
  return 0;
}

}  // namespace

}  // namespace obit
