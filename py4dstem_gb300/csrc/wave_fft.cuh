// 2D transforms of one wave held in shared memory, two samples to a register
// pair, for square waves of S = 8 RI samples an edge (RI = 4, 6, 8, 12, 16).
//
// Bound: FP32 pipe and shared-memory bandwidth. A 1D transform of S points is
// two in-register passes, radix 8 and radix RI, with one twiddle multiplication
// and one shared-memory round trip between them. The radix-8 pass is the outer
// one: it is next to the elementwise step (real space along rows, Fourier space
// along columns), so a step, the last pass before it and the first pass after it
// run on the same registers and the wave never goes to shared memory between
// them. A forward / inverse pair of 2D transforms around two elementwise steps
// costs 6 round trips, where separate passes and steps cost 10.
//
// Every sample pair is two neighbours of the same row, (re0, re1, im0, im1) in
// one 16-byte cell, and the arithmetic is packed (add / mul / fma of float2, one
// instruction for two samples): half the issue slots of scalar code.
//
// Owners: a warp owns 8 rows in the row passes and 8 columns (4 cells) in the
// column passes, S / 8 warps in all, so passes along one axis synchronise inside
// a warp and only a turn from rows to columns needs the block.
//
// Shared-memory layout: cell (x, c) at pitch x + 4 (x / 8) + c with the odd pitch
// S / 2 + 1. The eight lanes of a 16-byte access phase then always fall into
// eight different groups of four banks:
//   row passes, radix RI:  lane = r + 8 a, row 8 w + r, cells of one index
//   row passes, radix 8:   tasks t = jp + (RI / 2) i, row order row_of(i)
//   column passes, radix RI: lanes (c, j) and (c, j + 4) share a phase
//   column passes, radix 8:  lanes (c, k1) and (c, k1 + 1) share a phase
//
// Index splits (forward; the inverse walks them backwards):
//   rows     y = j + RI m (j < RI, m < 8), fy = k1 + 8 k2 (k1 < 8, k2 < RI)
//            radix 8 over m on lanes (j, j + 1); its last butterfly regroups the
//            lanes to (k1, k1 + 1), so that fy leaves the radix-RI pass (over j)
//            in natural order, neighbours in one cell
//   columns  x = j + 8 k (j < 8, k < RI), fx = k1 + RI k2 (k1 < RI, k2 < 8)
//            in place: row 8 k1 + k2 of the Fourier-space wave is fx = k1 + RI k2
#pragma once

#include <cuda_runtime.h>

#include "fft_smem.cuh"

namespace pty {
namespace {

// two complex samples: lanes x and y of each part
struct Cx2 {
  float2 re, im;
};

__device__ __forceinline__ float2 dup(float v) { return make_float2(v, v); }
// (negations fold into the packed instructions' operands)
__device__ __forceinline__ float2 neg2(float2 v) { return make_float2(-v.x, -v.y); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  return __fadd2_rn(a, neg2(b));
}
__device__ __forceinline__ Cx2 add(const Cx2& a, const Cx2& b) {
  return {add2(a.re, b.re), add2(a.im, b.im)};
}
__device__ __forceinline__ Cx2 sub(const Cx2& a, const Cx2& b) {
  return {sub2(a.re, b.re), sub2(a.im, b.im)};
}
// a + (DIR i) b
template <int DIR>
__device__ __forceinline__ Cx2 add_i(const Cx2& a, const Cx2& b) {
  return DIR < 0 ? Cx2{add2(a.re, b.im), sub2(a.im, b.re)}
                 : Cx2{sub2(a.re, b.im), add2(a.im, b.re)};
}
// a + s b for a real factor
__device__ __forceinline__ Cx2 fma_r(const Cx2& b, float s, const Cx2& a) {
  return {__ffma2_rn(b.re, dup(s), a.re), __ffma2_rn(b.im, dup(s), a.im)};
}
// a - s b
__device__ __forceinline__ Cx2 fms_r(const Cx2& b, float s, const Cx2& a) {
  return {__ffma2_rn(neg2(b.re), dup(s), a.re), __ffma2_rn(neg2(b.im), dup(s), a.im)};
}
// a + (DIR i) s b for a positive factor
template <int DIR>
__device__ __forceinline__ Cx2 fma_i(const Cx2& b, float s, const Cx2& a) {
  return DIR < 0 ? Cx2{__ffma2_rn(b.im, dup(s), a.re), __ffma2_rn(neg2(b.re), dup(s), a.im)}
                 : Cx2{__ffma2_rn(neg2(b.im), dup(s), a.re), __ffma2_rn(b.re, dup(s), a.im)};
}
__device__ __forceinline__ Cx2 scale(const Cx2& a, float s) {
  return {__fmul2_rn(a.re, dup(s)), __fmul2_rn(a.im, dup(s))};
}
__device__ __forceinline__ Cx2 mul(const Cx2& a, const Cx2& b) {
  return {__ffma2_rn(a.re, b.re, neg2(__fmul2_rn(a.im, b.im))),
          __ffma2_rn(a.re, b.im, __fmul2_rn(a.im, b.re))};
}
// conj(a) b
__device__ __forceinline__ Cx2 conj_mul(const Cx2& a, const Cx2& b) {
  return {__ffma2_rn(a.re, b.re, __fmul2_rn(a.im, b.im)),
          __ffma2_rn(a.re, b.im, neg2(__fmul2_rn(a.im, b.re)))};
}
// a times the table entry w = exp(-i t) (DIR < 0) or its conjugate
template <int DIR>
__device__ __forceinline__ Cx2 twiddle(const Cx2& a, float4 w) {
  const Cx2 t{make_float2(w.x, w.y), make_float2(w.z, w.w)};
  return DIR < 0 ? mul(a, t) : conj_mul(t, a);
}
template <int DIR>
__device__ __forceinline__ Cx2 twiddle(const Cx2& a, float2 w) {
  return twiddle<DIR>(a, make_float4(w.x, w.x, w.y, w.y));
}
// a times the constant c + DIR i s (c, s > 0; one register pair each)
template <int DIR>
__device__ __forceinline__ Cx2 rotate(const Cx2& a, float c, float s) {
  return fma_i<DIR>(a, s, scale(a, c));
}

__device__ __forceinline__ Cx2 as_cx2(float4 v) {
  return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ float4 as_cell(const Cx2& v) {
  return make_float4(v.re.x, v.re.y, v.im.x, v.im.y);
}
// interleaved complex64 pair <-> Cx2
__device__ __forceinline__ Cx2 from_pair(float4 v) {
  return {make_float2(v.x, v.z), make_float2(v.y, v.w)};
}
__device__ __forceinline__ float4 to_pair(const Cx2& v) {
  return make_float4(v.re.x, v.im.x, v.re.y, v.im.y);
}

constexpr float kSqrtHalf = 0.70710678118654752f;
constexpr float kCos16 = 0.92387953251128674f;  // cos, sin of pi / 8
constexpr float kSin16 = 0.38268343236508977f;
constexpr double kSin60 = 0.86602540378443864676;  // sin of pi / 3

// DFT of length 4 in place, natural order.
template <int DIR>
__device__ __forceinline__ void dft4(Cx2& a0, Cx2& a1, Cx2& a2, Cx2& a3) {
  const Cx2 s0 = add(a0, a2), d0 = sub(a0, a2), s1 = add(a1, a3), d1 = sub(a1, a3);
  a0 = add(s0, s1);
  a2 = sub(s0, s1);
  a1 = add_i<DIR>(d0, d1);
  a3 = add_i<-DIR>(d0, d1);
}
// DFT of length 4 of (a0, w a1, w^2 a2, w^3 a3), w = exp(DIR 2 pi i / 8): the
// factor sqrt(1/2) of w and w^3 moves into the last additions.
template <int DIR>
__device__ __forceinline__ void dft4_w8(Cx2& a0, Cx2& a1, Cx2& a2, Cx2& a3) {
  const Cx2 s0 = add_i<DIR>(a0, a2), d0 = add_i<-DIR>(a0, a2);
  const Cx2 p1 = add_i<DIR>(a1, a1);              // sqrt(2) w a1
  const Cx2 p3 = add_i<DIR>(a3, a3);              // sqrt(2) w a3; w^3 a3 = (DIR i) of it
  const Cx2 s1 = add_i<DIR>(p1, p3), d1 = add_i<-DIR>(p1, p3);
  a0 = fma_r(s1, kSqrtHalf, s0);
  a2 = fms_r(s1, kSqrtHalf, s0);
  a1 = fma_i<DIR>(d1, kSqrtHalf, d0);
  a3 = fma_i<-DIR>(d1, kSqrtHalf, d0);
}
// a sin(pi / 3), the factor as two floats: its float alone is a third of an ulp
// off, the same way in every transform, which the sums over positions keep (the
// probe of a 96 x 96 batch came out 10% further from float64 with it).
__device__ __forceinline__ float2 times_sin60(float2 v) {
  constexpr float hi = (float)kSin60, lo = (float)(kSin60 - (double)hi);
  return __ffma2_rn(v, dup(hi), __fmul2_rn(v, dup(lo)));
}
__device__ __forceinline__ Cx2 times_sin60(const Cx2& a) {
  return {times_sin60(a.re), times_sin60(a.im)};
}
// a exp(DIR i pi / 6) and a exp(DIR i pi / 3)
template <int DIR>
__device__ __forceinline__ Cx2 rotate30(const Cx2& a) {
  return fma_i<DIR>(a, 0.5f, times_sin60(a));
}
template <int DIR>
__device__ __forceinline__ Cx2 rotate60(const Cx2& a) {
  const Cx2 u = times_sin60(a);
  return fma_r(a, 0.5f, DIR < 0 ? Cx2{u.im, neg2(u.re)} : Cx2{neg2(u.im), u.re});
}
template <int DIR>
__device__ __forceinline__ Cx2 rotate120(const Cx2& a) {
  const Cx2 u = times_sin60(a);
  return fms_r(a, 0.5f, DIR < 0 ? Cx2{u.im, neg2(u.re)} : Cx2{neg2(u.im), u.re});
}

template <int DIR>
__device__ __forceinline__ void dft3(Cx2& a0, Cx2& a1, Cx2& a2) {
  const Cx2 t = add(a1, a2), d = times_sin60(sub(a1, a2));
  const Cx2 m = fms_r(t, 0.5f, a0);
  a0 = add(a0, t);
  a1 = add_i<DIR>(m, d);
  a2 = add_i<-DIR>(m, d);
}

// DFT of length R in place, natural order in and out.
template <int R, int DIR>
__device__ __forceinline__ void dft_pair(Cx2 (&a)[R]) {
  if constexpr (R == 4) {
    dft4<DIR>(a[0], a[1], a[2], a[3]);
  } else if constexpr (R == 8) {
    Cx2 d[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      d[k] = sub(a[k], a[k + 4]);
      a[k] = add(a[k], a[k + 4]);
    }
    dft4<DIR>(a[0], a[1], a[2], a[3]);
    dft4_w8<DIR>(d[0], d[1], d[2], d[3]);
    Cx2 e[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) e[k] = a[k];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      a[2 * k] = e[k];
      a[2 * k + 1] = d[k];
    }
  } else if constexpr (R == 16) {
    // n = n2 + 4 n1, k = k1 + 4 k2
#pragma unroll
    for (int n = 0; n < 4; ++n) dft4<DIR>(a[n], a[n + 4], a[n + 8], a[n + 12]);
    a[5] = rotate<DIR>(a[5], kCos16, kSin16);
    const Cx2 p6 = add_i<DIR>(a[6], a[6]);  // sqrt(2) w8 a6
    a[7] = rotate<DIR>(a[7], kSin16, kCos16);
    a[13] = rotate<DIR>(a[13], kSin16, kCos16);
    const Cx2 p14 = add_i<DIR>(a[14], a[14]);  // w8^3 a14 = (DIR i) sqrt(1/2) p14
    const Cx2 m15 = rotate<DIR>(a[15], kCos16, kSin16);  // minus w16^9 a15
    dft4<DIR>(a[0], a[1], a[2], a[3]);
    {
      const Cx2 s0 = fma_r(p6, kSqrtHalf, a[4]), d0 = fms_r(p6, kSqrtHalf, a[4]);
      const Cx2 s1 = add(a[5], a[7]), d1 = sub(a[5], a[7]);
      a[4] = add(s0, s1);
      a[6] = sub(s0, s1);
      a[5] = add_i<DIR>(d0, d1);
      a[7] = add_i<-DIR>(d0, d1);
    }
    dft4_w8<DIR>(a[8], a[9], a[10], a[11]);
    {
      const Cx2 s0 = fma_i<DIR>(p14, kSqrtHalf, a[12]), d0 = fma_i<-DIR>(p14, kSqrtHalf, a[12]);
      const Cx2 s1 = sub(a[13], m15), d1 = add(a[13], m15);
      a[12] = add(s0, s1);
      a[14] = sub(s0, s1);
      a[13] = add_i<DIR>(d0, d1);
      a[15] = add_i<-DIR>(d0, d1);
    }
    Cx2 t[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) t[k] = a[k];
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
      for (int k2 = 0; k2 < 4; ++k2) a[k1 + 4 * k2] = t[4 * k1 + k2];
  } else if constexpr (R == 12) {
    // n = n2 + 4 n1 (n1 < 3), k = k1 + 3 k2
#pragma unroll
    for (int n = 0; n < 4; ++n) dft3<DIR>(a[n], a[n + 4], a[n + 8]);
    a[5] = rotate30<DIR>(a[5]);
    a[6] = rotate60<DIR>(a[6]);
    a[9] = rotate60<DIR>(a[9]);
    a[10] = rotate120<DIR>(a[10]);
    dft4<DIR>(a[0], a[1], a[2], a[3]);
    {  // a7 carries the factor DIR i
      const Cx2 s0 = add(a[4], a[6]), d0 = sub(a[4], a[6]);
      const Cx2 s1 = add_i<DIR>(a[5], a[7]), d1 = add_i<-DIR>(a[5], a[7]);
      a[4] = add(s0, s1);
      a[6] = sub(s0, s1);
      a[5] = add_i<DIR>(d0, d1);
      a[7] = add_i<-DIR>(d0, d1);
    }
    {  // a11 carries the factor -1
      const Cx2 s0 = add(a[8], a[10]), d0 = sub(a[8], a[10]);
      const Cx2 s1 = sub(a[9], a[11]), d1 = add(a[9], a[11]);
      a[8] = add(s0, s1);
      a[10] = sub(s0, s1);
      a[9] = add_i<DIR>(d0, d1);
      a[11] = add_i<-DIR>(d0, d1);
    }
    Cx2 t[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) t[k] = a[k];
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1)
#pragma unroll
      for (int k2 = 0; k2 < 4; ++k2) a[k1 + 3 * k2] = t[4 * k1 + k2];
  } else {
    static_assert(R == 6, "radix");
    // n = n2 + 2 n1 (n1 < 3), k = k1 + 3 k2
    dft3<DIR>(a[0], a[2], a[4]);
    dft3<DIR>(a[1], a[3], a[5]);
    const Cx2 w1 = rotate60<DIR>(a[3]), w2 = rotate120<DIR>(a[5]);
    const Cx2 e0 = a[0], e1 = a[2], e2 = a[4], o0 = a[1];
    a[0] = add(e0, o0);
    a[3] = sub(e0, o0);
    a[1] = add(e1, w1);
    a[4] = sub(e1, w1);
    a[2] = add(e2, w2);
    a[5] = sub(e2, w2);
  }
}

// Forward DFT of length 8 of v (lanes j, j + 1), the last butterfly regrouping
// to cells c[e][a]: lane e's outputs (2 a, 2 a + 1) as a pair.
__device__ __forceinline__ void dft8_to_k_pairs(Cx2 (&v)[8], Cx2 (&c)[2][4]) {
  dft4<-1>(v[0], v[2], v[4], v[6]);
  dft4<-1>(v[1], v[3], v[5], v[7]);
  const Cx2 p1 = add_i<-1>(v[3], v[3]), p3 = add_i<-1>(v[7], v[7]);
  // even part E[k] = v[2 k]; odd part times w8^k: o0, sqrt(1/2) p1, -i v5, -i sqrt(1/2) p3
  const float h = kSqrtHalf;
  auto put = [&](int e, int k, float re, float im) {
    float2& r = c[e][k >> 1].re;
    float2& i = c[e][k >> 1].im;
    if (k & 1) {
      r.y = re;
      i.y = im;
    } else {
      r.x = re;
      i.x = im;
    }
  };
  auto lanes = [&](int e) {
    auto L = [e](float2 t) { return e ? t.y : t.x; };
    put(e, 0, L(v[0].re) + L(v[1].re), L(v[0].im) + L(v[1].im));
    put(e, 4, L(v[0].re) - L(v[1].re), L(v[0].im) - L(v[1].im));
    put(e, 1, fmaf(L(p1.re), h, L(v[2].re)), fmaf(L(p1.im), h, L(v[2].im)));
    put(e, 5, fmaf(L(p1.re), -h, L(v[2].re)), fmaf(L(p1.im), -h, L(v[2].im)));
    put(e, 2, L(v[4].re) + L(v[5].im), L(v[4].im) - L(v[5].re));
    put(e, 6, L(v[4].re) - L(v[5].im), L(v[4].im) + L(v[5].re));
    put(e, 3, fmaf(L(p3.im), h, L(v[6].re)), fmaf(L(p3.re), -h, L(v[6].im)));
    put(e, 7, fmaf(L(p3.im), -h, L(v[6].re)), fmaf(L(p3.re), h, L(v[6].im)));
  };
  lanes(0);
  lanes(1);
}

// Inverse DFT of length 8 of the cells c[e][a] (k1 = 2 a, 2 a + 1 in the lanes),
// the first butterfly regrouping to lanes e: v[m], natural order.
__device__ __forceinline__ void dft8_from_k_pairs(const Cx2 (&c)[2][4], Cx2 (&v)[8]) {
  Cx2 s[4], d[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int a = k >> 1;
    auto L = [k](float2 t) { return k & 1 ? t.y : t.x; };
    s[k].re = make_float2(L(c[0][a].re) + L(c[0][a + 2].re), L(c[1][a].re) + L(c[1][a + 2].re));
    s[k].im = make_float2(L(c[0][a].im) + L(c[0][a + 2].im), L(c[1][a].im) + L(c[1][a + 2].im));
    d[k].re = make_float2(L(c[0][a].re) - L(c[0][a + 2].re), L(c[1][a].re) - L(c[1][a + 2].re));
    d[k].im = make_float2(L(c[0][a].im) - L(c[0][a + 2].im), L(c[1][a].im) - L(c[1][a + 2].im));
  }
  dft4<1>(s[0], s[1], s[2], s[3]);
  dft4_w8<1>(d[0], d[1], d[2], d[3]);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[2 * k] = s[k];
    v[2 * k + 1] = d[k];
  }
}

// Geometry and passes of one S x S wave; see the file header.
template <int S>
struct WaveFft {
  static constexpr int RI = S / 8;
  static constexpr int N = S * S;
  static constexpr int WARPS = S / 8;
  static constexpr int NT = 32 * WARPS;
  static constexpr int PITCH = S / 2 + 1;          // cells a row
  static constexpr int BLOCK = 8 * PITCH + 4;      // cells per 8 rows
  static constexpr int CELLS = BLOCK * (S / 8);
  static constexpr int TCOL = 9 * RI;              // column twiddles, [k1][j] at 9 k1 + j
  static constexpr int TROW = 4 * RI;              // row twiddles, [a][j parity][j / 2]
  static constexpr int TASKS = 4 * RI;             // radix-8 tasks of a warp
  static constexpr int TITER = (TASKS + 31) / 32;  // radix-8 tasks of a thread
  static constexpr int HALF = RI / 2;
  static_assert(S % 16 == 0 && (RI == 4 || RI == 6 || RI == 8 || RI == 12 || RI == 16), "S");

  float4* wave;
  float2* tcol;
  float4* trow;
  int warp, lane;

  // row of the warp's i-th group of HALF radix-8 tasks (distinct bank groups for
  // the eight tasks of an access phase)
  static __device__ __forceinline__ int row_of(int i) {
    constexpr int period = HALF % 8 == 0 ? 1 : HALF % 4 == 0 ? 2 : HALF % 2 == 0 ? 4 : 8;
    return (HALF * i) % 8 + i / period;
  }
  // fill the twiddle tables (block-cooperative, no barrier)
  __device__ __forceinline__ void tables(int tid) const {
    for (int i = tid; i < RI * 8; i += NT) {
      const int k1 = i / 8, j = i % 8;
      const float2 w = twiddle_detail::kTable<S>.v[j * k1];
      tcol[9 * k1 + j] = w;
    }
    for (int i = tid; i < TROW; i += NT) {
      const int a = i / RI, j = 2 * (i % HALF) + (i / HALF) % 2;
      const float2 w0 = twiddle_detail::kTable<S>.v[j * 2 * a];
      const float2 w1 = twiddle_detail::kTable<S>.v[j * (2 * a + 1)];
      trow[i] = make_float4(w0.x, w1.x, w0.y, w1.y);
    }
  }

  // ---- columns: 4 cells x S rows of this warp
  __device__ __forceinline__ float4* col_inner() const {  // radix RI: cell c, j
    const int c = lane & 3, j = ((lane >> 2) & 1) * 4 + (lane >> 3);
    return wave + PITCH * j + 4 * warp + c;
  }
  __device__ __forceinline__ const float2* col_inner_tw() const {
    return tcol + ((lane >> 2) & 1) * 4 + (lane >> 3);
  }
  __device__ __forceinline__ void col_inner_forward() const {
    float4* p = col_inner();
    const float2* w = col_inner_tw();
    Cx2 a[RI];
#pragma unroll
    for (int k = 0; k < RI; ++k) a[k] = as_cx2(p[BLOCK * k]);
    dft_pair<RI, -1>(a);
    p[0] = as_cell(a[0]);
#pragma unroll
    for (int k = 1; k < RI; ++k) p[BLOCK * k] = as_cell(twiddle<-1>(a[k], w[9 * k]));
  }
  __device__ __forceinline__ void col_inner_inverse() const {
    float4* p = col_inner();
    Cx2 a[RI];
#pragma unroll
    for (int k = 0; k < RI; ++k) a[k] = as_cx2(p[BLOCK * k]);
    dft_pair<RI, 1>(a);
#pragma unroll
    for (int k = 0; k < RI; ++k) p[BLOCK * k] = as_cell(a[k]);
  }
  // radix-8 task t < TASKS of the warp: cell t & 3, k1 = t >> 2; rows 8 k1 + i hold
  // fx = k1 + RI i
  __device__ __forceinline__ float4* col_outer(int t) const {
    return wave + BLOCK * (t >> 2) + 4 * warp + (t & 3);
  }
  __device__ __forceinline__ void col_outer_load(int t, Cx2 (&v)[8]) const {
    const float4* p = col_outer(t);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = as_cx2(p[PITCH * i]);
    dft_pair<8, -1>(v);
  }
  __device__ __forceinline__ void col_outer_store(int t, Cx2 (&v)[8]) const {
    dft_pair<8, 1>(v);
    float4* p = col_outer(t);
    const float2* w = tcol + 9 * (t >> 2);
    p[0] = as_cell(v[0]);
#pragma unroll
    for (int i = 1; i < 8; ++i) p[PITCH * i] = as_cell(twiddle<1>(v[i], w[i]));
  }

  // ---- rows: 8 rows of this warp
  __device__ __forceinline__ float4* row_inner() const {  // radix RI: row r, pair a
    return wave + BLOCK * warp + PITCH * (lane & 7);
  }
  __device__ __forceinline__ void row_inner_forward() const {
    float4* p = row_inner();
    const int a = lane >> 3;
    Cx2 v[RI];
#pragma unroll
    for (int j = 0; j < RI; ++j) v[j] = as_cx2(p[RI * a + (j & 1) * HALF + (j >> 1)]);
    dft_pair<RI, -1>(v);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < RI; ++k) p[a + 4 * k] = as_cell(v[k]);
  }
  __device__ __forceinline__ void row_inner_inverse() const {
    float4* p = row_inner();
    const int a = lane >> 3;
    const float4* w = trow + RI * a;
    Cx2 v[RI];
#pragma unroll
    for (int k = 0; k < RI; ++k) v[k] = as_cx2(p[a + 4 * k]);
    dft_pair<RI, 1>(v);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < RI; ++j) {
      const int i = (j & 1) * HALF + (j >> 1);
      p[RI * a + i] = as_cell(twiddle<1>(v[j], w[i]));
    }
  }
  // radix-8 task t of the warp: jp = t % HALF, row row_of(t / HALF); samples
  // y = 2 jp + e + RI m
  static __device__ __forceinline__ int task_jp(int t) { return t % HALF; }
  static __device__ __forceinline__ int task_row(int t) { return row_of(t / HALF); }
  __device__ __forceinline__ float4* row_outer(int t) const {
    return wave + BLOCK * warp + PITCH * task_row(t) + task_jp(t);
  }
  __device__ __forceinline__ void row_outer_load(int t, Cx2 (&v)[8]) const {
    const float4* p = row_outer(t);
    Cx2 c[2][4];
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int a = 0; a < 4; ++a) c[e][a] = as_cx2(p[RI * a + HALF * e]);
    dft8_from_k_pairs(c, v);
  }
  __device__ __forceinline__ void row_outer_store(int t, Cx2 (&v)[8]) const {
    Cx2 c[2][4];
    dft8_to_k_pairs(v, c);
    float4* p = row_outer(t);
    const float4* w = trow + task_jp(t);
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int a = 0; a < 4; ++a)
        p[RI * a + HALF * e] = as_cell(twiddle<-1>(c[e][a], w[RI * a + HALF * e]));
  }
};

}  // namespace
}  // namespace pty
