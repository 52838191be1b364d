// Per-position kernels on the packed in-shared-memory transforms of
// wave_fft.cuh: the same forward model, projection and adjoint terms as
// position_one (ptycho_position.cuh) for square regions of interest.
//
// One block of 4 S threads per position. The model is a walk over phases that
// alternate between the axes: a column phase (Fourier space) transforms the
// columns forward, applies a Fourier-space step and transforms them back; a row
// phase (real space) does the same around a real-space step; a block barrier
// turns from one to the other. Phase n of single-slice / multislice models:
//   columns n = 0: spectrum x ramp           rows n < T: P_n, psi = P_n O_n
//           n < T: x propagator n - 1             n >= T: adjoint of slice 2 T - 1 - n
//           n = T: Fourier projection
//           n > T: x conj(propagator 2 T - 1 - n)
// so single-slice gradient descent is two turns of one loop and needs 5 block
// barriers. Mixed states run the forward half for every mode, keeping the far
// fields, and then the other half for every mode.
#pragma once

#include "ptycho_internal.h"
#include "tc_gemm.cuh"
#include "wave_fft.cuh"

namespace pty {
namespace {

// The transmission functions of the slices (complex objects as they are, exp(iV)
// of potentials) in two copies, one starting at column 0 and one at column 1, in
// cells of two columns (re0, re1, im0, im1), each row wrapped on by S + 2 columns:
// the patch of a position starts at a whole cell of one of the copies whatever
// its parity, so its rows are read as aligned 16-byte cells with neither index
// wraps nor regrouping. (Pairs of 8-byte loads from the object moved twice the
// sectors: 40% of the L1 wavefronts of the 128 x 128 kernel.) One launch a batch;
// the copies live where the batch's reductions write later.
__host__ __device__ __forceinline__ int transmission_pitch(int Py, int S) {
  return (Py + S + 3) / 2;
}

__global__ void __launch_bounds__(256) transmission_kernel(BatchArgs a, int pitch) {
  // (rows on the first grid axis: the others end at 65535)
  const int x = blockIdx.x, s = blockIdx.z;
  const int c = blockIdx.y * 256 + threadIdx.x;  // cell of the row
  if (c >= pitch) return;
  const size_t row = ((size_t)s * a.Px + x) * a.Py;
  float2 v[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    int y = 2 * c + k;
    while (y >= a.Py) y -= a.Py;
    if (a.potential) {
      float sv, cv;
      sincosf(reinterpret_cast<const float*>(a.object)[row + y], &sv, &cv);
      v[k] = make_float2(cv, sv);
    } else {
      v[k] = reinterpret_cast<const float2*>(a.object)[row + y];
    }
  }
#pragma unroll
  for (int q = 0; q < 2; ++q)
    a.trans[(((size_t)q * a.T + s) * a.Px + x) * pitch + c] =
        make_float4(v[q].x, v[q + 1].x, v[q].y, v[q + 1].y);
}

inline cudaError_t launch_transmission(const BatchArgs& a, cudaStream_t s) {
  const int pitch = transmission_pitch(a.Py, a.Sy);
  transmission_kernel<<<dim3(a.Px, (pitch + 255) / 256, a.T), 256, 0, s>>>(a, pitch);
  return cudaGetLastError();
}

// What a block keeps of its position.
template <int S>
struct WavePosition {
  using W = WaveFft<S>;
  // shared memory: wave, twiddle tables, two buffers of sub-pixel shift ramps
  // (x: (re, re, im, im) per fx; y: one cell per pair of fy), the slots
  static constexpr int RAMPS = S + S / 2;
  static constexpr int CELLS = W::CELLS + W::TROW + 2 * RAMPS + (W::TCOL + 1) / 2;
  W w;
  float4* ramps;
  int x0, y0;  // rounded position
  int bx, by;  // object pixel of patch corner (S / 2, S / 2)

  // slots: one float2 per Fourier sample pair of a thread (the amplitudes, or
  // the mixed-state intensity sums)
  static constexpr size_t smem_bytes(bool slots) {
    return sizeof(float4) * (size_t)CELLS +
           (slots ? sizeof(float2) * (size_t)(8 * W::TITER * W::NT) : 0);
  }

  __device__ __forceinline__ void carve(float4* smem) {
    w.wave = smem;
    w.trow = smem + W::CELLS;
    ramps = smem + W::CELLS + W::TROW;
    w.tcol = reinterpret_cast<float2*>(ramps + 2 * RAMPS);
    w.warp = threadIdx.x >> 5;
    w.lane = threadIdx.x & 31;
  }

  // scan position of batch entry b
  static __device__ __forceinline__ float2 position(const BatchArgs& a, const float* positions,
                                                    int b) {
    const int prow = a.pos_rows ? a.pos_rows[b] : b;
    return make_float2(positions[2 * prow], positions[2 * prow + 1]);
  }

  // patch and ramps (buffer k) of the position (qx, qy), no barrier; false when it
  // is not finite (then taken as 0)
  __device__ __forceinline__ bool locate(const BatchArgs& a, float qx, float qy, int k) {
    const float posx = finite_or_zero(qx), posy = finite_or_zero(qy);
    const float rx = rintf(posx), ry = rintf(posy);  // numpy.round: half to even
    x0 = (int)rx;
    y0 = (int)ry;
    bx = pmod(x0 - S / 2, a.Px);
    by = pmod(y0 - S / 2, a.Py);
    // the phase in float32 like the reference's complex64 expression, its cos /
    // sin rounded once; frequency -f has the conjugate of f's
    const int axis = threadIdx.x / (S / 2 + 1), f = threadIdx.x % (S / 2 + 1);
    if (axis < 2) {
      const float q = (float)f / (float)S;
      const float2 r = cis_rounded(
          __fmul_rn(__fmul_rn(-6.2831855f, q), axis == 0 ? posx - rx : posy - ry));
      float4* const px = ramps + RAMPS * k;
      auto put = [&](int i, float im) {
        if (axis == 0) {
          px[i] = make_float4(r.x, r.x, im, im);
        } else {
          float* c = reinterpret_cast<float*>(px + S + (i >> 1)) + (i & 1);
          c[0] = r.x;
          c[2] = im;
        }
      };
      if (f < S / 2) put(f, r.y);
      if (f > 0) put(S - f, -r.y);  // f = S / 2 is the frequency -S / 2
    }
    return isfinite(qx) && isfinite(qy);
  }

  // ramp at Fourier sample i of task t
  __device__ __forceinline__ Cx2 ramp(int t, int i, int k = 0) const {
    const float4* px = ramps + RAMPS * k;
    return mul(as_cx2(px[(t >> 2) + W::RI * i]), as_cx2(px[S + 4 * w.warp + (t & 3)]));
  }
  // index of Fourier sample i (lane 0) of task t in an S x S array
  __device__ __forceinline__ int fourier(int t, int i) const {
    return ((t >> 2) + W::RI * i) * S + 8 * w.warp + 2 * (t & 3);
  }
  // index of real-space sample m (lane 0) of task t
  __device__ __forceinline__ int real(int t, int m) const {
    return (8 * w.warp + W::task_row(t)) * S + 2 * W::task_jp(t) + W::RI * m;
  }
  // transmission samples of slice s, real-space task t, with the patch moved by
  // (sx, sy) in {0, 1}
  __device__ __forceinline__ void load_patch(const BatchArgs& a, int s, int t, int sx, int sy,
                                             Cx2 (&o)[8]) const {
    const int x = 8 * w.warp + W::task_row(t);
    int ox = bx + (x + S / 2) % S + sx;
    if (ox >= a.Px) ox -= a.Px;
    const int y = by + sy;
    const float4* __restrict__ q =
        a.trans + (((size_t)(y & 1) * a.T + s) * a.Px + ox) * transmission_pitch(a.Py, S) +
        (y >> 1) + W::task_jp(t);
#pragma unroll
    for (int m = 0; m < 8; ++m) o[m] = as_cx2(__ldg(q + W::HALF * ((m + 4) & 7)));
  }
};

__device__ __forceinline__ float4 ld_cell(const float2* p) {
  return *reinterpret_cast<const float4*>(p);
}
__device__ __forceinline__ void st_cell(float2* p, float4 v) {
  *reinterpret_cast<float4*>(p) = v;
}
__device__ __forceinline__ float2 ld_two(const float* p) {
  return *reinterpret_cast<const float2*>(p);
}
__device__ __forceinline__ void st_two(float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; }
__device__ __forceinline__ float rsqrt_approx(float v) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
// asynchronous 8-byte copy from global to shared memory
__device__ __forceinline__ void copy_async8(float2* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_async_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}
__device__ __forceinline__ float2 abs2(const Cx2& v) {
  return __ffma2_rn(v.re, v.re, __fmul2_rn(v.im, v.im));
}

// A exp(i angle f) (gd: minus f) for one lane, the expressions of position_one.
__device__ __noinline__ float3 project_lane(bool gd, float A, float re, float im) {
  const float af = c_abs(make_float2(re, im));
  const float d = A - af;
  const float q = af > 0.0f ? A / af : 0.0f;
  float3 r;
  if (gd) {
    r.x = af > 0.0f ? fmaf(re, q, -re) : A - re;
    r.y = af > 0.0f ? fmaf(im, q, -im) : -im;
  } else {
    r.x = af > 0.0f ? re * q : A;
    r.y = af > 0.0f ? im * q : 0.0f;
  }
  r.z = d * d;
  return r;
}

// The Fourier projection of a task's eight cells: |f| and A / |f| from one
// reciprocal square root and Newton steps on the residuals s - |f|^2 and
// A - q |f|, packed, where the IEEE square root and quotient took 25 instructions a
// sample. Each residual is one fused multiply-add, so a step ends in one rounding of a
// value accurate to about 2^-45 (the method: P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990): the results are the
// correctly rounded ones but for values that close to a tie. Restated with any error
// the reciprocal root may have, one in 2e6 differs, by an ulp; here none of 2e8 did. A
// task with a square outside [1e-30, 1e30] other than 0 takes project_lane.
__device__ __forceinline__ void project(bool gd, const float2 (&A)[8], Cx2 (&f)[8], float2& err) {
  float2 s[8], g[8];  // |f|^2, and the same with 1 for 0
  float lo = 1.0f, hi = 1.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    s[i] = abs2(f[i]);
    g[i] = make_float2(s[i].x == 0.0f ? 1.0f : s[i].x, s[i].y == 0.0f ? 1.0f : s[i].y);
    lo = fminf(lo, fminf(g[i].x, g[i].y));
    hi = fmaxf(hi, fmaxf(g[i].x, g[i].y));
  }
  // (a NaN square passes the minimum and maximum and stays NaN below)
  if (lo < 1e-30f || hi > 1e30f) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float3 u = project_lane(gd, A[i].x, f[i].re.x, f[i].im.x);
      const float3 v = project_lane(gd, A[i].y, f[i].re.y, f[i].im.y);
      f[i] = {make_float2(u.x, v.x), make_float2(u.y, v.y)};
      err = add2(err, make_float2(u.z, v.z));
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 y = make_float2(rsqrt_approx(g[i].x), rsqrt_approx(g[i].y));
    const float2 a0 = __fmul2_rn(s[i], y);
    const float2 e = __ffma2_rn(neg2(a0), a0, s[i]);
    const float2 a = __ffma2_rn(__fmul2_rn(dup(0.5f), y), e, a0);  // |f|
    const float2 t = __ffma2_rn(neg2(a), y, dup(1.0f));
    const float2 y1 = __ffma2_rn(y, t, y);                         // 1 / |f|
    const float2 q0 = __fmul2_rn(A[i], y1);
    const float2 q = __ffma2_rn(__ffma2_rn(neg2(q0), a, A[i]), y1, q0);  // A / |f|
    const float2 d = sub2(A[i], a);
    err = __ffma2_rn(d, d, err);
    if (gd) {
      f[i] = {__ffma2_rn(f[i].re, q, neg2(f[i].re)), __ffma2_rn(f[i].im, q, neg2(f[i].im))};
    } else {
      f[i] = {__fmul2_rn(f[i].re, q), __fmul2_rn(f[i].im, q)};
    }
    // phase 0 where the model is 0
    if (s[i].x == 0.0f) f[i].re.x = A[i].x;
    if (s[i].y == 0.0f) f[i].re.y = A[i].y;
  }
}

// f times the detector mask at the samples of Fourier-space task t
template <int S>
__device__ __forceinline__ void apply_mask(const WavePosition<S>& p, const float* mask, int t,
                                           Cx2 (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 mk = ld_two(mask + p.fourier(t, i));
    f[i] = {__fmul2_rn(f[i].re, mk), __fmul2_rn(f[i].im, mk)};
  }
}

// Tensor memory as this thread's own storage: `words` consecutive 32-bit columns
// of its lane (warp w owns lanes 32 (w % 4) .. + 31).
__device__ __forceinline__ void tmem_put(uint32_t addr, const Cx2 (&v)[8]) {
#define PTY_CELL(k)                                                                     \
  "r"(__float_as_uint(v[k].re.x)), "r"(__float_as_uint(v[k].re.y)),                     \
      "r"(__float_as_uint(v[k].im.x)), "r"(__float_as_uint(v[k].im.y))
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(
          addr),
      PTY_CELL(0), PTY_CELL(1), PTY_CELL(2), PTY_CELL(3), PTY_CELL(4), PTY_CELL(5), PTY_CELL(6),
      PTY_CELL(7)
      : "memory");
#undef PTY_CELL
}
__device__ __forceinline__ void tmem_put(uint32_t addr, const float2 (&v)[8]) {
#define PTY_TWO(k) "r"(__float_as_uint(v[k].x)), "r"(__float_as_uint(v[k].y))
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(addr),
      PTY_TWO(0), PTY_TWO(1), PTY_TWO(2), PTY_TWO(3), PTY_TWO(4), PTY_TWO(5), PTY_TWO(6),
      PTY_TWO(7)
      : "memory");
#undef PTY_TWO
}
// (the values arrive at tmem_wait_load)
__device__ __forceinline__ void tmem_get(uint32_t addr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tmem_wait_load(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) asm volatile("" : "+r"(r[i]));  // uses stay below the wait
}
__device__ __forceinline__ void tmem_wait_store() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ Cx2 tmem_cell(const uint32_t (&r)[32], int k) {
  return {make_float2(__uint_as_float(r[4 * k]), __uint_as_float(r[4 * k + 1])),
          make_float2(__uint_as_float(r[4 * k + 2]), __uint_as_float(r[4 * k + 3]))};
}

// kKind 0: plain single-slice single-probe gradient descent; 1: any single-probe
// model (multislice, projection sets, kept far fields, forward only, exact probe
// gradient); 2: any mixed-state model (likewise).
// Bound: shared memory (two round trips an axis) and the L2 traffic of the stashed
// P_s, patches and terms, one block of 128 x 128 an SM. 256 positions at 128 x 128:
// 8 slices 490 us (557 with the block-wide walk by groups of warps), 4 modes 324
// (340); both are 1.7 rounds of 152 blocks and pay two.
template <int S, int kKind>
__global__ void __launch_bounds__(WaveFft<S>::NT) wave_position_kernel(BatchArgs a) {
  using W = WaveFft<S>;
  using P = WavePosition<S>;
  constexpr int N = W::N;
  constexpr bool kPlain = kKind == 0;
  constexpr bool kMixed = kKind == 2;
  extern __shared__ float4 smem4[];
  __shared__ float red[W::NT / 32];

  const int tid = threadIdx.x;
  const int T = kPlain ? 1 : a.T;
  const int M = kMixed ? a.M : 1;
  P p;
  p.carve(smem4);
  p.w.tables(tid);
  // single-slice mixed states sum the modes' object terms and |P|^2 in tensor
  // memory (48 words a task of this thread) and write them once
  constexpr bool kTmem = kMixed && S == 128;
  constexpr int WORDS = 48 * W::TITER;
  __shared__ uint32_t tmem_base;
  uint32_t tm = 0;
  if constexpr (kTmem) {
    if (p.w.warp == 0) nn::tmem_alloc(&tmem_base, 512);
    nn::tc_fence_before();
    __syncthreads();
    nn::tc_fence_after();
    tm = tmem_base + ((uint32_t)(p.w.warp & 3) << 21) + (p.w.warp >> 2) * WORDS;
  }
  const bool mode_sums = kTmem && T == 1 && M > 1;

  // (resident blocks walk the batch where the launch has fewer blocks)
#pragma unroll 1
  for (int b = blockIdx.x; b < a.B; b += gridDim.x) {
  const int prow = a.pos_rows ? a.pos_rows[b] : b;
  const int arow = a.amp_rows ? a.amp_rows[b] : b;
  const float2 at = P::position(a, a.positions, b);
  const bool pos_ok = p.locate(a, at.x, at.y, 0);
  if (tid == 0) a.pos_round[b] = make_int2(p.x0, p.y0);
  __syncthreads();

  const W& w = p.w;
  const float invN = 1.0f / (float)N;
  const float* amp = a.amplitudes + (size_t)arow * N;
  const bool ps = !kPlain && a.projection != 0;
  const bool fwd = !kPlain && a.forward_only != 0;
  const bool exact = !kPlain && a.exact_probe_grad != 0;
  const float px_ = 1.0f - a.pa - a.pb;  // projection x
  const float py_ = 1.0f - a.pc;          // projection y
  float2* const itot = reinterpret_cast<float2*>(smem4 + P::CELLS);
  float err = 0.0f;
  float2 err2 = make_float2(0.0f, 0.0f);
  if constexpr (!kMixed) {
    // this thread's amplitudes travel to its own slots meanwhile
#pragma unroll 1
    for (int it = 0; it < W::TITER; ++it) {
      const int t = w.lane + 32 * it;
      if (W::TASKS % 32 != 0 && t >= W::TASKS) break;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        copy_async8(itot + (8 * it + i) * W::NT + tid, amp + p.fourier(t, i));
    }
  }

  // the forward half of every mode, then the other half of every mode; a single
  // probe walks through in one pass
#pragma unroll 1
  for (int pass = 0; pass < (kMixed && !fwd ? 2 : 1); ++pass) {
#pragma unroll 1
    for (int m = 0; m < M; ++m) {
      const float2* __restrict__ spec = a.probe_spec + (size_t)m * N;
      float2* const far = a.scratch_f + ((size_t)b * M + m) * N;
      float2* const probe_term = a.st_probe + ((size_t)b * M + m) * N;
      // stash of P_{s,m}: the rows that the adjoint's terms overwrite, or st_pm
      auto stash = [&](int s) {
        return T == 1 ? probe_term
               : !kMixed ? a.st_obj + ((size_t)s * a.B + b) * N
                         : a.st_pm + (((size_t)s * a.B + b) * M + m) * N;
      };
      float2* const ew = ps ? a.exit_waves + ((size_t)prow * M + m) * N : nullptr;
      const int n0 = pass == 0 ? 0 : T;
      const int n1 = kMixed && pass == 0 ? T + 1 : exact ? 2 * T + 1 : 2 * T;
#pragma unroll 1
      for (int n = n0; n < n1; ++n) {
        // ------------------------------------------------ columns, Fourier space
        const bool col_fwd = n > 0 && !(kMixed && pass == 1 && n == T);
        // the far field of a forward half and the exact probe term end here
        const bool col_end = (n == T && ((kMixed && pass == 0) || fwd)) || n == 2 * T;
        if (col_fwd) {
          w.col_inner_forward();
          __syncwarp();
        }
#pragma unroll 1
        for (int it = 0; it < W::TITER; ++it) {
          const int t = w.lane + 32 * it;
          if (W::TASKS % 32 != 0 && t >= W::TASKS) break;
          Cx2 v[8];
          if (n == 0) {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = from_pair(ld_cell(spec + p.fourier(t, i)));
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = mul(v[i], p.ramp(t, i));
          } else if (n == T && (!kMixed || pass == 0)) {
            if constexpr (!kMixed) {
              w.col_outer_load(t, v);
              copy_async_wait();
              float2 A[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) A[i] = itot[(8 * it + i) * W::NT + tid];
              if (!kPlain && a.keep_farfield) {
#pragma unroll
                for (int i = 0; i < 8; ++i) st_cell(far + p.fourier(t, i), to_pair(v[i]));
              }
              if (a.det_mask) apply_mask(p, a.det_mask, t, v);
              project(!ps, A, v, err2);
              if (a.det_mask && !ps) apply_mask(p, a.det_mask, t, v);
            } else {
              w.col_outer_load(t, v);
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                st_cell(far + p.fourier(t, i), to_pair(v[i]));
                float2& tot = itot[(8 * it + i) * W::NT + tid];
                const float2 h = abs2(v[i]);
                tot = m == 0 ? h : add2(tot, h);
              }
            }
          } else if (kMixed && n == T) {  // pass 1
            if constexpr (kMixed) {
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] = from_pair(ld_cell(far + p.fourier(t, i)));
              if (a.det_mask) apply_mask(p, a.det_mask, t, v);
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const float2 q = itot[(8 * it + i) * W::NT + tid];
                const Cx2 r{__fmul2_rn(v[i].re, q), __fmul2_rn(v[i].im, q)};
                v[i] = ps ? r : sub(r, v[i]);
              }
              if (a.det_mask && !ps) apply_mask(p, a.det_mask, t, v);
            }
          } else if constexpr (!kPlain) {
            w.col_outer_load(t, v);
            if (n == 2 * T) {
              // exact probe gradient: back through the sub-pixel shift
#pragma unroll
              for (int i = 0; i < 8; ++i)
                st_cell(probe_term + p.fourier(t, i), to_pair(conj_mul(p.ramp(t, i), v[i])));
            } else {
              const bool back = n > T;
              const float2* __restrict__ h = a.props + (size_t)(back ? 2 * T - 1 - n : n - 1) * N;
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                Cx2 hv = from_pair(__ldg(reinterpret_cast<const float4*>(h + p.fourier(t, i))));
                if (back) hv.im = neg2(hv.im);
                v[i] = mul(v[i], hv);
              }
            }
          }
          if (!col_end) w.col_outer_store(t, v);
        }
        if (!kPlain && col_end) {
          __syncthreads();  // the next walk rewrites the wave
          break;
        }
        __syncwarp();
        w.col_inner_inverse();
        __syncthreads();

        // --------------------------------------------------- rows, real space
        const bool row_fwd = n + 1 < n1;
        w.row_inner_inverse();
        __syncwarp();
#pragma unroll 1
        for (int it = 0; it < W::TITER; ++it) {
          const int t = w.lane + 32 * it;
          if (W::TASKS % 32 != 0 && t >= W::TASKS) break;
          Cx2 o[8], v[8];
          if (n < T) {
            const int s = n;
            p.load_patch(a, s, t, 0, 0, o);
            w.row_outer_load(t, v);
            float2* const st = stash(s);
            const bool mix = !kPlain && ps && s == T - 1;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int e = p.real(t, i);
              v[i] = scale(v[i], invN);
              st_cell(st + e, as_cell(v[i]));
              v[i] = mul(v[i], o[i]);
              if (mix) {
                const Cx2 wv = a.ew_valid ? from_pair(ld_cell(ew + e)) : v[i];
                v[i] = fma_r(wv, py_, scale(v[i], a.pc));
              }
            }
          } else {
            const int s = 2 * T - 1 - n;
            float2* const st = stash(s);
            p.load_patch(a, s, t, 0, 0, o);
            Cx2 pr[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) pr[i] = as_cx2(ld_cell(st + p.real(t, i)));
            w.row_outer_load(t, v);
            float2* const gobj = a.st_obj + ((size_t)s * a.B + b) * N;
            float* const nobj = a.st_nobj + ((size_t)s * a.B + b) * N;
            const bool mix = !kPlain && ps && n == T;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int e = p.real(t, i);
              Cx2 chi = scale(v[i], invN);
              if (mix) {
                // new exit wave x w + a psi + b projected
                const Cx2 psi = mul(pr[i], o[i]);
                const Cx2 wv = a.ew_valid ? from_pair(ld_cell(ew + e)) : psi;
                chi = fma_r(chi, a.pb, fma_r(psi, a.pa, scale(wv, px_)));
                st_cell(ew + e, to_pair(chi));
              }
              Cx2 g = conj_mul(pr[i], chi);
              if (a.potential) {
                // Re(-i conj(O) conj(P) chi)
                g.re = conj_mul(o[i], g).im;
                g.im = make_float2(0.0f, 0.0f);
              }
              const float2 pn = abs2(pr[i]);
              v[i] = conj_mul(o[i], chi);
              if (s == 0) {
                if (!exact) st_cell(probe_term + e, to_pair(v[i]));
                if (!kPlain && m == 0 && !a.nprobe_from_object)
                  st_two(a.st_nprobe + (size_t)b * N + e, abs2(o[i]));
              }
              if (mode_sums) {
                pr[i] = g;  // summed below
                o[i].re = pn;
              } else if (kMixed && m > 0) {
                st_cell(gobj + e, to_pair(add(from_pair(ld_cell(gobj + e)), g)));
                st_two(nobj + e, add2(ld_two(nobj + e), pn));
              } else {
                st_cell(gobj + e, to_pair(g));
                st_two(nobj + e, pn);
              }
            }
            if constexpr (kTmem) {
              if (mode_sums) {
                const uint32_t tg = tm + 48 * it;
                float2 pn[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) pn[i] = o[i].re;
                if (m > 0) {
                  uint32_t r[32];
                  float q[16];
                  tmem_get(tg, r);
                  tmem_wait_load(r);
#pragma unroll
                  for (int i = 0; i < 8; ++i) pr[i] = add(tmem_cell(r, i), pr[i]);
                  nn::tmem_load16(tg + 32, q);
#pragma unroll
                  for (int i = 0; i < 8; ++i)
                    pn[i] = add2(make_float2(q[2 * i], q[2 * i + 1]), pn[i]);
                }
                if (m + 1 < M) {
                  tmem_put(tg, pr);
                  tmem_put(tg + 32, pn);
                  tmem_wait_store();
                } else {
#pragma unroll
                  for (int i = 0; i < 8; ++i) {
                    const int e = p.real(t, i);
                    st_cell(gobj + e, to_pair(pr[i]));
                    st_two(nobj + e, pn[i]);
                  }
                }
              }
            }
          }
          if (row_fwd) w.row_outer_store(t, v);
        }
        if (row_fwd) {
          __syncwarp();
          w.row_inner_forward();
        }
        __syncthreads();
      }
    }
    if constexpr (kMixed) {
      if (pass == 0) {
        // the shared ratio A / sqrt(sum_m |F_m|^2), 0 where the model is 0
#pragma unroll 1
        for (int it = 0; it < W::TITER; ++it) {
          const int t = w.lane + 32 * it;
          if (W::TASKS % 32 != 0 && t >= W::TASKS) break;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int e = p.fourier(t, i);
            const float2 A = __ldg(reinterpret_cast<const float2*>(amp + e));
            float2 s2 = itot[(8 * it + i) * W::NT + tid];
            if (a.det_mask) {
              const float2 mk = ld_two(a.det_mask + e);
              s2 = __fmul2_rn(__fmul2_rn(s2, mk), mk);
            }
            const float t0 = sqrtf(s2.x), t1 = sqrtf(s2.y);
            const float d0 = A.x - t0, d1 = A.y - t1;
            err += d0 * d0;
            err += d1 * d1;
            itot[(8 * it + i) * W::NT + tid] =
                make_float2(t0 == 0.0f ? 0.0f : A.x / t0, t1 == 0.0f ? 0.0f : A.y / t1);
          }
        }
      }
    }
  }
  const float tot = block_sum<W::NT>(err + (err2.x + err2.y), red);
  if (tid == 0) a.err[b] = pos_ok ? tot : __int_as_float(0x7fc00000);
  __syncthreads();  // red and the ramps are rewritten by the next position
  }
  if constexpr (kTmem) {
    nn::tc_fence_before();
    __syncthreads();
    nn::tc_fence_after();
    if (p.w.warp == 0) nn::tmem_dealloc(tmem_base, 512);
  }
}

// Plain single-slice single-probe gradient descent: one resident block per SM
// walks the batch (b = blockIdx.x, + gridDim.x, ...).
//
// Bound: the traffic between the SM and L2, and shared memory. Against the
// one-position-per-block kernel a position moves 640 KB instead of 1020: the
// shifted probe waits for the adjoint in tensor memory (thread-private, no
// 128 KB out and back through L2), and the probe terms conj(O) chi of the
// block's positions are summed there too and leave once per block, as row
// blockIdx.x of st_probe (probe_reduce_kernel then adds gridDim.x rows instead
// of B). Positions go to blocks by index, so every sum has a fixed order. A
// position's amplitudes travel while its first column and row passes run; the spectrum
// and ramps of the next position follow this one's adjoint.
// 128 x 128, per 1024 positions: 172 us, where the block-wide walk with named
// barriers took 250 and one position per block of this one 219.
// kFull adds the projection sets and the kept far field: 4096 positions of a
// difference map 765 us (one position per block: 1066, and 140 us more to add the
// probe terms of all positions), 1024 positions with the far field kept 182 (233).
template <int S, bool kFull>
__global__ void __launch_bounds__(WaveFft<S>::NT) wave_gd_kernel(BatchArgs a) {
  using W = WaveFft<S>;
  using P = WavePosition<S>;
  constexpr int N = W::N;
  constexpr int WORDS = 64 * W::TITER;             // tensor-memory columns of a warp
  constexpr int COLS = WORDS * (W::WARPS / 4);
  static_assert(W::TASKS % 32 == 0 && W::WARPS % 4 == 0 && COLS <= 512, "tensor memory");
  extern __shared__ float4 smem4[];
  __shared__ float red[W::WARPS];
  __shared__ uint32_t tmem_base;

  const int tid = threadIdx.x;
  P p;
  p.carve(smem4);
  const W& w = p.w;
  if (w.warp == 0) nn::tmem_alloc(&tmem_base, COLS);
  w.tables(tid);

  // the amplitudes, rows of S padded so that the (fy pair, fx) walk of the
  // Fourier-space tasks is free of bank conflicts
  constexpr int AP = S + 8;
  float* const amps = reinterpret_cast<float*>(smem4 + P::CELLS);
  const float invN = 1.0f / (float)N;
  const bool ps = kFull && a.projection != 0;
  const float px_ = 1.0f - a.pa - a.pb;  // projection x
  const float py_ = 1.0f - a.pc;          // projection y
  const float2* __restrict__ spec = a.probe_spec;
  // `count` of the PARTS 16-byte pieces that each thread copies, from piece q on
  constexpr int PARTS = N / 4 / W::NT;
  auto fetch_amplitudes = [&](int arow, int q, int count) {
    const float* src = a.amplitudes + (size_t)arow * N;
#pragma unroll
    for (int r = 0; r < count; ++r) {
      const int i = tid + (q + r) * W::NT;
      copy_async16(amps + (i / (S / 4)) * AP + 4 * (i % (S / 4)), src + 4 * i);
    }
  };
  float4 sp[W::TITER][8];  // the probe spectrum at this thread's Fourier samples
  auto load_spectrum = [&]() {
#pragma unroll
    for (int it = 0; it < W::TITER; ++it)
#pragma unroll
      for (int i = 0; i < 8; ++i) sp[it][i] = ld_cell(spec + p.fourier(w.lane + 32 * it, i));
  };
  int b = blockIdx.x;
  int row = a.amp_rows ? a.amp_rows[b] : b;
  int prow = kFull && a.pos_rows ? a.pos_rows[b] : b;
  load_spectrum();
  const float2 at = P::position(a, a.positions, b);
  bool pos_ok = p.locate(a, at.x, at.y, 0);
  nn::tc_fence_before();
  __syncthreads();
  nn::tc_fence_after();
  const uint32_t tm = tmem_base + ((uint32_t)(w.warp & 3) << 21) + (w.warp >> 2) * WORDS;
  bool first = true;

#pragma unroll 1
  for (int k = 0; b < a.B; k ^= 1) {
    const int next = b + gridDim.x;
    const bool cur_ok = pos_ok;
    // (a position behind the end is read as this one again)
    const int nb = next < a.B ? next : b;
    const int next_row = a.amp_rows ? a.amp_rows[nb] : nb;
    const int next_prow = a.pos_rows ? a.pos_rows[nb] : nb;
    float2 next_at;
    float2* const ew = ps ? a.exit_waves + (size_t)prow * N : nullptr;
    P cur = p;  // (patch corner of this position; p moves on to the next below)
    if (tid == 0) a.pos_round[b] = make_int2(p.x0, p.y0);
    // columns: spectrum x ramp, back to real space
#pragma unroll
    for (int it = 0; it < W::TITER; ++it) {
      const int t = w.lane + 32 * it;
      Cx2 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = mul(from_pair(sp[it][i]), p.ramp(t, i, k));
      fetch_amplitudes(row, it * (PARTS / W::TITER), PARTS / W::TITER);
      w.col_outer_store(t, v);
    }
    __syncwarp();
    w.col_inner_inverse();
    __syncthreads();
#pragma unroll 1
    for (int n = 0; n < 2; ++n) {
      // rows: n = 0 psi = P O, n = 1 adjoint terms; a task's patch is loaded while
      // the pass before it runs
      w.row_inner_inverse();
      __syncwarp();
#pragma unroll 1
      for (int it = 0; it < W::TITER; ++it) {
        const int t = w.lane + 32 * it;
        const uint32_t tp = tm + 32 * it, ta = tm + 32 * (W::TITER + it);
        Cx2 v[8], o[8];
        cur.load_patch(a, 0, t, 0, 0, o);
        w.row_outer_load(t, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = scale(v[i], invN);
        if (n == 0) {
          tmem_put(tp, v);
          // (staged here: the adjoint phase has the other stores)
          float* const nobj = a.st_nobj + (size_t)b * N;
#pragma unroll
          for (int i = 0; i < 8; ++i) st_two(nobj + p.real(t, i), abs2(v[i]));
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = mul(v[i], o[i]);
          if (ps) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const Cx2 wv = a.ew_valid ? from_pair(ld_cell(ew + p.real(t, i))) : v[i];
              v[i] = fma_r(wv, py_, scale(v[i], a.pc));
            }
          }
          w.row_outer_store(t, v);
          tmem_wait_store();
        } else {
          uint32_t pr[32];
          tmem_get(tp, pr);
          tmem_wait_load(pr);
          float2* const gobj = a.st_obj + (size_t)b * N;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int e = p.real(t, i);
            const Cx2 q = tmem_cell(pr, i);
            if (ps) {
              // new exit wave x w + a psi + b projected
              const Cx2 psi = mul(q, o[i]);
              const Cx2 wv = a.ew_valid ? from_pair(ld_cell(ew + e)) : psi;
              v[i] = fma_r(v[i], a.pb, fma_r(psi, a.pa, scale(wv, px_)));
              st_cell(ew + e, to_pair(v[i]));
            }
            Cx2 g = conj_mul(q, v[i]);
            if (a.potential) {
              // Re(-i conj(O) conj(P) chi)
              g.re = conj_mul(o[i], g).im;
              g.im = make_float2(0.0f, 0.0f);
            }
            st_cell(gobj + e, to_pair(g));
            v[i] = conj_mul(o[i], v[i]);
          }
          if (!first) {
            tmem_get(ta, pr);
            tmem_wait_load(pr);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = add(tmem_cell(pr, i), v[i]);
          }
          tmem_put(ta, v);
          tmem_wait_store();
        }
      }
      if (n == 1) break;
      __syncwarp();
      w.row_inner_forward();
      copy_async_wait();
      __syncthreads();
      next_at = make_float2(a.positions[2 * next_prow], a.positions[2 * next_prow + 1]);

      // columns: Fourier projection
      w.col_inner_forward();
      __syncwarp();
      float2 err2 = make_float2(0.0f, 0.0f);
#pragma unroll 1
      for (int it = 0; it < W::TITER; ++it) {
        const int t = w.lane + 32 * it;
        Cx2 v[8];
        w.col_outer_load(t, v);
        float2 A[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
          A[i] = ld_two(amps + ((t >> 2) + W::RI * i) * AP + 8 * w.warp + 2 * (t & 3));
        if (kFull && a.keep_farfield) {
          float2* const far = a.scratch_f + (size_t)b * N;
#pragma unroll
          for (int i = 0; i < 8; ++i) st_cell(far + p.fourier(t, i), to_pair(v[i]));
        }
        if (a.det_mask) apply_mask(p, a.det_mask, t, v);
        project(!ps, A, v, err2);
        if (a.det_mask && !ps) apply_mask(p, a.det_mask, t, v);
        w.col_outer_store(t, v);
      }
      __syncwarp();
      w.col_inner_inverse();
      float e = err2.x + err2.y;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
      if (w.lane == 0) red[w.warp] = e;
      __syncthreads();
      if (tid == 0) {
        float total = 0.0f;
        for (int i = 0; i < W::WARPS; ++i) total += red[i];
        a.err[b] = cur_ok ? total : __int_as_float(0x7fc00000);
      }
    }
    load_spectrum();
    if (next < a.B) pos_ok = p.locate(a, next_at.x, next_at.y, k ^ 1);
    row = next_row;
    prow = next_prow;
    __syncthreads();
    first = false;
    b = next;
  }
  // the block's summed probe terms
  float2* const out = a.st_probe + (size_t)blockIdx.x * N;
#pragma unroll 1
  for (int it = 0; it < W::TITER; ++it) {
    uint32_t r[32];
    tmem_get(tm + 32 * (W::TITER + it), r);
    tmem_wait_load(r);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      st_cell(out + p.real(w.lane + 32 * it, i), to_pair(tmem_cell(r, i)));
  }
  nn::tc_fence_before();
  __syncthreads();
  nn::tc_fence_after();
  if (w.warp == 0) nn::tmem_dealloc(tmem_base, COLS);
}

// Position correction of a single-slice batch: the expressions of
// position_correction_kernel. The shifted probe is transformed once per mode and
// waits in st_probe (which the batch's reductions have consumed) for the second
// direction. For a single probe at 128 x 128 (kTmem) the blocks are resident and
// the probe and the far field of the batch wait in tensor memory, the x derivative
// in shared memory. Bound: L2 traffic, 580 KB a position (1090 through memory).
// 128 x 128, 1024 positions: 191 us; through memory, with the sums of all threads
// in double: 303; the block-wide walk: 465.
template <int S, bool kTmem>
__global__ void __launch_bounds__(WaveFft<S>::NT) wave_correction_kernel(BatchArgs a) {
  using W = WaveFft<S>;
  using P = WavePosition<S>;
  constexpr int N = W::N;
  extern __shared__ float4 smem4[];
  __shared__ double sums[5];
  __shared__ uint32_t tmem_base;
  constexpr int WORDS = 64 * W::TITER;  // tensor-memory columns of a warp
  constexpr int COLS = WORDS * (W::WARPS / 4);
  static_assert(!kTmem || (W::TASKS % 32 == 0 && W::WARPS % 4 == 0 && COLS <= 512),
                "tensor memory");

  const int tid = threadIdx.x;
  const int M = kTmem ? 1 : a.M;
  P p;
  p.carve(smem4);
  p.w.tables(tid);
  uint32_t tm = 0;
  if constexpr (kTmem) {
    if (p.w.warp == 0) nn::tmem_alloc(&tmem_base, COLS);
    nn::tc_fence_before();
    __syncthreads();
    nn::tc_fence_after();
    tm = tmem_base + ((uint32_t)(p.w.warp & 3) << 21) + (p.w.warp >> 2) * WORDS;
  }
  // this thread's d|F|^2/dx samples, in its own slots
  float2* const own_gx = reinterpret_cast<float2*>(smem4 + P::CELLS);

#pragma unroll 1
  for (int b = blockIdx.x; b < a.B; b += gridDim.x) {
  const int prow = a.pos_rows ? a.pos_rows[b] : b;
  const int arow = a.amp_rows ? a.amp_rows[b] : b;
  const float2 at = P::position(a, a.positions_rw, b);
  const bool pos_ok = p.locate(a, at.x, at.y, 0);
  const float posx = finite_or_zero(at.x);
  const float posy = finite_or_zero(at.y);
  __syncthreads();

  const W& w = p.w;
  const float invN = 1.0f / (float)N;
  float* const gx = a.st_nobj + (size_t)b * N;
  float* const gy = a.st_nprobe + (size_t)b * N;
  const float* amp = a.amplitudes + (size_t)arow * N;
  // sums of the normal equations: float over the 16 samples of a task, as many as a
  // thread of the block-wide walk adds at 128 x 128
  float sxx = 0.f, sxy = 0.f, syy = 0.f, sxd = 0.f, syd = 0.f;
  float first[5] = {0.f, 0.f, 0.f, 0.f, 0.f};  // task 0's where a thread has two
  static_assert(W::TITER <= 2, "tasks of a thread");
#pragma unroll 1
  for (int m = 0; m < M; ++m) {
    const float2* __restrict__ spec = a.probe_spec + (size_t)m * N;
    const float2* __restrict__ f0 = a.scratch_f + ((size_t)b * M + m) * N;
    float2* const stash = a.st_probe + ((size_t)b * M + m) * N;
    // P_m shifted as in the forward pass
#pragma unroll 1
    for (int it = 0; it < W::TITER; ++it) {
      const int t = w.lane + 32 * it;
      if (W::TASKS % 32 != 0 && t >= W::TASKS) break;
      Cx2 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = from_pair(ld_cell(spec + p.fourier(t, i)));
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = mul(v[i], p.ramp(t, i));
      w.col_outer_store(t, v);
    }
    __syncwarp();
    w.col_inner_inverse();
    __syncthreads();
    w.row_inner_inverse();
    __syncwarp();
#pragma unroll 1
    for (int dir = 0; dir < 2; ++dir) {
      // times the object patch moved one pixel along x (dir 0) or y (dir 1)
#pragma unroll 1
      for (int it = 0; it < W::TITER; ++it) {
        const int t = w.lane + 32 * it;
        if (W::TASKS % 32 != 0 && t >= W::TASKS) break;
        Cx2 o[8], v[8];
        p.load_patch(a, 0, t, dir == 0 ? 1 : 0, dir, o);
        if (dir == 0) {
          w.row_outer_load(t, v);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            v[i] = scale(v[i], invN);
            if (!kTmem) st_cell(stash + p.real(t, i), as_cell(v[i]));
          }
          if constexpr (kTmem) {
            tmem_put(tm + 32 * it, v);
            tmem_wait_store();
          }
        } else if constexpr (kTmem) {
          uint32_t c[32];
          tmem_get(tm + 32 * it, c);
          tmem_wait_load(c);
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = tmem_cell(c, i);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = as_cx2(ld_cell(stash + p.real(t, i)));
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = mul(v[i], o[i]);
        w.row_outer_store(t, v);
      }
      __syncwarp();
      w.row_inner_forward();
      __syncthreads();
      w.col_inner_forward();
      __syncwarp();
      float* const g = dir == 0 ? gx : gy;
      const bool last = dir == 1 && m == M - 1;
#pragma unroll 1
      for (int it = 0; it < W::TITER; ++it) {
        const int t = w.lane + 32 * it;
        if (W::TASKS % 32 != 0 && t >= W::TASKS) break;
        Cx2 r[8], v[8];
        const uint32_t tf = tm + 32 * (W::TITER + it);
        if (W::TITER > 1 && last && it == 1) {
          first[0] = sxx;
          first[1] = sxy;
          first[2] = syy;
          first[3] = sxd;
          first[4] = syd;
          sxx = sxy = syy = sxd = syd = 0.f;
        }
        if (!kTmem || dir == 0) {
#pragma unroll
          for (int i = 0; i < 8; ++i) r[i] = from_pair(ld_cell(f0 + p.fourier(t, i)));
        }
        w.col_outer_load(t, v);
        if constexpr (kTmem) {
          if (dir == 0) {
            tmem_put(tf, r);
            tmem_wait_store();
          } else {
            uint32_t c[32];
            tmem_get(tf, c);
            tmem_wait_load(c);
#pragma unroll
            for (int i = 0; i < 8; ++i) r[i] = tmem_cell(c, i);
          }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int e = p.fourier(t, i);
          const Cx2 d = sub(r[i], v[i]);
          float2 u = __fmul2_rn(dup(2.0f), add2(__fmul2_rn(d.re, r[i].re),
                                                __fmul2_rn(d.im, r[i].im)));
          if (m > 0) u = add2(ld_two(g + e), u);
          float2& kept = own_gx[(8 * it + i) * W::NT + tid];
          if (!last) {
            if (kTmem) kept = u;
            else st_two(g + e, u);
            continue;
          }
          // the normal equations of this thread's samples
          float2 est = abs2(r[i]);
          for (int k = 0; k < M - 1; ++k)
            est = add2(est, abs2(from_pair(ld_cell(
                                a.scratch_f + ((size_t)b * M + k) * N + e))));
          const float2 A = __ldg(reinterpret_cast<const float2*>(amp + e));
          const float2 gv = kTmem ? kept : ld_two(gx + e);
          auto add_terms = [&](float px, float py, float d2) {
            sxx = fmaf(px, px, sxx);
            sxy = fmaf(px, py, sxy);
            syy = fmaf(py, py, syy);
            sxd = fmaf(px, d2, sxd);
            syd = fmaf(py, d2, syd);
          };
          add_terms(gv.x, u.x, __fsub_rn(__fmul_rn(A.x, A.x), est.x));
          add_terms(gv.y, u.y, __fsub_rn(__fmul_rn(A.y, A.y), est.y));
        }
      }
      __syncthreads();  // the wave is rewritten by rows (dir 1) or the next mode
    }
  }
  // the block's sums over the tasks' partials (the wave's shared memory is free by
  // now): a warp per sum, each lane adding its partials as a float and the sum of the
  // rounding errors (TwoSum, so about 46 bits), the lanes in double. (Partials added in
  // double cost 2.5 us a position with two tasks a thread: conversions and additions
  // run at a sixtieth of the float rate.)
  float* const part = reinterpret_cast<float*>(smem4);
  const float last_task[5] = {sxx, sxy, syy, sxd, syd};
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    part[k * W::NT + tid] = last_task[k];
    if (W::TITER > 1) part[(5 + k) * W::NT + tid] = first[k];
  }
  __syncthreads();
  for (int k = w.warp; k < 5; k += W::WARPS) {
    cis_detail::DF x{part[k * W::NT + w.lane], 0.0f};
#pragma unroll
    for (int j = 1; j < W::TITER * W::WARPS; ++j) {
      const cis_detail::DF t = cis_detail::two_sum(
          x.hi, part[(j / W::WARPS * 5 + k) * W::NT + 32 * (j % W::WARPS) + w.lane]);
      x = {t.hi, __fadd_rn(x.lo, t.lo)};
    }
    double sum = (double)x.hi + x.lo;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (w.lane == 0) sums[k] = sum;
  }
  __syncthreads();
  if (tid == 0) correction_update(a, prow, posx, posy, pos_ok, sums);
  }
  if constexpr (kTmem) {
    nn::tc_fence_before();
    __syncthreads();
    nn::tc_fence_after();
    if (p.w.warp == 0) nn::tmem_dealloc(tmem_base, COLS);
  }
}

// |P_b|^2 of the sub-pixel shifted probe (mode 0), as probe_intensity_kernel: the
// first two phases of the position kernel.
template <int S>
__global__ void __launch_bounds__(WaveFft<S>::NT) wave_intensity_kernel(BatchArgs a) {
  using W = WaveFft<S>;
  using P = WavePosition<S>;
  constexpr int N = W::N;
  extern __shared__ float4 smem4[];
  const int b = blockIdx.x;
  P p;
  p.carve(smem4);
  p.w.tables(threadIdx.x);
  const float2 at = P::position(a, a.positions, b);
  p.locate(a, at.x, at.y, 0);
  if (threadIdx.x == 0) a.pos_round[b] = make_int2(p.x0, p.y0);
  __syncthreads();
  const W& w = p.w;
  const float invN = 1.0f / (float)N;
#pragma unroll 1
  for (int it = 0; it < W::TITER; ++it) {
    const int t = w.lane + 32 * it;
    if (W::TASKS % 32 != 0 && t >= W::TASKS) break;
    Cx2 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = from_pair(ld_cell(a.probe_spec + p.fourier(t, i)));
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = mul(v[i], p.ramp(t, i));
    w.col_outer_store(t, v);
  }
  __syncwarp();
  w.col_inner_inverse();
  __syncthreads();
  w.row_inner_inverse();
  __syncwarp();
  float* const dst = a.st_nobj + (size_t)b * N;
#pragma unroll 1
  for (int it = 0; it < W::TITER; ++it) {
    const int t = w.lane + 32 * it;
    if (W::TASKS % 32 != 0 && t >= W::TASKS) break;
    Cx2 v[8];
    w.row_outer_load(t, v);
#pragma unroll
    for (int i = 0; i < 8; ++i) st_two(dst + p.real(t, i), abs2(scale(v[i], invN)));
  }
}

// The wider loads and stores of these kernels need the caller's arrays aligned
// (16-byte cells of the amplitudes, exit waves and propagators, float2 pairs of
// the mask); a batch whose pointers are not takes the general kernel. At 128 x 128
// amplitudes off the boundary are copied to one first (realign_amplitudes, 21 us per
// 1024 positions): an iteration of 4096 positions takes 1.16 ms that way (1.08 with
// aligned amplitudes, 1.55 in the general kernel), of 8 slices 9.98 (9.87, 13.6), of 4
// modes 6.36 (6.25, 7.24).
inline bool aligned_to(const void* p, size_t n) { return reinterpret_cast<size_t>(p) % n == 0; }
inline bool wave_aligned(const BatchArgs& a) {
  return (a.Sx == 128 || aligned_to(a.amplitudes, 16)) && aligned_to(a.det_mask, 8) &&
         aligned_to(a.exit_waves, 16) && aligned_to(a.props, 16);
}

// the amplitude rows of the batch, in order, to the aligned array `dst`
template <int N>
__global__ void __launch_bounds__(256) realign_kernel(const float* __restrict__ src,
                                                      const int* __restrict__ rows, float* dst) {
  const int b = blockIdx.x, e = 4 * (blockIdx.y * 256 + threadIdx.x);
  const float* s = src + (size_t)(rows ? rows[b] : b) * N + e;
  *reinterpret_cast<float4*>(dst + (size_t)b * N + e) = make_float4(s[0], s[1], s[2], s[3]);
}

// A batch with aligned amplitudes: `a` itself, or `a` reading the copy that is made in
// `room` (B S S floats that the kernel does not write before it has read them).
template <int S>
cudaError_t realign_amplitudes(BatchArgs& a, float* room, cudaStream_t s) {
  constexpr int N = S * S;
  if (S != 128 || aligned_to(a.amplitudes, 16)) return cudaSuccess;
  static_assert(N % 1024 == 0 || S != 128, "pieces of a row");
  realign_kernel<N><<<dim3(a.B, N / 1024), 256, 0, s>>>(a.amplitudes, a.amp_rows, room);
  a.amplitudes = room;
  a.amp_rows = nullptr;
  return cudaGetLastError();
}

// They also need room for the transmission copies in the workspace (a.trans;
// ptycho_workspace_bytes() includes it, a caller's workspace may hold less).
// Projection sets that keep the far field of psi (position correction) run the
// general kernel.
inline bool wave_batch(const BatchArgs& a) {
  return a.trans && wave_aligned(a) && !(a.projection && a.keep_farfield);
}

inline bool wave_mixed(const BatchArgs& a) { return a.M > 1 || (a.T == 1 && a.mixed_formula); }
inline bool wave_plain(const BatchArgs& a) {
  return !wave_mixed(a) && a.T == 1 && !a.projection && !a.forward_only && !a.keep_farfield &&
         !a.exact_probe_grad;
}

// One block per SM (its shared memory holds one wave of 128 x 128).
inline int resident_blocks(int B) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 0;
  return B < sms ? B : sms;
}

// Blocks of the resident single-slice single-probe kernel for this batch (the rows
// of st_probe that hold probe terms), 0 when the batch runs another kernel.
template <int S>
int wave_gd_blocks(const BatchArgs& a) {
  return S == 128 && !wave_mixed(a) && a.T == 1 && !a.forward_only && !a.exact_probe_grad
             ? resident_blocks(a.B)
             : 0;
}

template <int S>
cudaError_t launch_wave_position(BatchArgs a, cudaStream_t s) {
  using W = WaveFft<S>;
  int blocks = wave_gd_blocks<S>(a);
  const size_t smem = blocks > 0 ? sizeof(float4) * WavePosition<S>::CELLS + 4 * S * (S + 8)
                                 : WavePosition<S>::smem_bytes(true);
  void (*fn)(BatchArgs) = wave_mixed(a) ? wave_position_kernel<S, 2> : wave_position_kernel<S, 1>;
  if constexpr (S == 128) {
    if (blocks > 0) fn = wave_plain(a) ? wave_gd_kernel<S, false> : wave_gd_kernel<S, true>;
  } else if constexpr (S > 32) {
    if (wave_plain(a)) fn = wave_position_kernel<S, 0>;
  }
  cudaError_t e = ensure_smem_limit(reinterpret_cast<const void*>(fn), (int)smem);
  if (e != cudaSuccess) return e;
  if ((e = launch_transmission(a, s)) != cudaSuccess) return e;
  // (a position's |O|^2 go there after its amplitudes have been read, if at all)
  if ((e = realign_amplitudes<S>(a, a.st_nprobe, s)) != cudaSuccess) return e;
  timing_before(s);
  if (S == 128 && blocks == 0 && wave_mixed(a)) blocks = resident_blocks(a.B);
  fn<<<blocks > 0 ? blocks : a.B, W::NT, smem, s>>>(a);
  e = cudaGetLastError();
  timing_after(s);
  return e;
}

template <int S>
cudaError_t launch_wave_intensity(const BatchArgs& a, cudaStream_t s) {
  const size_t smem = WavePosition<S>::smem_bytes(false);
  const cudaError_t e =
      ensure_smem_limit(reinterpret_cast<const void*>(wave_intensity_kernel<S>), (int)smem);
  if (e != cudaSuccess) return e;
  wave_intensity_kernel<S><<<a.B, WaveFft<S>::NT, smem, s>>>(a);
  return cudaGetLastError();
}

template <int S>
cudaError_t launch_wave_correction(BatchArgs a, cudaStream_t s) {
  using W = WaveFft<S>;
  size_t smem = WavePosition<S>::smem_bytes(false);
  void (*fn)(BatchArgs) = wave_correction_kernel<S, false>;
  int blocks = a.B;
  if constexpr (S == 128) {
    if (a.M == 1 && resident_blocks(a.B) > 0) {
      fn = wave_correction_kernel<S, true>;
      smem = WavePosition<S>::smem_bytes(true);
      blocks = resident_blocks(a.B);
    }
  }
  cudaError_t e = ensure_smem_limit(reinterpret_cast<const void*>(fn), (int)smem);
  if (e != cudaSuccess) return e;
  if ((e = launch_transmission(a, s)) != cudaSuccess) return e;
  // (the object terms have been summed by now)
  if ((e = realign_amplitudes<S>(a, reinterpret_cast<float*>(a.st_obj), s)) != cudaSuccess)
    return e;
  fn<<<blocks, W::NT, smem, s>>>(a);
  return cudaGetLastError();
}

}  // namespace
}  // namespace pty
