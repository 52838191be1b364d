// Volume operations of ptychographic tomography: rotating the (Z, Px, Py)
// potential volume into each tilt's frame, projecting it onto the multislice
// slices, expanding a slice update back onto the voxels, and the per-iteration
// volume constraints.
//
// Reference (py4DSTEM 0.14.18):
//   _rotate_zxy_volume      ptychographic_methods.py:849-868
//     scipy.ndimage.affine_transform(volume, tf, offset, order=3), mode
//     "constant" (cval 0), prefilter on, output in the input's type
//   _project_sliced_object  ptychographic_methods.py:783-812
//   _expand_sliced_object   ptychographic_methods.py:814-847
//   collective update, object constraints
//                           ptychographic_tomography.py:991-1240,
//                           ptychographic_constraints.py:60-118, 836-887
//
// Rotation. The volume is first turned into cubic B-spline coefficients, one
// separable recursive filter per axis (Unser, Aldroubi & Eden, "B-spline signal
// processing", IEEE Trans. Signal Process. 41 (1993); the single pole of the cubic
// spline z = sqrt(3) - 2 and gain (1 - z)(1 - 1/z)), with the exact initial values
// of a mirror-symmetric (whole-sample) extension. Each output voxel o then reads
// the input at c = offset + M o; a coordinate outside [0, n - 1] on any axis gives
// 0, otherwise the 4 x 4 x 4 cubic B-spline weights of c around floor(c) - 1
// combine the coefficients (indices mirrored at the edges). Float64 results run
// in float64, like SciPy's, float32 results in pairs of floats (below); where the
// face of the volume is decided the coordinate is formed in float64 as offset + m0 o0 + m1 o1 +
// m2 o2 in that order and without fused multiply-adds, so that the in/out
// decision at the volume's faces falls the same way as SciPy's.

#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "ptycho_internal.h"

namespace pty {
namespace {

constexpr int kThreads = 256;

struct Affine {
  double m[9];
  double off[3];
};

__global__ void volume_load_kernel(const void* in, int in_is_double, double* c, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    c[i] = in_is_double ? static_cast<const double*>(in)[i]
                        : (double)static_cast<const float*>(in)[i];
  }
}

// First sample and sample stride of line `line` along `axis` of (n0, n1, n2).
__device__ __forceinline__ void line_geometry(size_t line, int n1, int n2, int axis,
                                              size_t& base, size_t& stride) {
  if (axis == 0) {
    base = line;
    stride = (size_t)n1 * n2;
  } else if (axis == 1) {
    const size_t i0 = line / n2, i2 = line % n2;
    base = i0 * (size_t)n1 * n2 + i2;
    stride = n2;
  } else {
    base = line * (size_t)n2;
    stride = 1;
  }
}

// Cubic B-spline coefficients of one line of L >= 2 samples x[0], x[stride], ...
// in place: gain, causal recursion from the exact initial value of the
// mirror-symmetric extension (period 2L - 2: the sum over one period of z^k x_k
// divided by 1 - z^(2L-2)), anti-causal recursion from its initial value.
__device__ __forceinline__ void spline_line(double* x, size_t stride, int L) {
  const double z = __dadd_rn(sqrt(3.0), -2.0);
  const double gain = __dmul_rn(__dadd_rn(1.0, -z), __dadd_rn(1.0, -__ddiv_rn(1.0, z)));
  for (int i = 0; i < L; ++i) x[i * stride] = __dmul_rn(x[i * stride], gain);
  double zl = 1.0;
  for (int i = 0; i < L - 1; ++i) zl = __dmul_rn(zl, z);  // z^(L-1)
  double s = __dadd_rn(x[0], __dmul_rn(zl, x[(size_t)(L - 1) * stride]));
  double zi = z;
  for (int i = 1; i < L - 1; ++i) {
    const double pair = __dadd_rn(x[i * stride], __dmul_rn(zl, x[(size_t)(L - 1 - i) * stride]));
    s = __dadd_rn(s, __dmul_rn(zi, pair));
    zi = __dmul_rn(zi, z);
  }
  x[0] = __ddiv_rn(s, __dadd_rn(1.0, -__dmul_rn(zl, zl)));
  for (int i = 1; i < L; ++i)
    x[i * stride] = __dadd_rn(x[i * stride], __dmul_rn(z, x[(size_t)(i - 1) * stride]));
  const size_t last = (size_t)(L - 1) * stride;
  x[last] = __ddiv_rn(
      __dmul_rn(__dadd_rn(__dmul_rn(z, x[last - stride]), x[last]), z),
      __dadd_rn(__dmul_rn(z, z), -1.0));
  for (int i = L - 2; i >= 0; --i)
    x[i * stride] = __dmul_rn(z, __dadd_rn(x[(size_t)(i + 1) * stride], -x[i * stride]));
}

// One thread per line along `axis`, in global memory (lines too long to stage).
__global__ void spline_prefilter_kernel(double* c, int n0, int n1, int n2, int axis) {
  const int L = axis == 0 ? n0 : axis == 1 ? n1 : n2;
  const size_t lines = (size_t)n0 * n1 * n2 / (size_t)L;
  const size_t line = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (line >= lines || L < 2) return;
  size_t base, stride;
  line_geometry(line, n1, n2, axis, base, stride);
  spline_line(c + base, stride, L);
}

// Lines staged in shared memory: each warp of the block owns 32 consecutive
// lines, loaded and stored with coalesced accesses (row by row for the
// contiguous axis), and runs the recursions there. Sample i of the warp's line l
// sits at s[i * kLineLD + l]; the odd pitch spreads a row's samples over banks.
constexpr int kLineLD = 33;

__global__ void spline_prefilter_staged_kernel(double* c, int n0, int n1, int n2, int axis) {
  extern __shared__ double staged[];
  const int L = axis == 0 ? n0 : axis == 1 ? n1 : n2;
  const size_t lines = (size_t)n0 * n1 * n2 / (size_t)L;
  const int warps = blockDim.x / 32;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const size_t first = ((size_t)blockIdx.x * warps + warp) * 32;
  if (first >= lines || L < 2) return;  // the same for every lane of the warp
  double* s = staged + (size_t)warp * kLineLD * L;
  const size_t line = first + lane;
  const bool active = line < lines;
  const int nl = (int)(lines - first < 32 ? lines - first : 32);
  size_t base = 0, stride = 1;
  if (active) line_geometry(line, n1, n2, axis, base, stride);
  if (axis == 2) {
    for (int l = 0; l < nl; ++l) {
      const double* row = c + (first + l) * (size_t)n2;
      for (int i = lane; i < L; i += 32) s[i * kLineLD + l] = row[i];
    }
  } else if (active) {
    for (int i = 0; i < L; ++i) s[i * kLineLD + lane] = c[base + (size_t)i * stride];
  }
  __syncwarp();
  if (active) spline_line(s + lane, kLineLD, L);
  __syncwarp();
  if (axis == 2) {
    for (int l = 0; l < nl; ++l) {
      double* row = c + (first + l) * (size_t)n2;
      for (int i = lane; i < L; i += 32) row[i] = s[i * kLineLD + l];
    }
  } else if (active) {
    for (int i = 0; i < L; ++i) c[base + (size_t)i * stride] = s[i * kLineLD + lane];
  }
}

__device__ __forceinline__ int mirror_index(int i, int n) {
  if (n == 1) return 0;
  const int period = 2 * n - 2;
  i = i < 0 ? -i : i;
  i %= period;
  return i >= n ? period - i : i;
}

// Cubic B-spline weights of the four samples floor(x) - 1 .. floor(x) + 2.
__device__ __forceinline__ void cubic_weights(double t, double w[4]) {
  const double u = __dadd_rn(1.0, -t);
  const double t2 = __dmul_rn(t, t), u2 = __dmul_rn(u, u);
  const double sixth = __ddiv_rn(1.0, 6.0), two3 = __ddiv_rn(2.0, 3.0);
  w[0] = __dmul_rn(__dmul_rn(u2, u), sixth);
  w[1] = __dadd_rn(__dadd_rn(two3, -t2), __dmul_rn(__dmul_rn(t2, t), 0.5));
  w[2] = __dadd_rn(__dadd_rn(two3, -u2), __dmul_rn(__dmul_rn(u2, u), 0.5));
  w[3] = __dmul_rn(__dmul_rn(t2, t), sixth);
}

// out_mode 0: float32 out; 1: float64 out; 2: float32 out += value (the sum
// formed in float64 and rounded once).
__global__ void volume_affine_kernel(const double* __restrict__ c, void* out, int out_mode,
                                     int n0, int n1, int n2, Affine tf) {
  const size_t total = (size_t)n0 * n1 * n2;
  const int n[3] = {n0, n1, n2};
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x) {
    const double o[3] = {(double)(i / ((size_t)n1 * n2)), (double)((i / n2) % n1),
                         (double)(i % n2)};
    double x[3];
    bool inside = true;
#pragma unroll
    for (int h = 0; h < 3; ++h) {
      double v = tf.off[h];
#pragma unroll
      for (int l = 0; l < 3; ++l) v = __dadd_rn(v, __dmul_rn(tf.m[h * 3 + l], o[l]));
      x[h] = v;
      inside = inside && !(v < 0.0) && !(v > (double)(n[h] - 1));
    }
    double value = 0.0;
    if (inside) {
      int idx[3][4];
      double w[3][4];
#pragma unroll
      for (int h = 0; h < 3; ++h) {
        const double f = floor(x[h]);
        const int start = (int)f - 1;
        cubic_weights(__dadd_rn(x[h], -f), w[h]);
#pragma unroll
        for (int k = 0; k < 4; ++k) idx[h][k] = mirror_index(start + k, n[h]);
      }
      for (int a = 0; a < 4; ++a) {
        const size_t ra = (size_t)idx[0][a] * n1;
        for (int b = 0; b < 4; ++b) {
          const double wab = __dmul_rn(w[0][a], w[1][b]);
          const double* row = c + (ra + idx[1][b]) * n2;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            value = __dadd_rn(value, __dmul_rn(__dmul_rn(wab, w[2][k]), row[idx[2][k]]));
        }
      }
    }
    if (out_mode == 0) {
      static_cast<float*>(out)[i] = (float)value;
    } else if (out_mode == 1) {
      static_cast<double*>(out)[i] = value;
    } else {
      float* dst = static_cast<float*>(out) + i;
      *dst = (float)__dadd_rn((double)*dst, value);
    }
  }
}

// ---------------------------------------------------- float32 results: float pairs
// The same rotation for float32 results (out_mode 0 and 2) on the float32 units:
// every coefficient, weight, coordinate and sum is an unevaluated pair hi + lo of
// floats (about 46 bits), rounded once at the end. These are fewer bits than the 53
// of float64, in float64 input too: a result is within half an ulp and 1e-12 of the
// largest coefficient of the exact one (a coordinate near 100 carries an error of
// about 1e-12), so where a value is small against its neighbours' coefficients it can
// be another float than float64 arithmetic gives. Over 25 volumes of 24 x 40 x 40 to
// 96 x 160 x 160 voxels, 221 of 2.1e7 results are, by at most 9e-9 of the largest value, and the
// error against 64 bits is that of the final rounding either way (ratio 1.000000).
// The sums and products are the error-free transformations TwoSum (Knuth) and
// TwoProduct with a fused multiply-add (Ogita, Rump and Oishi 2005).
// GB300 does 60 times as many float32 as float64 operations: 96 x 160 x 160 voxels
// took 1286 us of resampling and 3 x 98 us of prefilters in float64.
//
// The coefficients carry a factor 2^-9. With the gain of the filters (6 per axis,
// 216 in all, applied first) the causal recursion reaches 216 / (1 - |pole|) = 295
// times the largest voxel and the anticausal one adds at most 108 to that: 403, so
// every finite float volume stays in range. Below about 1e-28 the error terms of the
// pairs run out of exponents: there the error is up to 2^-135.
constexpr float kPairScale = 512.0f;

__device__ __forceinline__ float2 pair_of(double v) {
  const float hi = (float)v;
  return make_float2(hi, (float)(v - (double)hi));
}
__device__ __forceinline__ float2 pair_renorm(float a, float b) {  // |a| >= |b|
  const float s = __fadd_rn(a, b);
  return make_float2(s, __fsub_rn(b, __fsub_rn(s, a)));
}
__device__ __forceinline__ float2 pair_sum(float a, float b) {  // a + b exactly
  const float s = __fadd_rn(a, b);
  const float t = __fsub_rn(s, a);
  return make_float2(s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t)));
}
__device__ __forceinline__ float2 pair_add(float2 a, float2 b) {
  const float2 s = pair_sum(a.x, b.x);
  return pair_renorm(s.x, __fadd_rn(s.y, __fadd_rn(a.y, b.y)));
}
__device__ __forceinline__ float2 pair_neg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 pair_mul(float2 a, float2 b) {
  const float p = __fmul_rn(a.x, b.x);
  float e = __fmaf_rn(a.x, b.x, -p);
  e = __fmaf_rn(a.x, b.y, e);
  e = __fmaf_rn(a.y, b.x, e);
  return pair_renorm(p, e);
}
// s += w c, s.y collecting the rounding errors
__device__ __forceinline__ void pair_accumulate(float2& s, float2 w, float2 c) {
  const float p = __fmul_rn(w.x, c.x);
  float e = __fmaf_rn(w.x, c.x, -p);
  e = __fmaf_rn(w.x, c.y, e);
  e = __fmaf_rn(w.y, c.x, e);
  const float2 t = pair_sum(s.x, p);
  s = make_float2(t.x, __fadd_rn(s.y, __fadd_rn(t.y, e)));
}

constexpr double kPole = -0.26794919243112270647;  // sqrt(3) - 2
constexpr float2 pair_constant(double v) { return {(float)v, (float)(v - (double)(float)v)}; }

// The axes in the order the coefficients are stored: (p, q) and the innermost h.
struct Axes {
  int p, q, h;
  int n[3];  // extents in that order
};

// Cubic B-spline recursions (see spline_line) along a line of L >= 2 pairs at
// s[i * kLineLD], the gain already applied. The sum that starts the causal filter
// ends after 40 terms (pole^40 = 1.4e-23).
__device__ __forceinline__ void spline_line_pairs(float2* s, int L) {
  constexpr float2 z = pair_constant(kPole);
  constexpr float2 last = pair_constant(kPole / (kPole * kPole - 1.0));
  const int period = 2 * L - 2;
  const int terms = period < 40 ? period : 40;
  auto mirrored = [&](int i) { return s[(i < L ? i : period - i) * kLineLD]; };
  float2 y = mirrored(terms - 1);
  for (int i = terms - 2; i >= 0; --i) y = pair_add(pair_mul(z, y), mirrored(i));
  if (period <= 40) {
    double zp = 1.0;
    for (int i = 0; i < period; ++i) zp *= kPole;
    y = pair_mul(y, pair_of(1.0 / (1.0 - zp)));
  }
  s[0] = y;
  float2 before = y;
  for (int i = 1; i < L; ++i) {
    before = y;
    y = pair_add(s[i * kLineLD], pair_mul(z, y));
    s[i * kLineLD] = y;
  }
  y = pair_mul(pair_add(pair_mul(z, before), y), last);
  s[(L - 1) * kLineLD] = y;
  for (int i = L - 2; i >= 0; --i) {
    y = pair_mul(z, pair_add(y, pair_neg(s[i * kLineLD])));
    s[i * kLineLD] = y;
  }
}

// One prefilter pass; a warp owns 32 lines in shared memory as in
// spline_prefilter_staged_kernel. axis 2 (the first pass) reads the volume `in`
// (float32 or float64, its own axis order), applies the gain and writes c in the
// order of `ax`; axes 0 and 1 of that order then run in place on c. Bound: the
// dependent pair operations of a line (about 60 cycles a sample and direction).
__global__ void __launch_bounds__(32) pair_prefilter_kernel(const void* __restrict__ in,
                                                            int in_is_double, float2* c, Axes ax,
                                                            size_t stride_p, size_t stride_q,
                                                            size_t stride_h, int axis,
                                                            float gain) {
  extern __shared__ float2 lines2[];
  const int lane = threadIdx.x;
  const int n0 = ax.n[0], n1 = ax.n[1], n2 = ax.n[2];
  const int L = ax.n[axis];
  const size_t lines = (size_t)n0 * n1 * n2 / (size_t)L;
  const size_t first = (size_t)blockIdx.x * 32;
  const size_t line = first + lane;
  const bool active = line < lines;
  const int nl = (int)(lines - first < 32 ? lines - first : 32);
  auto load = [&](size_t at) {
    return in_is_double
               ? pair_of(static_cast<const double*>(in)[at] * (double)gain)
               : pair_mul(make_float2(static_cast<const float*>(in)[at], 0.0f),
                          make_float2(gain, 0.0f));
  };
  size_t base = 0, stride = 1;
  if (axis == 2) {
    if (stride_h == 1) {  // lines are rows of the volume
      for (int l = 0; l < nl; ++l) {
        const size_t row = (first + l) / n1 * stride_p + (first + l) % n1 * stride_q;
        for (int i = lane; i < L; i += 32) lines2[i * kLineLD + l] = load(row + i);
      }
    } else if (active) {
      base = line / n1 * stride_p + line % n1 * stride_q;
      for (int i = 0; i < L; ++i) lines2[i * kLineLD + lane] = load(base + i * stride_h);
    }
  } else if (active) {
    line_geometry(line, n1, n2, axis, base, stride);
    for (int i = 0; i < L; ++i) lines2[i * kLineLD + lane] = c[base + (size_t)i * stride];
  }
  __syncwarp();
  if (active && L >= 2) spline_line_pairs(lines2 + lane, L);
  __syncwarp();
  if (axis == 2) {
    for (int l = 0; l < nl; ++l)
      for (int i = lane; i < L; i += 32) c[(first + l) * (size_t)L + i] = lines2[i * kLineLD + l];
  } else if (active) {
    for (int i = 0; i < L; ++i) c[base + (size_t)i * stride] = lines2[i * kLineLD + lane];
  }
}

// The indices of the four taps from `start`, mirrored at the edges (start >= -1,
// start + 3 <= n + 1).
__device__ __forceinline__ void mirror_taps(int start, int n, int (&idx)[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    int i = abs(start + k);
    if (i >= n) i = abs(2 * n - 2 - i);
    idx[k] = n == 1 ? 0 : i;
  }
}

__device__ __forceinline__ void cubic_weights(float2 t, float2 (&w)[4]) {
  constexpr float2 sixth = pair_constant(1.0 / 6.0), two3 = pair_constant(2.0 / 3.0);
  const float2 u = pair_add(make_float2(1.0f, 0.0f), pair_neg(t));
  const float2 t2 = pair_mul(t, t), u2 = pair_mul(u, u);
  const float2 t3 = pair_mul(t2, t), u3 = pair_mul(u2, u);
  auto half = [](float2 a) { return make_float2(0.5f * a.x, 0.5f * a.y); };
  w[0] = pair_mul(u3, sixth);
  w[1] = pair_add(pair_add(two3, pair_neg(t2)), half(t3));
  w[2] = pair_add(pair_add(two3, pair_neg(u2)), half(u3));
  w[3] = pair_mul(t3, sixth);
}

// Resampling of the pair coefficients; out_mode 0 or 2. A warp walks a row along
// the stored innermost axis h, chosen so that its samples read neighbouring
// coefficients (the axis of a tilt, where there is one). The sum is separable (84
// multiply-adds a voxel). A voxel within 1e-6 of a face takes the float64
// coordinate of volume_affine_kernel, whose rounding decides whether it is inside.
__global__ void __launch_bounds__(kThreads) pair_affine_kernel(const float2* __restrict__ c,
                                                               float* __restrict__ out,
                                                               int out_mode, Axes ax, int m0,
                                                               int m1, int m2, Affine tf) {
  const int lane = threadIdx.x & 31;
  const size_t rows = (size_t)ax.n[0] * ax.n[1];
  const int axis[3] = {ax.p, ax.q, ax.h};
  const size_t stride[3] = {(size_t)m1 * m2, (size_t)m2, 1};
  for (size_t row = ((size_t)blockIdx.x * kThreads + threadIdx.x) >> 5; row < rows;
       row += (size_t)gridDim.x * (kThreads / 32)) {
    const int op = (int)(row / ax.n[1]), oq = (int)(row % ax.n[1]);
    float2 base[3], slope[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const double* m = tf.m + 3 * axis[r];
      base[r] = pair_of(tf.off[axis[r]] + m[ax.p] * (double)op + m[ax.q] * (double)oq);
      slope[r] = pair_of(m[ax.h]);
    }
    const size_t out_row = op * stride[ax.p] + oq * stride[ax.q];
    for (int oh = lane; oh < ax.n[2]; oh += 32) {
      bool inside = true, near = false;
      int idx[3][4];
      float2 w[3][4];
      float2 t[3];
      int start[3];
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const float2 x = pair_add(base[r], pair_mul(slope[r], make_float2((float)oh, 0.0f)));
        const float end = (float)(ax.n[r] - 1);
        const float above = __fadd_rn(x.x, x.y);
        const float below = __fadd_rn(__fsub_rn(end, x.x), -x.y);
        near = near || fabsf(above) < 1e-6f || fabsf(below) < 1e-6f;
        inside = inside && above >= 0.0f && below >= 0.0f;
        const float f = floorf(x.x);
        t[r] = pair_sum(__fsub_rn(x.x, f), x.y);
        start[r] = (int)f - 1;
        if (t[r].x < 0.0f) {  // hi is whole, lo negative
          t[r] = pair_add(t[r], make_float2(1.0f, 0.0f));
          --start[r];
        }
      }
      if (near) {
        double o[3];
        o[ax.p] = op;
        o[ax.q] = oq;
        o[ax.h] = oh;
        inside = true;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          double v = tf.off[axis[r]];
#pragma unroll
          for (int l = 0; l < 3; ++l) v = __dadd_rn(v, __dmul_rn(tf.m[axis[r] * 3 + l], o[l]));
          inside = inside && !(v < 0.0) && !(v > (double)(ax.n[r] - 1));
          const double f = floor(v);
          t[r] = pair_of(v - f);
          start[r] = (int)f - 1;
        }
      }
      float2 value = make_float2(0.0f, 0.0f);
      if (inside) {
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          cubic_weights(t[r], w[r]);
          mirror_taps(start[r], ax.n[r], idx[r]);
        }
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          float2 plane = make_float2(0.0f, 0.0f);
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const float2* line = c + ((size_t)idx[0][a] * ax.n[1] + idx[1][b]) * ax.n[2];
            float2 sum = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int k = 0; k < 4; ++k) pair_accumulate(sum, w[2][k], __ldg(line + idx[2][k]));
            pair_accumulate(plane, w[1][b], sum);
          }
          pair_accumulate(value, w[0][a], plane);
        }
      }
      const float hi = kPairScale * value.x, lo = kPairScale * value.y;
      float* dst = out + out_row + oh * stride[ax.h];
      if (out_mode == 0) {
        *dst = __fadd_rn(hi, lo);
      } else if (fabsf(hi) < 1e38f && fabsf(*dst) < 1e38f) {
        const float2 sum = pair_sum(*dst, hi);
        *dst = __fadd_rn(sum.x, __fadd_rn(sum.y, lo));
      } else {  // (TwoSum is not for sums beyond the float range)
        *dst = (float)((double)*dst + (double)kPairScale * ((double)value.x + (double)value.y));
      }
    }
  }
}

// sliced[t] = volume[t*vps] + volume[t*vps + 1] + ... (float32, in voxel order;
// voxels past the end count as the zero padding of the reference).
__global__ void volume_project_kernel(const float* __restrict__ vol, int n0, int T, size_t P,
                                      int vps, float* __restrict__ sliced) {
  const size_t total = (size_t)T * P;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x) {
    const int t = (int)(i / P);
    const size_t p = i % P;
    float s = 0.0f;
    for (int k = 0; k < vps; ++k) {
      const int zz = t * vps + k;
      const float v = zz < n0 ? vol[(size_t)zz * P + p] : 0.0f;
      s = k == 0 ? v : __fadd_rn(s, v);
    }
    sliced[i] = s;
  }
}

// Voxel z of slice t = z / vps receives (sliced - sliced_old)[t] / count_t in
// float64 (count_t = vps, or the remainder for the last slice), one division per
// slice pixel. out_mode 1: float64 out; 2: float32 out += value.
__global__ void volume_expand_kernel(const float* __restrict__ sliced,
                                     const float* __restrict__ old, int n0, size_t P, int vps,
                                     int T, int last_count, void* out, int out_mode) {
  const size_t total = (size_t)T * P;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x) {
    const int t = (int)(i / P);
    const size_t p = i % P;
    const float u = __fsub_rn(sliced[i], old[i]);
    const double v = __ddiv_rn((double)u, (double)(t == T - 1 ? last_count : vps));
    const int end = min(n0, (t + 1) * vps);
    for (int zz = t * vps; zz < end; ++zz) {
      if (out_mode == 1) {
        static_cast<double*>(out)[(size_t)zz * P + p] = v;
      } else {
        float* dst = static_cast<float*>(out) + (size_t)zz * P + p;
        *dst = (float)__dadd_rn((double)*dst, v);
      }
    }
  }
}

__global__ void volume_add_scaled_kernel(float* vol, const float* addend, size_t n, float div) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    vol[i] = __fadd_rn(vol[i], __fdiv_rn(addend[i], div));
}

__global__ void volume_constraints_kernel(float* vol, size_t n, float shrinkage,
                                          int apply_shrinkage, int positivity) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    float v = vol[i];
    if (apply_shrinkage) v = __fsub_rn(v, shrinkage);
    if (positivity && v < 0.0f) v = 0.0f;
    vol[i] = v;
  }
}

unsigned grid_for(size_t n) {
  const size_t blocks = (n + kThreads - 1) / kThreads;
  return (unsigned)(blocks < 152 * 16 ? (blocks ? blocks : 1) : 152 * 16);
}

cudaError_t launch_rotate_pairs(const void* in, int in_is_double, float* out, int out_mode,
                                const int* n, const Affine& tf, float2* c, cudaStream_t s) {
  // the stored innermost axis: the one along which an output step is nearest to
  // an input step of the same axis (the last on equal terms)
  int h = 2;
  for (int k = 1; k >= 0; --k)
    if (fabs(tf.m[4 * k]) > fabs(tf.m[4 * h]) && n[k] >= 32) h = k;
  Axes ax;
  ax.h = h;
  ax.p = h == 0 ? 1 : 0;
  ax.q = h == 2 ? 1 : 2;
  ax.n[0] = n[ax.p];
  ax.n[1] = n[ax.q];
  ax.n[2] = n[h];
  const size_t stride[3] = {(size_t)n[1] * n[2], (size_t)n[2], 1};
  const size_t total = (size_t)n[0] * n[1] * n[2];
  float gain = 1.0f / kPairScale;
  for (int k = 0; k < 3; ++k)
    if (n[k] >= 2) gain *= 6.0f;
  for (int axis = 2; axis != -1; axis = axis == 2 ? 0 : axis == 0 ? 1 : -1) {
    const int L = ax.n[axis];
    if (axis != 2 && L < 2) continue;
    const size_t lines = total / (size_t)L;
    pair_prefilter_kernel<<<(unsigned)((lines + 31) / 32), 32, sizeof(float2) * kLineLD * L, s>>>(
        in, in_is_double, c, ax, stride[ax.p], stride[ax.q], stride[ax.h], axis, gain);
  }
  const size_t rows = (size_t)ax.n[0] * ax.n[1];
  pair_affine_kernel<<<grid_for(rows * 32), kThreads, 0, s>>>(c, out, out_mode, ax, n[0], n[1],
                                                              n[2], tf);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_volume_rotate(const void* in, int in_is_double, void* out, int out_mode,
                                 int n0, int n1, int n2, const double* matrix,
                                 const double* offset, double* scratch, cudaStream_t s) {
  const size_t total = (size_t)n0 * n1 * n2;
  Affine tf;
  for (int k = 0; k < 9; ++k) tf.m[k] = matrix[k];
  for (int k = 0; k < 3; ++k) tf.off[k] = offset[k];
  int smem_optin = 0;
  {
    // the staged prefilter may use up to the device's opt-in limit of dynamic
    // shared memory; the attribute is set per device
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess)
      e = cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess)
      e = ensure_smem_limit(reinterpret_cast<const void*>(spline_prefilter_staged_kernel),
                            smem_optin);
    if (e == cudaSuccess)
      e = ensure_smem_limit(reinterpret_cast<const void*>(pair_prefilter_kernel), smem_optin);
    if (e != cudaSuccess) return e;
  }
  const int n[3] = {n0, n1, n2};
  const int longest = n0 > n1 ? (n0 > n2 ? n0 : n2) : (n1 > n2 ? n1 : n2);
  // float32 results in float pairs, unless a line does not fit in shared memory
  if (out_mode != 1 && sizeof(float2) * kLineLD * (size_t)longest <= (size_t)smem_optin)
    return launch_rotate_pairs(in, in_is_double, static_cast<float*>(out), out_mode, n, tf,
                               reinterpret_cast<float2*>(scratch), s);
  volume_load_kernel<<<grid_for(total), kThreads, 0, s>>>(in, in_is_double, scratch, total);
  for (int axis = 0; axis < 3; ++axis) {
    if (n[axis] < 2) continue;
    const size_t lines = total / (size_t)n[axis];
    const size_t per_warp = sizeof(double) * kLineLD * (size_t)n[axis];
    if (per_warp <= (size_t)smem_optin) {
      int warps = 4;
      while (warps > 1 && (size_t)warps * per_warp > (size_t)smem_optin) warps /= 2;
      const size_t per_block = (size_t)warps * 32;
      spline_prefilter_staged_kernel<<<(unsigned)((lines + per_block - 1) / per_block),
                                       warps * 32, warps * per_warp, s>>>(scratch, n0, n1, n2,
                                                                          axis);
    } else {
      spline_prefilter_kernel<<<(unsigned)((lines + 127) / 128), 128, 0, s>>>(scratch, n0, n1,
                                                                             n2, axis);
    }
  }
  volume_affine_kernel<<<grid_for(total), kThreads, 0, s>>>(scratch, out, out_mode, n0, n1, n2,
                                                            tf);
  return cudaGetLastError();
}

cudaError_t launch_volume_project(const float* vol, int n0, size_t P, int T, float* sliced,
                                  cudaStream_t s) {
  const int vps = (n0 + T - 1) / T;
  volume_project_kernel<<<grid_for((size_t)T * P), kThreads, 0, s>>>(vol, n0, T, P, vps,
                                                                     sliced);
  return cudaGetLastError();
}

cudaError_t launch_volume_expand(const float* sliced, const float* old, int T, int n0, size_t P,
                                 void* out, int out_mode, cudaStream_t s) {
  const int vps = (n0 + T - 1) / T;
  const int rem = vps - (vps * T - n0);
  const int last_count = rem > 0 ? rem : vps;
  volume_expand_kernel<<<grid_for((size_t)T * P), kThreads, 0, s>>>(sliced, old, n0, P, vps, T,
                                                                    last_count, out, out_mode);
  return cudaGetLastError();
}

cudaError_t launch_volume_add_scaled(float* vol, const float* addend, size_t n, int divisor,
                                     cudaStream_t s) {
  volume_add_scaled_kernel<<<grid_for(n), kThreads, 0, s>>>(vol, addend, n, (float)divisor);
  return cudaGetLastError();
}

cudaError_t launch_volume_constraints(float* vol, size_t n, float shrinkage, int apply_shrinkage,
                                      int positivity, cudaStream_t s) {
  volume_constraints_kernel<<<grid_for(n), kThreads, 0, s>>>(vol, n, shrinkage, apply_shrinkage,
                                                             positivity);
  return cudaGetLastError();
}

}  // namespace pty
