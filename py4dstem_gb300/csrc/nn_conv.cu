// Convolution and elementwise kernels of the learned initializer (a BF16 U-Net
// that maps virtual bright-field and centre-of-mass images of a scan to an
// initial object phase). There is no counterpart in the reference.
//
// Activations are NHWC bfloat16 with a channel count that is a multiple of 8.
// The 3 x 3 convolutions (stride 1, zero padding 1) are implicit GEMMs on the
// tensor cores, from halo tiles in shared memory (nn_conv_tile.cuh) or, for image
// rows too wide for one, gathered by tc_gemm_kernel (tc_gemm.cuh):
//   forward         y[p, co]   = sum_{tap, ci} x[p + off(tap), ci] w[co, tap, ci]
//                   rows = pixels p, columns = co, K = 9 Cin
//   input gradient  dx[p, ci]  = sum_{tap, co} dy[p - off(tap), co] wt[ci, tap, co]
//                   rows = pixels, columns = ci, K = 9 Cout (wt: w transposed)
//   weight gradient dw[co, tap, ci] = sum_p dy[p, co] x[p + off(tap), ci]
//                   rows = (tap, ci), columns = co, K = pixels, split over K
//                   into fixed chunks whose partial sums are added in order
// with off(tap) = (tap / 3 - 1, tap % 3 - 1) in (y, x). Every reduction here is
// deterministic (no float atomics).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "nn_conv_tile.cuh"
#include "nn_internal.h"
#include "tc_gemm.cuh"

namespace pty {
namespace nn {
namespace {

constexpr int kEw = 256;  // threads of the elementwise kernels

__device__ __forceinline__ uint4 zero16() { return make_uint4(0u, 0u, 0u, 0u); }

// ------------------------------------------------------------ GEMM operands
struct RowMajorBf16 {  // rows x K, row-major
  const bf16* p;
  int rows, K;
  __device__ uint4 operator()(int r, int kc) const {
    if (r >= rows) return zero16();
    return *reinterpret_cast<const uint4*>(p + (size_t)r * K + 8 * kc);
  }
};

struct StoreF32 {  // C (M, N) row-major float
  float* c;
  int M, N;
  __device__ void operator()(int r, int c0, const float (&v)[16], int) const {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (c0 + i < N) c[(size_t)r * N + c0 + i] = v[i];
  }
};

struct Im2colFwd {  // rows = pixels, K = 9 Cin: 8 channels of one tap per chunk
  const bf16* x;
  int nb, H, W, C;
  __device__ uint4 operator()(int r, int kc) const {
    if (r >= nb * H * W) return zero16();
    const int k = 8 * kc;
    const int tap = k / C;
    const int ci = k - tap * C;
    const int xx = r % W;
    const int t = r / W;
    const int yy = t % H;
    const int n = t / H;
    const int sy = yy + tap / 3 - 1;
    const int sx = xx + tap % 3 - 1;
    if (sy < 0 || sy >= H || sx < 0 || sx >= W) return zero16();
    return *reinterpret_cast<const uint4*>(x + (((size_t)n * H + sy) * W + sx) * C + ci);
  }
};

struct Im2colBwdData {  // rows = pixels, K = 9 Cout: dy at p - off(tap)
  const bf16* dy;
  int nb, H, W, C;
  __device__ uint4 operator()(int r, int kc) const {
    if (r >= nb * H * W) return zero16();
    const int k = 8 * kc;
    const int tap = k / C;
    const int co = k - tap * C;
    const int xx = r % W;
    const int t = r / W;
    const int yy = t % H;
    const int n = t / H;
    const int sy = yy - (tap / 3 - 1);
    const int sx = xx - (tap % 3 - 1);
    if (sy < 0 || sy >= H || sx < 0 || sx >= W) return zero16();
    return *reinterpret_cast<const uint4*>(dy + (((size_t)n * H + sy) * W + sx) * C + co);
  }
};

// rows = (tap, ci) (9 Cin), K = pixels (8 consecutive pixels of one image row:
// the width is a multiple of 8)
struct Im2colWgradA {
  const bf16* x;
  int nb, H, W, C;
  __device__ uint4 operator()(int r, int kc) const {
    if (r >= 9 * C) return zero16();
    const int tap = r / C;
    const int ci = r - tap * C;
    const int p0 = 8 * kc;
    if (p0 >= nb * H * W) return zero16();
    const int x0 = p0 % W;
    const int t = p0 / W;
    const int yy = t % H;
    const int n = t / H;
    const int sy = yy + tap / 3 - 1;
    if (sy < 0 || sy >= H) return zero16();
    const int dx = tap % 3 - 1;
    const bf16* row = x + (((size_t)n * H + sy) * W) * C + ci;
    __align__(16) bf16 v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int sx = x0 + j + dx;
      v[j] = (sx >= 0 && sx < W) ? row[(size_t)sx * C] : __float2bfloat16(0.0f);
    }
    return *reinterpret_cast<const uint4*>(v);
  }
};

struct WgradB {  // rows = co, K = pixels: dy[p, co] for 8 consecutive pixels
  const bf16* dy;
  int npix, C;
  __device__ uint4 operator()(int r, int kc) const {
    if (r >= C) return zero16();
    const int p0 = 8 * kc;
    if (p0 >= npix) return zero16();
    __align__(16) bf16 v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = dy[(size_t)(p0 + j) * C + r];
    return *reinterpret_cast<const uint4*>(v);
  }
};

struct StoreActivation {  // y[p, co] = bf16(act(v + bias[co])), Cout a multiple of 16
  static constexpr bool kWarp = false;
  bf16* y;
  const float* bias;
  int Cout, relu;
  __device__ void operator()(int r, int c0, const float (&v)[16], int) const {
    __align__(16) bf16 o[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float t = v[i] + (bias ? bias[c0 + i] : 0.0f);
      if (relu) t = fmaxf(t, 0.0f);
      o[i] = __float2bfloat16(t);
    }
    uint4* dst = reinterpret_cast<uint4*>(y + (size_t)r * Cout + c0);
    dst[0] = reinterpret_cast<const uint4*>(o)[0];
    dst[1] = reinterpret_cast<const uint4*>(o)[1];
  }
};

struct StoreGradInput {  // dx[p, ci] (float), columns beyond Cin dropped
  float* dx;
  int Cin;
  bool whole;  // rows start on 16 bytes
  static constexpr bool kWarp = true;
  // a warp's 32 rows of 16 columns through shared memory, so that four lanes
  // write the 64 bytes of a row together (32 rows of 16 bytes each otherwise)
  __device__ void store(float* buf, int lane, int pixel, int c0, const float (&v)[16]) const {
#pragma unroll
    for (int i = 0; i < 16; i += 4)
      *reinterpret_cast<float4*>(buf + lane * kEpiPitch + i) =
          make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    __syncwarp();
    const int c = 4 * (lane & 3);
#pragma unroll
    for (int r = 0; r < 32; r += 8) {
      const int row = r + (lane >> 2);
      const int px = __shfl_sync(0xffffffffu, pixel, row);
      const float4 u = *reinterpret_cast<const float4*>(buf + row * kEpiPitch + c);
      if (px >= 0 && c0 + c < Cin) {
        float* dst = dx + (size_t)px * Cin + c0 + c;
        if (whole) {
          *reinterpret_cast<float4*>(dst) = u;
        } else {  // (Cin is a multiple of 8)
          dst[0] = u.x;
          dst[1] = u.y;
          dst[2] = u.z;
          dst[3] = u.w;
        }
      }
    }
    __syncwarp();
  }
  __device__ void operator()(int r, int c0, const float (&v)[16], int) const {
    float* dst = dx + (size_t)r * Cin + c0;
    if (whole) {
#pragma unroll
      for (int i = 0; i < 16; i += 4)
        if (c0 + i < Cin)
          *reinterpret_cast<float4*>(dst + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (c0 + i < Cin) dst[i] = v[i];
    }
  }
};

struct StoreWgradPartial {  // part[z][co][r] with r = (tap, ci)
  float* part;
  int rows, Cout;
  __device__ void operator()(int r, int c0, const float (&v)[16], int z) const {
    float* base = part + (size_t)z * Cout * rows;
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (c0 + i < Cout) base[(size_t)(c0 + i) * rows + r] = v[i];
  }
};

template <int BN, class LA, class LB, class EP>
cudaError_t launch_gemm(int M, int N, int K, int splits, int k_per_split, LA la, LB lb, EP ep,
                        int* err, cudaStream_t s) {
  auto kern = tc_gemm_kernel<BN, LA, LB, EP>;
  const int smem = GemmSmem<BN>::kBytes;
  cudaError_t e = ensure_smem_limit(reinterpret_cast<const void*>(kern), smem);
  if (e != cudaSuccess) return e;
  dim3 grid((M + kBM - 1) / kBM, (N + BN - 1) / BN, splits);
  kern<<<grid, kGemmThreads, smem, s>>>(M, N, K, k_per_split, la, lb, ep, err);
  return cudaGetLastError();
}

// Largest of 256/128/64/32 that divides n (n a multiple of 8 and >= 32), else 32.
int pick_bn(int n) {
  for (int bn : {256, 128, 64, 32})
    if (n % bn == 0) return bn;
  return 32;
}

template <class LA, class LB, class EP>
cudaError_t launch_gemm_bn(int bn, int M, int N, int K, int splits, int kps, LA la, LB lb, EP ep,
                           int* err, cudaStream_t s) {
  switch (bn) {
    case 256: return launch_gemm<256>(M, N, K, splits, kps, la, lb, ep, err, s);
    case 128: return launch_gemm<128>(M, N, K, splits, kps, la, lb, ep, err, s);
    case 64: return launch_gemm<64>(M, N, K, splits, kps, la, lb, ep, err, s);
    default: return launch_gemm<32>(M, N, K, splits, kps, la, lb, ep, err, s);
  }
}

// ------------------------------------------------------------ elementwise
constexpr int kReduceLanes = 32;              // outputs of a block
constexpr int kReduceGroups = kEw / kReduceLanes;

__global__ void __launch_bounds__(kEw) wgrad_reduce_kernel(const float* __restrict__ part,
                                                           int splits, size_t n, float* dw) {
  __shared__ float sums[kReduceGroups][kReduceLanes];
  const int lane = threadIdx.x % kReduceLanes, group = threadIdx.x / kReduceLanes;
  const size_t i = (size_t)blockIdx.x * kReduceLanes + lane;
  float s = 0.0f;
  if (i < n) {
#pragma unroll 8  // (the loads of 8 parts in flight, the sum in order)
    for (int z = group; z < splits; z += kReduceGroups) s += part[(size_t)z * n + i];
  }
  sums[group][lane] = s;
  __syncthreads();
  if (group == 0 && i < n) {
    for (int g = 1; g < kReduceGroups; ++g) s += sums[g][lane];
    dw[i] = s;
  }
}

// bias gradient: sum over pixels of dy[:, c]; one block per channel, fixed order
__global__ void bias_grad_kernel(const bf16* dy, int npix, int C, float* db) {
  __shared__ float red[kEw / 32];
  const int c = blockIdx.x;
  float s = 0.0f;
  for (int p = threadIdx.x; p < npix; p += kEw) s += __bfloat162float(dy[(size_t)p * C + c]);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.0f;
    for (int w = 0; w < kEw / 32; ++w) t += red[w];
    db[c] = t;
  }
}

}  // namespace

cudaError_t gemm_bf16(const bf16* a, const bf16* b, float* c, int M, int N, int K, int* err,
                      cudaStream_t s) {
  return launch_gemm_bn(pick_bn(N), M, N, K, 1, K, RowMajorBf16{a, M, K}, RowMajorBf16{b, N, K},
                        StoreF32{c, M, N}, err, s);
}

// Tile shape of the rows kernel: columns a block (all of them up to 128) and 128-row
// tiles a block, fewer of both while the launch would not give every SM a block;
// smem 0 when a row of the image is too wide for a tile (the gathered GEMM then).
struct RowsTile {
  int BN, G, buffers;
  size_t smem;
};

size_t rows_smem(int BN, int G, int pitch, int buffers) {
  const size_t P = tile_pixels(128 * G, pitch);
  const size_t need = buffers * (2 * P * 16 + 18 * (size_t)BN * 16) + 4 * P;
  const size_t epilogue = sizeof(float) * kTileThreads * kEpiPitch;
  return need > epilogue ? need : epilogue;
}

RowsTile rows_tile(const ConvLine& g, int C, int N) {
  const int stages = (C + kStageChannels - 1) / kStageChannels;
  RowsTile t{N <= 128 ? (N + 15) / 16 * 16 : 128, 4, stages < 3 ? (stages < 2 ? 2 : stages) : 3, 0};
  auto blocks = [&] {
    return ((g.Q + 128 * t.G - 1) / (128 * t.G)) * ((N + t.BN - 1) / t.BN);
  };
  auto smem = [&] { return rows_smem(t.BN, t.G, g.pitch, t.buffers); };
  while (t.G > 1 && (blocks() < 152 || t.G * t.BN > 256 || smem() > 110 * 1024)) t.G /= 2;
  while (t.BN > 32 && t.BN % 32 == 0 && blocks() < 152) t.BN /= 2;
  if (smem() > 220 * 1024) t.buffers = 2;
  t.smem = smem() <= 220 * 1024 ? smem() : 0;
  return t;
}

template <class Epi>
cudaError_t launch_rows(const bf16* x, const ConvLine& g, int C, const bf16* w, int N, int sign,
                        const RowsTile& t, Epi epi, int* err, cudaStream_t s) {
  auto kern = conv_rows_kernel<Epi>;
  const cudaError_t e = ensure_smem_limit(reinterpret_cast<const void*>(kern), (int)t.smem);
  if (e != cudaSuccess) return e;
  kern<<<dim3((g.Q + 128 * t.G - 1) / (128 * t.G), (N + t.BN - 1) / t.BN), kTileThreads, t.smem,
         s>>>(x, g, C, w, N, t.BN, t.G, t.buffers, sign, epi, err);
  return cudaGetLastError();
}

size_t wgrad_smem(int pitch, int buffers) {
  const size_t P = wgrad_pixels(kWgradPixels, pitch);
  return buffers * (kWgradRows / 8 * P * 16 + (size_t)kWgradColumns / 8 * kWgradPixels * 16) +
         4 * P;
}

// the padded line of pixels has to fit an int index
bool line_fits(int nb, int H, int W) {
  return (size_t)nb * ((size_t)H + 1) * ((size_t)W + 1) < (size_t)1 << 30;
}

cudaError_t conv3x3_forward(const bf16* x, int nb, int H, int W, int cin, const bf16* w,
                            const float* bias, int cout, int relu, bf16* y, int* err,
                            cudaStream_t s) {
  if (line_fits(nb, H, W)) {
    const ConvLine g = conv_line(nb, H, W);
    const RowsTile t = rows_tile(g, cin, cout);
    if (t.smem)
      return launch_rows(x, g, cin, w, cout, 1, t, StoreActivation{y, bias, cout, relu}, err, s);
  }
  const int M = nb * H * W;
  return launch_gemm_bn(pick_bn(cout), M, cout, 9 * cin, 1, 9 * cin,
                        Im2colFwd{x, nb, H, W, cin}, RowMajorBf16{w, cout, 9 * cin},
                        StoreActivation{y, bias, cout, relu}, err, s);
}

cudaError_t conv3x3_backward_data(const bf16* dy, int nb, int H, int W, int cout, const bf16* wt,
                                  int cin, float* dx, int* err, cudaStream_t s) {
  const bool whole = cin % 4 == 0 && reinterpret_cast<uintptr_t>(dx) % 16 == 0;
  if (line_fits(nb, H, W)) {
    const ConvLine g = conv_line(nb, H, W);
    const RowsTile t = rows_tile(g, cout, cin);
    if (t.smem)
      return launch_rows(dy, g, cout, wt, cin, -1, t, StoreGradInput{dx, cin, whole}, err, s);
  }
  const int M = nb * H * W;
  return launch_gemm_bn(pick_bn(cin), M, cin, 9 * cout, 1, 9 * cout,
                        Im2colBwdData{dy, nb, H, W, cout}, RowMajorBf16{wt, cin, 9 * cout},
                        StoreGradInput{dx, cin, whole}, err, s);
}

// Parts of the weight gradient (K chunks): of at least 2048 pixels, at most 64 of
// them, which any workspace holds; with room, one for every SM.
int wgrad_splits(int npix) {
  int splits = (npix + 2047) / 2048;
  return splits > 64 ? 64 : (splits < 1 ? 1 : splits);
}

size_t conv3x3_wgrad_workspace_min(int nb, int H, int W, int cin, int cout) {
  return sizeof(float) * (size_t)wgrad_splits(nb * H * W) * 9 * cin * cout;
}

size_t conv3x3_wgrad_workspace(int nb, int H, int W, int cin, int cout) {
  const size_t least = conv3x3_wgrad_workspace_min(nb, H, W, cin, cout);
  if (!line_fits(nb, H, W)) return least;  // (the gathered GEMM's parts)
  const int tiles = (nb * (H + 1) * (W + 1) + kWgradPixels - 1) / kWgradPixels;
  const int blocks = ((cin + kWgradRows - 1) / kWgradRows) *
                     ((cout + kWgradColumns - 1) / kWgradColumns);
  int splits = (152 + blocks - 1) / blocks;
  if (splits > tiles) splits = tiles;
  const size_t want = sizeof(float) * ((size_t)splits * 9 * cin * cout +
                                       (size_t)kBiasBlocks * cout);
  return want > least ? want : least;
}

cudaError_t conv3x3_backward_weight(const bf16* x, const bf16* dy, int nb, int H, int W, int cin,
                                    int cout, float* dw, float* db, float* part,
                                    size_t part_bytes, int* err, cudaStream_t s) {
  const int npix = nb * H * W;
  const int M = 9 * cin;
  const size_t n = (size_t)M * cout;
  const int buffers = wgrad_smem(W + 1, 2) <= 220 * 1024 ? 2 : 1;
  const size_t smem = wgrad_smem(W + 1, buffers);
  // the tile copies and the bias partials read 16 bytes at a time; x and dy that start
  // elsewhere take the gathered GEMM and the one-kernel bias sum, which read elements
  const bool x_aligned = reinterpret_cast<uintptr_t>(x) % 16 == 0;
  const bool dy_aligned = reinterpret_cast<uintptr_t>(dy) % 16 == 0;
  // bias partials first, then as many weight parts as fit
  const size_t bias_floats = (size_t)kBiasBlocks * cout;
  const bool bias_parts = dy_aligned && part_bytes / sizeof(float) >= bias_floats + n;
  float* wpart = part + (bias_parts ? bias_floats : 0);
  const size_t room = (part_bytes / sizeof(float) - (bias_parts ? bias_floats : 0)) / n;
  int splits;
  cudaError_t e;
  if (x_aligned && dy_aligned && line_fits(nb, H, W) && smem <= 220 * 1024) {
    const ConvLine g = conv_line(nb, H, W);
    const int tiles = (g.Q + kWgradPixels - 1) / kWgradPixels;
    const int bm = (cin + kWgradRows - 1) / kWgradRows;
    const int bn = (cout + kWgradColumns - 1) / kWgradColumns;
    splits = (152 + bm * bn - 1) / (bm * bn);
    if (splits > tiles) splits = tiles;
    if ((size_t)splits > room) splits = (int)room;
    if ((e = ensure_smem_limit(reinterpret_cast<const void*>(conv_wgrad_kernel), (int)smem)) !=
        cudaSuccess)
      return e;
    conv_wgrad_kernel<<<dim3(splits, bm, bn), kTileThreads, smem, s>>>(x, dy, g, cin, cout, buffers,
                                                                       wpart, err);
    e = cudaGetLastError();
  } else {
    splits = wgrad_splits(npix);
    if ((size_t)splits > room) splits = (int)room;
    int kps = (npix + splits - 1) / splits;
    kps = (kps + kBK - 1) / kBK * kBK;
    e = launch_gemm_bn(pick_bn(cout), M, cout, npix, splits, kps, Im2colWgradA{x, nb, H, W, cin},
                       WgradB{dy, npix, cout}, StoreWgradPartial{wpart, M, cout}, err, s);
  }
  if (e != cudaSuccess) return e;
  auto blocks = [](size_t v) { return (unsigned)((v + kReduceLanes - 1) / kReduceLanes); };
  wgrad_reduce_kernel<<<blocks(n), kEw, 0, s>>>(wpart, splits, n, dw);
  if (db) {
    if (bias_parts) {
      bias_partial_kernel<<<kBiasBlocks, kTileThreads, 0, s>>>(dy, npix, cout, part);
      wgrad_reduce_kernel<<<blocks(cout), kEw, 0, s>>>(part, kBiasBlocks, cout, db);
    } else {
      bias_grad_kernel<<<cout, kEw, 0, s>>>(dy, npix, cout, db);
    }
  }
  return cudaGetLastError();
}

}  // namespace nn
}  // namespace pty

// ------------------------------------------------------------------ C ABI
// (declared in include/ptycho_gb300.h; bf16 arrays are passed as raw 16-bit
// words)
#include "../../include/ptycho_gb300.h"

namespace {
int conv_shape_ok(int nb, int H, int W, int cin, int cout) {
  return nb >= 1 && H >= 1 && W >= 8 && W % 8 == 0 && cin >= 8 && cin % 8 == 0 && cout >= 16 &&
         cout % 16 == 0;
}
}  // namespace

extern "C" {

int ptycho_nn_gemm_bf16(const void* a, const void* b, float* c, int32_t m, int32_t n, int32_t k,
                        int32_t* err_flag, void* stream) {
  if (!a || !b || !c || !err_flag || m < 1 || n < 16 || n % 16 || k < 8 || k % 8)
    return PTYCHO_ERR_INVALID_ARGUMENT;
  using pty::nn::bf16;
  cudaError_t e = pty::nn::gemm_bf16(static_cast<const bf16*>(a), static_cast<const bf16*>(b), c,
                                     m, n, k, err_flag, static_cast<cudaStream_t>(stream));
  return e == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_CUDA;
}

int ptycho_nn_conv3x3_forward(const void* x, int32_t batch, int32_t height, int32_t width,
                              int32_t cin, const void* weight, const float* bias, int32_t cout,
                              int32_t relu, void* y, int32_t* err_flag, void* stream) {
  if (!x || !weight || !y || !err_flag || !conv_shape_ok(batch, height, width, cin, cout))
    return PTYCHO_ERR_INVALID_ARGUMENT;
  using pty::nn::bf16;
  cudaError_t e = pty::nn::conv3x3_forward(
      static_cast<const bf16*>(x), batch, height, width, cin, static_cast<const bf16*>(weight),
      bias, cout, relu ? 1 : 0, static_cast<bf16*>(y), err_flag, static_cast<cudaStream_t>(stream));
  return e == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_CUDA;
}

int ptycho_nn_conv3x3_backward_data(const void* dy, int32_t batch, int32_t height,
                                    int32_t width, int32_t cout, const void* weight_t,
                                    int32_t cin, float* dx, int32_t* err_flag, void* stream) {
  if (!dy || !weight_t || !dx || !err_flag || !conv_shape_ok(batch, height, width, cin, cout))
    return PTYCHO_ERR_INVALID_ARGUMENT;
  using pty::nn::bf16;
  cudaError_t e = pty::nn::conv3x3_backward_data(
      static_cast<const bf16*>(dy), batch, height, width, cout,
      static_cast<const bf16*>(weight_t), cin, dx, err_flag, static_cast<cudaStream_t>(stream));
  return e == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_CUDA;
}

size_t ptycho_nn_conv3x3_wgrad_workspace_bytes(int32_t batch, int32_t height, int32_t width,
                                               int32_t cin, int32_t cout) {
  if (!conv_shape_ok(batch, height, width, cin, cout)) return 0;
  return pty::nn::conv3x3_wgrad_workspace(batch, height, width, cin, cout);
}

int ptycho_nn_conv3x3_backward_weight(const void* x, const void* dy, int32_t batch,
                                      int32_t height, int32_t width, int32_t cin, int32_t cout,
                                      float* dweight, float* dbias, void* workspace,
                                      size_t workspace_bytes, int32_t* err_flag, void* stream) {
  if (!x || !dy || !dweight || !workspace || !err_flag ||
      !conv_shape_ok(batch, height, width, cin, cout))
    return PTYCHO_ERR_INVALID_ARGUMENT;
  if (workspace_bytes < pty::nn::conv3x3_wgrad_workspace_min(batch, height, width, cin, cout))
    return PTYCHO_ERR_WORKSPACE;
  using pty::nn::bf16;
  cudaError_t e = pty::nn::conv3x3_backward_weight(
      static_cast<const bf16*>(x), static_cast<const bf16*>(dy), batch, height, width, cin, cout,
      dweight, dbias, static_cast<float*>(workspace), workspace_bytes, err_flag,
      static_cast<cudaStream_t>(stream));
  return e == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_CUDA;
}

}  // extern "C"
