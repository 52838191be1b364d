// 3 x 3 convolutions on the tensor cores from halo tiles held once in shared
// memory.
//
// The images of a batch are laid end to end as one line of pixels with one zero
// column after each row and one zero row after each image: pixel (n, y, x) is
// q = (n (H + 1) + y) (W + 1) + x, and the neighbour of every tap is q + dy (W + 1)
// + dx, with zeros outside. A tile is a run of consecutive q with (W + 2) more on
// each side. In shared memory eight channels of a pixel are 16 bytes and the
// pixels of a channel chunk follow one another, [chunk][pixel][8]: this is the
// canonical layout of an operand without swizzle whose row groups are 128 bytes
// apart, and because it has no gaps, starting it dy (W + 1) + dx pixels (x 16
// bytes) further gives the operand of that tap. So one copy of the tile serves all
// nine taps; the gathered implicit GEMM that this replaces copied it nine times,
// element by element for the weight gradient (16 images of 128 x 128, 96 -> 32
// channels: 240 us forward, 384 us input gradient, 620 us weight gradient).
//
//   forward, input gradient   rows = pixels (K-major operand), K = channels of a tap
//   weight gradient           rows = input channels, columns = output channels,
//                             K = pixels (both operands MN-major, same layout); one
//                             accumulator per tap
//
// Bound: the copy of the tiles from L2 (about twice the input) and, for narrow
// layers, the A operand's 4 KB per MMA. Every wait is bounded as in tc_gemm.cuh.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "nn_internal.h"
#include "tc_gemm.cuh"

namespace pty {
namespace nn {
namespace {

constexpr int kTileThreads = 256;
constexpr int kStageChannels = 16;  // channels of one pipeline stage (one MMA of K)

struct ConvLine {
  int nb, H, W;
  int pitch;  // W + 1
  int Q;      // nb (H + 1) (W + 1)
};

__host__ inline ConvLine conv_line(int nb, int H, int W) {
  return ConvLine{nb, H, W, W + 1, nb * (H + 1) * (W + 1)};
}

// index of the image pixel at q, -1 for the zeros
__device__ __forceinline__ int line_pixel(const ConvLine& g, int q) {
  if (q < 0 || q >= g.Q) return -1;
  const int r = q / g.pitch, x = q - r * g.pitch;
  const int n = r / (g.H + 1), y = r - n * (g.H + 1);
  return x < g.W && y < g.H ? (n * g.H + y) * g.W + x : -1;
}

// pixels of a tile of `rows` with its halo, = 4 mod 8 so that the two chunks of a
// stage fall into different banks
__host__ __device__ constexpr int tile_pixels(int rows, int pitch) {
  return (rows + 2 * (pitch + 1) + 3) / 8 * 8 + 4;
}

// 16 bytes from global to shared memory, zeros when !valid
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src),
               "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
}

__host__ __device__ constexpr int tmem_columns(int n) {
  return n <= 32 ? 32 : n <= 64 ? 64 : n <= 128 ? 128 : n <= 256 ? 256 : 512;
}

// Rows = pixels. Each block computes G x 128 consecutive q and BN columns (a
// multiple of 16) over all channels: stage = 16 channels of the tile and of the
// weights of the nine taps, two stages in flight. w: (N, 9, C). sign +1 reads x at
// q + off(tap), -1 at q - off(tap). epi(pixel, column, v[16]) receives the sums.
template <class Epi>
__global__ void __launch_bounds__(kTileThreads) conv_rows_kernel(const bf16* __restrict__ x,
                                                                 ConvLine g, int C,
                                                                 const bf16* __restrict__ w,
                                                                 int N, int BN, int G, int sign,
                                                                 Epi epi, int* err) {
  extern __shared__ __align__(1024) unsigned char tile_smem[];
  __shared__ uint64_t bar[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int P = tile_pixels(128 * G, g.pitch);
  const uint32_t a_bytes = 2u * P * 16u, b_bytes = 18u * BN * 16u;
  const uint32_t base = smem_u32(tile_smem);
  int* const offs = reinterpret_cast<int*>(tile_smem + 2 * (a_bytes + b_bytes));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int q0 = blockIdx.x * 128 * G, col0 = blockIdx.y * BN;
  const int cols = tmem_columns(G * BN);
  const int halo = g.pitch + 1;

  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(&tmem_slot, cols);
  for (int i = tid; i < P; i += kTileThreads)
    offs[i] = i < 128 * G + 2 * halo ? line_pixel(g, q0 - halo + i) : -1;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const uint32_t idesc = idesc_bf16_f32(128, BN);
  const int stages = (C + kStageChannels - 1) / kStageChannels;

  auto fill = [&](int st) {
    const uint32_t a = base + (st & 1) * (a_bytes + b_bytes), b = a + a_bytes;
    const int c0 = st * kStageChannels;
    for (int i = tid; i < 2 * P; i += kTileThreads) {
      const int p = i >> 1, kc = i & 1, c = c0 + 8 * kc;
      const int o = offs[p];
      const bool ok = o >= 0 && c < C;
      copy16(a + (kc * P + p) * 16, ok ? x + (size_t)o * C + c : x, ok);
    }
    for (int i = tid; i < 18 * BN; i += kTileThreads) {
      const int kc = i & 1, tap = (i >> 1) % 9, n = i / 18, c = c0 + 8 * kc;
      const bool ok = col0 + n < N && c < C;
      copy16(b + ((tap * 2 + kc) * BN + n) * 16,
             ok ? w + ((size_t)(col0 + n) * 9 + tap) * C + c : w, ok);
    }
    copy_commit();
  };
  auto multiply = [&](int st) {  // one thread
    tc_fence_after();
    const uint32_t a = base + (st & 1) * (a_bytes + b_bytes), b = a + a_bytes;
    for (int t = 0; t < G; ++t) {
#pragma unroll 1
      for (int tap = 0; tap < 9; ++tap) {
        const int off = sign * ((tap / 3 - 1) * g.pitch + tap % 3 - 1);
        mma_bf16(tmem + t * BN, smem_desc(a + (halo + 128 * t + off) * 16, P * 16, 128),
                 smem_desc(b + tap * 2 * BN * 16, BN * 16, 128), idesc,
                 st > 0 || tap > 0 ? 1u : 0u);
      }
    }
    mma_commit(&bar[st & 1]);
  };

  int issued = -1;
  for (int st = 0; st <= stages; ++st) {
    if (st < stages) {
      // the MMAs of stage st - 2 read this buffer
      if (st >= 2 && !mbar_wait_bounded(&bar[st & 1], ((st >> 1) - 1) & 1))
        atomicExch(&abort_flag, 2 + st);
      __syncthreads();
      if (abort_flag) break;
      fill(st);
    }
    if (st > 0) {
      if (st < stages) copy_wait<1>();
      else copy_wait<0>();
      fence_async_smem();
      __syncthreads();
      if (tid == 0) multiply(st - 1);
      issued = st - 1;
    }
  }
  if (abort_flag) copy_wait<0>();
  if (issued >= 0 && !mbar_wait_bounded(&bar[issued & 1], (issued >> 1) & 1))
    atomicExch(&abort_flag, 1);
  __syncthreads();
  tc_fence_after();
  const bool ok = !abort_flag;
  if (!ok && tid == 0) atomicMax(err, abort_flag);
  if (ok) {
    // warps w and w + 4 share a lane quarter and take every other 128 rows
    for (int t = warp >> 2; t < G; t += 2) {
      const int pixel = offs[halo + 128 * t + 32 * (warp & 3) + lane];
#pragma unroll 1
      for (int c = 0; c < BN; c += 16) {
        float v[16];
        tmem_load16(tmem + t * BN + c + (static_cast<uint32_t>(32 * (warp & 3)) << 16), v);
        if (pixel >= 0 && col0 + c < N) epi(pixel, col0 + c, v, 0);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, cols);
}

// Instruction descriptor with both operands MN-major.
__host__ __device__ constexpr uint32_t idesc_bf16_f32_mn(int M, int N) {
  return idesc_bf16_f32(M, N) | (1u << 15) | (1u << 16);
}

constexpr int kWgradPixels = 256;   // K of a tile
constexpr int kWgradColumns = 32;   // output channels of a block (9 accumulators)
constexpr int kWgradRows = 128;     // input channels of a block

// Partial weight gradient of the pixel tiles z, z + splits, ...: part[z][co][tap
// cin + ci]. Block (z, ci block, co block).
__global__ void __launch_bounds__(kTileThreads) conv_wgrad_kernel(
    const bf16* __restrict__ x, const bf16* __restrict__ dy, ConvLine g, int cin, int cout,
    float* __restrict__ part, int* err) {
  extern __shared__ __align__(1024) unsigned char tile_smem[];
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  constexpr int KT = kWgradPixels, BN = kWgradColumns;
  const int halo = g.pitch + 1;
  const int P = tile_pixels(KT, g.pitch);
  const uint32_t base = smem_u32(tile_smem);
  const uint32_t b_base = base + (kWgradRows / 8) * P * 16;
  int* const offs = reinterpret_cast<int*>(tile_smem + (kWgradRows / 8) * P * 16 + BN / 8 * KT * 16);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int splits = gridDim.x;
  const int ci0 = blockIdx.y * kWgradRows, co0 = blockIdx.z * BN;
  const int chunks = min(kWgradRows, cin - ci0) / 8;
  const int tiles = (g.Q + KT - 1) / KT;

  if (tid == 0) {
    mbar_init(&bar, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(&tmem_slot, 512);
  // (channel chunks beyond cin feed accumulator rows that are not stored)
  for (int i = tid; i < (kWgradRows / 8 - chunks) * P; i += kTileThreads)
    reinterpret_cast<uint4*>(tile_smem)[chunks * P + i] = make_uint4(0, 0, 0, 0);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const uint32_t idesc = idesc_bf16_f32_mn(kWgradRows, BN);

  int done = 0;
  for (int tile = blockIdx.x; tile < tiles; tile += splits, ++done) {
    const int q0 = tile * KT;
    if (done > 0 && !mbar_wait_bounded(&bar, (done - 1) & 1)) atomicExch(&abort_flag, 1 + done);
    for (int i = tid; i < P; i += kTileThreads)
      offs[i] = i < KT + 2 * halo ? line_pixel(g, q0 - halo + i) : -1;
    __syncthreads();
    if (abort_flag) break;
    for (int i = tid; i < chunks * P; i += kTileThreads) {
      const int p = i / chunks, kc = i - p * chunks;
      const int o = offs[p];
      copy16(base + (kc * P + p) * 16, o >= 0 ? x + (size_t)o * cin + ci0 + 8 * kc : x, o >= 0);
    }
    for (int i = tid; i < BN / 8 * KT; i += kTileThreads) {
      const int p = i / (BN / 8), kc = i % (BN / 8);
      const int o = offs[halo + p];
      const bool ok = o >= 0 && co0 + 8 * kc < cout;
      copy16(b_base + (kc * KT + p) * 16, ok ? dy + (size_t)o * cout + co0 + 8 * kc : dy, ok);
    }
    copy_commit();
    copy_wait<0>();
    fence_async_smem();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
#pragma unroll 1
      for (int k = 0; k < KT / 16; ++k)
#pragma unroll 1
        for (int tap = 0; tap < 9; ++tap) {
          const int off = (tap / 3 - 1) * g.pitch + tap % 3 - 1;
          mma_bf16(tmem + tap * BN, smem_desc(base + (halo + 16 * k + off) * 16, 128, P * 16),
                   smem_desc(b_base + 16 * k * 16, 128, KT * 16), idesc,
                   done > 0 || k > 0 ? 1u : 0u);
        }
      mma_commit(&bar);
    }
  }
  if (done > 0 && !abort_flag && !mbar_wait_bounded(&bar, (done - 1) & 1))
    atomicExch(&abort_flag, 1);
  __syncthreads();
  tc_fence_after();
  const bool ok = !abort_flag;
  if (!ok && tid == 0) atomicMax(err, abort_flag);
  const int ci = ci0 + 32 * (warp & 3) + lane;
  if (ok) {
    const size_t rows = 9 * (size_t)cin;
    for (int tap = warp >> 2; tap < 9; tap += 2) {
#pragma unroll 1
      for (int c = 0; c < BN; c += 16) {
        float v[16];
        if (done > 0) {
          tmem_load16(tmem + tap * BN + c + (static_cast<uint32_t>(32 * (warp & 3)) << 16), v);
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = 0.0f;
        }
        if (ci < cin) {
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (co0 + c + i < cout)
              part[((size_t)blockIdx.x * cout + co0 + c + i) * rows + (size_t)tap * cin + ci] =
                  v[i];
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

// Bias gradient: block b sums its pixels of all channels into part[b][c] (lanes
// over channels, 16-byte loads; the threads of a channel chunk in thread order).
constexpr int kBiasBlocks = 152;

__global__ void __launch_bounds__(kTileThreads) bias_partial_kernel(const bf16* __restrict__ dy,
                                                                    int npix, int C,
                                                                    float* __restrict__ part) {
  __shared__ float sums[kTileThreads][8];
  const int chunks = C / 8;
  const int lanes = kTileThreads / min(chunks, kTileThreads);  // pixels at a time
  const int per = (npix + gridDim.x - 1) / gridDim.x;
  const int p0 = min(npix, (int)blockIdx.x * per), p1 = min(npix, p0 + per);
  for (int cb = 0; cb < chunks; cb += kTileThreads) {
    const int kc = cb + threadIdx.x % min(chunks, kTileThreads);
    const int pl = threadIdx.x / min(chunks, kTileThreads);
    float s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = 0.0f;
    if (pl < lanes && kc < chunks) {
#pragma unroll 4
      for (int p = p0 + pl; p < p1; p += lanes) {
        const uint4 u = *reinterpret_cast<const uint4*>(dy + (size_t)p * C + 8 * kc);
        const bf16* b = reinterpret_cast<const bf16*>(&u);
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i] += __bfloat162float(b[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) sums[threadIdx.x][i] = s[i];
    __syncthreads();
    const int width = min(chunks, kTileThreads);
    for (int i = threadIdx.x; i < 8 * width; i += kTileThreads) {
      if (cb + i / 8 >= chunks) continue;
      float t = 0.0f;
      for (int l = 0; l < lanes; ++l) t += sums[l * width + i / 8][i % 8];
      part[(size_t)blockIdx.x * C + 8 * cb + i] = t;
    }
    __syncthreads();
  }
}

}  // namespace
}  // namespace nn
}  // namespace pty
