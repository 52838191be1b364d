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
// channels: 240 us forward, 384 us input gradient, 620 us weight gradient; now 51,
// 65 and 72 us).
//
//   forward, input gradient   rows = pixels (K-major operand), K = channels of a tap
//   weight gradient           rows = input channels, columns = output channels,
//                             K = pixels (both operands MN-major, same layout); one
//                             accumulator per tap
//
// The zeros take part in the products, on both sides of the weight gradient: an
// infinite or NaN activation at an image's border reaches the taps that pair it
// with the zeros too (0 x inf), beside those that pair it with gradients.
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
constexpr int kEpiPitch = 20;  // floats a row of a warp's epilogue buffer
constexpr int kRowBuffers = 3;      // most stages in shared memory
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

// the same for the weight gradient, whose copies put the chunks of a pixel side by
// side: an odd pitch spreads them over the banks
__host__ __device__ constexpr int wgrad_pixels(int rows, int pitch) {
  return (rows + 2 * (pitch + 1)) | 1;
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

// The issuing thread's work per MMA is what a narrow layer is bound by: the
// descriptors of a stage differ only in their start address (the low word, in
// units of 16 bytes), so an MMA costs two additions (rebuilding both descriptors
// for every MMA took about 240 cycles, eight times the MMA itself).
struct OperandBase {
  uint32_t lo, hi;
};
__device__ __forceinline__ OperandBase operand_base(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  const uint64_t d = smem_desc(addr, lbo, sbo);
  return {(uint32_t)d, (uint32_t)(d >> 32)};
}
__device__ __forceinline__ void mma_at(uint32_t d_tmem, OperandBase a, uint32_t a_off,
                                       OperandBase b, uint32_t b_off, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}" ::"r"(d_tmem),
      "r"(a.lo + a_off), "r"(a.hi), "r"(b.lo + b_off), "r"(b.hi), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Rows = pixels. Each block computes G x 128 consecutive q and BN columns (a
// multiple of 16) over all channels: stage = 16 channels of the tile and of the
// weights of the nine taps in `buffers` (2 or 3) buffers: all stages at once if they
// fit, else one under the MMAs and the others on their way. w: (N, 9, C). sign +1 reads x at
// q + off(tap), -1 at q - off(tap). epi(pixel, column, v[16]) receives the sums.
template <class Epi>
__global__ void __launch_bounds__(kTileThreads) conv_rows_kernel(const bf16* __restrict__ x,
                                                                 ConvLine g, int C,
                                                                 const bf16* __restrict__ w,
                                                                 int N, int BN, int G, int buffers,
                                                                 int sign, Epi epi, int* err) {
  extern __shared__ __align__(1024) unsigned char tile_smem[];
  __shared__ uint64_t bar[kRowBuffers];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int P = tile_pixels(128 * G, g.pitch);
  const uint32_t a_bytes = 2u * P * 16u, b_bytes = 18u * BN * 16u;
  const uint32_t base = smem_u32(tile_smem);
  int* const offs = reinterpret_cast<int*>(tile_smem + buffers * (a_bytes + b_bytes));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int q0 = blockIdx.x * 128 * G, col0 = blockIdx.y * BN;
  const int cols = tmem_columns(G * BN);
  const int halo = g.pitch + 1;

  if (tid == 0) {
    for (int i = 0; i < kRowBuffers; ++i) mbar_init(&bar[i], 1);
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
    const uint32_t a = base + (st % buffers) * (a_bytes + b_bytes), b = a + a_bytes;
    const int c0 = st * kStageChannels;
#pragma unroll 4
    for (int i = tid; i < 2 * P; i += kTileThreads) {
      const int p = i >> 1, kc = i & 1, c = c0 + 8 * kc;
      const int o = offs[p];
      const bool ok = o >= 0 && c < C;
      copy16(a + (kc * P + p) * 16, ok ? x + (size_t)o * C + c : x, ok);
    }
#pragma unroll 4
    for (int i = tid; i < 18 * BN; i += kTileThreads) {
      const int kc = i & 1, tap = (i >> 1) % 9, n = i / 18, c = c0 + 8 * kc;
      const bool ok = col0 + n < N && c < C;
      copy16(b + ((tap * 2 + kc) * BN + n) * 16,
             ok ? w + ((size_t)(col0 + n) * 9 + tap) * C + c : w, ok);
    }
  };
  auto multiply = [&](int st) {  // one thread
    tc_fence_after();
    const uint32_t a = base + (st % buffers) * (a_bytes + b_bytes), b = a + a_bytes;
    const OperandBase da = operand_base(a + halo * 16, P * 16, 128);
    const OperandBase db = operand_base(b, BN * 16, 128);
#pragma unroll 1
    for (int t = 0; t < G; ++t) {
#pragma unroll
      for (int tap = 0; tap < 9; ++tap)
        mma_at(tmem + t * BN, da,
               128 * t + sign * ((tap / 3 - 1) * g.pitch + tap % 3 - 1), db, tap * 2 * BN, idesc,
               st > 0 || tap > 0 ? 1u : 0u);
    }
    mma_commit(&bar[st % buffers]);
  };

  const int ahead = stages <= buffers ? stages : buffers - 1;  // stages in flight
  for (int st = 0; st < ahead; ++st) {
    fill(st);
    copy_commit();
  }
  int issued = -1;
  for (int st = 0; st < stages; ++st) {
    if (ahead == 1) copy_wait<0>();
    else if (ahead == 2) copy_wait<1>();
    else copy_wait<2>();
    fence_async_smem();
    __syncthreads();
    if (abort_flag) break;
    if (tid == 0) multiply(st);
    issued = st;
    if (st + ahead < stages) {
      // (ahead = buffers - 1: the buffer of stage st - 1, once its MMAs are done)
      if (st > 0 && !mbar_wait_bounded(&bar[(st - 1) % buffers], ((st - 1) / buffers) & 1))
        atomicExch(&abort_flag, 2 + st);
      fill(st + ahead);
    }
    copy_commit();
  }
  copy_wait<0>();
  if (issued >= 0 &&
      !mbar_wait_bounded(&bar[issued % buffers], (issued / buffers) & 1))
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
        if constexpr (Epi::kWarp) {
          // (the operand buffers are free by now)
          epi.store(reinterpret_cast<float*>(tile_smem) + warp * 32 * kEpiPitch, lane, pixel,
                    col0 + c, v);
        } else {
          if (pixel >= 0 && col0 + c < N) epi(pixel, col0 + c, v, 0);
        }
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
// cin + ci]. Block (z, ci block, co block). `buffers` (1 or 2) tiles in shared
// memory: with two, a tile is copied while the MMAs of the one before run.
__global__ void __launch_bounds__(kTileThreads) conv_wgrad_kernel(
    const bf16* __restrict__ x, const bf16* __restrict__ dy, ConvLine g, int cin, int cout,
    int buffers, float* __restrict__ part, int* err) {
  extern __shared__ __align__(1024) unsigned char tile_smem[];
  __shared__ uint64_t bar[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  constexpr int KT = kWgradPixels, BN = kWgradColumns;
  const int halo = g.pitch + 1;
  const int P = wgrad_pixels(KT, g.pitch);
  const uint32_t base = smem_u32(tile_smem);
  const uint32_t a_bytes = (kWgradRows / 8) * P * 16, b_bytes = BN / 8 * KT * 16;
  int* const offs = reinterpret_cast<int*>(tile_smem + buffers * (a_bytes + b_bytes));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int splits = gridDim.x;
  const int ci0 = blockIdx.y * kWgradRows, co0 = blockIdx.z * BN;
  const int chunks = min(kWgradRows, cin - ci0) / 8;
  const int tiles = (g.Q + KT - 1) / KT;
  const int mine = (int)blockIdx.x < tiles ? (tiles - 1 - (int)blockIdx.x) / splits + 1 : 0;
  // this thread's first piece of the x tile, and the step to its next
  const int p_first = tid / chunks, c_first = tid % chunks;
  const int p_step = kTileThreads / chunks, c_step = kTileThreads % chunks;

  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(&tmem_slot, 512);
  // (channel chunks beyond cin feed accumulator rows that are not stored)
  for (int b = 0; b < buffers; ++b)
    for (int i = tid; i < (kWgradRows / 8 - chunks) * P; i += kTileThreads)
      *reinterpret_cast<uint4*>(tile_smem + b * (a_bytes + b_bytes) + (chunks * P + i) * 16) =
          make_uint4(0, 0, 0, 0);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const uint32_t idesc = idesc_bf16_f32_mn(kWgradRows, BN);

  auto fill = [&](int k) {  // (block-wide: every thread calls it)
    const int q0 = ((int)blockIdx.x + k * splits) * KT;
    const uint32_t a = base + (k % buffers) * (a_bytes + b_bytes), b = a + a_bytes;
    for (int i = tid; i < P; i += kTileThreads)
      offs[i] = i < KT + 2 * halo ? line_pixel(g, q0 - halo + i) : -1;
    __syncthreads();
    int p = p_first, c = c_first;
#pragma unroll 4
    for (int i = tid; i < chunks * P; i += kTileThreads) {
      const int o = offs[p];
      copy16(a + (c * P + p) * 16, o >= 0 ? x + (size_t)o * cin + ci0 + 8 * c : x, o >= 0);
      p += p_step;
      c += c_step;
      if (c >= chunks) {
        c -= chunks;
        ++p;
      }
    }
#pragma unroll
    for (int i = tid; i < BN / 8 * KT; i += kTileThreads) {
      const int pp = i / (BN / 8), kc = i % (BN / 8);
      const int o = offs[halo + pp];
      const bool ok = o >= 0 && co0 + 8 * kc < cout;
      copy16(b + (kc * KT + pp) * 16, ok ? dy + (size_t)o * cout + co0 + 8 * kc : dy, ok);
    }
  };

  int done = 0;
  if (buffers == 2 && mine > 0) fill(0);
  for (int k = 0; k < mine; ++k) {
    if (buffers == 1) {
      if (k > 0 && !mbar_wait_bounded(&bar[(k - 1) & 1], ((k - 1) >> 1) & 1))
        atomicExch(&abort_flag, 1 + k);
      fill(k);
    }
    copy_commit();
    copy_wait<0>();
    fence_async_smem();
    __syncthreads();
    if (abort_flag) break;
    if (tid == 0) {
      tc_fence_after();
      const uint32_t a = base + (k % buffers) * (a_bytes + b_bytes), b = a + a_bytes;
      const OperandBase da = operand_base(a + halo * 16, 128, P * 16);
      const OperandBase db = operand_base(b, 128, KT * 16);
#pragma unroll 1
      for (int s = 0; s < KT / 16; ++s)
#pragma unroll
        for (int tap = 0; tap < 9; ++tap)
          mma_at(tmem + tap * BN, da, 16 * s + (tap / 3 - 1) * g.pitch + tap % 3 - 1, db, 16 * s,
                 idesc, k > 0 || s > 0 ? 1u : 0u);
      mma_commit(&bar[k & 1]);
    }
    done = k + 1;
    if (buffers == 2 && k + 1 < mine) {
      if (k > 0 && !mbar_wait_bounded(&bar[(k - 1) & 1], ((k - 1) >> 1) & 1))
        atomicExch(&abort_flag, 1 + k);
      fill(k + 1);
    }
  }
  copy_wait<0>();
  if (done > 0 && !mbar_wait_bounded(&bar[(done - 1) & 1], ((done - 1) >> 1) & 1))
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
#pragma unroll 16  // (latency-bound: 16 loads in flight)
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
