// Layout and type changes ahead of the tensor-core kernels.
//
// ib::transpose_batched rewrites [b][r][c] as [b][c][r] (K-major operands for tcgen05, and the
// `ij~ji` copies); the rest rounds or converts the operands of contractions and of fused attention.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "sm100.cuh"

namespace ib {
namespace {

// Round-to-nearest fp32 -> tf32 (10-bit mantissa, low 13 bits cleared).  The
// tensor core itself truncates; rounding operands first halves the error and
// removes its bias.
__device__ __forceinline__ float round_tf32(float x) {
  uint32_t u;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(x));
  return __uint_as_float(u);
}

// out[c][r] = in[r][c] through a 64 x 64 tile in shared memory.  Whole tiles of 16-byte-aligned
// arrays move as 16-byte accesses on both sides (a thread loads four neighbouring columns of a row
// and stores four neighbouring rows of a column); unaligned arrays go element by element.
template <bool ROUND>
__global__ void __launch_bounds__(256)
transpose_kernel(const float* __restrict__ in, float* __restrict__ out, size_t rows, size_t cols,
                 size_t out_pitch, bool vec) {
  constexpr int kT = 64;
  __shared__ float tile[kT][kT + 1];
  const size_t batch = blockIdx.z;
  in += batch * rows * cols;
  out += batch * cols * out_pitch;
  const size_t c0 = static_cast<size_t>(blockIdx.x) * kT, r0 = static_cast<size_t>(blockIdx.y) * kT;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  // Every load of a tile is in flight before the first is used, on ragged tiles too: one element after
  // the other they took sixteen round trips, and the last row of tiles was most of the kernel (700 x
  // 3000: 12.5 us, now 5.6).
  if (vec) {
    const size_t c = c0 + 4 * tx;                        // cols is a multiple of four
    float4 v[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const size_t r = r0 + ty + 16 * p;
      v[p] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (r < rows && c < cols) v[p] = *reinterpret_cast<const float4*>(in + r * cols + c);
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      float* at = &tile[ty + 16 * p][4 * tx];
      at[0] = v[p].x; at[1] = v[p].y; at[2] = v[p].z; at[3] = v[p].w;
    }
  } else {
    float v[16];
#pragma unroll
    for (int p = 0; p < 16; ++p) {
      const size_t r = r0 + threadIdx.x / kT + 4 * p, c = c0 + threadIdx.x % kT;
      v[p] = r < rows && c < cols ? in[r * cols + c] : 0.0f;
    }
#pragma unroll
    for (int p = 0; p < 16; ++p) tile[threadIdx.x / kT + 4 * p][threadIdx.x % kT] = v[p];
  }
  __syncthreads();
  if (vec) {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int c = ty + 16 * p;
      const size_t r = r0 + 4 * tx;
      float4 v = make_float4(tile[4 * tx + 0][c], tile[4 * tx + 1][c], tile[4 * tx + 2][c], tile[4 * tx + 3][c]);
      if (ROUND) v = make_float4(round_tf32(v.x), round_tf32(v.y), round_tf32(v.z), round_tf32(v.w));
      float* at = out + (c0 + c) * out_pitch + r;
      if (c0 + c < cols && r + 4 <= rows) {
        *reinterpret_cast<float4*>(at) = v;
      } else if (c0 + c < cols) {
        if (r + 0 < rows) at[0] = v.x;
        if (r + 1 < rows) at[1] = v.y;
        if (r + 2 < rows) at[2] = v.z;
      }
    }
  } else {
#pragma unroll
    for (int p = 0; p < 16; ++p) {
      const int c = threadIdx.x / kT + 4 * p, r = threadIdx.x % kT;
      if (r0 + r < rows && c0 + c < cols)
        out[(c0 + c) * out_pitch + r0 + r] = ROUND ? round_tf32(tile[r][c]) : tile[r][c];
    }
  }
}

// out[r][c] = round_tf32(in[r][c]) for up to two row-major arrays in one launch
// (blockIdx.y selects the array); pitches in elements.
struct RoundJob {
  const float* in;
  float* out;
  size_t rows, cols, in_pitch, out_pitch;
};

__global__ void __launch_bounds__(256)
round_rows_kernel(RoundJob j0, RoundJob j1) {
  const RoundJob j = blockIdx.y == 0 ? j0 : j1;
  const size_t n = j.rows * j.cols;
  const size_t stride = static_cast<size_t>(gridDim.x) * 256;
  const bool vec = j.cols % 4 == 0 && j.in_pitch % 4 == 0 && j.out_pitch % 4 == 0 &&
                   (reinterpret_cast<uintptr_t>(j.in) & 15u) == 0 &&
                   (reinterpret_cast<uintptr_t>(j.out) & 15u) == 0;
  if (vec) {
    const size_t cvec = j.cols / 4;
    for (size_t i = static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x; i < n / 4; i += stride) {
      const size_t r = i / cvec, c = (i - r * cvec) * 4;
      float4 v = *reinterpret_cast<const float4*>(j.in + r * j.in_pitch + c);
      v.x = round_tf32(v.x); v.y = round_tf32(v.y); v.z = round_tf32(v.z); v.w = round_tf32(v.w);
      *reinterpret_cast<float4*>(j.out + r * j.out_pitch + c) = v;
    }
  } else {
    for (size_t i = static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x; i < n; i += stride) {
      const size_t r = i / j.cols, c = i - r * j.cols;
      j.out[r * j.out_pitch + c] = round_tf32(j.in[r * j.in_pitch + c]);
    }
  }
}

// Operand preparation for the fused attention kernel in one launch:
// blockIdx.y = 0 rounds Q, 1 rounds K (both plain copies with TF32 rounding),
// 2 writes V^T = round(V)^T with 64x64 tiles through shared memory.
struct PrepareArgs {
  const float* q; float* qr; size_t q_elems;
  const float* k; float* kr; size_t k_elems;
  const float* v; float* vt; size_t batch, nk, dv, pitch;
};

__global__ void __launch_bounds__(256)
prepare_attention_kernel(PrepareArgs a) {
  __shared__ float tile[64][65];
  // The attention kernel may be scheduled once every CTA of this grid has started;
  // it waits for this grid's completion before it reads K or V^T.
  sm100::trigger_dependent_launch();
  if (blockIdx.y < 2) {
    const float* in = blockIdx.y == 0 ? a.q : a.k;
    float* out = blockIdx.y == 0 ? a.qr : a.kr;
    const size_t n4 = (blockIdx.y == 0 ? a.q_elems : a.k_elems) / 4;   // element counts are multiples of 4
    const size_t stride = static_cast<size_t>(gridDim.x) * 256;
    for (size_t i = static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x; i < n4; i += stride) {
      float4 x = __ldcs(reinterpret_cast<const float4*>(in) + i);
      x.x = round_tf32(x.x); x.y = round_tf32(x.y); x.z = round_tf32(x.z); x.w = round_tf32(x.w);
      reinterpret_cast<float4*>(out)[i] = x;
    }
    return;
  }
  const size_t tiles_k = (a.nk + 63) / 64, tiles_d = (a.dv + 63) / 64;
  const size_t total = a.batch * tiles_k * tiles_d;
  const bool vec_in = a.dv % 4 == 0 && (reinterpret_cast<uintptr_t>(a.v) & 15u) == 0;
  const bool vec_out = a.pitch % 4 == 0 && (reinterpret_cast<uintptr_t>(a.vt) & 15u) == 0;
  for (size_t t = blockIdx.x; t < total; t += gridDim.x) {
    const size_t b = t / (tiles_k * tiles_d);
    const size_t rem = t - b * tiles_k * tiles_d;
    const size_t k0 = (rem / tiles_d) * 64, d0 = (rem % tiles_d) * 64;
    const float* src = a.v + b * a.nk * a.dv;
    float* dst = a.vt + b * a.dv * a.pitch;
    // 64 keys x 64 features in: 16 float4 per key row, 4 rows per thread.
    for (int e = threadIdx.x; e < 64 * 16; e += 256) {
      const int r = e >> 4, c = (e & 15) * 4;           // r: key, c: feature (contiguous in V)
      float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (k0 + r < a.nk) {
        const float* row = src + (k0 + r) * a.dv + d0 + c;
        if (vec_in && d0 + c + 4 <= a.dv) {
          x = __ldcs(reinterpret_cast<const float4*>(row));
        } else {
          if (d0 + c + 0 < a.dv) x.x = row[0];
          if (d0 + c + 1 < a.dv) x.y = row[1];
          if (d0 + c + 2 < a.dv) x.z = row[2];
          if (d0 + c + 3 < a.dv) x.w = row[3];
        }
      }
      tile[r][c + 0] = round_tf32(x.x);
      tile[r][c + 1] = round_tf32(x.y);
      tile[r][c + 2] = round_tf32(x.z);
      tile[r][c + 3] = round_tf32(x.w);
    }
    __syncthreads();
    // 64 features x 64 keys out: 16 float4 per feature row.
    for (int e = threadIdx.x; e < 64 * 16; e += 256) {
      const int c = e >> 4, r = (e & 15) * 4;           // c: feature, r: key (contiguous in V^T)
      if (d0 + c >= a.dv) continue;
      float* row = dst + (d0 + c) * a.pitch + k0 + r;
      const float4 x = make_float4(tile[r][c], tile[r + 1][c], tile[r + 2][c], tile[r + 3][c]);
      if (vec_out && k0 + r + 4 <= a.nk) {
        *reinterpret_cast<float4*>(row) = x;
      } else {
        if (k0 + r + 0 < a.nk) row[0] = x.x;
        if (k0 + r + 1 < a.nk) row[1] = x.y;
        if (k0 + r + 2 < a.nk) row[2] = x.z;
        if (k0 + r + 3 < a.nk) row[3] = x.w;
      }
    }
    __syncthreads();
  }
}

__device__ __forceinline__ uint2 pack4_bf16(float a, float b, float c, float d) {
  const __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

__global__ void __launch_bounds__(256)
convert_bf16_kernel(const float* __restrict__ in, __nv_bfloat16* __restrict__ out, size_t rows,
                    size_t cols, size_t out_pitch) {
  // Four output columns per thread: a 16-byte load and an 8-byte store (out_pitch is a
  // multiple of 8, so every row starts 16-byte aligned).
  const size_t quads = out_pitch / 4;
  const size_t total = rows * quads;
  const size_t stride = static_cast<size_t>(gridDim.x) * 256;
  const bool vec = cols % 4 == 0 && (reinterpret_cast<uintptr_t>(in) & 15u) == 0;
  for (size_t i = static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x; i < total; i += stride) {
    const size_t r = i / quads, c = (i - r * quads) * 4;
    float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float* src = in + r * cols + c;
    if (vec && c + 4 <= cols) {
      x = __ldcs(reinterpret_cast<const float4*>(src));
    } else {
      if (c + 0 < cols) x.x = src[0];
      if (c + 1 < cols) x.y = src[1];
      if (c + 2 < cols) x.z = src[2];
      if (c + 3 < cols) x.w = src[3];
    }
    *reinterpret_cast<uint2*>(out + r * out_pitch + c) = pack4_bf16(x.x, x.y, x.z, x.w);
  }
}

// bf16 operand preparation for attention, one launch: blockIdx.y = 0 converts K
// ([rows][d] -> [rows][d_pitch]), blockIdx.y = 1 writes V^T ([nk][dv] -> [dv][nk_pitch])
// through 64x64 shared-memory tiles.  Pad columns are written as zero.
struct PrepareBf16Args {
  const float* k; __nv_bfloat16* k16; size_t k_rows, d, d_pitch;
  const float* v; __nv_bfloat16* vt16; size_t batch, nk, dv, nk_pitch;
};

__global__ void __launch_bounds__(256)
prepare_attention_bf16_kernel(PrepareBf16Args a) {
  __shared__ float tile[64][65];
  sm100::trigger_dependent_launch();       // see prepare_attention_kernel
  if (blockIdx.y == 0) {
    // Four columns per thread: one 16-byte load, one 8-byte store (d_pitch is a multiple of 8).
    const size_t quads = a.d_pitch / 4, total = a.k_rows * quads;
    const size_t stride = static_cast<size_t>(gridDim.x) * 256;
    const bool vec = a.d % 4 == 0 && (reinterpret_cast<uintptr_t>(a.k) & 15u) == 0;
    for (size_t i = static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x; i < total; i += stride) {
      const size_t r = i / quads, c = (i - r * quads) * 4;
      float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      const float* src = a.k + r * a.d + c;
      if (vec && c + 4 <= a.d) {
        x = __ldcs(reinterpret_cast<const float4*>(src));
      } else {
        if (c + 0 < a.d) x.x = src[0];
        if (c + 1 < a.d) x.y = src[1];
        if (c + 2 < a.d) x.z = src[2];
        if (c + 3 < a.d) x.w = src[3];
      }
      *reinterpret_cast<uint2*>(a.k16 + r * a.d_pitch + c) = pack4_bf16(x.x, x.y, x.z, x.w);
    }
    return;
  }
  const size_t tiles_k = (a.nk_pitch + 63) / 64, tiles_d = (a.dv + 63) / 64;
  const size_t total = a.batch * tiles_k * tiles_d;
  const bool vec_in = a.dv % 4 == 0 && (reinterpret_cast<uintptr_t>(a.v) & 15u) == 0;
  for (size_t t = blockIdx.x; t < total; t += gridDim.x) {
    const size_t b = t / (tiles_k * tiles_d);
    const size_t rem = t - b * tiles_k * tiles_d;
    const size_t k0 = (rem / tiles_d) * 64, d0 = (rem % tiles_d) * 64;
    const float* src = a.v + b * a.nk * a.dv;
    __nv_bfloat16* dst = a.vt16 + b * a.dv * a.nk_pitch;
    // 64 keys x 64 features in: 16 float4 per key row.
    for (int e = threadIdx.x; e < 64 * 16; e += 256) {
      const int r = e >> 4, c = (e & 15) * 4;           // r: key, c: feature (contiguous in V)
      float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (k0 + r < a.nk) {
        const float* row = src + (k0 + r) * a.dv + d0 + c;
        if (vec_in && d0 + c + 4 <= a.dv) {
          x = __ldcs(reinterpret_cast<const float4*>(row));
        } else {
          if (d0 + c + 0 < a.dv) x.x = row[0];
          if (d0 + c + 1 < a.dv) x.y = row[1];
          if (d0 + c + 2 < a.dv) x.z = row[2];
          if (d0 + c + 3 < a.dv) x.w = row[3];
        }
      }
      tile[r][c + 0] = x.x; tile[r][c + 1] = x.y; tile[r][c + 2] = x.z; tile[r][c + 3] = x.w;
    }
    __syncthreads();
    // 64 features x 64 keys out: 16 groups of 4 keys (8 bytes) per feature row; keys past nk
    // (up to the pitch) are written as the zeros the load left in the tile.
    for (int e = threadIdx.x; e < 64 * 16; e += 256) {
      const int c = e >> 4, r = (e & 15) * 4;           // c: feature, r: first key of the group
      if (d0 + c < a.dv && k0 + r < a.nk_pitch)
        *reinterpret_cast<uint2*>(dst + (d0 + c) * a.nk_pitch + k0 + r) =
            pack4_bf16(tile[r][c], tile[r + 1][c], tile[r + 2][c], tile[r + 3][c]);
    }
    __syncthreads();
  }
}

// ---- mixed arm: K rounded to TF32, V^T as fp16 scaled per head into fp16's range ----

// Largest |v| of each head, in kAbsmaxBlocks partial maxima per head (no atomics).  gridDim.y <=
// kAbsmaxBlocks blocks share a head, each thread keeping eight 16-byte loads in flight; the slots of
// the blocks a short head does not need are written as zero by its first block.
__global__ void __launch_bounds__(256)
absmax_heads_kernel(const float* __restrict__ v, float* __restrict__ block_max, size_t per_head) {
  __shared__ float warp_max[8];
  // The conversion kernel behind this one may start now: its K half does not need these maxima,
  // its V half waits for this grid before it reads them.
  sm100::trigger_dependent_launch();
  // blockIdx.x = head, blockIdx.y = slice of the head
  const float* base = v + static_cast<size_t>(blockIdx.x) * per_head;
  float m = 0.0f;
  const bool vec = per_head % 4 == 0 && (reinterpret_cast<uintptr_t>(base) & 15u) == 0;
  const size_t stride = static_cast<size_t>(gridDim.y) * 256;
  if (vec) {
    const float4* b4 = reinterpret_cast<const float4*>(base);
    const size_t n4 = per_head / 4;
    for (size_t i0 = static_cast<size_t>(blockIdx.y) * 256 + threadIdx.x; i0 < n4; i0 += 8 * stride) {
      float4 x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)   // plain loads: the conversion pass reads V again
        x[u] = i0 + u * stride < n4 ? b4[i0 + u * stride] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
      for (int u = 0; u < 8; ++u)
        m = fmaxf(m, fmaxf(fmaxf(fabsf(x[u].x), fabsf(x[u].y)), fmaxf(fabsf(x[u].z), fabsf(x[u].w))));
    }
  } else {
    for (size_t i = static_cast<size_t>(blockIdx.y) * 256 + threadIdx.x; i < per_head; i += stride)
      m = fmaxf(m, fabsf(base[i]));
  }
  m = warp_fold<IB_OP_MAX>(m);
  if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = m;
  __syncthreads();
  float* slots = block_max + static_cast<size_t>(blockIdx.x) * kAbsmaxBlocks;
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) m = fmaxf(m, warp_max[w]);
    slots[blockIdx.y] = m;
  }
  if (blockIdx.y == 0)
    for (int i = gridDim.y + threadIdx.x; i < kAbsmaxBlocks; i += 256) slots[i] = 0.0f;
}

// The power of two that brings a head's largest magnitude into [2^14, 2^15): large values fit
// fp16 (which holds up to 65504) and small ones keep their mantissa instead of falling into
// fp16's subnormals.  1 for an all-zero head or one holding inf / NaN (which then propagate as
// they would anyway).
__device__ __forceinline__ float f16_scale_for(float absmax) {
  if (!(absmax > 0.0f) || !(absmax < CUDART_INF_F)) return 1.0f;
  int e;
  frexpf(absmax, &e);                          // absmax = f * 2^e, f in [0.5, 1)
  return ldexpf(1.0f, max(e - 15, -120));      // absmax / scale = f * 2^15
}

// Every thread returns the scale of head b (reduces that head's partial maxima).
__device__ __forceinline__ float head_scale(const float* block_max, size_t b, float* scratch) {
  float m = threadIdx.x < kAbsmaxBlocks ? block_max[b * kAbsmaxBlocks + threadIdx.x] : 0.0f;
  m = warp_fold<IB_OP_MAX>(m);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = m;
  __syncthreads();
  float all = scratch[0];
  for (int w = 1; w < 8; ++w) all = fmaxf(all, scratch[w]);
  return f16_scale_for(all);
}

__device__ __forceinline__ uint2 pack4_f16(float a, float b, float c, float d) {
  const __half2 lo = __floats2half2_rn(a, b), hi = __floats2half2_rn(c, d);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

struct PrepareMixedArgs {
  const float* k; float* kr; size_t k_elems;
  const float* v; __half* vt16; float* scale; const float* block_max;
  size_t batch, nk, dv, nk_pitch;
  int v_kmajor;
  // fp16 arm only: K as fp16 [batch][nk][d_pitch], each tile of 128 keys over its own power of two.
  __half* k16; float* k_tile_scale; size_t d, d_pitch, kv_tiles;
};

// fp16(V^T / scale[head]) — through shared memory in steps of 64 keys when V is [keys][dv], as plain
// rows when it is already [dv][keys].  The per-head maxima come from the kernel before this one.
__device__ __forceinline__ void prepare_v_f16(const PrepareMixedArgs& a, uint32_t (*words)[32],
                                              float* scratch) {
  sm100::grid_dependency_wait();
  if (a.v_kmajor) {
    // Rows [batch * dv][nk] -> [batch * dv][nk_pitch], one row per block at a time.
    const size_t quads = a.nk_pitch / 4;
    const bool vec = a.nk % 4 == 0 && (reinterpret_cast<uintptr_t>(a.v) & 15u) == 0;
    size_t scaled_for = static_cast<size_t>(-1);
    float inv = 1.0f;
    for (size_t row = blockIdx.x; row < a.batch * a.dv; row += gridDim.x) {
      const size_t b = row / a.dv;
      if (b != scaled_for) {
        inv = 1.0f / head_scale(a.block_max, b, scratch);
        scaled_for = b;
      }
      if (row == b * a.dv && threadIdx.x == 0) a.scale[b] = 1.0f / inv;
      for (size_t q = threadIdx.x; q < quads; q += 256) {
        const size_t c = q * 4;
        const float* src = a.v + row * a.nk + c;
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (vec && c + 4 <= a.nk) {
          x = __ldcs(reinterpret_cast<const float4*>(src));
        } else {
          if (c + 0 < a.nk) x.x = src[0];
          if (c + 1 < a.nk) x.y = src[1];
          if (c + 2 < a.nk) x.z = src[2];
          if (c + 3 < a.nk) x.w = src[3];
        }
        *reinterpret_cast<uint2*>(a.vt16 + row * a.nk_pitch + c) =
            pack4_f16(x.x * inv, x.y * inv, x.z * inv, x.w * inv);
      }
    }
    return;
  }
  // 64 keys x all dv features per step.  Warp w takes key pairs 4w .. 4w + 3 of the step; lane l
  // loads features 4l .. 4l + 3 of both keys of a pair (two coalesced 512-byte rows), so eight
  // 16-byte loads are in flight per thread.  A pair of keys of one feature is one fp16x2 word of
  // V^T; it goes through shared memory as word [feature][pair ^ (feature / 4)]: the 32 lanes of a
  // store (32 feature groups, one pair) and the 32 lanes of a read (one feature, 32 pairs) each
  // hit 32 different banks.  A warp then writes a feature's 64 keys as one 128-byte line.
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t tiles_k = (a.nk_pitch + 63) / 64;
  const size_t total = a.batch * tiles_k;
  const bool vec_in = a.dv % 4 == 0 && (reinterpret_cast<uintptr_t>(a.v) & 15u) == 0;
  size_t scaled_for = static_cast<size_t>(-1);
  float inv = 1.0f;
  for (size_t t = blockIdx.x; t < total; t += gridDim.x) {
    const size_t b = t / tiles_k;
    const size_t k0 = (t - b * tiles_k) * 64;
    if (b != scaled_for) {
      inv = 1.0f / head_scale(a.block_max, b, scratch);
      scaled_for = b;
    }
    if (k0 == 0 && threadIdx.x == 0) a.scale[b] = 1.0f / inv;   // the block with the head's first tile
    const float* src = a.v + b * a.nk * a.dv;
    __half* dst = a.vt16 + b * a.dv * a.nk_pitch;
    const int c = lane * 4;                               // first feature of this lane's group
    float4 x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const size_t key = k0 + static_cast<size_t>(2 * (warp * 4 + (u >> 1)) + (u & 1));
      x[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (key < a.nk && static_cast<size_t>(c) < a.dv) {
        const float* row = src + key * a.dv + c;
        if (vec_in && static_cast<size_t>(c) + 4 <= a.dv) {
          x[u] = __ldcs(reinterpret_cast<const float4*>(row));
        } else {
          x[u].x = row[0];
          if (static_cast<size_t>(c) + 1 < a.dv) x[u].y = row[1];
          if (static_cast<size_t>(c) + 2 < a.dv) x[u].z = row[2];
          if (static_cast<size_t>(c) + 3 < a.dv) x[u].w = row[3];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 8; u += 2) {
      const int pair = warp * 4 + (u >> 1);
      const int col = pair ^ lane;                        // (feature / 4) & 31 == lane for all four
      const __half2 w0 = __floats2half2_rn(x[u].x * inv, x[u + 1].x * inv);
      const __half2 w1 = __floats2half2_rn(x[u].y * inv, x[u + 1].y * inv);
      const __half2 w2 = __floats2half2_rn(x[u].z * inv, x[u + 1].z * inv);
      const __half2 w3 = __floats2half2_rn(x[u].w * inv, x[u + 1].w * inv);
      words[c + 0][col] = *reinterpret_cast<const uint32_t*>(&w0);
      words[c + 1][col] = *reinterpret_cast<const uint32_t*>(&w1);
      words[c + 2][col] = *reinterpret_cast<const uint32_t*>(&w2);
      words[c + 3][col] = *reinterpret_cast<const uint32_t*>(&w3);
    }
    __syncthreads();
    // Feature rows warp, warp + 8, ...: lane = key pair.  Keys past nk (up to the pitch, which is
    // even) are written as the zeros the loads left.
#pragma unroll 4
    for (int f = warp; f < 128; f += 8) {
      if (static_cast<size_t>(f) < a.dv && k0 + 2 * lane < a.nk_pitch)
        *reinterpret_cast<uint32_t*>(dst + static_cast<size_t>(f) * a.nk_pitch + k0 + 2 * lane) =
            words[f][lane ^ ((f >> 2) & 31)];
    }
    __syncthreads();
  }
}

// The same in steps of 64 keys x 64 features (53 registers: for the grid whose other half is a plain
// elementwise pass and lives on occupancy).  fp16(V^T / scale[head]) — through 64x64 shared-memory tiles when V is [keys][dv], as plain rows
// when it is already [dv][keys].  The per-head maxima come from the kernel before this one.
__device__ __forceinline__ void prepare_v_f16_by_quarters(const PrepareMixedArgs& a, float (*tile)[65],
                                              float* scratch) {
  sm100::grid_dependency_wait();
  if (a.v_kmajor) {
    // Rows [batch * dv][nk] -> [batch * dv][nk_pitch], one row per block at a time.
    const size_t quads = a.nk_pitch / 4;
    const bool vec = a.nk % 4 == 0 && (reinterpret_cast<uintptr_t>(a.v) & 15u) == 0;
    size_t scaled_for = static_cast<size_t>(-1);
    float inv = 1.0f;
    for (size_t row = blockIdx.x; row < a.batch * a.dv; row += gridDim.x) {
      const size_t b = row / a.dv;
      if (b != scaled_for) {
        inv = 1.0f / head_scale(a.block_max, b, scratch);
        scaled_for = b;
      }
      if (row == b * a.dv && threadIdx.x == 0) a.scale[b] = 1.0f / inv;
      for (size_t q = threadIdx.x; q < quads; q += 256) {
        const size_t c = q * 4;
        const float* src = a.v + row * a.nk + c;
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (vec && c + 4 <= a.nk) {
          x = __ldcs(reinterpret_cast<const float4*>(src));
        } else {
          if (c + 0 < a.nk) x.x = src[0];
          if (c + 1 < a.nk) x.y = src[1];
          if (c + 2 < a.nk) x.z = src[2];
          if (c + 3 < a.nk) x.w = src[3];
        }
        *reinterpret_cast<uint2*>(a.vt16 + row * a.nk_pitch + c) =
            pack4_f16(x.x * inv, x.y * inv, x.z * inv, x.w * inv);
      }
    }
    return;
  }
  const size_t tiles_k = (a.nk_pitch + 63) / 64, tiles_d = (a.dv + 63) / 64;
  const size_t total = a.batch * tiles_k * tiles_d;
  const bool vec_in = a.dv % 4 == 0 && (reinterpret_cast<uintptr_t>(a.v) & 15u) == 0;
  size_t scaled_for = static_cast<size_t>(-1);
  float inv = 1.0f;
  for (size_t t = blockIdx.x; t < total; t += gridDim.x) {
    const size_t b = t / (tiles_k * tiles_d);
    const size_t rem = t - b * tiles_k * tiles_d;
    if (b != scaled_for) {
      inv = 1.0f / head_scale(a.block_max, b, scratch);
      scaled_for = b;
    }
    if (rem == 0 && threadIdx.x == 0) a.scale[b] = 1.0f / inv;   // the block with the head's first tile
    const size_t k0 = (rem / tiles_d) * 64, d0 = (rem % tiles_d) * 64;
    const float* src = a.v + b * a.nk * a.dv;
    __half* dst = a.vt16 + b * a.dv * a.nk_pitch;
    for (int e = threadIdx.x; e < 64 * 16; e += 256) {
      const int r = e >> 4, c = (e & 15) * 4;           // r: key, c: feature (contiguous in V)
      float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (k0 + r < a.nk) {
        const float* row = src + (k0 + r) * a.dv + d0 + c;
        if (vec_in && d0 + c + 4 <= a.dv) {
          x = __ldcs(reinterpret_cast<const float4*>(row));
        } else {
          if (d0 + c + 0 < a.dv) x.x = row[0];
          if (d0 + c + 1 < a.dv) x.y = row[1];
          if (d0 + c + 2 < a.dv) x.z = row[2];
          if (d0 + c + 3 < a.dv) x.w = row[3];
        }
      }
      tile[r][c + 0] = x.x * inv; tile[r][c + 1] = x.y * inv;
      tile[r][c + 2] = x.z * inv; tile[r][c + 3] = x.w * inv;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 64 * 16; e += 256) {
      const int c = e >> 4, r = (e & 15) * 4;           // c: feature, r: first key of the group
      if (d0 + c < a.dv && k0 + r < a.nk_pitch)
        *reinterpret_cast<uint2*>(dst + (d0 + c) * a.nk_pitch + k0 + r) =
            pack4_f16(tile[r][c], tile[r + 1][c], tile[r + 2][c], tile[r + 3][c]);
    }
    __syncthreads();
  }
}

// blockIdx.y = 0 rounds K to TF32; blockIdx.y = 1 writes the fp16 V^T.
__global__ void __launch_bounds__(256)
prepare_attention_mixed_kernel(PrepareMixedArgs a) {
  __shared__ float tile[64][65];
  __shared__ float scratch[8];
  sm100::trigger_dependent_launch();       // see prepare_attention_kernel
  if (blockIdx.y == 0) {
    const size_t n4 = a.k_elems / 4;          // d is a multiple of 4
    const size_t stride = static_cast<size_t>(gridDim.x) * 256;
    const bool vec = (reinterpret_cast<uintptr_t>(a.k) & 15u) == 0;
    for (size_t i = static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x; i < n4; i += stride) {
      float4 x;
      if (vec) {
        x = __ldcs(reinterpret_cast<const float4*>(a.k) + i);
      } else {
        x = make_float4(a.k[4 * i], a.k[4 * i + 1], a.k[4 * i + 2], a.k[4 * i + 3]);
      }
      x.x = round_tf32(x.x); x.y = round_tf32(x.y); x.z = round_tf32(x.z); x.w = round_tf32(x.w);
      reinterpret_cast<float4*>(a.kr)[i] = x;
    }
    return;
  }
  prepare_v_f16_by_quarters(a, tile, scratch);
}

// fp16 arm.  K, one tile of 128 keys per block at a time: a thread keeps its share of the tile in registers
// (sixteen 16-byte loads in flight), the tile's largest magnitude decides the power of two that brings it into
// [2^14, 2^15), and fp16(K / that) is written with rows padded to d_pitch (pad columns zero).  An outlier
// key therefore costs precision only to the 127 keys beside it.  V: the fp16 V^T as in the mixed arm.
// HALVES: K and V in one grid (blockIdx.y picks), or either in a grid of its own, since the registers that
// hold K's tile would leave the V half of a large grid two blocks per SM.
// Bound by HBM.  A thread's place in the tile comes from shifts: with a division of 64-bit numbers
// by the row length per 16-byte load the K half of 64 heads x 2048 x 128 took 35 us for 100 MB, now 21.
enum class Halves { Both, K, V };
template <Halves HALVES>
__global__ void __launch_bounds__(256)
prepare_attention_f16_kernel(PrepareMixedArgs a) {
  __shared__ float scratch[8];
  sm100::trigger_dependent_launch();       // see prepare_attention_kernel
  if constexpr (HALVES != Halves::K) {
    __shared__ uint32_t words[128][32];    // a step of V^T: 128 features x 32 key pairs (fp16x2)
    if (HALVES == Halves::V || blockIdx.y == 1) {
      prepare_v_f16(a, words, scratch);
      return;
    }
  }
  // 4-column groups per (padded) key row: at most 32, rounded up to a power of two.
  const unsigned across = 32 - __clz(static_cast<unsigned>(a.d_pitch / 4) - 1);
  const bool vec = (reinterpret_cast<uintptr_t>(a.k) & 15u) == 0;   // d is a multiple of 4
  constexpr int kBatch = 16;                 // 128 keys x 32 groups over 256 threads
  for (size_t t = blockIdx.x; t < a.batch * a.kv_tiles; t += gridDim.x) {
    const size_t b = t / a.kv_tiles, key0 = (t - b * a.kv_tiles) * 128;
    const size_t keys = a.nk - key0 < 128 ? a.nk - key0 : 128;
    const float* src = a.k + (b * a.nk + key0) * a.d;
    __half* dst = a.k16 + (b * a.nk + key0) * a.d_pitch;
    // 2^across lanes take a row (at most 32, the rest of them idle past quads); a tile is
    // 128 << across such places, at most 16 a thread.
    const unsigned places = static_cast<unsigned>(keys) << across;
    auto fetch = [&](unsigned g) {
      const unsigned r = g >> across, c = (g & ((1u << across) - 1)) * 4;
      if (g >= places || c >= a.d) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      const float* at = src + r * static_cast<unsigned>(a.d) + c;
      return vec ? *reinterpret_cast<const float4*>(at) : make_float4(at[0], at[1], at[2], at[3]);
    };
    float m = 0.0f;
    float4 x[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) x[u] = fetch(threadIdx.x + u * 256);
#pragma unroll
    for (int u = 0; u < kBatch; ++u)
      m = fmaxf(m, fmaxf(fmaxf(fabsf(x[u].x), fabsf(x[u].y)), fmaxf(fabsf(x[u].z), fabsf(x[u].w))));
    m = warp_fold<IB_OP_MAX>(m);
    __syncthreads();                         // scratch may still be read from the tile before
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = m;
    __syncthreads();
    float all = scratch[0];
    for (int w = 1; w < 8; ++w) all = fmaxf(all, scratch[w]);
    const float scale = f16_scale_for(all);
    const float inv = 1.0f / scale;
    if (threadIdx.x == 0) a.k_tile_scale[t] = scale;
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const unsigned g = threadIdx.x + u * 256;
      const unsigned r = g >> across, c = (g & ((1u << across) - 1)) * 4;
      if (g < places && c < a.d_pitch) {
        *reinterpret_cast<uint2*>(dst + r * static_cast<unsigned>(a.d_pitch) + c) =
            pack4_f16(x[u].x * inv, x[u].y * inv, x[u].z * inv, x[u].w * inv);
      }
    }
  }
  // Launched on its own under the tail of the maxima kernel (many tiles): this grid then only
  // completes once that one has, so that whoever waits for this grid has waited for both.
  if (HALVES == Halves::K) sm100::grid_dependency_wait();
}

// ---- operands of a contraction for the 16-bit tensor arms: both in one launch ----------------
//
// [batch][rows][kp] of 16-bit values, kp the depth rounded up to 8 (pad zero): bf16, or (SCALED) fp16
// over one power of two per row, which brings the row's largest magnitude into [2^14, 2^15) and goes to
// `scale` for the epilogue to multiply back.  Bound by HBM: one read of fp32, one write of half that.
//   stored [rows][k]: TPR threads a row, which stays in their registers up to 32 TPR values, so that the
//     maximum and the conversion share one read (2048 x 2048 x 2048 in fp16: 21 us with a CTA a row and
//     two loads in flight a thread, 10.5 with 64 threads and eight);
//   stored [k][rows]: a strip of 32 rows (128 bytes of every line), its k range divided between the CTAs
//     of a cluster where the strips alone are too few; the parts' maxima meet in distributed shared
//     memory, the conversion reads the strip again (from L2) and turns it through shared memory.
// Before, such an operand was transposed in fp32 first and the two converted one after the other:
// 4096 x 4096 x 4096 with B stored k first, whole call in bf16 174 -> 133 us, in fp16 195 -> 166.
struct ContractOperand {
  const float* in;
  void* out;
  float* scale;
  size_t rows;
  int kmajor;              // stored [rows][k]
  unsigned blocks;
};

constexpr int kStripK = 128;

template <bool SCALED>
__device__ __forceinline__ uint2 pack4_16(float4 x, float inv) {
  return SCALED ? pack4_f16(x.x * inv, x.y * inv, x.z * inv, x.w * inv) : pack4_bf16(x.x, x.y, x.z, x.w);
}

template <bool SCALED>
__device__ __forceinline__ void prepare_strip(const ContractOperand& o, unsigned block, size_t k, size_t kp,
                                              unsigned parts, float (*tile)[34], float (*warp_max)[32],
                                              float* part_max) {
  namespace cg = cooperative_groups;
  const size_t strips = (o.rows + 31) / 32;
  const unsigned part = block % parts;
  const size_t strip = block / parts, b = strip / strips, i0 = (strip - b * strips) * 32;
  const float* src = o.in + b * o.rows * k + i0;
  const size_t k_len = ((kp + kStripK - 1) / kStripK + parts - 1) / parts * kStripK;
  const size_t k_lo = part * k_len, k_hi = k_lo + k_len < kp ? k_lo + k_len : kp;
  const int quad = (threadIdx.x & 7) * 4, line = threadIdx.x >> 3;       // eight threads a line of 32 rows
  const size_t left = o.rows - i0;                                       // rows from here on
  const bool vec = o.rows % 4 == 0 && (reinterpret_cast<uintptr_t>(o.in) & 15u) == 0;
  auto fetch = [&](size_t kk) {
    float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (kk >= k || kk >= k_hi) return x;
    const float* at = src + kk * o.rows + quad;
    if (vec && static_cast<size_t>(quad) < left) return __ldg(reinterpret_cast<const float4*>(at));
    if (static_cast<size_t>(quad) + 0 < left) x.x = __ldg(at);
    if (static_cast<size_t>(quad) + 1 < left) x.y = __ldg(at + 1);
    if (static_cast<size_t>(quad) + 2 < left) x.z = __ldg(at + 2);
    if (static_cast<size_t>(quad) + 3 < left) x.w = __ldg(at + 3);
    return x;
  };

  if (SCALED) {
    float4 m = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (size_t kk = k_lo + line; kk < k_hi; kk += 32 * 8) {
      float4 x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = fetch(kk + u * 32);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        m.x = fmaxf(m.x, fabsf(x[u].x)); m.y = fmaxf(m.y, fabsf(x[u].y));
        m.z = fmaxf(m.z, fabsf(x[u].z)); m.w = fmaxf(m.w, fabsf(x[u].w));
      }
    }
#pragma unroll
    for (int d = 8; d < 32; d *= 2) {
      m.x = fmaxf(m.x, __shfl_xor_sync(0xffffffffu, m.x, d)); m.y = fmaxf(m.y, __shfl_xor_sync(0xffffffffu, m.y, d));
      m.z = fmaxf(m.z, __shfl_xor_sync(0xffffffffu, m.z, d)); m.w = fmaxf(m.w, __shfl_xor_sync(0xffffffffu, m.w, d));
    }
    if ((threadIdx.x & 31) < 8) *reinterpret_cast<float4*>(&warp_max[threadIdx.x >> 5][quad]) = m;
    __syncthreads();
    if (threadIdx.x < 32) {
      float all = 0.0f;
#pragma unroll
      for (int w = 0; w < 8; ++w) all = fmaxf(all, warp_max[w][threadIdx.x]);
      part_max[threadIdx.x] = all;
    }
    if (parts > 1) cg::this_cluster().sync();
    if (threadIdx.x < 32) {
      float all = part_max[threadIdx.x];
      if (parts > 1)
        for (unsigned q = 0; q < parts; ++q)
          all = fmaxf(all, cg::this_cluster().map_shared_rank(part_max, q)[threadIdx.x]);
      const float scale = f16_scale_for(all);
      warp_max[0][threadIdx.x] = 1.0f / scale;
      if (part == 0 && threadIdx.x < left) o.scale[b * o.rows + i0 + threadIdx.x] = scale;
    }
    __syncthreads();
  }

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = (warp & 1) * 16 + (lane & 15), group = (warp >> 1) * 2 + (lane >> 4);
  const float inv = SCALED ? warp_max[0][row] : 1.0f;
  uint16_t* dst = static_cast<uint16_t*>(o.out) + (b * o.rows + i0 + row) * kp;
  for (size_t k0 = k_lo; k0 < k_hi; k0 += kStripK) {
    float4 x[kStripK / 32];
#pragma unroll
    for (int u = 0; u < kStripK / 32; ++u) x[u] = fetch(k0 + line + u * 32);
#pragma unroll
    for (int u = 0; u < kStripK / 32; ++u) {
      float* at = &tile[line + u * 32][quad];           // rows of 34: 8-byte stores, no bank met twice
      *reinterpret_cast<float2*>(at) = make_float2(x[u].x, x[u].y);
      *reinterpret_cast<float2*>(at + 2) = make_float2(x[u].z, x[u].w);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kStripK / 64; ++u) {
      const int g = (group + u * 8) * 8;
      if (static_cast<size_t>(row) < left && k0 + g < k_hi) {
        const uint2 lo = pack4_16<SCALED>(make_float4(tile[g][row], tile[g + 1][row], tile[g + 2][row], tile[g + 3][row]), inv);
        const uint2 hi = pack4_16<SCALED>(make_float4(tile[g + 4][row], tile[g + 5][row], tile[g + 6][row], tile[g + 7][row]), inv);
        *reinterpret_cast<uint4*>(dst + k0 + g) = make_uint4(lo.x, lo.y, hi.x, hi.y);
      }
    }
    __syncthreads();
  }
  if (SCALED && parts > 1) cg::this_cluster().sync();      // nobody leaves while its maxima are read
}

// SHORT: rows of at most TPR quads.
template <bool SCALED, int TPR, bool SHORT>
__global__ void __launch_bounds__(256)
prepare_contract_kernel(const ContractOperand a, const ContractOperand b, size_t batch, size_t k, size_t kp,
                        unsigned parts) {
  __shared__ __align__(16) float tile[kStripK][34];      // rows of 34: stored to as pairs
  __shared__ __align__(16) float warp_max[8][32];
  __shared__ float part_max[32];
  sm100::trigger_dependent_launch();       // the GEMM's set-up may run under this grid
  const bool first = blockIdx.x < a.blocks;
  const ContractOperand& o = first ? a : b;
  const unsigned block = first ? blockIdx.x : blockIdx.x - a.blocks;
  if (!o.kmajor) {
    prepare_strip<SCALED>(o, block, k, kp, parts, tile, warp_max, part_max);
    return;
  }
  const size_t quads = kp / 4, rows = batch * o.rows;
  const unsigned at = threadIdx.x % TPR;
  const bool vec = k % 4 == 0 && (reinterpret_cast<uintptr_t>(o.in) & 15u) == 0;
  constexpr unsigned kGroups = 256 / TPR;
  if constexpr (SHORT) {
    // A quad a thread and row: eight rows at a time, so that as many loads are in flight.
    const size_t c = at * 4;
    for (size_t r0 = static_cast<size_t>(block) * kGroups * 8; r0 < rows; r0 += static_cast<size_t>(o.blocks) * kGroups * 8) {
      float4 x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const size_t r = r0 + u * kGroups + threadIdx.x / TPR;
        x[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (r >= rows || c >= k) continue;
        const float* src = o.in + r * k + c;
        if (vec) {
          x[u] = __ldg(reinterpret_cast<const float4*>(src));
        } else {
          x[u].x = src[0];
          if (c + 1 < k) x[u].y = src[1];
          if (c + 2 < k) x[u].z = src[2];
          if (c + 3 < k) x[u].w = src[3];
        }
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const size_t r = r0 + u * kGroups + threadIdx.x / TPR;
        float inv = 1.0f;
        if (SCALED) {
          float m = fmaxf(fmaxf(fabsf(x[u].x), fabsf(x[u].y)), fmaxf(fabsf(x[u].z), fabsf(x[u].w)));
#pragma unroll
          for (int d = TPR / 2; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
          const float scale = f16_scale_for(m);
          inv = 1.0f / scale;
          if (at == 0 && r < rows) o.scale[r] = scale;
        }
        if (r < rows && at < quads)
          *reinterpret_cast<uint2*>(static_cast<uint16_t*>(o.out) + r * kp + c) = pack4_16<SCALED>(x[u], inv);
      }
    }
  } else {
    const bool held = quads <= TPR * 8;
    for (size_t r0 = static_cast<size_t>(block) * kGroups; r0 < rows; r0 += static_cast<size_t>(o.blocks) * kGroups) {
      const size_t r = r0 + threadIdx.x / TPR;
      const bool live = r < rows;
      const float* src = o.in + r * k;
      uint16_t* dst = static_cast<uint16_t*>(o.out) + r * kp;
      float4 x[8];
      auto fetch = [&](size_t q0) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const size_t c = (q0 + u * TPR) * 4;
          x[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if (live && vec && c < k) {
            x[u] = __ldg(reinterpret_cast<const float4*>(src + c));
          } else if (live && c < k) {
            x[u].x = src[c];
            if (c + 1 < k) x[u].y = src[c + 1];
            if (c + 2 < k) x[u].z = src[c + 2];
            if (c + 3 < k) x[u].w = src[c + 3];
          }
        }
      };
      float inv = 1.0f;
      if (SCALED) {
        float m = 0.0f;
        for (size_t q0 = at; q0 < quads; q0 += TPR * 8) {
          fetch(q0);
#pragma unroll
          for (int u = 0; u < 8; ++u)
            m = fmaxf(m, fmaxf(fmaxf(fabsf(x[u].x), fabsf(x[u].y)), fmaxf(fabsf(x[u].z), fabsf(x[u].w))));
        }
        m = warp_fold<IB_OP_MAX>(m);
        if (TPR > 32) {
          __syncthreads();                     // part_max may still be read for the rows before
          if ((threadIdx.x & 31) == 0) part_max[threadIdx.x >> 5] = m;
          __syncthreads();
#pragma unroll
          for (int w = 0; w < TPR / 32; ++w) m = fmaxf(m, part_max[threadIdx.x / TPR * (TPR / 32) + w]);
        }
        const float scale = f16_scale_for(m);
        inv = 1.0f / scale;
        if (at == 0 && live) o.scale[r] = scale;
      }
      for (size_t q0 = at; q0 < quads; q0 += TPR * 8) {
        if (!SCALED || !held) fetch(q0);
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (live && q0 + u * TPR < quads)
            *reinterpret_cast<uint2*>(dst + (q0 + u * TPR) * 4) = pack4_16<SCALED>(x[u], inv);
      }
    }
  }
}

}  // namespace

// Blocks that share a head in absmax_heads_kernel: one per 32 KB of the head (eight 16-byte loads
// per thread), at most kAbsmaxBlocks.
unsigned absmax_blocks_per_head(size_t per_head) {
  const size_t per_block = 256 * 4 * 8;
  size_t blocks = (per_head + per_block - 1) / per_block;
  if (blocks < 1) blocks = 1;
  if (blocks > static_cast<size_t>(kAbsmaxBlocks)) blocks = kAbsmaxBlocks;
  return static_cast<unsigned>(blocks);
}

int prepare_attention_operands_bf16(const float* k, void* k16, const float* v, void* vt16,
                                    size_t batch, size_t nk, size_t d, size_t dv, size_t d_pitch,
                                    size_t nk_pitch, bool v_kmajor, cudaStream_t s) {
  if (v_kmajor) {
    // V already [dv][nk]: both operands are plain row conversions.
    if (int rc = convert_bf16_rows(k, k16, batch * nk, d, d_pitch, s)) return rc;
    return convert_bf16_rows(v, vt16, batch * dv, nk, nk_pitch, s);
  }
  PrepareBf16Args a{k, static_cast<__nv_bfloat16*>(k16), batch * nk, d, d_pitch,
                    v, static_cast<__nv_bfloat16*>(vt16), batch, nk, dv, nk_pitch};
  const size_t most = std::max(batch * nk * d_pitch / 4 / 256 + 1,
                               batch * ((nk_pitch + 63) / 64) * ((dv + 63) / 64));
  const size_t cap = static_cast<size_t>(kNumSMs) * 8;
  dim3 grid(static_cast<unsigned>(std::min(most, cap)), 2);
  prepare_attention_bf16_kernel<<<grid, 256, 0, s>>>(a);
  return check_launch("prepare_attention_operands_bf16");
}

int prepare_attention_operands_mixed(const float* k, float* kr, const float* v, void* vt16,
                                     float* scale, float* block_max, size_t batch, size_t nk,
                                     size_t d, size_t dv, size_t nk_pitch, bool v_kmajor,
                                     cudaStream_t s) {
  dim3 agrid(static_cast<unsigned>(batch), absmax_blocks_per_head(nk * dv));
  absmax_heads_kernel<<<agrid, 256, 0, s>>>(v, block_max, nk * dv);
  if (int rc = check_launch("absmax_heads")) return rc;
  PrepareMixedArgs a{k, kr, batch * nk * d, v, static_cast<__half*>(vt16), scale, block_max,
                     batch, nk, dv, nk_pitch, v_kmajor ? 1 : 0, nullptr, nullptr, d, d, 0};
  const size_t v_blocks = v_kmajor ? batch * dv : batch * ((nk_pitch + 63) / 64) * ((dv + 63) / 64);
  const size_t most = std::max(batch * nk * d / 4 / 256 + 1, v_blocks);
  const size_t cap = static_cast<size_t>(kNumSMs) * 8;
  // Launched so that it may overlap the maxima kernel (see the wait in its V half).
  cudaLaunchAttribute overlap{};
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(std::min(most, cap)), 2);
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cfg.attrs = &overlap;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, prepare_attention_mixed_kernel, a) != cudaSuccess)
    return fail(std::string("prepare_attention_operands_mixed: ") + cudaGetErrorString(cudaGetLastError()));
  count_launch();
  return 0;
}

int prepare_attention_operands_f16(const float* k, void* k16, float* k_tile_scale, const float* v,
                                   void* vt16, float* v_scale, float* block_max, size_t batch,
                                   size_t nk, size_t d, size_t dv, size_t d_pitch, size_t nk_pitch,
                                   bool v_kmajor, cudaStream_t s) {
  dim3 agrid(static_cast<unsigned>(batch), absmax_blocks_per_head(nk * dv));
  absmax_heads_kernel<<<agrid, 256, 0, s>>>(v, block_max, nk * dv);
  if (int rc = check_launch("absmax_heads")) return rc;
  const size_t kv_tiles = (nk + 127) / 128;
  PrepareMixedArgs a{k, nullptr, batch * nk * d, v, static_cast<__half*>(vt16), v_scale, block_max,
                     batch, nk, dv, nk_pitch, v_kmajor ? 1 : 0,
                     static_cast<__half*>(k16), k_tile_scale, d, d_pitch, kv_tiles};
  const size_t v_blocks = v_kmajor ? batch * dv : batch * ((nk_pitch + 63) / 64);
  const size_t cap = static_cast<size_t>(kNumSMs) * 8;
  // Launched so that it may overlap the maxima kernel (see the wait in the V half).
  cudaLaunchAttribute overlap{};
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cfg.attrs = &overlap;
  cfg.numAttrs = 1;
  cudaError_t launched;
  if (batch * kv_tiles <= 512) {
    // Few tiles: one grid, both halves.
    cfg.gridDim = dim3(static_cast<unsigned>(std::min(std::max(batch * kv_tiles, v_blocks), cap)), 2);
    launched = cudaLaunchKernelEx(&cfg, prepare_attention_f16_kernel<Halves::Both>, a);
  } else {
    // Many tiles: K in a grid of its own (with two passes per tile instead of the tile in registers, both in
    // one grid, it measured 1.8x the bf16 conversion's time), running beside the maxima kernel, which it does not need but whose
    // completion it waits for before it ends; then V, which waits for the K grid and so for the
    // maxima.  The attention kernel that waits for the V grid thereby waits for all three.
    cfg.gridDim = dim3(static_cast<unsigned>(std::min(batch * kv_tiles, cap * 2)), 1);
    launched = cudaLaunchKernelEx(&cfg, prepare_attention_f16_kernel<Halves::K>, a);
    if (launched == cudaSuccess) {
      count_launch();
      cfg.gridDim = dim3(static_cast<unsigned>(std::min(v_blocks, cap)), 1);
      launched = cudaLaunchKernelEx(&cfg, prepare_attention_f16_kernel<Halves::V>, a);
    }
  }
  if (launched != cudaSuccess)
    return fail(std::string("prepare_attention_operands_f16: ") + cudaGetErrorString(cudaGetLastError()));
  count_launch();
  return 0;
}

int convert_bf16_rows(const float* in, void* out, size_t rows, size_t cols, size_t out_pitch,
                      cudaStream_t s) {
  if (rows == 0 || cols == 0) return 0;
  size_t blocks = (rows * (out_pitch / 4) + 255) / 256;
  if (blocks > static_cast<size_t>(kNumSMs) * 16) blocks = static_cast<size_t>(kNumSMs) * 16;
  convert_bf16_kernel<<<static_cast<unsigned>(blocks), 256, 0, s>>>(
      in, static_cast<__nv_bfloat16*>(out), rows, cols, out_pitch);
  return check_launch("convert_bf16");
}

int prepare_contract_operands(const float* a, bool a_kmajor, void* a16, float* a_scale, const float* b,
                              bool b_kmajor, void* b16, float* b_scale, size_t batch, size_t m, size_t n,
                              size_t k, size_t kp, cudaStream_t s) {
  if (batch == 0 || m == 0 || n == 0 || k == 0) return 0;
  const bool scaled = a_scale != nullptr;
  // As few threads a row as hold it (32 values each): the more loads a thread has in flight, the less the
  // wait for the row's maximum shows.  Rows of up to 128 values take a thread a quad, eight rows at a time:
  // with a warp a row and one load a thread, 9 x 4048 rows of 29 took 14.5 us, 10^6 rows of 24 260.
  const int tpr = kp <= 32 ? 8 : kp <= 64 ? 16 : kp <= 1024 ? 32 : kp <= 2048 ? 64 : kp <= 4096 ? 128 : 256;
  const size_t at_once = kp <= 128 ? 8 : 1;
  // A strip's k range is divided until there are about two CTAs an SM or a part has 128 lines left.
  auto strips = [&](size_t rows, bool kmajor) { return kmajor ? 0 : batch * ((rows + 31) / 32); };
  const size_t n_strips = strips(m, a_kmajor) + strips(n, b_kmajor);
  unsigned parts = 1;
  while (n_strips && parts < 8 && n_strips * parts < 2 * static_cast<size_t>(kNumSMs) && kp / (parts * 2) >= kStripK)
    parts *= 2;
  auto blocks_for = [&](size_t rows, bool kmajor) {
    const size_t blocks = kmajor ? std::min((batch * rows * tpr + 256 * at_once - 1) / (256 * at_once),
                                            static_cast<size_t>(kNumSMs) * 32)
                                 : strips(rows, kmajor) * parts;
    return (blocks + parts - 1) / parts * parts;            // a cluster serves one operand
  };
  const size_t a_blocks = blocks_for(m, a_kmajor), b_blocks = blocks_for(n, b_kmajor);
  if (a_blocks + b_blocks >= (1u << 31)) return fail("ib_contract: operands too large to convert");
  const ContractOperand oa{a, a16, a_scale, m, a_kmajor ? 1 : 0, static_cast<unsigned>(a_blocks)};
  const ContractOperand ob{b, b16, b_scale, n, b_kmajor ? 1 : 0, static_cast<unsigned>(b_blocks)};
  cudaLaunchAttribute cluster{};
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim.x = parts;
  cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(a_blocks + b_blocks));
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cfg.attrs = &cluster;
  cfg.numAttrs = parts > 1 ? 1 : 0;
  auto pick = [tpr, at_once](auto is_scaled) {
    constexpr bool kScaled = decltype(is_scaled)::value;
    return tpr == 8    ? &prepare_contract_kernel<kScaled, 8, true>
           : tpr == 16  ? &prepare_contract_kernel<kScaled, 16, true>
           : at_once > 1 ? &prepare_contract_kernel<kScaled, 32, true>
           : tpr == 32  ? &prepare_contract_kernel<kScaled, 32, false>
           : tpr == 64  ? &prepare_contract_kernel<kScaled, 64, false>
           : tpr == 128 ? &prepare_contract_kernel<kScaled, 128, false>
                        : &prepare_contract_kernel<kScaled, 256, false>;
  };
  auto* kernel = scaled ? pick(std::true_type{}) : pick(std::false_type{});
  if (cudaLaunchKernelEx(&cfg, kernel, oa, ob, batch, k, kp, parts) != cudaSuccess)
    return fail(std::string("prepare_contract_operands: ") + cudaGetErrorString(cudaGetLastError()));
  count_launch();
  return 0;
}

int prepare_attention_operands(const float* q, float* qr, size_t q_elems, const float* k,
                               float* kr, size_t k_elems, const float* v, float* vt, size_t batch,
                               size_t nk, size_t dv, size_t pitch, cudaStream_t s) {
  PrepareArgs a{q, qr, q_elems, k, kr, k_elems, v, vt, batch, nk, dv, pitch};
  const size_t most = std::max(std::max(q_elems, k_elems) / 4 / 256 + 1,
                               batch * ((nk + 63) / 64) * ((dv + 63) / 64));
  const size_t cap = static_cast<size_t>(kNumSMs) * 8;
  dim3 grid(static_cast<unsigned>(std::min(most, cap)), 3);
  prepare_attention_kernel<<<grid, 256, 0, s>>>(a);
  return check_launch("prepare_attention_operands");
}

int round_tf32_rows(const float* in0, float* out0, size_t rows0, size_t cols0, size_t in_pitch0,
                    size_t out_pitch0, const float* in1, float* out1, size_t rows1, size_t cols1,
                    size_t in_pitch1, size_t out_pitch1, cudaStream_t s) {
  RoundJob j0{in0, out0, rows0, cols0, in_pitch0, out_pitch0};
  RoundJob j1{in1, out1, rows1, cols1, in_pitch1, out_pitch1};
  const size_t n = std::max(rows0 * cols0, in1 ? rows1 * cols1 : 0);
  if (n == 0) return 0;
  size_t blocks = (n / 4 + 255) / 256 + 1;
  if (blocks > static_cast<size_t>(kNumSMs) * 16) blocks = static_cast<size_t>(kNumSMs) * 16;
  dim3 grid(static_cast<unsigned>(blocks), in1 ? 2 : 1);
  round_rows_kernel<<<grid, 256, 0, s>>>(j0, j1);
  return check_launch("round_tf32");
}

int transpose_batched(const float* in, float* out, size_t batch, size_t rows, size_t cols,
                      size_t out_pitch, bool round, cudaStream_t s) {
  if (batch == 0 || rows == 0 || cols == 0) return 0;
  if (batch > 65535 || (rows + 63) / 64 > 65535) return fail("transpose: shape too large");
  dim3 grid(static_cast<unsigned>((cols + 63) / 64), static_cast<unsigned>((rows + 63) / 64),
            static_cast<unsigned>(batch));
  // 16-byte accesses need every row of either side, in every batch entry, to start on 16 bytes.
  const bool vec = cols % 4 == 0 && out_pitch % 4 == 0 && (rows * cols) % 4 == 0 &&
                   (reinterpret_cast<uintptr_t>(in) & 15u) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  if (round)
    transpose_kernel<true><<<grid, 256, 0, s>>>(in, out, rows, cols, out_pitch, vec);
  else
    transpose_kernel<false><<<grid, 256, 0, s>>>(in, out, rows, cols, out_pitch, vec);
  return check_launch("transpose");
}

}  // namespace ib
