// Sum of a row's shifted exponentials in one read: y[r] = sum_c powf(2.71828175f, x[r][c] - max_c x[r][c]),
// with unary operators on the result (`>ij~i`, `ij-i~ij`, `^ij~ij`, `+ij~i`, `$i~i`: a log-sum-exp).
//
// Bound: reading x once.  As a fold and a chained fold x was read twice and the second pass ran the
// operator interpreter (8192 x 8192 on B200: 39 + 117 us and a 3 us map; floor of one read 42 us).
// Every thread keeps a running maximum and the sum relative to it: 32 values are loaded, their
// maximum raises the running one (one rescale per 32 values), then their exponentials are added, two
// at a time in packed fp32 instructions.  No row has to fit on chip, so all lengths share the loop; short
// rows take a warp each, long ones a CTA, few very long ones a cluster whose CTAs meet in distributed
// shared memory.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "epilogue.cuh"
#include "kernels.h"

namespace ib {
namespace {

namespace cg = cooperative_groups;
using pair_t = unsigned long long;

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kUnroll = 8;                 // 16-byte loads in flight per thread

__device__ __forceinline__ pair_t pack(float lo, float hi) {
  pair_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack(pair_t x) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x));
  return r;
}
__device__ __forceinline__ pair_t add2(pair_t a, pair_t b) {
  pair_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ pair_t mul2(pair_t a, pair_t b) {
  pair_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ pair_t fma2(pair_t a, pair_t b, pair_t c) {
  pair_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float exp2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// max(x, floor) that lets a NaN through.
__device__ __forceinline__ float not_below(float x, float floor) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(floor));
  return r;
}

// powf(2.71828175f, d) of two differences d <= 0: 2^h with h = fp32(d * log2 e32), times one plus the
// rest of that product (what its rounding lost, and the low part of log2 e32) times ln 2; 2 ulp as in
// exp_e32_fast.  Results below 2^-126 are zero, which a sum that holds a one cannot tell; differences
// are held above -150 so that -inf - m does not turn the correction into NaN.
__device__ __forceinline__ pair_t exp_pair(pair_t d) {
  constexpr float l_hi = 1.4426950216293335f, l_lo = -2.4551930266625277e-08f, ln2 = 0.693147182464599609375f;
  const float2 raw = unpack(d);
  d = pack(not_below(raw.x, -150.0f), not_below(raw.y, -150.0f));
  const pair_t minus_h = mul2(d, pack(-l_hi, -l_hi));
  const pair_t lost = fma2(d, pack(l_hi, l_hi), minus_h);
  const pair_t rest = fma2(d, pack(l_lo * ln2, l_lo * ln2), mul2(lost, pack(ln2, ln2)));
  const float2 mh = unpack(minus_h);
  const pair_t r = pack(exp2_approx(-mh.x), exp2_approx(-mh.y));
  return fma2(r, rest, r);
}

// What an exponent is taken relative to: the maximum, or 0 while that is -inf (so that -inf counts as
// weight 0 until a finite value comes).
__device__ __forceinline__ float anchor(float m) { return m == -CUDART_INF_F ? 0.0f : m; }

struct Running {
  float m, l;
  __device__ Running() : m(-INFINITY), l(0.0f) {}

  // N values, an even number; absent ones are -inf.
  template <int N>
  __device__ __forceinline__ void take(const float (&v)[N]) {
    float top = m;
#pragma unroll
    for (int i = 0; i < N; ++i) top = fmaxf(top, v[i]);
    const float at = anchor(top);
    if (top != m) l *= exp_e32_fast(m - at);
    m = top;
    const pair_t shift = pack(-at, -at);
    pair_t sum = 0;
#pragma unroll
    for (int i = 0; i < N; i += 2) sum = add2(sum, exp_pair(add2(pack(v[i], v[i + 1]), shift)));
    const float2 s = unpack(sum);
    l += s.x + s.y;
  }
  __device__ __forceinline__ void merge(float m2, float l2) {
    const float top = fmaxf(m, m2), at = anchor(top);
    l = l * exp_e32_fast(m - at) + l2 * exp_e32_fast(m2 - at);
    m = top;
  }
};

// The values [lo, hi) of a row, shared by `across` threads of which this is number t.
template <bool VEC>
__device__ __forceinline__ Running scan(const float* row, size_t lo, size_t hi, size_t t, size_t across) {
  Running run;
  if (VEC) {
    const float4* row4 = reinterpret_cast<const float4*>(row);
    const size_t end = hi / 4;
    for (size_t i = lo / 4 + t; i < end; i += kUnroll * across) {
      float v[4 * kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const size_t at = i + u * across;
        const float4 q = at < end ? __ldcs(row4 + at)
                                  : make_float4(-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F);
        v[4 * u] = q.x; v[4 * u + 1] = q.y; v[4 * u + 2] = q.z; v[4 * u + 3] = q.w;
      }
      run.take(v);
    }
  } else {
    for (size_t i = lo + t; i < hi; i += kUnroll * across) {
      float v[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const size_t at = i + u * across;
        v[u] = at < hi ? __ldcs(row + at) : -CUDART_INF_F;
      }
      run.take(v);
    }
  }
  return run;
}

// The lanes of a warp (LANES of them hold something) meet: one rescale each to the common maximum.
template <int LANES = 32>
__device__ __forceinline__ void merge_warp(Running& run) {
  float top = run.m;
#pragma unroll
  for (int s = LANES / 2; s > 0; s >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, s));
  run.l *= exp_e32_fast(run.m - anchor(top));
  run.m = top;
#pragma unroll
  for (int s = LANES / 2; s > 0; s >>= 1) run.l += __shfl_xor_sync(0xffffffffu, run.l, s);
}

// A row of -inf alone has no finite maximum: the reference's -inf - (-inf) is NaN.
__device__ __forceinline__ float total(const Running& run, size_t cols) {
  return run.m == -CUDART_INF_F && cols > 0 ? CUDART_NAN_F : run.l;
}

template <bool VEC>
__global__ void __launch_bounds__(kThreads)
row_expsum_warp(const float* __restrict__ x, float* __restrict__ y, size_t rows, size_t cols,
                const __grid_constant__ GemmEpilogue post) {
  const size_t r = static_cast<size_t>(blockIdx.x) * kWarps + (threadIdx.x >> 5);
  if (r >= rows) return;
  Running run = scan<VEC>(x + r * cols, 0, cols, threadIdx.x & 31, 32);
  merge_warp(run);
  if ((threadIdx.x & 31) == 0) y[r] = epilogue_value(post, total(run, cols), r, 0, 1);
}

// One row per CTA, or per cluster of `parts` CTAs with equal shares of a multiple of four columns.
template <bool VEC, bool CLUSTER>
__global__ void __launch_bounds__(kThreads)
row_expsum_block(const float* __restrict__ x, float* __restrict__ y, size_t rows, size_t cols, unsigned parts,
                 const __grid_constant__ GemmEpilogue post) {
  __shared__ float2 warps[kWarps];
  __shared__ float2 share;
  const size_t r = CLUSTER ? blockIdx.x / parts : blockIdx.x;
  const unsigned part = CLUSTER ? blockIdx.x - static_cast<unsigned>(r) * parts : 0;
  const size_t len = CLUSTER ? ((cols + parts - 1) / parts + 3) / 4 * 4 : cols;
  const size_t lo = part * len < cols ? part * len : cols, hi = lo + len < cols ? lo + len : cols;
  Running run = scan<VEC>(x + r * cols, lo, hi, threadIdx.x, kThreads);
  merge_warp(run);
  if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = make_float2(run.m, run.l);
  __syncthreads();
  if (threadIdx.x < 32) {
    const float2 mine = warps[threadIdx.x % kWarps];
    run.m = mine.x;
    run.l = mine.y;
    merge_warp<kWarps>(run);
  }
  if (threadIdx.x == 0) {
    if (CLUSTER) share = make_float2(run.m, run.l);
    else y[r] = epilogue_value(post, total(run, cols), r, 0, 1);
  }
  if (!CLUSTER) return;
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  if (part == 0 && threadIdx.x == 0) {
    for (unsigned p = 1; p < parts; ++p) {
      const float2 other = *cluster.map_shared_rank(&share, p);
      run.merge(other.x, other.y);
    }
    y[r] = epilogue_value(post, total(run, cols), r, 0, 1);
  }
  cluster.sync();                            // nobody leaves while its shared memory is read
}

}  // namespace
}  // namespace ib

extern "C" int ib_row_expsum(const float* x, float* y, size_t rows, size_t cols, int n_post, const int* post_ops,
                             void* stream) {
  using namespace ib;
  if (rows == 0) return 0;
  if (!y || (!x && cols != 0)) return fail("ib_row_expsum: null pointer");
  if (n_post < 0 || n_post > IB_MAX_CHAIN_OPS || (n_post > 0 && !post_ops))
    return fail("ib_row_expsum: between 0 and " + std::to_string(IB_MAX_CHAIN_OPS) + " operators");
  GemmEpilogue post;
  post.n_ops = n_post;
  for (int k = 0; k < n_post; ++k) {
    if (post_ops[k] < IB_OP_ADD || post_ops[k] > IB_OP_NOT) return fail("ib_row_expsum: unknown operator");
    post.op[k] = post_ops[k];
    post.which[k] = -1;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool vec = cols % 4 == 0 && aligned16(x);
  // A warp per row up to 2048 columns (as the plain row folds): a CTA's 256 threads would hold fewer
  // than two 16-byte loads each.
  if (cols <= 2048) {
    // As many rows a launch as its grid holds (2^34; a loop over rows inside the kernel cost short rows 10 %).
    constexpr size_t kMost = static_cast<size_t>(0x7fffffff) * kWarps;
    for (size_t r0 = 0; r0 < rows; r0 += kMost) {
      const size_t n = std::min(rows - r0, kMost);
      const unsigned blocks = static_cast<unsigned>((n + kWarps - 1) / kWarps);
      if (vec) row_expsum_warp<true><<<blocks, kThreads, 0, s>>>(x + r0 * cols, y + r0, n, cols, post);
      else row_expsum_warp<false><<<blocks, kThreads, 0, s>>>(x + r0 * cols, y + r0, n, cols, post);
      if (int rc = check_launch("ib_row_expsum")) return rc;
    }
    return 0;
  }
  if (rows > 0x7fffffff) return fail("ib_row_expsum: more than 2^31 - 1 rows of more than 2048 columns");
  // Rows too few to give every SM several CTAs are cut into up to eight parts of at least 4096 columns.
  size_t parts = static_cast<size_t>(kNumSMs) * 4 / rows;
  if (parts > cols / 4096) parts = cols / 4096;
  if (parts > 8) parts = 8;
  if (parts < 2) {
    if (vec) row_expsum_block<true, false><<<static_cast<unsigned>(rows), kThreads, 0, s>>>(x, y, rows, cols, 1u, post);
    else row_expsum_block<false, false><<<static_cast<unsigned>(rows), kThreads, 0, s>>>(x, y, rows, cols, 1u, post);
    return check_launch("ib_row_expsum");
  }
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = static_cast<unsigned>(parts);
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(rows * parts));
  cfg.blockDim = dim3(kThreads);
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const unsigned p = static_cast<unsigned>(parts);
  const cudaError_t err = vec ? cudaLaunchKernelEx(&cfg, row_expsum_block<true, true>, x, y, rows, cols, p, post)
                              : cudaLaunchKernelEx(&cfg, row_expsum_block<false, true>, x, y, rows, cols, p, post);
  if (err != cudaSuccess) {
    cudaGetLastError();
    return fail(std::string("ib_row_expsum: ") + cudaGetErrorString(err));
  }
  count_launch();
  return 0;
}
