// Attention in fp32 straight from the caller's K and V: one pass, no score matrix, no converted
// operands.  What serves few queries against long contexts (decoding) and attention too small for
// the tensor-core kernels.
//
// Bound: with few queries per head every K and V element is used by a handful of multiply-adds, so
// the pass is bound by reading K and V once; small problems are bound by the length of one warp's
// chain.  Both ask for many independent warps and no staging.  A warp therefore works alone on blocks
// of 32 keys: lanes side by side hold one key row (LP lanes of four features; 128 features fill
// the warp, 32 features let four keys share it), NQ queries live in registers, eight rows are in
// flight per lane, and the partial dot products of eight rows are summed across lanes by a halving
// exchange (9 shuffles for 8 sums of 32 lanes, where 8 plain sums take 40) that leaves every lane with
// the score of one key.  The softmax is online per warp; the same lanes then read V rows and add
// p * v into NQ x 4 accumulators.  Warps meet in shared memory, key ranges of one head (splits) in
// distributed shared memory when a cluster holds them, else through partial results and a second kernel.
//
// Measured on B200, 32 heads x 1 query x 10000 keys x 128 (328 MB): 597 us as row folds per head
// (97 launches), here in one launch; figures in the table of the dispatch rule (dispatch.cu).
#include <cooperative_groups.h>

#include <cmath>

#include "common.cuh"
#include "kernels.h"

namespace ib {
namespace {

namespace cg = cooperative_groups;

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kBlockKeys = 32;             // keys a warp takes at a time: one score per lane
constexpr int kMaxCluster = 8;             // portable cluster size

struct DirectArgs {
  const float* q;
  const float* k;
  const float* v;
  float* o;
  float* partial_o;                        // [row][split][dv] when key ranges meet in a second kernel
  float2* partial_ml;                      // [row][split]: maximum, sum
  const float* logit_scale;
  size_t nq, nk, groups;
  int d, dv, splits, blocks_per_split, logit_divide;
  bool vec;                                // rows of q, k and v start on 16 bytes
};

__device__ __forceinline__ float4 load_chunk(const float* row, int at, int width, bool vec) {
  if (at >= width) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (vec) return __ldg(reinterpret_cast<const float4*>(row + at));
  float4 x = make_float4(__ldg(row + at), 0.0f, 0.0f, 0.0f);
  if (at + 1 < width) x.y = __ldg(row + at + 1);
  if (at + 2 < width) x.z = __ldg(row + at + 2);
  if (at + 3 < width) x.w = __ldg(row + at + 3);
  return x;
}

// exp(x - m) where a maximum of -inf (no key with a finite score yet) counts as 0, so that keys at
// -inf weigh nothing instead of turning the row into NaN.
__device__ __forceinline__ float weight_of(float x, float m) {
  return exp_e32_fast(x - (m == -CUDART_INF_F ? 0.0f : m));
}

// Two products or multiply-adds in one instruction, each lane rounded as the plain one.
using pair_t = unsigned long long;
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

// Sums v[0..7] across the LP lanes of a key row.  Lane `sub` returns the sum of v[sub / (LP / 8)].
template <int LP>
__device__ __forceinline__ float sum_eight(float (&v)[8], int sub) {
  int half = 4;
#pragma unroll
  for (int off = LP / 2; off >= LP / 8; off >>= 1, half >>= 1) {
    const bool up = (sub & off) != 0;
#pragma unroll
    for (int j = 0; j < half; ++j) {
      const float keep = up ? v[j + half] : v[j];
      const float send = up ? v[j] : v[j + half];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
#pragma unroll
  for (int off = LP / 16; off > 0; off >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
  return v[0];
}

template <int LP, int NQ, bool CLUSTER>
__global__ void __launch_bounds__(kThreads, NQ >= 4 ? 2 : 3)
attention_direct_kernel(DirectArgs a) {
  constexpr int kKeysPerLoad = 32 / LP;
  constexpr int kBatches = LP / 8;           // of eight loads: together one block of 32 keys
  constexpr int kWidth = LP * 4;             // features a warp covers
  // With four or eight queries the registers are the accumulators': the queries stay in shared
  // memory (one 16-byte read per eight rows and query), and a weight reaches the lanes as a
  // duplicated pair from shared memory (a 16-byte broadcast for two queries, where a shuffle serves one).
  constexpr bool kWide = NQ >= 4;
  constexpr int kBatchUnroll = kWide ? 1 : kBatches;      // unrolled, the wide forms outgrow the instruction cache
  constexpr int kRow = kWidth < 2 * kBlockKeys ? 2 * kBlockKeys : kWidth;   // a warp's part also holds its weights
  __shared__ __align__(16) float sm_o[kWarps][NQ][kRow];
  __shared__ __align__(16) float sm_q[kWide ? NQ : 1][kWide ? kWidth : 4];
  __shared__ float sm_m[kWarps][NQ], sm_l[kWarps][NQ];
  __shared__ float cta_m[NQ], cta_l[NQ];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane % LP, grp = lane / LP;
  const size_t unit = blockIdx.x / static_cast<unsigned>(a.splits);
  const int split = static_cast<int>(blockIdx.x - unit * a.splits);
  const size_t head = unit / a.groups, q0 = (unit - head * a.groups) * NQ;
  const float* kh = a.k + head * a.nk * a.d;
  const float* vh = a.v + head * a.nk * a.dv;

  float4 q[kWide ? 1 : NQ];
  auto query = [&](int i, int chunk) {
    return q0 + i < a.nq ? load_chunk(a.q + (head * a.nq + q0 + i) * a.d, chunk * 4, a.d, a.vec)
                         : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  };
  if constexpr (kWide) {
    for (int e = threadIdx.x; e < NQ * LP; e += kThreads)
      *reinterpret_cast<float4*>(&sm_q[e / LP][e % LP * 4]) = query(e / LP, e % LP);
    __syncthreads();
  } else {
#pragma unroll
    for (int i = 0; i < NQ; ++i) q[i] = query(i, sub);
  }
  // This warp's weights: its own part of sm_o, which is written after its last block of keys.
  float2(*sm_p)[NQ] = reinterpret_cast<float2(*)[NQ]>(sm_o[warp]);
  static_assert(sizeof(float2) * kBlockKeys * NQ <= sizeof(sm_o[0]), "the weights fit the warp's part");
  const float scale = a.logit_scale ? __ldg(a.logit_scale) : 1.0f;

  float m[NQ], l[NQ];
  pair_t o[NQ][2];
#pragma unroll
  for (int i = 0; i < NQ; ++i) {
    m[i] = -CUDART_INF_F;
    l[i] = 0.0f;
    o[i][0] = o[i][1] = 0;
  }

  const size_t n_blocks = (a.nk + kBlockKeys - 1) / kBlockKeys;
  const size_t b_lo = static_cast<size_t>(split) * a.blocks_per_split;
  const size_t b_hi = b_lo + a.blocks_per_split < n_blocks ? b_lo + a.blocks_per_split : n_blocks;
  for (size_t blk = b_lo + warp; blk < b_hi; blk += kWarps) {
    const size_t key0 = blk * kBlockKeys;
    float s[NQ];
#pragma unroll kBatchUnroll
    for (int b = 0; b < kBatches; ++b) {
      float4 x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const size_t key = key0 + (b * 8 + u) * kKeysPerLoad + grp;
        x[u] = key < a.nk ? load_chunk(kh + key * a.d, sub * 4, a.d, a.vec)
                          : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
#pragma unroll
      for (int i = 0; i < NQ; ++i) {
        float part[8];
        const float4 qi = kWide ? *reinterpret_cast<const float4*>(&sm_q[kWide ? i : 0][kWide ? sub * 4 : 0]) : q[kWide ? 0 : i];
        const pair_t q_lo = pack(qi.x, qi.y), q_hi = pack(qi.z, qi.w);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const float2 t = unpack(fma2(q_hi, pack(x[u].z, x[u].w), mul2(q_lo, pack(x[u].x, x[u].y))));
          part[u] = t.x + t.y;
        }
        const float sum = sum_eight<LP>(part, sub);
        if (b == 0 || sub % kBatches == b) s[i] = sum;
      }
    }
    // This lane's key: load (sub % kBatches) * 8 + sub / kBatches of the block.
    const size_t key = key0 + ((sub % kBatches) * 8 + sub / kBatches) * kKeysPerLoad + grp;
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
      if (a.logit_scale) s[i] = a.logit_divide ? __fdiv_rn(s[i], scale) : s[i] * scale;
      if (key >= a.nk) s[i] = -CUDART_INF_F;
      const float top = fmaxf(m[i], warp_fold<IB_OP_MAX>(s[i]));
      if (top != m[i]) {                       // uniform: every lane holds the same two values
        const float shrink = weight_of(m[i], top);
        l[i] *= shrink;
        o[i][0] = mul2(o[i][0], pack(shrink, shrink));
        o[i][1] = mul2(o[i][1], pack(shrink, shrink));
        m[i] = top;
      }
      s[i] = key < a.nk ? weight_of(s[i], top) : 0.0f;
      l[i] += s[i];
    }
    if constexpr (kWide) {
      __syncwarp();                            // the lanes have read the weights of the block before
      const int slot = ((sub % kBatches) * 8 + sub / kBatches) * kKeysPerLoad + grp;
#pragma unroll
      for (int i = 0; i < NQ; i += 2)
        *reinterpret_cast<float4*>(&sm_p[slot][i]) = make_float4(s[i], s[i], s[i + 1], s[i + 1]);
      __syncwarp();
    }
#pragma unroll kBatchUnroll
    for (int b = 0; b < kBatches; ++b) {
      float4 x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const size_t at = key0 + (b * 8 + u) * kKeysPerLoad + grp;
        x[u] = at < a.nk ? load_chunk(vh + at * a.dv, sub * 4, a.dv, a.vec)
                         : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const pair_t x_lo = pack(x[u].x, x[u].y), x_hi = pack(x[u].z, x[u].w);
        if constexpr (kWide) {
          const int slot = (b * 8 + u) * kKeysPerLoad + grp;
#pragma unroll
          for (int i = 0; i < NQ; i += 2) {
            const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(&sm_p[slot][i]);
            o[i][0] = fma2(p.x, x_lo, o[i][0]);
            o[i][1] = fma2(p.x, x_hi, o[i][1]);
            o[i + 1][0] = fma2(p.y, x_lo, o[i + 1][0]);
            o[i + 1][1] = fma2(p.y, x_hi, o[i + 1][1]);
          }
        } else {
          const int holder = grp * LP + u * kBatches + b;
#pragma unroll
          for (int i = 0; i < NQ; ++i) {
            const float w = __shfl_sync(0xffffffffu, s[i], holder);
            o[i][0] = fma2(pack(w, w), x_lo, o[i][0]);
            o[i][1] = fma2(pack(w, w), x_hi, o[i][1]);
          }
        }
      }
    }
  }

  // The warps of the CTA meet.
  __syncwarp();
#pragma unroll
  for (int i = 0; i < NQ; ++i) {
    l[i] = warp_fold<IB_OP_ADD>(l[i]);
    const float2 lo = unpack(o[i][0]), hi = unpack(o[i][1]);
    float4 sum = make_float4(lo.x, lo.y, hi.x, hi.y);
#pragma unroll
    for (int off = LP; off < 32; off <<= 1) {
      sum.x += __shfl_xor_sync(0xffffffffu, sum.x, off);
      sum.y += __shfl_xor_sync(0xffffffffu, sum.y, off);
      sum.z += __shfl_xor_sync(0xffffffffu, sum.z, off);
      sum.w += __shfl_xor_sync(0xffffffffu, sum.w, off);
    }
    if (grp == 0) *reinterpret_cast<float4*>(&sm_o[warp][i][sub * 4]) = sum;
    if (lane == 0) {
      sm_m[warp][i] = m[i];
      sm_l[warp][i] = l[i];
    }
  }
  __syncthreads();
  const bool alone = a.splits == 1;
  for (int e = threadIdx.x; e < NQ * kWidth; e += kThreads) {
    const int i = e / kWidth, c = e % kWidth;
    if (c >= a.dv || q0 + i >= a.nq) continue;
    float top = sm_m[0][i];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) top = fmaxf(top, sm_m[w][i]);
    float sum = 0.0f, acc = 0.0f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = weight_of(sm_m[w][i], top);
      sum = fmaf(sm_l[w][i], f, sum);
      acc = fmaf(sm_o[w][i][c], f, acc);
    }
    const size_t row = head * a.nq + q0 + i;
    if (alone) {
      a.o[row * a.dv + c] = acc / sum;
    } else if (CLUSTER) {
      sm_o[0][i][c] = acc;                   // only this thread reads or writes column (i, c)
      if (c == 0) {
        cta_m[i] = top;
        cta_l[i] = sum;
      }
    } else {
      a.partial_o[(row * a.splits + split) * a.dv + c] = acc;
      if (c == 0) a.partial_ml[row * a.splits + split] = make_float2(top, sum);
    }
  }
  if (!CLUSTER) return;
  // The key ranges of this head meet in distributed shared memory; the CTAs share the columns.
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  for (int e = threadIdx.x + split * kThreads; e < NQ * kWidth; e += kThreads * a.splits) {
    const int i = e / kWidth, c = e % kWidth;
    if (c >= a.dv || q0 + i >= a.nq) continue;
    float top = -CUDART_INF_F;
    for (int r = 0; r < a.splits; ++r) top = fmaxf(top, *cluster.map_shared_rank(&cta_m[i], r));
    float sum = 0.0f, acc = 0.0f;
    for (int r = 0; r < a.splits; ++r) {
      const float f = weight_of(*cluster.map_shared_rank(&cta_m[i], r), top);
      sum = fmaf(*cluster.map_shared_rank(&cta_l[i], r), f, sum);
      acc = fmaf(*cluster.map_shared_rank(&sm_o[0][i][c], r), f, acc);
    }
    a.o[(head * a.nq + q0 + i) * a.dv + c] = acc / sum;
  }
  cluster.sync();                            // nobody leaves while its shared memory is read
}

// One CTA per query row: merges the row's key ranges.  The ranges' weights are computed once, then
// groups of 128 threads (one per column) each add a share of the ranges and meet in shared memory.
constexpr int kMergeThreads = 512, kMergeGroups = kMergeThreads / 128, kMaxSplits = 512;

__global__ void __launch_bounds__(kMergeThreads)
attention_direct_merge_kernel(const float* __restrict__ partial_o, const float2* __restrict__ partial_ml,
                              float* __restrict__ o, int splits, int dv) {
  __shared__ float weight[kMaxSplits], scratch[kMergeThreads / 32][2], meet[kMergeGroups][128];
  const size_t row = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool mine = static_cast<int>(threadIdx.x) < splits;               // at most one range per thread
  const float2 ml = mine ? partial_ml[row * splits + threadIdx.x] : make_float2(-CUDART_INF_F, 0.0f);
  float top = warp_fold<IB_OP_MAX>(ml.x);
  if (lane == 0) scratch[warp][0] = top;
  __syncthreads();
  top = scratch[0][0];
#pragma unroll
  for (int w = 1; w < kMergeThreads / 32; ++w) top = fmaxf(top, scratch[w][0]);
  const float f = mine ? weight_of(ml.x, top) : 0.0f;
  if (mine) weight[threadIdx.x] = f;
  const float part = warp_fold<IB_OP_ADD>(ml.y * f);
  if (lane == 0) scratch[warp][1] = part;
  __syncthreads();
  const int c = threadIdx.x % 128, group = threadIdx.x / 128;
  float acc = 0.0f;
  if (c < dv) {
    const float* at = partial_o + row * splits * dv + c;
#pragma unroll 8
    for (int s = group; s < splits; s += kMergeGroups) acc = fmaf(at[static_cast<size_t>(s) * dv], weight[s], acc);
  }
  meet[group][c] = acc;
  __syncthreads();
  if (group != 0 || c >= dv) return;
  float sum = 0.0f;
#pragma unroll
  for (int w = 0; w < kMergeThreads / 32; ++w) sum += scratch[w][1];
#pragma unroll
  for (int g = 1; g < kMergeGroups; ++g) acc += meet[g][c];
  o[row * dv + c] = acc / sum;
}

struct DirectPlan {
  int nq_per_cta, splits, blocks_per_split;
  size_t groups;
  bool cluster;
};

// Queries per CTA: as many as are there, up to eight, but fewer while the warps (one per 32 keys and
// group of queries) would not give every scheduler of the machine one.  Key ranges: enough CTAs
// for two or three per SM (what fits), each at least one block of keys per warp; up to eight of
// them form a cluster, more (few heads, long contexts) meet in a second kernel.
DirectPlan direct_plan(size_t batch, size_t nq, size_t nk) {
  DirectPlan p;
  const size_t blocks = (nk + kBlockKeys - 1) / kBlockKeys;
  int n = 1;
  while (n < 8 && static_cast<size_t>(n) < nq) n *= 2;
  while (n > 1 && batch * ((nq + n - 1) / n) * blocks < static_cast<size_t>(kNumSMs) * 4) n /= 2;
  p.nq_per_cta = n;
  p.groups = (nq + n - 1) / n;
  const size_t units = batch * p.groups;
  const size_t room = static_cast<size_t>(kNumSMs) * (n >= 4 ? 2 : 3);
  size_t splits = units ? room / units : 1;
  if (splits > blocks / kWarps) splits = blocks / kWarps;
  if (splits > static_cast<size_t>(kMaxSplits)) splits = kMaxSplits;
  if (splits > static_cast<size_t>(kMaxCluster) && splits < 2 * static_cast<size_t>(kMaxCluster)) splits = kMaxCluster;
  if (splits < 1) splits = 1;
  const size_t per = (blocks + splits - 1) / splits;
  p.blocks_per_split = static_cast<int>(per);
  p.splits = static_cast<int>((blocks + per - 1) / per);
  p.cluster = p.splits > 1 && p.splits <= kMaxCluster;
  return p;
}

template <int LP, int NQ>
cudaError_t launch_direct(const DirectArgs& a, size_t ctas, bool cluster, cudaStream_t s) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = static_cast<unsigned>(a.splits);
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(ctas));
  cfg.blockDim = dim3(kThreads);
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = cluster ? 1 : 0;
  return cluster ? cudaLaunchKernelEx(&cfg, attention_direct_kernel<LP, NQ, true>, a)
                 : cudaLaunchKernelEx(&cfg, attention_direct_kernel<LP, NQ, false>, a);
}

template <int LP>
cudaError_t launch_direct_nq(int nq, const DirectArgs& a, size_t ctas, bool cluster, cudaStream_t s) {
  if (nq == 1) return launch_direct<LP, 1>(a, ctas, cluster, s);
  if (nq == 2) return launch_direct<LP, 2>(a, ctas, cluster, s);
  if (nq == 4) return launch_direct<LP, 4>(a, ctas, cluster, s);
  return launch_direct<LP, 8>(a, ctas, cluster, s);
}

}  // namespace

bool attention_direct_shape_ok(size_t batch, size_t nq, size_t nk, size_t d, size_t dv) {
  if (d < 1 || d > 128 || dv < 1 || dv > 128 || nk < 1 || nq < 1 || batch < 1) return false;
  if (nk > (static_cast<size_t>(1) << 35)) return false;                 // blocks per split are an int
  return batch <= (static_cast<size_t>(1) << 24) && nq <= (static_cast<size_t>(1) << 24) &&
         batch * nq <= (static_cast<size_t>(1) << 27);                   // CTAs are a 31-bit grid
}

// Estimated time.  A CTA takes about as long with one warp busy (32 keys or fewer) as with all eight (256
// keys), so the time is the number of rounds of CTAs, times the blocks of keys a warp takes in turn, times
// what a block takes for so many queries and features; the last round counts in full.
double attention_direct_us(size_t batch, size_t nq, size_t nk, size_t d, size_t dv) {
  const DirectPlan p = direct_plan(batch, nq, nk);
  const size_t widest = d > dv ? d : dv, features = widest <= 32 ? 32 : widest <= 64 ? 64 : 128;
  const size_t room = static_cast<size_t>(kNumSMs) * (p.nq_per_cta >= 4 ? 2 : 3);
  const size_t rounds = (batch * p.groups * static_cast<size_t>(p.splits) + room - 1) / room;
  const size_t blocks = (static_cast<size_t>(p.blocks_per_split) + kWarps - 1) / kWarps;
  return 2.0 + static_cast<double>(rounds * blocks) *
                   (1.5 + 0.55 * p.nq_per_cta + (0.04 + 0.004 * p.nq_per_cta) * static_cast<double>(features));
}

// Whether the last round of CTAs leaves much of the machine idle, where there are too many heads to divide
// their keys evenly.
bool attention_direct_idles(size_t batch, size_t nq, size_t nk) {
  const DirectPlan p = direct_plan(batch, nq, nk);
  const double room = kNumSMs * (p.nq_per_cta >= 4 ? 2.0 : 3.0);
  const double units = static_cast<double>(batch * p.groups), ctas = units * p.splits;
  return units * 3.0 > room && ctas < (p.splits > 1 ? 0.7 : 0.6) * room * std::ceil(ctas / room);
}

size_t attention_direct_floats(size_t batch, size_t nq, size_t nk, size_t dv) {
  const DirectPlan p = direct_plan(batch, nq, nk);
  return p.splits == 1 || p.cluster ? 0 : batch * nq * static_cast<size_t>(p.splits) * (dv + 2);
}

int attention_direct(const float* q, const float* k, const float* v, float* o, size_t batch, size_t nq,
                     size_t nk, size_t d, size_t dv, const float* logit_scale, bool logit_divide,
                     float* partials, cudaStream_t s) {
  const DirectPlan p = direct_plan(batch, nq, nk);
  DirectArgs a{};
  a.q = q;
  a.k = k;
  a.v = v;
  a.o = o;
  if (partials) {
    a.partial_ml = reinterpret_cast<float2*>(partials);                  // 8-byte aligned: ahead of the odd-sized part
    a.partial_o = partials + 2 * batch * nq * static_cast<size_t>(p.splits);
  }
  a.logit_scale = logit_scale;
  a.logit_divide = logit_divide ? 1 : 0;
  a.nq = nq;
  a.nk = nk;
  a.groups = p.groups;
  a.d = static_cast<int>(d);
  a.dv = static_cast<int>(dv);
  a.splits = p.splits;
  a.blocks_per_split = p.blocks_per_split;
  a.vec = d % 4 == 0 && dv % 4 == 0 && aligned16(q) && aligned16(k) && aligned16(v);
  const size_t ctas = batch * p.groups * static_cast<size_t>(p.splits);
  const size_t widest = d > dv ? d : dv;
  const cudaError_t err = widest <= 32   ? launch_direct_nq<8>(p.nq_per_cta, a, ctas, p.cluster, s)
                          : widest <= 64 ? launch_direct_nq<16>(p.nq_per_cta, a, ctas, p.cluster, s)
                                         : launch_direct_nq<32>(p.nq_per_cta, a, ctas, p.cluster, s);
  if (err != cudaSuccess) {
    cudaGetLastError();
    return fail(std::string("ib_attention (fp32): ") + cudaGetErrorString(err));
  }
  count_launch();
  if (p.splits == 1 || p.cluster) return 0;
  attention_direct_merge_kernel<<<static_cast<unsigned>(batch * nq), kMergeThreads, 0, s>>>(
      a.partial_o, a.partial_ml, o, p.splits, a.dv);
  return check_launch("ib_attention (fp32 merge)");
}

}  // namespace ib
