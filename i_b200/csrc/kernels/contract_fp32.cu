// CUDA-core fp32 contraction: the IB_PRECISION_FP32 arm of ib_contract, and what AUTO takes for
// products too small or too ragged for the tensor path (odd K, tiny tiles such as the 8x16x7 product
// of ilang-python/test.py:52-56).  C[b][i][j] = sum_k A(b,i,k) B(b,j,k), the arithmetic of the
// reference's loop nest (ilang-python/annotated-flashattn.c:57-89) up to summation order and FMA
// contraction.
//
// Bound: the FMA pipes, 128 multiply-adds per clock and SM.  What keeps a tile kernel from them is
// issue slots and shared-memory reads, so a thread owns TM x TN results (8 x 8 in the large tiles),
// reads both operands as 16-byte quads (4 reads for 64 multiply-adds) and multiplies with fma.rn.f32x2,
// two results per instruction (32 instead of 64 a step, each lane rounded as a plain fma).  Tiles of
// both operands go through registers into [k][row] shared memory whatever their layout, the next
// tile's loads in flight while the current one is multiplied, one barrier per tile.
//
// Results too few for the machine: a product is cut along k into up to eight parts, the CTAs of one
// cluster, whose sums meet in distributed shared memory: no workspace, no second launch, a fixed
// order.  Tile and parts are chosen by an estimate (choose below).  Where even eight parts leave SMs
// idle on a deep product, several clusters take a tile and their sums go through copies of the result
// (fp32_copies).
//
// Measured on B200, against 64 x 64 tiles of 4 x 4 results with 4-byte shared-memory reads: 1024 x
// 1000 x 1001 145 -> 62 us, 2048 x 2048 x 512 105 us (41 TFLOP/s), 32 x 32 x 2048 226 -> 10 us.  At 1024 x 1000 x
// 1001 the FMA pipe is busy 62 % of the time; stalls: the pipe itself, and waits between a quad's packing and its use.
#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.h"

namespace ib {
namespace {

namespace cg = cooperative_groups;

constexpr int kMaxParts = 8;               // portable cluster size

struct Operand {
  const float* p;
  size_t rows;                             // m or n
  bool vec;                                // 16-byte loads along its contiguous axis
};

struct Fp32Args {
  Operand a, b;
  float* c;
  size_t k, k_len;
  unsigned tiles_n, parts, copies;         // blockIdx.y = batch entry * copies + copy
  bool c_vec;
};

__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long both(float x) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ unsigned long long joined(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 halves(unsigned long long x) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x));
  return r;
}

// A thread's share of an operand's ROWS x TK tile on its way to shared memory.
template <int ROWS, int TK, int THREADS, bool KMAJOR>
struct Stage {
  static constexpr int kPer = ROWS * TK / THREADS;
  static_assert(kPer % 4 == 0, "whole quads per thread");
  float v[kPer];

  __device__ __forceinline__ void load(const Operand& op, const float* base, size_t row0, size_t k, size_t k0,
                                       size_t k_hi) {
    if (op.vec) {
#pragma unroll
      for (int i = 0; i < kPer / 4; ++i) {
        const int e = threadIdx.x + i * THREADS;
        const int row = KMAJOR ? e / (TK / 4) : (e % (ROWS / 4)) * 4, kk = KMAJOR ? (e % (TK / 4)) * 4 : e / (ROWS / 4);
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (row0 + row < op.rows && k0 + kk < k_hi)
          x = __ldg(reinterpret_cast<const float4*>(KMAJOR ? base + (row0 + row) * k + k0 + kk
                                                           : base + (k0 + kk) * op.rows + row0 + row));
        v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const int e = threadIdx.x + i * THREADS;
        const int row = KMAJOR ? e / TK : e % ROWS, kk = KMAJOR ? e % TK : e / ROWS;
        v[i] = row0 + row < op.rows && k0 + kk < k_hi
                   ? __ldg(KMAJOR ? base + (row0 + row) * k + k0 + kk : base + (k0 + kk) * op.rows + row0 + row)
                   : 0.0f;
      }
    }
  }

  __device__ __forceinline__ void store(float (*tile)[ROWS + 4], bool vec) const {
    if (vec) {
#pragma unroll
      for (int i = 0; i < kPer / 4; ++i) {
        const int e = threadIdx.x + i * THREADS;
        if (KMAJOR) {
#pragma unroll
          for (int j = 0; j < 4; ++j) tile[(e % (TK / 4)) * 4 + j][e / (TK / 4)] = v[4 * i + j];
        } else {
          *reinterpret_cast<float4*>(&tile[e / (ROWS / 4)][(e % (ROWS / 4)) * 4]) =
              make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const int e = threadIdx.x + i * THREADS;
        tile[KMAJOR ? e % TK : e / ROWS][KMAJOR ? e / TK : e % ROWS] = v[i];
      }
    }
  }
};

// v = op(v, t), or op(t, v) with `right`: the arithmetic of the pointwise kernels, for the operators that
// may follow a contraction.  One operator of the caller's list at a time, behind a switch in a loop that is
// not unrolled, so nothing is contracted across operators.
template <int N>
__device__ __forceinline__ void apply_operator(int op, bool right, float (&v)[N], const float (&t)[N]) {
#define IB_FP32_CASE(OP)                                                                             \
  case OP:                                                                                           \
    if (right) {                                                                                     \
      _Pragma("unroll") for (int j = 0; j < N; ++j) v[j] = apply_binary(OP, t[j], v[j]);             \
    } else {                                                                                         \
      _Pragma("unroll") for (int j = 0; j < N; ++j) v[j] = apply_binary(OP, v[j], t[j]);             \
    }                                                                                                \
    break;
  switch (op) {
    IB_FP32_CASE(IB_OP_ADD)
    IB_FP32_CASE(IB_OP_SUB)
    IB_FP32_CASE(IB_OP_MUL)
    IB_FP32_CASE(IB_OP_MAX)
    IB_FP32_CASE(IB_OP_MIN)
  }
#undef IB_FP32_CASE
}

// The one-operand form is the two-operand one with 0 in front, but for + and *, which change nothing.
__device__ __forceinline__ bool changes_nothing(const GemmEpilogue& e, int k) {
  return e.which[k] < 0 && (e.op[k] == IB_OP_ADD || e.op[k] == IB_OP_MUL);
}

__device__ __forceinline__ void load_quad(float* t, const float* p, size_t col, size_t n, bool vec) {
  if (vec && col < n) {
    const float4 x = __ldg(reinterpret_cast<const float4*>(p + col));
    t[0] = x.x; t[1] = x.y; t[2] = x.z; t[3] = x.w;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) t[j] = col + j < n ? __ldg(p + col + j) : 0.0f;
  }
}

// The caller's operators on all results of a thread, four rows at a time so that an operand's loads are in
// flight together.  (A call per four results, each waiting for its own loads and switching over all
// eighteen operators, took longer than a pass of its own where the product is short: 4096 x 4096 x 16 with
// a row factor and a rectifier 139 us, as two passes 60, now 27; 8000 x 8000 x 9 with bias and rectifier 484,
// 206, now 94.)
template <int TM, int TN, int BM, int BN>
__device__ __forceinline__ void fp32_epilogue(const GemmEpilogue& e, unsigned long long (&acc)[TM][TN / 2],
                                              size_t first_row, size_t i0, size_t m, size_t j0, size_t n, int ty,
                                              int tx) {
  constexpr int kQm = TM / 4, kQn = TN / 4;
#pragma unroll 1
  for (int k = 0; k < e.n_ops; ++k) {
    if (changes_nothing(e, k)) continue;
    const int w = e.which[k];
    const float* p = w < 0 ? nullptr : e.operand[w];
    const int mode = w < 0 ? 4 : e.mode[w];
    const bool vec = n % 4 == 0 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0;
#pragma unroll
    for (int h = 0; h < kQm; ++h) {
      const size_t row = i0 + h * (BM / kQm) + ty * 4;
      float t[4 * TN], v[4 * TN];
      if (mode == 0) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int q = 0; q < kQn; ++q)
            load_quad(&t[u * TN + 4 * q], p + (first_row + row + u) * n, j0 + q * (BN / kQn) + tx * 4,
                      row + u < m ? n : 0, vec);
      } else if (mode == 2) {
#pragma unroll
        for (int q = 0; q < kQn; ++q) load_quad(&t[4 * q], p, j0 + q * (BN / kQn) + tx * 4, n, vec);
#pragma unroll
        for (int j = TN; j < 4 * TN; ++j) t[j] = t[j % TN];
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float x = mode == 1 ? (row + u < m ? __ldg(p + first_row + row + u) : 0.0f) : mode == 3 ? __ldg(p) : 0.0f;
#pragma unroll
          for (int j = 0; j < TN; ++j) t[u * TN + j] = x;
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int c = 0; c < TN / 2; ++c) {
          const float2 x = halves(acc[4 * h + u][c]);
          v[u * TN + 2 * c] = x.x;
          v[u * TN + 2 * c + 1] = x.y;
        }
      apply_operator(e.op[k], w < 0 || e.acc_right[k] != 0, v, t);
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int c = 0; c < TN / 2; ++c) acc[4 * h + u][c] = joined(v[u * TN + 2 * c], v[u * TN + 2 * c + 1]);
    }
  }
}

// The same on four neighbouring results of one row, for the sums of a product cut along k.
__device__ __noinline__ float4 fp32_epilogue_quad(const GemmEpilogue& e, float4 r, size_t grow, size_t col, size_t n) {
  float v[4] = {r.x, r.y, r.z, r.w};
#pragma unroll 1
  for (int k = 0; k < e.n_ops; ++k) {
    if (changes_nothing(e, k)) continue;
    const int w = e.which[k];
    const float* p = w < 0 ? nullptr : e.operand[w];
    const int mode = w < 0 ? 4 : e.mode[w];
    float t[4];
    if (mode == 0 || mode == 2) {
      load_quad(t, mode == 0 ? p + grow * n : p, col, n, n % 4 == 0 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0);
    } else {
      t[0] = t[1] = t[2] = t[3] = mode == 4 ? 0.0f : __ldg(mode == 1 ? p + grow : p);
    }
    apply_operator(e.op[k], w < 0 || e.acc_right[k] != 0, v, t);
  }
  return make_float4(v[0], v[1], v[2], v[3]);
}

__device__ __forceinline__ void put_quad(float* c, float4 r, size_t grow, size_t col, size_t n, bool vec) {
  float* at = c + grow * n + col;
  if (vec && col + 4 <= n) {
    *reinterpret_cast<float4*>(at) = r;
  } else {
    if (col < n) at[0] = r.x;
    if (col + 1 < n) at[1] = r.y;
    if (col + 2 < n) at[2] = r.z;
    if (col + 3 < n) at[3] = r.w;
  }
}

template <int BM, int BN, int TK, int TM, int TN, bool AK, bool BK>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), 512 / ((BM / TM) * (BN / TN)))
contract_fp32_kernel(const __grid_constant__ Fp32Args g, const __grid_constant__ GemmEpilogue epilogue) {
  constexpr int kThreads = (BM / TM) * (BN / TN);
  constexpr int kQm = TM / 4, kQn = TN / 4;
  constexpr int kAcross = BN / TN;           // threads along a row of results
  constexpr size_t kTileFloats = 2 * TK * (BM + 4 + BN + 4);
  constexpr size_t kMeetFloats = BM * BN <= 64 * 128 ? BM * BN : 0;      // larger tiles are never cut along k
  __shared__ __align__(16) float smem[kTileFloats > kMeetFloats ? kTileFloats : kMeetFloats];
  float(*sa)[TK][BM + 4] = reinterpret_cast<float(*)[TK][BM + 4]>(smem);
  float(*sb)[TK][BN + 4] = reinterpret_cast<float(*)[TK][BN + 4]>(smem + 2 * TK * (BM + 4));

  const unsigned tile = blockIdx.x / g.parts, part = blockIdx.x - tile * g.parts;
  const size_t i0 = static_cast<size_t>(tile / g.tiles_n) * BM, j0 = static_cast<size_t>(tile % g.tiles_n) * BN;
  const size_t m = g.a.rows, n = g.b.rows, out = blockIdx.y, batch = out / g.copies;
  const float* a = g.a.p + batch * m * g.k;
  const float* b = g.b.p + batch * n * g.k;
  const size_t k_lo = ((out - batch * g.copies) * g.parts + part) * g.k_len, k_hi = k_lo + g.k_len < g.k ? k_lo + g.k_len : g.k;
  const int tx = threadIdx.x % kAcross, ty = threadIdx.x / kAcross;

  unsigned long long acc[TM][TN / 2];
#pragma unroll
  for (int u = 0; u < TM; ++u)
#pragma unroll
    for (int w = 0; w < TN / 2; ++w) acc[u][w] = 0;

  Stage<BM, TK, kThreads, AK> fa;
  Stage<BN, TK, kThreads, BK> fb;
  if (k_lo < k_hi) {
    fa.load(g.a, a, i0, g.k, k_lo, k_hi);
    fb.load(g.b, b, j0, g.k, k_lo, k_hi);
    fa.store(sa[0], g.a.vec);
    fb.store(sb[0], g.b.vec);
  }
  __syncthreads();
  int buf = 0;
  for (size_t k0 = k_lo; k0 < k_hi; k0 += TK) {
    const bool more = k0 + TK < k_hi;
    if (more) {
      fa.load(g.a, a, i0, g.k, k0 + TK, k_hi);
      fb.load(g.b, b, j0, g.k, k0 + TK, k_hi);
    }
#pragma unroll
    for (int kk = 0; kk < TK; ++kk) {
      float av[TM];
      unsigned long long bv[TN / 2];
#pragma unroll
      for (int q = 0; q < kQm; ++q)
        *reinterpret_cast<float4*>(&av[4 * q]) = *reinterpret_cast<const float4*>(&sa[buf][kk][q * (BM / kQm) + ty * 4]);
#pragma unroll
      for (int q = 0; q < kQn; ++q)
        *reinterpret_cast<ulonglong2*>(&bv[2 * q]) =
            *reinterpret_cast<const ulonglong2*>(&sb[buf][kk][q * (BN / kQn) + tx * 4]);
#pragma unroll
      for (int u = 0; u < TM; ++u) {
        const unsigned long long aa = both(av[u]);
#pragma unroll
        for (int w = 0; w < TN / 2; ++w) fma2(acc[u][w], aa, bv[w]);
      }
    }
    if (more) {
      fa.store(sa[buf ^ 1], g.a.vec);
      fb.store(sb[buf ^ 1], g.b.vec);
    }
    __syncthreads();
    buf ^= 1;
  }

  if (g.parts == 1) {
    if (epilogue.n_ops) fp32_epilogue<TM, TN, BM, BN>(epilogue, acc, out * m, i0, m, j0, n, ty, tx);
#pragma unroll
    for (int u = 0; u < TM; ++u) {
      const size_t gi = i0 + (u / 4) * (BM / kQm) + ty * 4 + u % 4;
      if (gi >= m) continue;
#pragma unroll
      for (int q = 0; q < kQn; ++q) {
        const float2 lo = halves(acc[u][2 * q]), hi = halves(acc[u][2 * q + 1]);
        put_quad(g.c, make_float4(lo.x, lo.y, hi.x, hi.y), out * m + gi, j0 + q * (BN / kQn) + tx * 4, n, g.c_vec);
      }
    }
    return;
  }
  if constexpr (kMeetFloats > 0) {
    // The parts meet: every CTA leaves its sums in shared memory, each adds a share of the tile.
    float4* meet = reinterpret_cast<float4*>(smem);
#pragma unroll
    for (int u = 0; u < TM; ++u)
#pragma unroll
      for (int q = 0; q < kQn; ++q) {
        const float2 lo = halves(acc[u][2 * q]), hi = halves(acc[u][2 * q + 1]);
        meet[((u / 4) * (BM / kQm) + ty * 4 + u % 4) * (BN / 4) + q * (BN / kQn) / 4 + tx] =
            make_float4(lo.x, lo.y, hi.x, hi.y);
      }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    for (unsigned e = part * kThreads + threadIdx.x; e < BM * BN / 4; e += g.parts * kThreads) {
      const size_t gi = i0 + e / (BN / 4), gj = j0 + (e % (BN / 4)) * 4;
      if (gi >= m || gj >= n) continue;
      float4 x[kMaxParts];
#pragma unroll
      for (unsigned p = 0; p < kMaxParts; ++p)
        if (p < g.parts) x[p] = *cluster.map_shared_rank(&meet[e], p);
      float4 sum = x[0];
#pragma unroll
      for (unsigned p = 1; p < kMaxParts; ++p)
        if (p < g.parts) {
          sum.x += x[p].x; sum.y += x[p].y; sum.z += x[p].z; sum.w += x[p].w;
        }
      if (epilogue.n_ops) sum = fp32_epilogue_quad(epilogue, sum, out * m + gi, gj, n);
      put_quad(g.c, sum, out * m + gi, gj, n, g.c_vec);
    }
    cluster.sync();                          // nobody leaves while its shared memory is read
  }
}

struct Choice {
  int tile;                                  // index into the tile list
  size_t parts;
};

struct TileShape {
  size_t bm, bn;
  double one, most;                          // share of the FMA rate with one CTA on an SM, with several
};
constexpr TileShape kTiles[] = {{128, 128, 0.53, 0.68}, {64, 128, 0.45, 0.65}, {64, 64, 0.30, 0.55}, {32, 32, 0.13, 0.34}};

// Tile and parts with the least estimated time: the busiest SM's share of the multiply-adds at the
// rate its number of resident CTAs reaches, plus a cost for the meeting of parts.  The rates are
// measured (one CTA: latency of shared memory and loads is exposed; several: it is covered), as is the
// meeting (about 1.5 us more for a cluster launch and its two barriers).
Choice choose(size_t batch, size_t m, size_t n, size_t k) {
  Choice best{3, 1};
  double best_time = 1e300;
  for (int t = 0; t < 4; ++t) {
    const TileShape& s = kTiles[t];
    const double tiles = static_cast<double>(batch) * ((m + s.bm - 1) / s.bm) * ((n + s.bn - 1) / s.bn);
    for (size_t parts = 1; parts <= static_cast<size_t>(kMaxParts); ++parts) {
      if (parts > 1 && (t == 0 || k < parts * 2 * 16)) break;
      const double per_sm = static_cast<double>(static_cast<size_t>((tiles * parts + kNumSMs - 1) / kNumSMs));
      const size_t k_len = ((k + parts - 1) / parts + 16 - 1) / 16 * 16;
      const double rate = s.one * per_sm < s.most ? s.one * per_sm : s.most;
      const double time = per_sm * k_len * s.bm * s.bn / 128 / rate + (parts > 1 ? 3000 + 0.15 * s.bm * s.bn / 4 : 0);
      if (time < best_time) {
        best_time = time;
        best = Choice{t, parts};
      }
    }
  }
  return best;
}

template <int BM, int BN, int TK, int TM, int TN>
cudaError_t launch_tile(Fp32Args g, const GemmEpilogue& e, size_t batch, size_t parts, size_t copies, bool ak,
                        bool bk, cudaStream_t s) {
  const size_t tiles_m = (g.a.rows + BM - 1) / BM, tiles_n = (g.b.rows + BN - 1) / BN;
  const size_t ctas = tiles_m * tiles_n * parts;
  if (ctas > 0x7fffffffu || tiles_n > 0x7fffffffu) return cudaErrorInvalidConfiguration;
  g.tiles_n = static_cast<unsigned>(tiles_n);
  g.parts = static_cast<unsigned>(parts);
  g.copies = static_cast<unsigned>(copies);
  // Whole k-tiles per part, so that every part but the last ones is full.
  const size_t cuts = parts * copies;
  g.k_len = ((g.k + cuts - 1) / cuts + TK - 1) / TK * TK;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = static_cast<unsigned>(parts);
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(ctas), static_cast<unsigned>(batch * copies));
  cfg.blockDim = dim3((BM / TM) * (BN / TN));
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = parts > 1 ? 1 : 0;
  if (ak) return bk ? cudaLaunchKernelEx(&cfg, contract_fp32_kernel<BM, BN, TK, TM, TN, true, true>, g, e)
                    : cudaLaunchKernelEx(&cfg, contract_fp32_kernel<BM, BN, TK, TM, TN, true, false>, g, e);
  return bk ? cudaLaunchKernelEx(&cfg, contract_fp32_kernel<BM, BN, TK, TM, TN, false, true>, g, e)
            : cudaLaunchKernelEx(&cfg, contract_fp32_kernel<BM, BN, TK, TM, TN, false, false>, g, e);
}

}  // namespace

// Copies of the result a deep product with few tiles is summed into (1 = none): two CTAs per SM, at
// least 128 terms each.  The copies cost a second launch (3-4 us with the fold), so only where they
// halve the chain of a part: 30 x 257 x 12288 on B200 43 us with one cluster per tile.
size_t fp32_copies(size_t batch, size_t m, size_t n, size_t k) {
  const Choice pick = choose(batch, m, n, k);
  if (pick.parts != static_cast<size_t>(kMaxParts)) return 1;
  const TileShape& s = kTiles[pick.tile];
  const size_t ctas = batch * ((m + s.bm - 1) / s.bm) * ((n + s.bn - 1) / s.bn) * pick.parts;
  size_t copies = 2 * static_cast<size_t>(kNumSMs) / ctas;
  if (copies > k / (pick.parts * 128)) copies = k / (pick.parts * 128);
  if (copies > 16) copies = 16;
  if (batch * copies > 65535) return 1;
  return copies < 2 ? 1 : copies;
}

int contract_fp32(const float* a, const float* b, float* c, size_t batch, size_t m, size_t n, size_t k,
                  bool a_kmajor, bool b_kmajor, cudaStream_t s, const GemmEpilogue* e, float* copies) {
  if (batch == 0 || m == 0 || n == 0) return 0;
  if (batch > 65535) return fail("ib_contract: more than 65535 batch entries");
  // 16-byte loads need every row of the operand, in every batch entry, to start on 16 bytes.
  Fp32Args g{};
  g.a = Operand{a, m, (a_kmajor ? k : m) % 4 == 0 && aligned16(a)};
  g.b = Operand{b, n, (b_kmajor ? k : n) % 4 == 0 && aligned16(b)};
  const size_t n_copies = copies ? fp32_copies(batch, m, n, k) : 1;
  g.c = n_copies > 1 ? copies : c;
  g.k = k;
  g.c_vec = n % 4 == 0 && aligned16(g.c);
  const Choice pick = choose(batch, m, n, k);
  const GemmEpilogue none{};
  const GemmEpilogue& ep = e && n_copies == 1 ? *e : none;
  cudaError_t err;
  switch (pick.tile) {
    case 0: err = launch_tile<128, 128, 16, 8, 8>(g, ep, batch, pick.parts, n_copies, a_kmajor, b_kmajor, s); break;
    case 1: err = launch_tile<64, 128, 16, 8, 8>(g, ep, batch, pick.parts, n_copies, a_kmajor, b_kmajor, s); break;
    case 2: err = launch_tile<64, 64, 32, 8, 4>(g, ep, batch, pick.parts, n_copies, a_kmajor, b_kmajor, s); break;
    default: err = launch_tile<32, 32, 32, 4, 4>(g, ep, batch, pick.parts, n_copies, a_kmajor, b_kmajor, s); break;
  }
  if (err != cudaSuccess) {
    cudaGetLastError();
    return fail(std::string("ib_contract (fp32): ") + cudaGetErrorString(err));
  }
  count_launch();
  return n_copies > 1 ? sum_partials(copies, c, batch, n_copies, m * n, s) : 0;
}

}  // namespace ib
