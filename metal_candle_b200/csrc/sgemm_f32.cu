// float32 path of the fused LoRA linear on CUDA cores with float32 FMA accumulation.  tcgen05 has no float32 MMA and a
// single TF32 pass cannot hold the 1e-4 bound against the reference's f32 CPU arithmetic, so the contractions run on
// the FMA pipes (148 SMs x 128 lanes = 74 TFLOP/s at the maximum clock), as four kinds of kernel:
//
//   tile_kernel    C = A B (+ bias) (+ residual) with the rank-r update as extra reduction steps: 128 x 64 tiles,
//                  the reduction split over the CTAs of a cluster when a shape has too few tiles for the chip
//   rank_kernel    the [M, r] intermediates scale * x A and scale * dy B^T
//   grad_kernel    dA and dB, reductions over tokens
//   lora_delta_cluster_kernel   scale * (x A) B of few tokens in one launch (also for bfloat16 x)
#include <cooperative_groups.h>

#include "lora_internal.cuh"

namespace cg = cooperative_groups;

namespace mcb {
namespace f32path {
namespace {

// ---- asynchronous copies (0 source bytes: the destination is zero-filled) ------------------------------------------
__device__ __forceinline__ void cp4(uint32_t dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp4_or_zero(uint32_t dst, const float* src, const float* any, bool in) {
  const int n = in ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(in ? src : any), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ---- tile kernel -------------------------------------------------------------------------------------------------
// An operand as the kernel reads it: element (row, k) at p[row * sr + k * sk].
struct Operand {
  const float* p;
  int64_t sr, sk;
};
struct TileParams {
  Operand a, b;      // [M, K] and [N, K]
  Operand ra, rb;    // rank part: [M, R] and [N, R]
  int M, N, K, R;    // C = alpha (A B + ra rb) (+ bias) (+ residual) (+ C)
  float alpha;
  const float *bias, *residual;         // [N]; laid out like C
  float* C;                             // element (m, n) at C[m * cm + n * cn]
  int64_t cm, cn;
  int accumulate;
  int n_tiles, splits;
};

constexpr int kTileM = 128, kTileN = 64, kStep = 32, kStages = 2, kTileThreads = 64;
// A stage holds both tiles as [k][row]; the row pitches are 4 mod 32 words, so that the 8 k x 4 rows (or 32 rows) a warp
// copies at a time fall into 32 different banks.
constexpr int kPitchA = kTileM + 4, kPitchB = kTileN + 4;
constexpr int kStageFloats = kStep * (kPitchA + kPitchB);
constexpr int kOutPitch = kTileN + 4, kMaxSplits = 8;
static_assert(kTileM * kOutPitch <= kStages * kStageFloats, "the output tile reuses the stage ring");

// Word copies serve every stride and alignment and transpose on the way; neighbouring lanes read neighbouring words
// (8 k of a row where k is the contiguous index, else consecutive rows).  Whole tiles skip the bounds checks.
template <int ROWS, int PITCH>
__device__ __forceinline__ void load_tile(uint32_t dst, const Operand& o, int row0, int rows, int k0, int kend) {
  const int t = threadIdx.x;
  const bool whole = row0 + ROWS <= rows && k0 + kStep <= kend;
  if (o.sk == 1) {
    const int kk = t & 7, rr = t >> 3;   // 8 rows x 8 k per round of the CTA's two warps
    const float* src = o.p + (row0 + rr) * o.sr + k0 + kk;
    dst += (kk * PITCH + rr) * 4;
    const int64_t jump = 8 * o.sr;
    if (whole) {
#pragma unroll 4
      for (int i = 0; i < ROWS / 8; ++i, src += jump) {
#pragma unroll
        for (int h = 0; h < kStep / 8; ++h) cp4(dst + (8 * h * PITCH + 8 * i) * 4, src + 8 * h);
      }
    } else {
      for (int i = 0; i < ROWS / 8; ++i, src += jump) {
        const bool row_in = row0 + rr + 8 * i < rows;
#pragma unroll
        for (int h = 0; h < kStep / 8; ++h)
          cp4_or_zero(dst + (8 * h * PITCH + 8 * i) * 4, src + 8 * h, o.p, row_in && k0 + kk + 8 * h < kend);
      }
    }
  } else {
    const int r = t % ROWS, k = t / ROWS;   // 64 threads: half of A's rows, or all of B's, at one k
    constexpr int kSub = ROWS > kTileThreads ? ROWS / kTileThreads : 1;
    const float* src = o.p + (row0 + r) * o.sr + (k0 + k) * o.sk;
    dst += (k * PITCH + r) * 4;
    const int64_t hop = kTileThreads * o.sr;
    for (int i = 0; i < kStep; ++i, src += o.sk)
#pragma unroll
      for (int h = 0; h < kSub; ++h) {
        const uint32_t d = dst + (i * PITCH + h * kTileThreads) * 4;
        if (whole) cp4(d, src + h * hop);
        else cp4_or_zero(d, src + h * hop, o.p, row0 + r + h * kTileThreads < rows && k0 + i < kend);
      }
  }
}

// Bound: the FMA pipe, with shared-memory reads next.  A thread owns 16 x 8 outputs: 6 LDS.128 feed 128 FMAs, which keeps
// the reads below the 128 bytes per cycle an SM has; the FMAs are packed pairs (fma.rn.f32x2), which leaves issue slots
// for the copies.  2048 x 1536 x 1536: 262 us (37 TFLOP/s; 64 x 64 tiles of 4 x 4 outputs took 480), 512 x 768 x 768: 29
// us (240).  A shape with few tiles (512 x 768 x 768: 48) leaves SMs idle, so up to 8 CTAs of a cluster share a tile's
// reduction and add their partial tiles through distributed shared memory, in rank order: deterministic, no workspace.
__global__ void __launch_bounds__(kTileThreads, 4) tile_kernel(const TileParams p) {
  extern __shared__ __align__(16) float smem[];
  const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const int split = blockIdx.x % p.splits, tile = blockIdx.x / p.splits;
  const int m0 = (tile / p.n_tiles) * kTileM, n0 = (tile % p.n_tiles) * kTileN;
  // main steps are shared out evenly; the rank steps go to the last CTA of the cluster
  const int ksteps = (p.K + kStep - 1) / kStep;
  const int s_begin = static_cast<int>(static_cast<int64_t>(ksteps) * split / p.splits);
  const int s_end = static_cast<int>(static_cast<int64_t>(ksteps) * (split + 1) / p.splits);
  const int main_steps = s_end - s_begin;
  const int steps = main_steps + (split == p.splits - 1 ? (p.R + kStep - 1) / kStep : 0);
  auto load_step = [&](int s) {
    const uint32_t da = sbase + (s % kStages) * kStageFloats * 4, db = da + kStep * kPitchA * 4;
    if (s < main_steps) {
      const int k0 = (s_begin + s) * kStep;
      load_tile<kTileM, kPitchA>(da, p.a, m0, p.M, k0, p.K);
      load_tile<kTileN, kPitchB>(db, p.b, n0, p.N, k0, p.K);
    } else if (s < steps) {
      const int k0 = (s - main_steps) * kStep;
      load_tile<kTileM, kPitchA>(da, p.ra, m0, p.M, k0, p.R);
      load_tile<kTileN, kPitchB>(db, p.rb, n0, p.N, k0, p.R);
    }
    cp_commit();   // one group per step, empty or not
  };
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;   // rows 4 ty + 32 i + (0..3), columns 4 tx + 32 j + (0..3)
  float2 acc[16][4];
#pragma unroll
  for (int i = 0; i < 16; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
  for (int s = 0; s < kStages - 1; ++s) load_step(s);
  for (int s = 0; s < steps; ++s) {
    cp_wait<kStages - 2>();
    __syncthreads();            // step s has landed, and every thread is through with step s - 1
    load_step(s + kStages - 1);
    const float* sa = smem + (s % kStages) * kStageFloats + 4 * ty;
    const float* sb = smem + (s % kStages) * kStageFloats + kStep * kPitchA + 4 * tx;
    // a step's indices behind the end are zeros: a rank of 8 is a quarter of a step, and that step is the last CTA's fourth
    // at 512 x 768 x 768 (forward 39.0 -> 34.9 us, 1024 x 768 -> 768 59.5 -> 55.4)
    const int left = s < main_steps ? p.K - (s_begin + s) * kStep : p.R - (s - main_steps) * kStep;
    const int kn = left < kStep ? left : kStep;
#pragma unroll 2
    for (int k = 0; k < kn; ++k) {
      float a[16];
      float4 b[2];
#pragma unroll
      for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(a + 4 * i) = *reinterpret_cast<const float4*>(sa + k * kPitchA + 32 * i);
#pragma unroll
      for (int j = 0; j < 2; ++j) b[j] = *reinterpret_cast<const float4*>(sb + k * kPitchB + 32 * j);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float2 aa = make_float2(a[i], a[i]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          acc[i][2 * j] = __ffma2_rn(aa, make_float2(b[j].x, b[j].y), acc[i][2 * j]);
          acc[i][2 * j + 1] = __ffma2_rn(aa, make_float2(b[j].z, b[j].w), acc[i][2 * j + 1]);
        }
      }
    }
  }
  cp_wait<0>();
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 16; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
      *reinterpret_cast<float4*>(smem + (4 * ty + 32 * (i >> 2) + (i & 3)) * kOutPitch + 4 * tx + 32 * j) =
          make_float4(acc[i][2 * j].x, acc[i][2 * j].y, acc[i][2 * j + 1].x, acc[i][2 * j + 1].y);
  cg::cluster_group cl = cg::this_cluster();
  if (p.splits > 1) cl.sync();
  else __syncthreads();
  // each CTA of the cluster finishes its share of the tile's rows
  const int row_begin = kTileM * split / p.splits, row_end = kTileM * (split + 1) / p.splits;
  const bool vec_out = p.cn == 1 && p.cm % 4 == 0 && p.N % 4 == 0 && (reinterpret_cast<uintptr_t>(p.C) & 15u) == 0;
  for (int e = threadIdx.x; e < (row_end - row_begin) * (kTileN / 4); e += kTileThreads) {
    const int r = row_begin + e / (kTileN / 4), c = (e % (kTileN / 4)) * 4;
    const int gm = m0 + r, gn = n0 + c;
    if (gm >= p.M || gn >= p.N) continue;
    // all parts' loads in flight before the first sum: one after the other, a thread's 32 remote reads of 8 parts are 32
    // trips through the cluster's network (64 x 256 -> 128 r8: forward 22.6 -> 20.6 us, backward 28.8 -> 26.8)
    float4 part[kMaxSplits];
#pragma unroll
    for (int q = 0; q < kMaxSplits; ++q)
      if (q < p.splits)
        part[q] = *reinterpret_cast<const float4*>((p.splits > 1 ? cl.map_shared_rank(smem, q) : smem) + r * kOutPitch + c);
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int q = 0; q < kMaxSplits; ++q)
      if (q < p.splits) { v[0] += part[q].x; v[1] += part[q].y; v[2] += part[q].z; v[3] += part[q].w; }
    const int64_t o = gm * p.cm + gn * p.cn;
    const int live = min(4, p.N - gn);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      if (x >= live) break;
      v[x] *= p.alpha;
      if (p.bias != nullptr) v[x] += p.bias[gn + x];
      if (p.residual != nullptr) v[x] += p.residual[o + x * p.cn];
      if (p.accumulate) v[x] += p.C[o + x * p.cn];
    }
    if (vec_out) {
      *reinterpret_cast<float4*>(p.C + o) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int x = 0; x < 4; ++x)
        if (x < live) p.C[o + x * p.cn] = v[x];
    }
  }
  if (p.splits > 1) cl.sync();   // nobody leaves while a peer still reads its tile
}

// ---- rank intermediates ------------------------------------------------------------------------------------------
// out(m, j) = scale * sum_k x[m, k] F(k, j), F(k, j) = F[k * fk + j * fj]; out(m, j) at out[m * om + j * oj].
// Bound: latency (6 MFLOP at 512 x 768, r = 8).  A CTA takes 4 tokens and 8 rank columns; its 8 warps share the
// reduction (an eighth each, lanes over k, so that x is read coalesced and once per 8 columns) and meet in shared
// memory.  One 4-token CTA per 128 KFLOP keeps 128 CTAs busy at 512 tokens; the 64 x 64 tile kernel had 8.
constexpr int kRankTokens = 4, kRankCols = 8, kRankWarps = 8;
__global__ void __launch_bounds__(kRankWarps * 32)
rank_kernel(const float* __restrict__ x, const float* __restrict__ F, int64_t fk, int64_t fj, float* __restrict__ out, int64_t om,
            int64_t oj, int M, int K, int r, float scale) {
  __shared__ float red[kRankWarps][kRankTokens * kRankCols];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t m0 = static_cast<int64_t>(blockIdx.x) * kRankTokens;
  const int j0 = blockIdx.y * kRankCols;
  float acc[kRankTokens][kRankCols] = {};
  const bool vec_f = fj == 1 && (fk & 3) == 0 && j0 + kRankCols <= r && (reinterpret_cast<uintptr_t>(F) & 15u) == 0;
#pragma unroll 2
  for (int k = warp * 32 + lane; k < K; k += kRankWarps * 32) {
    float f[kRankCols], xv[kRankTokens];
#pragma unroll
    for (int t = 0; t < kRankTokens; ++t) xv[t] = m0 + t < M ? x[(m0 + t) * K + k] : 0.0f;
    if (vec_f) {
      const float4 a = *reinterpret_cast<const float4*>(F + k * fk + j0), b = *reinterpret_cast<const float4*>(F + k * fk + j0 + 4);
      f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    } else {
#pragma unroll
      for (int j = 0; j < kRankCols; ++j) f[j] = j0 + j < r ? F[k * fk + (j0 + j) * fj] : 0.0f;
    }
#pragma unroll
    for (int t = 0; t < kRankTokens; ++t)
#pragma unroll
      for (int j = 0; j < kRankCols; ++j) acc[t][j] = fmaf(xv[t], f[j], acc[t][j]);
  }
  // butterfly over the lanes that halves the values as it goes: lane l ends with the warp's sum of value l
  float v[32];
#pragma unroll
  for (int e = 0; e < 32; ++e) v[e] = acc[e / kRankCols][e % kRankCols];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool upper = (lane & o) != 0;
#pragma unroll
    for (int e = 0; e < o; ++e) {
      const float give = upper ? v[e] : v[e + o], keep = upper ? v[e + o] : v[e];
      v[e] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  red[warp][lane] = v[0];
  __syncthreads();
  if (warp == 0) {
    float s = 0.0f;
#pragma unroll
    for (int w = 0; w < kRankWarps; ++w) s += red[w][lane];
    const int t = lane / kRankCols, j = j0 + lane % kRankCols;
    if (m0 + t < M && j < r) out[(m0 + t) * om + j * oj] = s * scale;
  }
}

// ---- weight gradients --------------------------------------------------------------------------------------------
// out(c, j) (+)= sum_m X[m, c] H(m, j), H(m, j) = H[m * hm + j * hj]; out(c, j) at out[c * oc + j * oj].  Two problems
// (dA: X = x, H = scale dy B^T; dB: X = dy, H = scale x A) in one launch.
// Bound: reading X once from L2 / HBM (latency at small sizes).  A CTA takes 32 columns of X (lanes, coalesced) and 8
// rank columns; its 8 warps and the CTAs of its cluster share the tokens, so that even 768 columns make
// 24 x 8 CTAs; sums meet in shared and distributed shared memory in a fixed order (deterministic, no workspace).
struct GradProblemF32 {
  const float *X, *H;
  int64_t hm, hj, oc, oj;
  float* out;
  int C, blocks;   // columns; column blocks of 32
};
constexpr int kGradWarps = 8, kGradCols = 8;
__global__ void __launch_bounds__(kGradWarps * 32)
grad_kernel(const GradProblemF32 qa, const GradProblemF32 qb, int M, int r, int accumulate, int splits) {
  __shared__ float red[kGradWarps][kGradCols][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = blockIdx.x % splits;
  int cb = blockIdx.x / splits;
  const bool second = cb >= qa.blocks;
  const GradProblemF32& q = second ? qb : qa;
  if (second) cb -= qa.blocks;
  const int c = cb * 32 + lane, j0 = blockIdx.y * kGradCols;
  const int part = split * kGradWarps + warp, parts = splits * kGradWarps;
  float acc[kGradCols] = {};
#pragma unroll 4
  for (int m = part; m < M; m += parts) {
    const float xv = c < q.C ? q.X[static_cast<int64_t>(m) * q.C + c] : 0.0f;
#pragma unroll
    for (int j = 0; j < kGradCols; ++j)
      if (j0 + j < r) acc[j] = fmaf(xv, __ldg(q.H + m * q.hm + (j0 + j) * q.hj), acc[j]);
  }
#pragma unroll
  for (int j = 0; j < kGradCols; ++j) red[warp][j][lane] = acc[j];
  __syncthreads();
  // thread (j, lane) adds the warps' sums
  float s = 0.0f;
#pragma unroll
  for (int w = 0; w < kGradWarps; ++w) s += red[w][warp][lane];
  cg::cluster_group cl = cg::this_cluster();
  if (splits > 1) {
    __syncthreads();
    red[0][warp][lane] = s;
    cl.sync();
    s = 0.0f;
    if (split == 0)
      for (int p = 0; p < splits; ++p) s += cl.map_shared_rank(&red[0][0][0], p)[warp * 32 + lane];
  }
  if (split == 0 && c < q.C && j0 + warp < r) {
    float* o = q.out + c * q.oc + (j0 + warp) * q.oj;
    *o = accumulate ? *o + s : s;
  }
  if (splits > 1) cl.sync();
}
static_assert(kGradWarps == kGradCols, "a warp finishes one rank column");

// ---- the adapter delta of few tokens, in one launch ----------------------------------------------------------------
// out[m, n] = scale * sum_j (sum_k x[m,k] A[k,j]) B[j,n], everything in float32.
// Bound: latency, and reading A and B from L2 once per cluster.  A cluster of 8 CTAs takes TOK tokens: each CTA reduces
// an eighth of K for all ranks, the partial intermediates are added through distributed shared memory in rank order, and
// each CTA then writes an eighth of the columns.  One CTA alone would read all of A through a single SM; two launches
// would pay the launch gap twice.  1 x 512 -> 512, r = 8: 62 us of kernels before (two 64 x 64-tile GEMMs on one SM).
constexpr int kDeltaThreads = 256, kDeltaCtas = 8, kDeltaChunk = 256, kDeltaMaxRank = 64;

template <typename T, int TOK>
__global__ void __launch_bounds__(kDeltaThreads)
lora_delta_cluster_kernel(const T* __restrict__ x, const float* __restrict__ A, const float* __restrict__ B, T* __restrict__ out,
                          int M, int K, int N, int r, float scale) {
  __shared__ float xs[TOK][kDeltaChunk];
  __shared__ float part[kDeltaThreads][TOK];
  __shared__ float hp[TOK * kDeltaMaxRank], h[TOK * kDeltaMaxRank];
  cg::cluster_group cl = cg::this_cluster();
  const int rank = cl.block_rank(), t = threadIdx.x;
  const int m0 = (blockIdx.x / kDeltaCtas) * TOK;
  // phase 1: this CTA's eighth of the reduction; thread (g, j) takes every groups-th k of rank column j
  const int kper = (K + kDeltaCtas - 1) / kDeltaCtas;
  const int k_begin = min(K, rank * kper), k_end = min(K, k_begin + kper);
  const int groups = kDeltaThreads / r;
  const int j = t % r, g = t / r;
  float acc[TOK] = {};
  for (int kc = k_begin; kc < k_end; kc += kDeltaChunk) {
    const int len = min(kDeltaChunk, k_end - kc);
    __syncthreads();
    for (int e = t; e < TOK * len; e += kDeltaThreads) {
      const int i = e / len, k = e - i * len;
      xs[i][k] = m0 + i < M ? to_f32(x[static_cast<int64_t>(m0 + i) * K + kc + k]) : 0.0f;
    }
    __syncthreads();
    if (g < groups) {
#pragma unroll 4
      for (int k = g; k < len; k += groups) {
        const float a = __ldg(A + static_cast<int64_t>(kc + k) * r + j);
#pragma unroll
        for (int i = 0; i < TOK; ++i) acc[i] = fmaf(xs[i][k], a, acc[i]);
      }
    }
  }
  // sum over the groups: lanes of the same column first where a warp holds whole columns, then through shared memory
  int n_parts = groups;
  if (r <= 32 && (r & (r - 1)) == 0) {
    for (int o = r; o < 32; o <<= 1) {
#pragma unroll
      for (int i = 0; i < TOK; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
    }
    n_parts = kDeltaThreads / 32;
    if ((t & 31) < r) {
#pragma unroll
      for (int i = 0; i < TOK; ++i) part[(t >> 5) * r + j][i] = acc[i];
    }
  } else if (g < groups) {
#pragma unroll
    for (int i = 0; i < TOK; ++i) part[g * r + j][i] = acc[i];
  }
  __syncthreads();
  for (int e = t; e < TOK * r; e += kDeltaThreads) {
    const int jj = e % r, i = e / r;
    float s = 0.0f;
    for (int q = 0; q < n_parts; ++q) s += part[q * r + jj][i];
    hp[e] = s;
  }
  cl.sync();
  for (int e = t; e < TOK * r; e += kDeltaThreads) {
    float s = 0.0f;
#pragma unroll
    for (int q = 0; q < kDeltaCtas; ++q) s += cl.map_shared_rank(hp, q)[e];
    h[e] = s * scale;
  }
  __syncthreads();
  cl.barrier_arrive();   // this CTA has read its peers' sums
  // phase 2: an eighth of the output columns, one column per thread
  const int nper = (N + kDeltaCtas - 1) / kDeltaCtas;
  const int n_end = min(N, (rank + 1) * nper);
  for (int n = rank * nper + t; n < n_end; n += kDeltaThreads) {
    float o[TOK] = {};
#pragma unroll 8
    for (int jj = 0; jj < r; ++jj) {
      const float b = __ldg(B + static_cast<int64_t>(jj) * N + n);
#pragma unroll
      for (int i = 0; i < TOK; ++i) o[i] = fmaf(h[i * r + jj], b, o[i]);
    }
#pragma unroll
    for (int i = 0; i < TOK; ++i)
      if (m0 + i < M) out[static_cast<int64_t>(m0 + i) * N + n] = from_f32<T>(o[i]);
  }
  cl.barrier_wait();     // and the peers have read its own
}

cudaError_t launch_cluster(const void* kernel, dim3 grid, int threads, size_t smem, int cluster, cudaStream_t st, void** args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = dim3(static_cast<unsigned>(threads)); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(cluster); attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 1 : 0;
  return cudaLaunchKernelExC(&cfg, kernel, args);
}

template <typename T, int TOK>
int launch_delta(const LoraArgs& a) {
  const T* x = static_cast<const T*>(a.x);
  T* out = static_cast<T*>(a.y);
  int M = static_cast<int>(a.M), K = static_cast<int>(a.K), N = static_cast<int>(a.N), r = static_cast<int>(a.r);
  float scale = a.scale;
  const float *A = a.A, *B = a.B;
  void* args[] = {&x, &A, &B, &out, &M, &K, &N, &r, &scale};
  const unsigned clusters = static_cast<unsigned>((M + TOK - 1) / TOK);
  const cudaError_t e = launch_cluster(reinterpret_cast<const void*>(&lora_delta_cluster_kernel<T, TOK>), dim3(clusters * kDeltaCtas),
                                       kDeltaThreads, 0, kDeltaCtas, a.stream, args);
  if (e != cudaSuccess) return cuda_fail(e, "lora_delta_cluster_kernel launch");
  MCB_CHECK_LAUNCH("lora_delta_cluster_kernel");
  return MCB_OK;
}

// ---- host side ---------------------------------------------------------------------------------------------------
constexpr size_t kTileSmem = static_cast<size_t>(kStages) * kStageFloats * sizeof(float);

// CTAs that share a tile's reduction.  In cycles: a CTA-step of one reduction index is 64 cycles of an SM's FMA pipes, but
// a CTA has two warps and so reaches only half of them alone; the tiles x splits units are dealt out to the SMs in whole
// units; a partial tile's write and exchange costs 1000 per unit and 2000 for the cluster.
int pick_splits(int64_t tiles, int64_t K, int sm_count) {
  int best = 1;
  double best_cost = 0.0;
  for (int s = 1; s <= kMaxSplits; s *= 2) {
    if (s > 1 && K < static_cast<int64_t>(s) * 2 * kStep) break;
    const double n = static_cast<double>((tiles * s + sm_count - 1) / sm_count);
    const double cost = (n < 2.0 ? 2.0 : n) * 64.0 * static_cast<double>(K) / s + 1000.0 * n + (s > 1 ? 2000.0 : 0.0);
    if (s == 1 || cost < best_cost) { best = s; best_cost = cost; }
  }
  return best;
}

// C = alpha A B, row-major unless the caller changes cm / cn
TileParams product(const Operand& a, const Operand& b, float* C, int64_t M, int64_t N, int64_t K) {
  TileParams p = {};
  p.a = p.ra = a; p.b = p.rb = b;
  p.M = static_cast<int>(M); p.N = static_cast<int>(N); p.K = static_cast<int>(K);
  p.alpha = 1.0f;
  p.C = C; p.cm = N; p.cn = 1;
  return p;
}

int gemm(cudaStream_t st, TileParams p) {
  DeviceState* ds = current_device_state();
  if (!ds) return MCB_ERR_NOT_INIT;
  if (p.residual != nullptr && p.residual == p.C) return fail(MCB_ERR_UNSUPPORTED, "f32 path: residual must not alias the output");
  p.n_tiles = (p.N + kTileN - 1) / kTileN;
  const int64_t tiles = static_cast<int64_t>((p.M + kTileM - 1) / kTileM) * p.n_tiles;
  p.splits = pick_splits(tiles, p.K, ds->sm_count);
  if (tiles * p.splits > 0x7fffffffll) return fail(MCB_ERR_SHAPE, "f32 path: %d x %d outputs", p.M, p.N);
  if (!ds->f32_tile_smem) {
    MCB_CHECK_CUDA(cudaFuncSetAttribute(tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kTileSmem)));
    ds->f32_tile_smem = true;
  }
  void* args[] = {&p};
  const cudaError_t e = launch_cluster(reinterpret_cast<const void*>(&tile_kernel), dim3(static_cast<unsigned>(tiles * p.splits)),
                                       kTileThreads, kTileSmem, p.splits, st, args);
  if (e != cudaSuccess) return cuda_fail(e, "f32 tile_kernel launch");
  MCB_CHECK_LAUNCH("f32 tile_kernel");
  return MCB_OK;
}

// From here on a rank fills enough of a 64-wide tile that the tile kernel's reuse beats the lean kernels' short start.
constexpr int64_t kTileRank = 24;

int rank_product(cudaStream_t st, const float* x, const float* F, int64_t fk, int64_t fj, float* out, int64_t om, int64_t oj, int64_t M,
                 int64_t K, int64_t r, float scale) {
  if (r >= kTileRank) {
    TileParams p = product({x, K, 1}, {F, fj, fk}, out, M, r, K);
    p.cm = om; p.cn = oj; p.alpha = scale;
    return gemm(st, p);
  }
  const dim3 grid(static_cast<unsigned>((M + kRankTokens - 1) / kRankTokens), static_cast<unsigned>((r + kRankCols - 1) / kRankCols));
  rank_kernel<<<grid, kRankWarps * 32, 0, st>>>(x, F, fk, fj, out, om, oj, static_cast<int>(M), static_cast<int>(K), static_cast<int>(r), scale);
  MCB_CHECK_LAUNCH("f32 rank_kernel");
  return MCB_OK;
}

int check_sizes(const LoraArgs& a) {
  if (a.M > 0x7fffff00ll || a.N > 0x7fffff00ll || a.K > 0x7fffff00ll) return fail(MCB_ERR_SHAPE, "LoRA kernels: dimension exceeds 2^31");
  return MCB_OK;
}

}  // namespace

int matmul(const float* a, const float* b, float* out, int64_t M, int64_t K, int64_t N, cudaStream_t st) {
  if (M > 0x7fffff00ll || N > 0x7fffff00ll || K > 0x7fffff00ll) return fail(MCB_ERR_SHAPE, "f32 path: dimension exceeds 2^31");
  return gemm(st, product({a, K, 1}, {b, 1, N}, out, M, N, K));
}

size_t workspace_bytes(int64_t M, int64_t K, int64_t N, int64_t r) {
  (void)K; (void)N;
  return (static_cast<size_t>(M) + static_cast<size_t>(h_pitch(M))) * static_cast<size_t>(rank_padded(r)) * sizeof(float);
}

bool delta_small(int64_t M, int64_t r) { return M <= kDeltaMaxTokens && r <= kDeltaMaxRank; }

int delta_cluster(const LoraArgs& a, int dtype) {
  if (int rc = check_sizes(a)) return rc;
  // one token per cluster is the quicker form while a thread's share of A is a few words
  const bool one = a.M <= 18 && a.r * a.K <= 8192;
  if (dtype == MCB_F32) return one ? launch_delta<float, 1>(a) : launch_delta<float, 4>(a);
  return one ? launch_delta<__nv_bfloat16, 1>(a) : launch_delta<__nv_bfloat16, 4>(a);
}

int delta_fwd(const LoraArgs& a) {
  if (int rc = check_sizes(a)) return rc;
  const int64_t rp = rank_padded(a.r);
  if (a.ws_bytes < workspace_bytes(a.M, a.K, a.N, a.r) || !a.ws)
    return fail(MCB_ERR_WORKSPACE, "lora_delta_fwd(f32): workspace too small");
  if (delta_small(a.M, a.r)) return delta_cluster(a, MCB_F32);
  float* h = static_cast<float*>(a.ws);
  // h = scale * x A ; out = h B   (src/training/lora.rs:323,336,339)
  if (int rc = rank_product(a.stream, static_cast<const float*>(a.x), a.A, a.r, 1, h, rp, 1, a.M, a.K, a.r, a.scale)) return rc;
  return gemm(a.stream, product({h, rp, 1}, {a.B, 1, a.N}, static_cast<float*>(a.y), a.M, a.N, a.r));
}

int linear_fwd(const LoraArgs& a) {
  if (int rc = check_sizes(a)) return rc;
  const int64_t pitch = h_pitch(a.M);
  const float *x = static_cast<const float*>(a.x), *W = static_cast<const float*>(a.W);
  const Operand w = a.w_layout == MCB_W_OUT_IN ? Operand{W, a.K, 1} : Operand{W, 1, a.N};
  TileParams p = product({x, a.K, 1}, w, static_cast<float*>(a.y), a.M, a.N, a.K);
  p.bias = static_cast<const float*>(a.bias); p.residual = static_cast<const float*>(a.residual);
  if (a.r > 0) {
    // hs = scale * (x A), kept transposed [rp, pitch] like the bf16 path's saved intermediate
    float* hs = static_cast<float*>(a.h_save);
    if (hs == nullptr) {
      if (a.ws_bytes < workspace_bytes(a.M, a.K, a.N, a.r) || !a.ws)
        return fail(MCB_ERR_WORKSPACE, "lora_linear_fwd(f32): workspace too small");
      hs = static_cast<float*>(a.ws);
    }
    if (int rc = rank_product(a.stream, x, a.A, a.r, 1, hs, 1, pitch, a.M, a.K, a.r, a.scale)) return rc;
    p.ra = {hs, 1, pitch}; p.rb = {a.B, 1, a.N}; p.R = static_cast<int>(a.r);
  }
  return gemm(a.stream, p);
}

int linear_bwd(const LoraArgs& a) {
  if (int rc = check_sizes(a)) return rc;
  const int64_t rp = rank_padded(a.r);
  const int64_t pitch = h_pitch(a.M);
  const float *x = static_cast<const float*>(a.x), *dy = static_cast<const float*>(a.dy), *W = static_cast<const float*>(a.W);
  float* dh = nullptr;                                    // scale * dy B^T   [M, rp]
  if (a.r > 0) {
    if (a.ws_bytes < workspace_bytes(a.M, a.K, a.N, a.r) || !a.ws)
      return fail(MCB_ERR_WORKSPACE, "lora_linear_bwd(f32): workspace too small");
    dh = static_cast<float*>(a.ws);
    if (int rc = rank_product(a.stream, dy, a.B, 1, a.N, dh, rp, 1, a.M, a.N, a.r, a.scale)) return rc;
  }
  if (a.dx != nullptr) {
    const Operand w = a.w_layout == MCB_W_OUT_IN ? Operand{W, 1, a.K} : Operand{W, a.N, 1};
    TileParams p = product({dy, a.N, 1}, w, static_cast<float*>(a.dx), a.M, a.K, a.N);
    p.residual = static_cast<const float*>(a.residual);
    if (a.r > 0) { p.ra = {dh, rp, 1}; p.rb = {a.A, a.r, 1}; p.R = static_cast<int>(a.r); }
    if (int rc = gemm(a.stream, p)) return rc;
  }
  if (a.r == 0 || (a.dA == nullptr && a.dB == nullptr)) return MCB_OK;
  const float* hs = static_cast<const float*>(a.h_save);
  if (a.dB != nullptr && hs == nullptr) {
    float* hs_ws = dh + a.M * rp;                         // scale * x A      [rp, pitch] when not saved
    if (int rc = rank_product(a.stream, x, a.A, a.r, 1, hs_ws, 1, pitch, a.M, a.K, a.r, a.scale)) return rc;
    hs = hs_ws;
  }
  // dA[k, j] = sum_m x[m,k] dh[m,j];  dB[j, n] = sum_m hs[j,m] dy[m,n]
  if (a.r >= kTileRank) {
    if (a.dA != nullptr) {
      TileParams p = product({x, 1, a.K}, {dh, 1, rp}, a.dA, a.K, a.r, a.M);
      p.accumulate = a.accumulate;
      if (int rc = gemm(a.stream, p)) return rc;
    }
    if (a.dB != nullptr) {
      TileParams p = product({dy, 1, a.N}, {hs, pitch, 1}, a.dB, a.N, a.r, a.M);
      p.cm = 1; p.cn = a.N; p.accumulate = a.accumulate;
      if (int rc = gemm(a.stream, p)) return rc;
    }
    return MCB_OK;
  }
  const DeviceState* ds = current_device_state();
  if (!ds) return MCB_ERR_NOT_INIT;
  GradProblemF32 qa = {x, dh, rp, 1, a.r, 1, a.dA, static_cast<int>(a.K), a.dA ? static_cast<int>((a.K + 31) / 32) : 0};
  GradProblemF32 qb = {dy, hs, 1, pitch, 1, a.N, a.dB, static_cast<int>(a.N), a.dB ? static_cast<int>((a.N + 31) / 32) : 0};
  const int64_t jb = (a.r + kGradCols - 1) / kGradCols;
  const int64_t blocks = (qa.blocks + qb.blocks) * jb;
  // share the tokens out until there are four CTAs per SM (eight fit), as long as every warp keeps 8 tokens
  int splits = 1;
  while (splits < 8 && blocks * splits < 4ll * ds->sm_count && a.M >= 2ll * splits * kGradWarps * 8) splits *= 2;
  int M = static_cast<int>(a.M), r = static_cast<int>(a.r), acc = a.accumulate;
  void* args[] = {&qa, &qb, &M, &r, &acc, &splits};
  const cudaError_t e = launch_cluster(reinterpret_cast<const void*>(&grad_kernel),
                                       dim3(static_cast<unsigned>((qa.blocks + qb.blocks) * splits), static_cast<unsigned>(jb)),
                                       kGradWarps * 32, 0, splits, a.stream, args);
  if (e != cudaSuccess) return cuda_fail(e, "f32 grad_kernel launch");
  MCB_CHECK_LAUNCH("f32 grad_kernel");
  return MCB_OK;
}

}  // namespace f32path
}  // namespace mcb
