// float32 path of the fused LoRA linear.  tcgen05 has no float32 MMA and a single TF32 pass cannot hold the 1e-4 bound against
// the reference's f32 CPU arithmetic; eight bfloat16 products of operands taken apart into three parts each can, with a smaller error
// than a chain of float32 FMAs (tile_kernel).  The kinds of kernel:
//
//   tile_kernel    C = A B (+ bias) (+ residual) with the rank-r update as extra reduction steps, on the tensor cores: 128 x
//                  128 (64) tiles, the reduction split over the CTAs of a cluster when a shape has too few tiles for the chip
//   short_kernel   the same for reductions of at most 32, on the FMA pipes
//   rank_kernel    the [M, r] intermediates scale * x A and scale * dy B^T
//   grad_kernel    dA and dB, reductions over tokens
//   lora_delta_cluster_kernel   scale * (x A) B of few tokens in one launch (also for bfloat16 x)
#include <cooperative_groups.h>

#include "lora_internal.cuh"
#include "umma_ptx.cuh"

namespace cg = cooperative_groups;

namespace mcb {
namespace f32path {
using namespace umma;
namespace {

// ---- tile kernel -------------------------------------------------------------------------------------------------
// An operand as the kernel reads it: element (row, k) at p[row * sr + k * sk]; one of the strides is 1.
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
  int* status;
};

// The tensor cores take bfloat16, whose eight significant bits are a third of float32's: x = h + m + l, each part what is left
// of x rounded to nearest bfloat16.  A remainder is at most half a unit of the part before it, so the three hold all 24 bits,
// and it has either sign, so that nothing that is left out of a product adds up over many of them.  Both operands are scaled by 2^24
// first, so that the parts of the smallest normal numbers are normal themselves; what overflows for it (operands beyond 2^103,
// products beyond 2^79) is computed again, see redo_outputs.  Of the nine products of the parts l x l alone is left out: below 2^-33 of
// the product, where one float32 rounding is up to 2^-24.
constexpr int kTileM = 128, kStep = 64, kStages = 2, kParts = 3, kMaxSplits = 8;
constexpr int kSumWarps = 8, kCopyWarps = 7, kCopyThreads = 32 * kCopyWarps, kTileThreads = 32 * kSumWarps + kCopyThreads + 32;
constexpr float kPartScale = 16777216.0f, kPartUnscale = 1.0f / 16777216.0f / 16777216.0f;

template <int BN>
struct TileSmem {
  static constexpr uint32_t kPlaneA = kTileM * kStep * 2, kPlaneB = BN * kStep * 2;
  static constexpr uint32_t kStage = kParts * (kPlaneA + kPlaneB), kBars = kStages * kStage;
  static constexpr size_t kBytes = kBars + 128 + 1024;
  static constexpr int kOutPitch = BN + 4;   // the output tile reuses the stages; rows four banks apart
  static_assert((kTileM * kOutPitch + kTileM * 36 + 32 * (BN + 4)) * 4 <= kBars, "output tile, and what redo_outputs stages behind it");
  static_assert(kTileM * (BN / 4) <= 8 * kTileThreads, "32 bits say which of a thread's outputs are spoilt");
};

// two values rounded to bfloat16 (the first in the lower half), and what the rounding left of them
__device__ __forceinline__ uint32_t take_part(float2& x) {
  const __nv_bfloat162 r = __float22bfloat162_rn(x);
  const uint32_t w = *reinterpret_cast<const uint32_t*>(&r);
  x = __ffma2_rn(make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)), make_float2(-1.0f, -1.0f), x);
  return w;
}
// the three parts of four values, 8 bytes each, `plane` bytes apart
__device__ __forceinline__ void store_parts(uint8_t* dst, uint32_t plane, const float4& v) {
  const float2 scale = make_float2(kPartScale, kPartScale);
  float2 x = __fmul2_rn(make_float2(v.x, v.y), scale), y = __fmul2_rn(make_float2(v.z, v.w), scale);
#pragma unroll
  for (int s = 0; s < kParts; ++s) {
    const uint32_t lo = take_part(x), hi = take_part(y);
    *reinterpret_cast<uint2*>(dst + s * plane) = make_uint2(lo, hi);
  }
}

__device__ __forceinline__ bool is_k_major(const Operand& o) { return o.sk == 1; }
__device__ __forceinline__ bool is_vec(const Operand& o) {
  return (reinterpret_cast<uintptr_t>(o.p) & 15u) == 0 && ((o.sk == 1 ? o.sr : o.sk) & 3) == 0;
}

// One step's tile of an operand, ROWS x 64 reduction indices, as ROWS * 16 pieces of four neighbouring values dealt out to THREADS
// threads.  In shared memory, per part: k contiguous: rows of 128 bytes (64 k); rows contiguous: blocks of 64 rows, each
// 64 k of 128 bytes; the 16-byte groups of a line in 128-byte swizzle order either way.  Half a warp reads 256 neighbouring bytes and
// writes a line.
template <int ROWS, int THREADS>
struct Copy {
  static constexpr int kTotal = ROWS * 16, kPieces = (kTotal + THREADS - 1) / THREADS;
  static constexpr int kHop = THREADS / 16, kHopAcross = THREADS / (ROWS / 4);   // lines from a thread's piece to its next
  static_assert(THREADS % 16 == 0 && THREADS % (ROWS / 4) == 0, "a thread keeps its place in the line");
  float4 v[kPieces];
  // line (row, or index k if the rows are contiguous) of piece i of thread t, and its place in it, in values
  __device__ __forceinline__ static int line_of(bool k_major, int t, int i) { return k_major ? (t >> 4) + i * kHop : t / (ROWS / 4) + i * kHopAcross; }
  __device__ __forceinline__ static int at_of(bool k_major, int t) { return (k_major ? t & 15 : t % (ROWS / 4)) * 4; }
  __device__ __forceinline__ static bool has(int t, int i) { return (i + 1) * THREADS <= kTotal || t + i * THREADS < kTotal; }
  // rows [row0, row0 + ROWS) and indices [k0, k0 + 64); zeros beyond `rows` and `kend`
  __device__ __forceinline__ void load(const Operand& o, int t, int row0, int rows, int k0, int kend) {
    const bool k_major = is_k_major(o);
    const int64_t pitch = k_major ? o.sr : o.sk;
    const int line0 = k_major ? row0 : k0, lines = k_major ? rows : kend, at = (k_major ? k0 : row0) + at_of(k_major, t), end = k_major ? kend : rows;
    const float* q = from_here(o.p) + (line0 + line_of(k_major, t, 0)) * pitch + at;
    const int64_t hop = (k_major ? kHop : kHopAcross) * pitch;
    if (is_vec(o) && row0 + ROWS <= rows && k0 + kStep <= kend) {
#pragma unroll
      for (int i = 0; i < kPieces; ++i, q += hop)
        if (has(t, i)) v[i] = __ldg(reinterpret_cast<const float4*>(q));
    } else {
#pragma unroll
      for (int i = 0; i < kPieces; ++i, q += hop) {
        const int left = has(t, i) && line0 + line_of(k_major, t, i) < lines ? end - at : 0;
        v[i].x = left > 0 ? __ldg(q) : 0.0f;
        v[i].y = left > 1 ? __ldg(q + 1) : 0.0f;
        v[i].z = left > 2 ? __ldg(q + 2) : 0.0f;
        v[i].w = left > 3 ? __ldg(q + 3) : 0.0f;
      }
    }
  }
  // the parts of the indices below kn (nobody reads beyond the step's last 16); a whole step without a branch, so that the pieces'
  // dependent instructions run side by side (2048 x 1536 x 1536 111 -> 102 us)
  template <bool K_MAJOR, bool WHOLE>
  __device__ __forceinline__ void store_as(uint8_t* dst, uint32_t plane, int t, int kn) const {
    const int at = at_of(K_MAJOR, t), group = (at & 63) >> 3;
    dst += (K_MAJOR ? 0 : (at >> 6) * (kStep * 128)) + (at & 4) * 2;
#pragma unroll
    for (int i = 0; i < kPieces; ++i) {
      const int line = line_of(K_MAJOR, t, i);
      if (has(t, i) && (WHOLE || (K_MAJOR ? at : line) < kn)) store_parts(dst + line * 128 + ((group ^ (line & 7)) << 4), plane, v[i]);
    }
  }
  __device__ __forceinline__ void store(uint8_t* dst, uint32_t plane, bool k_major, int t, int kn) const {
    if (kn == kStep) {
      if (k_major) store_as<true, true>(dst, plane, t, kn);
      else store_as<false, true>(dst, plane, t, kn);
    } else {
      if (k_major) store_as<true, false>(dst, plane, t, kn);
      else store_as<false, false>(dst, plane, t, kn);
    }
  }
};

// What a CTA has to do to an output besides the sum.
__device__ __forceinline__ float finish_output(const TileParams& p, float v, int gn, int64_t at) {
  v *= p.alpha;
  if (p.bias != nullptr) v += p.bias[gn];
  if (p.residual != nullptr) v += p.residual[at];
  if (p.accumulate) v += p.C[at];
  return v;
}

// The outputs of `bad` (bit 4 i + x: column x of the four that the thread has of its i-th row) in plain float32 arithmetic, a chain of FMAs
// over K and R.  An operand that is infinite, or becomes so by the scaling, has no parts (inf - inf), so an output that is not finite
// may be one the parts have spoilt: it is computed again, and is then what float32 gives.  Rare, or a run that has diverged, which should
// not take a hundred times as long either: the CTA goes over the reduction together, 32 indices at a time.  us, a serial sum
// by the thread that has the output / this (all clean): 512 x 768 x 768 all NaN 1703 / 101 (21), a row with an infinity 253 / 73;
// 2048 x 1536 x 1536 20313 / 643 (113), 522 / 161; 4096^3 249700 / 5450 (1075), 1737 / 1175.  (FMA tiles took 33, 259 and 2834 for any values.)
template <int BN>
struct Redo {
  static constexpr int kTerms = 32, kPitchA = kTerms + 4, kPitchB = BN + 4;
  static constexpr int kHop = kTileThreads / (BN / 4), kRows = kTileM / kHop;   // rows from one of a thread's to the next, and how many it has
  static constexpr int kFloats = kTileM * kPitchA + kTerms * kPitchB;
};
// 32 indices of an operand's ROWS rows, a word a thread at a time, neighbours next to each other
template <int ROWS>
struct RedoCopy {
  static constexpr int kWords = ROWS * 32 / kTileThreads;
  float v[kWords];
  __device__ __forceinline__ void load(const Operand& o, int row0, int first, int last, int rows, int k0, int kend) {
#pragma unroll
    for (int j = 0; j < kWords; ++j) {
      const int e = threadIdx.x + j * kTileThreads, r = is_k_major(o) ? e >> 5 : e % ROWS, k = k0 + (is_k_major(o) ? e & 31 : e / ROWS);
      v[j] = r >= first && r < last && row0 + r < rows && k < kend ? o.p[(row0 + r) * o.sr + k * o.sk] : 0.0f;
    }
  }
  // element (row, k) to dst[row * sr + k * sk]
  __device__ __forceinline__ void store(float* dst, int sr, int sk, bool k_major) const {
#pragma unroll
    for (int j = 0; j < kWords; ++j) {
      const int e = threadIdx.x + j * kTileThreads;
      dst[(k_major ? e >> 5 : e % ROWS) * sr + (k_major ? e & 31 : e / ROWS) * sk] = v[j];
    }
  }
};
// NR: of how many of its rows a thread has outputs
template <int BN, int NR>
__device__ __noinline__ void redo_rows(const TileParams& p, float* sa, int m0, int n0, int row_begin, int row_end, uint32_t bad) {
  using D = Redo<BN>;
  float* sb = sa + kTileM * D::kPitchA;
  const int c = (threadIdx.x % (BN / 4)) * 4, r0 = row_begin + threadIdx.x / (BN / 4);
  const bool any = __any_sync(0xffffffffu, bad != 0);
  float2 acc[NR][2] = {};
  RedoCopy<kTileM> ca;
  RedoCopy<BN> cb;
  auto add = [&](const Operand& a, const Operand& b, int len) {
    auto load = [&](int k0) {
      ca.load(a, m0, row_begin, row_end, p.M, k0, len);
      cb.load(b, n0, 0, BN, p.N, k0, len);
    };
    if (len > 0) load(0);
    for (int k0 = 0; k0 < len; k0 += D::kTerms) {
      __syncthreads();   // the terms before have been read
      ca.store(sa, D::kPitchA, 1, is_k_major(a));
      cb.store(sb, 1, D::kPitchB, is_k_major(b));
      __syncthreads();
      if (k0 + D::kTerms < len) load(k0 + D::kTerms);
      if (!any) continue;
#pragma unroll 2
      for (int k = 0; k < D::kTerms; k += 4) {   // behind the end both are zeros
        float4 x[NR], y[4];
#pragma unroll
        for (int i = 0; i < NR; ++i) x[i] = *reinterpret_cast<const float4*>(sa + min(r0 + i * D::kHop, kTileM - 1) * D::kPitchA + k);
#pragma unroll
        for (int t = 0; t < 4; ++t) y[t] = *reinterpret_cast<const float4*>(sb + (k + t) * D::kPitchB + c);
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
          for (int i = 0; i < NR; ++i) {
            const float v = t == 0 ? x[i].x : t == 1 ? x[i].y : t == 2 ? x[i].z : x[i].w;
            acc[i][0] = __ffma2_rn(make_float2(v, v), make_float2(y[t].x, y[t].y), acc[i][0]);
            acc[i][1] = __ffma2_rn(make_float2(v, v), make_float2(y[t].z, y[t].w), acc[i][1]);
          }
      }
    }
  };
  add(p.a, p.b, p.K);
  add(p.ra, p.rb, p.R);
#pragma unroll
  for (int i = 0; i < NR; ++i)
#pragma unroll
    for (int x = 0; x < 4; ++x)
      if (bad >> (4 * i + x) & 1u) {
        const int gm = m0 + r0 + i * D::kHop, gn = n0 + c + x;
        const int64_t at = gm * p.cm + gn * p.cn;
        p.C[at] = finish_output(p, x == 0 ? acc[i][0].x : x == 1 ? acc[i][0].y : x == 2 ? acc[i][1].x : acc[i][1].y, gn, at);
      }
}
template <int BN>
__device__ __forceinline__ void redo_outputs(const TileParams& p, float* stage, int m0, int n0, int row_begin, int row_end, uint32_t bad) {
  const int nr = (row_end - row_begin + Redo<BN>::kHop - 1) / Redo<BN>::kHop;
  if (nr <= 1) redo_rows<BN, 1>(p, stage, m0, n0, row_begin, row_end, bad);
  else if (nr <= 2) redo_rows<BN, 2>(p, stage, m0, n0, row_begin, row_end, bad);
  else if (nr <= 4) redo_rows<BN, 4>(p, stage, m0, n0, row_begin, row_end, bad);
  else redo_rows<BN, 8>(p, stage, m0, n0, row_begin, row_end, bad);
}

// A step of 64 reduction indices: seven warps take the values they loaded a step earlier apart (two stages of shared memory), one issues
// the products, and eight add the step before's accumulators to float32 sums in registers (having taken their half of the first step).
// The tensor core adds an MMA's 16 products and its accumulator exactly down to 2^-25 of the largest of them and cuts the rest off, always
// towards zero, where float32 rounds to nearest: terms of one sign lose half a unit of the sum with every MMA that adds to it.
// So the h x h products, which make the sum, get an accumulator for every 16 indices (16 products of eight bits by eight fit the 24 bits
// of a sum but for their smallest terms); the seven small ones, whose cut-off is 2^-8 of that, share one.
// Relative error to float64, in brackets that of float32 FMAs split likewise and of six products of cut parts in one accumulator per step:
//   512 x 768 x 768      normal 7.3e-8 (1.9e-7, 1.3e-7)   uniform(0, 1) 4.8e-8 (7.0e-8, 1.2e-7)   uniform(1, 2) 4.1e-8 (6.7e-8, 9.7e-8)
//   300 x 65 x 200              5.5e-8 (1.4e-7, 1.2e-7)                 5.1e-8 (1.2e-7, 1.2e-7)                 4.6e-8 (1.2e-7, 9.8e-8)
//   2048 x 1536 x 1536          8.8e-8 (2.5e-7, 1.4e-7)                 5.3e-8 (8.7e-8, 1.2e-7)                 4.7e-8 (8.3e-8, 9.9e-8)
// and the mean deviation of positive terms is -1e-8 to -2e-8 (0, -1e-7).  Larger than the FMAs' where one term of a short sum dwarfs the
// others, whose last bits it pushes out: exp(2 normal), 65 indices 1.8e-7 (1.0e-7, 7.4e-7), 768 indices 1.4e-7 (1.5e-7, 4.8e-7).
// Bound: taking the values apart (about 4800 cycles a step of seven warps; the products are 16 BN), then a CTA's start and the exchange of
// partial tiles.  us, FMAs / six products / this: 512 x 768 x 768 28.8 / 14.3 / 14.7, 2048 x 1536 x 1536 253 / 105 / 99, 256 x 1536 x 128
// 28.8 / 14.3 / 14.4, 1200 x 200 x 1100 34.1 / 17.1 / 17.5, 1000^3 70.3 / 32.3 / 31.1, 300 x 1001 x 130 22.7 / 13.6 / 13.6.
// (All 16 warps at everything, a barrier a half step: 18.5 and 151 for the first two; one warp issuing beside its other work: 16.9 and 133.)
// A shape with few tiles (512 x 768 x 768: 24) leaves SMs idle, so up to 8 CTAs of a cluster share a tile's reduction and add their
// partial tiles through distributed shared memory, in rank order: deterministic, no workspace.
template <int BN>
__global__ void __launch_bounds__(kTileThreads, 1) tile_kernel(const __grid_constant__ TileParams p) {
  using S = TileSmem<BN>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // (known to be the warp's, not a lane's)
  const uint32_t stage_free0 = base + S::kBars, parts_ready0 = stage_free0 + 8 * kStages, high_full = parts_ready0 + 8 * kStages, high_read = high_full + 8;
  const uint32_t all_full = high_read + 8, low_read = all_full + 8, first_ready = low_read + 8, tmem_slot = first_ready + 8;
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(gen + (tmem_slot - base));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + (tmem_slot + 4 - base));

  if (threadIdx.x == 0) {
    // a barrier per stage where one side can be a stage ahead of the other: a wait tells a phase from the next one only
    for (int a = 0; a < kStages; ++a) {
      mbar_init(stage_free0 + 8 * a, 1);
      mbar_init(parts_ready0 + 8 * a, kCopyWarps);
    }
    mbar_init(high_full, 1);
    mbar_init(all_full, 1);
    mbar_init(high_read, kSumWarps);
    mbar_init(low_read, kSumWarps);
    mbar_init(first_ready, kSumWarps);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async_smem();
  }
  constexpr uint32_t kCols = 4 * BN;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(kCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  grid_launch_dependents();
  grid_dependency_wait();   // the set-up above ran under the tail of the kernel before
  const int split = blockIdx.x % p.splits, tile = blockIdx.x / p.splits;
  const int m0 = (tile / p.n_tiles) * kTileM, n0 = (tile % p.n_tiles) * BN;
  // main steps are shared out evenly; the rank steps go to the first CTA of the cluster, which has the fewest
  const int ksteps = (p.K + kStep - 1) / kStep;
  const int s_begin = static_cast<int>(static_cast<int64_t>(ksteps) * split / p.splits);
  const int s_end = static_cast<int>(static_cast<int64_t>(ksteps) * (split + 1) / p.splits);
  const int main_steps = s_end - s_begin;
  const int steps = main_steps + (split == 0 ? (p.R + kStep - 1) / kStep : 0);

  // Four accumulators take turns: step s has number s % 4 for all small products, the next three for the h x h products of its second to
  // last 16 indices; the first 16 go to the last of the three where it is free (a short step, as of a rank), else to the small products.
  // The three are filled between the small products' halves: they are read under the second half, the first accumulator under the next
  // step's first half, and either is free when its turn comes without the tensor pipe having waited.
  auto indices = [&](int s) { return min(kStep, s < main_steps ? p.K - (s_begin + s) * kStep : p.R - (s - main_steps) * kStep); };
  auto wait = [&](uint32_t bar, int n, int code) { return __all_sync(0xffffffffu, mbar_wait(bar, n & 1, abort_flag, code, p.status)) != 0; };
  if (warp >= kSumWarps && warp < kSumWarps + kCopyWarps) {
    // ---------------- copy ----------------
    // (tb: what is left over of either operand goes to another warp)
    const int t = threadIdx.x - 32 * kSumWarps, tb = t >= 96 ? t - 96 : t + kCopyThreads - 96;
    Copy<kTileM, kCopyThreads> ca;
    Copy<BN, kCopyThreads> cb;
    auto load_a = [&](int s) {
      const bool main = s < main_steps;
      ca.load(main ? p.a : p.ra, t, m0, p.M, (main ? s_begin + s : s - main_steps) * kStep, main ? p.K : p.R);
    };
    auto load_b = [&](int s) {
      const bool main = s < main_steps;
      cb.load(main ? p.b : p.rb, tb, n0, p.N, (main ? s_begin + s : s - main_steps) * kStep, main ? p.K : p.R);
    };
    load_a(0);
    if (steps > 1) load_b(1);   // step 0's is the sum warps', which have nothing to add yet
    for (int s = 0; s < steps; ++s) {
      const bool main = s < main_steps;
      const int kn = (indices(s) + 15) & ~15;   // the MMAs' reduction is 16 long
      uint8_t* dst = gen + (s & 1) * S::kStage;
      if (s >= kStages && !wait(stage_free0 + 8 * (s & 1), (s >> 1) - 1, 100)) break;
      ca.store(dst, S::kPlaneA, is_k_major(main ? p.a : p.ra), t, kn);
      if (s > 0) cb.store(dst + kParts * S::kPlaneA, S::kPlaneB, is_k_major(main ? p.b : p.rb), tb, kn);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(parts_ready0 + 8 * (s & 1));
      if (s + 1 < steps) {
        load_a(s + 1);
        if (s > 0) load_b(s + 1);
      }
    }
  } else if (warp >= kSumWarps) {
    // ---------------- MMA issuer ----------------
    // Smallest products first, so that what the running sum loses to them is small.
    for (int s = 0; s < steps; ++s) {
      constexpr int kA[7] = {2, 1, 2, 0, 1, 1, 0}, kB[7] = {1, 2, 0, 2, 1, 0, 1};
      const bool main = s < main_steps, ak = is_k_major(main ? p.a : p.ra), bk = is_k_major(main ? p.b : p.rb);
      const uint32_t idesc = make_idesc(BN) | (ak ? 0u : 1u << 15) | (bk ? 0u : 1u << 16);
      const uint32_t pa = base + (s & 1) * S::kStage, pb = pa + kParts * S::kPlaneA, acc = tmem_base + (s & 3) * BN;
      // 16 reduction indices further: 32 bytes along a line, or two groups of eight lines
      const uint64_t da0 = ak ? desc_sw128(pa) : desc_sw128_mn(pa, kStep * 128, 1024);
      const uint64_t db0 = bk ? desc_sw128(pb) : desc_sw128_mn(pb, kStep * 128, 1024);
      const uint32_t ja = ak ? 32 : 2048, jb = bk ? 32 : 2048;
      const int k16 = (indices(s) + 15) >> 4;   // the MMAs' reduction is 16 long
      auto product = [&](uint32_t d, int qa, int qb, int k, uint32_t add) {
        umma_bf16(d, desc_advance(da0, qa * S::kPlaneA + k * ja), desc_advance(db0, qb * S::kPlaneB + k * jb), idesc, add);
      };
      if (!wait(parts_ready0 + 8 * (s & 1), s >> 1, 101) || !(s > 0 ? wait(high_read, s - 1, 102) : wait(first_ready, 0, 102))) break;
      tcgen05_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (k >= k16) break;
#pragma unroll
          for (int q = 0; q < 4; ++q) product(acc, kA[q], kB[q], k, q + k > 0);
        }
      }
      __syncwarp();
      if (s > 0 && !wait(low_read, s - 1, 103)) break;
      tcgen05_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int k = 1; k < 4; ++k)
          if (k < k16) product(tmem_base + ((s + k) & 3) * BN, 0, 0, k, 0);
        if (k16 < 4) product(tmem_base + ((s + 3) & 3) * BN, 0, 0, 0, 0);
        umma_commit(high_full);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (k >= k16) break;
#pragma unroll
          for (int q = 4; q < 7; ++q) product(acc, kA[q], kB[q], k, 1);
        }
        if (k16 == 4) product(acc, 0, 0, 0, 1);
        umma_commit(all_full);
        umma_commit(stage_free0 + 8 * (s & 1));
      }
      __syncwarp();
    }
  }
  // the sums: row 32 (warp % 4) + lane, BN / 2 columns from (warp / 4) BN / 2 on
  const int quad = warp & 3, col0 = (warp >> 2) * (BN / 2);
  if (warp < kSumWarps) {
    const uint32_t own = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + col0;
    {
      Copy<BN, 32 * kSumWarps> first;
      first.load(p.b, threadIdx.x, n0, p.N, s_begin * kStep, p.K);
      first.store(gen + kParts * S::kPlaneA, S::kPlaneB, is_k_major(p.b), threadIdx.x, (indices(0) + 15) & ~15);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(first_ready);
    }
    float sum[BN / 2];
#pragma unroll
    for (int i = 0; i < BN / 2; ++i) sum[i] = 0.0f;
    auto arrive = [&](uint32_t bar) {
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    for (int s = 0; s < steps; ++s) {
      const int k16 = (indices(s) + 15) >> 4;
      if (!wait(high_full, s, 104)) break;
      tcgen05_fence_after();
#pragma unroll
      for (int c = 0; c < BN / 2; c += 16) {
        uint32_t x[16], y[16], z[16];
        tmem_ld_x16(own + ((s + 3) & 3) * BN + c, z);
        if (k16 > 1) tmem_ld_x16(own + ((s + 1) & 3) * BN + c, x);
        if (k16 > 2) tmem_ld_x16(own + ((s + 2) & 3) * BN + c, y);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          float2 t = make_float2(__uint_as_float(z[i]), __uint_as_float(z[i + 1]));
          if (k16 > 1) t = __fadd2_rn(t, make_float2(__uint_as_float(x[i]), __uint_as_float(x[i + 1])));
          if (k16 > 2) t = __fadd2_rn(t, make_float2(__uint_as_float(y[i]), __uint_as_float(y[i + 1])));
          t = __fadd2_rn(t, make_float2(sum[c + i], sum[c + i + 1]));
          sum[c + i] = t.x;
          sum[c + i + 1] = t.y;
        }
      }
      arrive(high_read);
      if (!wait(all_full, s, 105)) break;
      tcgen05_fence_after();
#pragma unroll
      for (int c = 0; c < BN / 2; c += 32) {
        uint32_t x[32];
        tmem_ld_x16(own + (s & 3) * BN + c, *reinterpret_cast<uint32_t(*)[16]>(&x[0]));
        tmem_ld_x16(own + (s & 3) * BN + c + 16, *reinterpret_cast<uint32_t(*)[16]>(&x[16]));
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) sum[c + i] += __uint_as_float(x[i]);
      }
      arrive(low_read);
    }
    // every product has been waited for: nothing reads the stages any more
    float* out = reinterpret_cast<float*>(gen) + (quad * 32 + lane) * S::kOutPitch + col0;
#pragma unroll
    for (int i = 0; i < BN / 2; i += 4) *reinterpret_cast<float4*>(out + i) = make_float4(sum[i], sum[i + 1], sum[i + 2], sum[i + 3]);
  }
  __syncwarp();
  if (*abort_flag != 0) {
    for (int k = 0; k < 200; ++k) __nanosleep(1000);
  }
  tcgen05_fence_before();
  cg::cluster_group cl = cg::this_cluster();
  if (p.splits > 1) cl.sync();
  else __syncthreads();
  if (warp == 0) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kCols) : "memory");
  }
  // each CTA of the cluster finishes its share of the tile's rows
  float* tile_out = reinterpret_cast<float*>(gen);
  const int row_begin = kTileM * split / p.splits, row_end = kTileM * (split + 1) / p.splits;
  const bool vec_out = p.cn == 1 && p.cm % 4 == 0 && p.N % 4 == 0 && (reinterpret_cast<uintptr_t>(p.C) & 15u) == 0;
  uint32_t bad = 0;   // see redo_outputs
#pragma unroll 2
  for (int i = 0; i < Redo<BN>::kRows; ++i) {
    const int r = row_begin + threadIdx.x / (BN / 4) + i * Redo<BN>::kHop, c = (threadIdx.x % (BN / 4)) * 4;
    const int gm = m0 + r, gn = n0 + c;
    if (r >= row_end || gm >= p.M) break;
    if (gn >= p.N) continue;
    // all parts' loads in flight before the first sum: one after the other, a thread's remote reads are as many trips
    // through the cluster's network
    float4 part[kMaxSplits];
#pragma unroll
    for (int q = 0; q < kMaxSplits; ++q)
      if (q < p.splits)
        part[q] = *reinterpret_cast<const float4*>((p.splits > 1 ? cl.map_shared_rank(tile_out, q) : tile_out) + r * S::kOutPitch + c);
    // the rank update, which can be most of the output, comes with the first part: added last, it is rounded once
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int q = 1; q <= kMaxSplits; ++q)
      if (q < p.splits || q == kMaxSplits) {
        const float4 t = part[q % kMaxSplits];
        v[0] += t.x; v[1] += t.y; v[2] += t.z; v[3] += t.w;
      }
    const int64_t o = gm * p.cm + gn * p.cn;
    const int live = min(4, p.N - gn);
    // (no branch: with one around each output's arithmetic 4096 x 64 x 4096 took 74.7 us instead of 65.9)
    uint32_t spoilt = 0;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      if (x >= live) break;
      spoilt |= fabsf(v[x]) < INFINITY ? 0u : 1u << x;
      v[x] = finish_output(p, v[x] * kPartUnscale, gn + x, o + x * p.cn);
    }
    bad |= spoilt << (4 * i);
    // what is computed again may be stored here first, unless C is one of its terms
    if (vec_out && (spoilt == 0 || !p.accumulate)) {
      *reinterpret_cast<float4*>(p.C + o) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int x = 0; x < 4; ++x)
        if (x < live && (spoilt >> x & 1u) == 0) p.C[o + x * p.cn] = v[x];
    }
  }
  if (__syncthreads_or(bad != 0)) redo_outputs<BN>(p, tile_out + kTileM * S::kOutPitch, m0, n0, row_begin, row_end, bad);
  if (p.splits > 1) cl.sync();   // nobody leaves while a peer still reads its tile
}

// ---- short reductions ----------------------------------------------------------------------------------------------
// The same product where K and R are at most 32, with float32 FMAs: there is no reduction to speed up, and taking a step's values
// apart costs more than multiplying them.  Bound: writing C, 16 bytes a thread and row, 256 next to each other.  A CTA holds both
// operands' 64 rows whole; a thread owns 8 x 4 outputs.  us, copies of 64-wide FMA tiles / single words stored and staged in 32 / this:
// 4096 x 8 x 4096 41.0 / 50.8 / 25.5, 4096 x 16 x 4096 45.1 / 56.4 / 35.5, 4096 x 32 x 4096 53.4 / 70.5 / 54.3, 8192 x 16 x 896 26.7 / 31.1 / 17.2,
// delta of 4096 tokens 4096 -> 4096 r8 74.9 / 84.7 / 59.4.  Beyond 32 tile_kernel, which errs less (64 terms 4.9e-8 against 1.4e-7):
// 4096 x 40 x 4096 62.8 / 78.0 / 69.1, 2048 x 40 x 2048 21.5 / 27.5 / 20.1, 4096 x 64 x 4096 75.8 / 112 / 65.6.
constexpr int kShort = 32, kShortRows = 64, kShortThreads = 128, kShortPitch = kShortRows + 4;
__global__ void __launch_bounds__(kShortThreads) short_kernel(const __grid_constant__ TileParams p) {
  __shared__ __align__(16) float sa[kShort][kShortPitch], sb[kShort][kShortPitch];   // [k][row]
  const int m0 = (blockIdx.x / p.n_tiles) * kShortRows, n0 = (blockIdx.x % p.n_tiles) * kShortRows;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;   // rows 8 ty.., columns 4 tx..
  grid_launch_dependents();
  grid_dependency_wait();
  float2 sum[8][2] = {};
  auto stage = [&](float (&dst)[kShort][kShortPitch], const Operand& o, int row0, int rows, int len) {
    const float* src = from_here(o.p);
    if (is_k_major(o)) {
      for (int e = threadIdx.x; e < len * kShortRows; e += kShortThreads) {   // neighbouring threads, neighbouring words
        const int r = e / len, k = e - r * len;
        dst[k][r] = row0 + r < rows ? src[(row0 + r) * o.sr + k] : 0.0f;
      }
    } else {
      for (int e = threadIdx.x; e < len * kShortRows; e += kShortThreads) {
        const int k = e / kShortRows, r = e % kShortRows;
        dst[k][r] = row0 + r < rows ? src[row0 + r + k * o.sk] : 0.0f;
      }
    }
  };
  auto run = [&](const Operand& a, const Operand& b, int len) {
    stage(sa, a, m0, p.M, len);
    stage(sb, b, n0, p.N, len);
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < len; ++k) {
      const float4 a0 = *reinterpret_cast<const float4*>(&sa[k][8 * ty]), a1 = *reinterpret_cast<const float4*>(&sa[k][8 * ty + 4]);
      const float4 b0 = *reinterpret_cast<const float4*>(&sb[k][4 * tx]);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        sum[i][0] = __ffma2_rn(make_float2(av[i], av[i]), make_float2(b0.x, b0.y), sum[i][0]);
        sum[i][1] = __ffma2_rn(make_float2(av[i], av[i]), make_float2(b0.z, b0.w), sum[i][1]);
      }
    }
  };
  run(p.a, p.b, p.K);
  if (p.R > 0) {
    __syncthreads();
    run(p.ra, p.rb, p.R);
  }
  const bool vec = p.cn == 1 && p.cm % 4 == 0 && p.N % 4 == 0 && (reinterpret_cast<uintptr_t>(p.C) & 15u) == 0;
  const int gn0 = n0 + 4 * tx;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int gm = m0 + 8 * ty + i;
    if (gm >= p.M || gn0 >= p.N) continue;
    const int64_t o = gm * p.cm + gn0 * p.cn;
    float v[4] = {sum[i][0].x, sum[i][0].y, sum[i][1].x, sum[i][1].y};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (gn0 + j >= p.N) break;
      v[j] *= p.alpha;
      if (p.bias != nullptr) v[j] += p.bias[gn0 + j];
      if (p.residual != nullptr) v[j] += p.residual[o + j * p.cn];
      if (p.accumulate) v[j] += p.C[o + j * p.cn];
      if (!vec) p.C[o + j * p.cn] = v[j];
    }
    if (vec) *reinterpret_cast<float4*>(p.C + o) = make_float4(v[0], v[1], v[2], v[3]);
  }
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
  grid_launch_dependents();
  grid_dependency_wait();
  x = from_here(x);
  F = from_here(F);
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
  grid_launch_dependents();
  grid_dependency_wait();
  const float *X = from_here(q.X), *H = from_here(q.H);
#pragma unroll 4
  for (int m = part; m < M; m += parts) {
    const float xv = c < q.C ? X[static_cast<int64_t>(m) * q.C + c] : 0.0f;
#pragma unroll
    for (int j = 0; j < kGradCols; ++j)
      if (j0 + j < r) acc[j] = fmaf(xv, __ldg(H + m * q.hm + (j0 + j) * q.hj), acc[j]);
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
  grid_launch_dependents();
  grid_dependency_wait();
  x = from_here(x);
  A = from_here(A);
  B = from_here(B);
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
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = chained_launch() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(cluster); attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
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
// CTAs that share a tile's reduction (0: no cluster of that size fits the device).  In steps of 64 reduction indices: a CTA's
// start, drain and write-out cost some four steps, and the exchange of the partial tiles two more; tiles go over the resident clusters
// in whole rounds.
int pick_splits(int64_t tiles, int64_t ksteps, const int (&resident)[kMaxSplits + 1]) {
  int best = 1;
  double best_cost = 0.0;
  for (int s = 1; s <= kMaxSplits && (s == 1 || s <= ksteps); ++s) {
    if (resident[s] <= 0) continue;
    const double rounds = static_cast<double>((tiles + resident[s] - 1) / resident[s]);
    const double cost = rounds * (static_cast<double>((ksteps + s - 1) / s) + 4.0 + (s > 1 ? 2.0 : 0.0));
    if (best_cost == 0.0 || cost < best_cost) { best = s; best_cost = cost; }
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

template <int BN>
int launch_tiles(DeviceState* ds, TileParams p, cudaStream_t st) {
  const void* kernel = reinterpret_cast<const void*>(&tile_kernel<BN>);
  constexpr size_t smem = TileSmem<BN>::kBytes;
  int (&resident)[kMaxSplits + 1] = ds->f32_tile_clusters[BN == 64];
  if (resident[1] == 0) {
    MCB_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    for (int s = kMaxSplits; s >= 1; --s) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = static_cast<unsigned>(s); attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
      cfg.gridDim = dim3(static_cast<unsigned>(s)); cfg.blockDim = dim3(kTileThreads); cfg.dynamicSmemBytes = smem;
      cfg.attrs = attr; cfg.numAttrs = 1;
      int n = 0;
      if (s == 1) n = ds->sm_count;
      else if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) { cudaGetLastError(); n = -1; }
      resident[s] = n > 0 ? n : -1;
    }
  }
  p.n_tiles = (p.N + BN - 1) / BN;
  const int64_t tiles = static_cast<int64_t>((p.M + kTileM - 1) / kTileM) * p.n_tiles;
  p.splits = pick_splits(tiles, (p.K + kStep - 1) / kStep, resident);
  if (tiles * p.splits > 0x7fffffffll) return fail(MCB_ERR_SHAPE, "f32 path: %d x %d outputs", p.M, p.N);
  void* args[] = {&p};
  const cudaError_t e = launch_cluster(kernel, dim3(static_cast<unsigned>(tiles * p.splits)), kTileThreads, smem, p.splits, st, args);
  if (e != cudaSuccess) return cuda_fail(e, "f32 tile_kernel launch");
  MCB_CHECK_LAUNCH("f32 tile_kernel");
  return MCB_OK;
}

int gemm(cudaStream_t st, TileParams p) {
  DeviceState* ds = current_device_state();
  if (!ds) return MCB_ERR_NOT_INIT;
  if (p.residual != nullptr && p.residual == p.C) return fail(MCB_ERR_UNSUPPORTED, "f32 path: residual must not alias the output");
  p.status = ds->status_word;
  if (p.K <= kShort && p.R <= kShort) {
    p.n_tiles = (p.N + kShortRows - 1) / kShortRows;
    const int64_t tiles = static_cast<int64_t>((p.M + kShortRows - 1) / kShortRows) * p.n_tiles;
    if (tiles > 0x7fffffffll) return fail(MCB_ERR_SHAPE, "f32 path: %d x %d outputs", p.M, p.N);
    MCB_CHECK_CUDA(launch_kernel(short_kernel, dim3(static_cast<unsigned>(tiles)), dim3(kShortThreads), 0, st, chained_launch(), p));
    MCB_CHECK_LAUNCH("f32 short_kernel");
    return MCB_OK;
  }
  return p.N <= 64 ? launch_tiles<64>(ds, p, st) : launch_tiles<128>(ds, p, st);
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
  MCB_CHECK_CUDA(launch_kernel(rank_kernel, grid, dim3(kRankWarps * 32), 0, st, chained_launch(), x, F, fk, fj, out, om, oj, static_cast<int>(M),
                               static_cast<int>(K), static_cast<int>(r), scale));
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
