// The fused linear for shapes with too few output tiles for the chip:
//     Y[M,N] = X[M,K] . W[N,K]^T (+ bias) (+ residual) + (scale X P^T) Q^T        (as umma_gemm.cu)
// and its gate/up/SwiGLU form, on tcgen05 tiles of 128 x BN with the reduction shared by the CTAs of a cluster.
//
// Bound: latency, and the L2 feed of the few SMs that have a tile.  333 tokens x 896 outputs are 12 tiles of 128 x 224: on
// the persistent kernel 12 of 148 SMs stream the whole weight, and a down projection's 76 k-blocks (or the 2374 of the
// lm_head backward) run one after the other.  Here the tile is narrowed and its reduction cut into up to 8 parts until the
// chip is full (the choice is `split_plan` below); a CTA computes one part of one tile:
//   warp 0  TMA loads (128B swizzle) into a stage ring    warp 1  tcgen05.mma, accumulator in tensor memory
//   warps 2-9  stage Q in shared memory meanwhile, then move the float32 accumulator into shared memory (over the ring)
// and after the cluster barrier each CTA adds up its share of the tile's rows from all parts through distributed shared
// memory, in rank order (deterministic, no workspace), finishes the rank path (sum, scale, round to bf16, multiply by Q:
// the operands and roundings of the tensor-core form, accumulated in float32) and writes whole 8-byte pieces of rows.
// Every wait is bounded; a CTA whose wait ran out still meets its cluster's barriers.
#include <cooperative_groups.h>
#include <cuda.h>
#include <string.h>

#include "lora_internal.cuh"
#include "umma_ptx.cuh"

namespace cg = cooperative_groups;

namespace mcb {
namespace bf16path {
using namespace umma;
namespace {

constexpr int kSplitThreads = 320, kSplitMaxStages = 8, kSplitBK = 64;
constexpr int kSplitAhead = 16;   // k-blocks of the weight that a CTA asks for ahead: at most 148 x 16 x 32 KB, within L2
constexpr uint32_t kSplitSmemMax = 227 * 1024 - 1024;

struct SplitParams {
  int M, N, K;
  int BN, rp, stages, splits, nkb, m_tiles;
  int swiglu;        // 1: columns [0, 128) of a tile are gate features, [128, 256) the same features of up
  float scale;
  __nv_bfloat16* Y;  // swiglu: gate [M, F]
  __nv_bfloat16 *up, *act;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* R;
  const __nv_bfloat16* Q;   // [N, rp]
  __nv_bfloat16* H;
  int64_t h_pitch;
  int* status;
  uint32_t stage_bytes, w_off, p_off;
  uint32_t qs_off, hs_off, bar_off;
  int pitch;         // floats per row of the partial tile: 4 mod 32
};

__device__ __forceinline__ float4 ld_peer4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float2 ld_peer2(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}

// S: reduction parts = CTAs of the cluster
template <int S>
__global__ void __launch_bounds__(kSplitThreads, 1)
lora_gemm_split_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW,
                       const __grid_constant__ CUtensorMap tmP, const SplitParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen_base = smem_raw + (base - smem_u32(smem_raw));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t full0 = base + p.bar_off, empty0 = full0 + 8 * kSplitMaxStages, done_bar = empty0 + 8 * kSplitMaxStages;
  const uint32_t tmem_slot = done_bar + 8, abort_addr = tmem_slot + 4;
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(gen_base + (tmem_slot - base));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen_base + (abort_addr - base));
  cg::cluster_group cl = cg::this_cluster();
  const int split = blockIdx.x % S, tile = blockIdx.x / S;
  const int m0 = (tile % p.m_tiles) * BM, nt = tile / p.m_tiles, n0 = nt * p.BN;   // neighbours share the W tile
  const int kb_begin = static_cast<int>(static_cast<int64_t>(p.nkb) * split / S);
  const int kb_end = static_cast<int>(static_cast<int64_t>(p.nkb) * (split + 1) / S);
  const int cols = p.BN + p.rp;
  const uint32_t tmem_cols = cols <= 32 ? 32u : cols <= 64 ? 64u : cols <= 128 ? 128u : 256u;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
    mbar_init(done_bar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  grid_launch_dependents();
  // The set-up above runs under the tail of the kernel before, and so does the weight's way from HBM to L2: a model's weights are
  // more than L2 holds, so with 333 tokens every launch finds them cold and its first k-blocks waited for HBM.  The CTAs of the
  // m-tiles that share a weight tile ask for its k-blocks in turn.  With the like of it in the pack, RMSNorm and rotary kernels: forward of
  // 24 layers with 333 tokens 1817 -> 1665 us, with 128 tokens and four adapters a layer 1865 -> 1677, training pass of 6 layers with 512
  // tokens 1673 -> 1610.  (Two CTAs per SM, so that the next launch's could ask even earlier, cost the ring its depth: 1809 and 1735.)
  if (warp == 0 && lane == 0) {
    prefetch_map(&tmX);
    if (p.rp > 0) prefetch_map(&tmP);
    const int kb_ahead = min(kb_end, kb_begin + kSplitAhead * p.m_tiles);
    for (int kb = kb_begin + tile % p.m_tiles; kb < kb_ahead; kb += p.m_tiles) tma_prefetch_l2_2d(&tmW, kb * kSplitBK, n0);
  } else if (warp == 2 && p.bias != nullptr && !p.swiglu) {
    for (int c = lane * 64; c < p.BN && n0 + c < p.N; c += 32 * 64) prefetch_l2(p.bias + n0 + c);
  }
  grid_dependency_wait();
  float* part = reinterpret_cast<float*>(gen_base);                    // [128][pitch], over the stage ring
  uint32_t* qs = reinterpret_cast<uint32_t*>(gen_base + p.qs_off);     // [rp / 2][BN]: pairs of rank columns of Q
  uint32_t* hs = reinterpret_cast<uint32_t*>(gen_base + p.hs_off);     // [128 rows][rp / 2]

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb_begin; kb < kb_end; ++kb) {
        if (!mbar_wait(empty0 + 8 * stage, phase ^ 1, abort_flag, 13, p.status)) break;
        const uint32_t fb = full0 + 8 * stage, sb = base + stage * p.stage_bytes;
        mbar_expect_tx(fb, p.stage_bytes);
        tma_load_2d(sb, &tmX, fb, kb * kSplitBK, m0);
        tma_load_2d(sb + p.w_off, &tmW, fb, kb * kSplitBK, n0);
        if (p.rp > 0) tma_load_2d(sb + p.p_off, &tmP, fb, kb * kSplitBK, 0);
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = make_idesc(cols);   // P lies behind W in a stage: one MMA fills main and rank columns
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = kb_begin; kb < kb_end; ++kb) {
        ok = mbar_wait(full0 + 8 * stage, phase, abort_flag, 25, p.status);
        if (!ok) break;
        tcgen05_fence_after();
        const uint32_t sb = base + stage * p.stage_bytes;
#pragma unroll
        for (int k4 = 0; k4 < kSplitBK / 16; ++k4)
          umma_bf16(tmem_base, desc_sw128(sb + k4 * 32), desc_sw128(sb + p.w_off + k4 * 32), idesc, (kb > kb_begin || k4 > 0) ? 1u : 0u);
        umma_commit(empty0 + 8 * stage);
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
      if (ok) umma_commit(done_bar);
    }
  } else {
    constexpr int kEpi = kSplitThreads - 64;
    for (int e = threadIdx.x - 64; e < p.BN * p.rp / 2; e += kEpi) {
      const int n = e % p.BN, j2 = e / p.BN;
      qs[e] = n0 + n < p.N ? reinterpret_cast<const uint32_t*>(p.Q + static_cast<int64_t>(n0 + n) * p.rp)[j2] : 0u;
    }
    const bool ok = __all_sync(0xffffffffu, mbar_wait(done_bar, 0, abort_flag, 33, p.status));
    if (ok) {
      // two warps per lane quadrant take alternate blocks of 32 columns (both loads of a block in flight)
      tcgen05_fence_after();
      const int quad = warp & 3;
      float* prow = part + (quad * 32 + lane) * p.pitch;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
      for (int c = ((warp - 2) >> 2) * 32; c < cols; c += 64) {
        uint32_t v[2][16];
        tmem_ld_x16(taddr + c, v[0]);
        if (c + 16 < cols) tmem_ld_x16(taddr + c + 16, v[1]);
        tmem_ld_wait();
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (c + 16 * h < cols)
#pragma unroll
            for (int q = 0; q < 4; ++q)
              *reinterpret_cast<uint4*>(prow + c + 16 * h + 4 * q) = make_uint4(v[h][4 * q], v[h][4 * q + 1], v[h][4 * q + 2], v[h][4 * q + 3]);
      }
    }
  }
  __syncwarp();
  if (*abort_flag != 0) {
    for (int k = 0; k < 200; ++k) __nanosleep(1000);
  }
  tcgen05_fence_before();
  if constexpr (S > 1) cl.sync();
  else __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
  }
  // ---- each CTA finishes its share of the rows ----
  constexpr int kRows = BM / S;
  const int r_begin = kRows * split;
  uint32_t peers[S];   // every part's copy of this CTA's rows
#pragma unroll
  for (int q = 0; q < S; ++q) {
    const uint32_t at = base + static_cast<uint32_t>(r_begin * p.pitch) * 4;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peers[q]) : "r"(at), "r"(q));
  }
  auto sum4 = [&](int row, int col) {   // parts in rank order, all loads in flight
    const uint32_t off = static_cast<uint32_t>(row * p.pitch + col) * 4;
    float4 v[S];
#pragma unroll
    for (int q = 0; q < S; ++q) v[q] = ld_peer4(peers[q] + off);
#pragma unroll
    for (int q = 1; q < S; ++q) { v[0].x += v[q].x; v[0].y += v[q].y; v[0].z += v[q].z; v[0].w += v[q].w; }
    return v[0];
  };
  if (p.rp > 0) {
    const int half = p.rp / 2;
    for (int e = threadIdx.x; e < kRows * half; e += kSplitThreads) {
      const int r = e % kRows, j2 = e / kRows;
      float2 v[S];
#pragma unroll
      for (int q = 0; q < S; ++q) v[q] = ld_peer2(peers[q] + static_cast<uint32_t>(r * p.pitch + p.BN + 2 * j2) * 4);
#pragma unroll
      for (int q = 1; q < S; ++q) { v[0].x += v[q].x; v[0].y += v[q].y; }
      const uint32_t w = pack_bf16(v[0].x * p.scale, v[0].y * p.scale);
      hs[r * half + j2] = w;
      const int64_t grow = m0 + r_begin + r;
      if (p.H != nullptr && nt == 0 && grow < p.M) {
        p.H[static_cast<int64_t>(2 * j2) * p.h_pitch + grow] = __ushort_as_bfloat16(static_cast<unsigned short>(w & 0xffffu));
        p.H[static_cast<int64_t>(2 * j2 + 1) * p.h_pitch + grow] = __ushort_as_bfloat16(static_cast<unsigned short>(w >> 16));
      }
    }
    __syncthreads();
  }
  const int rows = min(kRows, p.M - m0 - r_begin);   // rows of the share that exist (may be negative)
  const int out_cols = p.swiglu ? 128 : p.BN;
  const int groups = out_cols / 4, lanes_r = kSplitThreads / groups;   // a thread keeps 4 columns and walks over rows
  const int c = (threadIdx.x % groups) * 4, tr = threadIdx.x / groups;
  constexpr int kBatch = S >= 4 ? 2 : 4;             // rows in flight per thread
  if (tr < lanes_r) {
    if (p.swiglu) {
      const int F = p.N >> 1, f0 = nt * 128 + c;
#pragma unroll 2
      for (int r = tr; r < rows; r += lanes_r) {
        const float4 g = sum4(r, c), u = sum4(r, 128 + c);
        const int64_t o = static_cast<int64_t>(m0 + r_begin + r) * F + f0;
        *reinterpret_cast<uint2*>(p.Y + o) = make_uint2(pack_bf16(g.x, g.y), pack_bf16(g.z, g.w));
        *reinterpret_cast<uint2*>(p.up + o) = make_uint2(pack_bf16(u.x, u.y), pack_bf16(u.z, u.w));
        *reinterpret_cast<uint2*>(p.act + o) = make_uint2(pack_bf16(silu_mul(g.x, u.x), silu_mul(g.y, u.y)),
                                                          pack_bf16(silu_mul(g.z, u.z), silu_mul(g.w, u.w)));
      }
    } else if (n0 + c < p.N) {
      float bias[4] = {};
      if (p.bias != nullptr) {
#pragma unroll
        for (int j = 0; j < 4; ++j) bias[j] = __bfloat162float(p.bias[n0 + c + j]);
      }
      for (int r0 = tr; r0 < rows; r0 += kBatch * lanes_r) {
        float4 v[kBatch];
        uint2 rv[kBatch];
        int64_t o[kBatch];
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
          const int r = min(r0 + b * lanes_r, rows - 1);   // (rows beyond the end repeat the last one and are not stored)
          o[b] = static_cast<int64_t>(m0 + r_begin + r) * p.N + n0 + c;
          v[b] = sum4(r, c);
          if (p.R != nullptr) rv[b] = *reinterpret_cast<const uint2*>(p.R + o[b]);
        }
        for (int j2 = 0; j2 < p.rp / 2; ++j2) {
          const uint4 q4 = *reinterpret_cast<const uint4*>(qs + j2 * p.BN + c);
#pragma unroll
          for (int b = 0; b < kBatch; ++b) {
            const uint32_t h2 = hs[min(r0 + b * lanes_r, rows - 1) * (p.rp / 2) + j2];
            const float ha = __uint_as_float(h2 << 16), hb = __uint_as_float(h2 & 0xffff0000u);
            v[b].x = fmaf(hb, __uint_as_float(q4.x & 0xffff0000u), fmaf(ha, __uint_as_float(q4.x << 16), v[b].x));
            v[b].y = fmaf(hb, __uint_as_float(q4.y & 0xffff0000u), fmaf(ha, __uint_as_float(q4.y << 16), v[b].y));
            v[b].z = fmaf(hb, __uint_as_float(q4.z & 0xffff0000u), fmaf(ha, __uint_as_float(q4.z << 16), v[b].z));
            v[b].w = fmaf(hb, __uint_as_float(q4.w & 0xffff0000u), fmaf(ha, __uint_as_float(q4.w << 16), v[b].w));
          }
        }
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
          if (r0 + b * lanes_r >= rows) break;
          float f[4] = {v[b].x + bias[0], v[b].y + bias[1], v[b].z + bias[2], v[b].w + bias[3]};
          if (p.R != nullptr) {
            f[0] += __uint_as_float(rv[b].x << 16); f[1] += __uint_as_float(rv[b].x & 0xffff0000u);
            f[2] += __uint_as_float(rv[b].y << 16); f[3] += __uint_as_float(rv[b].y & 0xffff0000u);
          }
          *reinterpret_cast<uint2*>(p.Y + o[b]) = make_uint2(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]));
        }
      }
    }
  }
  if constexpr (S > 1) cl.sync();   // nobody leaves while a peer still reads its part
}

typedef CUresult (*EncodeTiledFnS)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
int split_map(const DeviceState* ds, CUtensorMap* map, const void* ptr, int64_t inner, int64_t outer, int box_outer, const char* what) {
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(inner), static_cast<cuuint64_t>(outer)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(inner) * 2};
  cuuint32_t box[2] = {kSplitBK, static_cast<cuuint32_t>(box_outer)};
  cuuint32_t estr[2] = {1, 1};
  const CUresult r = reinterpret_cast<EncodeTiledFnS>(ds->encode_tiled)(
      map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(MCB_ERR_ALIGN, "split GEMM: tensor map for %s rejected (CUresult %d)", what, static_cast<int>(r));
  return MCB_OK;
}

// Cycles of one k-block (64 of the reduction) of a CTA: what it pulls from L2, or the tensor pipe (one cycle per
// accumulator column).
double kblock_cycles(double rows, double cols, double bytes_per_cycle) {
  const double feed = rows * 128.0 / bytes_per_cycle;
  return feed > cols ? feed : cols;
}

typedef void (*SplitKernel)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const SplitParams);
SplitKernel split_kernel(int s) {
  return s == 8 ? lora_gemm_split_kernel<8> : s == 4 ? lora_gemm_split_kernel<4> : s == 2 ? lora_gemm_split_kernel<2> : lora_gemm_split_kernel<1>;
}

}  // namespace

// Raises the kernels' shared-memory limits and asks how many clusters of each size the device runs at once: a GPC's SMs do
// not divide evenly into clusters, so 8 x 18 or 148 is not the number.
int init_split_kernel(DeviceState* ds) {
  for (int s : {1, 2, 4, 8}) {
    const cudaError_t e = cudaFuncSetAttribute(split_kernel(s), cudaFuncAttributeMaxDynamicSharedMemorySize, kSplitSmemMax + 1024);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(lora_gemm_split_kernel)");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(s)); cfg.blockDim = dim3(kSplitThreads); cfg.dynamicSmemBytes = kSplitSmemMax + 1024;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(s); attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int n = 0;
    const cudaError_t q = cudaOccupancyMaxActiveClusters(&n, split_kernel(s), &cfg);
    if (q != cudaSuccess) return cuda_fail(q, "cudaOccupancyMaxActiveClusters(lora_gemm_split_kernel)");
    ds->split_clusters[s] = n > 0 ? n : 1;
  }
  return MCB_OK;
}

// Tile width and reduction parts for a shape, or BN = 0 where the persistent kernels (umma_gemm.cu, umma_gemm2.cu) are
// expected to be about as fast.  Estimated cycles: rounds of CTAs over the SMs x (k-blocks of a part + what a tile costs
// once).  The constants are fitted to launches of 64 .. 2048 tokens and reductions of 896 .. 151936, measured in us (graph
// replay, weights from HBM), persistent kernel / this one:
//   64 x 896 -> 896        10.9 /  5.9      512 x 896 -> 896        13.5 /  7.8      2048 x 896 -> 896     11.3 /  9.4
//   333 x 896 -> 896 r16   13.0 / 10.1      333 x 4864 -> 896       40.4 / 13.4      2048 x 4864 -> 896    32.9 / 21.3
//   512 x 151936 -> 896    1023 / 189       1000 x 896 -> 896 r16   13.2 / 11.7      512 x 896 -> 4864     12.9 / 10.0
SplitPlan split_plan(int64_t M, int64_t N, int64_t K, int rp, bool pair_kernel, const DeviceState* ds) {
  SplitPlan best;
  const int nkb = static_cast<int>((K + kSplitBK - 1) / kSplitBK);
  const int64_t mt = (M + BM - 1) / BM;
  const int cap = rp > 0 ? ((256 - rp) / 32) * 32 : 256;
  double best_cost;
  {
    // the persistent kernel that would run instead
    const int64_t tiles_n = (N + cap - 1) / cap;
    const int bn = static_cast<int>(((N + tiles_n - 1) / tiles_n + 31) / 32 * 32);
    const int64_t tiles = pair_kernel ? (M + 255) / 256 * tiles_n : mt * tiles_n, slots = pair_kernel ? ds->sm_count / 2 : ds->sm_count;
    if (tiles > slots) return best;   // the chip is full
    best_cost = 0.93 * (13700.0 + nkb * kblock_cycles(pair_kernel ? 128 + (bn + rp) / 2 : 128 + bn + rp, bn + rp, 50.0));
  }
  for (int bn = 32; bn <= cap; bn += 32) {
    const int64_t nt = (N + bn - 1) / bn;
    if (bn > 32 && nt == (N + bn - 33) / (bn - 32)) continue;   // the narrower tile needs no more of them
    for (int s = 1; s <= 8; s *= 2) {
      if (s > 1 && nkb < 2 * s) break;
      const double rounds = static_cast<double>((mt * nt + ds->split_clusters[s] - 1) / ds->split_clusters[s]);
      const double rank = 128.0 / s * bn / 4.0 / kSplitThreads * rp * 28.0;
      const double main = (nkb + s - 1) / s * kblock_cycles(128 + bn + rp, bn + rp, 55.0);
      const double cost = 9900.0 + (s > 1 ? 1900.0 + 230.0 * s : 0.0) + rounds * (main + rank) + (rounds - 1.0) * 6500.0;
      if (cost < best_cost) { best_cost = cost; best.bn = bn; best.splits = s; }
    }
  }
  return best;
}

int launch_split(const SplitPlan& plan, const GemmCall& c, __nv_bfloat16* up, __nv_bfloat16* act, const DeviceState* ds, cudaStream_t st) {
  SplitParams p;
  memset(&p, 0, sizeof(p));
  p.M = static_cast<int>(c.M); p.N = static_cast<int>(c.N); p.K = static_cast<int>(c.K);
  p.BN = plan.bn; p.splits = plan.splits; p.rp = c.rp;
  p.nkb = (p.K + kSplitBK - 1) / kSplitBK;
  p.m_tiles = (p.M + BM - 1) / BM;
  p.swiglu = act != nullptr ? 1 : 0;
  p.scale = c.scale;
  p.Y = c.Y; p.up = up; p.act = act; p.bias = c.bias; p.R = c.R; p.Q = c.Q; p.H = c.H; p.h_pitch = c.h_pitch; p.status = ds->status_word;
  p.w_off = BM * kSplitBK * 2;
  p.p_off = p.w_off + p.BN * kSplitBK * 2;
  p.stage_bytes = p.p_off + p.rp * kSplitBK * 2;
  p.pitch = (p.BN + p.rp + 31) / 32 * 32 + 4;
  const uint32_t part_bytes = static_cast<uint32_t>(BM * p.pitch * 4 + 1023) & ~1023u;
  const uint32_t qs_bytes = static_cast<uint32_t>(p.BN) * p.rp * 2, hs_bytes = BM * p.rp * 2u;
  const uint32_t fixed = qs_bytes + hs_bytes + 512;
  int stages = static_cast<int>((kSplitSmemMax - fixed) / p.stage_bytes);
  const int per_cta = (p.nkb + p.splits - 1) / p.splits;
  if (stages > kSplitMaxStages) stages = kSplitMaxStages;
  if (stages > per_cta) stages = per_cta;
  p.stages = stages;
  const uint32_t ring = stages * p.stage_bytes;
  p.qs_off = ring > part_bytes ? ring : part_bytes;
  p.hs_off = p.qs_off + qs_bytes;
  p.bar_off = p.hs_off + hs_bytes;
  const uint32_t smem = p.bar_off + 256 + 1024;
  if (stages < 1 || smem > kSplitSmemMax + 1024) return fail(MCB_ERR_UNSUPPORTED, "split GEMM: tile does not fit shared memory (BN=%d rp=%d)", p.BN, p.rp);
  CUtensorMap tmX, tmW, tmP;
  if (int rc = split_map(ds, &tmX, c.X, c.K, c.M, BM, "X")) return rc;
  if (int rc = split_map(ds, &tmW, c.W, c.K, c.N, p.BN, "W")) return rc;
  if (p.rp > 0) { if (int rc = split_map(ds, &tmP, c.P, c.K, p.rp, p.rp, "P")) return rc; }
  else tmP = tmX;
  const int64_t n_tiles = (c.N + p.BN - 1) / p.BN;
  const bool prof = profile_on();
  if (prof) {
    const double m = static_cast<double>(c.M), n = static_cast<double>(c.N), k = static_cast<double>(c.K);
    profile_begin(c.rp > 0 ? kProfGemmLora : kProfGemm, 2.0 * m * n * k + 2.0 * m * c.r_true * (k + n),
                  2.0 * (m * k + n * k + (act ? 1.5 : 1.0) * m * n) + 2.0 * c.rp * (k + n), st);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(p.m_tiles * n_tiles * p.splits)); cfg.blockDim = dim3(kSplitThreads);
  cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (p.splits > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = static_cast<unsigned>(p.splits); attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = 1;
    ++na;
  }
  if (chained_launch()) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr; cfg.numAttrs = na;
  const cudaError_t le = cudaLaunchKernelEx(&cfg, split_kernel(p.splits), tmX, tmW, tmP, p);
  if (le != cudaSuccess) return cuda_fail(le, "lora_gemm_split_kernel launch");
  if (prof) profile_end(st);
  MCB_CHECK_LAUNCH("lora_gemm_split_kernel");
  return MCB_OK;
}

}  // namespace bf16path
}  // namespace mcb
