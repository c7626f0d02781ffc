// Linear without a rank path of its own,  Y[M,N] = X[M,K] . W[N,K]^T (+ X2[M,K2] . W2[N,K2]^T) (+ bias) (+ residual),  and the
// gate/up/SwiGLU form of umma_gemm2.cu, on CTA pairs with tiles of 256 x up to 512.
//
// Bound: what an SM pulls from L2, about 42 bytes per cycle whatever the shape.  The pair kernel's 256 x 256 tile needs 32 KB per
// CTA and 64-wide k-block, 780 cycles of that feed for 512 cycles of the tensor pipe; a 256 x 512 tile needs 48 KB for 1024.
// Its accumulators fill tensor memory (two halves of BN / 2 columns, one pair MMA each), so they cannot be doubled; instead the
// halves take turns at a tile's ends.  The first `turn` k-blocks of a tile go into half 0 while the epilogue still empties half 1
// of the tile before, then into half 1; the last `turn` are finished in half 0 first, which is emptied while half 1 gets them:
//   half 0:  k 0..t-1          |  k t .. n-t-1 |  k n-t..n-1                   | (emptied)
//   half 1:           k 0..t-1 |  (both)       |              k n-t..n-1       |           (emptied under the next tile's first)
// A k-block's stage is given back when both halves have used it.
//
// Per CTA: warp 0 loads its own 128 rows of X and a quarter of the W tile's rows for either half (TMA, 128B swizzle); warp 1 of
// the pair's leader issues the MMAs; warps 2-9 empty the accumulators, two warps per 32 rows, every other block of 32 columns.
// Barriers as in umma_gemm2.cu: full[s] in the leader counts both CTAs' bytes, empty[s] and done[h] are committed to both CTAs,
// acc_empty[h] in the leader counts the epilogue warps of both.  No load uses cluster multicast.  Every wait is bounded.
#include <cuda.h>
#include <string.h>

#include "lora_internal.cuh"
#include "umma_ptx.cuh"

namespace mcb {
namespace bf16path {
using namespace umma;
namespace {

constexpr int kWideBK = 64, kWideThreads = 320, kWideEpiWarps = 8, kWideMaxStages = 6;
constexpr int kWideSmem = 227 * 1024 - 1024;

struct WideParams {
  int M, N;          // swiglu: N = 2 F, the outputs are [M, F]
  int BN, stages, turn, swiglu, epi_bufs;
  int num_m_tiles, num_n_tiles, num_tiles, nkb, k1_blocks, group_m;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* R;
  int* status;
  uint32_t stage_bytes, w_off, w_half, epi_off, bar_off;
};

__device__ __forceinline__ void wide_tile(const WideParams& p, int t, int& mt, int& nt) {
  const int per_band = p.group_m * p.num_n_tiles;
  const int band = t / per_band, in = t - band * per_band, m_first = band * p.group_m;
  const int gm = min(p.group_m, p.num_m_tiles - m_first);
  nt = in / gm;
  mt = m_first + in % gm;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kWideThreads, 1)
gemm_wide_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX2,
                 const __grid_constant__ CUtensorMap tmW2, const __grid_constant__ CUtensorMap tmY, const __grid_constant__ CUtensorMap tmU,
                 const __grid_constant__ CUtensorMap tmAct, const WideParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen_base = smem_raw + (base - smem_u32(smem_raw));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const uint32_t full0 = base + p.bar_off, empty0 = full0 + 8 * kWideMaxStages, done0 = empty0 + 8 * kWideMaxStages;
  const uint32_t acc_empty0 = done0 + 16, tmem_slot = acc_empty0 + 16, abort_addr = tmem_slot + 4;
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(gen_base + (tmem_slot - base));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen_base + (abort_addr - base));

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
    for (int h = 0; h < 2; ++h) { mbar_init(done0 + 8 * h, 1); mbar_init(acc_empty0 + 8 * h, 2 * kWideEpiWarps); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anything arrives on them remotely
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  grid_launch_dependents();
  grid_dependency_wait();   // the set-up above ran under the tail of the kernel before
  const int half_n = p.BN / 2, quarter_n = p.BN / 4;

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs) ----------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = pair; ok && t < p.num_tiles; t += npairs) {
        int mt, nt;
        wide_tile(p, t, mt, nt);
        const int m0 = mt * 256 + static_cast<int>(rank) * 128;
        const int n0 = nt * p.BN + static_cast<int>(rank) * quarter_n;
        for (int kb = 0; kb < p.nkb; ++kb) {
          ok = mbar_wait(empty0 + 8 * stage, phase ^ 1, abort_flag, 110, p.status);
          if (!ok) break;
          const uint32_t fb = map_to_cta(full0 + 8 * stage, 0);  // the leader's barrier
          const uint32_t sb = base + stage * p.stage_bytes;
          const bool first = kb < p.k1_blocks;
          const int k0 = (first ? kb : kb - p.k1_blocks) * kWideBK;
          if (rank == 0) mbar_expect_tx(full0 + 8 * stage, 2 * p.stage_bytes);
          tma_load_2d_pair(sb, first ? &tmX : &tmX2, fb, k0, m0);
          tma_load_2d_pair(sb + p.w_off, first ? &tmW : &tmW2, fb, k0, n0);
          tma_load_2d_pair(sb + p.w_off + p.w_half, first ? &tmW : &tmW2, fb, k0, n0 + half_n);
          if (++stage == p.stages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA only) ----------------
    if (lane == 0 && rank == 0) {
      const uint32_t idesc = make_idesc2(half_n);
      int stage = 0;
      uint32_t phase = 0, acc_phase = 1;
      bool ok = true;
      auto mma = [&](int st, int h, bool add) {
        const uint32_t sb = base + st * p.stage_bytes, wb = sb + p.w_off + h * p.w_half;
#pragma unroll
        for (int k4 = 0; k4 < kWideBK / 16; ++k4)
          umma2_bf16(tmem_base + h * 256, desc_sw128(sb + k4 * 32), desc_sw128(wb + k4 * 32), idesc, add || k4 > 0 ? 1u : 0u);
      };
      auto next = [&](int& st, uint32_t& ph) { if (++st == p.stages) { st = 0; ph ^= 1; } };
      // k-blocks [k0, k1): all of them into half 0, then all into half 1
      auto in_turn = [&](int k0, int k1, bool first, bool last) -> bool {
        int st = stage;
        uint32_t ph = phase;
        if (first && !mbar_wait(acc_empty0, acc_phase, abort_flag, 111, p.status)) return false;
        tcgen05_fence_after();
        for (int kb = k0; kb < k1; ++kb) {
          if (!mbar_wait(full0 + 8 * st, ph, abort_flag, 112, p.status)) return false;
          tcgen05_fence_after();
          mma(st, 0, kb > 0);
          next(st, ph);
        }
        if (last) umma2_commit_both(done0);
        if (first && !mbar_wait(acc_empty0 + 8, acc_phase, abort_flag, 113, p.status)) return false;
        tcgen05_fence_after();
        for (int kb = k0; kb < k1; ++kb) {
          mma(stage, 1, kb > 0);
          umma2_commit_both(empty0 + 8 * stage);
          next(stage, phase);
        }
        if (last) umma2_commit_both(done0 + 8);
        return true;
      };
      for (int t = pair; ok && t < p.num_tiles; t += npairs) {
        ok = in_turn(0, p.turn, true, false);
        for (int kb = p.turn; ok && kb < p.nkb - p.turn; ++kb) {
          ok = mbar_wait(full0 + 8 * stage, phase, abort_flag, 114, p.status);
          if (!ok) break;
          tcgen05_fence_after();
          mma(stage, 0, kb > 0);
          mma(stage, 1, kb > 0);
          umma2_commit_both(empty0 + 8 * stage);
          next(stage, phase);
        }
        if (ok) ok = in_turn(p.nkb - p.turn, p.nkb, false, true);
        acc_phase ^= 1;
      }
    }
  } else {
    // ---------------- epilogue (warps 2-9, both CTAs): own 128 rows of the pair's tile ----------------
    const int quad = warp & 3, part = (warp - 2) >> 2;
    const int row_in_tile = quad * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t epi_base = base + p.epi_off + static_cast<uint32_t>((warp - 2) * p.epi_bufs) * kEpiBufBytes;
    int sbuf = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = pair; ok && t < p.num_tiles; t += npairs) {
      int mt, nt;
      wide_tile(p, t, mt, nt);
      const int m0 = mt * 256 + static_cast<int>(rank) * 128;
      const int64_t grow = static_cast<int64_t>(m0) + row_in_tile;
      const bool rows_ok = m0 + quad * 32 < p.M;
      for (int h = 0; h < 2; ++h) {
        ok = __all_sync(0xffffffffu, mbar_wait(done0 + 8 * h, phase, abort_flag, 115, p.status));
        if (!ok) break;
        tcgen05_fence_after();
        const uint32_t d = tmem_base + lane_addr + h * 256;
        if (p.swiglu) {
          // columns [0, 128) of a half are gate features, [128, 256) the same features of up
          const int F = p.N >> 1;
          for (int c = 32 * part; c < 128; c += 64) {
            const int fcol = (2 * nt + h) * 128 + c;
            if (fcol >= F) break;
            uint32_t g[2][16], u[2][16];
            tmem_ld_x16(d + c, g[0]);
            tmem_ld_x16(d + c + 16, g[1]);
            tmem_ld_x16(d + 128 + c, u[0]);
            tmem_ld_x16(d + 128 + c + 16, u[1]);
            if (lane == 0) bulk_wait_group_read<0>();  // all three staging buffers have been read
            __syncwarp();
            tmem_ld_wait();
            uint32_t wg[16], wu[16], wa[16];
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
              for (int j = 0; j < 16; j += 2) {
                const float ga = __uint_as_float(g[q][j]), gb = __uint_as_float(g[q][j + 1]);
                const float ua = __uint_as_float(u[q][j]), ub = __uint_as_float(u[q][j + 1]);
                wg[8 * q + (j >> 1)] = pack_bf16(ga, gb);
                wu[8 * q + (j >> 1)] = pack_bf16(ua, ub);
                wa[8 * q + (j >> 1)] = pack_bf16(silu_mul(ga, ua), silu_mul(gb, ub));
              }
            uint8_t* buf = gen_base + (epi_base - base);
            stage_row(buf, lane, wg);
            stage_row(buf + kEpiBufBytes, lane, wu);
            stage_row(buf + 2 * kEpiBufBytes, lane, wa);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0 && rows_ok) {
              tma_store_2d(&tmY, epi_base, fcol, m0 + quad * 32);
              tma_store_2d(&tmU, epi_base + kEpiBufBytes, fcol, m0 + quad * 32);
              tma_store_2d(&tmAct, epi_base + 2 * kEpiBufBytes, fcol, m0 + quad * 32);
              bulk_commit_group();
            }
          }
        } else {
          for (int c = 32 * part; c < half_n; c += 64) {
            const int gcol = nt * p.BN + h * half_n + c;
            if (gcol >= p.N) break;
            uint32_t v0[16], v1[16];
            tmem_ld_x16(d + c, v0);
            tmem_ld_x16(d + c + 16, v1);
            if (lane == 0) bulk_wait_group_read_n(p.epi_bufs - 1);  // the store that last used this buffer has read it
            __syncwarp();
            tmem_ld_wait();
            float f[32];
#pragma unroll
            for (int j = 0; j < 16; ++j) { f[j] = __uint_as_float(v0[j]); f[16 + j] = __uint_as_float(v1[j]); }
            uint32_t w[16];
            finish_cols(f, p.bias, p.R, grow, gcol, p.M, p.N, w);
            const uint32_t buf = epi_base + static_cast<uint32_t>(sbuf) * kEpiBufBytes;
            stage_row(gen_base + (buf - base), lane, w);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0 && rows_ok) {
              tma_store_2d(&tmY, buf, gcol, m0 + quad * 32);
              bulk_commit_group();
            }
            if (++sbuf == p.epi_bufs) sbuf = 0;
          }
        }
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (rank == 0) mbar_arrive(acc_empty0 + 8 * h);
          else mbar_arrive_remote(acc_empty0 + 8 * h, 0);
        }
      }
      phase ^= 1;
    }
    if (lane == 0) bulk_wait_group<0>();  // this warp's output stores are complete before the CTA may exit
  }

  // ---------------- common exit: both CTAs meet before either lets go of shared or tensor memory ----------------
  __syncwarp();
  if (*abort_flag != 0) {
    for (int k = 0; k < 200; ++k) __nanosleep(1000);
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

typedef CUresult (*EncodeTiledFnW)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
int wide_map(const DeviceState* ds, CUtensorMap* map, const void* ptr, int64_t inner, int64_t outer, int box_inner, int box_outer, const char* what) {
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(inner), static_cast<cuuint64_t>(outer)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(inner) * 2};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(box_inner), static_cast<cuuint32_t>(box_outer)};
  cuuint32_t estr[2] = {1, 1};
  const CUresult r = reinterpret_cast<EncodeTiledFnW>(ds->encode_tiled)(
      map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
      box_inner == kWideBK ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(MCB_ERR_ALIGN, "wide GEMM: tensor map for %s rejected (CUresult %d)", what, static_cast<int>(r));
  return MCB_OK;
}

}  // namespace

int init_wide_kernel() {
  const cudaError_t e = cudaFuncSetAttribute(gemm_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kWideSmem + 1024);
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(gemm_wide_kernel)");
  return MCB_OK;
}

// Tile width (a multiple of 64, 320 to 512), or 0 where the pair kernel's tiles of up to 256 columns are expected to be as fast.  Both
// in cycles: rounds of tiles over the pairs x the k-blocks' feed at 42 bytes per cycle (never below the tensor pipe's two cycles per
// column), and for this kernel 6500 per tile for the turns at its ends, during which the stages come back late: K = 896 is
// quicker on the pair kernel (32768 x 896 -> 4864 231 us against 268 here), 4096 here.  Pair kernel / this one, us: 32768 x 4096
// -> 4096 779 / 717, 32768 x 4864 -> 896 252 / 220, 9472 x 151936 -> 896 2260 / 1662.  *cycles: of the better one.
int wide_bn(int64_t M, int64_t N, int64_t nkb, bool swiglu, const DeviceState* ds, double* cycles) {
  const int64_t pairs = ds->sm_count / 2, mt = (M + 255) / 256;
  auto estimate = [&](int64_t bn, double extra) {
    const double rounds = static_cast<double>((mt * ((N + bn - 1) / bn) + pairs - 1) / pairs);
    const double feed = (128.0 + bn / 2.0) * 128.0 / 42.0, pipe = 2.0 * bn;
    return rounds * (nkb * (feed > pipe ? feed : pipe) + extra);
  };
  const int64_t t = (N + 255) / 256;
  double best = 0.97 * estimate(swiglu ? 256 : ((N + t - 1) / t + 31) / 32 * 32, 0.0);
  int bn = 0;
  for (int cand = swiglu ? 512 : 320; nkb >= 4 && cand <= 512; cand += 64) {
    const double c = estimate(cand, 6500.0);
    if (c < best) { best = c; bn = cand; }
  }
  if (cycles != nullptr) *cycles = best;
  return bn;
}

// The call with tiles of `bn` columns.  act != null: c.W holds gate and up interleaved in blocks of 128 rows, c.N = 2 F, and c.Y, up, act
// [M, F] receive gate, up and silu(gate) * up (bn 512).
int launch_wide(int bn, const GemmCall& c, __nv_bfloat16* up, __nv_bfloat16* act, const DeviceState* ds, cudaStream_t st) {
  WideParams p;
  memset(&p, 0, sizeof(p));
  p.M = static_cast<int>(c.M); p.N = static_cast<int>(c.N);
  p.BN = bn;
  p.swiglu = act != nullptr ? 1 : 0;
  p.k1_blocks = static_cast<int>((c.K + kWideBK - 1) / kWideBK);
  p.nkb = p.k1_blocks + static_cast<int>((c.K2 + kWideBK - 1) / kWideBK);
  p.num_m_tiles = static_cast<int>((c.M + 255) / 256);
  p.num_n_tiles = static_cast<int>((c.N + bn - 1) / bn);
  p.num_tiles = p.num_m_tiles * p.num_n_tiles;
  p.group_m = p.num_m_tiles < 8 ? p.num_m_tiles : 8;
  p.bias = c.bias; p.R = c.R; p.status = ds->status_word;
  p.w_off = 128 * kWideBK * 2;
  p.w_half = static_cast<uint32_t>(bn / 4) * kWideBK * 2;   // bn / 4 is a multiple of 16: whole 1024-byte groups of 8 rows
  p.stage_bytes = p.w_off + 2 * p.w_half;
  p.epi_bufs = p.swiglu ? 3 : 2;
  const uint32_t epi_bytes = kWideEpiWarps * static_cast<uint32_t>(p.epi_bufs) * kEpiBufBytes;
  p.stages = static_cast<int>((kWideSmem - epi_bytes - 256) / p.stage_bytes);
  if (p.stages > kWideMaxStages) p.stages = kWideMaxStages;
  if (p.stages < 3) return fail(MCB_ERR_UNSUPPORTED, "wide GEMM: tile does not fit shared memory (BN=%d)", bn);
  // a turn holds its stages until half 1 has used them: one stage stays for the loads ahead
  p.turn = p.stages - 1 < p.nkb / 2 ? p.stages - 1 : p.nkb / 2;
  p.epi_off = static_cast<uint32_t>(p.stages) * p.stage_bytes;
  p.bar_off = p.epi_off + epi_bytes;
  const int64_t cols = p.swiglu ? c.N / 2 : c.N;
  CUtensorMap tmX, tmW, tmX2, tmW2, tmY, tmU, tmA;
  if (int rc = wide_map(ds, &tmX, c.X, c.K, c.M, kWideBK, 128, "X")) return rc;
  if (int rc = wide_map(ds, &tmW, c.W, c.K, c.N, kWideBK, bn / 4, "W")) return rc;
  tmX2 = tmX; tmW2 = tmW;
  if (c.X2 != nullptr) {
    if (int rc = wide_map(ds, &tmX2, c.X2, c.K2, c.M, kWideBK, 128, "X2")) return rc;
    if (int rc = wide_map(ds, &tmW2, c.W2, c.K2, c.N, kWideBK, bn / 4, "W2")) return rc;
  }
  if (int rc = wide_map(ds, &tmY, c.Y, cols, c.M, 32, 32, "Y")) return rc;
  tmU = tmY; tmA = tmY;
  if (p.swiglu) {
    if (int rc = wide_map(ds, &tmU, up, cols, c.M, 32, 32, "up")) return rc;
    if (int rc = wide_map(ds, &tmA, act, cols, c.M, 32, 32, "act")) return rc;
  }
  int pairs = ds->sm_count / 2;
  if (pairs > p.num_tiles) pairs = p.num_tiles;
  const bool prof = profile_on();
  if (prof) {
    const double m = static_cast<double>(c.M), n = static_cast<double>(c.N), k = static_cast<double>(c.K + c.K2);
    profile_begin(gemm_kind(c), gemm_flops(c), 2.0 * (m * k + n * k + (act ? 1.5 : 1.0) * m * n), st);
  }
  const cudaError_t le = launch_kernel(gemm_wide_kernel, dim3(2 * pairs), dim3(kWideThreads), kWideSmem + 1024, st, chained_launch(), tmX, tmW, tmX2,
                                       tmW2, tmY, tmU, tmA, p);
  if (le != cudaSuccess) return cuda_fail(le, "gemm_wide_kernel launch");
  if (prof) profile_end(st);
  MCB_CHECK_LAUNCH("gemm_wide_kernel");
  return MCB_OK;
}

}  // namespace bf16path
}  // namespace mcb
