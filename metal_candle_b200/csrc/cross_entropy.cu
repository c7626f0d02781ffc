// Cross-entropy over logits [M, V], forward and backward (src/training/loss.rs:58-147): nll[row] = logsumexp - logit[target]
// (0 for ignored rows), and with write_grad d loss / d logits = (softmax - onehot) / count, zeros for ignored rows, either
// over the logits or into a tensor of its own.  A second tiny kernel sums nll in row order, so the loss is deterministic.
#include <cooperative_groups.h>

#include <mutex>

#include "common.cuh"
#include "umma_ptx.cuh"

namespace cg = cooperative_groups;

namespace mcb {
namespace {
using namespace umma;

constexpr float kLog2e = 1.4426950408889634f;
// 2^x with denormal results flushed to zero: one instruction, where __expf's denormal handling takes several
// (relative error about 2^-22; the long-row loops below are bound by their instruction count)
__device__ __forceinline__ float ex2_ftz(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void online_combine(float& m, float& s, float m2, float s2) {
  const float mm = fmaxf(m, m2);
  if (mm == -INFINITY) { m = mm; s += s2; return; }   // nothing kept yet: both sums are 0, or NaN from a NaN logit
  s = s * __expf(m - mm) + s2 * __expf(m2 - mm);
  m = mm;
}

// Beyond this magnitude a maximum times log2(e) may overflow: -m log2(e) is then infinite and the fused form
// 2^(x log2e - m log2e) is inf or 0 where x equals m (a row, or a share of one, masked with the type's lowest value).  Such
// maxima take differences first, 2^((x - m) log2e), in loops of their own; no logit in earnest gets there.
constexpr float kFusedMax = 8.507059e37f;   // 2^126
__device__ __forceinline__ bool beyond_fused(float m) { return fabsf(m) > kFusedMax && fabsf(m) != INFINITY; }
__device__ __forceinline__ float exp_diff(float x, float m) { return ex2_ftz((x - m) * kLog2e); }

// Every call in place (the training step's form), and the rows the cluster kernel below does not take: short ones, rows of
// more than 800 KB, and input and output that start differently far from a 16-byte boundary.  Persistent: block b takes rows b, b + gridDim.x, ...; sweep 1 takes the maximum and the sum, sweep 2 reads the
// row again (from L2 while the rows in flight fit it) and writes the gradient.
template <typename T>
__global__ void __launch_bounds__(1024)
cross_entropy_kernel(const T* in, T* out, const int32_t* __restrict__ targets, float* __restrict__ nll,
                     const int32_t* __restrict__ count_ptr, int64_t M, int V, int write_grad) {
  __shared__ float sm[32], ss[32];
  grid_launch_dependents();
  grid_dependency_wait();
  targets = from_here(targets);
  const float inv_count = 1.0f / static_cast<float>(max(1, *from_here(count_ptr)));
  using VT = Vec16<T>;
  constexpr int NV = VT::N;
  const int bd = blockDim.x;
  for (int64_t row = blockIdx.x; row < M; row += gridDim.x) {
    const T* lr = in + row * V;
    T* gr = out + row * V;   // may be the same row
    const int32_t tgt = targets[row];
    const bool ignored = tgt < 0 || tgt >= V;  // u32::MAX (src/training/trainer.rs:385) reads as -1
    if (ignored) {   // the same for every thread of the block
      if (threadIdx.x == 0) nll[row] = 0.0f;
      if (write_grad)
        for (int c = threadIdx.x; c < V; c += bd) gr[c] = from_f32<T>(0.0f);
      continue;
    }
    const bool vec = (V % NV == 0) && (((reinterpret_cast<uintptr_t>(lr) | reinterpret_cast<uintptr_t>(gr)) & 15u) == 0);
    float m = -INFINITY, s = 0.0f;
    if (vec) {
      float m2 = 0.0f;   // -m log2(e), finite also for the lowest values (a row whose maximum is one is summed again below)
      const int nvec = V / NV;
      const auto* src = reinterpret_cast<const decltype(VT::raw)*>(lr);
      auto absorb = [&](const VT& t) {
        float f[NV];
        t.to_float(f);
        float vm = f[0];
#pragma unroll
        for (int j = 1; j < NV; ++j) vm = fmaxf(vm, f[j]);
        if (vm > m) { s *= __expf(m - vm); m = vm; m2 = -fmaxf(m, -kFusedMax) * kLog2e; }
        // exp(f - m) = 2^(f log2e - m log2e): one fused multiply-add and one special function; masked logits add 0, with
        // nothing kept yet (m2 = 0) as well, and a NaN among them reaches the sum
#pragma unroll
        for (int j = 0; j < NV; ++j) s += ex2_ftz(fmaf(f[j], kLog2e, m2));
      };
      int c = threadIdx.x;
      for (; c + 3 * bd < nvec; c += 4 * bd) {   // four loads in flight per thread
        VT t0, t1, t2, t3;
        t0.raw = src[c]; t1.raw = src[c + bd]; t2.raw = src[c + 2 * bd]; t3.raw = src[c + 3 * bd];
        absorb(t0); absorb(t1); absorb(t2); absorb(t3);
      }
      for (; c < nvec; c += bd) {
        VT t; t.raw = src[c];
        absorb(t);
      }
    } else {
      for (int c = threadIdx.x; c < V; c += bd) {
        const float v = to_f32(lr[c]);
        if (v > m) { s = s * __expf(m - v) + 1.0f; m = v; } else if (v != -INFINITY) { s += __expf(v - m); }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float mo = __shfl_xor_sync(0xffffffffu, m, o), so = __shfl_xor_sync(0xffffffffu, s, o);
      online_combine(m, s, mo, so);
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = bd >> 5;
    if (lane == 0) { sm[warp] = m; ss[warp] = s; }
    __syncthreads();
    m = sm[0]; s = ss[0];
    for (int w = 1; w < nw; ++w) online_combine(m, s, sm[w], ss[w]);
    if (beyond_fused(m)) {   // the same for every thread of the block
      float d = 0.0f;
      for (int c = threadIdx.x; c < V; c += bd) d += exp_diff(to_f32(lr[c]), m);
      d = warp_sum(d);
      __syncthreads();   // everyone has read ss
      if (lane == 0) ss[warp] = d;
      __syncthreads();
      s = 0.0f;
      for (int w = 0; w < nw; ++w) s += ss[w];
      if (threadIdx.x == 0) nll[row] = (m - to_f32(lr[tgt])) + logf(s);   // (m + log s would lose the logarithm)
      __syncthreads();
      if (write_grad)
        for (int c = threadIdx.x; c < V; c += bd)
          gr[c] = from_f32<T>((exp_diff(to_f32(lr[c]), m) / s - (c == tgt ? 1.0f : 0.0f)) * inv_count);
      continue;
    }
    const float lse = m + logf(s);
    if (threadIdx.x == 0) nll[row] = lse - to_f32(lr[tgt]);
    __syncthreads();  // thread 0 has read lr[tgt] before anyone overwrites it; sm / ss are free for the next row
    if (write_grad) {
      if (vec) {
        const int nvec = V / NV;
        const auto* src = reinterpret_cast<const decltype(VT::raw)*>(lr);
        auto* dst = reinterpret_cast<decltype(VT::raw)*>(gr);
        const float lse2 = -lse * kLog2e;
        auto grad = [&](VT& t, int c) {
          float f[NV];
          t.to_float(f);
#pragma unroll
          for (int j = 0; j < NV; ++j) {
            float p = ex2_ftz(fmaf(f[j], kLog2e, lse2));
            if (c * NV + j == tgt) p -= 1.0f;
            f[j] = p * inv_count;
          }
          t.from_float(f);
          dst[c] = t.raw;
        };
        int c = threadIdx.x;
        for (; c + 3 * bd < nvec; c += 4 * bd) {
          VT t0, t1, t2, t3;
          t0.raw = src[c]; t1.raw = src[c + bd]; t2.raw = src[c + 2 * bd]; t3.raw = src[c + 3 * bd];
          grad(t0, c); grad(t1, c + bd); grad(t2, c + 2 * bd); grad(t3, c + 3 * bd);
        }
        for (; c < nvec; c += bd) {
          VT t; t.raw = src[c];
          grad(t, c);
        }
      } else {
        for (int c = threadIdx.x; c < V; c += bd) {
          float p = __expf(to_f32(lr[c]) - lse);
          if (c == tgt) p -= 1.0f;
          gr[c] = from_f32<T>(p * inv_count);
        }
      }
    }
  }
}

// ---- rows held in shared memory ------------------------------------------------------------------------------------
// Bound: HBM.  A vocabulary row (304 KB at 151936 bf16) is needed three times (maximum, sum, gradient); read twice from
// memory it cost 151 us for 1000 rows, 0.61 of the copy bandwidth counted once.  Here a cluster of up to 8 CTAs holds the
// row in its shared memory, each CTA its share by one bulk copy: one read and one write of HBM per element.  Shares of at
// most 40 KB let five CTAs of different rows sit on an SM, so that one's loads and stores run under another's arithmetic;
// only four warps work on a share, because with more of them a row's fixed costs (waits, reductions, the exchange) outweigh
// its dozen vectors per lane.  (maximum, sum) are exchanged through distributed shared memory, once per row, in rank order.
// 1000 x 151936 bf16: 129 us = 4.7 TB/s; 12 warps on 76 KB in 8 pieces 179, 7 warps on 38 KB in 2 pieces 137.  With the
// kernel that checks the targets in front, 137 us; 138 since rows of extreme values have loops of their own.
//
// Rows lie back to back and need not be whole 16-byte vectors: a row is the vectors that cover it (`mis` elements of
// misalignment at the start of the tensor, the same in input and output); the neighbours' elements in its first and last
// vector are masked on the way in and not written.
constexpr int kCeWarps = 4, kCeThreads = (kCeWarps + 1) * 32;
constexpr int kCeMaxBytes = 100 * 1024, kCeGoodBytes = 40 * 1024;

struct CeParams {
  const void* in;
  void* out;
  const int32_t* targets;
  float* nll;
  const int32_t* count;
  int64_t M;
  int V, write_grad, mis;
  // The loss itself, or null: the last CTA to finish (done counts them, from 0) sums nll in row order.
  float* loss;
  int* done;
  int* status;
};

__device__ __forceinline__ void ce_bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// Bounded like every wait of the library, with acquire at cluster scope: the data came from a peer's store.
__device__ __forceinline__ void ce_wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status) {
  const long long t0 = clock64();
  while (true) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok || *abort_flag != 0) return;
    if (clock64() - t0 > kWaitLimitCycles) { *abort_flag = 57; atomicCAS(status, 0, 57); return; }
  }
}

template <typename T>
struct CeMath;
template <>
struct CeMath<__nv_bfloat16> {
  // maximum of a vector of 8, two lanes at a time
  static __device__ __forceinline__ float vec_max(const Vec16<__nv_bfloat16>& v) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v.raw);
    const __nv_bfloat162 m = __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3]));
    return fmaxf(__low2float(m), __high2float(m));
  }
};
template <>
struct CeMath<float> {
  static __device__ __forceinline__ float vec_max(const Vec16<float>& v) {
    return fmaxf(fmaxf(v.raw.x, v.raw.y), fmaxf(v.raw.z, v.raw.w));
  }
};

template <typename T>
__global__ void __launch_bounds__(kCeThreads, 5)
cross_entropy_cluster_kernel(const CeParams p) {
  using VT = Vec16<T>;
  using Raw = decltype(VT::raw);
  constexpr int N = VT::N;
  extern __shared__ __align__(128) uint8_t ce_smem[];
  __shared__ __align__(8) uint64_t bars[2];
  __shared__ float red[2][kCeWarps];
  __shared__ __align__(8) uint64_t slot_bars[2];
  __shared__ float2 slots[2][8];   // every CTA's (maximum, sum), by row parity; the peers write theirs here
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  cg::cluster_group cl = cg::this_cluster();
  const int ctas = static_cast<int>(cl.num_blocks()), rank = static_cast<int>(cl.block_rank());
  const int64_t first = blockIdx.x / ctas, step = gridDim.x / ctas;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8, sbase = smem_u32(ce_smem);
  if (threadIdx.x == 0) {
    mbar_init(full0, 1);
    mbar_init(empty0, kCeWarps);
    for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&slot_bars[i]), ctas);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async_smem();
  }
  cl.sync();   // every CTA's barriers exist before a peer arrives on them
  grid_launch_dependents();
  grid_dependency_wait();
  const float inv_count = 1.0f / static_cast<float>(max(1, *p.count));
  const T* in = static_cast<const T*>(p.in) - p.mis;    // 16-byte boundaries
  T* out = static_cast<T*>(p.out) - p.mis;              // (not touched without write_grad)
  // this CTA's share of a row: vectors [v_begin, v_end) counted from the boundary
  auto share = [&](int64_t row, int64_t& v_begin, int& n) {
    const int64_t e0 = row * p.V + p.mis, v0 = e0 / N, v1 = (e0 + p.V + N - 1) / N;
    const int per = static_cast<int>((v1 - v0 + ctas - 1) / ctas);
    v_begin = min(v1, v0 + static_cast<int64_t>(rank) * per);
    n = static_cast<int>(min(v1, v_begin + per) - v_begin);
  };
  auto kept_row = [&](int64_t row) { const int t = p.targets[row]; return t >= 0 && t < p.V; };

  if (warp == kCeWarps) {
    // ---------------- producer ----------------
    if (lane == 0) {
      uint32_t phase = 0;
      bool ok = true;
      for (int64_t row = first; ok && row < p.M; row += step) {
        if (!kept_row(row)) continue;
        int64_t v_begin;
        int n;
        share(row, v_begin, n);
        ok = mbar_wait(empty0, phase ^ 1, abort_flag, 55, p.status);
        if (!ok) break;
        mbar_expect_tx(full0, n * 16);   // a share with nothing in it completes at once
        if (n > 0) ce_bulk_load(sbase, in + v_begin * N, n * 16, full0);
        phase ^= 1;
      }
    }
  } else {
    // ---------------- consumers ----------------
    // A wait that runs out leaves wrong results and a status code, but every CTA still meets every cluster barrier.
    constexpr int kLanes = kCeWarps * 32;
    const int tid = threadIdx.x;
    uint32_t phase = 0, slot_phase = 0;   // bit i: parity of slot barrier i's next completion
    int par = 0;
    for (int64_t row = first; row < p.M; row += step) {
      int64_t v_begin;
      int n;
      share(row, v_begin, n);
      const int64_t e0 = row * p.V + p.mis;
      const int lo = static_cast<int>(max(static_cast<int64_t>(0), e0 - v_begin * N));              // kept elements of the share
      const int hi = static_cast<int>(min(static_cast<int64_t>(n) * N, e0 + p.V - v_begin * N));
      T* orow = out + v_begin * N;
      // Whole vectors [fa, fb) take the vector loops; the elements [lo, head) and [tail, hi) in the vectors shared with the
      // neighbouring rows (none where rows are whole vectors) go to threads 0 and 1.  Masking them in the loops instead
      // cost every vector some 40 predicated instructions (185 us for 1000 rows).
      const int fa = (lo + N - 1) / N, fb = max(fa, hi / N);
      const int head = min(fa * N, hi), tail = max(fb * N, head);
      const int edge_b = tid == 0 ? lo : tid == 1 ? tail : 0, edge_e = tid == 0 ? head : tid == 1 ? hi : 0;
      if (!kept_row(row)) {
        if (rank == 0 && tid == 0) p.nll[row] = 0.0f;
        if (p.write_grad) {
          VT z;
          float f[N];
#pragma unroll
          for (int j = 0; j < N; ++j) f[j] = 0.0f;
          z.from_float(f);
          for (int vi = fa + tid; vi < fb; vi += kLanes) __stcs(reinterpret_cast<Raw*>(orow) + vi, z.raw);
          for (int e = edge_b; e < edge_e; ++e) orow[e] = from_f32<T>(0.0f);
        }
        continue;   // the same decision in every CTA of the cluster
      }
      const int tgt = static_cast<int>(e0 + p.targets[row] - v_begin * N);   // within the share, or outside it
      const Raw* srow = reinterpret_cast<const Raw*>(ce_smem);
      const T* selem = reinterpret_cast<const T*>(ce_smem);
      // pass 1: maximum
      float m = -INFINITY;
      mbar_wait(full0, phase, abort_flag, 56, p.status);
#pragma unroll 4
      for (int vi = fa + tid; vi < fb; vi += kLanes) {
        VT t;
        t.raw = srow[vi];
        m = fmaxf(m, CeMath<T>::vec_max(t));
      }
      for (int e = edge_b; e < edge_e; ++e) m = fmaxf(m, to_f32(selem[e]));
      m = warp_max(m);
      if (lane == 0) red[0][warp] = m;
      asm volatile("bar.sync 1, %0;" ::"n"(kLanes) : "memory");
      m = red[0][0];
#pragma unroll
      for (int w = 1; w < kCeWarps; ++w) m = fmaxf(m, red[0][w]);
      // pass 2: sum of 2^((x - m) log2 e), two lanes at a time
      const float2 l2 = make_float2(kLog2e, kLog2e);
      float2 s2 = make_float2(0.0f, 0.0f);
      if (!beyond_fused(m)) {
        const float nm1 = m == -INFINITY ? 0.0f : -m * kLog2e;   // a wholly masked share adds 0, or NaN if it holds one
        const float2 nm = make_float2(nm1, nm1);
#pragma unroll 4
        for (int vi = fa + tid; vi < fb; vi += kLanes) {
          VT t;
          t.raw = srow[vi];
          float f[N];
          t.to_float(f);
#pragma unroll
          for (int j = 0; j < N; j += 2) {
            const float2 a = __ffma2_rn(make_float2(f[j], f[j + 1]), l2, nm);
            s2 = __fadd2_rn(s2, make_float2(ex2_ftz(a.x), ex2_ftz(a.y)));
          }
        }
        for (int e = edge_b; e < edge_e; ++e) s2.x += ex2_ftz(fmaf(to_f32(selem[e]), kLog2e, nm.x));
      } else {
        for (int e = lo + tid; e < hi; e += kLanes) s2.x += exp_diff(to_f32(selem[e]), m);
      }
      const float sw = warp_sum(s2.x + s2.y);
      if (lane == 0) red[1][warp] = sw;
      asm volatile("bar.sync 1, %0;" ::"n"(kLanes) : "memory");
      float s = 0.0f;
#pragma unroll
      for (int w = 0; w < kCeWarps; ++w) s += red[1][w];
      if (ctas > 1) {
        // Thread q hands this CTA's pair to CTA q.  A slot is written again two rows later, when its readers have passed
        // the exchange in between.
        const uint32_t slot = smem_u32(&slots[par][rank]), bar = smem_u32(&slot_bars[par]);
        if (tid < ctas)
          asm volatile("{\n\t.reg .b32 rs, rb;\n\t"
                       "mapa.shared::cluster.u32 rs, %0, %2;\n\t"
                       "mapa.shared::cluster.u32 rb, %1, %2;\n\t"
                       "st.shared::cluster.v2.f32 [rs], {%3, %4};\n\t"
                       "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [rb];\n\t}"
                       ::"r"(slot), "r"(bar), "r"(tid), "f"(m), "f"(s) : "memory");
        ce_wait_cluster(bar, (slot_phase >> par) & 1u, abort_flag, p.status);
        slot_phase ^= 1u << par;
        m = slots[par][0].x; s = slots[par][0].y;
        for (int q = 1; q < ctas; ++q) online_combine(m, s, slots[par][q].x, slots[par][q].y);
        par ^= 1;
      }
      const float lse = m + logf(s);
      const bool diff = beyond_fused(m);   // the same in every CTA of the cluster
      if (tid == 0 && tgt >= lo && tgt < hi) p.nll[row] = diff ? (m - to_f32(selem[tgt])) + logf(s) : lse - to_f32(selem[tgt]);
      // pass 3: the gradient
      const float2 nl = make_float2(-lse * kLog2e, -lse * kLog2e), ic = make_float2(inv_count, inv_count);
      auto grad_one = [&](float x, bool is_target) { return from_f32<T>((ex2_ftz(fmaf(x, kLog2e, nl.x)) - (is_target ? 1.0f : 0.0f)) * inv_count); };
      float x_target = 0.0f;
      bool owner = false;   // this thread writes the target's vector below, and that element once more behind the loop
      if (p.write_grad && diff) {
        for (int e = lo + tid; e < hi; e += kLanes)
          orow[e] = from_f32<T>((exp_diff(to_f32(selem[e]), m) / s - (e == tgt ? 1.0f : 0.0f)) * inv_count);
      } else if (p.write_grad) {
        if (tgt >= fa * N && tgt < fb * N) {
          owner = (tgt / N - fa) % kLanes == tid;
          x_target = to_f32(selem[tgt]);
        }
        for (int e = edge_b; e < edge_e; ++e) orow[e] = grad_one(to_f32(selem[e]), e == tgt);
#pragma unroll 4
        for (int vi = fa + tid; vi < fb; vi += kLanes) {
          VT t;
          t.raw = srow[vi];
          float f[N];
          t.to_float(f);
#pragma unroll
          for (int j = 0; j < N; j += 2) {
            const float2 a = __ffma2_rn(make_float2(f[j], f[j + 1]), l2, nl);
            const float2 e = __fmul2_rn(make_float2(ex2_ftz(a.x), ex2_ftz(a.y)), ic);
            f[j] = e.x; f[j + 1] = e.y;
          }
          t.from_float(f);
          __stcs(reinterpret_cast<Raw*>(orow) + vi, t.raw);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty0);   // the next row may come in
      if (owner) orow[tgt] = grad_one(x_target, true);
      phase ^= 1;
    }
  }
  __syncwarp();
  if (*abort_flag != 0) {
    for (int k = 0; k < 200; ++k) __nanosleep(1000);   // loads in flight land before the shared memory is released
  }
  cl.sync();   // no peer still writes here
  if (p.loss != nullptr) {
    // release this CTA's nll, and let the last CTA of the grid sum all of them (a fixed order whichever CTA it is)
    __shared__ int last;
    if (threadIdx.x == 0) {
      __threadfence();
      last = atomicAdd(p.done, 1) == static_cast<int>(gridDim.x) - 1;
    }
    __syncthreads();
    if (last) {
      __threadfence();
      double* sums = reinterpret_cast<double*>(ce_smem);   // (not a static array: 1.3 KB more would cost float32 its third CTA per SM)
      double acc = 0.0;
      for (int64_t i = threadIdx.x; i < p.M; i += kCeThreads) acc += static_cast<double>(__ldcg(p.nll + i));
      sums[threadIdx.x] = acc;
      __syncthreads();
      if (threadIdx.x == 0) {
        double t = 0.0;
        for (int i = 0; i < kCeThreads; ++i) t += sums[i];
        p.loss[1] = static_cast<float>(t);
        p.loss[0] = static_cast<float>(t / static_cast<double>(max(1, *p.count)));
      }
    }
  }
}

__global__ void count_valid_kernel(const int32_t* __restrict__ targets, int64_t M, int V, int32_t* __restrict__ count) {
  __shared__ int red[32];
  int c = 0;
  grid_launch_dependents();
  grid_dependency_wait();
  targets = from_here(targets);
  for (int64_t i = threadIdx.x; i < M; i += blockDim.x) c += (targets[i] >= 0 && targets[i] < V) ? 1 : 0;
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int w = 0; w < (blockDim.x >> 5); ++w) t += red[w];
    *count = t;
  }
}

// loss[0] = sum(nll) / count, loss[1] = sum(nll); serial tree in fixed order (one block).
__global__ void reduce_nll_kernel(const float* __restrict__ nll, int64_t M, const int32_t* __restrict__ count,
                                  float* __restrict__ loss) {
  __shared__ double red[1024];
  double acc = 0.0;
  grid_launch_dependents();
  grid_dependency_wait();
  nll = from_here(nll);
  count = from_here(count);
  for (int64_t i = threadIdx.x; i < M; i += blockDim.x) acc += static_cast<double>(nll[i]);
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    loss[1] = static_cast<float>(red[0]);
    loss[0] = static_cast<float>(red[0] / static_cast<double>(max(1, *count)));
  }
}


// Targets as a caller has them (int64 or int32, possibly with an ignore index of its own) to the int32 the kernels take:
// -1 is ignored; info[0] = targets that count, info[1] = targets that are neither ignored nor in [0, V).
template <typename I>
__global__ void __launch_bounds__(1024)
prepare_targets_kernel(const I* __restrict__ targets, int32_t* __restrict__ t32, int64_t M, int64_t V, int has_ignore, int64_t ignore,
                       int32_t* __restrict__ info, int32_t* info_host) {
  __shared__ int red[2][32];
  int good = 0, bad = 0;
  grid_launch_dependents();
  grid_dependency_wait();
  targets = from_here(targets);
  for (int64_t i = threadIdx.x; i < M; i += blockDim.x) {
    int64_t t = targets[i];
    if (has_ignore && t == ignore) t = -1;
    const bool in = t >= 0 && t < V;
    good += in;
    bad += !in && t != -1;
    t32[i] = in ? static_cast<int32_t>(t) : -1;
  }
  good = __reduce_add_sync(0xffffffffu, good);
  bad = __reduce_add_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = good; red[1][threadIdx.x >> 5] = bad; }
  __syncthreads();
  if (threadIdx.x < 2) {
    int t = 0;
    for (int w = 0; w < (blockDim.x >> 5); ++w) t += red[threadIdx.x][w];
    info[threadIdx.x] = t;
    if (info_host != nullptr) info_host[threadIdx.x] = t;   // page-locked: written in place, no copy to enqueue
  }
  if (threadIdx.x == 2) info[2] = 0;   // the row kernel's count of finished CTAs
}

// Clusters of the launch `cfg` describes that the device runs at once.  The answer depends on the vocabulary through the
// CTAs' shared memory (float32, 8 CTAs a row: 25 KB at 50257 columns, 76 KB at 151936, 688 and 384 CTAs); the query
// takes microseconds, so the last few answers are kept.
template <typename T>
int resident_clusters(const cudaLaunchConfig_t& cfg, DeviceState::ResidentClusters (&kept)[4], int* count) {
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  for (const auto& k : kept)
    if (k.smem == cfg.dynamicSmemBytes) { *count = k.count; return MCB_OK; }
  int n = 0;
  MCB_CHECK_CUDA(cudaOccupancyMaxActiveClusters(&n, cross_entropy_cluster_kernel<T>, &cfg));
  for (int i = 3; i > 0; --i) kept[i] = kept[i - 1];
  kept[0].smem = cfg.dynamicSmemBytes;
  kept[0].count = *count = n > 0 ? n : 1;
  return MCB_OK;
}

// Row kernel launch: in -> out (which may be the same tensor); out is null when no gradient is wanted.
template <typename T>
int launch_rows(const void* in, void* out, const int32_t* targets, float* nll, const int32_t* count, int64_t M, int64_t V, int write_grad,
                float* loss, int* done, DeviceState* ds, cudaStream_t st) {
  constexpr int N = Vec16<T>::N;
  const uintptr_t ai = reinterpret_cast<uintptr_t>(in), ao = reinterpret_cast<uintptr_t>(out ? out : in);
  const int64_t row_vecs = (V + 2 * N - 2) / N;   // vectors that cover a row at most
  int ctas = 1;
  while (ctas < 8 && (row_vecs + ctas - 1) / ctas * 16 > kCeGoodBytes) ctas *= 2;
  const int64_t cta_vecs = (row_vecs + ctas - 1) / ctas;
  // In place (the training step, a chunk of tokens at a time) the block kernel stays, although it is 12 % slower there: the
  // step's losses and gradients keep its order of summation.
  // From 16 KB on a CTA's 128 lanes have at least eight vectors each.  Measured with the line at 1 KB, block kernel / this
  // one: 1000 rows of 2 KB 10.9 / 11.5 us, of 8 KB 16.3 / 15.3; 16000 rows of 2 KB 88 / 61 us, of 8 KB 131 / 84.  So it is
  // only few and very short rows that the block kernel is quicker with.
  if (in != out && row_vecs * 16 >= 16 * 1024 && cta_vecs * 16 <= kCeMaxBytes && ((ai ^ ao) & 15u) == 0 && ai % sizeof(T) == 0) {
    CeParams p;
    p.in = in; p.out = out; p.targets = targets; p.nll = nll; p.count = count;
    p.M = M; p.V = static_cast<int>(V); p.write_grad = write_grad; p.mis = static_cast<int>((ai & 15u) / sizeof(T));
    p.loss = loss; p.done = done;
    p.status = ds->status_word;
    const size_t smem = static_cast<size_t>(cta_vecs) * 16;
    bool& ready = ds->ce_smem[sizeof(T) == 4];
    if (!ready) {
      MCB_CHECK_CUDA(cudaFuncSetAttribute(cross_entropy_cluster_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kCeMaxBytes));
      MCB_CHECK_CUDA(cudaFuncSetAttribute(cross_entropy_cluster_kernel<T>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                          cudaSharedmemCarveoutMaxShared));
      ready = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(ctas)); cfg.blockDim = dim3(kCeThreads); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(ctas); attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    // as many clusters as are resident together: a later one would start its share of the rows when the others are done
    int resident = 0;
    if (int rc = resident_clusters<T>(cfg, ds->ce_clusters[sizeof(T) == 4][ctas], &resident)) return rc;
    cfg.gridDim = dim3(static_cast<unsigned>((M < resident ? M : resident) * ctas));
    if (chained_launch()) cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, cross_entropy_cluster_kernel<T>, p);
    if (e != cudaSuccess) return cuda_fail(e, "cross_entropy_cluster_kernel launch");
    MCB_CHECK_LAUNCH("cross_entropy_cluster_kernel");
    return MCB_OK;   // (the last CTA has summed the loss, if that was asked for)
  }
  // eight blocks of 256 threads per SM, fewer when there are fewer rows
  const int64_t blocks = static_cast<int64_t>(ds->sm_count) * 8;
  MCB_CHECK_CUDA(launch_kernel(cross_entropy_kernel<T>, dim3(static_cast<unsigned>(M < blocks ? M : blocks)), dim3(256), 0, st, chained_launch(),
                               static_cast<const T*>(in), static_cast<T*>(out), targets, nll, count, M, static_cast<int>(V), write_grad));
  MCB_CHECK_LAUNCH("cross_entropy");
  if (loss != nullptr) {
    MCB_CHECK_CUDA(launch_kernel(reduce_nll_kernel, dim3(1), dim3(1024), 0, st, chained_launch(), nll, M, count, loss));
    MCB_CHECK_LAUNCH("reduce_nll");
  }
  return MCB_OK;
}
int launch_rows(const void* in, void* out, const int32_t* targets, float* nll, const int32_t* count, int64_t M, int64_t V, int write_grad,
                int dtype, float* loss, int* done, DeviceState* ds, cudaStream_t st) {
  if (dtype == MCB_F32) return launch_rows<float>(in, out, targets, nll, count, M, V, write_grad, loss, done, ds, st);
  if (dtype == MCB_BF16) return launch_rows<__nv_bfloat16>(in, out, targets, nll, count, M, V, write_grad, loss, done, ds, st);
  return fail(MCB_ERR_UNSUPPORTED, "dtype %d", dtype);
}

}  // namespace
}  // namespace mcb

using namespace mcb;

extern "C" int mcb_cross_entropy(void* logits, const int32_t* targets, float* nll, int32_t* count, float* loss,
                                 int64_t M, int64_t V, int write_grad, int dtype, void* stream) {
  MCB_NVTX_RANGE("mcb_cross_entropy");
  if (!logits || !targets || !nll || !count || !loss) return fail(MCB_ERR_NULL, "cross_entropy: null pointer");
  if (M <= 0 || V <= 0 || M > 0x7fffffff || V > 0x7fffffff) return fail(MCB_ERR_SHAPE, "cross_entropy: bad shape");
  DeviceState* ds = current_device_state();
  if (!ds) return MCB_ERR_NOT_INIT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  MCB_CHECK_CUDA(launch_kernel(count_valid_kernel, dim3(1), dim3(1024), 0, st, chained_launch(), targets, M, (int)V, count));
  MCB_CHECK_LAUNCH("count_valid");
  if (int rc = launch_rows(logits, logits, targets, nll, count, M, V, write_grad, dtype, nullptr, nullptr, ds, st)) return rc;
  MCB_CHECK_CUDA(launch_kernel(reduce_nll_kernel, dim3(1), dim3(1024), 0, st, chained_launch(), nll, M, count, loss));
  MCB_CHECK_LAUNCH("reduce_nll");
  return MCB_OK;
}

// The three stages of mcb_cross_entropy as separate calls, so that the logits can be produced, consumed and
// discarded a chunk of tokens at a time (the [tokens, vocabulary] matrix of the whole batch never exists).
extern "C" int mcb_cross_entropy_count(const int32_t* targets, int32_t* count, int64_t M, int64_t V, void* stream) {
  MCB_NVTX_RANGE("mcb_cross_entropy_count");
  if (!targets || !count) return fail(MCB_ERR_NULL, "cross_entropy_count: null pointer");
  if (M <= 0 || V <= 0 || M > 0x7fffffff || V > 0x7fffffff) return fail(MCB_ERR_SHAPE, "cross_entropy_count: bad shape");
  if (!current_device_state()) return MCB_ERR_NOT_INIT;
  MCB_CHECK_CUDA(launch_kernel(count_valid_kernel, dim3(1), dim3(1024), 0, static_cast<cudaStream_t>(stream), chained_launch(), targets, M, (int)V, count));
  MCB_CHECK_LAUNCH("count_valid");
  return MCB_OK;
}

extern "C" int mcb_cross_entropy_chunk(void* logits, const int32_t* targets, float* nll, const int32_t* count, int64_t rows,
                                       int64_t V, int write_grad, int dtype, void* stream) {
  MCB_NVTX_RANGE("mcb_cross_entropy_chunk");
  if (!logits || !targets || !nll || !count) return fail(MCB_ERR_NULL, "cross_entropy_chunk: null pointer");
  if (rows <= 0 || V <= 0 || rows > 0x7fffffff || V > 0x7fffffff) return fail(MCB_ERR_SHAPE, "cross_entropy_chunk: bad shape");
  DeviceState* ds = current_device_state();
  if (!ds) return MCB_ERR_NOT_INIT;
  return launch_rows(logits, logits, targets, nll, count, rows, V, write_grad, dtype, nullptr, nullptr, ds, static_cast<cudaStream_t>(stream));
}

extern "C" int mcb_cross_entropy_finish(const float* nll, const int32_t* count, float* loss, int64_t M, void* stream) {
  MCB_NVTX_RANGE("mcb_cross_entropy_finish");
  if (!nll || !count || !loss) return fail(MCB_ERR_NULL, "cross_entropy_finish: null pointer");
  if (M <= 0 || M > 0x7fffffff) return fail(MCB_ERR_SHAPE, "cross_entropy_finish: bad shape");
  if (!current_device_state()) return MCB_ERR_NOT_INIT;
  MCB_CHECK_CUDA(launch_kernel(reduce_nll_kernel, dim3(1), dim3(1024), 0, static_cast<cudaStream_t>(stream), chained_launch(), nll, M, count, loss));
  MCB_CHECK_LAUNCH("reduce_nll");
  return MCB_OK;
}


extern "C" int mcb_cross_entropy_out(const void* logits, void* dlogits, const void* targets, int target_bytes, int has_ignore,
                                     int64_t ignore_index, int32_t* t32, int32_t* info, int32_t* info_host, void* info_event,
                                     float* nll, float* loss, int64_t M, int64_t V, int dtype, void* stream) {
  MCB_NVTX_RANGE("mcb_cross_entropy_out");
  if (!logits || !targets || !t32 || !info || !nll || !loss) return fail(MCB_ERR_NULL, "cross_entropy_out: null pointer");
  if (M <= 0 || V <= 0 || M > 0x7fffffff || V > 0x7fffffff) return fail(MCB_ERR_SHAPE, "cross_entropy_out: bad shape");
  if (target_bytes != 4 && target_bytes != 8) return fail(MCB_ERR_UNSUPPORTED, "cross_entropy_out: targets of %d bytes", target_bytes);
  DeviceState* ds = current_device_state();
  if (!ds) return MCB_ERR_NOT_INIT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (target_bytes == 8) {
    MCB_CHECK_CUDA(launch_kernel(prepare_targets_kernel<int64_t>, dim3(1), dim3(1024), 0, st, chained_launch(), static_cast<const int64_t*>(targets), t32, M, V,
                                 has_ignore, ignore_index, info, info_host));
  } else {
    MCB_CHECK_CUDA(launch_kernel(prepare_targets_kernel<int32_t>, dim3(1), dim3(1024), 0, st, chained_launch(), static_cast<const int32_t*>(targets), t32, M, V,
                                 has_ignore, ignore_index, info, info_host));
  }
  MCB_CHECK_LAUNCH("prepare_targets");
  if (info_event != nullptr) MCB_CHECK_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(info_event), st));
  const bool grad = dlogits != nullptr;
  if (int rc = launch_rows(logits, dlogits, t32, nll, info, M, V, grad ? 1 : 0, dtype, loss, info + 2, ds, st)) return rc;
  return MCB_OK;
}
