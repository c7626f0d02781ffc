// The element-wise "frame" of the Qwen-shaped training step around the LoRA hot path: embedding
// gather, rotary embedding with the head-major re-layout attention wants, SwiGLU and residual add.  All
// are HBM-bound streaming kernels; float32 or bfloat16 storage, float32 arithmetic.
#include "common.cuh"

namespace mcb {
namespace {

// ---- embedding (candle_nn::embedding, src/models/qwen.rs:189; gather of table rows) -----------------
template <typename T>
__global__ void embedding_fwd_kernel(const int32_t* __restrict__ ids, const T* __restrict__ table, T* __restrict__ out,
                                     int64_t M, int H, int vocab) {
  const int64_t row = blockIdx.x;
  grid_launch_dependents();
  grid_dependency_wait();
  ids = from_here(ids);
  table = from_here(table);
  if (row >= M) return;
  int32_t id = ids[row];
  if (id < 0 || id >= vocab) id = 0;  // ids are validated on the host; never read out of range
  const T* src = table + static_cast<int64_t>(id) * H;
  T* dst = out + row * H;
  if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0 && (H * sizeof(T)) % 16 == 0) {
    const int nv = H * sizeof(T) / 16;
    for (int i = threadIdx.x; i < nv; i += blockDim.x)
      reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
  } else {
    for (int i = threadIdx.x; i < H; i += blockDim.x) dst[i] = src[i];
  }
}

// ---- rotary embedding + [B,S,H,d] -> [B,H,S,d] (src/models/transformer.rs:47-120,255-257) ----------------
// Half-split rotation: (x1, x2) -> (x1 cos - x2 sin, x1 sin + x2 cos), angle = pos * theta^(-2i/d).
// inverse != 0 applies the transposed rotation and the inverse layout change (the backward pass).
// rotate == 0 only changes the layout (used for V).
template <typename T>
__global__ void rope_relayout_kernel(const T* __restrict__ src, T* __restrict__ dst, int B, int S, int H, int d,
                                     float theta, int rotate, int inverse, int64_t pitch, int64_t offset) {
  // One thread owns a 16-byte chunk of the first half of a head (and the matching chunk of the second
  // half) at one (batch, position), computes its sines and cosines once, and walks over the heads.
  using V = Vec16<T>;
  constexpr int N = V::N;
  const int half = d / 2;
  const int chunks = half / N;  // host guarantees half % N == 0
  const int64_t total = static_cast<int64_t>(B) * S * chunks;
  for (int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
       idx += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(idx % chunks);
    const int64_t bs = idx / chunks;
    const int s = static_cast<int>(bs % S);
    const int b = static_cast<int>(bs / S);
    float cs[N], sn[N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
      if (rotate) {
        // 1 / theta^(2i/d) as in the reference's table (float32 powf), angle = position * inv_freq
        const int i = c * N + j;
        const float inv_freq = 1.0f / powf(theta, static_cast<float>(2 * i) / static_cast<float>(d));
        sincosf(static_cast<float>(s) * inv_freq, &sn[j], &cs[j]);
        if (inverse) sn[j] = -sn[j];
      } else {
        cs[j] = 1.0f; sn[j] = 0.0f;
      }
    }
    for (int h = 0; h < H; ++h) {
      // [B,S,H,d] side: token rows `pitch` elements apart, the heads starting `offset` elements into a row
      const int64_t bshd = (static_cast<int64_t>(b) * S + s) * pitch + offset + static_cast<int64_t>(h) * d;
      const int64_t bhsd = ((static_cast<int64_t>(b) * H + h) * S + s) * d;   // [B,H,S,d]
      const int64_t in = inverse ? bhsd : bshd, out = inverse ? bshd : bhsd;
      V a, bb;
      a.raw = *reinterpret_cast<const decltype(a.raw)*>(src + in + c * N);
      bb.raw = *reinterpret_cast<const decltype(bb.raw)*>(src + in + half + c * N);
      float x1[N], x2[N], o1[N], o2[N];
      a.to_float(x1); bb.to_float(x2);
#pragma unroll
      for (int j = 0; j < N; ++j) {
        o1[j] = x1[j] * cs[j] - x2[j] * sn[j];
        o2[j] = x1[j] * sn[j] + x2[j] * cs[j];
      }
      a.from_float(o1); bb.from_float(o2);
      *reinterpret_cast<decltype(a.raw)*>(dst + out + c * N) = a.raw;
      *reinterpret_cast<decltype(bb.raw)*>(dst + out + half + c * N) = bb.raw;
    }
  }
}

// The same for the query, key and value heads of a fused q/k/v row in one launch: the sines and cosines of a
// (position, chunk) are computed once and used for the rotated segments (q and k); v is only re-laid out.  grid.y shares
// the heads: at 333 tokens one thread per (token, chunk) is 11 blocks, each thread working through 18 heads one after the
// other (10.4 us); with the heads spread over as many blocks as fill the chip the launch takes 6.3 us, although
// every share computes the sines again.  Many tokens keep one share: 32768 x 18 heads move 151 MB and are HBM-bound.
template <typename T>
struct RopeSegment {
  T* head_major;    // [B, H, S, d]
  int H;
  int64_t offset;   // first column of the segment's heads in a token row
  int rotate;
};
template <typename T>
__global__ void rope_relayout_qkv_kernel(T* __restrict__ fused, RopeSegment<T> s0, RopeSegment<T> s1, RopeSegment<T> s2, int B, int S,
                                         int d, float theta, int inverse, int64_t pitch) {
  using V = Vec16<T>;
  constexpr int N = V::N;
  grid_launch_dependents();
  const int half = d / 2;
  const int chunks = half / N;
  const int64_t total = static_cast<int64_t>(B) * S * chunks;
  const int heads = s0.H + s1.H + s2.H;
  const int h_begin = static_cast<int>(static_cast<int64_t>(heads) * blockIdx.y / gridDim.y);
  const int h_end = static_cast<int>(static_cast<int64_t>(heads) * (blockIdx.y + 1) / gridDim.y);
  const int64_t first_idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  float cs[N], sn[N];
  auto angles = [&](int64_t idx) {
    const int c = static_cast<int>(idx % chunks), s = static_cast<int>(idx / chunks % S);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const int i = c * N + j;
      const float inv_freq = 1.0f / powf(theta, static_cast<float>(2 * i) / static_cast<float>(d));
      sincosf(static_cast<float>(s) * inv_freq, &sn[j], &cs[j]);
      if (inverse) sn[j] = -sn[j];
    }
  };
  // The first (with few tokens the only) sines and cosines, some 1500 instructions, under the tail of the kernel before.
  if (first_idx < total) angles(first_idx);
  grid_dependency_wait();
  fused = from_here(fused);
  s0.head_major = from_here(s0.head_major);
  s1.head_major = from_here(s1.head_major);
  s2.head_major = from_here(s2.head_major);
  for (int64_t idx = first_idx; idx < total; idx += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(idx % chunks);
    const int64_t bs = idx / chunks;
    const int s = static_cast<int>(bs % S);
    const int b = static_cast<int>(bs / S);
    if (idx != first_idx) angles(idx);
#pragma unroll
    for (int g = 0; g < 3; ++g) {
      const RopeSegment<T>& sg = g == 0 ? s0 : g == 1 ? s1 : s2;
      const int first = g == 0 ? 0 : g == 1 ? s0.H : s0.H + s1.H;   // the segment's part of heads [h_begin, h_end)
      for (int h = max(0, h_begin - first); h < min(sg.H, h_end - first); ++h) {
        const int64_t tok = (static_cast<int64_t>(b) * S + s) * pitch + sg.offset + static_cast<int64_t>(h) * d;
        const int64_t hm = ((static_cast<int64_t>(b) * sg.H + h) * S + s) * d;
        const T* in = inverse ? sg.head_major + hm : fused + tok;
        T* out = inverse ? fused + tok : sg.head_major + hm;
        V a, bb;
        a.raw = *reinterpret_cast<const decltype(a.raw)*>(in + c * N);
        bb.raw = *reinterpret_cast<const decltype(bb.raw)*>(in + half + c * N);
        if (sg.rotate) {
          float x1[N], x2[N], o1[N], o2[N];
          a.to_float(x1); bb.to_float(x2);
#pragma unroll
          for (int j = 0; j < N; ++j) {
            o1[j] = x1[j] * cs[j] - x2[j] * sn[j];
            o2[j] = x1[j] * sn[j] + x2[j] * cs[j];
          }
          a.from_float(o1); bb.from_float(o2);
        }
        *reinterpret_cast<decltype(a.raw)*>(out + c * N) = a.raw;
        *reinterpret_cast<decltype(bb.raw)*>(out + half + c * N) = bb.raw;
      }
    }
  }
}

// Scalar variant for head sizes whose half is not a multiple of the vector width.
template <typename T>
__global__ void rope_relayout_scalar_kernel(const T* __restrict__ src, T* __restrict__ dst, int B, int S, int H, int d,
                                            float theta, int rotate, int inverse, int64_t pitch, int64_t offset) {
  const int half = d / 2;
  const int64_t total = static_cast<int64_t>(B) * S * H * half;
  for (int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
       idx += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int i = static_cast<int>(idx % half);
    int64_t t = idx / half;
    const int h = static_cast<int>(t % H); t /= H;
    const int s = static_cast<int>(t % S);
    const int b = static_cast<int>(t / S);
    const int64_t bshd = (static_cast<int64_t>(b) * S + s) * pitch + offset + static_cast<int64_t>(h) * d;
    const int64_t bhsd = ((static_cast<int64_t>(b) * H + h) * S + s) * d;
    const int64_t in = inverse ? bhsd : bshd, out = inverse ? bshd : bhsd;
    const float x1 = to_f32(src[in + i]), x2 = to_f32(src[in + half + i]);
    float o1 = x1, o2 = x2;
    if (rotate) {
      const float inv_freq = 1.0f / powf(theta, static_cast<float>(2 * i) / static_cast<float>(d));
      float sn, cs;
      sincosf(static_cast<float>(s) * inv_freq, &sn, &cs);
      if (inverse) sn = -sn;
      o1 = x1 * cs - x2 * sn;
      o2 = x1 * sn + x2 * cs;
    }
    dst[out + i] = from_f32<T>(o1);
    dst[out + half + i] = from_f32<T>(o2);
  }
}

// ---- SwiGLU (src/models/transformer.rs:389-395) ---------------------------------------------------------
template <typename T>
__global__ void swiglu_fwd_kernel(const T* __restrict__ gate, const T* __restrict__ up, T* __restrict__ out, int64_t n) {
  using V = Vec16<T>;
  constexpr int N = V::N;
  grid_launch_dependents();
  grid_dependency_wait();
  gate = from_here(gate);
  up = from_here(up);
  out = from_here(out);
  const int64_t nv = n / N;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < nv;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    V g, u, o;
    g.raw = reinterpret_cast<const decltype(g.raw)*>(gate)[i];
    u.raw = reinterpret_cast<const decltype(u.raw)*>(up)[i];
    float gf[N], uf[N], of[N];
    g.to_float(gf); u.to_float(uf);
#pragma unroll
    for (int j = 0; j < N; ++j) of[j] = gf[j] / (1.0f + __expf(-gf[j])) * uf[j];
    o.from_float(of);
    reinterpret_cast<decltype(o.raw)*>(out)[i] = o.raw;
  }
}

// d_gate = d_out * up * sig(g) * (1 + g (1 - sig(g))),  d_up = d_out * silu(g).  In place on gate/up allowed.
template <typename T>
__global__ void swiglu_bwd_kernel(const T* __restrict__ gate, const T* __restrict__ up, const T* __restrict__ dout,
                                  T* __restrict__ dgate, T* __restrict__ dup, int64_t n) {
  using V = Vec16<T>;
  constexpr int N = V::N;
  grid_launch_dependents();
  grid_dependency_wait();
  gate = from_here(gate);
  up = from_here(up);
  dout = from_here(dout);
  dgate = from_here(dgate);
  dup = from_here(dup);
  const int64_t nv = n / N;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < nv;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    V g, u, d, og, ou;
    g.raw = reinterpret_cast<const decltype(g.raw)*>(gate)[i];
    u.raw = reinterpret_cast<const decltype(u.raw)*>(up)[i];
    d.raw = reinterpret_cast<const decltype(d.raw)*>(dout)[i];
    float gf[N], uf[N], df[N], a[N], b[N];
    g.to_float(gf); u.to_float(uf); d.to_float(df);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const float sg = 1.0f / (1.0f + __expf(-gf[j]));
      a[j] = df[j] * uf[j] * sg * (1.0f + gf[j] * (1.0f - sg));
      b[j] = df[j] * gf[j] * sg;
    }
    og.from_float(a); ou.from_float(b);
    reinterpret_cast<decltype(og.raw)*>(dgate)[i] = og.raw;
    reinterpret_cast<decltype(ou.raw)*>(dup)[i] = ou.raw;
  }
}

template <typename T>
__global__ void add_kernel(const T* __restrict__ a, const T* __restrict__ b, T* __restrict__ out, int64_t n) {
  using V = Vec16<T>;
  constexpr int N = V::N;
  const int64_t nv = n / N;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < nv;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    V x, y, o;
    x.raw = reinterpret_cast<const decltype(x.raw)*>(a)[i];
    y.raw = reinterpret_cast<const decltype(y.raw)*>(b)[i];
    float xf[N], yf[N];
    x.to_float(xf); y.to_float(yf);
#pragma unroll
    for (int j = 0; j < N; ++j) xf[j] += yf[j];
    o.from_float(xf);
    reinterpret_cast<decltype(o.raw)*>(out)[i] = o.raw;
  }
}

template <typename T>
__global__ void add_scalar_kernel(const T* __restrict__ a, const T* __restrict__ b, T* __restrict__ out, int64_t n) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    out[i] = from_f32<T>(to_f32(a[i]) + to_f32(b[i]));
}

// out = a * b (mode 0) or out = a * scalar (mode 1): Operation::Mul / Operation::MulScalar of the lazy graph
// (src/graph/executor.rs:97-120).
template <typename T>
__global__ void mul_kernel(const T* __restrict__ a, const T* __restrict__ b, T* __restrict__ out, int64_t n, float scalar,
                           int mode) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    out[i] = from_f32<T>(to_f32(a[i]) * (mode == 0 ? to_f32(b[i]) : scalar));
}

// out[n,k] = W[n,k] + scale * sum_j A[k,j] B[j,n]   (LoRAAdapter::merge_weights, src/training/adapter.rs:315-354:
// base + scaling * (A B)^T for a base weight stored [out, in]).  One thread per 4 consecutive k of one n; A rows
// and the B column are read through the read-only cache, the product is accumulated in float32.
template <typename T>
__global__ void merge_weights_kernel(const T* __restrict__ W, const float* __restrict__ A, const float* __restrict__ B,
                                     T* __restrict__ out, int K, int N, int r, float scale) {
  const int64_t total = static_cast<int64_t>(N) * ((K + 3) / 4);
  for (int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
       idx += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int kq = static_cast<int>(idx % ((K + 3) / 4));
    const int n = static_cast<int>(idx / ((K + 3) / 4));
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int j = 0; j < r; ++j) {
      const float b = __ldg(B + static_cast<int64_t>(j) * N + n);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int k = kq * 4 + e;
        if (k < K) acc[e] = fmaf(__ldg(A + static_cast<int64_t>(k) * r + j), b, acc[e]);
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int k = kq * 4 + e;
      if (k < K) {
        const int64_t o = static_cast<int64_t>(n) * K + k;
        out[o] = from_f32<T>(to_f32(W[o]) + scale * acc[e]);
      }
    }
  }
}

int grid_for(int64_t work_items, int threads, int sm_count) {
  int64_t g = (work_items + threads - 1) / threads;
  const int64_t cap = static_cast<int64_t>(sm_count) * 16;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return static_cast<int>(g);
}

}  // namespace
}  // namespace mcb

using namespace mcb;

#define MCB_DTYPE_SWITCH(dtype, CALL)                                    \
  if ((dtype) == MCB_F32) { using T = float; CALL; }                     \
  else if ((dtype) == MCB_BF16) { using T = __nv_bfloat16; CALL; }       \
  else return fail(MCB_ERR_UNSUPPORTED, "dtype %d", (dtype));

extern "C" int mcb_embedding_fwd(const int32_t* ids, const void* table, void* out, int64_t M, int64_t H, int64_t vocab,
                                 int dtype, void* stream) {
  MCB_NVTX_RANGE("mcb_embedding_fwd");
  if (!ids || !table || !out) return fail(MCB_ERR_NULL, "embedding_fwd: null pointer");
  if (M <= 0 || H <= 0 || vocab <= 0 || M > 0x7fffffff) return fail(MCB_ERR_SHAPE, "embedding_fwd: bad shape");
  if (!current_device_state()) return MCB_ERR_NOT_INIT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t le = cudaSuccess;
  MCB_DTYPE_SWITCH(dtype, (le = launch_kernel(embedding_fwd_kernel<T>, dim3((unsigned)M), dim3(128), 0, st, chained_launch(), ids, (const T*)table, (T*)out, M, (int)H, (int)vocab)));
  if (le != cudaSuccess) return cuda_fail(le, "embedding_fwd launch");
  MCB_CHECK_LAUNCH("embedding_fwd");
  return MCB_OK;
}

extern "C" int mcb_rope_relayout_qkv(void* fused, void* q, void* k, void* v, int64_t B, int64_t S, int64_t Hq, int64_t Hk, int64_t d,
                                     float theta, int inverse, int64_t token_pitch, int dtype, void* stream) {
  MCB_NVTX_RANGE("mcb_rope_relayout_qkv");
  if (!fused || !q || !k || !v) return fail(MCB_ERR_NULL, "rope_relayout_qkv: null pointer");
  if (B <= 0 || S <= 0 || Hq <= 0 || Hk <= 0 || d <= 0 || d % 2 != 0)
    return fail(MCB_ERR_SHAPE, "rope_relayout_qkv: bad shape (head_dim must be even)");
  const int64_t width = (Hq + 2 * Hk) * d;
  if (token_pitch == 0) token_pitch = width;
  if (token_pitch < width)
    return fail(MCB_ERR_SHAPE, "rope_relayout_qkv: %lld + 2 x %lld heads of %lld do not fit a row of %lld", (long long)Hq, (long long)Hk,
                (long long)d, (long long)token_pitch);
  DeviceState* ds = current_device_state();
  if (!ds) return MCB_ERR_NOT_INIT;
  const int64_t half = d / 2;
  const int vec_n = dtype == MCB_F32 ? 4 : 8;
  if (dtype != MCB_F32 && dtype != MCB_BF16) return fail(MCB_ERR_UNSUPPORTED, "rope_relayout_qkv: dtype %d", dtype);
  if (!(half % vec_n == 0 && aligned16(fused) && aligned16(q) && aligned16(k) && aligned16(v) && token_pitch % vec_n == 0)) {
    // shapes the vector kernel does not take: the three single calls (same arithmetic)
    const void* src[3] = {inverse ? q : fused, inverse ? k : fused, inverse ? v : fused};
    void* dst[3] = {inverse ? fused : q, inverse ? fused : k, inverse ? fused : v};
    const int64_t H[3] = {Hq, Hk, Hk}, off[3] = {0, Hq * d, (Hq + Hk) * d};
    for (int g = 0; g < 3; ++g)
      if (int rc = mcb_rope_relayout_ex(src[g], dst[g], B, S, H[g], d, theta, g < 2 ? 1 : 0, inverse, token_pitch, off[g], dtype, stream))
        return rc;
    return MCB_OK;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t heads = Hq + 2 * Hk;
  const int blocks = grid_for(B * S * (half / vec_n), 128, ds->sm_count);
  int64_t shares = (4 * static_cast<int64_t>(ds->sm_count) + blocks - 1) / blocks;   // four blocks per SM
  if (shares > heads) shares = heads;
  if (shares > 65535) shares = 65535;
  const dim3 grid(static_cast<unsigned>(blocks), static_cast<unsigned>(shares));
  MCB_DTYPE_SWITCH(dtype, ({
    RopeSegment<T> s0{static_cast<T*>(q), static_cast<int>(Hq), 0, 1};
    RopeSegment<T> s1{static_cast<T*>(k), static_cast<int>(Hk), Hq * d, 1};
    RopeSegment<T> s2{static_cast<T*>(v), static_cast<int>(Hk), (Hq + Hk) * d, 0};
    const cudaError_t le = launch_kernel(rope_relayout_qkv_kernel<T>, grid, dim3(128), 0, st, chained_launch(), static_cast<T*>(fused), s0, s1, s2,
                                         (int)B, (int)S, (int)d, theta, inverse, token_pitch);
    if (le != cudaSuccess) return cuda_fail(le, "rope_relayout_qkv launch");
  }));
  MCB_CHECK_LAUNCH("rope_relayout_qkv");
  return MCB_OK;
}

extern "C" int mcb_rope_relayout_ex(const void* src, void* dst, int64_t B, int64_t S, int64_t H, int64_t d, float theta,
                                    int rotate, int inverse, int64_t token_pitch, int64_t col_offset, int dtype, void* stream) {
  MCB_NVTX_RANGE("mcb_rope_relayout");
  if (!src || !dst) return fail(MCB_ERR_NULL, "rope_relayout: null pointer");
  if (B <= 0 || S <= 0 || H <= 0 || d <= 0 || d % 2 != 0) return fail(MCB_ERR_SHAPE, "rope_relayout: bad shape (head_dim must be even)");
  if (token_pitch == 0) token_pitch = H * d;
  if (col_offset < 0 || col_offset + H * d > token_pitch)
    return fail(MCB_ERR_SHAPE, "rope_relayout: %lld heads x %lld at column %lld do not fit a row of %lld", (long long)H, (long long)d,
                (long long)col_offset, (long long)token_pitch);
  DeviceState* ds = current_device_state();
  if (!ds) return MCB_ERR_NOT_INIT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t half = d / 2;
  const int vec_n = dtype == MCB_F32 ? 4 : 8;
  if (half % vec_n == 0 && aligned16(src) && aligned16(dst) && token_pitch % vec_n == 0 && col_offset % vec_n == 0) {
    const int grid = grid_for(B * S * (half / vec_n), 128, ds->sm_count);
    MCB_DTYPE_SWITCH(dtype, (rope_relayout_kernel<T><<<grid, 128, 0, st>>>((const T*)src, (T*)dst, (int)B, (int)S, (int)H, (int)d, theta, rotate, inverse, token_pitch, col_offset)));
  } else {
    const int grid = grid_for(B * S * H * half, 256, ds->sm_count);
    MCB_DTYPE_SWITCH(dtype, (rope_relayout_scalar_kernel<T><<<grid, 256, 0, st>>>((const T*)src, (T*)dst, (int)B, (int)S, (int)H, (int)d, theta, rotate, inverse, token_pitch, col_offset)));
  }
  MCB_CHECK_LAUNCH("rope_relayout");
  return MCB_OK;
}

extern "C" int mcb_rope_relayout(const void* src, void* dst, int64_t B, int64_t S, int64_t H, int64_t d, float theta,
                                 int rotate, int inverse, int dtype, void* stream) {
  return mcb_rope_relayout_ex(src, dst, B, S, H, d, theta, rotate, inverse, 0, 0, dtype, stream);
}

extern "C" int mcb_swiglu_fwd(const void* gate, const void* up, void* out, int64_t n, int dtype, void* stream) {
  MCB_NVTX_RANGE("mcb_swiglu_fwd");
  if (!gate || !up || !out) return fail(MCB_ERR_NULL, "swiglu_fwd: null pointer");
  if (n <= 0 || n % 8 != 0) return fail(MCB_ERR_SHAPE, "swiglu_fwd: element count must be a positive multiple of 8");
  if (!aligned16(gate) || !aligned16(up) || !aligned16(out)) return fail(MCB_ERR_ALIGN, "swiglu_fwd: 16-byte alignment");
  DeviceState* ds = current_device_state();
  if (!ds) return MCB_ERR_NOT_INIT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = grid_for(n / 4, 256, ds->sm_count);
  cudaError_t le = cudaSuccess;
  MCB_DTYPE_SWITCH(dtype, (le = launch_kernel(swiglu_fwd_kernel<T>, dim3(grid), dim3(256), 0, st, chained_launch(), (const T*)gate, (const T*)up, (T*)out, n)));
  if (le != cudaSuccess) return cuda_fail(le, "swiglu_fwd launch");
  MCB_CHECK_LAUNCH("swiglu_fwd");
  return MCB_OK;
}

extern "C" int mcb_swiglu_bwd(const void* gate, const void* up, const void* dout, void* dgate, void* dup, int64_t n,
                              int dtype, void* stream) {
  MCB_NVTX_RANGE("mcb_swiglu_bwd");
  if (!gate || !up || !dout || !dgate || !dup) return fail(MCB_ERR_NULL, "swiglu_bwd: null pointer");
  if (n <= 0 || n % 8 != 0) return fail(MCB_ERR_SHAPE, "swiglu_bwd: element count must be a positive multiple of 8");
  if (!aligned16(gate) || !aligned16(up) || !aligned16(dout) || !aligned16(dgate) || !aligned16(dup))
    return fail(MCB_ERR_ALIGN, "swiglu_bwd: 16-byte alignment");
  DeviceState* ds = current_device_state();
  if (!ds) return MCB_ERR_NOT_INIT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = grid_for(n / 4, 256, ds->sm_count);
  cudaError_t le = cudaSuccess;
  MCB_DTYPE_SWITCH(dtype, (le = launch_kernel(swiglu_bwd_kernel<T>, dim3(grid), dim3(256), 0, st, chained_launch(), (const T*)gate, (const T*)up, (const T*)dout, (T*)dgate, (T*)dup, n)));
  if (le != cudaSuccess) return cuda_fail(le, "swiglu_bwd launch");
  MCB_CHECK_LAUNCH("swiglu_bwd");
  return MCB_OK;
}

extern "C" int mcb_add(const void* a, const void* b, void* out, int64_t n, int dtype, void* stream) {
  MCB_NVTX_RANGE("mcb_add");
  if (!a || !b || !out) return fail(MCB_ERR_NULL, "add: null pointer");
  if (n <= 0) return fail(MCB_ERR_SHAPE, "add: element count must be positive");
  DeviceState* ds = current_device_state();
  if (!ds) return MCB_ERR_NOT_INIT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = grid_for(n / 4 + 1, 256, ds->sm_count);
  if (n % 8 != 0 || !aligned16(a) || !aligned16(b) || !aligned16(out)) {
    MCB_DTYPE_SWITCH(dtype, (add_scalar_kernel<T><<<grid, 256, 0, st>>>((const T*)a, (const T*)b, (T*)out, n)));
  } else {
    MCB_DTYPE_SWITCH(dtype, (add_kernel<T><<<grid, 256, 0, st>>>((const T*)a, (const T*)b, (T*)out, n)));
  }
  MCB_CHECK_LAUNCH("add");
  return MCB_OK;
}

extern "C" int mcb_mul(const void* a, const void* b, void* out, int64_t n, int dtype, void* stream) {
  MCB_NVTX_RANGE("mcb_mul");
  if (!a || !b || !out) return fail(MCB_ERR_NULL, "mul: null pointer");
  if (n <= 0) return fail(MCB_ERR_SHAPE, "mul: element count must be positive");
  DeviceState* ds = current_device_state();
  if (!ds) return MCB_ERR_NOT_INIT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = grid_for(n, 256, ds->sm_count);
  MCB_DTYPE_SWITCH(dtype, (mul_kernel<T><<<grid, 256, 0, st>>>((const T*)a, (const T*)b, (T*)out, n, 0.0f, 0)));
  MCB_CHECK_LAUNCH("mul");
  return MCB_OK;
}

// Inverted dropout with a counter-based generator: element i of the call is kept when the 24 high bits of
// splitmix64(seed, offset + i), read as a fraction of one, are >= p.  The mask depends on (seed, offset + i) only,
// so the same call on the upstream gradient is the backward pass, whatever the launch shape.
__device__ __forceinline__ bool dropout_keep(uint64_t seed, uint64_t index, float p) {
  uint64_t z = seed ^ (index * 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z = z ^ (z >> 31);
  return static_cast<float>(z >> 40) * (1.0f / 16777216.0f) >= p;
}
template <typename T>
__global__ void dropout_kernel(const T* __restrict__ x, T* __restrict__ out, int64_t n, float p, float keep_scale, uint64_t seed,
                               uint64_t offset) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    out[i] = dropout_keep(seed, offset + static_cast<uint64_t>(i), p) ? from_f32<T>(to_f32(x[i]) * keep_scale) : from_f32<T>(0.0f);
}

extern "C" int mcb_dropout(const void* x, void* out, int64_t n, float p, uint64_t seed, uint64_t offset, int dtype, void* stream) {
  MCB_NVTX_RANGE("mcb_dropout");
  if (!x || !out) return fail(MCB_ERR_NULL, "dropout: null pointer");
  if (n <= 0) return fail(MCB_ERR_SHAPE, "dropout: element count must be positive");
  if (!(p >= 0.0f && p < 1.0f)) return fail(MCB_ERR_SHAPE, "dropout: probability %g is not in [0, 1)", static_cast<double>(p));
  DeviceState* ds = current_device_state();
  if (!ds) return MCB_ERR_NOT_INIT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = grid_for(n, 256, ds->sm_count);
  const float keep_scale = 1.0f / (1.0f - p);
  MCB_DTYPE_SWITCH(dtype, (dropout_kernel<T><<<grid, 256, 0, st>>>((const T*)x, (T*)out, n, p, keep_scale, seed, offset)));
  MCB_CHECK_LAUNCH("dropout");
  return MCB_OK;
}

extern "C" int mcb_mul_scalar(const void* a, void* out, int64_t n, float value, int dtype, void* stream) {
  MCB_NVTX_RANGE("mcb_mul_scalar");
  if (!a || !out) return fail(MCB_ERR_NULL, "mul_scalar: null pointer");
  if (n <= 0) return fail(MCB_ERR_SHAPE, "mul_scalar: element count must be positive");
  DeviceState* ds = current_device_state();
  if (!ds) return MCB_ERR_NOT_INIT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = grid_for(n, 256, ds->sm_count);
  MCB_DTYPE_SWITCH(dtype, (mul_kernel<T><<<grid, 256, 0, st>>>((const T*)a, (const T*)a, (T*)out, n, value, 1)));
  MCB_CHECK_LAUNCH("mul_scalar");
  return MCB_OK;
}

extern "C" int mcb_lora_merge_weights(const void* W, const float* A, const float* B, void* out, int64_t K, int64_t N,
                                      int64_t r, float scale, int dtype, void* stream) {
  MCB_NVTX_RANGE("mcb_lora_merge_weights");
  if (!W || !A || !B || !out) return fail(MCB_ERR_NULL, "lora_merge_weights: null pointer");
  if (K <= 0 || N <= 0 || r <= 0 || K > 0x7fffffff || N > 0x7fffffff || r > 0x7fffffff)
    return fail(MCB_ERR_SHAPE, "lora_merge_weights: K=%lld N=%lld r=%lld", (long long)K, (long long)N, (long long)r);
  DeviceState* ds = current_device_state();
  if (!ds) return MCB_ERR_NOT_INIT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = grid_for(N * ((K + 3) / 4), 256, ds->sm_count);
  MCB_DTYPE_SWITCH(dtype, (merge_weights_kernel<T><<<grid, 256, 0, st>>>((const T*)W, A, B, (T*)out, (int)K, (int)N, (int)r, scale)));
  MCB_CHECK_LAUNCH("merge_weights");
  return MCB_OK;
}
