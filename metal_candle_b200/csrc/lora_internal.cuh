// Internal interface between the C-ABI LoRA entry points (lora_api.cu) and the two implementations:
// the float32 validation path on CUDA cores (sgemm_f32.cu) and the bfloat16 production path on
// tcgen05 tensor cores (umma_gemm.cu).
#pragma once
#include "common.cuh"

namespace mcb {

struct LoraArgs {
  const void* x = nullptr;     // [M,K]
  const void* W = nullptr;     // [N,K] or [K,N] per w_layout
  const void* bias = nullptr;  // [N] or null
  const void* residual = nullptr;  // added to y (forward, [M,N]) or to dx (backward, [M,K]); may alias the output
  const float* A = nullptr;    // [K,r] float32
  const float* B = nullptr;    // [r,N] float32
  void* y = nullptr;           // [M,N]
  void* h_save = nullptr;      // [rp, h_pitch(M)] scale*(x A) transposed, optional
  const void* dy = nullptr;    // [M,N]
  void* dx = nullptr;          // [M,K]
  void* swiglu_up = nullptr;   // backward, with dx: dx holds gate and this holds up [M,K]; both are replaced by the
                               // SwiGLU backward of the input gradient, which itself is not stored
  float* dA = nullptr;         // [K,r]
  float* dB = nullptr;         // [r,N]
  int accumulate = 0;
  int64_t M = 0, K = 0, N = 0, r = 0;
  float scale = 1.0f;
  int w_layout = MCB_W_OUT_IN;
  void* ws = nullptr;
  size_t ws_bytes = 0;
  cudaStream_t stream = nullptr;
};

// Several projections that share one input, computed as ONE linear with a block-diagonal rank path: segment i owns
// output columns [n_off, n_off + n) of the fused output and has its own adapter (A_i [K,r], B_i [r,n]).
constexpr int kMaxSegments = 4;
struct LoraSegments {
  int count = 0;
  const float* A[kMaxSegments] = {nullptr, nullptr, nullptr, nullptr};
  const float* B[kMaxSegments] = {nullptr, nullptr, nullptr, nullptr};
  float* dA[kMaxSegments] = {nullptr, nullptr, nullptr, nullptr};
  float* dB[kMaxSegments] = {nullptr, nullptr, nullptr, nullptr};
  int64_t n_off[kMaxSegments] = {0, 0, 0, 0};
  int64_t n[kMaxSegments] = {0, 0, 0, 0};
};

inline int64_t rank_padded(int64_t r) { return r <= 0 ? 0 : ((r + 15) / 16) * 16; }
// Row pitch (in elements) of the saved rank intermediate [rp, pitch]: tokens rounded up to 64.
inline int64_t h_pitch(int64_t M) { return ((M + 63) / 64) * 64; }

namespace f32path {
size_t workspace_bytes(int64_t M, int64_t K, int64_t N, int64_t r);
int delta_fwd(const LoraArgs& a);
// The delta of few tokens in one cluster launch, float32 arithmetic for either dtype of x and out.  Up to 512 tokens it
// beats the two float32 launches (400 x 4096 -> 4096 r64: 52 us against 91).
constexpr int64_t kDeltaMaxTokens = 512;
bool delta_small(int64_t M, int64_t r);
int delta_cluster(const LoraArgs& a, int dtype);
int linear_fwd(const LoraArgs& a);
int linear_bwd(const LoraArgs& a);
// out[M,N] = a[M,K] b[K,N]
int matmul(const float* a, const float* b, float* out, int64_t M, int64_t K, int64_t N, cudaStream_t st);
}  // namespace f32path

namespace bf16path {
struct GradRequest;
// One call of the fused GEMM  Y = X W^T (+bias) (+R) + (scale X P^T) Q^T ; all operands bf16, K-major.
struct GemmCall {
  const __nv_bfloat16* X = nullptr;   // [M,K]
  const __nv_bfloat16* W = nullptr;   // [N,K] or null
  const __nv_bfloat16* P = nullptr;   // [rp,K] or null
  const __nv_bfloat16* Q = nullptr;   // [N,rp] or null
  const __nv_bfloat16* bias = nullptr;
  const __nv_bfloat16* R = nullptr;   // [M,N] or null
  __nv_bfloat16* Y = nullptr;         // [M,N] or null
  __nv_bfloat16* H = nullptr;         // [rp,h_pitch] or null
  int64_t h_pitch = 0;
  int64_t M = 0, N = 0, K = 0;
  // A second pair of operands whose product is added in the same accumulators, X2 [M,K2] . W2 [N,K2]^T, or null (rp = 0 only): a
  // rank update whose intermediate a launch ahead has computed.
  const __nv_bfloat16* X2 = nullptr;
  const __nv_bfloat16* W2 = nullptr;
  int64_t K2 = 0;
  // Scratch [M, rp] for a rank intermediate that is computed apart (launch_gemm decides), or null: always in the product's own tiles.
  __nv_bfloat16* Hr = nullptr;
  int rp = 0;
  int r_true = 0;  // unpadded rank, for the algorithmic flop count
  float scale = 1.0f;
  // Weight-gradient problems to run as a tail phase of the same launch (one-CTA kernel only), or null.  Problem 0
  // reads the H this call writes.
  const GradRequest* grads = nullptr;
  // Y is the gate buffer of a SwiGLU and this its up buffer: the product is d act, and the epilogue replaces gate and
  // up by d gate and d up instead of storing it (pair kernel only).
  __nv_bfloat16* swiglu_up = nullptr;
};
// What the per-kernel profile records of a product on its own: an update from a second operand pair counts with the unpadded rank.
inline double gemm_flops(const GemmCall& c) {
  const double m = static_cast<double>(c.M), n = static_cast<double>(c.N), k = static_cast<double>(c.K), r = c.r_true;
  return 2.0 * m * n * k + (c.rp > 0 ? 2.0 * m * r * (k + n) : c.X2 != nullptr ? 2.0 * m * r * n : 0.0);
}
inline int gemm_kind(const GemmCall& c) { return c.rp > 0 || c.X2 != nullptr ? kProfGemmLora : kProfGemm; }
// Tile width and reduction parts of the split-reduction kernel (umma_split.cu); bn == 0: the persistent kernels run.
struct SplitPlan {
  int bn = 0, splits = 1;
};
SplitPlan split_plan(int64_t M, int64_t N, int64_t K, int rp, bool pair_kernel, const DeviceState* ds);
// Runs the call with that plan; with act != null its columns are blocks of 128 gate and 128 up features (bn 256) and c.Y,
// up, act receive gate, up and silu(gate) * up.
int launch_split(const SplitPlan& plan, const GemmCall& c, __nv_bfloat16* up, __nv_bfloat16* act, const DeviceState* ds, cudaStream_t st);
// Tiles of 256 x up to 512 on CTA pairs (umma_wide.cu): their width for a call without a rank path, or 0 (the other kernels run),
// and the better one's estimated cycles.
int wide_bn(int64_t M, int64_t N, int64_t nkb, bool swiglu, const DeviceState* ds, double* cycles = nullptr);
int launch_wide(int bn, const GemmCall& c, __nv_bfloat16* up, __nv_bfloat16* act, const DeviceState* ds, cudaStream_t st);
size_t workspace_bytes(int64_t M, int64_t K, int64_t N, int64_t r);
int delta_fwd(const LoraArgs& a, const DeviceState* ds);
int linear_fwd(const LoraArgs& a, const DeviceState* ds);
int linear_bwd(const LoraArgs& a, const DeviceState* ds);
// Whether linear_bwd can run the SwiGLU backward in the epilogue of its input-gradient product (a.swiglu_up).
bool swiglu_bwd_supported(int64_t M, int64_t K, int64_t N, int64_t r);
// The same two passes for a fused projection with one adapter of rank a.r per segment (a.A / a.B / a.dA / a.dB unused).
size_t fused_workspace_bytes(int64_t M, int64_t K, int64_t N, int64_t r, int segments);
int linear_fused_fwd(const LoraArgs& a, const LoraSegments& sg, const DeviceState* ds);
int linear_fused_bwd(const LoraArgs& a, const LoraSegments& sg, const DeviceState* ds);
// out[M,N] = a[M,K] bt[N,K]^T (bt is b transposed, both operands K-major)
int matmul_nt(const void* a, const void* bt, void* out, int64_t M, int64_t K, int64_t N, const DeviceState* ds,
              cudaStream_t st);
// gate, up [M,F] = x w_gu^T (w_gu: gate and up rows interleaved in blocks of 128), act = silu(gate) * up
int launch_gemm2_swiglu(const __nv_bfloat16* X, const __nv_bfloat16* Wgu, __nv_bfloat16* G, __nv_bfloat16* U,
                        __nv_bfloat16* Act, int64_t M, int64_t K, int64_t F, const DeviceState* ds, cudaStream_t st);
}  // namespace bf16path

}  // namespace mcb
