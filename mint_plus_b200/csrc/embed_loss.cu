// The two ends of the model around the layer stack, as HBM-bound kernels:
//   embed_fwd / embed_bwd   token embedding with the token-dropout rescale, <mask> and <pad> zeroing of MINT.forward and the
//                           (B,T,E) -> (T,B,E) layout change, in one pass; its weight gradient by per-CTA private sums
//   masked_ce_fwd / _bwd    the masked-language-model loss of the training step: cross-entropy over the vocabulary at the
//                           target positions, averaged over them, and its gradient with respect to the logits
#include <type_traits>

#include "common.cuh"

namespace mintb {

namespace {

template <typename T>
__device__ __forceinline__ float to_f(T v);
template <>
__device__ __forceinline__ float to_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T>
__device__ __forceinline__ T from_f(float v);
template <>
__device__ __forceinline__ float from_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Factor of token (b, t): 0 for <pad>, 0 for <mask> under token dropout, else the row's rescale
// (1 - mask_ratio_train) / (1 - masked / unpadded) under token dropout, else 1.
__device__ __forceinline__ float row_scale(int n_mask, int n_real, int token_dropout, float mask_ratio_train) {
  if (!token_dropout) return 1.f;
  const float observed = float(n_mask) / float(n_real);      // 0 / 0 -> NaN, as the tensor expression gives for an all-pad row
  return (1.f - mask_ratio_train) / (1.f - observed);
}

// out[t][b][:] = W[tok] * factor.  grid = (B, slabs of t): every CTA counts the <mask> and unpadded tokens of its row again (16 KB
// at T = 2048, from L2) and writes its own slab; with one CTA per row, B of the 148 SMs did all the writing (B8 T2048 E2560 bf16,
// 84 MB: 302 us, now 24 us).
template <typename T>
__global__ void __launch_bounds__(256) embed_fwd_kernel(const long long* __restrict__ tokens, const T* __restrict__ w, T* __restrict__ out,
                                                       float* __restrict__ scales, int B, int Tn, int E, int V, int pad_idx,
                                                       int mask_idx, int token_dropout, float mask_ratio_train, int slab) {
  __shared__ int s_cnt[2];
  const int b = blockIdx.x;
  const long long* row = tokens + size_t(b) * Tn;
  float scale = 1.f;
  if (token_dropout) {
    if (threadIdx.x < 2) s_cnt[threadIdx.x] = 0;
    __syncthreads();
    int nm = 0, nr = 0;
    for (int t = threadIdx.x; t < Tn; t += blockDim.x) {
      const long long tok = row[t];
      nm += tok == mask_idx;
      nr += tok != pad_idx;
    }
    nm = __reduce_add_sync(0xffffffffu, nm);
    nr = __reduce_add_sync(0xffffffffu, nr);
    if (threadIdx.x % 32 == 0) {
      atomicAdd(&s_cnt[0], nm);
      atomicAdd(&s_cnt[1], nr);
    }
    __syncthreads();
    scale = row_scale(s_cnt[0], s_cnt[1], token_dropout, mask_ratio_train);
  }
  if (blockIdx.y == 0 && threadIdx.x == 0 && scales != nullptr) scales[b] = scale;
  constexpr int VEC = 16 / sizeof(T);
  const int nvec = E / VEC;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, nwarps = blockDim.x / 32;
  const int t1 = min(Tn, int(blockIdx.y + 1) * slab);
  for (int t = blockIdx.y * slab + warp; t < t1; t += nwarps) {
    const long long tok = row[t];
    const bool zero = tok == pad_idx || (token_dropout && tok == mask_idx) || tok < 0 || tok >= V;
    const uint4* src = reinterpret_cast<const uint4*>(w + size_t(zero ? 0 : tok) * E);
    uint4* dst = reinterpret_cast<uint4*>(out + (size_t(t) * B + b) * E);
#pragma unroll 4
    for (int v = lane; v < nvec; v += 32) {
      uint4 q = make_uint4(0u, 0u, 0u, 0u);
      if (!zero) {
        q = __ldg(src + v);
        if (scale != 1.f) {
          T* e = reinterpret_cast<T*>(&q);
#pragma unroll
          for (int j = 0; j < VEC; ++j) e[j] = from_f<T>(to_f<T>(e[j]) * scale);
        }
      }
      dst[v] = q;
    }
  }
}

__device__ __forceinline__ float2 ld_two(const __nv_bfloat16* p) {
  const uint32_t u = *reinterpret_cast<const uint32_t*>(p);
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}
__device__ __forceinline__ float2 ld_two(const float* p) { return *reinterpret_cast<const float2*>(p); }

constexpr int kEmbCols = 256;    // columns of an embed_bwd CTA, two per thread
constexpr int kEmbBatch = 16;    // gradient rows that a thread has in flight

// dW[v][:] += factor(b, t) * d_out[t][b][:] over the tokens with tok == v.  A CTA walks a slab of tokens of one batch row with a
// private [V][256] sum in shared memory (a thread owns its two columns, so no two threads meet), then adds the slab's sums to the
// fp32 result, two columns per atomic.  grid = (slabs, B, column chunks).  Bound by the read of d_out, so the rows of sixteen tokens
// are requested before the first is added (one at a time, B16 T2048 E1280 bf16, 84 MB, took 171 us; now 34 us).
template <typename T>
__global__ void __launch_bounds__(kEmbCols / 2) embed_bwd_kernel(const long long* __restrict__ tokens, const T* __restrict__ d_out,
                                                                const float* __restrict__ scales, float* __restrict__ dw, int B, int Tn, int E,
                                                                int V, int pad_idx, int mask_idx, int token_dropout, int slab) {
  extern __shared__ float2 s_acc[];   // [V][128]
  const int b = blockIdx.y, c = blockIdx.z * kEmbCols + 2 * threadIdx.x;
  const bool mine = c < E;
  for (int v = 0; v < V; ++v) s_acc[v * (kEmbCols / 2) + threadIdx.x] = make_float2(0.f, 0.f);
  const float scale = scales[b];
  const int t0 = blockIdx.x * slab, t1 = min(Tn, t0 + slab);
  const long long* row = tokens + size_t(b) * Tn;
  if (mine) {
    for (int t = t0; t < t1; t += kEmbBatch) {
      int tok[kEmbBatch];
      float2 g[kEmbBatch];
#pragma unroll
      for (int k = 0; k < kEmbBatch; ++k) {
        const long long v = row[min(t + k, Tn - 1)];
        const bool skip = t + k >= t1 || v == pad_idx || (token_dropout && v == mask_idx) || v < 0 || v >= V;   // uniform over the CTA
        tok[k] = skip ? -1 : int(v);
      }
#pragma unroll
      for (int k = 0; k < kEmbBatch; ++k)
        g[k] = tok[k] < 0 ? make_float2(0.f, 0.f) : ld_two(d_out + (size_t(t + k) * B + b) * E + c);
#pragma unroll
      for (int k = 0; k < kEmbBatch; ++k)
        if (tok[k] >= 0) {
          float2& a = s_acc[tok[k] * (kEmbCols / 2) + threadIdx.x];
          a.x += g[k].x * scale;
          a.y += g[k].y * scale;
        }
    }
    for (int v = 0; v < V; ++v) {
      const float2 a = s_acc[v * (kEmbCols / 2) + threadIdx.x];
      if (a.x != 0.f || a.y != 0.f)
        asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(dw + size_t(v) * E + c), "f"(a.x), "f"(a.y) : "memory");
    }
  }
}

// One thread per token row of the logits [N][ld] (the first V columns count): log-sum-exp, the loss at the target where the
// row is a target position, and the two sums (loss, count) by one atomic per warp.
__global__ void __launch_bounds__(256) masked_ce_fwd_kernel(const __nv_bfloat16* __restrict__ logits, const long long* __restrict__ targets,
                                                           const unsigned char* __restrict__ mask, float* __restrict__ lse_out,
                                                           float* __restrict__ sums, int N, int ld, int V) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  float loss = 0.f, cnt = 0.f;
  if (i < N) {
    const __nv_bfloat16* row = logits + size_t(i) * ld;
    float m = -INFINITY;
    for (int v = 0; v < V; ++v) m = fmaxf(m, __bfloat162float(row[v]));
    float s = 0.f;
    for (int v = 0; v < V; ++v) s += __expf(__bfloat162float(row[v]) - m);
    const float lse = m + __logf(s);
    lse_out[i] = lse;
    if (mask[i]) {
      const long long tg = targets[i];
      loss = lse - (tg >= 0 && tg < V ? __bfloat162float(row[tg]) : 0.f);
      cnt = 1.f;
    }
  }
  for (int off = 16; off > 0; off >>= 1) {
    loss += __shfl_xor_sync(0xffffffffu, loss, off);
    cnt += __shfl_xor_sync(0xffffffffu, cnt, off);
  }
  if ((threadIdx.x % 32) == 0 && cnt > 0.f) {
    atomicAdd(sums, loss);
    atomicAdd(sums + 1, cnt);
  }
}

// d_logits[i][v] = (softmax(logits[i])[v] - [v == target]) * g / count at target rows, 0 elsewhere and in the pad columns.
__global__ void __launch_bounds__(256) masked_ce_bwd_kernel(const __nv_bfloat16* __restrict__ logits, const long long* __restrict__ targets,
                                                           const unsigned char* __restrict__ mask, const float* __restrict__ lse,
                                                           const float* __restrict__ sums, const float* __restrict__ g,
                                                           __nv_bfloat16* __restrict__ d_logits, int N, int ld, int V) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  __nv_bfloat16* drow = d_logits + size_t(i) * ld;
  if (!mask[i]) {
    for (int v = 0; v < ld; ++v) drow[v] = __float2bfloat16_rn(0.f);
    return;
  }
  const float coef = g[0] / sums[1];
  const __nv_bfloat16* row = logits + size_t(i) * ld;
  const float l = lse[i];
  const long long tg = targets[i];
  for (int v = 0; v < ld; ++v) {
    float d = 0.f;
    if (v < V) d = (__expf(__bfloat162float(row[v]) - l) - (v == tg ? 1.f : 0.f)) * coef;
    drow[v] = __float2bfloat16_rn(d);
  }
}

// The masked-language-model corruption from its three draws: a residue (not one of the special tokens) is a target where
// u_target < 0.15; a target becomes <mask> where u_kind < 0.8 and the drawn residue where u_kind > 0.9.
__global__ void __launch_bounds__(256) mlm_corrupt_kernel(const long long* __restrict__ tokens, const float* __restrict__ u_target, const float* __restrict__ u_kind,
                                                          const long long* __restrict__ residue, long long* __restrict__ out, uint8_t* __restrict__ target,
                                                          long long n, int cls, int eos, int pad, int mask) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long t = tokens[i];
  const bool tg = u_target[i] < 0.15f && t != cls && t != eos && t != pad;
  const float k = u_kind[i];
  out[i] = tg && k > 0.9f ? residue[i] : tg && k < 0.8f ? mask : t;
  target[i] = tg ? 1 : 0;
}

}  // namespace
}  // namespace mintb

using namespace mintb;

static int el_fail(const char* what, cudaError_t e) {
  set_error("%s: %s", what, cudaGetErrorString(e));
  return MINTB_ECUDA;
}

extern "C" int mintb_embed_fwd(const long long* tokens, const void* weight, void* out, float* row_scales, int B, int T, int E, int V,
                               int dtype, int pad_idx, int mask_idx, int token_dropout, float mask_ratio_train, void* stream) {
  const int esz = dtype == MINTB_F32 ? 4 : 2;
  if (tokens == nullptr || weight == nullptr || out == nullptr || B <= 0 || T <= 0 || E <= 0 || V <= 0 ||
      (dtype != MINTB_F32 && dtype != MINTB_BF16) || (E * esz) % 16 != 0 || (reinterpret_cast<uintptr_t>(weight) & 15) ||
      (reinterpret_cast<uintptr_t>(out) & 15)) {
    set_error("mintb_embed_fwd: tokens, weight, out, positive sizes, an f32 / bf16 weight with 16-byte rows and aligned pointers are required");
    return MINTB_EINVAL;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int slab = T > 1024 ? 32 : 16;   // two or four rows per warp: thousands of CTAs at full size, and a short batch still spreads out
  const dim3 grid(B, (T + slab - 1) / slab);
  if (dtype == MINTB_F32)
    embed_fwd_kernel<float><<<grid, 256, 0, st>>>(tokens, static_cast<const float*>(weight), static_cast<float*>(out), row_scales, B, T, E, V,
                                               pad_idx, mask_idx, token_dropout, mask_ratio_train, slab);
  else
    embed_fwd_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(tokens, static_cast<const __nv_bfloat16*>(weight), static_cast<__nv_bfloat16*>(out),
                                                       row_scales, B, T, E, V, pad_idx, mask_idx, token_dropout, mask_ratio_train, slab);
  count_launches(1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MINTB_OK : el_fail("mintb_embed_fwd launch", e);
}

extern "C" int mintb_embed_bwd(const long long* tokens, const void* d_out, const float* row_scales, float* d_weight, int B, int T, int E,
                               int V, int dtype, int pad_idx, int mask_idx, int token_dropout, void* stream) {
  if (tokens == nullptr || d_out == nullptr || row_scales == nullptr || d_weight == nullptr || B <= 0 || T <= 0 || E <= 0 || V <= 0 ||
      V > 64 || (dtype != MINTB_F32 && dtype != MINTB_BF16)) {
    set_error("mintb_embed_bwd: tokens, d_out, row_scales, d_weight, positive sizes, a vocabulary of at most 64 and f32 / bf16 are required");
    return MINTB_EINVAL;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(d_weight, 0, size_t(V) * E * sizeof(float), st);
  if (e != cudaSuccess) return el_fail("mintb_embed_bwd memset", e);
  if (E % 2 != 0 || reinterpret_cast<uintptr_t>(d_out) % 8 != 0 || reinterpret_cast<uintptr_t>(d_weight) % 8 != 0) {
    set_error("mintb_embed_bwd: an even E, d_out and d_weight aligned to 8 bytes are required");
    return MINTB_EINVAL;
  }
  const size_t smem = size_t(V) * kEmbCols * sizeof(float);   // at most 64 KB
  // a slab's sums cost up to V atomics per column pair, so slabs grow with the batch: from 32 tokens on a small one to 128
  const int chunks = (E + kEmbCols - 1) / kEmbCols;
  const int slab = size_t(B) * T * chunks > size_t(128) * 1024 ? 128 : 32;
  const dim3 grid((T + slab - 1) / slab, B, chunks);
  auto run = [&](auto* g) {
    using G = typename std::remove_cv<typename std::remove_pointer<decltype(g)>::type>::type;
    cudaError_t err = cudaSuccess;
    if (smem > 48 * 1024) err = cudaFuncSetAttribute(embed_bwd_kernel<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (err != cudaSuccess) return err;
    embed_bwd_kernel<G><<<grid, kEmbCols / 2, smem, st>>>(tokens, g, row_scales, d_weight, B, T, E, V, pad_idx, mask_idx, token_dropout, slab);
    return cudaSuccess;
  };
  e = dtype == MINTB_F32 ? run(static_cast<const float*>(d_out)) : run(static_cast<const __nv_bfloat16*>(d_out));
  if (e != cudaSuccess) return el_fail("cudaFuncSetAttribute", e);
  count_launches(1);
  e = cudaGetLastError();
  return e == cudaSuccess ? MINTB_OK : el_fail("mintb_embed_bwd launch", e);
}

extern "C" int mintb_masked_ce_fwd(const void* logits, const long long* targets, const unsigned char* mask, float* lse, float* sums,
                                   int N, int ld, int V, void* stream) {
  if (logits == nullptr || targets == nullptr || mask == nullptr || lse == nullptr || sums == nullptr || N <= 0 || V <= 0 || ld < V) {
    set_error("mintb_masked_ce_fwd: logits (bf16 [N][ld], ld >= V), targets, mask, lse, sums and positive sizes are required");
    return MINTB_EINVAL;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(sums, 0, 2 * sizeof(float), st);
  if (e != cudaSuccess) return el_fail("mintb_masked_ce_fwd memset", e);
  masked_ce_fwd_kernel<<<(N + 255) / 256, 256, 0, st>>>(static_cast<const __nv_bfloat16*>(logits), targets, mask, lse, sums, N, ld, V);
  count_launches(1);
  e = cudaGetLastError();
  return e == cudaSuccess ? MINTB_OK : el_fail("mintb_masked_ce_fwd launch", e);
}

extern "C" int mintb_masked_ce_bwd(const void* logits, const long long* targets, const unsigned char* mask, const float* lse,
                                   const float* sums, const float* grad_loss, void* d_logits, int N, int ld, int V, void* stream) {
  if (logits == nullptr || targets == nullptr || mask == nullptr || lse == nullptr || sums == nullptr || grad_loss == nullptr ||
      d_logits == nullptr || N <= 0 || V <= 0 || ld < V) {
    set_error("mintb_masked_ce_bwd: every pointer and positive sizes (ld >= V) are required");
    return MINTB_EINVAL;
  }
  masked_ce_bwd_kernel<<<(N + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(logits), targets, mask, lse, sums, grad_loss, static_cast<__nv_bfloat16*>(d_logits), N, ld, V);
  count_launches(1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MINTB_OK : el_fail("mintb_masked_ce_bwd launch", e);
}

extern "C" int mintb_mlm_corrupt(const long long* tokens, const float* u_target, const float* u_kind, const long long* residue, long long* out,
                                 unsigned char* target, long long n, int cls, int eos, int pad, int mask, void* stream) {
  if (tokens == nullptr || u_target == nullptr || u_kind == nullptr || residue == nullptr || out == nullptr || target == nullptr || n <= 0 || n > (1ll << 38)) {
    set_error("mintb_mlm_corrupt: every pointer and a positive size are required");
    return MINTB_EINVAL;
  }
  mlm_corrupt_kernel<<<unsigned((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(tokens, u_target, u_kind, residue, out, target, n, cls, eos, pad, mask);
  count_launches(1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MINTB_OK : el_fail("mintb_mlm_corrupt launch", e);
}
