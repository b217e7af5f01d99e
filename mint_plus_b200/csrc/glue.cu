// HBM-bound kernels around the projection GEMMs and the attention (bf16 tensors, fp32 arithmetic):
//
//   add_layernorm_fwd / _bwd   s = a x + b r, y = LayerNorm(s) gamma + beta  — the residual-and-norm glue of the Pre-LN layer
//                              (a = b = 1; modules.py:179-195 of the reference) and of the muS layer (a = sqrt(1 - tau),
//                              b = sqrt(tau); mu_scaling/layer.py:259-280); without gamma it is the scaled residual add alone.
//   gelu_bwd_colsum            dz = dy * gelu'(z) and the bias gradient sum_rows(dz) in the same pass; without z the column
//                              sum of dy alone (bias gradient of a plain projection).
//   qkv_grad_pack              gradients of the head-major q, k, v (B,H,T,D) -> one row-major [T*B][3E] matrix for the
//                              dgrad / wgrad products: un-rotates dq and dk of the self pathway (transpose of the RoPE
//                              rotation) and applies the q scale.
//
// Every kernel reads each input once and writes each output once, 16 bytes per thread and access, rows walked by whole warps.
#include <cuda_fp8.h>

#include <type_traits>

#include "common.cuh"
#include "ptx.cuh"

namespace mintb {
namespace {

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

// Two fp32 values in one 64-bit register, for the packed instructions.
__device__ __forceinline__ uint64_t pk(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void upk(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t bf2(uint32_t w) { return pk(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
__device__ __forceinline__ uint32_t to_bf2(uint64_t v) {
  float a, b;
  upk(v, a, b);
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
__device__ __forceinline__ uint32_t word(const uint4& q, int i) { return i == 0 ? q.x : i == 1 ? q.y : i == 2 ? q.z : q.w; }

__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return u;
}

__device__ __forceinline__ uint2 pack8_e4m3(const float (&f)[8], float inv) {
  uint2 u;
  __nv_fp8x2_storage_t* h = reinterpret_cast<__nv_fp8x2_storage_t*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __nv_cvt_float2_to_fp8x2(make_float2(f[2 * i] * inv, f[2 * i + 1] * inv), __NV_SATFINITE, __NV_E4M3);
  return u;
}

// eight values -> e5m2 (saturating at +-57344) after multiplication by inv; `f` is overwritten with the values the
// 8-bit numbers stand for, times `scale` (an e5m2 number is the upper byte of the fp16 number with the same value)
__device__ __forceinline__ uint2 pack8_e5m2_roundtrip(float (&f)[8], float inv, float scale) {
  uint2 u;
  __nv_fp8x2_storage_t* h = reinterpret_cast<__nv_fp8x2_storage_t*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    h[i] = __nv_cvt_float2_to_fp8x2(make_float2(f[2 * i] * inv, f[2 * i + 1] * inv), __NV_SATFINITE, __NV_E5M2);
    const unsigned short lo = static_cast<unsigned short>((h[i] & 0xffu) << 8), hi = static_cast<unsigned short>(h[i] & 0xff00u);
    f[2 * i] = __half2float(__ushort_as_half(lo)) * scale;
    f[2 * i + 1] = __half2float(__ushort_as_half(hi)) * scale;
  }
  return u;
}

__device__ __forceinline__ float ld_param(const void* p, int dtype, int i) {
  return dtype == MINTB_F32 ? static_cast<const float*>(p)[i] : __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
}

constexpr int kLnWarps = 4;

struct LnParams {
  const __nv_bfloat16 *x, *r;       // r may be null (then s = a x)
  float a, b;
  const void *gamma, *beta;         // null: no normalisation, only s
  int param_dtype;                  // MINTB_F32 or MINTB_BF16
  __nv_bfloat16 *s_out, *y_out;     // either may be null
  __nv_fp8_storage_t* q_out;        // e4m3 copy of the main result (y with gamma, else s), sat(value * q_inv); may be null
  float q_inv;
  float2* stats;                    // [rows] (mean, rstd); written by forward, read by backward
  const __nv_bfloat16 *dy, *ds_in;  // backward inputs (either may be null)
  int ds_apart;                     // ds_in is added to dx as a gradient of its own: after dx = a ds has been rounded
  __nv_bfloat16 *dx, *dr;           // backward outputs (dr may be null)
  float* partial;                   // backward: [gridDim.x][2][E] sums of dy * xhat and of dy
  int rows, E;
  float eps;
};

// gamma and beta as they are in memory, requested without waiting for them; 16 bytes at a time where their alignment allows it.
struct RawParams {
  template <int THREADS>
  static __device__ __forceinline__ void request(unsigned char* dst, const void* src, int bytes) {
    if (src == nullptr) {
      for (int i = threadIdx.x * 16; i < bytes; i += THREADS * 16) *reinterpret_cast<uint4*>(dst + i) = make_uint4(0u, 0u, 0u, 0u);
    } else if (reinterpret_cast<uintptr_t>(src) % 16 == 0) {
      for (int i = threadIdx.x * 16; i < bytes; i += THREADS * 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ptx::smem_u32(dst + i)), "l"(static_cast<const unsigned char*>(src) + i) : "memory");
    } else {
      for (int i = threadIdx.x * 2; i < bytes; i += THREADS * 2)
        *reinterpret_cast<uint16_t*>(dst + i) = *reinterpret_cast<const uint16_t*>(static_cast<const unsigned char*>(src) + i);
    }
  }
  static __device__ __forceinline__ void arrived() { asm volatile("cp.async.wait_all;" ::: "memory"); }
  // vector vi (eight values) of the copy
  static __device__ __forceinline__ void read(const unsigned char* src, int dtype, int vi, float (&f)[8]) {
    if (dtype == MINTB_F32) {
      *reinterpret_cast<float4*>(f) = *reinterpret_cast<const float4*>(src + vi * 32);
      *reinterpret_cast<float4*>(f + 4) = *reinterpret_cast<const float4*>(src + vi * 32 + 16);
    } else {
      unpack8(*reinterpret_cast<const uint4*>(src + vi * 16), f);
    }
  }
};

// MAXV: 16-byte vectors per lane (E <= MAXV * 256).  A warp owns a row and holds it packed, as it was loaded, through the passes for
// the mean, the variance and the result: as fp32 values (and with registers for a second tensor that is not there) the wide rows
// left 12 warps on an SM and half of the memory's rate (16384 x 2560, no residual, back to back: 56 us; now 39 us, 4.3 TB/s).
// The parameters are read behind the wait like everything else (the kernel before may be an optimizer's), but no row waits for them: they
// travel to shared memory while the first row does, out of L2, where the prefetch has brought them meanwhile (it delivers nothing, so it
// may run ahead).  Loaded and converted first, they held up every pass of a chain of short kernels (one pair through the 33-layer FP8 650M
// model: 2435 us, 2389 so).
template <int MAXV, bool HAS_R>
__global__ void __launch_bounds__(kLnWarps * 32, MAXV == 10 ? 4 : (MAXV == 5 ? 6 : 8)) add_layernorm_fwd_kernel(LnParams p) {
  __shared__ __align__(16) unsigned char s_gamma[MAXV * 256 * 4], s_beta[MAXV * 256 * 4];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int nvec = p.E / 8;
  const float inv_e = 1.f / float(p.E);
  const int param_bytes = p.E * (p.param_dtype == MINTB_F32 ? 4 : 2);
  if (p.gamma != nullptr && int(threadIdx.x) * 128 < param_bytes) {
    ptx::prefetch_l2(static_cast<const unsigned char*>(p.gamma) + threadIdx.x * 128);
    if (p.beta != nullptr) ptx::prefetch_l2(static_cast<const unsigned char*>(p.beta) + threadIdx.x * 128);
  }
  ptx::griddep_wait();
  ptx::griddep_launch();
  if (p.gamma != nullptr) {
    RawParams::request<kLnWarps * 32>(s_gamma, p.gamma, param_bytes);
    RawParams::request<kLnWarps * 32>(s_beta, p.beta, param_bytes);
  }
  for (int first = blockIdx.x * kLnWarps; first < p.rows; first += gridDim.x * kLnWarps) {
    const int row = first + warp;
    const bool ok = row < p.rows;
    const uint4* xr = reinterpret_cast<const uint4*>(p.x + size_t(row) * p.E);
    const uint4* rr = reinterpret_cast<const uint4*>(p.r + size_t(row) * p.E);
    // every load of the row is issued before the first use (a store between two loads would order them)
    uint4 xq[MAXV], rq[HAS_R ? MAXV : 1];
#pragma unroll
    for (int k = 0; k < MAXV; ++k) {
      const int vi = lane + 32 * k;
      xq[k] = make_uint4(0u, 0u, 0u, 0u);
      if (HAS_R) rq[k] = xq[k];
      if (ok && vi < nvec) {
        xq[k] = __ldg(xr + vi);
        if (HAS_R) rq[k] = __ldg(rr + vi);
      }
    }
    if (p.gamma != nullptr && first == int(blockIdx.x) * kLnWarps) {
      RawParams::arrived();
      __syncthreads();
    }
    if (!ok) break;   // (of this CTA's last rows)
    auto value = [&](int k, float (&v)[8]) {   // a x + b r of vector k
      unpack8(xq[k], v);
      if constexpr (HAS_R) {
        float rv[8];
        unpack8(rq[k], rv);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = fmaf(p.a, v[j], p.b * rv[j]);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] *= p.a;
      }
    };
    auto repack = [&] {   // keeps the compiler from holding the unpacked row from one pass to the next
#pragma unroll
      for (int k = 0; k < MAXV; ++k) {
        asm volatile("" : "+r"(xq[k].x), "+r"(xq[k].y), "+r"(xq[k].z), "+r"(xq[k].w));
        if (HAS_R) asm volatile("" : "+r"(rq[k].x), "+r"(rq[k].y), "+r"(rq[k].z), "+r"(rq[k].w));
      }
    };
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < MAXV; ++k) {
      float v[8];
      value(k, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) sum += v[j];
      const int vi = lane + 32 * k;
      if (p.s_out != nullptr && vi < nvec) {
        const uint4 packed = pack8(v);
        reinterpret_cast<uint4*>(p.s_out + size_t(row) * p.E)[vi] = packed;
        if (p.q_out != nullptr && p.gamma == nullptr) {   // the e4m3 copy is taken from the rounded bf16 values
          float rb[8];
          unpack8(packed, rb);
          reinterpret_cast<uint2*>(p.q_out + size_t(row) * p.E)[vi] = pack8_e4m3(rb, p.q_inv);
        }
      }
    }
    if (p.gamma == nullptr) continue;
    repack();
    const float mean = warp_sum_f(sum) * inv_e;
    float sq = 0.f;
#pragma unroll
    for (int k = 0; k < MAXV; ++k) {
      if (lane + 32 * k < nvec) {
        float v[8];
        value(k, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float d = v[j] - mean;
          sq = fmaf(d, d, sq);
        }
      }
    }
    repack();
    const float rstd = rsqrtf(warp_sum_f(sq) * inv_e + p.eps);
    if (lane == 0 && p.stats != nullptr) p.stats[row] = make_float2(mean, rstd);
#pragma unroll
    for (int k = 0; k < MAXV; ++k) {
      const int vi = lane + 32 * k;
      if (vi < nvec) {
        float v[8], o[8], gm[8], bt[8];
        value(k, v);
        RawParams::read(s_gamma, p.param_dtype, vi, gm);
        RawParams::read(s_beta, p.param_dtype, vi, bt);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = fmaf((v[j] - mean) * rstd, gm[j], bt[j]);
        const uint4 packed = pack8(o);
        reinterpret_cast<uint4*>(p.y_out + size_t(row) * p.E)[vi] = packed;
        if (p.q_out != nullptr) {
          float rb[8];
          unpack8(packed, rb);
          reinterpret_cast<uint2*>(p.q_out + size_t(row) * p.E)[vi] = pack8_e4m3(rb, p.q_inv);
        }
      }
    }
  }
}

// ds = LayerNorm'(dy) + ds_in;  dx = a ds;  dr = b ds;  per-CTA partial sums for dgamma / dbeta.
// LayerNorm backward per row: g = dy gamma, xhat = (s - mean) rstd, ds = rstd (g - mean(g) - xhat mean(g xhat)).
//
// A CTA spans one row: thread i owns the 8 columns of 16-byte vector i for every row the CTA walks, so its share of
// dgamma / dbeta stays in 16 registers and no thread ever adds into another thread's columns.  kLnBwdRows rows are in
// flight at a time: every tensor's loads are issued before the first use.  Their 2 x kLnBwdRows row sums are reduced
// by nine warp shuffles, then across the warps through a double-buffered shared-memory slot with ONE barrier per batch of rows.
// Which tensors exist is a template argument (r, ds_in, parameter gradients), so that none costs registers that is not there, and
// the arithmetic is packed, two columns an instruction: with all of it in one body, single values and the load of ds_in behind the
// barrier, instructions and latency held 32768 x 640 at 2.1 TB/s (75 us; now 32 us).
#ifndef MINTB_LN_BWD_PER_SM
#define MINTB_LN_BWD_PER_SM 3
#endif
constexpr int kLnBwdRows = 4;

// Sums of eight values over the warp: afterwards the lanes with lane / 4 == i hold the sum of v[i].
__device__ __forceinline__ float warp_sum8(float (&v)[8], int lane) {
#pragma unroll
  for (int o = 16, n = 4; o >= 4; o >>= 1, n >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// NW: warps per CTA (E <= NW * 256); MINB: CTAs per SM the register budget is cut for.
template <int NW, int MINB, bool HAS_R, bool HAS_DS, bool PARAM>
__global__ void __launch_bounds__(NW * 32, MINB) add_layernorm_bwd_kernel(LnParams p) {
  __shared__ __align__(16) float red[2][NW][2 * kLnBwdRows];
  const int vi = threadIdx.x, warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int nvec = p.E / 8;
  const bool live = vi < nvec;
  const float inv_e = 1.f / float(p.E);
  uint64_t gm[4], rg[PARAM ? 4 : 1], rb[PARAM ? 4 : 1];
  ptx::griddep_wait();
  ptx::griddep_launch();
#pragma unroll
  for (int j = 0; j < 4; ++j)
    gm[j] = live ? pk(ld_param(p.gamma, p.param_dtype, vi * 8 + 2 * j), ld_param(p.gamma, p.param_dtype, vi * 8 + 2 * j + 1)) : pk(0.f, 0.f);
  if constexpr (PARAM) {
#pragma unroll
    for (int j = 0; j < 4; ++j) rg[j] = rb[j] = pk(0.f, 0.f);
  }
  const float nb = p.b;
  int parity = 0;
  for (int row0 = blockIdx.x * kLnBwdRows; row0 < p.rows; row0 += gridDim.x * kLnBwdRows, parity ^= 1) {
    uint4 xq[kLnBwdRows], dq[kLnBwdRows], rq[HAS_R ? kLnBwdRows : 1], eq[HAS_DS ? kLnBwdRows : 1];
    float2 st[kLnBwdRows];
    const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int r = 0; r < kLnBwdRows; ++r) {
      const int row = row0 + r;
      const bool ok = live && row < p.rows;
      const size_t off = size_t(row) * p.E;
      xq[r] = dq[r] = zero4;
      if (HAS_R) rq[r] = zero4;
      if (HAS_DS) eq[r] = zero4;
      st[r] = make_float2(0.f, 0.f);
      if (ok) {
        xq[r] = __ldg(reinterpret_cast<const uint4*>(p.x + off) + vi);
        dq[r] = __ldg(reinterpret_cast<const uint4*>(p.dy + off) + vi);
        if (HAS_R) rq[r] = __ldg(reinterpret_cast<const uint4*>(p.r + off) + vi);
        if (HAS_DS) eq[r] = __ldg(reinterpret_cast<const uint4*>(p.ds_in + off) + vi);
        st[r] = __ldg(p.stats + row);
      }
    }
    // xhat = (a x + b r - mean) rstd of columns 2 j, 2 j + 1 of row r; rows past the end: all zeros
    auto xhat = [&](int r, int j) {
      const float m = -st[r].x * st[r].y, sa = p.a * st[r].y;
      uint64_t t = pk(m, m);
      if (HAS_R) {
        const float sb = nb * st[r].y;
        t = fma2(bf2(word(rq[r], j)), pk(sb, sb), t);
      }
      return fma2(bf2(word(xq[r], j)), pk(sa, sa), t);
    };
    float c[2 * kLnBwdRows];
#pragma unroll
    for (int r = 0; r < kLnBwdRows; ++r) {
      uint64_t c1 = pk(0.f, 0.f), c2 = c1;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint64_t x = xhat(r, j), d = bf2(word(dq[r], j)), g = mul2(d, gm[j]);
        c1 = add2(c1, g);
        c2 = fma2(g, x, c2);
        if constexpr (PARAM) {
          rg[j] = fma2(d, x, rg[j]);
          rb[j] = add2(rb[j], d);
        }
      }
      float u, v;
      upk(c1, u, v);
      c[2 * r] = u + v;
      upk(c2, u, v);
      c[2 * r + 1] = u + v;
    }
    const float mine = warp_sum8(c, lane);
    if (lane % 4 == 0) red[parity][warp][lane / 4] = mine;
    __syncthreads();   // the slot of the other parity is free again once every thread is past this barrier
#pragma unroll
    for (int i = 0; i < 2 * kLnBwdRows; ++i) c[i] = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) {   // same order in every thread: all of them hold identical sums
#pragma unroll
      for (int i = 0; i < 2 * kLnBwdRows; i += 4) {
        const float4 t = *reinterpret_cast<const float4*>(&red[parity][w][i]);
        c[i] += t.x; c[i + 1] += t.y; c[i + 2] += t.z; c[i + 3] += t.w;
      }
    }
    // The second pass unpacks the rows again instead of keeping their fp32 values alive across the barrier; the empty statements
    // stop the compiler from undoing that.
#pragma unroll
    for (int r = 0; r < kLnBwdRows; ++r) {
      asm volatile("" : "+r"(xq[r].x), "+r"(xq[r].y), "+r"(xq[r].z), "+r"(xq[r].w));
      asm volatile("" : "+r"(dq[r].x), "+r"(dq[r].y), "+r"(dq[r].z), "+r"(dq[r].w));
      if (HAS_R) asm volatile("" : "+r"(rq[r].x), "+r"(rq[r].y), "+r"(rq[r].z), "+r"(rq[r].w));
    }
#pragma unroll
    for (int r = 0; r < kLnBwdRows; ++r) {
      const int row = row0 + r;
      if (!(live && row < p.rows)) continue;
      const size_t off = size_t(row) * p.E;
      const float rstd = st[r].y, m1 = -rstd * c[2 * r] * inv_e, m2 = -rstd * c[2 * r + 1] * inv_e;
      uint4 o, o2;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint64_t g = mul2(bf2(word(dq[r], j)), gm[j]);
        uint64_t ds = fma2(g, pk(rstd, rstd), fma2(xhat(r, j), pk(m2, m2), pk(m1, m1)));
        if (HAS_DS && !p.ds_apart) ds = add2(ds, bf2(word(eq[r], j)));
        uint32_t w = to_bf2(mul2(ds, pk(p.a, p.a)));
        if (HAS_DS && p.ds_apart) w = to_bf2(add2(bf2(w), bf2(word(eq[r], j))));
        (j == 0 ? o.x : j == 1 ? o.y : j == 2 ? o.z : o.w) = w;
        if (HAS_R) {
          const uint32_t w2 = to_bf2(mul2(ds, pk(nb, nb)));
          (j == 0 ? o2.x : j == 1 ? o2.y : j == 2 ? o2.z : o2.w) = w2;
        }
      }
      reinterpret_cast<uint4*>(p.dx + off)[vi] = o;
      if (HAS_R && p.dr != nullptr) reinterpret_cast<uint4*>(p.dr + off)[vi] = o2;
    }
  }
  if constexpr (PARAM) {
    if (live) {
      float* dst = p.partial + size_t(blockIdx.x) * 2 * p.E + vi * 8;
      float f[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) upk(rg[j], f[2 * j], f[2 * j + 1]);
      *reinterpret_cast<float4*>(dst) = make_float4(f[0], f[1], f[2], f[3]);
      *reinterpret_cast<float4*>(dst + 4) = make_float4(f[4], f[5], f[6], f[7]);
#pragma unroll
      for (int j = 0; j < 4; ++j) upk(rb[j], f[2 * j], f[2 * j + 1]);
      *reinterpret_cast<float4*>(dst + p.E) = make_float4(f[0], f[1], f[2], f[3]);
      *reinterpret_cast<float4*>(dst + p.E + 4) = make_float4(f[4], f[5], f[6], f[7]);
    }
  }
}

// The scaled residual sum alone (no normalisation): dx = a ds_in, dr = b ds_in.
__global__ void __launch_bounds__(256) scaled_copies_kernel(LnParams p, size_t n_vec) {
  ptx::griddep_wait();
  ptx::griddep_launch();
  const size_t i = size_t(blockIdx.x) * 256 + threadIdx.x;
  if (i >= n_vec) return;
  const uint4 e = __ldg(reinterpret_cast<const uint4*>(p.ds_in) + i);
  float v[8], o[8];
  unpack8(e, v);
#pragma unroll
  for (int j = 0; j < 8; ++j) o[j] = p.a * v[j];
  reinterpret_cast<uint4*>(p.dx)[i] = pack8(o);
  if (p.dr != nullptr) {
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = p.b * v[j];
    reinterpret_cast<uint4*>(p.dr)[i] = pack8(o);
  }
}

__device__ __forceinline__ void st_param(void* p, int dtype, int i, float v) {
  if (dtype == MINTB_F32) static_cast<float*>(p)[i] = v;
  else static_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
}

// dgamma[e] = sum over CTAs of partial[c][0][e], dbeta likewise; fixed order.  CTA = 32 columns x 32 row lanes: each lane
// adds every 32nd partial, the sums meet in shared memory.
__global__ void __launch_bounds__(1024) ln_param_grad_kernel(const float* __restrict__ partial, int n_parts, int E, void* __restrict__ dgamma,
                                                             void* __restrict__ dbeta, int out_dtype) {
  __shared__ float red[32][33];
  ptx::griddep_wait();
  ptx::griddep_launch();
  const int cl = threadIdx.x % 32, rl = threadIdx.x / 32;
  const int i = blockIdx.x * 32 + cl;
  float t = 0.f;
  if (i < 2 * E) {
#pragma unroll 4
    for (int c = rl; c < n_parts; c += 32) t += partial[size_t(c) * 2 * E + i];
  }
  red[rl][cl] = t;
  __syncthreads();
  if (rl == 0 && i < 2 * E) {
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < 32; ++k) sum += red[k][cl];
    if (i < E) st_param(dgamma, out_dtype, i, sum); else st_param(dbeta, out_dtype, i - E, sum);
  }
}

// ------------------------------------------------------------------------------------------------ GELU backward + column sums
constexpr int kColRows = 256;   // rows per CTA strip of the gradient pack
constexpr int kSumRows = 64;    // rows per CTA strip of the column sums: every thread has its 8 rows in flight at once, and
                                // the grid is many waves deep (a 256-row strip left 1.6 to 2.2 waves at 32768 rows)
constexpr int kColLanes = 8;    // threads that share a column group, each taking every 8th row of the strip

// d/dz [z Phi(z)] = Phi(z) + z phi(z) of two values, and with VAL z Phi(z) itself.  Phi(-|z|) = exp(-z^2 / 2) Q(|z|) with Q a
// polynomial of degree 10 (least squares on Chebyshev nodes of [0, 6], weighted by exp(-a^2 / 2) and re-weighted towards the largest
// error; Q(a) = erfcx(a / sqrt 2) / 2): one special-function operation per value, shared with the density, and packed multiply-adds
// for the rest.  Largest error of Phi in fp32 arithmetic 1.5e-7 (the rational form it replaces, with a reciprocal as well: 2.9e-7).
template <bool VAL>
__device__ __forceinline__ uint64_t gelu_grad2(float z0, float z1, uint64_t& val) {
  const uint64_t z = pk(z0, z1), a = pk(fminf(fabsf(z0), 6.f), fminf(fabsf(z1), 6.f));
  constexpr float q[11] = {4.999999404e-01f, -3.989365101e-01f, 2.499167919e-01f, -1.325137913e-01f, 6.115488335e-02f, -2.431392856e-02f,
                           7.939389907e-03f, -1.974627143e-03f, 3.397383844e-04f, -3.520777682e-05f, 1.631689429e-06f};
  uint64_t s = pk(q[10], q[10]);
#pragma unroll
  for (int k = 9; k >= 0; --k) s = fma2(s, a, pk(q[k], q[k]));
  float x0, x1, e0, e1, t0, t1;
  upk(mul2(mul2(z, pk(-0.72134752044448170f, -0.72134752044448170f)), z), x0, x1);   // -z^2 / 2 log2 e
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(x0));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(x1));
  const uint64_t e = pk(e0, e1);
  upk(fma2(mul2(e, s), pk(-1.f, -1.f), pk(0.5f, 0.5f)), t0, t1);                       // 1/2 - Phi(-|z|)
  const uint64_t cdf = add2(pk(0.5f, 0.5f), pk(copysignf(t0, z0), copysignf(t1, z1)));
  if (VAL) val = mul2(z, cdf);
  return fma2(mul2(z, pk(0.3989422804014327f, 0.3989422804014327f)), e, cdf);
}

// CTA = 32 column groups (8 columns each: 256 columns) x 8 row lanes over a strip of kSumRows rows; a warp reads 512
// contiguous bytes of one row.  A thread issues the loads of all its rows of the strip (in two halves when z is read as
// well) before it touches the first value.  The 8 partial column sums meet in shared memory; db gets one atomicAdd per
// column and CTA, or, with a workspace, the sum of the strips' sums in its own type (no clearing and no conversion pass).
template <bool HAS_Z>
__global__ void __launch_bounds__(256) gelu_bwd_colsum_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ z,
                                                              __nv_bfloat16* __restrict__ dz, float* __restrict__ db, int M, int N,
                                                              __nv_bfloat16* __restrict__ act, __nv_fp8_storage_t* __restrict__ q8,
                                                              float q_inv, float q_scale, float* __restrict__ strips, int* __restrict__ arrived,
                                                              void* __restrict__ db_out, int db_dtype) {
  __shared__ float part[kColLanes][32][8];
  __shared__ bool s_last;
  ptx::griddep_wait();
  ptx::griddep_launch();
  const int cl = threadIdx.x % 32, rl = threadIdx.x / 32;
  const int cg = blockIdx.x * 32 + cl;   // column group
  const bool live = cg * 8 < N;
  const int m0 = blockIdx.y * kSumRows;
  constexpr int kPerThread = kSumRows / kColLanes;        // 8 rows of the strip per thread
  constexpr int kBatch = HAS_Z ? kPerThread / 2 : kPerThread;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (live) {
#pragma unroll
    for (int h = 0; h < kPerThread / kBatch; ++h) {
      uint4 gq[kBatch], zq[HAS_Z ? kBatch : 1];
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        const int m = m0 + rl + (h * kBatch + i) * kColLanes;
        const size_t off = size_t(m) * N + size_t(cg) * 8;
        gq[i] = make_uint4(0u, 0u, 0u, 0u);
        if (HAS_Z) zq[i] = gq[i];
        if (m < M) {
          gq[i] = __ldg(reinterpret_cast<const uint4*>(dy + off));
          if (HAS_Z) zq[i] = __ldg(reinterpret_cast<const uint4*>(z + off));
        }
      }
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        const int m = m0 + rl + (h * kBatch + i) * kColLanes;
        float g[8];
        unpack8(gq[i], g);
        if (HAS_Z) {
          float zv[8];
          unpack8(zq[i], zv);
          if (act != nullptr) {   // gelu(z) itself as well: the activation the next product's weight gradient needs
            float a[8];
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
              uint64_t v;
              upk(mul2(pk(g[j], g[j + 1]), gelu_grad2<true>(zv[j], zv[j + 1], v)), g[j], g[j + 1]);
              upk(v, a[j], a[j + 1]);
            }
            if (m < M) *reinterpret_cast<uint4*>(act + size_t(m) * N + size_t(cg) * 8) = pack8(a);
          } else {
            uint64_t unused;
#pragma unroll
            for (int j = 0; j < 8; j += 2) upk(mul2(pk(g[j], g[j + 1]), gelu_grad2<false>(zv[j], zv[j + 1], unused)), g[j], g[j + 1]);
          }
          if (dz != nullptr) {
            const uint4 packed = pack8(g);
            if (m < M) *reinterpret_cast<uint4*>(dz + size_t(m) * N + size_t(cg) * 8) = packed;
            if (q8 == nullptr) unpack8(packed, g);   // the bias gradient sums what the products will read
          }
        }
        if (q8 != nullptr) {   // the e5m2 operand of the 8-bit dgrad / wgrad products; the bias gradient sums these very numbers
          const uint2 pk = pack8_e5m2_roundtrip(g, q_inv, q_scale);
          if (m < M) *reinterpret_cast<uint2*>(q8 + size_t(m) * N + size_t(cg) * 8) = pk;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += g[j];   // rows past the end hold zeros
      }
    }
  }
  if (db == nullptr && strips == nullptr) return;
#pragma unroll
  for (int j = 0; j < 8; ++j) part[rl][cl][j] = acc[j];
  __syncthreads();
  // 256 threads <-> 256 columns of the CTA
  const int c = threadIdx.x;
  const int col = blockIdx.x * 256 + c;
  float t = 0.f;
  if (col < N) {
#pragma unroll
    for (int r = 0; r < kColLanes; ++r) t += part[r][c / 8][c % 8];
  }
  if (strips == nullptr) {
    if (col < N) atomicAdd(db + col, t);
    return;
  }
  if (col < N) strips[size_t(blockIdx.y) * N + col] = t;
  if (arrived == nullptr) return;   // many strips: a second pass adds them (waiting for this CTA's stores here would hold it up)
  // few: the CTA that comes last adds them, in strip order
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    s_last = atomicAdd(arrived + blockIdx.x, 1) == int(gridDim.y) - 1;
    if (s_last) arrived[blockIdx.x] = 0;   // as the next launch to get the counter expects it
  }
  __syncthreads();
  if (!s_last || col >= N) return;
  __threadfence();
  t = 0.f;
#pragma unroll 16
  for (unsigned r = 0; r < gridDim.y; ++r) t += strips[size_t(r) * N + col];
  st_param(db_out, db_dtype, col, t);
}

constexpr int kFewStrips = 32;
// db[n] = sum over the strips, in a fixed order: CTA = 32 columns x 32 strip lanes.
__global__ void __launch_bounds__(1024) strip_sum_kernel(const float* __restrict__ strips, int n_strips, int N, void* __restrict__ db, int db_dtype) {
  __shared__ float red[32][33];
  ptx::griddep_wait();
  ptx::griddep_launch();
  const int cl = threadIdx.x % 32, rl = threadIdx.x / 32, col = blockIdx.x * 32 + cl;
  float t = 0.f;
  if (col < N) {
#pragma unroll 8
    for (int r = rl; r < n_strips; r += 32) t += strips[size_t(r) * N + col];
  }
  red[rl][cl] = t;
  __syncthreads();
  if (rl == 0 && col < N) {
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < 32; ++k) sum += red[k][cl];
    st_param(db, db_dtype, col, sum);
  }
}

// ------------------------------------------------------------------------------------------------ QKV gradient pack
// g[(t * B + b)][which * E + h * D + d] = f(dsrc[which][b][h][t][d]), f = q scale and the transposed rotation for dq, dk;
// db[col] = sum over rows of g (the bias gradient of the fused projection) in the same pass.
// CTA = 32 column groups (8 columns each: 256 columns of g) x 8 row lanes over a strip of kColRows rows; a thread's column
// group — pathway third, head, 8 dimensions — is fixed, only (t, b) changes from row to row.
template <int D>
__global__ void __launch_bounds__(256) qkv_grad_pack_kernel(const __nv_bfloat16* __restrict__ dq, const __nv_bfloat16* __restrict__ dk,
                                                            const __nv_bfloat16* __restrict__ dv, __nv_bfloat16* __restrict__ g,
                                                            float* __restrict__ db, const float* __restrict__ cos_tab,
                                                            const float* __restrict__ sin_tab, const int32_t* __restrict__ row_map,
                                                            int M, int T, int B, int H, float q_scale) {
  __shared__ float part[kColLanes][32][8];
  constexpr int VPH = D / 8, hd = D / 2;             // vectors per head; rotation pairs dimension d with d + hd
  const int E = H * D, N = 3 * E;
  const int cl = threadIdx.x % 32, rl = threadIdx.x / 32;
  const int cg = blockIdx.x * 32 + cl;               // column group
  const bool live = cg * 8 < N;
  const int col = live ? cg * 8 : 0;
  const int which = col / E, e = col % E, h = e / D, dv8 = (e % D) / 8;
  const __nv_bfloat16* src = which == 0 ? dq : (which == 1 ? dk : dv);
  const bool rot = cos_tab != nullptr && which < 2;
  const bool upper = dv8 * 8 >= hd;
  const int pv = upper ? dv8 - VPH / 2 : dv8 + VPH / 2;   // the vector holding the partner dimensions
  const int f0 = upper ? dv8 * 8 - hd : dv8 * 8;
  const float scale = which == 0 ? q_scale : 1.f;
  const int m0 = blockIdx.y * kColRows, m1 = min(M, m0 + kColRows);
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (live) {
#pragma unroll 4
    for (int m = m0 + rl; m < m1; m += kColLanes) {
      const int mo = row_map != nullptr ? row_map[m] : m;   // packed rows: output row m is token mo = t * B + b
      const int t = mo / B, b = mo % B;
      const uint4* row = reinterpret_cast<const uint4*>(src + ((size_t(b) * H + h) * T + t) * D);
      float v[8];
      unpack8(__ldg(row + dv8), v);
      if (rot) {
        // y = R x rotated forward: y_lo = x_lo c - x_hi s, y_hi = x_hi c + x_lo s; the gradient takes the transpose:
        // dx_lo = dy_lo c + dy_hi s, dx_hi = dy_hi c - dy_lo s
        float o[8], c[8], sn[8];
        unpack8(__ldg(row + pv), o);
        const float4* c4 = reinterpret_cast<const float4*>(cos_tab + size_t(t) * hd + f0);
        const float4* s4 = reinterpret_cast<const float4*>(sin_tab + size_t(t) * hd + f0);
        *reinterpret_cast<float4*>(c) = __ldg(c4); *reinterpret_cast<float4*>(c + 4) = __ldg(c4 + 1);
        *reinterpret_cast<float4*>(sn) = __ldg(s4); *reinterpret_cast<float4*>(sn + 4) = __ldg(s4 + 1);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = upper ? v[j] * c[j] - o[j] * sn[j] : v[j] * c[j] + o[j] * sn[j];
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] *= scale;
      const uint4 packed = pack8(v);
      *reinterpret_cast<uint4*>(g + size_t(m) * N + col) = packed;
      unpack8(packed, v);   // the bias gradient sums what the products will read
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += v[j];
    }
  }
  if (db == nullptr) return;
#pragma unroll
  for (int j = 0; j < 8; ++j) part[rl][cl][j] = acc[j];
  __syncthreads();
  const int c = threadIdx.x;
  const int ocol = blockIdx.x * 256 + c;
  if (ocol < N) {
    float t = 0.f;
#pragma unroll
    for (int r = 0; r < kColLanes; ++r) t += part[r][c / 8][c % 8];
    atomicAdd(db + ocol, t);
  }
}

// ------------------------------------------------------------------------------------------------ LoRA operands
constexpr int kLoraMax = 8;   // projections per launch
struct LoraParams {
  const __nv_bfloat16* w[kLoraMax];   // W [out][in]
  const __nv_bfloat16 *delta, *b;     // B A [n][out][in], B [n][out][r]
  __nv_bfloat16* merged;              // [n][out][in]
  __nv_bfloat16* b_diag;              // [n][out][n r]: B of projection i in columns i r .. (i + 1) r, zeros elsewhere; may be null
  int n, out, in, r;
  float scaling;
};

// merged = W + scaling (B A), each step rounded to bf16 as the tensor expression rounds it, and b_diag, the B's as the operand of one
// product that forms g B of all projections (r a multiple of eight).  Eight values per thread; HBM-bound.
__global__ void __launch_bounds__(256) lora_operands_kernel(LoraParams p) {
  ptx::griddep_wait();
  ptx::griddep_launch();
  const size_t idx = size_t(blockIdx.x) * 256 + threadIdx.x;
  const size_t per_w = size_t(p.out) * p.in / 8, n_w = p.n * per_w;
  if (idx < n_w) {
    const size_t at = idx * 8;
    float w[8], d[8];
    unpack8(__ldg(reinterpret_cast<const uint4*>(p.w[idx / per_w]) + idx % per_w), w);
    unpack8(__ldg(reinterpret_cast<const uint4*>(p.delta + at)), d);
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] += __bfloat162float(__float2bfloat16_rn(p.scaling * d[j]));
    *reinterpret_cast<uint4*>(p.merged + at) = pack8(w);
  } else if (p.b_diag != nullptr) {
    const int nr = p.n * p.r;
    const size_t k = idx - n_w;
    if (k >= size_t(p.n) * p.out * nr / 8) return;
    const int row = int(k / (nr / 8)), c = int(k % (nr / 8)) * 8, i = row / p.out;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (c / p.r == i) v = __ldg(reinterpret_cast<const uint4*>(p.b + size_t(row) * p.r + c % p.r));
    *reinterpret_cast<uint4*>(p.b_diag + size_t(row) * nr + c) = v;
  }
}

int fail(const char* what, cudaError_t e) {
  set_error("%s: %s", what, cudaGetErrorString(e));
  return MINTB_ECUDA;
}

int ln_maxv(int E) { return E <= 512 ? 2 : (E <= 1280 ? 5 : (E <= 2560 ? 10 : 0)); }
// warps of a backward CTA: a thread per 16-byte vector of the row
int ln_bwd_warps(int E) { return E <= 512 ? 2 : (E <= 768 ? 3 : (E <= 1280 ? 5 : 10)); }

// Upper bound of the backward grid (sizes the partial-sum workspace); the launch takes min(this, 148 x resident CTAs per SM).
int ln_bwd_grid_max(int rows) {
  const int want = (rows + kLnBwdRows - 1) / kLnBwdRows;
  return want < 148 * 8 ? want : 148 * 8;
}

}  // namespace
}  // namespace mintb

extern "C" {

using namespace mintb;

int mintb_lora_operands(const void* const* w, const void* delta, const void* b, int n, int out, int in, int r, float scaling, void* merged,
                        void* b_diag, void* stream) {
  bool ok = w != nullptr && delta != nullptr && merged != nullptr && n > 0 && n <= kLoraMax && out > 0 && in > 0 && in % 8 == 0 &&
            (b_diag == nullptr || (b != nullptr && r > 0 && r % 8 == 0));
  LoraParams p{};
  for (int i = 0; ok && i < n; ++i) {
    p.w[i] = static_cast<const __nv_bfloat16*>(w[i]);
    ok = w[i] != nullptr && (reinterpret_cast<uintptr_t>(w[i]) & 15) == 0;
  }
  if (!ok) {
    set_error("mintb_lora_operands: 1 to 8 16-byte aligned weights, delta, merged, in a multiple of 8; b and r a multiple of 8 with b_diag");
    return MINTB_EINVAL;
  }
  p.delta = static_cast<const __nv_bfloat16*>(delta); p.b = static_cast<const __nv_bfloat16*>(b);
  p.merged = static_cast<__nv_bfloat16*>(merged); p.b_diag = static_cast<__nv_bfloat16*>(b_diag);
  p.n = n; p.out = out; p.in = in; p.r = r; p.scaling = scaling;
  const size_t vec = size_t(n) * out * in / 8 + (b_diag != nullptr ? size_t(n) * out * n * r / 8 : 0);
  const cudaError_t e = launch_dependent(lora_operands_kernel, dim3(unsigned((vec + 255) / 256)), dim3(256), 0, static_cast<cudaStream_t>(stream), p);
  count_launches(1);
  return e == cudaSuccess ? MINTB_OK : fail("mintb_lora_operands launch", e);
}

int mintb_add_layernorm_fwd_q(const void* x, const void* r, float a, float b, const void* gamma, const void* beta, int param_dtype,
                              void* s_out, void* y_out, float* stats, int rows, int E, float eps, void* q_out, float q_inv_scale,
                              void* stream) {
  if (x == nullptr || rows <= 0 || E <= 0 || (E % 8) != 0 || ln_maxv(E) == 0) {
    set_error("mintb_add_layernorm_fwd: x is required, rows > 0, E a multiple of 8 and at most 2560 (got rows %d, E %d)", rows, E);
    return x == nullptr || rows <= 0 || E <= 0 ? MINTB_EINVAL : MINTB_EUNSUPPORTED;
  }
  if ((gamma != nullptr && y_out == nullptr) || (gamma == nullptr && s_out == nullptr) ||
      (param_dtype != MINTB_F32 && param_dtype != MINTB_BF16)) {
    set_error("mintb_add_layernorm_fwd: y_out is required with gamma, s_out without; parameters are f32 or bf16");
    return MINTB_EINVAL;
  }
  LnParams p{};
  p.x = static_cast<const __nv_bfloat16*>(x); p.r = static_cast<const __nv_bfloat16*>(r);
  p.a = a; p.b = b; p.gamma = gamma; p.beta = beta; p.param_dtype = param_dtype;
  p.s_out = static_cast<__nv_bfloat16*>(s_out); p.y_out = static_cast<__nv_bfloat16*>(y_out);
  p.stats = reinterpret_cast<float2*>(stats); p.rows = rows; p.E = E; p.eps = eps;
  p.q_out = static_cast<__nv_fp8_storage_t*>(q_out); p.q_inv = q_inv_scale;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int want = (rows + kLnWarps - 1) / kLnWarps;
  const int grid = want < 148 * 16 ? want : 148 * 16;   // rows are walked with a grid stride
  void (*kern)(LnParams);
  switch (ln_maxv(E)) {
    case 2: kern = r != nullptr ? add_layernorm_fwd_kernel<2, true> : add_layernorm_fwd_kernel<2, false>; break;
    case 5: kern = r != nullptr ? add_layernorm_fwd_kernel<5, true> : add_layernorm_fwd_kernel<5, false>; break;
    default: kern = r != nullptr ? add_layernorm_fwd_kernel<10, true> : add_layernorm_fwd_kernel<10, false>; break;
  }
  const cudaError_t e = launch_dependent(kern, dim3(grid), dim3(kLnWarps * 32), 0, st, p);
  count_launches(1);
  return e == cudaSuccess ? MINTB_OK : fail("mintb_add_layernorm_fwd launch", e);
}

int mintb_add_layernorm_fwd(const void* x, const void* r, float a, float b, const void* gamma, const void* beta, int param_dtype,
                            void* s_out, void* y_out, float* stats, int rows, int E, float eps, void* stream) {
  return mintb_add_layernorm_fwd_q(x, r, a, b, gamma, beta, param_dtype, s_out, y_out, stats, rows, E, eps, nullptr, 1.f, stream);
}

size_t mintb_add_layernorm_bwd_workspace_bytes(int rows, int E) {
  if (rows <= 0 || E <= 0) return 0;
  return align256(size_t(ln_bwd_grid_max(rows)) * 2 * E * sizeof(float));
}

int mintb_add_layernorm_bwd(const void* dy, const void* ds_in, const void* x, const void* r, float a, float b, const void* gamma,
                            int param_dtype, const float* stats, void* dx, void* dr, float* dgamma, float* dbeta, void* workspace,
                            size_t workspace_bytes, int rows, int E, void* stream) {
  return mintb_add_layernorm_bwd_typed(dy, ds_in, 0, x, r, a, b, gamma, param_dtype, stats, dx, dr, dgamma, dbeta, MINTB_F32, workspace, workspace_bytes, rows, E,
                                       stream);
}

int mintb_add_layernorm_bwd_typed(const void* dy, const void* ds_in, int ds_apart, const void* x, const void* r, float a, float b, const void* gamma,
                                  int param_dtype, const float* stats, void* dx, void* dr, void* dgamma, void* dbeta, int grad_dtype, void* workspace,
                                  size_t workspace_bytes, int rows, int E, void* stream) {
  if (rows <= 0 || E <= 0 || (E % 8) != 0 || ln_maxv(E) == 0) {
    set_error("mintb_add_layernorm_bwd: rows > 0, E a multiple of 8 and at most 2560 (got rows %d, E %d)", rows, E);
    return rows <= 0 || E <= 0 ? MINTB_EINVAL : MINTB_EUNSUPPORTED;
  }
  const bool norm = gamma != nullptr;
  if (dx == nullptr || (norm && (dy == nullptr || x == nullptr || stats == nullptr || (dgamma == nullptr) != (dbeta == nullptr))) ||
      (!norm && ds_in == nullptr)) {
    set_error("mintb_add_layernorm_bwd: missing pointer (with gamma: dy, x, stats, dgamma and dbeta or neither; without: ds_in; always dx)");
    return MINTB_EINVAL;
  }
  const bool param_grads = norm && dgamma != nullptr;   // frozen parameters: no partial sums, no second pass
  if (param_grads && (workspace == nullptr || workspace_bytes < mintb_add_layernorm_bwd_workspace_bytes(rows, E))) {
    set_error("mintb_add_layernorm_bwd: workspace of %zu bytes required", mintb_add_layernorm_bwd_workspace_bytes(rows, E));
    return MINTB_EWORKSPACE;
  }
  LnParams p{};
  p.x = static_cast<const __nv_bfloat16*>(x); p.r = static_cast<const __nv_bfloat16*>(r);
  p.a = a; p.b = b; p.gamma = gamma; p.param_dtype = param_dtype;
  p.stats = const_cast<float2*>(reinterpret_cast<const float2*>(stats));
  p.dy = static_cast<const __nv_bfloat16*>(dy); p.ds_in = static_cast<const __nv_bfloat16*>(ds_in); p.ds_apart = ds_apart;
  p.dx = static_cast<__nv_bfloat16*>(dx); p.dr = static_cast<__nv_bfloat16*>(dr);
  p.partial = param_grads ? static_cast<float*>(workspace) : nullptr; p.rows = rows; p.E = E;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // one 16-byte vector of the row per thread; ONE wave of CTAs, each walking its share of the rows
  if (!norm) {
    const size_t n_vec = size_t(rows) * E / 8;
    const cudaError_t err = launch_dependent(scaled_copies_kernel, dim3(unsigned((n_vec + 255) / 256)), dim3(256), 0, st, p, n_vec);
    count_launches(1);
    return err == cudaSuccess ? MINTB_OK : fail("mintb_add_layernorm_bwd launch", err);
  }
  const int nw = ln_bwd_warps(E);
  const int per_sm = nw == 2 ? 8 : (nw == 3 ? 5 : (nw == 5 ? MINTB_LN_BWD_PER_SM : 1));
  const int grid_max = ln_bwd_grid_max(rows);
  const int grid = grid_max < 148 * per_sm ? grid_max : 148 * per_sm;
  auto pick = [&](auto nw_c, auto minb_c) -> void (*)(LnParams) {
    constexpr int NW = decltype(nw_c)::value, MINB = decltype(minb_c)::value;
    const bool hr = r != nullptr, hd = ds_in != nullptr;
    if (param_grads) return hr ? (hd ? add_layernorm_bwd_kernel<NW, MINB, true, true, true> : add_layernorm_bwd_kernel<NW, MINB, true, false, true>)
                               : (hd ? add_layernorm_bwd_kernel<NW, MINB, false, true, true> : add_layernorm_bwd_kernel<NW, MINB, false, false, true>);
    return hr ? (hd ? add_layernorm_bwd_kernel<NW, MINB, true, true, false> : add_layernorm_bwd_kernel<NW, MINB, true, false, false>)
              : (hd ? add_layernorm_bwd_kernel<NW, MINB, false, true, false> : add_layernorm_bwd_kernel<NW, MINB, false, false, false>);
  };
  using std::integral_constant;
  void (*kern)(LnParams) = nw == 2 ? pick(integral_constant<int, 2>(), integral_constant<int, 8>())
                         : nw == 3 ? pick(integral_constant<int, 3>(), integral_constant<int, 5>())
                         : nw == 5 ? pick(integral_constant<int, 5>(), integral_constant<int, MINTB_LN_BWD_PER_SM>())
                                   : pick(integral_constant<int, 10>(), integral_constant<int, 1>());
  cudaError_t e = launch_dependent(kern, dim3(grid), dim3(nw * 32), 0, st, p);
  count_launches(1);
  if (e == cudaSuccess && param_grads) {
    e = launch_dependent(ln_param_grad_kernel, dim3((2 * E + 31) / 32), dim3(1024), 0, st, p.partial, grid, E, dgamma, dbeta, grad_dtype);
    count_launches(1);
  }
  return e == cudaSuccess ? MINTB_OK : fail("mintb_add_layernorm_bwd launch", e);
}

static int gelu_bwd_colsum(const void* dy, const void* z, void* dz, void* act, void* db, int db_dtype, void* dz_e5m2, float e5m2_scale, void* workspace,
                           size_t workspace_bytes, int M, int N, void* stream) {
  if (dy == nullptr || M <= 0 || N <= 0 || (N % 8) != 0 || (z != nullptr && dz == nullptr && dz_e5m2 == nullptr) ||
      (z == nullptr && db == nullptr && dz_e5m2 == nullptr) || (z == nullptr && act != nullptr) || (dz_e5m2 != nullptr && !(e5m2_scale > 0.f))) {
    set_error("mintb_gelu_bwd_colsum: dy required, N a multiple of 8, a result to write (dz / dz_e5m2 with z, db / dz_e5m2 without), "
              "act only with z, a positive e5m2_scale with dz_e5m2");
    return MINTB_EINVAL;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const dim3 grid((N + 255) / 256, (M + kSumRows - 1) / kSumRows);
  float *acc = nullptr, *strips = nullptr;
  int* arrived = nullptr;
  if (db != nullptr && workspace != nullptr) {
    if (workspace_bytes < mintb_bias_grad_workspace_bytes(M, N)) {
      set_error("mintb_gelu_bwd_bias: workspace of %zu bytes required", mintb_bias_grad_workspace_bytes(M, N));
      return MINTB_EWORKSPACE;
    }
    strips = static_cast<float*>(workspace);
    if (int(grid.y) <= kFewStrips) {
      if (int rc = next_arrival_counters(int(grid.x), &arrived); rc != MINTB_OK) return rc;
    }
  } else if (db != nullptr) {
    acc = static_cast<float*>(db);
    cudaError_t e = cudaMemsetAsync(db, 0, size_t(N) * sizeof(float), st);
    if (e != cudaSuccess) return fail("mintb_gelu_bwd_colsum memset", e);
  }
  __nv_fp8_storage_t* q8 = static_cast<__nv_fp8_storage_t*>(dz_e5m2);
  const float q_inv = q8 != nullptr ? 1.f / e5m2_scale : 1.f, q_scale = q8 != nullptr ? e5m2_scale : 1.f;
  cudaError_t e = launch_dependent(z != nullptr ? gelu_bwd_colsum_kernel<true> : gelu_bwd_colsum_kernel<false>, grid, dim3(256), 0, st,
                                         static_cast<const __nv_bfloat16*>(dy), static_cast<const __nv_bfloat16*>(z), static_cast<__nv_bfloat16*>(dz), acc, M, N,
                                         static_cast<__nv_bfloat16*>(act), q8, q_inv, q_scale, strips, arrived, db, db_dtype);
  count_launches(1);
  if (e == cudaSuccess && strips != nullptr && arrived == nullptr) {
    e = launch_dependent(strip_sum_kernel, dim3((N + 31) / 32), dim3(1024), 0, st, static_cast<const float*>(strips), int(grid.y), N, db, db_dtype);
    count_launches(1);
  }
  return e == cudaSuccess ? MINTB_OK : fail("mintb_gelu_bwd_colsum launch", e);
}

int mintb_gelu_bwd_colsum_f8(const void* dy, const void* z, void* dz, void* act, float* db, void* dz_e5m2, float e5m2_scale, int M,
                             int N, void* stream) {
  return gelu_bwd_colsum(dy, z, dz, act, db, MINTB_F32, dz_e5m2, e5m2_scale, nullptr, 0, M, N, stream);
}

size_t mintb_bias_grad_workspace_bytes(int M, int N) {
  return M <= 0 || N <= 0 ? 0 : align256(size_t((M + kSumRows - 1) / kSumRows) * N * sizeof(float));
}

int mintb_gelu_bwd_bias(const void* dy, const void* z, void* dz, void* db, int db_dtype, void* dz_e5m2, float e5m2_scale, void* workspace,
                        size_t workspace_bytes, int M, int N, void* stream) {
  if (db != nullptr && (workspace == nullptr || (db_dtype != MINTB_F32 && db_dtype != MINTB_BF16))) {
    set_error("mintb_gelu_bwd_bias: a bias gradient is f32 or bf16 and needs the workspace");
    return MINTB_EINVAL;
  }
  return gelu_bwd_colsum(dy, z, dz, nullptr, db, db_dtype, dz_e5m2, e5m2_scale, workspace, workspace_bytes, M, N, stream);
}

int mintb_gelu_bwd_colsum_act(const void* dy, const void* z, void* dz, void* act, float* db, int M, int N, void* stream) {
  if ((z != nullptr && dz == nullptr) || (z == nullptr && db == nullptr)) {
    set_error("mintb_gelu_bwd_colsum: dy required, N a multiple of 8, dz with z, db without z, act only with z");
    return MINTB_EINVAL;
  }
  return mintb_gelu_bwd_colsum_f8(dy, z, dz, act, db, nullptr, 1.f, M, N, stream);
}

int mintb_gelu_bwd_colsum(const void* dy, const void* z, void* dz, float* db, int M, int N, void* stream) {
  return mintb_gelu_bwd_colsum_act(dy, z, dz, nullptr, db, M, N, stream);
}

int mintb_qkv_grad_pack(const void* dq, const void* dk, const void* dv, void* g, float* db, const float* rope_cos,
                        const float* rope_sin, const int32_t* row_map, int n_rows, int T, int B, int H, int D, float q_scale,
                        void* stream) {
  if (dq == nullptr || dk == nullptr || dv == nullptr || g == nullptr || T <= 0 || B <= 0 || H <= 0 ||
      (rope_cos == nullptr) != (rope_sin == nullptr)) {
    set_error("mintb_qkv_grad_pack: null pointer or non-positive size");
    return MINTB_EINVAL;
  }
  if (D != 16 && D != 32 && D != 64) {
    set_error("mintb_qkv_grad_pack: head_dim %d is not one of 16, 32, 64", D);
    return MINTB_EUNSUPPORTED;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int N = 3 * H * D, M = row_map != nullptr ? n_rows : T * B;
  if (M <= 0) {
    set_error("mintb_qkv_grad_pack: no rows");
    return MINTB_EINVAL;
  }
  if (db != nullptr) {
    cudaError_t e = cudaMemsetAsync(db, 0, size_t(N) * sizeof(float), st);
    if (e != cudaSuccess) return fail("mintb_qkv_grad_pack memset", e);
  }
  dim3 grid((N + 255) / 256, (M + kColRows - 1) / kColRows);
  const __nv_bfloat16 *q = static_cast<const __nv_bfloat16*>(dq), *k = static_cast<const __nv_bfloat16*>(dk),
                      *v = static_cast<const __nv_bfloat16*>(dv);
  __nv_bfloat16* o = static_cast<__nv_bfloat16*>(g);
  switch (D) {
    case 16: qkv_grad_pack_kernel<16><<<grid, 256, 0, st>>>(q, k, v, o, db, rope_cos, rope_sin, row_map, M, T, B, H, q_scale); break;
    case 32: qkv_grad_pack_kernel<32><<<grid, 256, 0, st>>>(q, k, v, o, db, rope_cos, rope_sin, row_map, M, T, B, H, q_scale); break;
    default: qkv_grad_pack_kernel<64><<<grid, 256, 0, st>>>(q, k, v, o, db, rope_cos, rope_sin, row_map, M, T, B, H, q_scale); break;
  }
  count_launches(1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MINTB_OK : fail("mintb_qkv_grad_pack launch", e);
}

}  // extern "C"
