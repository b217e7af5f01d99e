// Mask metadata and RoPE tables: small memory-bound kernels run once per batch.
#include "ptx.cuh"
#include "rope.cuh"

namespace mintb {

// All of the metadata from chain ids in one pass.  A CTA of eight warps owns 64 query rows of one sample, a warp every eighth of
// them; lane l of a warp holds word l of a group of 32.  A word of a row is one ballot over the 32 chain ids it covers, and rows of
// one chain share their words, so a warp forms them once per chain that it meets and otherwise only writes: bound by the two
// copies of the bits (B16 T2048: 34 MB, 245 us with 32 compares per thread and word, three launches and two casts before; 12 us).
// The relation is symmetric, so the key-major copy (bitsT) holds the same words.
template <typename Id>
__device__ __forceinline__ void meta_rows(int b, int qt, const Id* __restrict__ chain_ids, const uint8_t* __restrict__ key_pad, uint32_t* __restrict__ bits,
                                          uint32_t* __restrict__ bitsT, uint32_t* __restrict__ kpad, uint8_t* __restrict__ cls, int T, int TW, int NT) {
  __shared__ uint32_t s_seen[2][32];   // of the word group: keys that some row of the tile meets in its own / in another chain
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  chain_ids += size_t(b) * T;
  for (int w0 = 0; w0 < TW; w0 += 32) {
    const int nw = min(32, TW - w0);
    if (threadIdx.x < 64) s_seen[threadIdx.x / 32][lane] = 0;
    __syncthreads();
    uint32_t pad = 0xffffffffu;
#pragma unroll 8
    for (int w = 0; w < nw; ++w) {
      const int j = (w0 + w) * 32 + lane;
      const uint32_t v = __ballot_sync(0xffffffffu, j >= T || (key_pad != nullptr && key_pad[size_t(b) * T + j] != 0));
      if (lane == w) pad = v;
    }
    uint32_t word = 0, intra = 0, inter = 0;
    int chain = 0;
    bool have = false;
    for (int r = warp; r < kClassTile; r += 8) {
      const int i = qt * kClassTile + r;
      if (i >= T) break;
      const int ci = int(chain_ids[i]);
      if (!have || ci != chain) {
        have = true;
        chain = ci;
#pragma unroll 8
        for (int w = 0; w < nw; ++w) {
          const int j = (w0 + w) * 32 + lane;
          const uint32_t v = __ballot_sync(0xffffffffu, j < T && int(chain_ids[j]) != ci);
          if (lane == w) word = v;
        }
        inter |= word & ~pad;
        intra |= ~word & ~pad;
      }
      if (lane < nw) {
        const size_t at = (size_t(b) * T + i) * TW + w0 + lane;
        bits[at] = word;
        bitsT[at] = word;
      }
    }
    if (intra) atomicOr(&s_seen[0][lane], intra);
    if (inter) atomicOr(&s_seen[1][lane], inter);
    if (qt == 0 && warp == 0 && lane < nw) kpad[size_t(b) * TW + w0 + lane] = pad;
    __syncthreads();
    if (warp == 0) {   // two words make a 64-key tile; a group starts on a tile boundary
      const uint32_t pad_next = __shfl_down_sync(0xffffffffu, pad, 1);
      const int kt = (w0 + lane) / 2;
      if (lane % 2 == 0 && kt < NT)
        cls[(size_t(b) * NT + qt) * NT + kt] = uint8_t(((s_seen[0][lane] | s_seen[0][lane + 1]) ? kHasIntra : 0) |
                                                       ((s_seen[1][lane] | s_seen[1][lane + 1]) ? kHasInter : 0) | ((pad | pad_next) ? kHasPad : 0));
    }
    __syncthreads();
  }
}

template <typename Id>
__global__ void __launch_bounds__(256) meta_from_chain_ids_kernel(const Id* __restrict__ chain_ids, const uint8_t* __restrict__ key_pad,
                                                                  uint32_t* __restrict__ bits, uint32_t* __restrict__ bitsT, uint32_t* __restrict__ kpad,
                                                                  uint8_t* __restrict__ cls, int T, int TW, int NT) {
  meta_rows(blockIdx.x, blockIdx.y, chain_ids, key_pad, bits, bitsT, kpad, cls, T, TW, NT);
}

// The same with the rotation of the self pathway's Q and K, by further CTAs of the launch: what an attention call on chain ids and raw
// projections has to have done before it starts.  For short pairs, where a launch is what either costs (B1 H20 T187 D16: 18.6 us a call with
// two, 14.7 with one).
template <typename Id>
__global__ void __launch_bounds__(256) prepare_kernel(const Id* __restrict__ chain_ids, const uint8_t* __restrict__ key_pad, uint32_t* __restrict__ bits,
                                                      uint32_t* __restrict__ bitsT, uint32_t* __restrict__ kpad, uint8_t* __restrict__ cls, int B, int T, int TW, int NT,
                                                      const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k, __nv_bfloat16* __restrict__ qr,
                                                      __nv_bfloat16* __restrict__ kr, const float* __restrict__ cos_tab, const float* __restrict__ sin_tab, size_t rows, int D) {
  ptx::griddep_wait();
  ptx::griddep_launch();
  const unsigned n = unsigned(B) * NT;
  if (blockIdx.x < n) meta_rows(int(blockIdx.x) % B, int(blockIdx.x) / B, chain_ids, key_pad, bits, bitsT, kpad, cls, T, TW, NT);
  else rope_rotate_part(size_t(blockIdx.x - n) * blockDim.x + threadIdx.x, q, k, qr, kr, cos_tab, sin_tab, rows, T, D);
}

// Arbitrary (B,T,T) mask: row-major words, and the transposed relation for the key-major copy.
__global__ void meta_bits_from_mask(const uint8_t* __restrict__ mask, uint32_t* __restrict__ bits,
                                    uint32_t* __restrict__ bitsT, int B, int T, int TW) {
  size_t idx = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  size_t total = size_t(B) * T * TW;
  if (idx >= total) return;
  int w = int(idx % TW);
  size_t bi = idx / TW;
  int i = int(bi % T);
  int b = int(bi / T);
  const uint8_t* m = mask + size_t(b) * T * T;
  uint32_t word = 0, wordT = 0;
  int j0 = w * 32;
  for (int jj = 0; jj < 32; ++jj) {
    int j = j0 + jj;
    if (j < T) {
      if (m[size_t(i) * T + j]) word |= (1u << jj);
      if (m[size_t(j) * T + i]) wordT |= (1u << jj);  // row i of bitsT is KEY i; bit jj is QUERY j
    }
  }
  bits[idx] = word;
  bitsT[idx] = wordT;
}

__global__ void meta_kpad(const uint8_t* __restrict__ key_pad, uint32_t* __restrict__ kpad, int B, int T, int TW) {
  int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= B * TW) return;
  int w = idx % TW, b = idx / TW;
  uint32_t word = 0;
  for (int jj = 0; jj < 32; ++jj) {
    int j = w * 32 + jj;
    bool padded = (j >= T) || (key_pad != nullptr && key_pad[size_t(b) * T + j] != 0);
    if (padded) word |= (1u << jj);
  }
  kpad[idx] = word;
}

// One warp per 64x64 tile: lanes stride over the 64 query rows, two words per row.
__global__ void meta_tile_class(const uint32_t* __restrict__ bits, const uint32_t* __restrict__ kpad,
                                uint8_t* __restrict__ cls, int B, int T, int TW, int NT) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
  int lane = threadIdx.x % 32;
  if (warp >= B * NT * NT) return;
  int kt = warp % NT, qt = (warp / NT) % NT, b = warp / (NT * NT);
  uint32_t pad0 = kpad[size_t(b) * TW + 2 * kt], pad1 = kpad[size_t(b) * TW + 2 * kt + 1];
  uint32_t intra = 0, inter = 0;
  for (int r = lane; r < kClassTile; r += 32) {
    int i = qt * kClassTile + r;
    if (i < T) {
      const uint32_t* row = bits + (size_t(b) * T + i) * TW + 2 * kt;
      uint32_t w0 = row[0], w1 = row[1];
      inter |= (w0 & ~pad0) | (w1 & ~pad1);
      intra |= (~w0 & ~pad0) | (~w1 & ~pad1);
    }
  }
  intra = __reduce_or_sync(0xffffffffu, intra);
  inter = __reduce_or_sync(0xffffffffu, inter);
  if (lane == 0) {
    uint8_t c = 0;
    if (intra) c |= kHasIntra;
    if (inter) c |= kHasInter;
    if (pad0 | pad1) c |= kHasPad;
    cls[warp] = c;
  }
}

static cudaError_t finish_meta(const uint8_t* key_pad, void* meta, int B, int T, cudaStream_t s) {
  MetaLayout L = meta_layout(B, T);
  char* p = static_cast<char*>(meta);
  uint32_t* bits = reinterpret_cast<uint32_t*>(p + L.off_bits);
  uint32_t* kpad = reinterpret_cast<uint32_t*>(p + L.off_kpad);
  uint8_t* cls = reinterpret_cast<uint8_t*>(p + L.off_cls);
  meta_kpad<<<(B * L.TW + 127) / 128, 128, 0, s>>>(key_pad, kpad, B, T, L.TW);
  int warps = B * L.NT * L.NT;
  meta_tile_class<<<(warps * 32 + 127) / 128, 128, 0, s>>>(bits, kpad, cls, B, T, L.TW, L.NT);
  count_launches(3);  // bits + kpad + class
  return cudaGetLastError();
}

cudaError_t launch_meta_from_chain_ids(const void* chain_ids, bool ids64, const uint8_t* key_pad, void* meta, int B, int T, cudaStream_t s) {
  MetaLayout L = meta_layout(B, T);
  char* p = static_cast<char*>(meta);
  uint32_t* bits = reinterpret_cast<uint32_t*>(p + L.off_bits);
  uint32_t* bitsT = reinterpret_cast<uint32_t*>(p + L.off_bitsT);
  uint32_t* kpad = reinterpret_cast<uint32_t*>(p + L.off_kpad);
  uint8_t* cls = reinterpret_cast<uint8_t*>(p + L.off_cls);
  const dim3 grid(B, L.NT);
  if (ids64)
    meta_from_chain_ids_kernel<long long><<<grid, 256, 0, s>>>(static_cast<const long long*>(chain_ids), key_pad, bits, bitsT, kpad, cls, T, L.TW, L.NT);
  else
    meta_from_chain_ids_kernel<int32_t><<<grid, 256, 0, s>>>(static_cast<const int32_t*>(chain_ids), key_pad, bits, bitsT, kpad, cls, T, L.TW, L.NT);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_prepare(const AttnArgs& a, __nv_bfloat16* qr, __nv_bfloat16* kr) {
  const MetaLayout L = meta_layout(a.B, a.T);
  char* p = static_cast<char*>(a.meta_buf);
  uint32_t* bits = reinterpret_cast<uint32_t*>(p + L.off_bits);
  uint32_t* bitsT = reinterpret_cast<uint32_t*>(p + L.off_bitsT);
  uint32_t* kpad = reinterpret_cast<uint32_t*>(p + L.off_kpad);
  uint8_t* cls = reinterpret_cast<uint8_t*>(p + L.off_cls);
  const size_t rows = size_t(a.B) * a.H * a.T, parts = rows * (a.D / 16);
  const dim3 grid(unsigned(a.B) * L.NT + unsigned((parts + 255) / 256));
  auto launch = [&](auto kern, auto ids) {
    return launch_dependent(kern, grid, dim3(256), 0, a.stream, ids, a.key_pad, bits, bitsT, kpad, cls, a.B, a.T, L.TW, L.NT, static_cast<const __nv_bfloat16*>(a.q_s),
                            static_cast<const __nv_bfloat16*>(a.k_s), qr, kr, a.rope_cos, a.rope_sin, rows, a.D);
  };
  const cudaError_t e = a.ids64 ? launch(prepare_kernel<long long>, static_cast<const long long*>(a.chain_ids))
                                : launch(prepare_kernel<int32_t>, static_cast<const int32_t*>(a.chain_ids));
  count_launches(1);
  return e == cudaSuccess ? cudaGetLastError() : e;
}

cudaError_t launch_meta_from_mask(const uint8_t* mask, const uint8_t* key_pad, void* meta, int B, int T,
                                  cudaStream_t s) {
  MetaLayout L = meta_layout(B, T);
  char* p = static_cast<char*>(meta);
  size_t total = size_t(B) * T * L.TW;
  meta_bits_from_mask<<<unsigned((total + 255) / 256), 256, 0, s>>>(
      mask, reinterpret_cast<uint32_t*>(p + L.off_bits), reinterpret_cast<uint32_t*>(p + L.off_bitsT), B, T, L.TW);
  return finish_meta(key_pad, meta, B, T, s);
}

// cos/sin of float(position) * inv_freq[i], full-range accurate cosf/sinf (arguments reach ~T radians).
__global__ void rope_tables_kernel(const float* __restrict__ inv_freq, float* __restrict__ cos_tab,
                                   float* __restrict__ sin_tab, int T, int half) {
  int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= T * half) return;
  int i = idx % half, t = idx / half;
  float ang = __fmul_rn(float(t), inv_freq[i]);
  cos_tab[idx] = cosf(ang);
  sin_tab[idx] = sinf(ang);
}

cudaError_t launch_rope_tables(const float* inv_freq, float* cos_tab, float* sin_tab, int T, int D, cudaStream_t s) {
  int n = T * (D / 2);
  rope_tables_kernel<<<(n + 255) / 256, 256, 0, s>>>(inv_freq, cos_tab, sin_tab, T, D / 2);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace mintb
