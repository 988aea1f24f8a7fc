// Small row kernels around multi-head latent attention (MLA):
//   mla_prep:   from the fused projection row [q_a (q_lora) | c_kv (512) | k_rope (64)]:
//               q_a -> RMSNorm (learned gain) -> qa_out;  c_kv -> RMSNorm (learned gain) and k_rope -> split-half RoPE,
//               both written to the latent cache slot of the row ([c_kv_normed (512) | k_rope (64)]).
//   mla_q_rope: RoPE on the 64-dim rope part of every query head, written behind the absorbed 512 latent dims of
//               q_full[T, H, 576].
// Math of the reference MLA: src/models/k3/mla.rs:49-63,102-111 (eps 1e-6 inside MLA; the reference runs NoPE and an
// expanded cache — `inv_freq == nullptr` gives NoPE here, the latent cache is this build's).
#include "common.cuh"
#include "host_utils.h"

using namespace mary;

namespace {

__device__ __forceinline__ float block_sum_256(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (l < (blockDim.x >> 5)) ? red[l] : 0.f;
  t = warp_sum(t);
  __syncthreads();
  return t;
}

__global__ void mla_prep_kernel(const __nv_bfloat16* __restrict__ qakv, int64_t ld, int q_lora, const __nv_bfloat16* __restrict__ w_qa,
                                const __nv_bfloat16* __restrict__ w_kv, const float* __restrict__ inv_freq, const int* __restrict__ positions,
                                const int64_t* __restrict__ slots, __nv_bfloat16* __restrict__ qa_out, __nv_bfloat16* __restrict__ cache,
                                float eps, int64_t n_slots, int* __restrict__ status) {
  pdl_sync();
  __shared__ float red[32];
  const int t = blockIdx.x;
  const __nv_bfloat16* row = qakv + (int64_t)t * ld;
  // q_a norm
  float ss = 0.f;
  for (int i = threadIdx.x; i < q_lora; i += blockDim.x) { float v = __bfloat162float(row[i]); ss += v * v; }
  const float inv_q = rsqrtf(block_sum_256(ss, red) / q_lora + eps);
  for (int i = threadIdx.x; i < q_lora; i += blockDim.x)
    qa_out[(int64_t)t * q_lora + i] = __float2bfloat16(__bfloat162float(row[i]) * inv_q * __bfloat162float(w_qa[i]));
  // latent norm
  const __nv_bfloat16* ckv = row + q_lora;
  ss = 0.f;
  for (int i = threadIdx.x; i < 512; i += blockDim.x) { float v = __bfloat162float(ckv[i]); ss += v * v; }
  const float inv_k = rsqrtf(block_sum_256(ss, red) / 512 + eps);
  if (n_slots > 0 && (slots[t] < 0 || slots[t] >= n_slots)) {                 // a cache slot outside the cache: record it, skip the write
    if (threadIdx.x == 0) atomicCAS(status, 0, (int)MARY_ERR_BOUNDS);
    return;
  }
  __nv_bfloat16* dst = cache + slots[t] * 576;
  for (int i = threadIdx.x; i < 512; i += blockDim.x)
    dst[i] = __float2bfloat16(__bfloat162float(ckv[i]) * inv_k * __bfloat162float(w_kv[i]));
  // rope on the 64 carried dims (split-half pairs (i, i + 32))
  if (threadIdx.x < 32) {
    const int i = threadIdx.x;
    float a = __bfloat162float(ckv[512 + i]), b = __bfloat162float(ckv[512 + 32 + i]);
    if (inv_freq) {
      float s, c;
      sincosf((float)positions[t] * inv_freq[i], &s, &c);
      const float ra = a * c - b * s, rb = a * s + b * c;
      a = ra; b = rb;
    }
    dst[512 + i] = __float2bfloat16(a);
    dst[512 + 32 + i] = __float2bfloat16(b);
  }
}

// The same for 16-byte aligned rows with q_lora % 8 == 0 and q_lora <= 6144: warps 0-5 own the q_a part, warps 6-7 the latent, everything in registers
// after one load, both sums behind one barrier (4096 rows of 2112: 25 us by 2-byte accesses and four barriers, 10 us so).
constexpr int PREP_Q = 192, PREP_CH = 4;
__device__ __forceinline__ void wide8(const uint4& v, float* f) {
  const __nv_bfloat162* h = (const __nv_bfloat162*)&v;
#pragma unroll
  for (int j = 0; j < 4; ++j) { const float2 t = __bfloat1622float2(h[j]); f[2 * j] = t.x; f[2 * j + 1] = t.y; }
}
__device__ __forceinline__ uint4 scaled8(const uint4& v, const uint4& w, float inv) {
  float f[8], g[8];
  wide8(v, f);
  wide8(w, g);
  uint4 o;
  __nv_bfloat162* h = (__nv_bfloat162*)&o;
#pragma unroll
  for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(f[2 * j] * inv * g[2 * j], f[2 * j + 1] * inv * g[2 * j + 1]);
  return o;
}
__device__ __forceinline__ float squares8(const uint4& v) {
  float f[8], ss = 0.f;
  wide8(v, f);
#pragma unroll
  for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
  return ss;
}

__global__ void __launch_bounds__(256)
mla_prep_rows_kernel(const __nv_bfloat16* __restrict__ qakv, int64_t ld, int q_lora, const __nv_bfloat16* __restrict__ w_qa,
                     const __nv_bfloat16* __restrict__ w_kv, const float* __restrict__ inv_freq, const int* __restrict__ positions,
                     const int64_t* __restrict__ slots, __nv_bfloat16* __restrict__ qa_out, __nv_bfloat16* __restrict__ cache, float eps, int64_t n_slots,
                     int* __restrict__ status) {
  pdl_sync();
  __shared__ float red[8];
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const __nv_bfloat16* row = qakv + (int64_t)t * ld;
  const __nv_bfloat16* ckv = row + q_lora;
  const bool is_q = threadIdx.x < PREP_Q;
  const int kv_at = ((int)threadIdx.x - PREP_Q) * 8;               // of the other 64 threads
  uint4 v[PREP_CH], w[PREP_CH];
  float ss = 0.f;
  if (is_q) {
#pragma unroll
    for (int c = 0; c < PREP_CH; ++c) {
      const int i = (threadIdx.x + c * PREP_Q) * 8;
      if (i < q_lora) { v[c] = *(const uint4*)(row + i); w[c] = *(const uint4*)(w_qa + i); }
    }
#pragma unroll
    for (int c = 0; c < PREP_CH; ++c) if ((int)(threadIdx.x + c * PREP_Q) * 8 < q_lora) ss += squares8(v[c]);
  } else {
    v[0] = *(const uint4*)(ckv + kv_at);
    w[0] = *(const uint4*)(w_kv + kv_at);
    ss = squares8(v[0]);
  }
  float ra = 0.f, rb = 0.f;                                         // warp 7: rope on the 64 carried dims (split-half pairs (i, i + 32))
  if (warp == 7) {
    ra = __bfloat162float(ckv[512 + lane]); rb = __bfloat162float(ckv[512 + 32 + lane]);
    if (inv_freq) {
      float s, c;
      sincosf((float)positions[t] * inv_freq[lane], &s, &c);
      const float x = ra * c - rb * s, y = ra * s + rb * c;
      ra = x; rb = y;
    }
  }
  const int64_t slot = slots[t];
  ss = warp_sum(ss);
  if (lane == 0) red[warp] = ss;
  __syncthreads();
  if (is_q) {
    const float inv = rsqrtf((red[0] + red[1] + red[2] + red[3] + red[4] + red[5]) / q_lora + eps);
#pragma unroll
    for (int c = 0; c < PREP_CH; ++c) {
      const int i = (threadIdx.x + c * PREP_Q) * 8;
      if (i < q_lora) *(uint4*)(qa_out + (int64_t)t * q_lora + i) = scaled8(v[c], w[c], inv);
    }
    return;
  }
  if (n_slots > 0 && (slot < 0 || slot >= n_slots)) {               // a cache slot outside the cache: record it, skip the write
    if (threadIdx.x == PREP_Q) atomicCAS(status, 0, (int)MARY_ERR_BOUNDS);
    return;
  }
  __nv_bfloat16* dst = cache + slot * 576;
  *(uint4*)(dst + kv_at) = scaled8(v[0], w[0], rsqrtf((red[6] + red[7]) / 512 + eps));
  if (warp == 7) {
    dst[512 + lane] = __float2bfloat16(ra);
    dst[512 + 32 + lane] = __float2bfloat16(rb);
  }
}

// qb [T, H, 192] = [nope 128 | rope 64] per head -> q_full[T, H, 512 + i] for the rope part
__global__ void mla_q_rope_kernel(const __nv_bfloat16* qb, const float* __restrict__ inv_freq, const int* __restrict__ positions,
                                  __nv_bfloat16* q_full, int H, int T, int64_t dst_stride, int dst_off) {
  pdl_sync();
  const int64_t gw = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (gw >= (int64_t)T * H) return;
  const int t = (int)(gw / H), i = threadIdx.x & 31;
  const __nv_bfloat16* src = qb + gw * 192 + 128;
  float a = __bfloat162float(src[i]), b = __bfloat162float(src[32 + i]);
  if (inv_freq) {
    float s, c;
    sincosf((float)positions[t] * inv_freq[i], &s, &c);
    const float ra = a * c - b * s, rb = a * s + b * c;
    a = ra; b = rb;
  }
  __nv_bfloat16* dst = q_full + gw * dst_stride + dst_off;        // may be the source row itself: every lane has read its pair
  dst[i] = __float2bfloat16(a);
  dst[32 + i] = __float2bfloat16(b);
}

// The same for 8-byte aligned rows: eight lanes hold a head's 64 dims (lane j the pairs 4 j .. 4 j + 3), a warp walks QR_HEADS heads of one token, four at a
// time, with one set of angles (4096 tokens of 64 heads: 36 us by one head per warp and 2-byte accesses, 9.6 us so).  Up to 4096 heads in all, where every
// warp of the form above has one and its chain is the shorter one, that form stays (3 tokens of 64 heads: 2.6 us, 3.3 us by this one; 64 of 64: 2.9 / 3.2).
constexpr int QR_HEADS = 16;
__global__ void __launch_bounds__(256)
mla_q_rope_heads_kernel(const __nv_bfloat16* qb, const float* __restrict__ inv_freq, const int* __restrict__ positions, __nv_bfloat16* q_full, int H, int T,
                        int64_t dst_stride, int dst_off) {
  pdl_sync();
  const int groups = (H + QR_HEADS - 1) / QR_HEADS, lane = threadIdx.x & 31, j = lane & 7;
  const int64_t gw = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (gw >= (int64_t)T * groups) return;
  const int t = (int)(gw / groups), h0 = (int)(gw % groups) * QR_HEADS + (lane >> 3), h1 = min(H, (int)(gw % groups + 1) * QR_HEADS);
  union Piece { uint2 v; __nv_bfloat16 e[4]; };
  Piece a[QR_HEADS / 4], b[QR_HEADS / 4];
#pragma unroll
  for (int k = 0; k < QR_HEADS / 4; ++k) {
    if (h0 + 4 * k < h1) {
      const __nv_bfloat16* src = qb + ((int64_t)t * H + h0 + 4 * k) * 192 + 128;
      a[k].v = *(const uint2*)(src + 4 * j);
      b[k].v = *(const uint2*)(src + 32 + 4 * j);
    }
  }
  float s[4], c[4];
  if (inv_freq) {
    const float pos = (float)positions[t];
#pragma unroll
    for (int e = 0; e < 4; ++e) sincosf(pos * inv_freq[4 * j + e], &s[e], &c[e]);
  }
#pragma unroll
  for (int k = 0; k < QR_HEADS / 4; ++k) {
    if (h0 + 4 * k < h1) {
      if (inv_freq) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float x = __bfloat162float(a[k].e[e]), y = __bfloat162float(b[k].e[e]);
          a[k].e[e] = __float2bfloat16(x * c[e] - y * s[e]);
          b[k].e[e] = __float2bfloat16(x * s[e] + y * c[e]);
        }
      }
      __nv_bfloat16* dst = q_full + ((int64_t)t * H + h0 + 4 * k) * dst_stride + dst_off;
      *(uint2*)(dst + 4 * j) = a[k].v;
      *(uint2*)(dst + 32 + 4 * j) = b[k].v;
    }
  }
}

// The copy below for 16-byte aligned rows: a warp writes 16 heads of a row, four at a time, from one load (4096 rows of 64 heads: 36 us by words).
__global__ void __launch_bounds__(256)
mla_fill_k_rope_heads_kernel(const __nv_bfloat16* __restrict__ lat, int64_t lat_stride, __nv_bfloat16* __restrict__ k, int H, int64_t n_rows) {
  pdl_sync();
  const int groups = (H + 15) / 16, lane = threadIdx.x & 31;
  const int64_t gw = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (gw >= n_rows * groups) return;
  const int64_t n = gw / groups;
  const int g = (int)(gw % groups);
  const uint4 v = *(const uint4*)(lat + n * lat_stride + 512 + (lane & 7) * 8);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int h = g * 16 + i * 4 + (lane >> 3);
    if (h < H) *(uint4*)(k + (n * H + h) * 192 + 128 + (lane & 7) * 8) = v;
  }
}

// K rows of the expanded prefill: the 64 rotated dims every head shares, copied from the latent row behind each head's 128 own dims.
__global__ void mla_fill_k_rope_kernel(const __nv_bfloat16* __restrict__ lat, int64_t lat_stride, __nv_bfloat16* __restrict__ k, int H,
                                       int64_t n_rows) {
  pdl_sync();
  const int64_t gw = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (gw >= n_rows * H) return;
  const int64_t n = gw / H;
  const int i = threadIdx.x & 31;
  const uint32_t v = *(const uint32_t*)(lat + n * lat_stride + 512 + 2 * i);
  *(uint32_t*)(k + gw * 192 + 128 + 2 * i) = v;
}

}  // namespace

MARY_API int mary_mla_prep(const void* qakv, int64_t ld, int q_lora, const void* w_qa, const void* w_kv, const float* inv_freq,
                           const int* positions, const int64_t* slots, void* qa_out, void* cache, float eps, int T, int64_t n_slots,
                           cudaStream_t s) {
  if (T <= 0) return MARY_OK;
  const uintptr_t at = (uintptr_t)qakv | (uintptr_t)w_qa | (uintptr_t)w_kv | (uintptr_t)qa_out | (uintptr_t)cache;
  if (at % 16 == 0 && ld % 8 == 0 && q_lora % 8 == 0 && q_lora <= PREP_Q * 8 * PREP_CH) {
    MARY_LAUNCH(mla_prep_rows_kernel, T, 256, 0, s, (const __nv_bfloat16*)qakv, ld, q_lora, (const __nv_bfloat16*)w_qa, (const __nv_bfloat16*)w_kv, inv_freq,
                positions, slots, (__nv_bfloat16*)qa_out, (__nv_bfloat16*)cache, eps, n_slots, mary_status_ptr());
    MARY_CHECK_LAUNCH();
    return MARY_OK;
  }
  MARY_LAUNCH(mla_prep_kernel, T, 256, 0, s, (const __nv_bfloat16*)qakv, ld, q_lora, (const __nv_bfloat16*)w_qa, (const __nv_bfloat16*)w_kv, inv_freq,
                                    positions, slots, (__nv_bfloat16*)qa_out, (__nv_bfloat16*)cache, eps, n_slots, mary_status_ptr());
  MARY_CHECK_LAUNCH();
  return MARY_OK;
}

static int q_rope(const void* qb, const float* inv_freq, const int* positions, void* dst, int H, int T, int64_t stride, int off, cudaStream_t s) {
  if (T <= 0) return MARY_OK;
  if (((uintptr_t)qb | (uintptr_t)dst) % 8 == 0 && (int64_t)T * H > 4096) {
    const int64_t warps = (int64_t)T * ((H + QR_HEADS - 1) / QR_HEADS);
    MARY_LAUNCH(mla_q_rope_heads_kernel, (int)((warps + 7) / 8), 256, 0, s, (const __nv_bfloat16*)qb, inv_freq, positions, (__nv_bfloat16*)dst, H, T, stride, off);
  } else {
    const int64_t warps = (int64_t)T * H;
    MARY_LAUNCH(mla_q_rope_kernel, (int)((warps + 7) / 8), 256, 0, s, (const __nv_bfloat16*)qb, inv_freq, positions, (__nv_bfloat16*)dst, H, T, stride, off);
  }
  MARY_CHECK_LAUNCH();
  return MARY_OK;
}

MARY_API int mary_mla_q_rope(const void* qb, const float* inv_freq, const int* positions, void* q_full, int H, int T, cudaStream_t s) {
  return q_rope(qb, inv_freq, positions, q_full, H, T, 576, 512, s);
}

// The same rotation written back over the 64 rope dims of qb [T, H, 192] itself (the expanded prefill attends with 192-wide queries).
MARY_API int mary_mla_q_rope_inplace(void* qb, const float* inv_freq, const int* positions, int H, int T, cudaStream_t s) {
  return q_rope(qb, inv_freq, positions, qb, H, T, 192, 128, s);
}

// k [n_rows, H, 192]: dims 128..191 of every head <- dims 512..575 of latent row n (row pitch lat_stride elements).
MARY_API int mary_mla_fill_k_rope(const void* lat, int64_t lat_stride, void* k, int H, int64_t n_rows, cudaStream_t s) {
  if (n_rows <= 0) return MARY_OK;
  if (lat_stride & 1) return MARY_ERR_BAD_ARG;
  if (((uintptr_t)lat | (uintptr_t)k) % 16 == 0 && lat_stride % 8 == 0) {
    const int64_t w = n_rows * ((H + 15) / 16);
    MARY_LAUNCH(mla_fill_k_rope_heads_kernel, (int)((w + 7) / 8), 256, 0, s, (const __nv_bfloat16*)lat, lat_stride, (__nv_bfloat16*)k, H, n_rows);
    MARY_CHECK_LAUNCH();
    return MARY_OK;
  }
  const int64_t warps = n_rows * H;
  MARY_LAUNCH(mla_fill_k_rope_kernel, (int)((warps + 7) / 8), 256, 0, s, (const __nv_bfloat16*)lat, lat_stride, (__nv_bfloat16*)k, H, n_rows);
  MARY_CHECK_LAUNCH();
  return MARY_OK;
}
