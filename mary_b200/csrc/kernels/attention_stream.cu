// Decode attention over the paged cache for few query rows per kv head, as a stream of whole cache rows; bf16 and 8-bit caches.
//
// What bounds it.  With one to eight query rows per kv head a cache row of D values is used for a handful of products, so the cache stream is the bound:
// about 23 bytes a clock per SM at full memory rate.  A warp reads whole rows (lane i holds D / 32 neighbouring values of a key and of a value row), so
// the arithmetic has to stay under ~40 issue slots per 512 bytes for that.  That is why
//   * products are packed pairs (`fma.rn.f32x2`), 8-bit codes become floats by a byte permute and one exact subtraction (2^23 + code - 2^23 - 128; the
//     conversion instruction runs at an eighth of that rate), and the scale and the zero of a row are applied once per row, not once per element:
//     q . (s c + z) = s (q . c) + z sum(q), and sum_j p_j (s_j c_j + z_j) = sum_j (p_j s_j) c_j + sum_j p_j z_j;
//   * the dot products of a group of keys are completed by a halving exchange that leaves ONE (key, row) total in each lane; scale, mask, maximum,
//     exponential and sum then run once per (key, row), in parallel over the lanes, and only the weights are broadcast;
//   * every warp has a ring of groups of its own in shared memory, filled by asynchronous copies at least one group ahead (what is in flight does not live in
//     registers, and no warp waits for another).
//
// The key range of a (query block, kv head) is cut between the CTAs of a cluster, which merge their partial results through distributed shared
// memory: no scratch, no second launch.  Everything is f32 between the cache and the bf16 output.
#include <type_traits>

#include "common.cuh"
#include "host_utils.h"

using namespace mary;

namespace {

constexpr float LOG2E = 1.4426950408889634f;
constexpr int MAX_SPLIT = 8;                  // portable cluster size

struct StreamParams {
  const __nv_bfloat16* q; const void* kc; const void* vc; __nv_bfloat16* out;
  const int* page_table; const int* kv_len; const int* q_start; const int* blk_seq; const int* blk_q0;
  const float* k_sz; const float* v_sz;       // 8-bit cache: (scale, zero) of every (slot, kv head)
  int max_pages, page_size;
  int64_t k_tok, k_page, v_tok, v_page;       // elements
  int Hq, Hkv, G, RQ, nsplit, window;
  float scale, softcap;
  int64_t q_ld, out_ld;
};

typedef unsigned long long f2;                // two f32 in one register pair
__device__ __forceinline__ f2 pack2(float a, float b) { f2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ float2 unpack2(f2 v) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v)); return r; }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) { f2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) { f2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f2 add2(f2 a, f2 b) { f2 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }

// What a lane holds of a row: E bf16 values or E codes, in 32-bit words (16-bit ones where E codes are less than a word).
template <int E, bool Q8> struct Piece {
  static constexpr int W = Q8 ? (E + 3) / 4 : E / 2;
  uint32_t w[W];
  __device__ __forceinline__ void load(const void* base, int64_t at) {
    if constexpr (Q8) {
      const uint8_t* s = (const uint8_t*)base + at;
      if constexpr (E == 2) w[0] = *(const uint16_t*)s;
      else if constexpr (E == 4) w[0] = *(const uint32_t*)s;
      else { const uint2 v = *(const uint2*)s; w[0] = v.x; w[1] = v.y; }
    } else {
      const __nv_bfloat16* s = (const __nv_bfloat16*)base + at;
      if constexpr (E == 2) w[0] = *(const uint32_t*)s;
      else if constexpr (E == 4) { const uint2 v = *(const uint2*)s; w[0] = v.x; w[1] = v.y; }
      else { const uint4 v = *(const uint4*)s; w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w; }
    }
  }
  // values 2 j and 2 j + 1; codes less 128
  __device__ __forceinline__ f2 pair(int j) const {
    if constexpr (Q8) {
      const uint32_t x = w[j / 2];
      const uint32_t lo = __byte_perm(x, 0x4B000000u, (j & 1) ? 0x7652 : 0x7650), hi = __byte_perm(x, 0x4B000000u, (j & 1) ? 0x7653 : 0x7651);
      return add2(pack2(__uint_as_float(lo), __uint_as_float(hi)), pack2(-8388736.f, -8388736.f));
    } else {
      return pack2(__uint_as_float(w[j] << 16), __uint_as_float(w[j] & 0xffff0000u));
    }
  }
};

// Totals of V values (a power of two, at most 32) over the 32 lanes: lane l returns the total of value l % V.
template <int V>
__device__ __forceinline__ float totals(float* v, int lane) {
#pragma unroll
  for (int o = 16; o >= V; o >>= 1) {
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
  }
#pragma unroll
  for (int o = V / 2; o >= 1; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float send = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0];
}

__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ float ld_cluster(uint32_t a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

__device__ __forceinline__ void copy_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

constexpr int STREAM_GROUP = 8192;           // K and V bytes of a group at most
// Bytes of a warp's ring, but two groups at least: two of bf16 rows or of codes of 256 with their scales (16896 bytes), three to eight of smaller ones.  Three
// groups of bf16 rows: 120 us instead of 104, fewer CTAs fit.
constexpr int STREAM_RING = 16384;
template <int D, int R, bool Q8> struct Group {
  static constexpr int ROW = D * (Q8 ? 1 : 2);                         // bytes of a key or value row
  static constexpr int FIT = STREAM_GROUP / (2 * ROW);
  static constexpr int KG0 = FIT < 32 / R ? FIT : 32 / R;
  static constexpr int KG = KG0 > 16 ? 16 : KG0;                       // keys of a group: KG * R totals fit the lanes
  static constexpr int LPR = ROW / 16, KPI = 32 / LPR;                 // lanes per row, rows per copy instruction
  static constexpr int STAGE = 2 * KG * ROW + (Q8 ? 2 * KG * 8 : 0);   // [keys][values][(scale, zero) of the keys][of the values]
  static constexpr int STAGES = STREAM_RING / STAGE < 2 ? 2 : (STREAM_RING / STAGE > 8 ? 8 : STREAM_RING / STAGE);
  static_assert((KG % KPI == 0 || KG < KPI) && 2 * KG <= 32 && STAGE % 16 == 0, "group");
};

// R rows at most (RQ * G); rows beyond the block's are computed on zeros and not stored.
template <int D, int R, bool Q8, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 8 / WARPS)
attn_stream_kernel(const StreamParams p) {
  pdl_sync();
  constexpr int E = D / 32, KG = Group<D, R, Q8>::KG, V = KG * R;
  using P = Piece<E, Q8>;
  __shared__ float red_o[WARPS][R][D];
  __shared__ float red_m[WARPS][R], red_l[WARPS][R];
  __shared__ float part_m[R], part_l[R];
  float (*part_o)[D] = red_o[0];                    // the CTA's merged rows replace the first warp's
  const int split = blockIdx.x, nb = blockIdx.y, kvh = blockIdx.z;     // the splits of one problem are one cluster
  const int seq = p.blk_seq[nb], row0 = p.blk_q0[nb];
  const int seq0 = p.q_start[seq], q_end = p.q_start[seq + 1];
  const int nq = min(p.RQ, q_end - row0), rows = nq * p.G;
  const int kvlen = p.kv_len[seq];
  const int pos0 = kvlen - (q_end - seq0) + (row0 - seq0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  f2 q2[R][E / 2];
  float qsum = 0.f;                                 // of row lane % R
#pragma unroll
  for (int r = 0; r < R; ++r) {
    Piece<E, false> v;
    const int tq = row0 + r / p.G, h = kvh * p.G + r % p.G;
    float s = 0.f;
    if (r < rows) v.load(p.q, (int64_t)tq * p.q_ld + h * D + lane * E);
#pragma unroll
    for (int e = 0; e < E / 2; ++e) {
      q2[r][e] = r < rows ? mul2(v.pair(e), pack2(p.scale, p.scale)) : 0ull;
      const float2 f = unpack2(q2[r][e]);
      s += f.x + f.y;
    }
    if (Q8) { s = warp_sum(s); if (lane % R == r) qsum = s; }
  }
  const int k_hi = pos0 + nq, k_lo = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;
  const int per = ((k_hi - k_lo + p.nsplit - 1) / p.nsplit + KG - 1) / KG * KG;
  const int s_lo = k_lo + split * per, s_hi = min(k_hi, s_lo + per);
  const int my_row = lane % R, my_key = lane % V / R;                  // of the total that this lane finishes
  const int my_pos = pos0 + my_row / p.G;
  const int* pt = p.page_table + (int64_t)seq * p.max_pages;

  float m = -INFINITY, l = 0.f, zero = 0.f;         // of this lane's (row, key of the group) pairs; m of the row
  f2 o2[R][E / 2];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int e = 0; e < E / 2; ++e) o2[r][e] = 0ull;

  using GR = Group<D, R, Q8>;
  extern __shared__ __align__(16) uint8_t ring_raw[];
  uint8_t* const ring = ring_raw + warp * (GR::STAGES * GR::STAGE);
  const uint32_t ring_at = smem_u32(ring);
  const bool same = p.k_tok == p.v_tok && p.k_page == p.v_page;
  constexpr int ES = Q8 ? 1 : 2, STEP = WARPS * KG;
  const uint8_t* const kbase = (const uint8_t*)p.kc + (int64_t)kvh * D * ES + (lane % GR::LPR) * 16;
  const uint8_t* const vbase = (const uint8_t*)p.vc + (int64_t)kvh * D * ES + (lane % GR::LPR) * 16;
  // page of key `lane % KG` of the group at kb (keys past the end: the last one, masked below)
  auto page_of = [&](int kb) -> int { return kb < s_hi ? pt[min(kb + lane % KG, s_hi - 1) / p.page_size] : 0; };
  auto request = [&](int kb, int page, int stage) {
    if (kb < s_hi) {
      const int tok = min(kb + lane % KG, s_hi - 1) % p.page_size;
      const int64_t ko = (page * p.k_page + tok * p.k_tok) * ES, vo = (page * p.v_page + tok * p.v_tok) * ES;
      const uint32_t dst = ring_at + stage * GR::STAGE + lane * 16;
#pragma unroll
      for (int i = 0; i < (KG + GR::KPI - 1) / GR::KPI; ++i) {
        const int j = i * GR::KPI + lane / GR::LPR;
        const int64_t a = __shfl_sync(0xffffffffu, ko, j), b = same ? a : __shfl_sync(0xffffffffu, vo, j);
        if (KG % GR::KPI && j >= KG) continue;
        copy_async16(dst + i * 512, kbase + a);
        copy_async16(dst + KG * GR::ROW + i * 512, vbase + b);
      }
      if constexpr (Q8) {
        const int64_t at = ((int64_t)(page * p.page_size + tok) * p.Hkv + kvh) * 2;
        if (lane < 2 * KG) copy_async8(ring_at + stage * GR::STAGE + 2 * KG * GR::ROW + lane * 8, (lane < KG ? p.k_sz : p.v_sz) + at);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int first = s_lo + warp * KG;
  int page = page_of(first), ask = first, ask_stage = 0;
#pragma unroll
  for (int i = 0; i < GR::STAGES - 1; ++i) {
    const int next = page_of(ask + STEP);
    request(ask, page, i);
    page = next;
    ask += STEP;
  }
  ask_stage = GR::STAGES - 1;
  int stage = 0;
  for (int kb = first; kb < s_hi; kb += STEP) {
    {
      const int next = page_of(ask + STEP);
      request(ask, page, ask_stage);             // into the stage that the previous pass left
      page = next;
      ask += STEP;
      if (++ask_stage == GR::STAGES) ask_stage = 0;
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(GR::STAGES - 1) : "memory");
    __syncwarp();
    const uint8_t* const st = ring + stage * GR::STAGE;
    if (++stage == GR::STAGES) stage = 0;
    P kv[KG], vv[KG];
#pragma unroll
    for (int j = 0; j < KG; ++j) { kv[j].load(st, j * D + lane * E); vv[j].load(st + KG * GR::ROW, j * D + lane * E); }
    float2 ks = make_float2(1.f, 0.f), vs = ks;
    if constexpr (Q8) {
      ks = *(const float2*)(st + 2 * KG * GR::ROW + my_key * 8);
      vs = *(const float2*)(st + 2 * KG * GR::ROW + (KG + my_key) * 8);
    }
    float t[V];
#pragma unroll
    for (int j = 0; j < KG; ++j) {
      f2 a[R];
#pragma unroll
      for (int e = 0; e < E / 2; ++e) {
        const f2 k2 = kv[j].pair(e);
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = e == 0 ? mul2(q2[r][0], k2) : fma2(q2[r][e], k2, a[r]);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) { const float2 f = unpack2(a[r]); t[j * R + r] = f.x + f.y; }
    }
    float x = totals<V>(t, lane);
    if (Q8) x = fmaf(ks.x, x, fmaf(128.f, ks.x, ks.y) * qsum);
    if (p.softcap > 0.f) x = p.softcap * tanhf(x / p.softcap);
    const int kp = kb + my_key;
    const bool ok = kp < s_hi && kp <= my_pos && (p.window <= 0 || my_pos - kp < p.window);
    x = ok ? x * LOG2E : -INFINITY;
    float mx = x;
#pragma unroll
    for (int o = V / 2; o >= R; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    mx = fmaxf(mx, m);
    const float ref = mx == -INFINITY ? 0.f : mx;
    const float corr = exp2f(m - ref), w = exp2f(x - ref);
    m = mx;
    l = fmaf(l, corr, w);
    if (Q8) zero = fmaf(zero, corr, w * fmaf(128.f, vs.x, vs.y));
    const float pw = Q8 ? w * vs.x : w;
    if (__any_sync(0xffffffffu, corr != 1.f)) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float c = __shfl_sync(0xffffffffu, corr, r);
#pragma unroll
        for (int e = 0; e < E / 2; ++e) o2[r][e] = mul2(o2[r][e], pack2(c, c));
      }
    }
#pragma unroll
    for (int j = 0; j < KG; ++j) {
      f2 c[R];
#pragma unroll
      for (int r = 0; r < R; ++r) { const float b = __shfl_sync(0xffffffffu, pw, j * R + r); c[r] = pack2(b, b); }
#pragma unroll
      for (int e = 0; e < E / 2; ++e) {
        const f2 v2 = vv[j].pair(e);
#pragma unroll
        for (int r = 0; r < R; ++r) o2[r][e] = fma2(c[r], v2, o2[r][e]);
      }
    }
    __syncwarp();                                // every lane has read this stage: the next pass may refill it
  }
  // sums over the keys of a group; lane r then holds row r
#pragma unroll
  for (int o = V / 2; o >= R; o >>= 1) {
    l += __shfl_xor_sync(0xffffffffu, l, o);
    if (Q8) zero += __shfl_xor_sync(0xffffffffu, zero, o);
  }
  if (lane < R) { red_m[warp][lane] = m; red_l[warp][lane] = l; }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float z = Q8 ? __shfl_sync(0xffffffffu, zero, r) : 0.f;
#pragma unroll
    for (int e = 0; e < E / 2; ++e) {
      const float2 f = unpack2(o2[r][e]);
      *(float2*)&red_o[warp][r][lane * E + 2 * e] = make_float2(f.x + z, f.y + z);
    }
  }
  __syncthreads();
  // the CTA's warps, then the CTAs of the cluster
  for (int i = threadIdx.x; i < rows * D; i += WARPS * 32) {
    const int r = i / D, d = i % D;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) mm = fmaxf(mm, red_m[w][r]);
    float ll = 0.f, acc = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float c = red_m[w][r] == -INFINITY ? 0.f : exp2f(red_m[w][r] - mm);
      ll = fmaf(red_l[w][r], c, ll);
      acc = fmaf(red_o[w][r][d], c, acc);
    }
    if (p.nsplit == 1) {
      const int tq = row0 + r / p.G, h = kvh * p.G + r % p.G;
      p.out[(int64_t)tq * p.out_ld + (int64_t)h * D + d] = __float2bfloat16(ll > 0.f ? acc / ll : 0.f);
    } else {
      part_o[r][d] = acc;                           // nobody else reads this element of the first warp
      if (d == 0) { part_m[r] = mm; part_l[r] = ll; }
    }
  }
  if (p.nsplit > 1) {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    for (int i = split * (WARPS * 32) + threadIdx.x; i < rows * D; i += p.nsplit * WARPS * 32) {
      const int r = i / D, d = i % D;
      float pm[MAX_SPLIT], pl[MAX_SPLIT], po[MAX_SPLIT];
#pragma unroll
      for (int s = 0; s < MAX_SPLIT; ++s) {
        pm[s] = -INFINITY; pl[s] = po[s] = 0.f;
        if (s < p.nsplit) {
          pm[s] = ld_cluster(cluster_addr(&part_m[r], s));
          pl[s] = ld_cluster(cluster_addr(&part_l[r], s));
          po[s] = ld_cluster(cluster_addr(&part_o[r][d], s));
        }
      }
      float mm = -INFINITY, ll = 0.f, acc = 0.f;
#pragma unroll
      for (int s = 0; s < MAX_SPLIT; ++s) mm = fmaxf(mm, pm[s]);
#pragma unroll
      for (int s = 0; s < MAX_SPLIT; ++s) {
        const float c = pm[s] == -INFINITY ? 0.f : exp2f(pm[s] - mm);
        ll = fmaf(pl[s], c, ll);
        acc = fmaf(po[s], c, acc);
      }
      const int tq = row0 + r / p.G, h = kvh * p.G + r % p.G;
      p.out[(int64_t)tq * p.out_ld + (int64_t)h * D + d] = __float2bfloat16(ll > 0.f ? acc / ll : 0.f);
    }
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");      // shared memory stays until all have read it
  }
}

template <int D, int R, bool Q8, int WARPS>
int launch(const StreamParams& p, int NB, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(WARPS * 32);
  cfg.dynamicSmemBytes = WARPS * Group<D, R, Q8>::STAGES * Group<D, R, Q8>::STAGE;
  cfg.stream = s;
  static MarySmemSlots smem_set = {};
  if (int rc = mary_ensure_dyn_smem((const void*)attn_stream_kernel<D, R, Q8, WARPS>, cfg.dynamicSmemBytes, &smem_set)) return rc;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.nsplit;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  // More CTAs than SMs start after their predecessor: placed while it drains they would crowd three deep onto the SMs that are free first (256 CTAs of
  // 2048 bf16 keys: 80 us instead of 66).
  cfg.numAttrs = mary_pdl_enabled() && (int64_t)p.nsplit * NB * p.Hkv <= mary_num_sms() ? 2 : 1;
  // a grid has at most 65535 query blocks (as x instead, together with the splits, they took 92 -> 120 us: 8 sequences of 8000 bf16 keys, 8 kv heads)
  for (int at = 0; at < NB; at += 65535) {
    StreamParams part = p;
    part.blk_seq += at;
    part.blk_q0 += at;
    cfg.gridDim = dim3(p.nsplit, NB - at < 65535 ? NB - at : 65535, p.Hkv);
    if (cudaLaunchKernelEx(&cfg, attn_stream_kernel<D, R, Q8, WARPS>, part) != cudaSuccess) return MARY_ERR_CUDA;
    MARY_CHECK_LAUNCH();
  }
  return MARY_OK;
}

template <int D, int R, bool Q8>
int launch_warps(const StreamParams& p, int NB, int warps, cudaStream_t s) {
  return warps == 8 ? launch<D, R, Q8, 8>(p, NB, s) : launch<D, R, Q8, 4>(p, NB, s);
}
template <int D, int R>
int launch_cache(const StreamParams& p, int NB, int warps, cudaStream_t s) {
  if (p.k_sz) return launch_warps<D, R, true>(p, NB, warps, s);
  if constexpr (D == 256 && R <= 2) return launch_warps<D, R, false>(p, NB, warps, s);       // the other bf16 shapes are the tensor-core kernel's
  return MARY_ERR_BAD_ARG;
}

}  // namespace

// q [T, Hq, D] bf16 with row pitch q_ld, caches [pages, page, Hkv, D] with token and page strides in elements (k_sz / v_sz null: bf16; else unsigned
// codes with (scale, zero) per (slot, kv head)), out rows of out_ld elements.  D 64, 128 or 256, RQ * (Hq / Hkv) <= 4 (D 256) or 8 for codes; D 256 and
// RQ * (Hq / Hkv) <= 2 for bf16; nsplit 1, 2, 4 or 8;
// warps 4 or 8.  Query blocks as in mary_paged_attention.
MARY_API int mary_attention_stream(const void* q, const void* kc, const void* vc, const float* k_sz, const float* v_sz, void* out, const int* page_table,
                                   const int* kv_len, const int* q_start, const int* blk_seq, const int* blk_q0, int NB, int max_pages, int page_size,
                                   int64_t k_tok, int64_t k_page, int64_t v_tok, int64_t v_page, int64_t q_ld, int64_t out_ld, int Hq, int Hkv, int D,
                                   int RQ, int nsplit, int warps, int window, float scale, float softcap, cudaStream_t s) {
  if (NB <= 0) return MARY_OK;
  if (Hkv < 1 || Hq % Hkv || page_size < 1 || RQ < 1 || (nsplit != 1 && nsplit != 2 && nsplit != 4 && nsplit != 8) || (warps != 4 && warps != 8) ||
      (k_sz == nullptr) != (v_sz == nullptr) || Hkv > 65535)
    return MARY_ERR_BAD_ARG;
  // rows are copied 16 bytes at a time, a lane reads D / 32 neighbouring query values at once
  const int64_t es = k_sz ? 1 : 2, qb = D / 32 * 2;
  if ((k_tok * es) % 16 || (k_page * es) % 16 || (v_tok * es) % 16 || (v_page * es) % 16 || ((uintptr_t)kc % 16) || ((uintptr_t)vc % 16) ||
      ((uintptr_t)q % qb) || (q_ld * 2) % qb || ((uintptr_t)k_sz % 8) || ((uintptr_t)v_sz % 8))
    return MARY_ERR_BAD_ARG;
  StreamParams p;
  p.q = (const __nv_bfloat16*)q; p.kc = kc; p.vc = vc; p.out = (__nv_bfloat16*)out;
  p.page_table = page_table; p.kv_len = kv_len; p.q_start = q_start; p.blk_seq = blk_seq; p.blk_q0 = blk_q0;
  p.k_sz = k_sz; p.v_sz = v_sz;
  p.max_pages = max_pages; p.page_size = page_size; p.k_tok = k_tok; p.k_page = k_page; p.v_tok = v_tok; p.v_page = v_page;
  p.Hq = Hq; p.Hkv = Hkv; p.G = Hq / Hkv; p.RQ = RQ; p.nsplit = nsplit; p.window = window; p.scale = scale; p.softcap = softcap;
  p.q_ld = q_ld; p.out_ld = out_ld;
  const int R = RQ * p.G;
  if (D == 256) { if (R == 1) return launch_cache<256, 1>(p, NB, warps, s); if (R == 2) return launch_cache<256, 2>(p, NB, warps, s); if (R <= 4) return launch_cache<256, 4>(p, NB, warps, s); }
  if (D == 128) { if (R == 1) return launch_cache<128, 1>(p, NB, warps, s); if (R == 2) return launch_cache<128, 2>(p, NB, warps, s); if (R <= 4) return launch_cache<128, 4>(p, NB, warps, s);
                  if (R <= 8) return launch_cache<128, 8>(p, NB, warps, s); }
  if (D == 64) { if (R == 1) return launch_cache<64, 1>(p, NB, warps, s); if (R == 2) return launch_cache<64, 2>(p, NB, warps, s); if (R <= 4) return launch_cache<64, 4>(p, NB, warps, s);
                 if (R <= 8) return launch_cache<64, 8>(p, NB, warps, s); }
  return MARY_ERR_BAD_ARG;
}
