// bf16 GEMM by pairs of SMs: out[M, N] = X[M, K] * W[N, K]^T, both operands K-major, f32 accumulation in TMEM.
//
// What bounds it.  A 128 x 256 tile of one SM moves 48 KB from L2 for every 64 columns of K, and at full tensor rate that is about 96
// bytes a clock per SM, more than an SM can draw from L2.  Two SMs that work on one 256 x BN tile (`tcgen05.mma.cta_group::2`) hold
// half of the column operand each: 32 KB per SM for the same arithmetic.  Shapes with few output tiles are bound by something else: one
// tile per SM leaves SMs idle, or each of them walks a long K alone.  There a cluster of 2, 4 or 8 pairs cuts K between the pairs and adds the
// partial tiles through distributed shared memory, in a fixed order, without scratch memory and without atomics.
//
//   * cluster of 2 * S CTAs = S pairs; pair s multiplies the s-th part of K.  Per CTA: warp 0 issues the TMA loads of this CTA's 128
//     rows of the row operand and BN / 2 rows of the column operand, warp 1 of the pair's first CTA issues the MMAs (M = 256), warps
//     2-5 read this CTA's 128 x BN accumulator and store it;
//   * the loads of both CTAs of a pair complete on the FIRST CTA's "full" barrier; `tcgen05.commit` with the pair's mask frees a stage, or
//     publishes an accumulator, in both;
//   * S = 1 is persistent (one pair per two SMs, two accumulators, so that storing a tile overlaps the next one); S > 1 takes one tile per
//     cluster, and the idle load ring becomes the buffer that the partial sums are exchanged through;
//   * GLU: the first CTA of a pair loads gate rows, the second the matching up rows, so gate and up of an output feature sit BN / 2
//     columns apart in every CTA's accumulator and the [rows, 2 F] intermediate never exists;
//   * SWAP: the weights are the row operand (256 weight rows per tile) and the few tokens the columns.
//
// Measured (weights larger than L2, one-SM kernel -> this one): 8192 x 30720 x 3840 1345 -> 1235 us (1565 TFLOP/s), 8192 x 8192 x 3840 366 -> 324 us,
// 1024 x 3840 x 65536 540 -> 375 us, 701 x 3840 x 15360 104 -> 63 us; with K split 217 x 3840 x 4096 42 -> 15 us, 384 x 2112 x 7168 23 -> 20 us,
// 4096 x 48 x 3840 18 -> 12 us.  One tile per pair and no split, 217 x 8192 x 3840: 47 -> 20 us, 217 x 30720 x 3840: 77 -> 51 us (4.9 TB/s).
// Narrow outputs of a long K (4 -> 8 pairs): 3 x 48 x 15360 16.6 -> 11.8 us, 16 x 128 x 7168 11.5 -> 9.2 us, 257 x 128 x 7168 11.5 -> 10.0 us.  f32 results
// through TMA stores of 16 columns: 257 x 3840 x 256 at 256 columns 14.3 -> 10.1 us.
#include <type_traits>

#include "common.cuh"
#include "gemm_pair.h"
#include "host_utils.h"

using namespace mary;

namespace {

constexpr int BK = 64;
constexpr int ROWS = 128;                 // rows of the row operand per CTA
constexpr int A_BYTES = ROWS * BK * 2;
constexpr int NTHREADS = 192;
constexpr int MAX_STAGES = 12;
constexpr int SMEM = 226 * 1024;
constexpr int STORE_BYTES = 4 * 2 * 2048; // two chunks of 32 rows x 32 bf16 columns per epilogue warp on their way out
constexpr int RING = SMEM - 1024 - 512 - STORE_BYTES;

struct PairParams {
  int rows_r, rows_c;                     // extents of the row and the column operand (with GLU: output features)
  int tiles_r, tiles_c, k_blocks, kb_per_split, S;
  int bn, stages, stage_bytes;
  int raster;
  int act, glu_rows;                      // GLU: kind, rows between a gate row and its up row
  float glu_limit, alpha;
  int un_act, un_cols;
  int tma_box;                            // columns per TMA store (32 or 16; f32: 16); 0: plain stores
  int n_acc, acc_stride;                  // accumulators that the K blocks of a tile go round, their distance in TMEM columns
  int group, pitch;                       // group > 0 (TMA stores): output columns in groups, their starts `pitch` columns apart
  int64_t ldo;
  void* out;
  const float* bias;
  int w_static;
  int* status;
};

// ------------------------------------------------------------------------------------------------ pair and cluster forms
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ float4 ld_cluster4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, uint32_t src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(m), "r"(src), "r"(x), "r"(y) : "memory");
}
// `bar`: shared::cluster address; it may lie in the other CTA of the pair
__device__ __forceinline__ void tma_load_pair(void* dst, const CUtensorMap* m, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(m), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar, uint16_t mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"(mask) : "memory");
}

// tiles of this cluster, in bands of `raster` column tiles (rows of a band one after the other, its columns fastest) so that the clusters that run together
// cover a compact block of the output
__device__ __forceinline__ void tile_at(const PairParams& p, int t, int& tr, int& tc) {
  if (p.raster > 0) {
    const int band = t / (p.raster * p.tiles_r), base = band * p.raster;
    const int gw = min(p.raster, p.tiles_c - base), in = t - band * p.raster * p.tiles_r;
    tr = in / gw;
    tc = base + in % gw;
  } else {
    tc = t % p.tiles_c;
    tr = t / p.tiles_c;
  }
}

// F32: the result's type; CUT: K is cut between the pairs of a cluster (S > 1).  Each form has its own code: a launch of few blocks spends a good part of its
// time on fetching instructions for the first time.
template <bool GLU, bool SWAP, bool F32, bool CUT>
__global__ void __launch_bounds__(NTHREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tm_r, const __grid_constant__ CUtensorMap tm_c, const __grid_constant__ CUtensorMap tm_o,
                 const PairParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~uintptr_t(1023));
  uint64_t* full = (uint64_t*)(smem + RING + STORE_BYTES);
  uint64_t* empty = full + MAX_STAGES;
  uint64_t* acc_full = empty + MAX_STAGES;    // [2]
  uint64_t* acc_empty = acc_full + 2;         // [2], of the pair's first CTA
  uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int half = rank & 1, split = rank >> 1;
  const int bn = p.bn, stages = p.stages;
  const int cluster = blockIdx.x / (2 * p.S), n_clusters = gridDim.x / (2 * p.S);
  const int total = p.tiles_r * p.tiles_c;
  const int kb0 = split * p.kb_per_split, kb1 = min(kb0 + p.kb_per_split, p.k_blocks);
  const int n_acc = F32 ? min(p.n_acc, kb1 - kb0) : 1;                       // the last part of K may have fewer blocks than there are accumulators

  if (threadIdx.x < MAX_STAGES) { mbar_init(&full[threadIdx.x], 1); mbar_init(&empty[threadIdx.x], 1); }
  if (threadIdx.x >= 32 && threadIdx.x < 34) { mbar_init(&acc_full[threadIdx.x - 32], 1); mbar_init(&acc_empty[threadIdx.x - 32], 8); }
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    tma_prefetch_desc(&tm_r);
    tma_prefetch_desc(&tm_c);
  }
  fence_barrier_init();
  cluster_arrive();
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_wait();                             // the other CTA's barriers are ready before anything completes on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch();
  bool ok = true;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      const uint32_t full0 = mapa(smem_u32(full), rank & ~1u);       // the first CTA's barriers
      int stage = 0; uint32_t phase = 0;
      const int wrows = bn / 2;
      int pre = 0;
      // row of the weight operand (both CTAs of a pair hold different rows of it)
      auto w_row = [&](int tr, int tc) -> int {
        if (SWAP) return (tr * 2 + half) * ROWS;
        return GLU ? tc * wrows + half * p.glu_rows : tc * bn + half * wrows;
      };
      auto x_row = [&](int tr, int tc) -> int { return SWAP ? tc * bn + half * wrows : (tr * 2 + half) * ROWS; };
      if (p.w_static && cluster < total && kb0 < kb1) {
        // constant weights: the first tiles are requested before the previous kernel of the stream has finished
        int tr, tc;
        tile_at(p, cluster, tr, tc);
        pre = min(kb1 - kb0, stages);
        for (int i = 0; i < pre; ++i) {
          uint8_t* st = smem + i * p.stage_bytes;
          if (half == 0) mbar_expect_tx(&full[i], 2 * p.stage_bytes);
          if (SWAP) tma_load_pair(st, &tm_r, full0 + 8 * i, (kb0 + i) * BK, w_row(tr, tc));
          else tma_load_pair(st + A_BYTES, &tm_c, full0 + 8 * i, (kb0 + i) * BK, w_row(tr, tc));
        }
      }
      pdl_wait();
      for (int t = cluster; ok && t < total; t += n_clusters) {
        int tr, tc;
        tile_at(p, t, tr, tc);
        const int wr = w_row(tr, tc), xr = x_row(tr, tc);
        for (int kb = kb0; kb < kb1; ++kb) {
          uint8_t* st = smem + stage * p.stage_bytes;
          const uint32_t bar = full0 + 8 * stage;
          if (pre > 0) {
            --pre;
            if (SWAP) tma_load_pair(st + A_BYTES, &tm_c, bar, kb * BK, xr);
            else tma_load_pair(st, &tm_r, bar, kb * BK, xr);
          } else {
            if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.status, MARY_ERR_TIMEOUT_TMA)) { ok = false; break; }
            if (half == 0) mbar_expect_tx(&full[stage], 2 * p.stage_bytes);
            tma_load_pair(st, &tm_r, bar, kb * BK, SWAP ? wr : xr);
            tma_load_pair(st + A_BYTES, &tm_c, bar, kb * BK, SWAP ? xr : wr);
          }
          if (++stage == stages) { stage = 0; phase ^= 1; }
        }
      }
      // the commits that free the last stages arrive from the pair's first CTA: none may still be on its way when this CTA leaves
      for (int i = 0; ok && i < stages; ++i) {
        ok = mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.status, MARY_ERR_TIMEOUT_TMA);
        if (++stage == stages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer of the pair
    if (half == 0 && elect_one()) {
      const uint32_t idesc = idesc_bf16(2 * ROWS, bn);
      const uint16_t mask = (uint16_t)(3u << (rank & ~1u));
      int stage = 0; uint32_t phase = 0;
      int it = 0;
      for (int t = cluster; ok && t < total; t += n_clusters, ++it) {
        const int buf = it & 1;
        if (!mbar_wait(&acc_empty[buf], ((it >> 1) & 1) ^ 1, abort_flag, p.status, MARY_ERR_TIMEOUT_MMA)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d0 = tmem_base + buf * 256;
        int acc = 0;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&full[stage], phase, abort_flag, p.status, MARY_ERR_TIMEOUT_TMA)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * p.stage_bytes), sb = sa + A_BYTES;
          const uint32_t d = F32 ? d0 + acc * p.acc_stride : d0;
          const bool begun = kb - kb0 >= n_acc;
          if (F32 && ++acc == n_acc) acc = 0;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_f16_pair(d, umma_desc_sw128(sa + k * 32), umma_desc_sw128(sb + k * 32), idesc, (begun || k > 0) ? 1u : 0u);
          umma_commit_pair(&empty[stage], mask);
          if (++stage == stages) { stage = 0; phase ^= 1; }
        }
        if (ok) umma_commit_pair(&acc_full[buf], mask);
      }
    }
  }
  // ------------------------------------------------------------------ epilogue (warps 2..5)
  const int q = warp & 3;
  const int row = q * 32 + lane;
  auto activate = [&](auto width, int i, int j0, float* v) {
    constexpr int W = decltype(width)::value;
    const int left = SWAP ? (i < p.un_cols ? W : 0) : p.un_cols - j0;
    if (left <= 0) return;
    // x * sigmoid(g(x)): the chains side by side, without a branch between them
    const float c1 = p.un_act == 1 ? -2.302208198f : -1.4426950408889634f, c3 = p.un_act == 1 ? -0.1029432397f : 0.f;
    float e[W];
#pragma unroll
    for (int j = 0; j < W; ++j) e[j] = exp2f(v[j] * fmaf(c3 * v[j], v[j], c1));
#pragma unroll
    for (int j = 0; j < W; ++j) v[j] = j < left ? __fdividef(v[j], 1.0f + e[j]) : v[j];
  };
  // finishes W values of accumulator columns c0 .. (with GLU: output features) of this thread's row and stores them
  auto emit = [&](auto width, int tr, int tc, int c0, float* v) {
    constexpr int W = decltype(width)::value;
    const int i = (tr * 2 + half) * ROWS + row;
    const int j0 = tc * (GLU ? bn / 2 : bn) + c0;
    if (!GLU && p.un_act) activate(width, i, j0, v);
    if (i >= p.rows_r) return;
    if (SWAP) {
      const float b = p.bias ? p.bias[i] : 0.f;
#pragma unroll
      for (int j = 0; j < W; ++j) {
        if (j0 + j < p.rows_c) {
          const int64_t o = (int64_t)(j0 + j) * p.ldo + i;
          if (F32) ((float*)p.out)[o] = v[j] + b;
          else ((__nv_bfloat16*)p.out)[o] = __float2bfloat16(v[j] + b);
        }
      }
      return;
    }
    if (p.bias) {
#pragma unroll
      for (int j = 0; j < W; ++j) if (j0 + j < p.rows_c) v[j] += p.bias[j0 + j];
    }
    const int64_t o = (int64_t)i * p.ldo + j0;
    if (F32) {
      float* dst = (float*)p.out + o;
      if (j0 + W <= p.rows_c && ((uintptr_t)dst & 15) == 0) {
#pragma unroll
        for (int j = 0; j < W; j += 4) *(float4*)(dst + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
      } else {
#pragma unroll
        for (int j = 0; j < W; ++j) if (j0 + j < p.rows_c) dst[j] = v[j];
      }
    } else {
      __nv_bfloat16* dst = (__nv_bfloat16*)p.out + o;
      if (W % 8 == 0 && j0 + W <= p.rows_c && ((uintptr_t)dst & 15) == 0) {
#pragma unroll
        for (int j = 0; j < W / 8 * 8; j += 8) {
          uint4 w;
          uint32_t* wp = (uint32_t*)&w;
#pragma unroll
          for (int x = 0; x < 4; ++x) { __nv_bfloat162 h = __floats2bfloat162_rn(v[j + 2 * x], v[j + 2 * x + 1]); wp[x] = *(uint32_t*)&h; }
          *(uint4*)(dst + j) = w;
        }
      } else {
#pragma unroll
        for (int j = 0; j < W; ++j) if (j0 + j < p.rows_c) dst[j] = __float2bfloat16(v[j]);
      }
    }
  };
  // the same through shared memory and a TMA store, 32 columns of a warp's 32 rows at a time: a plain store instruction would touch 32 rows
  uint8_t* const stage_out = smem + RING + q * 4096;
  int n_stored = 0;
  auto emit_tma = [&](int tr, int tc, int c0, const float* v) {
    const int i0 = (tr * 2 + half) * ROWS + q * 32;
    const int j0 = tc * (GLU ? bn / 2 : bn) + c0;
    if constexpr (F32) {
      // f32: the 32 columns in two boxes of 16, rows of 64 bytes in the 64-byte swizzle
#pragma unroll
      for (int h = 0; h < 2; ++h, ++n_stored) {
        uint8_t* buf = stage_out + (n_stored & 1) * 2048;
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 4; ++c)
          *(float4*)(buf + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) =
              make_float4(v[16 * h + 4 * c], v[16 * h + 4 * c + 1], v[16 * h + 4 * c + 2], v[16 * h + 4 * c + 3]);
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
          if (i0 < p.rows_r && j0 + 16 * h < p.rows_c && c0 + 16 * h < (GLU ? bn / 2 : bn)) tma_store_2d(&tm_o, smem_u32(buf), j0 + 16 * h, i0);
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
      return;
    }
    uint8_t* buf = stage_out + (n_stored & 1) * 2048;
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");      // the store before last has read this buffer
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint4 w;
      uint32_t* wp = (uint32_t*)&w;
#pragma unroll
      for (int x = 0; x < 4; ++x) { __nv_bfloat162 h = __floats2bfloat162_rn(v[8 * c + 2 * x], v[8 * c + 2 * x + 1]); wp[x] = *(uint32_t*)&h; }
      // 32-column boxes: rows of 64 bytes in the 64-byte swizzle; 16-column boxes: two blocks of rows of 32 bytes in the 32-byte swizzle
      const int at = p.tma_box == 32 ? lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4) : (c >> 1) * 1024 + lane * 32 + (((c & 1) ^ ((lane >> 2) & 1)) << 4);
      *(uint4*)(buf + at) = w;
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) {
      if (i0 < p.rows_r) {
        if (p.tma_box == 32) {
          if (j0 < p.rows_c) tma_store_2d(&tm_o, smem_u32(buf), p.group > 0 ? j0 / p.group * p.pitch + j0 % p.group : j0, i0);
        } else {
          if (j0 < p.rows_c) tma_store_2d(&tm_o, smem_u32(buf), j0, i0);
          if (c0 + 16 < (GLU ? bn / 2 : bn) && j0 + 16 < p.rows_c) tma_store_2d(&tm_o, smem_u32(buf) + 1024, j0 + 16, i0);
        }
      }
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    ++n_stored;
  };
  // 32 columns of this thread's row: the sum of the tile's accumulators, in a fixed order
  auto read32 = [&](uint32_t at, uint32_t* r) {
    tmem_ld_32x32b_x32(at, r);
    tmem_ld_wait();
    if constexpr (!F32) return;
    for (int a = 1; a < n_acc; ++a) {
      uint32_t t[32];
      tmem_ld_32x32b_x32(at + a * p.acc_stride, t);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(t[j]));
    }
  };
  if (warp >= 2) {
    pdl_wait();                            // before the first store: an earlier kernel may still read what this one overwrites
    const uint32_t empty0 = mapa(smem_u32(acc_empty), rank & ~1u);
    int it = 0;
    for (int t = cluster; t < total; t += n_clusters, ++it) {
      const int buf = it & 1;
      if (!mbar_wait(&acc_full[buf], (it >> 1) & 1, abort_flag, p.status, MARY_ERR_TIMEOUT_MMA)) { ok = false; break; }
      tc_fence_after();
      const uint32_t taddr = tmem_base + buf * 256 + ((uint32_t)(q * 32) << 16);
      if constexpr (!CUT) {
        int tr, tc;
        tile_at(p, t, tr, tc);
#pragma unroll 1
        for (int c0 = 0; c0 < (GLU ? bn / 2 : bn); c0 += 32) {
          uint32_t r[32];
          float v[32];
          if (GLU) {
            uint32_t u[32];
            tmem_ld_32x32b_x32(taddr + c0, r);
            tmem_ld_32x32b_x32(taddr + bn / 2 + c0, u);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = glu_f(p.act, __uint_as_float(r[j]) * p.alpha, __uint_as_float(u[j]) * p.alpha, p.glu_limit);
          } else {
            read32(taddr + c0, r);
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]) * p.alpha;
          }
          // BN / 2 is a multiple of 16 with GLU: the last chunk may reach into the up columns, whose values are not output
          if (!SWAP && p.tma_box) {
            if (!GLU && p.un_act) activate(std::integral_constant<int, 32>{}, (tr * 2 + half) * ROWS + row, tc * bn + c0, v);
            if (p.bias) {
#pragma unroll
              for (int j = 0; j < 32; ++j) { const int col = tc * (GLU ? bn / 2 : bn) + c0 + j; if (col < p.rows_c) v[j] += p.bias[col]; }
            }
            emit_tma(tr, tc, c0, v);
          } else if (GLU && c0 + 32 > bn / 2) emit(std::integral_constant<int, 16>{}, tr, tc, c0, v);
          else emit(std::integral_constant<int, 32>{}, tr, tc, c0, v);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(empty0 + 8 * buf);
      } else {
        // partial sums, four columns of a row together, into the load ring, which nothing uses any more: all of this CTA's loads have
        // landed and the MMAs that read them are complete
        uint4* part = (uint4*)smem;
#pragma unroll 1
        for (int c0 = 0; c0 < bn; c0 += 32) {
          uint32_t r[32];
          read32(taddr + c0, r);
#pragma unroll
          for (int j = 0; j < 8; ++j) part[(c0 / 4 + j) * ROWS + row] = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
        }
      }
    }
  }
  __syncwarp();
  if constexpr (CUT) {
    cluster_sync_all();                    // every partial tile of the cluster is in shared memory
    if (warp >= 2 && ok && cluster < total && !*abort_flag) {
      int tr, tc;
      tile_at(p, cluster, tr, tc);
      const int share = (GLU ? bn / 2 : bn) / p.S;        // columns that this CTA finishes: a multiple of 8, or of 4 with 8 pairs
      const uint32_t mine = smem_u32(smem) + row * 16;
      // W columns at a time, all pairs' values of them requested before the first is used
      auto gather = [&](auto width, auto pairs, int c0) {
        constexpr int W = decltype(width)::value, S = decltype(pairs)::value, NV = W / 4;
        float4 a[S][NV], b[GLU ? S : 1][NV];
#pragma unroll
        for (int s = 0; s < S; ++s) {
          const uint32_t src = mapa(mine, 2 * s + half);
#pragma unroll
          for (int j = 0; j < NV; ++j) {
            a[s][j] = ld_cluster4(src + (c0 / 4 + j) * ROWS * 16);
            if (GLU) b[s][j] = ld_cluster4(src + ((bn / 2 + c0) / 4 + j) * ROWS * 16);
          }
        }
        float v[W];
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          float4 x = a[0][j], u = b[0][j];
#pragma unroll
          for (int s = 1; s < S; ++s) {
            x.x += a[s][j].x; x.y += a[s][j].y; x.z += a[s][j].z; x.w += a[s][j].w;
            if (GLU) { u.x += b[s][j].x; u.y += b[s][j].y; u.z += b[s][j].z; u.w += b[s][j].w; }
          }
          const float xs[4] = {x.x, x.y, x.z, x.w}, us[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) v[4 * j + e] = GLU ? glu_f(p.act, xs[e] * p.alpha, us[e] * p.alpha, p.glu_limit) : xs[e] * p.alpha;
        }
        emit(width, tr, tc, c0, v);
      };
      const int first = split * share;
      if (p.S == 2) {
        int c = 0;
        for (; c + 16 <= share; c += 16) gather(std::integral_constant<int, 16>{}, std::integral_constant<int, 2>{}, first + c);
        if (c < share) gather(std::integral_constant<int, 8>{}, std::integral_constant<int, 2>{}, first + c);
      } else if (p.S == 4) {
        int c = 0;
        for (; c + 16 <= share; c += 16) gather(std::integral_constant<int, 16>{}, std::integral_constant<int, 4>{}, first + c);
        if (c < share) gather(std::integral_constant<int, 8>{}, std::integral_constant<int, 4>{}, first + c);
      } else if constexpr (!GLU) {
        int c = 0;
        for (; c + 8 <= share; c += 8) gather(std::integral_constant<int, 8>{}, std::integral_constant<int, 8>{}, first + c);
        if (c < share) gather(std::integral_constant<int, 4>{}, std::integral_constant<int, 8>{}, first + c);
      }
    }
    __syncwarp();
  }
  if (!CUT && warp >= 2 && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");    // the stores are complete
  __syncwarp();
  tc_fence_before();
  cluster_sync_all();                      // neither shared memory nor TMEM goes while the other CTAs may still reach it
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
}

template <bool GLU, bool SWAP, bool F32, bool CUT>
int launch(const CUtensorMap& tr, const CUtensorMap& tc, const CUtensorMap& to, const PairParams& p, int clusters, cudaStream_t stream) {
  static MarySmemSlots smem_set = {};
  if (int rc = mary_ensure_dyn_smem((const void*)gemm_pair_kernel<GLU, SWAP, F32, CUT>, SMEM, &smem_set)) return rc;
  if (p.S > 4 && cudaFuncSetAttribute(gemm_pair_kernel<GLU, SWAP, F32, CUT>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return MARY_ERR_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(clusters * 2 * p.S);
  cfg.blockDim = dim3(NTHREADS);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2 * p.S;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = mary_pdl_enabled() ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, gemm_pair_kernel<GLU, SWAP, F32, CUT>, tr, tc, to, p) != cudaSuccess) return MARY_ERR_CUDA;
  MARY_CHECK_LAUNCH();
  return MARY_OK;
}

// output rows in boxes of 32 rows x `box` columns
int store_map(CUtensorMap* m, void* out, int f32, int rows, int cols, int64_t ld, int box) {
  PFN_encodeTiled enc = mary_encode_fn();
  if (!enc) return MARY_ERR_CUDA;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * (f32 ? 4 : 2)};
  cuuint32_t boxes[2] = {(cuuint32_t)box, 32}, estr[2] = {1, 1};
  CUresult r = enc(m, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, out, dims, strides, boxes, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   box * (f32 ? 4 : 2) == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? MARY_OK : MARY_ERR_CUDA;
}

}  // namespace

// Clusters of 2 S CTAs that the current device runs at a time: clusters of 4 and 8 leave some SMs of a processor cluster without a partner.
// Clusters of 16 are beyond what every device promises: 0 where there are none.
static int resident_clusters(int S) {
  static int known[MARY_MAX_DEVICES][4];                   // 0: not asked yet, -1: none
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MARY_MAX_DEVICES) return S == 8 ? 0 : 1;
  int& n = known[dev][S == 1 ? 0 : (S == 2 ? 1 : (S == 4 ? 2 : 3))];
  if (n) return n > 0 ? n : 0;
  static MarySmemSlots smem_set = {};
  if (mary_ensure_dyn_smem((const void*)gemm_pair_kernel<false, false, false, true>, SMEM, &smem_set)) return S == 8 ? 0 : 1;
  if (S == 8 && cudaFuncSetAttribute(gemm_pair_kernel<false, false, false, true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    n = -1;
    return 0;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(mary_num_sms() / (2 * S) * (2 * S));
  cfg.blockDim = dim3(NTHREADS);
  cfg.dynamicSmemBytes = SMEM;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2 * S;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int got = 0;
  if (cudaOccupancyMaxActiveClusters(&got, gemm_pair_kernel<false, false, false, true>, &cfg) != cudaSuccess || got < 1) { cudaGetLastError(); got = S == 8 ? -1 : 1; }
  n = got;
  return got > 0 ? got : 0;
}

// Width (32 .. max_bn) and K split with the smallest estimated time, in ns.  Measured: a K block of 64 takes 1.08 ns per column of the tile (the MMAs) and
// at least 172; with every SM busy the 16 KB + 64 BN bytes that an SM draws for it arrive at 110 GB/s; storing a tile takes 6 ns per column (16 with
// the GLU's exponentials) where no next tile hides it, and never less than that + 0.4 us per tile; an exchange of partial sums 0.5 us + 6.5 ns per
// column and pair (3.6 with 8 pairs, which read more of it at a time); memory gives 6.2 TB/s to all SMs and a quarter less to few of them.  Over 700
// shapes of 3 to 8192 rows, 16 to 3840 outputs and K of 128 to 15360 the choice takes 1.1 % longer on average than the fastest of all widths and splits.
int mary_gemm_pair_plan(int rows_r, int rows_c, int K, bool glu, int max_bn, PairPlan* plan) {
  const int sms = mary_num_sms();
  const int kb = (K + BK - 1) / BK;
  const int tr = (rows_r + 2 * ROWS - 1) / (2 * ROWS);
  const double memory = ((double)rows_c * (glu ? 2 : 1) + rows_r) * K * 2 / 6200.0;
  double best = 0;
  for (int bn = max_bn; bn >= 32; bn -= 32) {
    if (glu && bn < 64) continue;
    const int64_t tc = (rows_c + (glu ? bn / 2 : bn) - 1) / (glu ? bn / 2 : bn);
    for (int S = 1; S <= 8; S *= 2) {
      if (S > 1 && kb < 4 * S) continue;
      if (S > 4 && glu) continue;
      if (glu && bn % (16 * S)) continue;                  // every CTA of the cluster finishes a multiple of 8 outputs
      if (((kb + S - 1) / S) * (S - 1) >= kb) continue;
      const int64_t slots = resident_clusters(S), tiles = tr * tc;
      if (S > 1 && tiles > slots) continue;                // more tiles than clusters: the exchange would not overlap anything
      const int64_t waves = (tiles + slots - 1) / slots;
      const double busy = (double)(tiles < slots ? tiles : slots) * 2 * S / sms;
      const double per = fmax(fmax(1.08 * bn, 172.0), busy * (A_BYTES + bn * 64) / 110.0), store = (glu ? 16.0 : 6.0) * bn;
      double t = fmax((double)waves * fmax(((kb + S - 1) / S) * per, waves > 1 ? store + 390.0 : 0.0), memory * (1.25 - 0.25 * busy));
      t += S > 1 ? 500.0 + (S == 8 ? 3.6 : 6.5) * bn * S : store;
      if (best == 0 || t < best) { best = t; plan->bn = bn; plan->S = S; }
    }
  }
  return best > 0;
}

int mary_gemm_pair_run(const void* R, const void* C, int rows_r, int rows_c, int K, int64_t ldr, int64_t ldc, bool swap, const PairOut& o,
                       const PairPlan& plan, cudaStream_t stream) {
  PairParams p;
  const int bn = plan.bn;
  p.rows_r = rows_r; p.rows_c = rows_c;
  p.bn = bn; p.S = plan.S;
  p.tiles_r = (rows_r + 2 * ROWS - 1) / (2 * ROWS);
  p.tiles_c = (rows_c + (o.glu ? bn / 2 : bn) - 1) / (o.glu ? bn / 2 : bn);
  p.k_blocks = (K + BK - 1) / BK;
  p.kb_per_split = (p.k_blocks + p.S - 1) / p.S;
  if (bn % 32 || bn < 32 || bn > 256 || (o.glu && (swap || bn < 64 || p.S > 4 || bn % (16 * p.S))) || p.kb_per_split * (p.S - 1) >= p.k_blocks) return MARY_ERR_BAD_ARG;
  p.stage_bytes = A_BYTES + bn * BK;                       // BN / 2 rows of 128 bytes
  p.stages = RING / p.stage_bytes;
  if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
  p.raster = (p.tiles_c >= 16 && p.tiles_r >= 4) ? 8 : 0;
  p.act = o.glu ? o.glu - 1 : 0; p.glu_rows = rows_c;
  p.glu_limit = o.glu_limit; p.alpha = o.alpha;
  p.un_act = o.un_act; p.un_cols = o.un_cols;
  p.ldo = o.ldo; p.out = o.out; p.bias = o.bias;
  p.w_static = o.w_static; p.status = mary_status_ptr();
  const int total = p.tiles_r * p.tiles_c;
  const int slots = mary_num_sms() / 2;
  const int clusters = p.S > 1 ? total : (total < slots ? total : slots);
  // f32 results: the tensor core cuts off what an addition of 16 products leaves below the accumulator's last place, always downwards, so the error
  // grows with the length of a chain.  TMEM columns that the tile leaves free take further accumulators, until no chain is longer than the one-SM kernel's
  // dealing of K among all SMs makes it (at most 16 parts, at least 4 blocks), 3 x 128 x 7168: relative error 1.9e-6 -> 4e-7.
  p.acc_stride = bn <= 32 ? 32 : (bn <= 64 ? 64 : (bn <= 128 ? 128 : 256));
  p.n_acc = 1;
  if (o.f32 && !o.glu) {
    const int sms = mary_num_sms(), fit = (total <= clusters ? 512 : 256) / p.acc_stride;
    const int m = swap ? rows_c : rows_r, n = swap ? rows_r : rows_c;
    const int64_t tiles = m <= 256 ? (n + 127) / 128 : (int64_t)((m + 127) / 128) * ((n + 63) / 64);
    int chain = (int)((tiles * p.k_blocks + sms - 1) / sms);
    if (chain < (p.k_blocks + 15) / 16) chain = (p.k_blocks + 15) / 16;
    if (chain < 4) chain = 4;
    const int want = (p.kb_per_split + chain - 1) / chain;
    p.n_acc = want < fit ? want : fit;
  }
  CUtensorMap tr, tc;
  int rc = mary_make_tmap_2d(&tr, R, 4, rows_r, K, ldr, ROWS, BK, 1);
  if (rc) return rc;
  rc = mary_make_tmap_2d(&tc, C, 4, o.glu ? 2 * (uint64_t)rows_c : rows_c, K, ldc, bn / 2, BK, 1);
  if (rc) return rc;
  CUtensorMap to = tr;                                     // only read when tma_box is set
  p.tma_box = 0;
  if (!swap && p.S == 1 && ((uintptr_t)o.out & 15) == 0 && (o.ldo & (o.f32 ? 3 : 7)) == 0 && rows_c >= 32) {
    p.tma_box = (o.f32 || (o.glu && bn % 64)) ? 16 : 32;
    rc = store_map(&to, o.out, o.f32, rows_r, o.group > 0 ? rows_c / o.group * o.pitch : rows_c, o.ldo, p.tma_box);
    if (rc) return rc;
  }
  p.group = o.group; p.pitch = o.pitch;
  if (o.group > 0 && (p.tma_box != 32 || o.group % 32 || rows_c % o.group || o.pitch < o.group || o.pitch % 8)) return MARY_ERR_BAD_ARG;
  auto go = [&](auto glu, auto sw, auto f32) {
    return p.S > 1 ? launch<glu, sw, f32, true>(tr, tc, to, p, clusters, stream) : launch<glu, sw, f32, false>(tr, tc, to, p, clusters, stream);
  };
  const std::true_type yes;
  const std::false_type no;
  if (o.glu) return o.f32 ? go(yes, no, yes) : go(yes, no, no);
  if (swap) return o.f32 ? go(no, yes, yes) : go(no, yes, no);
  return o.f32 ? go(no, no, yes) : go(no, no, no);
}

// The kernel with a given width (a multiple of 32) and K split; swap as in mary_gemm_bf16.  glu: 0, or 1 + kind.
MARY_API int mary_gemm_bf16_pair(const void* X, const void* W, void* out, int M, int N, int K, int64_t ldx, int64_t ldw, int64_t ldo, int glu, int out_f32,
                                 int bn, int splits, int swap, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0 || (K & 7) || (ldx & 7) || (ldw & 7) || (splits != 1 && splits != 2 && splits != 4 && splits != 8)) return MARY_ERR_BAD_ARG;
  if (splits == 8 && resident_clusters(8) < 1) return MARY_ERR_BAD_ARG;
  PairOut o = {out, ldo, out_f32, glu, 0.f, 1.0f, 0, 0, nullptr, 0, 0, 0};
  PairPlan plan = {bn, splits};
  return swap ? mary_gemm_pair_run(W, X, N, M, K, ldw, ldx, true, o, plan, stream) : mary_gemm_pair_run(X, W, M, N, K, ldx, ldw, false, o, plan, stream);
}

// out[i, (j / group) * pitch + j % group] = X_i . W_j, bf16: the heads of a projection at a pitch of their own (group: a multiple of 32, N of group; rows of
// ldo elements, 16-byte aligned).  The values between the groups are not written.
MARY_API int mary_gemm_bf16_grouped_columns(const void* X, const void* W, void* out, int M, int N, int K, int64_t ldx, int64_t ldw, int64_t ldo, int group,
                                            int pitch, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0 || group <= 0 || (K & 7) || (ldx & 7) || (ldw & 7)) return MARY_ERR_BAD_ARG;
  PairOut o = {out, ldo, 0, 0, 0.f, 1.0f, 0, 0, nullptr, 0, group, pitch};
  PairPlan plan;
  if (!mary_gemm_pair_plan(M, N, K, false, 256, &plan)) return MARY_ERR_BAD_ARG;
  if (plan.S > 1) plan = {128, 1};                         // the exchange of a split stores plainly
  return mary_gemm_pair_run(X, W, M, N, K, ldx, ldw, false, o, plan, stream);
}
