// bf16 GEMM on CTA pairs (tcgen05 cta_group::2), optionally fused with a tensor-parallel collective.
//
//   C[M,N] (+)= op(A) * op(B)     same operand layouts as tplr_gemm_bf16 (K-major or MN-major)
//
// A cluster of two CTAs computes one tile of 256 rows and 256, 192 or 128 columns (see plan_cost): each CTA stages its own
// 128 rows of A and its own half of the tile's rows of B (so every shared-memory byte feeds two SMs' tensor cores), the even
// CTA issues tcgen05.mma.cta_group::2, and each CTA drains its 128 rows of the accumulator from its own tensor memory.  A ring
// of 192 KB per CTA (6 stages at 256 and 192 columns, 8 at 128), two accumulator buffers.
// The producer and the issuer are warp-uniform loops with one elected lane behind the issuing statements (see elect_one):
// 505 cycles a k block of 64 at 256 columns, which is the tensor pipe's 512 within the clock readings, for every operand layout; under
// `lane == 0` 620 to 625.  2048 x 18944 x 2048 (8 tiles a pair): 113 -> 102 us K-major, 123 -> 102 us MN-major.
//
// Fused collectives (one process per GPU, peers mapped through the symmetric heap):
//   gather  (all-gather -> GEMM): trailing "comm" CTAs of the same launch pull the peers' row
//           shards of one operand into this GPU's full buffer with bulk copies, 128 rows at a
//           time, and release one flag per 128 rows; the TMA producer of a compute CTA waits
//           (bounded) for the flags of the rows it is about to load.  Every remote byte crosses
//           NVLink once and the tiles of the local shard start at once.
//   scatter (GEMM -> reduce-scatter): the epilogue of every tile reduce-adds its 32 x 128-byte boxes
//           (bf16 or fp32) with TMA straight into the buffer of the rank that owns those rows, over
//           NVLink for a peer and in the local L2 for itself; tile rows are visited so that all
//           owners receive traffic all the time.  No staging buffer, no second pass.
// No load in this file carries a cluster-multicast qualifier; only tcgen05.commit does.
// Every wait is bounded by wall time; on expiry TPLR_ST_WAIT_TIMEOUT is set and all roles return.
//
// Replaces cuBLAS + NCCL behind the reference's tensor-parallel plan: colwise q/k/v/w1/w3,
// rowwise wo/w2 with sequence-sharded activations (torchtitan models/llama3/infra/parallelize.py:151-219).
#include "tcgen05.cuh"
#include <stdlib.h>

namespace {
using namespace tplr_tc;

constexpr int TILE_M = 256, CTA_M = 128, TILE_N = 256, CTA_N = 128, BK = 64, STAGES = 6, UMMA_K = 16;
constexpr int A_STAGE = CTA_M * BK * 2;            // 16 KB
constexpr int B_STAGE = CTA_N * BK * 2;            // 16 KB
constexpr int STAGE_BYTES = A_STAGE + B_STAGE;     // 32 KB
constexpr int EPI_STAGE_BYTES = 4 * 2 * 4096;      // 4 epilogue warps x 2 buffers x (32 rows x 128 B)
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_STAGE_BYTES + 1024;
constexpr int EPI5_STAGES = STAGES - 1;            // the SwiGLU backward has a second pair of staging buffers per warp instead
constexpr int MAX_STAGES = 8;                      // narrower tiles have smaller stages, so more of them fit the ring
static_assert(4 * 8192 <= STAGE_BYTES, "the freed stage holds four warps' second pair");
constexpr int NUM_THREADS = 192;
constexpr int MAX_RANKS = 8;
constexpr int CHUNK_ROWS = 128;                    // gather / scatter flag granularity (rows)

struct Gemm2Params {
  CUtensorMap tmA, tmB;
  CUtensorMap tmC;                   // output: box 64 x 32 bf16 or 32 x 32 fp32, 128-byte swizzle
  int c_tma;                         // 1: epilogue through TMA, 0: direct stores (unaligned C)
  CUtensorMap tmCr[MAX_RANKS];       // scatter: rank o's owned rows [rows_per_rank, N], same box as tmC
  void* C;
  long long ldc;
  int M, N, K;
  unsigned int* status;
  int tile_n;                        // columns of a pair's tile: 256, 192 or 128 (see plan_cost); each CTA stages half of them
  int n_compute_pairs;               // CTA pairs [0, n_compute_pairs) compute, the rest are comm CTAs
  int group_m;                       // tile order: bands of group_m tile rows, tile row fastest inside a band
  int m_rot;                         // rotation of the tile-row order (in 256-row tiles)
  int n_rot;                         // rotation of the tile-column order (in 256-column tiles)
  int m_inter;                       // > 1: logical tile row l is row (l % m_inter) * (tiles_m / m_inter) + l / m_inter
  int k_splits;                      // > 1 (reduce-add epilogues, or with plane_rows): a tile's K range is cut into this many work units
  int plane_rows;                    // > 0: the parts of a tile's K range go to planes of plane_rows rows, part s to plane s of tmC
                                     // (EPI 2), or part 0 into tmC and part s to plane s - 1 of tmCr[0] (EPI 1)
  int tri;                           // 1: C is symmetric (B is A): only tiles on or above the diagonal are computed
  int swiglu_f;                      // > 0 (EPI 3): B is the packed [w1; w3] weight of 2 * swiglu_f rows.  Tile column j pairs
                                     // gate rows [128 j, 128 j + 128) (staged by the even CTA) with up rows swiglu_f + the same
                                     // (odd CTA), so every accumulator row holds g and u of the same 128 features; the epilogue
                                     // stores both into C [M, 2 * swiglu_f] and silu(g) * u into tmCr[0]'s tensor [M, swiglu_f]
  // backward of the SwiGLU in the epilogue of the down projection's data gradient (EPI 5): the accumulator tile is
  // dh[M, swiglu_f] = dY W2; tmGU is the forward's packed [M, 2 * swiglu_f] projection (gate | up);
  // the epilogue stores dg | du (bf16) through tmC, a map over the [M, 2 * swiglu_f] gradient of that projection
  CUtensorMap tmGU;                  // EPI 5: the packed projection, box 64 x 32, 128-byte swizzle
  const __nv_bfloat16* gu;
  long long ld_gu;
  // data gradient of the attention output projection (EPI 6): C = dO [M, heads * attn_dh] stored as bf16, and for every row
  // and head delta = sum over the head's attn_dh (128 or 64) columns of dO * O, with O = gu (leading dimension ld_gu), written to
  // attn_delta[(row / attn_s * heads + head) * attn_s + row % attn_s]
  float* attn_delta;
  int attn_s, attn_heads, attn_dh;
  // rotary embedding in the epilogue (EPI 4): the first rope_cols columns of C are heads of rope_dh columns whose
  // interleaved pairs (2i, 2i + 1) are rotated by the angle of (row % rope_s, i); tables [rope_s, rope_dh / 2] fp32
  const float* rope_cos;
  const float* rope_sin;
  int rope_s, rope_cols, rope_dh;
  int world, rank;
  unsigned int epoch;
  // gather
  int ag_operand;                    // 0 none, 1 A, 2 B
  int ag_rows_per_rank;              // rows (outer dimension) of the gathered operand per rank
  long long ag_row_bytes;            // bytes of one dense row
  const uint8_t* ag_src[MAX_RANKS];  // base of every rank's full buffer (own entry unused)
  uint8_t* ag_dst;                   // base of this rank's full buffer
  unsigned int* ag_flags;            // one per CHUNK_ROWS rows of the full buffer (local memory)
  // scatter
  int rs_on;
  int rs_bound[MAX_RANKS + 1];       // owner o holds rows [rs_bound[o], rs_bound[o + 1]) of C; multiples of 32
};

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address of `saddr` (a shared::cta address of this CTA) inside CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA tile load of a CTA pair: data lands in this CTA, completion bytes go to `bar` which may live in the peer CTA.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar_cluster), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// Descriptors are given as (low word, high word): the low word carries the start address (bytes >> 4), so the
// issuing thread advances an operand by one 32-bit add instead of rebuilding a 64-bit descriptor per instruction.
__device__ __forceinline__ void umma_bf16_pair_lohi(uint32_t tmem_d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                                    uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "mov.b64 da, {%1, %2};\n\t"
      "mov.b64 db, {%3, %4};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %5, p;\n\t}"
      ::"r"(tmem_d), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void bulk_s2g(void* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async;" ::: "memory"); }

__device__ __forceinline__ unsigned int ld_acquire_gpu(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned int ld_acquire_sys(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_gpu(unsigned int* p, unsigned int v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Bounded wait for *flag == want (flags carry the call's epoch).  SYS selects the scope of the acquire.
template <bool SYS>
__device__ __forceinline__ bool flag_wait(const unsigned int* flag, unsigned int want, volatile int* abort_flag) {
  unsigned long long t0 = 0;
  for (uint32_t i = 0;; ++i) {
    const unsigned int v = SYS ? ld_acquire_sys(flag) : ld_acquire_gpu(flag);
    if (v == want) return true;
    if ((i & 7u) == 7u) {
      if (*abort_flag) return false;
      const unsigned long long now = gtimer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > WAIT_LIMIT_NS) break;
    }
  }
  *abort_flag = 1;
  return false;
}

// The work units of one CTA pair, walked identically by its producer, MMA and epilogue roles: units pair, pair + P,
// ... of the (tile, k split) list, k split fastest.  (A stream-K cut of the flattened (tile, k block) space, every pair
// an equal contiguous run, was measured on the weight-gradient shapes and lost 20-25 % to this static order: pairs
// that share operand tiles stop running in step, and the L2 reuse between them goes.)
struct Work {
  int t;                             // unit index
  int tile, kb0, nkb;                // current unit: tile index, first k block, k blocks
};
__device__ __forceinline__ void work_init(const Gemm2Params& p, Work& w, int pair) { w.t = pair; }
__device__ __forceinline__ bool work_get(const Gemm2Params& p, Work& w, int tiles, int k_blocks_all, int k_per) {
  if (w.t >= tiles * p.k_splits) return false;
  w.tile = w.t / p.k_splits;
  w.kb0 = (w.t % p.k_splits) * k_per;
  w.nkb = min(k_per, k_blocks_all - w.kb0);
  return true;
}
__device__ __forceinline__ void work_next(const Gemm2Params& p, Work& w) { w.t += p.n_compute_pairs; }

// tile index -> (tile row, tile column) under the launch's order
__device__ __forceinline__ void tile_coords(const Gemm2Params& p, int t, int tiles_m, int tiles_n, int& tm, int& tn) {
  if (p.tri) {                       // t-th tile of the upper triangle, row by row: row i holds tiles_n - i tiles
    int i = 0, left = t;
    while (left >= tiles_n - i) { left -= tiles_n - i; ++i; }
    tm = i;
    tn = i + left;
    return;
  }
  const int band = p.group_m * tiles_n;
  const int g = t / band, first = g * p.group_m;
  const int rows = p.group_m < tiles_m - first ? p.group_m : tiles_m - first;
  const int in = t - g * band;
  int tml = first + in % rows;
  tn = in / rows;
  if (p.m_inter > 1) tml = (tml % p.m_inter) * (tiles_m / p.m_inter) + tml / p.m_inter;
  tm = tml + p.m_rot;
  if (tm >= tiles_m) tm -= tiles_m;
  tn += p.n_rot;
  if (tn >= tiles_n) tn -= tiles_n;
}

// Epilogue without TMA (C not 16-byte aligned or odd leading dimension): each lane stores its own row.
template <int EPI>
__device__ __forceinline__ void epilogue_direct(const Gemm2Params& p, uint32_t tmem_acc, int quad, int lane, int m0, int n0) {
  const int row = m0 + quad * 32 + lane;
#pragma unroll 1
  for (int c = 0; c < p.tile_n / 32; ++c) {
    uint32_t r[32];
    tmem_ld32(tmem_acc + c * 32 + ((uint32_t)(quad * 32) << 16), r);
    const int col0 = n0 + c * 32;
    if (row < p.M && col0 < p.N) {
      if (EPI == 0 || EPI >= 3) {      // (the epilogue modes 3-5 never take this path: their entries require TMA stores)
        __nv_bfloat16* crow = reinterpret_cast<__nv_bfloat16*>(p.C) + (long long)row * p.ldc + col0;
        for (int e = 0; e < 32 && col0 + e < p.N; ++e) crow[e] = __float2bfloat16(__uint_as_float(r[e]));
      } else {
        float* crow = reinterpret_cast<float*>(p.C) + (long long)row * p.ldc + col0;
        for (int e = 0; e < 32 && col0 + e < p.N; ++e) {
          const float o = __uint_as_float(r[e]);
          crow[e] = (EPI == 1) ? crow[e] + o : o;
        }
      }
    }
  }
}

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(map), "r"(src), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* map, uint32_t src, int x, int y) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(map), "r"(src), "r"(x), "r"(y) : "memory");
}

// Rotary angles of one output row for a whole tile (EPI 4): the tile's heads share them, so a lane loads the head's DH / 2
// cosines and sines once into registers.  Loaded again for every 32 columns they cost 32 cache lines per instruction (each
// lane has a row of its own), which made the epilogue longer than a short main loop.  16384 x 768 -> 2304, heads of 64:
// 81 us then, 59 us here.
template <int DH>
struct RopeRow {
  float c[DH / 2], s[DH / 2];
  __device__ __forceinline__ void load(const Gemm2Params& p, int row) {
    const long long tb = (long long)(row % p.rope_s) * (DH / 2);
    const float4* cp = reinterpret_cast<const float4*>(p.rope_cos + tb);
    const float4* sp = reinterpret_cast<const float4*>(p.rope_sin + tb);
#pragma unroll
    for (int q = 0; q < DH / 8; ++q) {
      const float4 a = cp[q], b = sp[q];
      c[4 * q] = a.x; c[4 * q + 1] = a.y; c[4 * q + 2] = a.z; c[4 * q + 3] = a.w;
      s[4 * q] = b.x; s[4 * q + 1] = b.y; s[4 * q + 2] = b.z; s[4 * q + 3] = b.w;
    }
  }
  // 32 columns from column OFF of a head on
  template <int OFF>
  __device__ __forceinline__ void turn(uint32_t* r) const {
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const float a = __uint_as_float(r[2 * e]), b = __uint_as_float(r[2 * e + 1]);
      r[2 * e] = __float_as_uint(a * c[OFF / 2 + e] - b * s[OFF / 2 + e]);
      r[2 * e + 1] = __float_as_uint(a * s[OFF / 2 + e] + b * c[OFF / 2 + e]);
    }
  }
};

// Epilogue through shared memory and TMA: a warp stages 32 rows x 128 bytes (64 bf16 or 32 fp32
// columns) in 128-byte-swizzled order, then one lane stores (EPI 0, 2) or reduce-adds (EPI 1) the
// box.  Two staging buffers per warp; `n_boxes` counts the boxes this warp has issued so far.
template <int EPI>
__device__ __forceinline__ void epilogue_tma(const Gemm2Params& p, uint32_t tmem_acc, int quad, int lane, int m0, int n0,
                                             uint32_t stage_base, uint32_t& n_boxes, int part) {
  constexpr bool BF16_OUT = EPI == 0 || EPI == 4;
  constexpr int COLS = BF16_OUT ? 64 : 32;
  const int row0 = m0 + quad * 32;
  const uint32_t sw = (uint32_t)(lane & 7);
  const CUtensorMap* map = &p.tmC;
  int y = EPI == 2 ? row0 + part * p.plane_rows : row0;
  const bool plane = EPI == 1 && p.plane_rows > 0 && part > 0;
  if (plane) { map = &p.tmCr[0]; y = row0 + (part - 1) * p.plane_rows; }
  if (p.rs_on && row0 < p.M) {                       // the 32 rows of a warp have one owner (32 | every bound)
    int owner = 0;
    while (owner + 1 < p.world && row0 >= p.rs_bound[owner + 1]) ++owner;
    map = &p.tmCr[owner];
    y = row0 - p.rs_bound[owner];
  }
#pragma unroll 1
  for (int c = 0; c < p.tile_n / COLS; ++c) {
    const int col0 = n0 + c * COLS;
    if (row0 >= p.M || col0 >= p.N) break;          // warp-uniform: nothing of this box is inside C
    const uint32_t buf = stage_base + (n_boxes & 1u) * 4096u;
    if (n_boxes >= 2) {                              // the box issued two steps ago has left this buffer
      if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
      __syncwarp();
    }
    const uint32_t rowaddr = buf + (uint32_t)lane * 128u;
    if (BF16_OUT) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t r[32];
        tmem_ld32(tmem_acc + c * 64 + h * 32 + ((uint32_t)(quad * 32) << 16), r);
        if (EPI == 4 && col0 + h * 32 < p.rope_cols) {
          // rotary pairs of this lane's token: 16 angles starting at pair ((col % head) / 2) of position row % S
          const int row = min(row0 + lane, p.M - 1);
          const long long tb = (long long)(row % p.rope_s) * (p.rope_dh / 2) + ((col0 + h * 32) % p.rope_dh) / 2;
          const float4* cp = reinterpret_cast<const float4*>(p.rope_cos + tb);
          const float4* sp = reinterpret_cast<const float4*>(p.rope_sin + tb);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float4 cv = cp[q], sv = sp[q];
            const float cc[4] = {cv.x, cv.y, cv.z, cv.w}, ss[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float a = __uint_as_float(r[8 * q + 2 * e]), b = __uint_as_float(r[8 * q + 2 * e + 1]);
              r[8 * q + 2 * e] = __float_as_uint(a * cc[e] - b * ss[e]);
              r[8 * q + 2 * e + 1] = __float_as_uint(a * ss[e] + b * cc[e]);
            }
          }
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          uint32_t pw[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            __nv_bfloat162 hh = __floats2bfloat162_rn(__uint_as_float(r[8 * v + 2 * e]), __uint_as_float(r[8 * v + 2 * e + 1]));
            pw[e] = *reinterpret_cast<uint32_t*>(&hh);
          }
          const uint32_t j = (uint32_t)(h * 4 + v);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(rowaddr + ((j ^ sw) << 4)), "r"(pw[0]), "r"(pw[1]),
                       "r"(pw[2]), "r"(pw[3]) : "memory");
        }
      }
    } else {
      uint32_t r[32];
      tmem_ld32(tmem_acc + c * 32 + ((uint32_t)(quad * 32) << 16), r);
#pragma unroll
      for (int v = 0; v < 8; ++v)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(rowaddr + (((uint32_t)v ^ sw) << 4)), "r"(r[4 * v]),
                     "r"(r[4 * v + 1]), "r"(r[4 * v + 2]), "r"(r[4 * v + 3]) : "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
      if ((EPI == 1 && !plane) || p.rs_on) tma_reduce_add_2d(map, buf, col0, y);
      else                     tma_store_2d(map, buf, col0, y);
      bulk_commit();
    }
    ++n_boxes;
  }
}

// Staging of one 32 x 64 bf16 box in two halves of 32 columns (same double-buffer protocol as epilogue_tma):
// box_begin waits until the buffer is free, box_half writes this lane's 32 values of half `hh`, box_store issues the store.
__device__ __forceinline__ uint32_t box_begin(int lane, uint32_t stage_base, uint32_t n_boxes) {
  if (n_boxes >= 2) {
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
    __syncwarp();
  }
  return stage_base + (n_boxes & 1u) * 4096u;
}
__device__ __forceinline__ void box_half(uint32_t buf, int lane, int hh, const float* v) {
  const uint32_t rowaddr = buf + (uint32_t)lane * 128u, sw = (uint32_t)(lane & 7);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t pw[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      __nv_bfloat162 b2 = __floats2bfloat162_rn(v[8 * j + 2 * e], v[8 * j + 2 * e + 1]);
      pw[e] = *reinterpret_cast<uint32_t*>(&b2);
    }
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(rowaddr + (((uint32_t)(hh * 4 + j) ^ sw) << 4)), "r"(pw[0]),
                 "r"(pw[1]), "r"(pw[2]), "r"(pw[3]) : "memory");
  }
}
__device__ __forceinline__ void box_store(const CUtensorMap* map, uint32_t buf, int lane, uint32_t& n_boxes, int col0, int row0) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  if (lane == 0) {
    tma_store_2d(map, buf, col0, row0);
    bulk_commit();
  }
  ++n_boxes;
}

// The plain bf16 epilogue with the rotation, for heads of DH columns (tiles and heads start at multiples of DH).
template <int DH>
__device__ __forceinline__ void epilogue_rope(const Gemm2Params& p, uint32_t tmem_acc, int quad, int lane, int m0, int n0,
                                              uint32_t stage_base, uint32_t& n_boxes) {
  const int row0 = m0 + quad * 32;
  if (row0 >= p.M) return;                           // warp-uniform
  const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
  RopeRow<DH> rr;
  if (n0 < p.rope_cols) rr.load(p, min(row0 + lane, p.M - 1));
#pragma unroll 1
  for (int h = 0; h < p.tile_n / DH; ++h) {
    if (n0 + h * DH >= p.N) break;
    const bool rot = n0 + h * DH < p.rope_cols;      // whole heads (rope_cols is a multiple of DH)
#pragma unroll
    for (int q = 0; q < DH / 64; ++q) {
      const int col = h * DH + q * 64;
      if (n0 + col >= p.N) break;
      const uint32_t buf = box_begin(lane, stage_base, n_boxes);
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        uint32_t r[32];
        float v[32];
        tmem_ld32(tmem_acc + col + hh * 32 + lane_sel, r);
        if (rot) {
          if (q == 0 && hh == 0) rr.template turn<0>(r);
          if (q == 0 && hh == 1) rr.template turn<32>(r);
          if (q == 1 && hh == 0) rr.template turn<DH / 2>(r);
          if (q == 1 && hh == 1) rr.template turn<DH - 32>(r);
        }
#pragma unroll
        for (int e = 0; e < 32; ++e) v[e] = __uint_as_float(r[e]);
        box_half(buf, lane, hh, v);
      }
      box_store(&p.tmC, buf, lane, n_boxes, n0 + col, row0);
    }
  }
}

// Epilogue of the fused [w1; w3] projection (EPI 3): the first half of a row's accumulator columns are the gate values g of
// features [h tn, h tn + h) with h = tile_n / 2, the second half the up values u of the same features.  Per 64 features: g and
// u go to C (bf16, columns h tn + .. and swiglu_f + h tn + ..: what the backward pass reads) and h = silu(g) * u, computed from the fp32
// accumulators, goes to the [M, swiglu_f] tensor behind tmCr[0].  Replaces a separate pass that re-reads g and u
// (the reference's F.silu(w1(x)) * w3(x), torchtitan models/llama3/model/model.py FeedForward.forward).
// The accumulators are read twice (once for the g / u boxes, once for h): tensor-memory loads are cheap and 32 values
// at a time keep the register count of the epilogue warps where it was.
__device__ __forceinline__ void epilogue_swiglu(const Gemm2Params& p, uint32_t tmem_acc, int quad, int lane, int m0, int tn,
                                                uint32_t stage_base, uint32_t& n_boxes) {
  const int row0 = m0 + quad * 32;
  if (row0 >= p.M) return;                           // warp-uniform
  const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
  const int half = p.tile_n / 2;                     // features of a tile
#pragma unroll 1
  for (int c = 0; c < half / 64; ++c) {
    const int f0 = tn * half + c * 64;               // first feature of this box
    if (f0 >= p.swiglu_f) break;
#pragma unroll 1
    for (int part = p.C ? 0 : 2; part < 2; ++part) { // 0: g box, 1: u box; a caller without a backward pass has no C
      const uint32_t buf = box_begin(lane, stage_base, n_boxes);
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        uint32_t r[32];
        float v[32];
        tmem_ld32(tmem_acc + part * half + c * 64 + hh * 32 + lane_sel, r);
#pragma unroll
        for (int e = 0; e < 32; ++e) v[e] = __uint_as_float(r[e]);
        box_half(buf, lane, hh, v);
      }
      box_store(&p.tmC, buf, lane, n_boxes, part * p.swiglu_f + f0, row0);
    }
    const uint32_t buf = box_begin(lane, stage_base, n_boxes);
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      uint32_t rg[32], ru[32];
      float v[32];
      tmem_ld32(tmem_acc + c * 64 + hh * 32 + lane_sel, rg);
      tmem_ld32(tmem_acc + half + c * 64 + hh * 32 + lane_sel, ru);
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        const float g = __uint_as_float(rg[e]);
        v[e] = __fdividef(g, 1.f + __expf(-g)) * __uint_as_float(ru[e]);            // silu(g) * u
      }
      box_half(buf, lane, hh, v);
    }
    box_store(&p.tmCr[0], buf, lane, n_boxes, f0, row0);
  }
}

// Epilogue of the down projection's data gradient fused with the backward of the SwiGLU (EPI 5).  The accumulator row
// holds dh for 256 features; with g and u of the same row and features read from the forward's packed projection,
//   s = sigmoid(g),  du = dh * g * s,  dg = dh * u * s * (1 + g * (1 - s)),
// and dg / du are stored (bf16) at columns f and swiglu_f + f of the packed gradient.  This replaces a pass that writes
// dh, reads it back with g and u and writes dg | du (the backward of the reference's F.silu(w1(x)) * w3(x)).
// g and u come as TMA boxes of 32 rows x 64 columns into the staging buffers that dg and du leave from, in place: a lane
// reading its own row from global memory touches 32 lines per instruction, which made the epilogue longer than the main loop
// (2048 x 768 -> 3072: 67 -> 41 us in one run of all its products; 16384 x 2048 -> 8192: 651 -> 542 us).  Two pairs of buffers per warp (the operand ring has one stage less for them): the next
// pair is in flight while this one is computed, the first of a tile while its main loop runs.
struct GuLoads {
  uint32_t bar;                      // two mbarriers of this warp
  uint32_t base;                     // two pairs of 4 KB buffers
  uint32_t issued, used;             // box pairs asked for and consumed so far
};
__device__ __forceinline__ void gu_issue(const Gemm2Params& p, GuLoads& L, int lane, int f0, int row0) {
  if (lane == 0) {
    const uint32_t s = L.issued & 1u, bar = L.bar + 8u * s, buf = L.base + s * 8192u;
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");      // the stores that leave from this pair have read it
    mbar_expect_tx(bar, 8192);
    tma_load_2d(buf, &p.tmGU, bar, f0, row0);
    tma_load_2d(buf + 4096u, &p.tmGU, bar, p.swiglu_f + f0, row0);
  }
  ++L.issued;
}
__device__ __forceinline__ bool epilogue_swiglu_bwd(const Gemm2Params& p, uint32_t tmem_acc, int quad, int lane, int m0, int n0,
                                                    GuLoads& L, volatile int* abort_flag) {
  const int row0 = m0 + quad * 32;
  if (row0 >= p.M || n0 >= p.swiglu_f) return true;  // warp-uniform; nothing was asked for
  const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
  const uint32_t sw = (uint32_t)(lane & 7);
#pragma unroll 1
  for (int c = 0; c < p.tile_n / 64; ++c) {
    const int f0 = n0 + c * 64;
    if (f0 >= p.swiglu_f) break;                     // warp-uniform (swiglu_f is a multiple of 64)
    if (c + 1 < p.tile_n / 64 && f0 + 64 < p.swiglu_f) gu_issue(p, L, lane, f0 + 64, row0);
    const uint32_t s = L.used & 1u;
    const bool ok = mbar_wait(L.bar + 8u * s, (L.used >> 1) & 1u, abort_flag);
    if (!__all_sync(0xffffffffu, ok)) return false;
    ++L.used;
    const uint32_t grow = L.base + s * 8192u + (uint32_t)lane * 128u, urow = grow + 4096u;
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      uint32_t r[32];
      tmem_ld32(tmem_acc + c * 64 + hh * 32 + lane_sel, r);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t off = ((uint32_t)(hh * 4 + q) ^ sw) << 4;
        uint32_t gw[4], uw[4];
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(gw[0]), "=r"(gw[1]), "=r"(gw[2]), "=r"(gw[3]) : "r"(grow + off) : "memory");
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(uw[0]), "=r"(uw[1]), "=r"(uw[2]), "=r"(uw[3]) : "r"(urow + off) : "memory");
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 g2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gw[e]));
          const float2 u2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&uw[e]));
          const float gg[2] = {g2.x, g2.y}, uu[2] = {u2.x, u2.y};
          float dg[2], du[2];
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const float dh = __uint_as_float(r[8 * q + 2 * e + k]);
            const float sg = __fdividef(1.f, 1.f + __expf(-gg[k]));
            const float silu = gg[k] * sg;
            du[k] = dh * silu;
            dg[k] = dh * uu[k] * (sg + silu * (1.f - sg));
          }
          const __nv_bfloat162 hg = __floats2bfloat162_rn(dg[0], dg[1]), hu = __floats2bfloat162_rn(du[0], du[1]);
          gw[e] = *reinterpret_cast<const uint32_t*>(&hg);
          uw[e] = *reinterpret_cast<const uint32_t*>(&hu);
        }
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(grow + off), "r"(gw[0]), "r"(gw[1]), "r"(gw[2]), "r"(gw[3]) : "memory");
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(urow + off), "r"(uw[0]), "r"(uw[1]), "r"(uw[2]), "r"(uw[3]) : "memory");
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
      tma_store_2d(&p.tmC, L.base + s * 8192u, f0, row0);
      tma_store_2d(&p.tmC, L.base + s * 8192u + 4096u, p.swiglu_f + f0, row0);
      bulk_commit();
    }
  }
  return true;
}

// Epilogue of the attention output projection's data gradient (EPI 6): the accumulator row is dO for two
// heads of 128 columns or four of 64.  dO is stored as bf16 like a plain epilogue; on the way every lane multiplies its (bf16-rounded) values
// with the forward's attention output O of the same row and sums per head, which is the `delta` term of the attention
// backward (the row sum of dO * O): no separate pass over dO and O.  O is fetched one step of 32 columns ahead.
__device__ __forceinline__ void epilogue_attn_dout(const Gemm2Params& p, uint32_t tmem_acc, int quad, int lane, int m0, int n0,
                                                   uint32_t stage_base, uint32_t& n_boxes) {
  const int row0 = m0 + quad * 32;
  if (row0 >= p.M) return;                           // warp-uniform
  const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
  const int row = min(row0 + lane, p.M - 1);
  const bool live = row0 + lane < p.M;
  const __nv_bfloat16* orow = p.gu + (long long)row * p.ld_gu;
  const long long drow = (long long)(row / p.attn_s) * p.attn_heads * p.attn_s + row % p.attn_s;
  uint4 oq[4], on[4];
  auto fetch = [&](int step, uint4* o4) {
    const int f = n0 + step * 32;
    if (f < p.N) {
      const uint4* op = reinterpret_cast<const uint4*>(orow + f);
#pragma unroll
      for (int q = 0; q < 4; ++q) o4[q] = op[q];
    }
  };
  fetch(0, oq);
  float acc = 0.f;
  const int steps = p.tile_n / 32;
#pragma unroll 2
  for (int step = 0; step < steps; ++step) {
    const int c = step >> 1, hh = step & 1;
    const int f0 = n0 + c * 64;
    if (f0 >= p.N) break;                            // warp-uniform (N is a multiple of 64)
    if (step + 1 < steps) fetch(step + 1, on);
    uint32_t buf = 0;
    if (hh == 0) buf = box_begin(lane, stage_base, n_boxes); else buf = stage_base + (n_boxes & 1u) * 4096u;
    uint32_t r[32];
    tmem_ld32(tmem_acc + c * 64 + hh * 32 + lane_sel, r);
    float v[32];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t ow[4] = {oq[q].x, oq[q].y, oq[q].z, oq[q].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 o2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ow[e]));
        // the attention kernels read dO as bf16: the sum is taken over the values they will see
        const __nv_bfloat162 d2 = __floats2bfloat162_rn(__uint_as_float(r[8 * q + 2 * e]), __uint_as_float(r[8 * q + 2 * e + 1]));
        const float2 df = __bfloat1622float2(d2);
        v[8 * q + 2 * e] = df.x; v[8 * q + 2 * e + 1] = df.y;
        acc = fmaf(df.x, o2.x, acc);
        acc = fmaf(df.y, o2.y, acc);
      }
    }
    box_half(buf, lane, hh, v);
    if (hh == 1) box_store(&p.tmC, buf, lane, n_boxes, f0, row0);
    if (((step + 1) * 32) % p.attn_dh == 0) {        // a head is complete
      const int head = (n0 + step * 32) / p.attn_dh;
      if (live) p.attn_delta[drow + (long long)head * p.attn_s] = acc;
      acc = 0.f;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) oq[q] = on[q];
  }
}

// EPI: 0 store bf16, 1 fp32 accumulate (C += acc), 2 store fp32, 3 fused SwiGLU of a packed [w1; w3] projection,
// 4 store bf16 with the rotary embedding applied to the leading columns, 5 backward of the SwiGLU on the data gradient
// of the down projection, 6 data gradient of the attention output projection with the attention backward's delta term
template <bool A_MN, bool B_MN, int EPI>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm2_kernel(const __grid_constant__ Gemm2Params p) {
  constexpr int RING_BYTES = (EPI == 5 ? EPI5_STAGES : STAGES) * STAGE_BYTES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t bar_full[MAX_STAGES], bar_empty[MAX_STAGES], bar_tfull[2], bar_tempty[2];
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;
  __shared__ __align__(8) uint64_t bar_gu[EPI == 5 ? 8 : 1];      // EPI 5: two per epilogue warp
  __shared__ uint32_t s_ready[32];   // gather: bit c set once chunk c was seen ready (1024 chunks)

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const uint32_t cr = cluster_ctarank();
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const bool is_compute = pair < p.n_compute_pairs;
  const int tile_n = p.tile_n, cta_n = tile_n / 2;                  // cta_n: columns of B that each CTA stages
  const uint32_t b_stage = B_MN ? (uint32_t)((cta_n + 63) / 64) * (BK * 128) : (uint32_t)cta_n * 128u;
  const int n_stages = min(MAX_STAGES, (int)(RING_BYTES / (A_STAGE + b_stage)));
  const int tiles_m = (p.M + TILE_M - 1) / TILE_M, tiles_n = (p.N + tile_n - 1) / tile_n;
  const int k_blocks_all = (p.K + BK - 1) / BK;
  const int k_per = (k_blocks_all + p.k_splits - 1) / p.k_splits;   // k blocks per work unit (static mode)
  const int num_tiles = p.tri ? tiles_m * (tiles_m + 1) / 2 : tiles_m * tiles_n;
  volatile int* abort_flag = &s_abort;

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int s = 0; s < MAX_STAGES; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int s = 0; s < 2; ++s) { mbar_init(smem_u32(&bar_tfull[s]), 1); mbar_init(smem_u32(&bar_tempty[s]), 8); }
    if (EPI == 5)
      for (int s = 0; s < 8; ++s) mbar_init(smem_u32(&bar_gu[s]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (threadIdx.x == 32) { prefetch_map(&p.tmA); prefetch_map(&p.tmB); }
  if (threadIdx.x < 32) s_ready[threadIdx.x] = 0;
  if (warp == 1 && is_compute) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&s_tmem_base)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();   // the peer's barriers are initialised before any remote arrive or TMA completion
  tcgen05_fence_after();
  grid_wait();          // everything up to here ran beside the kernel before
  if (p.world == 1) grid_release();      // a fused collective has its SMs to itself until it ends
  const uint32_t tmem_base = s_tmem_base;
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sA = sbase, sB = sbase + n_stages * A_STAGE, sEpi = sbase + RING_BYTES;

  if (is_compute) {
    if (warp == 0) {
      // ----------------------------- TMA producer (both CTAs of the pair) ------------
      {
        const bool leader = elect_one();
        const int chunks_per_rank = p.ag_operand ? p.ag_rows_per_rank / CHUNK_ROWS : 1;
        // bounded wait until rows [r0, r0 + nrows) of the gathered operand are in local memory
        auto rows_ready = [&](int r0, int nrows) -> bool {
          const int c0 = r0 / CHUNK_ROWS, c1 = (r0 + nrows - 1) / CHUNK_ROWS;
          for (int c = c0; c <= c1; ++c) {
            if (c / chunks_per_rank == p.rank || c >= p.world * chunks_per_rank) continue;
            if (s_ready[(c >> 5) & 31] & (1u << (c & 31))) continue;
            if (!flag_wait<false>(p.ag_flags + c, p.epoch, abort_flag)) return false;
            fence_proxy_async();
            s_ready[(c >> 5) & 31] |= 1u << (c & 31);
          }
          return true;
        };
        // the lane that issues the loads waits for the rows; every lane gets the answer
        auto rows_ready_warp = [&](int r0, int nrows) -> bool { return __all_sync(0xffffffffu, !leader || rows_ready(r0, nrows)); };
        uint32_t it = 0, s = 0, ph = 0;                  // ring position of `it` (no division in the loop)
        const uint32_t full0 = smem_u32(&bar_full[0]), empty0 = smem_u32(&bar_empty[0]), fullp0 = mapa(full0, 0);
        bool ok = true;
        Work w;
        work_init(p, w, pair);
        for (; ok && work_get(p, w, num_tiles, k_blocks_all, k_per); work_next(p, w)) {
          int tm, tn;
          tile_coords(p, w.tile, tiles_m, tiles_n, tm, tn);
          const int kb0 = w.kb0;
          const int k_blocks = w.nkb;
          const int m0 = tm * TILE_M + (int)cr * CTA_M;
          const int n0 = EPI == 3 ? tn * cta_n + (int)cr * p.swiglu_f : tn * tile_n + (int)cr * cta_n;
          if (p.ag_operand == 1 && !A_MN) ok = rows_ready_warp(m0, CTA_M);
          if (p.ag_operand == 2 && !B_MN) ok = ok && rows_ready_warp(n0, cta_n);
          for (int kb = 0; kb < k_blocks && ok; ++kb, ++it) {
            // k order rotated so that the rows of the local shard come first when k is the gathered dimension
            int kbr = kb0 + kb;
            if ((p.ag_operand == 1 && A_MN) || (p.ag_operand == 2 && B_MN)) {
              kbr = kb + p.rank * (p.ag_rows_per_rank / BK);       // gathered k: never split (host side)
              if (kbr >= k_blocks) kbr -= k_blocks;
              if (!(ok = rows_ready_warp(kbr * BK, BK))) break;
            }
            if (!(ok = mbar_wait_warp(empty0 + 8u * s, ph ^ 1u, abort_flag))) break;
            if (leader) {
              if (cr == 0) mbar_expect_tx(full0 + 8u * s, 2 * (A_STAGE + b_stage));
              const uint32_t fb = fullp0 + 8u * s;
              const uint32_t a_dst = sA + s * A_STAGE, b_dst = sB + s * b_stage;
              const int k0 = kbr * BK;
              if (!A_MN) {
                tma_load_2d_pair(a_dst, &p.tmA, fb, k0, m0);
              } else {
#pragma unroll
                for (int j = 0; j < CTA_M / 64; ++j) tma_load_2d_pair(a_dst + j * (BK * 128), &p.tmA, fb, m0 + 64 * j, k0);
              }
              if (!B_MN) {
                tma_load_2d_pair(b_dst, &p.tmB, fb, k0, n0);
              } else {
                for (int j = 0; j < cta_n; j += 64) tma_load_2d_pair(b_dst + j * 128, &p.tmB, fb, n0 + j, k0);
              }
            }
            if (++s == (uint32_t)n_stages) { s = 0; ph ^= 1u; }
          }
        }
        // drain (even CTA): every armed stage has landed in both CTAs before the pair may retire
        if (leader && cr == 0) {
          Drain drain;
          for (uint32_t back = 0; back < (uint32_t)n_stages && back < it; ++back) {
            const uint32_t j = it - 1 - back;
            drain.wait(smem_u32(&bar_full[j % n_stages]), (j / n_stages) & 1);
          }
        }
      }
    } else if (warp == 1) {
      // ----------------------------- MMA issuer (even CTA only) ----------------------
      if (cr == 0) {
        const bool leader = elect_one();
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((A_MN ? 1u : 0u) << 15) |
                               ((B_MN ? 1u : 0u) << 16) | ((uint32_t)(tile_n >> 3) << 17) | ((uint32_t)(TILE_M >> 4) << 24);
        uint32_t tile_i = 0;
        bool ok = true;
        Work w;
        work_init(p, w, pair);
        // descriptors of stage 0, built once: a stage or a k step only moves the start address (bytes >> 4 in the low
        // word; the whole ring lies below 256 KB, so the additions never carry out of the 14-bit address field).
        const DescBase dA0 = A_MN ? desc_base(sA, BK * 128, 1024) : desc_base(sA, 16, 1024);
        const DescBase dB0 = B_MN ? desc_base(sB, BK * 128, 1024) : desc_base(sB, 16, 1024);
        constexpr uint32_t A_KSTEP = (A_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4, B_KSTEP = (B_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4;
        uint32_t s = 0, ph = 0;                          // ring position (no division in the loop)
        const uint32_t full0 = smem_u32(&bar_full[0]), empty0 = smem_u32(&bar_empty[0]);
        for (; ok && work_get(p, w, num_tiles, k_blocks_all, k_per); work_next(p, w), ++tile_i) {
          const int k_blocks = w.nkb;
          const uint32_t acc = tile_i & 1, acc_ph = (tile_i >> 1) & 1;
          if (!(ok = mbar_wait_warp(smem_u32(&bar_tempty[acc]), acc_ph ^ 1, abort_flag))) break;
          tcgen05_fence_after();
          const uint32_t d_tmem = tmem_base + acc * TILE_N;
          for (int kb = 0; kb < k_blocks; ++kb) {
            if (!(ok = mbar_wait_warp(full0 + 8u * s, ph, abort_flag))) break;
            tcgen05_fence_after();
            const uint32_t a_lo = dA0.lo + s * (A_STAGE >> 4), b_lo = dB0.lo + s * (b_stage >> 4);
            if (leader) {
#pragma unroll
              for (int kk = 0; kk < BK / UMMA_K; ++kk)
                umma_bf16_pair_lohi(d_tmem, a_lo + kk * A_KSTEP, dA0.hi, b_lo + kk * B_KSTEP, dB0.hi, idesc,
                                    (kb > 0 || kk > 0) ? 1u : 0u);
              umma_commit_pair(empty0 + 8u * s);
            }
            if (++s == (uint32_t)n_stages) { s = 0; ph ^= 1u; }
          }
          if (ok && leader) umma_commit_pair(smem_u32(&bar_tfull[acc]));
        }
      }
    } else {
      // ----------------------------- epilogue (warps 2..5 of both CTAs) --------------
      const int quad = warp & 3;
      uint32_t tile_i = 0, n_boxes = 0;
      GuLoads gl = {};
      if (EPI == 5) gl = {smem_u32(&bar_gu[EPI == 5 ? 2 * quad : 0]), sEpi + (uint32_t)quad * 16384u, 0u, 0u};
      bool ok = true;
      Work w;
      work_init(p, w, pair);
      for (; ok && work_get(p, w, num_tiles, k_blocks_all, k_per); work_next(p, w), ++tile_i) {
        int tm, tn;
        tile_coords(p, w.tile, tiles_m, tiles_n, tm, tn);
        const int m0 = tm * TILE_M + (int)cr * CTA_M, n0 = tn * tile_n;
        const uint32_t acc = tile_i & 1, acc_ph = (tile_i >> 1) & 1;
        if (EPI == 5 && m0 + quad * 32 < p.M && n0 < p.swiglu_f) gu_issue(p, gl, lane, n0, m0 + quad * 32);   // while the main loop runs
        ok = mbar_wait(smem_u32(&bar_tfull[acc]), acc_ph, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tcgen05_fence_after();
        const uint32_t tmem_acc = tmem_base + acc * TILE_N;
        if (EPI == 3)      epilogue_swiglu(p, tmem_acc, quad, lane, m0, tn, sEpi + (uint32_t)quad * 8192u, n_boxes);
        else if (EPI == 5) { if (!(ok = epilogue_swiglu_bwd(p, tmem_acc, quad, lane, m0, n0, gl, abort_flag))) break; }
        else if (EPI == 6) epilogue_attn_dout(p, tmem_acc, quad, lane, m0, n0, sEpi + (uint32_t)quad * 8192u, n_boxes);
        else if (EPI == 4 && p.rope_dh == 128 && p.rope_cols % 128 == 0)
          epilogue_rope<128>(p, tmem_acc, quad, lane, m0, n0, sEpi + (uint32_t)quad * 8192u, n_boxes);
        else if (EPI == 4 && p.rope_dh == 64 && p.rope_cols % 64 == 0)
          epilogue_rope<64>(p, tmem_acc, quad, lane, m0, n0, sEpi + (uint32_t)quad * 8192u, n_boxes);
        else if (p.c_tma)  epilogue_tma<EPI>(p, tmem_acc, quad, lane, m0, n0, sEpi + (uint32_t)quad * 8192u, n_boxes, w.t % p.k_splits);
        else               epilogue_direct<EPI>(p, tmem_acc, quad, lane, m0, n0);
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa(smem_u32(&bar_tempty[acc]), 0));
      }
      // a role that gave up leaves no load in flight into the shared memory that it returns
      if (EPI == 5) {
        Drain drain;
        for (; gl.used < gl.issued; ++gl.used) drain.wait(gl.bar + 8u * (gl.used & 1u), (gl.used >> 1) & 1u);
      }
      if (lane == 0) {
        bulk_wait0();                // staging buffers are read out and the stores / reductions are performed
        if (p.rs_on) __threadfence_system();
      }
    }
  } else if (p.ag_operand) {
    // ----------------------------- comm CTA: pull the peers' row shards -----------------
    if (warp == 0 && lane == 0) {
      const int ci = (pair - p.n_compute_pairs) * 2 + (int)cr, n_comm = (n_pairs - p.n_compute_pairs) * 2;
      const int chunks_per_rank = p.ag_rows_per_rank / CHUNK_ROWS;
      const long long chunk_bytes = (long long)CHUNK_ROWS * p.ag_row_bytes;
      const int spc = (int)((chunk_bytes + STAGE_BYTES - 1) / STAGE_BYTES);   // steps per chunk
      const int peer_chunks = (p.world - 1) * chunks_per_rank;
      const int my_chunks = ci < peer_chunks ? (peer_chunks - ci + n_comm - 1) / n_comm : 0;
      const long long total = (long long)my_chunks * spc;
      auto locate = [&](long long g, long long& off, uint32_t& bytes, int& chunk, int& src, bool& last) {
        const int q = ci + (int)(g / spc) * n_comm;          // q-th peer chunk in ring order
        const int piece = (int)(g % spc);
        src = (p.rank + 1 + q / chunks_per_rank) % p.world;
        chunk = src * chunks_per_rank + q % chunks_per_rank;
        off = (long long)chunk * chunk_bytes + (long long)piece * STAGE_BYTES;
        const long long left = chunk_bytes - (long long)piece * STAGE_BYTES;
        bytes = (uint32_t)(left < STAGE_BYTES ? left : STAGE_BYTES);
        last = piece == spc - 1;
      };
      long long issued = 0, stored = 0;
      bool ok = true;
      while (stored < total && ok) {
        // a stage is reused by load g only after the store of step g - STAGES finished reading it
        asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        while (issued < total && issued < stored + STAGES - 1) {
          long long off; uint32_t bytes; int chunk, src; bool last;
          locate(issued, off, bytes, chunk, src, last);
          const int s = (int)(issued % STAGES);
          const uint32_t fb = smem_u32(&bar_full[s]);
          mbar_expect_tx(fb, bytes);
          bulk_g2s(sbase + s * STAGE_BYTES, p.ag_src[src] + off, bytes, fb);
          ++issued;
        }
        long long off; uint32_t bytes; int chunk, src; bool last;
        locate(stored, off, bytes, chunk, src, last);
        const int s = (int)(stored % STAGES);
        if (!(ok = mbar_wait(smem_u32(&bar_full[s]), (uint32_t)((stored / STAGES) & 1), abort_flag))) break;
        bulk_s2g(p.ag_dst + off, sbase + s * STAGE_BYTES, bytes);
        bulk_commit();
        ++stored;
        if (last) {
          bulk_wait0();            // the whole chunk is written
          fence_proxy_async();
          __threadfence();
          st_release_gpu(p.ag_flags + chunk, p.epoch);
        }
      }
      bulk_wait0();
      // loads that were issued but never stored (abort path) must land before the CTA retires
      Drain drain;
      for (long long g = stored; g < issued; ++g) drain.wait(smem_u32(&bar_full[g % STAGES]), (uint32_t)((g / STAGES) & 1));
    }
  }
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();   // no CTA retires while its peer may still signal its barriers or read its smem
  if (warp == 1 && is_compute) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
  if (threadIdx.x == 0 && s_abort && p.status) atomicOr(p.status, TPLR_ST_WAIT_TIMEOUT);
}

// ------------------------------ host side ----------------------------------------------
template <bool A_MN, bool B_MN, int EPI>
int launch2(Gemm2Params& p, int n_comm_pairs, int max_pairs, cudaStream_t st) {
  auto kern = gemm2_kernel<A_MN, B_MN, EPI>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cfg.stream = st;
  // not for the fused collectives: their CTAs wait for other ranks' kernels and start as one
  attr[1] = pdl_attr(p.world == 1);
  cfg.attrs = attr; cfg.numAttrs = 2;
  // all CTAs must be resident at once: compute CTAs wait for comm CTAs of the same launch
  static int max_clusters[2][2][7] = {};
  int& mc = max_clusters[A_MN][B_MN][EPI];
  if (mc == 0) {
    cfg.gridDim = dim3(2 * (tplr_sm_count() / 2));
    int n = 0;
    e = cudaOccupancyMaxActiveClusters(&n, kern, &cfg);
    if (e != cudaSuccess) return (int)e;
    mc = n > 0 ? n : -1;
  }
  if (mc < 1) return -105;
  int pairs = mc < tplr_sm_count() / 2 ? mc : tplr_sm_count() / 2;
  if (max_pairs > 0 && pairs > max_pairs) pairs = max_pairs;
  if (n_comm_pairs >= pairs) return -106;
  const int tiles_m_h = (p.M + TILE_M - 1) / TILE_M;
  const int tiles = p.tri ? tiles_m_h * (tiles_m_h + 1) / 2 : tiles_m_h * ((p.N + p.tile_n - 1) / p.tile_n);
  int compute = pairs - n_comm_pairs;
  if (compute > tiles * p.k_splits) compute = tiles * p.k_splits;
  p.n_compute_pairs = compute;
  cfg.gridDim = dim3(2 * (compute + n_comm_pairs));
  return (int)cudaLaunchKernelEx(&cfg, kern, p);
}

int dispatch2(Gemm2Params& p, int a_mn, int b_mn, int epi, int n_comm_pairs, int max_pairs, cudaStream_t st) {
#define TPLR_GEMM2_CASE(AM, BMJ, E) \
  if (a_mn == AM && b_mn == BMJ && epi == E) return launch2<AM != 0, BMJ != 0, E>(p, n_comm_pairs, max_pairs, st);
  TPLR_GEMM2_CASE(0, 0, 0) TPLR_GEMM2_CASE(0, 0, 1) TPLR_GEMM2_CASE(0, 0, 2)
  TPLR_GEMM2_CASE(0, 1, 0) TPLR_GEMM2_CASE(0, 1, 1) TPLR_GEMM2_CASE(0, 1, 2)
  TPLR_GEMM2_CASE(1, 1, 0) TPLR_GEMM2_CASE(1, 1, 1) TPLR_GEMM2_CASE(1, 1, 2)
  TPLR_GEMM2_CASE(1, 0, 0) TPLR_GEMM2_CASE(1, 0, 1) TPLR_GEMM2_CASE(1, 0, 2)
  TPLR_GEMM2_CASE(0, 0, 3) TPLR_GEMM2_CASE(0, 0, 4) TPLR_GEMM2_CASE(0, 1, 5) TPLR_GEMM2_CASE(0, 1, 6)
#undef TPLR_GEMM2_CASE
  return -104;
}

int forced_splits() {                                     // tuning override
  static const int forced = [] { const char* e = getenv("TPLR_GEMM_KSPLITS"); return e ? atoi(e) : 0; }();
  return forced;
}

// Width of the tiles and parts of K of a product.
//
// A 256 x 256 tile takes 500 cycles for a k block of 64, which is the tensor pipe's own time.  A narrower one moves more bytes
// for each product: 400 cycles at 192, 345 at 128 while one wave of tiles covers the product and 400 to 440 with several (what
// the SMs can take from L2), 440 and 560 where an operand is M- or N-contiguous (twice the loads).  So narrow tiles pay where
// 256-wide ones leave CTA pairs idle or start a wave for a few of them: 2048 x 768 x 3072 (24 tiles on 74 pairs, 48 of 128)
// 22.6 -> 16.5 us, 8192 x 768 x 3072 (96 tiles in two waves, 128 of 192 in two shorter ones) 43.2 -> 34.0, 1024 x 6144 x 4096 47.2
// -> 39.0, 1111 x 8192 x 1536 30.7 -> 26.8, weight gradient 2304 x 768 x 2048 18.6 -> 16.5; at 16384 x 2048 x 2048 (512 tiles)
// 92.9 us with 256, 99.9 with 192, 112 with 128.  192 only with K-major B (whole 64-column blocks for each CTA otherwise).
//
// K is cut where even so most pairs would idle over a long K: every part stores fp32 (an accumulating product's part 0 adds into C)
// and a second kernel adds the planes in order, the same bits on every run, which parts added as they arrive would not give.
// It costs a launch (4000 cycles) and the planes' bytes, 5000 a cycle while they stay in L2 and 2700 beyond.  768 x 768 x 8192
// accumulating (9 tiles) 45.2 us whole, 18.8 in eight parts; 2304 x 768 x 8192 45.2 whole, 35.0 in two; 2048 x 768 x 6144 bf16 35.0
// whole, 24.0 in three; 8192 x 768 x 32000 341 and 294 in three.  A cut has to win 10 %, a narrower tile 3 %.  Where the result is
// stored in fp32, what bounds a short K is the store, so a narrower tile must not take more waves there: 472 x 9168 x 64 8.0 us
// in one wave of 256, 8.4 in two of 128; 712 x 5960 x 248 9.3 and 9.9; with K of 1000 the two are even.
//
// The costs (cycles) were fitted on 70 shapes of 300 to 16384 rows, K 300 to 32000, each with every width and 1 to 8 parts.
double plan_cost(int M, int N, int K, bool a_mn, bool b_mn, int epi, int tile_n, int parts) {
  const long long kb = (K + BK - 1) / BK, per = (kb + parts - 1) / parts;
  const long long tiles = (long long)((M + TILE_M - 1) / TILE_M) * ((N + tile_n - 1) / tile_n);
  const int pairs = tplr_sm_count() / 2;
  const long long waves = (tiles * parts + pairs - 1) / pairs;
  const double block = tile_n == 256 ? 500 : tile_n == 192 ? 400 : (a_mn || b_mn) ? (waves > 1 ? 560 : 440) : (waves > 1 ? 400 : 345);
  double cost = (double)waves * ((double)per * block + 900.0) + (epi == 1 || epi == 2 || parts > 1 ? 20.0 : 10.0) * tile_n;
  if (parts > 1) {
    const double bytes = (double)M * N * (epi == 1 ? 8.0 * parts : 8.0 * parts + 2.0);
    cost += 4000.0 + bytes / (bytes < 6e7 ? 5000.0 : 2700.0);
  }
  return cost;
}
// The widths that a layout takes; col_unit: what a tile's columns must be a multiple of (64-column boxes, whole heads).
int pick_tile(int M, int N, int K, bool a_mn, bool b_mn, int epi, int parts = 1, int col_unit = 64) {
  int best = TILE_N;
  double best_cost = plan_cost(M, N, K, a_mn, b_mn, epi, TILE_N, parts);
  const int pairs = tplr_sm_count() / 2;
  auto waves = [&](int tn) { return ((long long)((M + TILE_M - 1) / TILE_M) * ((N + tn - 1) / tn) + pairs - 1) / pairs; };
  for (const int tn : {192, 128}) {
    if (tn % col_unit || (tn == 192 && b_mn)) continue;
    if (epi == 2 && waves(tn) > waves(TILE_N)) continue;
    const double cost = plan_cost(M, N, K, a_mn, b_mn, epi, tn, parts);
    if (cost < 0.97 * best_cost) { best = tn; best_cost = cost; }
  }
  return best;
}
// Parts of K: epi 1 an accumulating product, 0 one with a bf16 result (K of 4096 or more and 64 tiles at most: others do not ask).
// The callers lay their workspace out by this number, so it does not depend on the operands' layout (the M-contiguous figures).
int pick_parts(int M, int N, int K, int epi) {
  const long long kb = (K + BK - 1) / BK, tiles = (long long)((M + TILE_M - 1) / TILE_M) * ((N + TILE_N - 1) / TILE_N);
  const int pairs = tplr_sm_count() / 2;
  if (N % 8) return 1;
  if (epi == 0 && (K < 4096 || tiles > 64)) return 1;
  if (epi == 1 && forced_splits() > 0) return kb / forced_splits() >= 1 ? forced_splits() : 1;
  if (kb < 32) return 1;
  auto cost = [&](int parts) {
    const double wide = plan_cost(M, N, K, true, true, epi, 256, parts), narrow = plan_cost(M, N, K, true, true, epi, 128, parts);
    return wide < narrow ? wide : narrow;
  };
  int best = 1;
  double best_cost = 0.90 * cost(1);
  for (int parts = 2; parts <= 8 && parts <= kb; ++parts) {
    const long long per = (kb + parts - 1) / parts;
    if ((parts - 1) * per >= kb || tiles * parts > 4 * pairs) continue;      // every unit has work
    const double c = cost(parts);
    if (c < best_cost) { best = parts; best_cost = c; }
  }
  return best;
}

// Parts of K of the triangle product for Newton-Schulz, by the same count of waves.  Two at most: replicas orthogonalise the
// same matrix each for itself, so the result must not depend on the order in which the parts arrive, and two parts added into
// zeros give the same sum in either order.
int pick_syrk_splits(int M, int K) {
  const long long t = (M + TILE_M - 1) / TILE_M, tiles = t * (t + 1) / 2, kb = (K + BK - 1) / BK, per = (kb + 1) / 2;
  const int pairs = tplr_sm_count() / 2;
  if (per >= kb) return 1;
  auto waves = [&](long long units) { return (double)((units + pairs - 1) / pairs); };
  return waves(2 * tiles) * (double)(per + 8) < 0.95 * waves(tiles) * (double)(kb + 8) ? 2 : 1;
}

// The scatter entry's rule: its reductions cross NVLink, so K is only halved, and only where that lifts the wave efficiency
// by more than 10 points (4 and 8 splits lost more than the fuller waves won).
int pick_scatter_splits(int M, int N, int K) {
  if (forced_splits() > 0) return (K + BK - 1) / BK / forced_splits() >= 1 ? forced_splits() : 1;
  const int pairs = tplr_sm_count() / 2;
  const long long tiles = (long long)((M + TILE_M - 1) / TILE_M) * ((N + TILE_N - 1) / TILE_N);
  if ((K + BK - 1) / BK < 128) return 1;
  auto eff = [&](long long units) { return (double)units / (double)(((units + pairs - 1) / pairs) * pairs); };
  return eff(2 * tiles) > eff(tiles) + 0.10 ? 2 : 1;
}

// C += the planes ([n_planes][plane] fp32, rows of N elements), in order; C: rows of ldc elements, all multiples of 4 and 16-byte
// aligned.
__global__ void __launch_bounds__(256) add_planes_kernel(const float* __restrict__ x, float* __restrict__ c, long long M, int n4, long long ldc,
                                                         int n_planes, long long plane) {
  grid_wait();
  grid_release();
  behind_grid_wait(x); behind_grid_wait(c);
  const long long total = M * n4;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < total; i += gridDim.x * 256LL) {
    const long long row = i / n4;
    float4* p = reinterpret_cast<float4*>(c + row * ldc) + (i - row * n4);
    float4 a = *p;
    for (int s = 0; s < n_planes; ++s) {
      const float4 q = reinterpret_cast<const float4*>(x + s * plane)[i];
      a.x += q.x; a.y += q.y; a.z += q.z; a.w += q.w;
    }
    *p = a;
  }
}

// The parts' planes ([parts][plane] fp32, rows of N elements) added in order -> bf16 rows of ldc elements; N, plane and ldc
// multiples of 8, 16-byte aligned.
__global__ void __launch_bounds__(256) round_rows_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ y, long long M, int n8,
                                                         long long ldc, int parts, long long plane) {
  grid_wait();
  grid_release();
  behind_grid_wait(x); behind_grid_wait(y);
  const long long total = M * n8;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < total; i += gridDim.x * 256LL) {
    float4 a = reinterpret_cast<const float4*>(x)[2 * i], b = reinterpret_cast<const float4*>(x)[2 * i + 1];
    for (int s = 1; s < parts; ++s) {
      const float4* q = reinterpret_cast<const float4*>(x + s * plane) + 2 * i;
      const float4 c = q[0], d = q[1];
      a.x += c.x; a.y += c.y; a.z += c.z; a.w += c.w;
      b.x += d.x; b.y += d.y; b.z += d.z; b.w += d.w;
    }
    const __nv_bfloat162 h[4] = {__floats2bfloat162_rn(a.x, a.y), __floats2bfloat162_rn(a.z, a.w), __floats2bfloat162_rn(b.x, b.y),
                                 __floats2bfloat162_rn(b.z, b.w)};
    const long long row = i / n8;
    *reinterpret_cast<uint4*>(y + row * ldc + (i - row * n8) * 8) = *reinterpret_cast<const uint4*>(h);
  }
}

// Fills the operand maps and the plain fields; returns 0 or a negative argument error.
int fill_common(Gemm2Params& p, const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                long long ldb, long long ldc, int a_mn, int b_mn, int epi, unsigned int* status, int tile_n = TILE_N) {
  if ((lda % 8) || (ldb % 8) || ((uintptr_t)A & 15) || ((uintptr_t)B & 15)) return -101;
  if (!(a_mn ? make_map(&p.tmA, A, M, K, lda, 64, BK) : make_map(&p.tmA, A, K, M, lda, BK, CTA_M))) return -102;
  if (!(b_mn ? make_map(&p.tmB, B, N, K, ldb, 64, BK) : make_map(&p.tmB, B, K, N, ldb, BK, tile_n / 2))) return -103;
  p.tile_n = tile_n;
  p.C = C; p.ldc = ldc; p.M = M; p.N = N; p.K = K; p.status = status;
  static const int group_m = [] { const char* e = getenv("TPLR_GEMM_GROUP_M"); const int v = e ? atoi(e) : 0; return v > 0 ? v : 8; }();
  p.world = 1; p.rank = 0; p.epoch = 0; p.group_m = group_m; p.m_rot = 0; p.n_rot = 0; p.m_inter = 1; p.k_splits = 1;
  p.tri = 0;
  p.ag_operand = 0; p.rs_on = 0;
  const bool f32 = epi != 0;
  p.c_tma = !((uintptr_t)C & 15) && (ldc * (f32 ? 4 : 2)) % 16 == 0;
  if (p.c_tma && C && !make_map(&p.tmC, C, N, M, ldc, f32 ? 32 : 64, 32, CU_TENSOR_MAP_SWIZZLE_128B, f32)) return -110;
  return 0;
}

}  // namespace

// Symmetric rank-k product for Newton-Schulz: the 256 x 256 tiles of C = A A^T (A: [M, K] bf16, K-major; C bf16) that
// lie on or above the diagonal.  Tiles below the diagonal are NOT written: tplr_sym_axpby mirrors them.  Half the
// tensor-core work of the full product, as the reference's Triton kernels ns_line_1 / ns_line_2 do with one triangle
// and a mirrored store (src/tplr/muon/newton_schulz_triton.py:62-131, :173-258).
TPLR_API int tplr_gemm2_syrk(const void* A, void* C, int M, int K, long long lda, long long ldc, unsigned int* status,
                             void* stream) {
  TPLR_ENTER();
  if (M <= 0 || K <= 0) return 0;
  Gemm2Params p = {};
  if (int r = fill_common(p, A, A, C, M, M, K, lda, lda, ldc, 0, 0, 0, status)) return r;
  p.tri = 1;
  return dispatch2(p, 0, 0, 0, 0, 0, (cudaStream_t)stream);
}

// K splits that tplr_gemm2_syrk_acc makes for this size (1: tplr_gemm2_syrk is the better call).
TPLR_API int tplr_gemm2_syrk_splits(int M, int K) { return pick_syrk_splits(M, K); }

// tplr_gemm2_syrk adding into an fp32 C (ldc a multiple of 4, zeroed by the caller) with K cut into two work units per
// tile: the triangle of a small matrix has fewer tiles than the chip has CTA pairs.  2048 x 8192 (36 tiles on 74 pairs):
// 49 us in one pass; an iteration's two products (K = 8192 and 2048) 64 us in one pass each, 44 us split.
TPLR_API int tplr_gemm2_syrk_acc(const void* A, float* C, int M, int K, long long lda, long long ldc, unsigned int* status,
                                 void* stream) {
  TPLR_ENTER();
  if (M <= 0 || K <= 0) return 0;
  if ((ldc % 4) || ((uintptr_t)C & 15)) return -101;
  Gemm2Params p = {};
  if (int r = fill_common(p, A, A, C, M, M, K, lda, lda, ldc, 0, 0, 1, status)) return r;
  p.tri = 1;
  p.k_splits = pick_syrk_splits(M, K);
  return dispatch2(p, 0, 0, 1, 0, 0, (cudaStream_t)stream);
}

// Same contract as tplr_gemm_bf16; max_pairs <= 0 uses every SM pair.
TPLR_API int tplr_gemm2_bf16(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                             long long ldb, long long ldc, int a_mn, int b_mn, int epi, unsigned int* status,
                             int max_pairs, void* stream) {
  TPLR_ENTER();
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  Gemm2Params p = {};
  if (int r = fill_common(p, A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, epi, status,
                          pick_tile(M, N, K, a_mn, b_mn, epi))) return r;
  return dispatch2(p, a_mn, b_mn, epi, 0, max_pairs, (cudaStream_t)stream);
}

// Parts that tplr_gemm2_acc_split cuts K into for this size; 1: no workspace, call tplr_gemm2_bf16 with epi 1.
TPLR_API int tplr_gemm2_acc_splits(int M, int N, int K) { return pick_parts(M, N, K, 1); }

// tplr_gemm2_bf16 with epi 1 (C fp32, C += ...) with K cut into parts: the workspace `ws` holds (parts - 1) * (M rounded up to
// 32) * N fp32 elements (contents irrelevant).  C and ws 16-byte aligned, ldc a multiple of 4, N a multiple of 8.
TPLR_API int tplr_gemm2_acc_split(const void* A, const void* B, float* C, float* ws, int M, int N, int K, long long lda, long long ldb,
                                  long long ldc, int a_mn, int b_mn, unsigned int* status, void* stream) {
  TPLR_ENTER();
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((N % 8) || (ldc % 4) || (((uintptr_t)C | (uintptr_t)ws) & 15)) return -101;
  Gemm2Params p = {};
  const int parts = pick_parts(M, N, K, 1);
  if (int r = fill_common(p, A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, 1, status, pick_tile(M, N, K, a_mn, b_mn, 1, parts))) return r;
  p.k_splits = parts;
  p.plane_rows = (M + 31) / 32 * 32;                    // a warp's box of 32 rows stays inside its plane
  const int n_planes = p.k_splits - 1;
  if (n_planes && !make_map(&p.tmCr[0], ws, N, (long long)n_planes * p.plane_rows, N, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B, true)) return -110;
  if (int r = dispatch2(p, a_mn, b_mn, 1, 0, 0, (cudaStream_t)stream)) return r;
  if (n_planes) {
    const long long n = ((long long)M * (N / 4) + 255) / 256;
    const unsigned grid = (unsigned)(n < 8LL * tplr_sm_count() ? n : 8LL * tplr_sm_count());
    return (int)launch_pdl(add_planes_kernel, grid, 256, 0, (cudaStream_t)stream, ws, C, M, N / 4, ldc, n_planes, (long long)p.plane_rows * N);
  }
  return (int)cudaGetLastError();
}

// Parts that tplr_gemm2_bf16_split would cut K into for a bf16 result of this size; 1: no workspace, call tplr_gemm2_bf16.
TPLR_API int tplr_gemm2_out_splits(int M, int N, int K) { return pick_parts(M, N, K, 0); }

// tplr_gemm2_bf16 with a bf16 result (epi 0) through an fp32 workspace `ws` of parts * (M rounded up to 32) * N elements
// (16-byte aligned, contents irrelevant); C 16-byte aligned with ldc a multiple of 8, N a multiple of 8.
TPLR_API int tplr_gemm2_bf16_split(const void* A, const void* B, void* C, float* ws, int M, int N, int K, long long lda,
                                   long long ldb, long long ldc, int a_mn, int b_mn, unsigned int* status, void* stream) {
  TPLR_ENTER();
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((N % 8) || (ldc % 8) || (((uintptr_t)C | (uintptr_t)ws) & 15)) return -101;
  Gemm2Params p = {};
  const int parts = pick_parts(M, N, K, 0);
  if (int r = fill_common(p, A, B, ws, M, N, K, lda, ldb, N, a_mn, b_mn, 2, status, pick_tile(M, N, K, a_mn, b_mn, 0, parts))) return r;
  p.k_splits = parts;
  p.plane_rows = (M + 31) / 32 * 32;                    // a warp's box of 32 rows stays inside its plane
  if (!make_map(&p.tmC, ws, N, (long long)p.k_splits * p.plane_rows, N, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B, true)) return -110;
  if (int r = dispatch2(p, a_mn, b_mn, 2, 0, 0, (cudaStream_t)stream)) return r;
  const long long n = (long long)M * (N / 8);
  const unsigned grid = (unsigned)((n + 255) / 256 < 8LL * tplr_sm_count() ? (n + 255) / 256 : 8LL * tplr_sm_count());
  return (int)launch_pdl(round_rows_kernel, grid, 256, 0, (cudaStream_t)stream, ws, (__nv_bfloat16*)C, M, N / 8, ldc, p.k_splits,
                         (long long)p.plane_rows * N);
}

// GU[M, 2F] = X W^T for the packed weight W = [w1; w3] ([2F, K] bf16, K-major) and H[M, F] = silu(GU[:, :F]) * GU[:, F:]
// in one launch (see Gemm2Params::swiglu_f).  F a multiple of 128; X, W, GU, H 16-byte aligned with leading dimensions
// that are multiples of 8 elements.  GU may be null: then only H is stored (a forward pass that nothing differentiates:
// two thirds of the entry's stores; 16384 x 768 -> 3072: 130 -> 119 us).  -111: shapes or alignment that this entry does not take (the caller runs the
// projection and the activation as two launches instead).
TPLR_API int tplr_gemm2_swiglu(const void* X, const void* W, void* GU, void* H, int M, int F, int K, long long ldx,
                               long long ldw, long long ldgu, long long ldh, unsigned int* status, void* stream) {
  TPLR_ENTER();
  if (M <= 0 || F <= 0 || K <= 0) return 0;
  if (F % CTA_N || ((uintptr_t)GU & 15) || ((uintptr_t)H & 15) || (ldgu % 8) || (ldh % 8)) return -111;
  Gemm2Params p = {};
  if (int r = fill_common(p, X, W, GU, M, 2 * F, K, ldx, ldw, ldgu, 0, 0, 0, status, pick_tile(M, 2 * F, K, false, false, 3, 1, 128))) return r;
  if (!p.c_tma) return -111;
  if (!make_map(&p.tmCr[0], H, F, M, ldh, 64, 32, CU_TENSOR_MAP_SWIZZLE_128B, false)) return -110;
  p.swiglu_f = F;
  return dispatch2(p, 0, 0, 3, 0, 0, (cudaStream_t)stream);
}

// dGU[M, 2F] = backward of the SwiGLU applied to dH = dY W2 (dY [M, K] bf16 K-major, W2 [K, F] bf16 with F contiguous:
// the down projection's weight as stored), with GU [M, 2F] the forward's packed gate | up projection: one launch instead
// of the data-gradient GEMM followed by an element-wise pass (see epilogue_swiglu_bwd).  F a multiple of 64, all tensors
// 16-byte aligned with leading dimensions that are multiples of 8; -111 when this entry does not take the arguments.
TPLR_API int tplr_gemm2_swiglu_bwd(const void* dY, const void* W2, const void* GU, void* dGU, int M, int F, int K,
                                   long long lddy, long long ldw2, long long ldgu, long long lddgu, unsigned int* status,
                                   void* stream) {
  TPLR_ENTER();
  if (M <= 0 || F <= 0 || K <= 0) return 0;
  if (F % 64 || ((uintptr_t)GU & 15) || ((uintptr_t)dGU & 15) || (ldgu % 8) || (lddgu % 8)) return -111;
  Gemm2Params p = {};
  // operands and tile grid of the [M, F] product; the output map then covers the [M, 2F] packed gradient
  if (int r = fill_common(p, dY, W2, dGU, M, F, K, lddy, ldw2, lddgu, 0, 1, 0, status, pick_tile(M, F, K, false, true, 5))) return r;
  if (!p.c_tma) return -111;
  if (!make_map(&p.tmC, dGU, 2LL * F, M, lddgu, 64, 32, CU_TENSOR_MAP_SWIZZLE_128B, false)) return -110;
  if (!make_map(&p.tmGU, GU, 2LL * F, M, ldgu, 64, 32, CU_TENSOR_MAP_SWIZZLE_128B, false)) return -110;
  p.swiglu_f = F;
  return dispatch2(p, 0, 1, 5, 0, 0, (cudaStream_t)stream);
}

// dO[M, N] = dY Wo (dY [M, K] bf16 K-major, Wo [K, N] bf16 with N contiguous: the attention output projection's weight
// as stored; N = heads * head_dim), and delta[b, h, s] = sum over head h's columns of dO * O for row b * S + s, with O
// [M, N] the forward's attention output (see epilogue_attn_dout).  -111 when this entry does not take the arguments.
TPLR_API int tplr_gemm2_attn_dout(const void* dY, const void* Wo, const void* O, void* dO, float* delta, int M, int N, int K,
                                  int S, int head_dim, long long lddy, long long ldwo, long long ldo, long long lddo,
                                  unsigned int* status, void* stream) {
  TPLR_ENTER();
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((head_dim != 128 && head_dim != 64) || N % head_dim || S <= 0 || M % S || ((uintptr_t)O & 15) || ((uintptr_t)dO & 15) || (ldo % 8) || (lddo % 8) || !delta) return -111;
  Gemm2Params p = {};
  if (int r = fill_common(p, dY, Wo, dO, M, N, K, lddy, ldwo, lddo, 0, 1, 0, status, pick_tile(M, N, K, false, true, 6, 1, head_dim))) return r;
  if (!p.c_tma) return -111;
  p.gu = (const __nv_bfloat16*)O; p.ld_gu = ldo;
  p.attn_delta = delta; p.attn_s = S; p.attn_heads = N / head_dim; p.attn_dh = head_dim;
  return dispatch2(p, 0, 1, 6, 0, 0, (cudaStream_t)stream);
}

// QKV[M, N] = X W^T (bf16, W K-major) with the rotary embedding applied to the first rope_cols columns in the epilogue:
// heads of `head_dim` columns, interleaved pairs, angle tables cos / sin [S, head_dim / 2] fp32, position = row % S
// (the reference's apply_rotary_emb on xq and xk, torchtitan models/llama3/model/model.py, after the wq / wk projections).
// rope_cols and head_dim multiples of 32 and 16-byte aligned tables; -111 when this entry does not take the arguments.
TPLR_API int tplr_gemm2_rope(const void* X, const void* W, void* QKV, int M, int N, int K, long long ldx, long long ldw,
                             long long ldc, const float* cosb, const float* sinb, int S, int rope_cols, int head_dim,
                             unsigned int* status, void* stream) {
  TPLR_ENTER();
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (S <= 0 || head_dim % 32 || rope_cols % 32 || rope_cols > N || ((uintptr_t)cosb & 15) || ((uintptr_t)sinb & 15)) return -111;
  Gemm2Params p = {};
  if (int r = fill_common(p, X, W, QKV, M, N, K, ldx, ldw, ldc, 0, 0, 0, status, head_dim == 64 || head_dim == 128 ? pick_tile(M, N, K, false, false, 4, 1, head_dim) : TILE_N)) return r;
  if (!p.c_tma) return -111;
  p.rope_cos = cosb; p.rope_sin = sinb; p.rope_s = S; p.rope_cols = rope_cols; p.rope_dh = head_dim;
  return dispatch2(p, 0, 0, 4, 0, 0, (cudaStream_t)stream);
}

// All-gather fused into the GEMM.  Operand `ag_operand` (1 = A, 2 = B) is the local FULL buffer
// whose rows (its outer dimension: m or n when K-major, k when MN-major) are sharded over `world`
// ranks, `rows_per_rank` (multiple of 128) each; rank r's rows are valid in rank r's buffer when the
// kernel starts (the caller runs a barrier first) and are copied from `peer_bases[r]` into the local
// buffer by `n_comm_pairs` CTA pairs while the other pairs compute.  `flags` holds one zero-initialised
// word per 128 rows of the full buffer; `epoch` must differ from every earlier call's on these flags.
TPLR_API int tplr_gemm2_gather(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                               long long ldb, long long ldc, int a_mn, int b_mn, int epi, int ag_operand,
                               int world, int rank, int rows_per_rank, const void* const* peer_bases,
                               unsigned int* flags, unsigned int epoch, int n_comm_pairs, unsigned int* status,
                               void* stream) {
  TPLR_ENTER();
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (world < 1 || world > MAX_RANKS || rank < 0 || rank >= world || (ag_operand != 1 && ag_operand != 2)) return -107;
  if (rows_per_rank % CHUNK_ROWS || (long long)world * rows_per_rank / CHUNK_ROWS > 1024 || n_comm_pairs < 1) return -107;
  const bool mn = ag_operand == 1 ? a_mn != 0 : b_mn != 0;
  const long long outer = mn ? K : (ag_operand == 1 ? M : N);
  if (outer != (long long)world * rows_per_rank) return -108;
  Gemm2Params p = {};
  if (int r = fill_common(p, A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, epi, status)) return r;
  p.world = world; p.rank = rank; p.epoch = epoch;
  p.ag_operand = ag_operand; p.ag_rows_per_rank = rows_per_rank;
  p.ag_row_bytes = (ag_operand == 1 ? lda : ldb) * 2;
  for (int r = 0; r < world; ++r) p.ag_src[r] = static_cast<const uint8_t*>(peer_bases[r]);
  p.ag_dst = static_cast<uint8_t*>(const_cast<void*>(ag_operand == 1 ? A : B));
  p.ag_flags = flags;
  if (!mn && ag_operand == 1) {           // tiles of the local row shard first, then the peers in ring order
    p.group_m = 1;
    p.m_rot = (int)(((long long)rank * rows_per_rank) / TILE_M);
  }
  if (!mn && ag_operand == 2) {           // gathered weight rows (FSDP shards): all tile rows of the local columns first
    p.group_m = (M + TILE_M - 1) / TILE_M;
    p.n_rot = (int)(((long long)rank * rows_per_rank) / TILE_N);
  }
  return dispatch2(p, a_mn, b_mn, epi, world > 1 ? n_comm_pairs : 0, 0, (cudaStream_t)stream);
}

// GEMM fused with a reduce-scatter over the rows of C.  Every rank computes its partial
// [M,N] = op(A) op(B) over its own K shard; rank o owns rows [o*rows_per_rank, (o+1)*rows_per_rank)
// and `peer_out[o]` is its [rows_per_rank, N] result buffer (leading dimension ld_out, bf16 or fp32
// by `out_fp32`) as mapped in this process.  The partial tiles are reduce-added into those buffers by
// the epilogue, so every buffer must be zero and all ranks past a barrier when the kernel starts,
// and the sums are complete once all ranks' kernels have finished (a barrier after it).
TPLR_API int tplr_gemm2_scatter(const void* A, const void* B, int M, int N, int K, long long lda, long long ldb,
                                int a_mn, int b_mn, int world, int rank, int rows_per_rank,
                                void* const* peer_out, long long ld_out, int out_fp32, unsigned int* status,
                                void* stream) {
  TPLR_ENTER();
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (world < 1 || world > MAX_RANKS || rank < 0 || rank >= world) return -107;
  const int esz = out_fp32 ? 4 : 2;
  if (rows_per_rank % CHUNK_ROWS || M != world * rows_per_rank || (ld_out * esz) % 16) return -108;
  Gemm2Params p = {};
  const int epi = out_fp32 ? 1 : 0;
  if (int r = fill_common(p, A, B, peer_out[rank], rows_per_rank, N, K, lda, ldb, ld_out, a_mn, b_mn, epi, status)) return r;
  if (!p.c_tma) return -108;
  p.M = M;                                 // fill_common built tmC over the owned rows only
  if (!(a_mn ? make_map(&p.tmA, A, M, K, lda, 64, BK) : make_map(&p.tmA, A, K, M, lda, BK, CTA_M))) return -102;
  p.world = world; p.rank = rank;
  p.rs_on = 1;
  for (int r = 0; r <= world; ++r) p.rs_bound[r] = r * rows_per_rank;
  for (int r = 0; r < world; ++r) {
    if ((uintptr_t)peer_out[r] & 15) return -108;
    if (!make_map(&p.tmCr[r], peer_out[r], N, rows_per_rank, ld_out, out_fp32 ? 32 : 64, 32, CU_TENSOR_MAP_SWIZZLE_128B,
                  out_fp32 != 0)) return -109;
  }
  // every band of tile rows touches every owner, so all links carry traffic throughout the GEMM
  const int tiles_m = (M + TILE_M - 1) / TILE_M;
  if (world > 1 && tiles_m % world == 0) p.m_inter = world;
  return dispatch2(p, a_mn, b_mn, epi, 0, 0, (cudaStream_t)stream);
}

// GEMM fused with a reduce-scatter over the rows of C whose owners hold UNEQUAL row ranges: owner o holds rows
// [bounds[o], bounds[o + 1]) (multiples of 32, bounds[0] = 0, bounds[world] = M; an owner may hold none) in
// `peer_out[o]`, a dense fp32 [rows_o, N] array as mapped in this process (its own, for o == rank).  This is the
// weight-gradient GEMM of sharded data parallelism: every rank multiplies its own tokens (the whole K range) and
// the epilogue reduce-adds each tile into the shard of the rank that owns those rows, over NVLink for a peer
// and in the local L2 for itself, so the fp32 gradient exists only as shards and the reduce-scatter ends with
// the backward pass.  Nothing is zeroed here: the shards accumulate over micro-batches; the caller zeroes them
// between inner steps and separates that from the next backward pass with a barrier.
// Replaces FSDP2's per-block fp32 reduce-scatter (src/tplr/model_factory.py:153,183).
TPLR_API int tplr_gemm2_scatter_v(const void* A, const void* B, int M, int N, int K, long long lda, long long ldb,
                                  int a_mn, int b_mn, int world, int rank, const int* bounds,
                                  void* const* peer_out, unsigned int* status, void* stream) {
  TPLR_ENTER();
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (world < 1 || world > MAX_RANKS || rank < 0 || rank >= world) return -107;
  if (bounds[0] != 0 || bounds[world] != M || (N * 4) % 16) return -108;
  for (int r = 0; r < world; ++r)
    if (bounds[r + 1] < bounds[r] || (bounds[r + 1] % 32)) return -108;
  int first = 0;
  while (first < world && bounds[first + 1] == bounds[first]) ++first;      // first owner that holds rows
  Gemm2Params p = {};
  if (int r = fill_common(p, A, B, peer_out[first], bounds[first + 1] - bounds[first], N, K, lda, ldb, N, a_mn, b_mn, 1,
                          status)) return r;
  if (!p.c_tma) return -108;
  p.M = M;
  if (!(a_mn ? make_map(&p.tmA, A, M, K, lda, 64, BK) : make_map(&p.tmA, A, K, M, lda, BK, CTA_M))) return -102;
  p.world = world; p.rank = rank;
  p.rs_on = 1;
  for (int r = 0; r <= world; ++r) p.rs_bound[r] = bounds[r];
  for (int r = 0; r < world; ++r) {
    const int rows = bounds[r + 1] - bounds[r];
    if (rows == 0) continue;
    if ((uintptr_t)peer_out[r] & 15) return -108;
    if (!make_map(&p.tmCr[r], peer_out[r], N, rows, N, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B, true)) return -109;
  }
  // ranks start on different owners and consecutive tile rows go to different owners where the tile rows
  // divide evenly, so that every owner's link receives traffic throughout the GEMM
  const int tiles_m = (M + TILE_M - 1) / TILE_M;
  if (world > 1 && tiles_m % world == 0) p.m_inter = world;
  if (world > 1) p.m_rot = (int)(((long long)rank * tiles_m) / world);
  p.k_splits = pick_scatter_splits(M, N, K);
  return dispatch2(p, a_mn, b_mn, 1, 0, 0, (cudaStream_t)stream);
}
