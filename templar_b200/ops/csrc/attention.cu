// Causal flash attention on tcgen05 (sm_100a): S = Q K^T and O += P V run on the 5th-generation
// tensor cores with the accumulators in tensor memory; the softmax reads its row of S straight
// from TMEM (lane = query row, so row max / row sum need no shuffles), writes P back into the
// same TMEM columns as packed bf16 and the second MMA takes P from TMEM as its A operand.
//
// Operands come from the packed projection output [B*S, (H + 2 KV) * 128] (q heads, k heads,
// v heads; RoPE already applied in place), loaded by TMA with 128-byte swizzle; no copy splits
// q, k and v.  Head dimension 128 or 64 (a template parameter), any sequence length, grouped-query heads.  The maps are
// three-dimensional (column, position, sequence): the rows of a last block that lie past the end of the sequence read as
// zeros and are not stored, and no block reads the next sequence.
//
// CTA = one 128-row query block of one head: warp 0 TMA producer, warp 1 MMA issuer + TMEM
// owner, warps 2-5 softmax / correction / epilogue.  256 TMEM columns and 97 KB of shared
// memory per CTA, so two CTAs share an SM and one's softmax overlaps the other's MMAs.
// The running maximum is only raised when it grows by more than 2^8 (any consistent reference
// value gives the same result), which keeps the O-rescale off the common path.
// Every mbarrier wait is bounded; on expiry TPLR_ST_WAIT_TIMEOUT is set and all roles return.
//
// Replaces F.scaled_dot_product_attention(is_causal=True) of the reference model
// (torchtitan models/llama3/model/model.py:203-206, :244-262).
#include "tcgen05.cuh"
#include <cuda/std/type_traits>
#include <stdlib.h>

namespace {
using namespace tplr_tc;

constexpr int BQ = 128, BKV = 128;
constexpr int PT_BYTES = 128 * 128 * 2;                  // one 128 x 128 bf16 tile (P, dS)
template <int DH> constexpr int tile_bytes() { return 128 * DH * 2; }            // one operand tile: 32 KB / 16 KB
template <int DH> constexpr int fwd_smem() { return 3 * tile_bytes<DH>() + 1024; }   // Q, K, V
constexpr int FWD_THREADS = 192;
constexpr float RESCALE_THRESHOLD = 8.0f;                // log2 units

struct AttnFwdParams {
  CUtensorMap tmQKV;      // [B, S, C] bf16, box 64 x 128 x 1, 128-byte swizzle
  CUtensorMap tmO;        // [B, S, H*DH] bf16, box 64 x 32 x 1, 128-byte swizzle
  float* lse;             // [B, H, S] natural-log sum-exp of the scaled scores
  int B, S, H, KV;
  float scale_log2;       // softmax scale * log2(e)
  unsigned int* status;
};

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(map), "r"(src), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, uint32_t src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(map), "r"(src), "r"(x), "r"(y), "r"(z) : "memory");
}
// 128 rows x DH columns of one head as DH / 64 boxes of 64 columns
template <int DH>
__device__ __forceinline__ void load_tile(uint32_t dst, const CUtensorMap* map, uint32_t bar, int col, int row, int b) {
#pragma unroll
  for (int q = 0; q < DH / 64; ++q) tma_load_3d(dst + q * (128 * 128), map, bar, col + 64 * q, row, b);
}
// [B, S, inner] tensor map (row stride ld elements, sequence stride S * ld), 128-byte swizzle, box box_inner x box_rows x 1
inline bool make_map3(CUtensorMap* map, const void* ptr, long long inner, int S, int B, long long ld, int box_inner, int box_rows,
                      bool fp32 = false) {
  auto enc = get_encode();
  if (!enc) return false;
  const cuuint64_t esz = fp32 ? 4 : 2;
  cuuint64_t dims[3] = {(cuuint64_t)inner, (cuuint64_t)S, (cuuint64_t)B};
  cuuint64_t strides[2] = {(cuuint64_t)ld * esz, (cuuint64_t)ld * esz * (cuuint64_t)S};
  cuuint32_t box[3] = {(cuuint32_t)box_inner, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  auto call = [&] {
    return enc(map, fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims,
               strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = call();
  if (r == CUDA_ERROR_INVALID_CONTEXT) {     // a thread that has made no runtime call yet (see make_map)
    cudaFree(0);
    r = call();
  }
  if (r != CUDA_SUCCESS)
    fprintf(stderr, "[tplr] cuTensorMapEncodeTiled failed (%d): ptr=%p inner=%lld S=%d B=%d ld=%lld box=%dx%d\n", (int)r, ptr,
            inner, S, B, ld, box_inner, box_rows);
  return r == CUDA_SUCCESS;
}

// instruction descriptor: fp32 accumulate, bf16 A and B, M = 128, N = n; a_mn / b_mn select an M- / N-contiguous operand
__device__ __forceinline__ uint32_t idesc_mn(int n, bool a_mn, bool b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

// Softmax over one row of S (128 fp32 columns in tensor memory, lane = query row).  DIAG = the block on the diagonal
// (columns above the row are masked); the other blocks run the variant without the per-element compare and select.
// At heads of 64 the row is read from tensor memory once and stays in registers, which lets the next S be computed ahead
// (B 8, S 2048, 12 heads: 125 us with two reads, 118 us).  At 128, where P lies over S, it is read twice, 32 columns at a time, for
// the maximum and for the exponentials: holding it spills and gains nothing there (16 heads, B 8, S 2048 189 us with two
// reads and 193 with one; B 2 56 and 65).
// packed fp32 pairs (sm_100): one instruction for two lanes of fma / add, and the three-input max
__device__ __forceinline__ unsigned long long pack_f32x2(uint32_t lo, uint32_t hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma_f32x2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long add_f32x2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// One row of S (128 fp32 columns): four loads in flight and one wait.  The empty statements make every register an output
// of something behind the wait, so that no use of it can be scheduled before.
__device__ __forceinline__ void tmem_ld32_nowait(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void behind_wait32(uint32_t* r) {
  asm volatile("" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
        "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
        "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
        "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31]));
}
__device__ __forceinline__ void tmem_ld128(uint32_t taddr, uint32_t (&v)[128]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) tmem_ld32_nowait(taddr + c * 32, v + c * 32);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int c = 0; c < 4; ++c) behind_wait32(v + c * 32);
}

template <bool DIAG>
__device__ __forceinline__ float attn_row_max(uint32_t (&v)[128], int r) {
  float mx = -INFINITY, mx2 = -INFINITY;
#pragma unroll
  for (int e = 0; e < 128; e += 4) {
    if (DIAG) {
#pragma unroll
      for (int k = 0; k < 4; ++k) if (e + k > r) v[e + k] = 0xff800000u;           // -inf: exp2 makes it zero
    }
    mx = max3(mx, __uint_as_float(v[e]), __uint_as_float(v[e + 1]));
    mx2 = max3(mx2, __uint_as_float(v[e + 2]), __uint_as_float(v[e + 3]));
  }
  return fmaxf(mx, mx2);
}
template <bool DIAG>
__device__ __forceinline__ float attn_row_max(uint32_t ts_lane, int r) {
  float mx = -INFINITY;
#pragma unroll 1
  for (int c = 0; c < 4; ++c) {
    uint32_t v[32];
    tmem_ld32(ts_lane + c * 32, v);
    if (DIAG) {
#pragma unroll
      for (int e = 0; e < 32; ++e) mx = fmaxf(mx, (c * 32 + e > r) ? -INFINITY : __uint_as_float(v[e]));
    } else {
#pragma unroll
      for (int e = 0; e < 16; ++e) mx = max3(mx, __uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1]));
    }
  }
  return mx;
}
// P = exp2(S * scale - m) written as packed bf16 to 64 columns; returns the row sum of P.
__device__ __forceinline__ float attn_row_exp(const uint32_t (&v)[128], uint32_t tp_lane, float sl2, float m_used) {
  const unsigned long long sl2x2 = pack_f32x2(__float_as_uint(sl2), __float_as_uint(sl2));
  const unsigned long long negm = pack_f32x2(__float_as_uint(-m_used), __float_as_uint(-m_used));
  unsigned long long sum = 0ull;                         // (0.f, 0.f)
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t pk[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      float a0, a1;
      unpack_f32x2(fma_f32x2(pack_f32x2(v[c * 32 + 2 * e], v[c * 32 + 2 * e + 1]), sl2x2, negm), a0, a1);
      const float p0 = exp2f(a0), p1 = exp2f(a1);
      sum = add_f32x2(sum, pack_f32x2(__float_as_uint(p0), __float_as_uint(p1)));
      __nv_bfloat162 hh = __floats2bfloat162_rn(p0, p1);
      pk[e] = *reinterpret_cast<uint32_t*>(&hh);
    }
    tmem_st16(tp_lane + c * 16, pk);
  }
  float s0, s1;
  unpack_f32x2(sum, s0, s1);
  return s0 + s1;
}

// the same over the first 64 columns of S
template <bool DIAG>
__device__ __forceinline__ float attn_row_exp(uint32_t ts_lane, int r, float sl2, float m_used) {
  const unsigned long long sl2x2 = pack_f32x2(__float_as_uint(sl2), __float_as_uint(sl2));
  const unsigned long long negm = pack_f32x2(__float_as_uint(-m_used), __float_as_uint(-m_used));
  unsigned long long sum = 0ull;                         // (0.f, 0.f)
#pragma unroll 1
  for (int c = 0; c < 4; ++c) {
    uint32_t v[32], pk[16];
    tmem_ld32(ts_lane + c * 32, v);
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      float a0, a1;
      unpack_f32x2(fma_f32x2(pack_f32x2(v[2 * e], v[2 * e + 1]), sl2x2, negm), a0, a1);
      float p0 = exp2f(a0), p1 = exp2f(a1);
      if (DIAG) {
        if (c * 32 + 2 * e > r) p0 = 0.f;
        if (c * 32 + 2 * e + 1 > r) p1 = 0.f;
      }
      sum = add_f32x2(sum, pack_f32x2(__float_as_uint(p0), __float_as_uint(p1)));
      __nv_bfloat162 hh = __floats2bfloat162_rn(p0, p1);
      pk[e] = *reinterpret_cast<uint32_t*>(&hh);
    }
    tmem_st16(ts_lane + c * 16, pk);
  }
  float s0, s1;
  unpack_f32x2(sum, s0, s1);
  return s0 + s1;
}

template <int DH>
__global__ void __launch_bounds__(FWD_THREADS, 2)
attn_fwd_kernel(const __grid_constant__ AttnFwdParams p) {
  constexpr int TILE_BYTES = tile_bytes<DH>();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t bar_q, bar_k_full, bar_k_empty, bar_v_full, bar_v_empty, bar_s_full, bar_s_read, bar_p_full, bar_o_full;
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int nQ = (p.S + BQ - 1) / BQ;
  // heavy (late) query blocks first
  const int hb = p.H * p.B;
  const int qi = nQ - 1 - (int)(blockIdx.x / hb);
  const int h = (int)(blockIdx.x % hb) % p.H, b = (int)(blockIdx.x % hb) / p.H;
  const int g = h / (p.H / p.KV);
  const int nb = qi + 1;                                   // causal: kv blocks 0..qi
  const int row0 = qi * BQ;                                // position of the first query row; rows past S read as zeros
  const int qcol = h * DH, kcol = (p.H + g) * DH, vcol = (p.H + p.KV + g) * DH;
  volatile int* abort_flag = &s_abort;

  if (threadIdx.x == 0) {
    s_abort = 0;
    mbar_init(smem_u32(&bar_q), 1);
    mbar_init(smem_u32(&bar_k_full), 1); mbar_init(smem_u32(&bar_k_empty), 1);
    mbar_init(smem_u32(&bar_v_full), 1); mbar_init(smem_u32(&bar_v_empty), 1);
    mbar_init(smem_u32(&bar_s_full), 1); mbar_init(smem_u32(&bar_s_read), 4); mbar_init(smem_u32(&bar_p_full), 4);
    mbar_init(smem_u32(&bar_o_full), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(&s_tmem_base)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  grid_wait();
  grid_release();
  const uint32_t tmem_base = s_tmem_base;
  // S columns 0..127, O from column 128.  P lies over S at DH = 128; at 64 it has the 64 columns that O leaves, so that the
  // next block's S is computed as soon as the softmax warps hold this one's in registers (AHEAD).
  constexpr bool AHEAD = DH == 64;
  const uint32_t tS = tmem_base, tO = tmem_base + 128, tP = AHEAD ? tmem_base + 192 : tmem_base;
  const uint32_t sQ = smem_u32(smem), sK = sQ + TILE_BYTES, sV = sK + TILE_BYTES;

  if (warp == 0) {
    {
      const bool leader = elect_one();
      if (leader) {
        mbar_expect_tx(smem_u32(&bar_q), TILE_BYTES);
        load_tile<DH>(sQ, &p.tmQKV, smem_u32(&bar_q), qcol, row0, b);
      }
      bool ok = true;
      int n_k = 0, n_v = 0;                                // tiles asked for
      for (int j = 0; j < nb && ok; ++j) {
        const uint32_t ph = j & 1;
        const int krow = j * BKV;
        if (!(ok = mbar_wait_warp(smem_u32(&bar_k_empty), ph ^ 1, abort_flag))) break;
        if (leader) {
          mbar_expect_tx(smem_u32(&bar_k_full), TILE_BYTES);
          load_tile<DH>(sK, &p.tmQKV, smem_u32(&bar_k_full), kcol, krow, b);
        }
        ++n_k;
        if (!(ok = mbar_wait_warp(smem_u32(&bar_v_empty), ph ^ 1, abort_flag))) break;
        if (leader) {
          mbar_expect_tx(smem_u32(&bar_v_full), TILE_BYTES);
          load_tile<DH>(sV, &p.tmQKV, smem_u32(&bar_v_full), vcol, krow, b);
        }
        ++n_v;
      }
      if (leader) {
        Drain drain;                                         // no load may land after the CTA has retired: a role may have given up
        drain.wait(smem_u32(&bar_q), 0);
        if (n_k) drain.wait(smem_u32(&bar_k_full), (uint32_t)((n_k - 1) & 1));
        if (n_v) drain.wait(smem_u32(&bar_v_full), (uint32_t)((n_v - 1) & 1));
      }
    }
  } else if (warp == 1) {
    {
      const bool leader = elect_one();
      const uint32_t id_qk = idesc_mn(128, false, false), id_pv = idesc_mn(DH, false, true);
      const DescBase bQ = desc_base(sQ, 16, 1024), bK = desc_base(sK, 16, 1024), bV = desc_base(sV, 128 * 128, 1024);
      auto issue_s = [&](int j) -> bool {                  // S(j) = Q K(j)^T
        if (!mbar_wait_warp(smem_u32(&bar_k_full), (uint32_t)(j & 1), abort_flag)) return false;
        tcgen05_fence_after();
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < DH / 16; ++kk) {
            const uint32_t off = (uint32_t)(kk >> 2) * (128u * 128u / 16u) + (uint32_t)(kk & 3) * 2u;    // 16-byte units
            umma_bf16_b(tS, bQ, off, bK, off, id_qk, kk > 0 ? 1u : 0u);
          }
          umma_commit(smem_u32(&bar_s_full));
          umma_commit(smem_u32(&bar_k_empty));
        }
        return true;
      };
      bool ok = mbar_wait_warp(smem_u32(&bar_q), 0, abort_flag);
      if (AHEAD && ok) ok = issue_s(0);
      for (int j = 0; j < nb && ok; ++j) {
        const uint32_t ph = j & 1;
        if (!AHEAD) {
          if (!(ok = issue_s(j))) break;
        } else if (j + 1 < nb) {
          if (!(ok = mbar_wait_warp(smem_u32(&bar_s_read), ph, abort_flag))) break;
          if (!(ok = issue_s(j + 1))) break;
        }
        if (!(ok = mbar_wait_warp(smem_u32(&bar_p_full), ph, abort_flag))) break;
        if (!(ok = mbar_wait_warp(smem_u32(&bar_v_full), ph, abort_flag))) break;
        tcgen05_fence_after();
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < BKV / 16; ++kk)
            umma_ts_bf16_b(tO, tP + 8 * kk, bV, (uint32_t)kk * 128u, id_pv, (j > 0 || kk > 0) ? 1u : 0u);
          umma_commit(smem_u32(&bar_v_empty));
          if (j == nb - 1) umma_commit(smem_u32(&bar_o_full));
        }
      }
    }
  } else {
    const int quad = warp & 3;
    const int r = quad * 32 + lane;                        // query row inside the block = TMEM lane
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < nb && ok; ++j) {
      ok = mbar_wait(smem_u32(&bar_s_full), j & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tcgen05_fence_after();
      const bool diag = j == qi;
      uint32_t sv[AHEAD ? 128 : 1];                        // AHEAD: the row, loaded once
      float mx;
      if constexpr (AHEAD) {
        tmem_ld128(tS + lane_off, sv);
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_s_read));
        mx = diag ? attn_row_max<true>(sv, r) : attn_row_max<false>(sv, r);
      } else {
        mx = diag ? attn_row_max<true>(tS + lane_off, r) : attn_row_max<false>(tS + lane_off, r);
      }
      if (AHEAD && j > 0) {                // O and the P columns: the product of block j-1 has finished with them
        ok = mbar_wait(smem_u32(&bar_v_empty), (uint32_t)((j - 1) & 1), abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tcgen05_fence_after();
      }
      const float m_new = fmaxf(m_used, mx * p.scale_log2);
      const bool need = m_new > m_used + RESCALE_THRESHOLD;       // true for the first block (m_used = -inf)
      if (__any_sync(0xffffffffu, need)) {
        const float alpha = need ? exp2f(m_used - m_new) : 1.f;   // 0 for the first block
        if (need) { m_used = m_new; l *= alpha; }
        if (j > 0) {
          // PV of block j-1 has finished with O: waited for above, or (not AHEAD) S of block j was issued behind it
#pragma unroll 1
          for (int c = 0; c < DH / 32; ++c) {
            uint32_t v[32];
            tmem_ld32(tO + c * 32 + lane_off, v);
#pragma unroll
            for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * alpha);
            tmem_st32(tO + c * 32 + lane_off, v);
          }
        }
      }
      if constexpr (AHEAD) l += attn_row_exp(sv, tP + lane_off, p.scale_log2, m_used);
      else l += diag ? attn_row_exp<true>(tS + lane_off, r, p.scale_log2, m_used) : attn_row_exp<false>(tS + lane_off, r, p.scale_log2, m_used);
      tmem_wait_st();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_p_full));
    }
    // epilogue: O / l -> bf16 -> swizzled staging (the Q tile is no longer read) -> TMA store
    if (ok) ok = mbar_wait(smem_u32(&bar_o_full), 0, abort_flag);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      tcgen05_fence_after();
      const float inv_l = 1.f / l;
      const uint32_t stage = sQ + (uint32_t)quad * (32u * DH * 2u);
      const int orow = row0 + quad * 32;
      const uint32_t sw = (uint32_t)(lane & 7);
#pragma unroll 1
      for (int c = 0; c < DH / 32; ++c) {
        uint32_t v[32];
        tmem_ld32(tO + c * 32 + lane_off, v);
        const uint32_t rowaddr = stage + (uint32_t)(c >> 1) * 4096u + (uint32_t)lane * 128u;
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          uint32_t pw[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            __nv_bfloat162 hh = __floats2bfloat162_rn(__uint_as_float(v[8 * q4 + 2 * e]) * inv_l,
                                                      __uint_as_float(v[8 * q4 + 2 * e + 1]) * inv_l);
            pw[e] = *reinterpret_cast<uint32_t*>(&hh);
          }
          const uint32_t jj = (uint32_t)((c & 1) * 4 + q4);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(rowaddr + ((jj ^ sw) << 4)), "r"(pw[0]), "r"(pw[1]),
                       "r"(pw[2]), "r"(pw[3]) : "memory");
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0 && orow < p.S) {
#pragma unroll
        for (int q = 0; q < DH / 64; ++q) tma_store_3d(&p.tmO, stage + 4096u * q, qcol + 64 * q, orow, b);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      }
      if (p.lse && row0 + r < p.S) p.lse[((long long)b * p.H + h) * p.S + row0 + r] = (m_used + log2f(l)) * 0.6931471805599453f;
    }
  }
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem_base) : "memory");
  }
  if (threadIdx.x == 0 && s_abort && p.status) atomicOr(p.status, TPLR_ST_WAIT_TIMEOUT);
}

}  // namespace

namespace {
template <int DH>
int launch_fwd(const void* qkv, void* out, float* lse, int B, int S, int H, int KV, long long ld_qkv, long long ld_o,
               float scale, unsigned int* status, cudaStream_t st) {
  AttnFwdParams p = {};
  if (!make_map3(&p.tmQKV, qkv, (long long)(H + 2 * KV) * DH, S, B, ld_qkv, 64, 128)) return -202;
  if (!make_map3(&p.tmO, out, (long long)H * DH, S, B, ld_o, 64, 32)) return -203;
  p.lse = lse; p.B = B; p.S = S; p.H = H; p.KV = KV;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.status = status;
  cudaError_t e = cudaFuncSetAttribute(attn_fwd_kernel<DH>, cudaFuncAttributeMaxDynamicSharedMemorySize, fwd_smem<DH>());
  if (e != cudaSuccess) return (int)e;
  const unsigned grid = (unsigned)(((S + BQ - 1) / BQ) * H * B);
  return (int)launch_pdl(attn_fwd_kernel<DH>, grid, FWD_THREADS, fwd_smem<DH>(), st, p);
}
}  // namespace

// qkv: packed [B*S, (H + 2*KV) * head_dim] bf16 (row stride ld_qkv elements); out: [B*S, H*head_dim] bf16 (row stride
// ld_o); lse: [B, H, S] fp32 or null.  head_dim 128 or 64, H a multiple of KV.
TPLR_API int tplr_attention_fwd(const void* qkv, void* out, float* lse, int B, int S, int H, int KV, int head_dim,
                                long long ld_qkv, long long ld_o, float scale, unsigned int* status, void* stream) {
  TPLR_ENTER();
  if (B <= 0 || S <= 0) return 0;
  if (H % KV || (ld_qkv % 8) || (ld_o % 8) || ((uintptr_t)qkv & 15) || ((uintptr_t)out & 15)) return -201;
  if (head_dim == 128) return launch_fwd<128>(qkv, out, lse, B, S, H, KV, ld_qkv, ld_o, scale, status, (cudaStream_t)stream);
  if (head_dim == 64) return launch_fwd<64>(qkv, out, lse, B, S, H, KV, ld_qkv, ld_o, scale, status, (cudaStream_t)stream);
  return -201;
}

// ------------------------------------------------------------------------------------------ //
// Backward.  CTA = one 128-row key/value block of one kv head and the query heads of its group, or a part of them; it
// walks those heads and the query blocks at or below the diagonal.  Per step:
//   S = Q K^T, dP = dO V^T            (tensor cores -> TMEM)
//   P = exp2(S*scale - lse), dS = P * (dP - delta) * scale   (softmax warps, one query row per thread;
//                                      P and dS go to shared memory as bf16 in 128-byte-swizzled tiles)
//   dV += P^T dO, dK += dS^T Q        (accumulated in TMEM over the whole walk)
//   dQ_partial = dS K                 (at DH = 128 into the dP columns, then TMA reduce-add into the fp32 dQ buffer)
// The same swizzled tile serves as a K-major operand of one MMA and an MN-major operand of another,
// so Q, dO, P and dS are each stored once.  K and V stay resident in shared memory.
//
// What bounds it is the chain of a step, not the tensor pipe (five products of 512 cycles each at DH = 128): so the step
// is split where P is ready.  S of the next step is issued as soon as every warp has read this one's (Q has two buffers
// for it) and runs, with dV, while the warps form dS; dK and dQ run while they take the next step's exponentials, and dQ is
// drained behind those (at 64 by warps of its own).  A step of 128 x 128 took 6400 to 7900 cycles at DH = 128 and 5200 at 64 with
// dQ drained at its own end, 5250 to 6300 and 3950 behind the exponentials; the shared-memory traffic of the products, P, dS and dQ
// would allow 4600 and 2900.  With the delta and rounding passes, B 8, S 2048: 16 heads of 128 728 us with the products issued
// under `lane == 0`, 718 from a warp-uniform loop (elect_one), 655 with the late drain; 12 heads of 64 349, 320 and 279, with warps of
// their own 263.  Forward, issued from a warp-uniform loop: 182 -> 170 us and 104 -> 89.
// ------------------------------------------------------------------------------------------ //
namespace {

// K, V, two Q, dO; P, dS; at 64 the staging of dQ
template <int DH> constexpr int bwd_smem() { return 5 * tile_bytes<DH>() + 2 * PT_BYTES + (DH == 64 ? 4 * 8192 : 0) + 1024; }
// TMA warp, MMA warp, 8 softmax warps (2 per TMEM lane quadrant); at 64 four more that drain dQ.  At 128 the softmax warps drain
// it: there is no shared memory left for a staging of its own, and warps that stage it in the dS tile hold back the next dS
// (8 x 2048 x 16 heads 655 us, 690 with them; at 64, 8 x 2048 x 12 279 -> 263, 2 x 8192 x 12 814 -> 743).
template <int DH> constexpr int bwd_threads() { return DH == 64 ? 448 : 320; }

struct AttnBwdParams {
  CUtensorMap tmQKV;    // [B, S, C] bf16, box 64 x 128 x 1
  CUtensorMap tmDO;     // [B, S, H*DH] bf16, box 64 x 128 x 1
  CUtensorMap tmDQ;     // [B, S, H*DH] fp32, box 32 x 32 x 1 (reduce-add target)
  CUtensorMap tmPart;   // split: [B, S, split*2*KV*DH] fp32, box 32 x 32 x 1 (dK | dV of every part)
  CUtensorMap tmDQKV;   // [B, S, C] bf16, box 64 x 32 x 1 (dK and dV stores)
  const float* lse;
  const float* delta;
  int B, S, H, KV;
  int split;            // CTAs that share a group's query heads; > 1: each stores its part of dK and dV in fp32
  float scale, scale_log2;
  unsigned int* status;
  // not null: q and k were rotated (rotary embedding, interleaved pairs, tables [S, DH / 2] fp32) by the producer of qkv and
  // the gradient is wanted with respect to the un-rotated projection: dK is rotated back in the epilogue
  const float* rope_cos;
  const float* rope_sin;
};

__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* map, uint32_t src, int x, int y) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(map), "r"(src), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tma_reduce_add_3d(const CUtensorMap* map, uint32_t src, int x, int y, int z) {
  asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(map), "r"(src), "r"(x), "r"(y), "r"(z) : "memory");
}

template <int DH>
__global__ void __launch_bounds__(bwd_threads<DH>(), 1)
attn_bwd_kernel(const __grid_constant__ AttnBwdParams p) {
  constexpr int TILE_BYTES = tile_bytes<DH>();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t bar_kv, bar_q_full[2], bar_q_empty[2], bar_do_full, bar_do_empty, bar_s_full, bar_dp_full,
      bar_p_ready, bar_ds_ready, bar_dq_full, bar_dq_free;
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int nQ = (p.S + BQ - 1) / BQ;
  const int gb = p.KV * p.B * p.split;
  const int j = (int)(blockIdx.x / gb);                    // kv block; small j (long walks) first
  const int sub = (int)(blockIdx.x % gb) % p.split;
  const int g = (int)(blockIdx.x % gb) / p.split % p.KV, b = (int)(blockIdx.x % gb) / p.split / p.KV;
  const int heads = p.H / p.KV / p.split;                  // query heads of this CTA
  const int h0 = (g * p.split + sub) * heads;
  const int n_i = nQ - j;                                  // query blocks j..nQ-1
  const int n_it = heads * n_i;
  const int kvrow0 = j * BKV;                              // position of the first key row; rows past S read as zeros
  const int kcol = (p.H + g) * DH, vcol = (p.H + p.KV + g) * DH;
  volatile int* abort_flag = &s_abort;

  if (threadIdx.x == 0) {
    s_abort = 0;
    mbar_init(smem_u32(&bar_kv), 1);
    for (int s = 0; s < 2; ++s) { mbar_init(smem_u32(&bar_q_full[s]), 1); mbar_init(smem_u32(&bar_q_empty[s]), 1); }
    mbar_init(smem_u32(&bar_do_full), 1); mbar_init(smem_u32(&bar_do_empty), 1);
    mbar_init(smem_u32(&bar_s_full), 1); mbar_init(smem_u32(&bar_dp_full), 1);
    mbar_init(smem_u32(&bar_p_ready), 8); mbar_init(smem_u32(&bar_ds_ready), 8);
    mbar_init(smem_u32(&bar_dq_full), 1); mbar_init(smem_u32(&bar_dq_free), DH == 64 ? 4 : 8);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&s_tmem_base)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  grid_wait();
  grid_release();
  const uint32_t tmem_base = s_tmem_base;
  // dQ of a step lies over its dP at DH = 128; at 64 it has columns of its own
  const uint32_t tS = tmem_base, tdP = tmem_base + 128, tdV = tmem_base + 256, tdK = tmem_base + 256 + DH, tdQ = DH == 64 ? tmem_base + 384 : tdP;
  const uint32_t sK = smem_u32(smem), sV = sK + TILE_BYTES, sQ = sV + TILE_BYTES, sdO = sQ + 2 * TILE_BYTES,
                 sP = sdO + TILE_BYTES, sdS = sP + PT_BYTES;

  if (warp == 0) {
    {
      const bool leader = elect_one();
      if (leader) {
        mbar_expect_tx(smem_u32(&bar_kv), 2 * TILE_BYTES);
        load_tile<DH>(sK, &p.tmQKV, smem_u32(&bar_kv), kcol, kvrow0, b);
        load_tile<DH>(sV, &p.tmQKV, smem_u32(&bar_kv), vcol, kvrow0, b);
      }
      bool ok = true;
      int n_q = 0, n_do = 0;                                 // tiles asked for
      for (int t = 0; t < n_it && ok; ++t) {
        const int h = h0 + t / n_i, i = j + t % n_i;
        const int qrow0 = i * BQ, qcol = h * DH, s = t & 1;
        if (!(ok = mbar_wait_warp(smem_u32(&bar_q_empty[s]), (uint32_t)(((t >> 1) & 1) ^ 1), abort_flag))) break;
        const uint32_t fq = smem_u32(&bar_q_full[s]);
        if (leader) {
          mbar_expect_tx(fq, TILE_BYTES);
          load_tile<DH>(sQ + s * TILE_BYTES, &p.tmQKV, fq, qcol, qrow0, b);
        }
        ++n_q;
        if (!(ok = mbar_wait_warp(smem_u32(&bar_do_empty), (uint32_t)((t & 1) ^ 1), abort_flag))) break;
        const uint32_t fd = smem_u32(&bar_do_full);
        if (leader) {
          mbar_expect_tx(fd, TILE_BYTES);
          load_tile<DH>(sdO, &p.tmDO, fd, qcol, qrow0, b);
        }
        ++n_do;
      }
      if (leader) {
        Drain drain;                                           // no load may land after the CTA has retired: a role may have given up
        drain.wait(smem_u32(&bar_kv), 0);
        for (int t = n_q > 2 ? n_q - 2 : 0; t < n_q; ++t) drain.wait(smem_u32(&bar_q_full[t & 1]), (uint32_t)((t >> 1) & 1));
        if (n_do) drain.wait(smem_u32(&bar_do_full), (uint32_t)((n_do - 1) & 1));
      }
    }
  } else if (warp == 1) {
    {
      const bool leader = elect_one();
      const uint32_t id_kk = idesc_mn(128, false, false), id_mm = idesc_mn(DH, true, true), id_km = idesc_mn(DH, false, true);
      // descriptor bases: "k" = contraction along the 128-byte rows, "m" = contraction along the tile rows
      // (every operand is made of 128-row blocks of 64 columns, 16 KB apart)
      const DescBase kQ = desc_base(sQ, 16, 1024), kK = desc_base(sK, 16, 1024), kdO = desc_base(sdO, 16, 1024),
                     kV = desc_base(sV, 16, 1024), kdS = desc_base(sdS, 16, 1024);
      const DescBase mP = desc_base(sP, 128 * 128, 1024), mdO = desc_base(sdO, 128 * 128, 1024),
                     mdS = desc_base(sdS, 128 * 128, 1024), mQ = desc_base(sQ, 128 * 128, 1024),
                     mK = desc_base(sK, 128 * 128, 1024);
#define TPLR_KOFF(kk) ((uint32_t)((kk) >> 2) * (128u * 128u / 16u) + (uint32_t)((kk) & 3) * 2u)
#define TPLR_MOFF(kk) ((uint32_t)(kk) * 128u)
      auto issue_s = [&](int t) {
        const uint32_t q = (uint32_t)(t & 1) * (TILE_BYTES / 16);
        if (!leader) return;
#pragma unroll
        for (int kk = 0; kk < DH / 16; ++kk)
          umma_bf16_b(tS, kQ, q + TPLR_KOFF(kk), kK, TPLR_KOFF(kk), id_kk, kk > 0 ? 1u : 0u);
        umma_commit(smem_u32(&bar_s_full));
      };
      auto issue_dp = [&] {
        if (!leader) return;
#pragma unroll
        for (int kk = 0; kk < DH / 16; ++kk) umma_bf16_b(tdP, kdO, TPLR_KOFF(kk), kV, TPLR_KOFF(kk), id_kk, kk > 0 ? 1u : 0u);
        umma_commit(smem_u32(&bar_dp_full));
      };
      bool ok = mbar_wait_warp(smem_u32(&bar_kv), 0, abort_flag);
      if (ok) ok = mbar_wait_warp(smem_u32(&bar_q_full[0]), 0, abort_flag);
      if (ok) { tcgen05_fence_after(); issue_s(0); }
      if (ok) ok = mbar_wait_warp(smem_u32(&bar_do_full), 0, abort_flag);
      if (ok) { tcgen05_fence_after(); issue_dp(); }
      for (int t = 0; t < n_it && ok; ++t) {
        const uint32_t ph = t & 1;
        if (!(ok = mbar_wait_warp(smem_u32(&bar_p_ready), ph, abort_flag))) break;      // P stored, S read by every warp
        tcgen05_fence_after();
        if (t + 1 < n_it) {
          if (!(ok = mbar_wait_warp(smem_u32(&bar_q_full[(t + 1) & 1]), (uint32_t)(((t + 1) >> 1) & 1), abort_flag))) break;
          tcgen05_fence_after();
          issue_s(t + 1);
        }
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)    // dV[kv, d] += P^T[kv, q] dO[q, d]
            umma_bf16_b(tdV, mP, TPLR_MOFF(kk), mdO, TPLR_MOFF(kk), id_mm, (t > 0 || kk > 0) ? 1u : 0u);
          umma_commit(smem_u32(&bar_do_empty));
        }
        if (!(ok = mbar_wait_warp(smem_u32(&bar_ds_ready), ph, abort_flag))) break;     // dS stored, dP read by every warp
        if (DH == 64 && t > 0 && !(ok = mbar_wait_warp(smem_u32(&bar_dq_free), ph ^ 1u, abort_flag))) break;      // dQ(t - 1) read
        tcgen05_fence_after();
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)    // dK[kv, d] += dS^T[kv, q] Q[q, d]
            umma_bf16_b(tdK, mdS, TPLR_MOFF(kk), mQ, ph * (TILE_BYTES / 16) + TPLR_MOFF(kk), id_mm, (t > 0 || kk > 0) ? 1u : 0u);
          umma_commit(smem_u32(&bar_q_empty[ph]));
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)    // dQ[q, d] = dS[q, kv] K[kv, d]; its commit covers every product before it
            umma_bf16_b(tdQ, kdS, TPLR_KOFF(kk), mK, TPLR_MOFF(kk), id_km, kk > 0 ? 1u : 0u);
          umma_commit(smem_u32(&bar_dq_full));
        }
        if (t + 1 < n_it) {
          if (!(ok = mbar_wait_warp(smem_u32(&bar_do_full), ph ^ 1u, abort_flag))) break;
          // dP(t + 1) lies over dQ(t) at 128; at 64 over dP(t), which dS(t) has read
          if (DH == 128 && !(ok = mbar_wait_warp(smem_u32(&bar_dq_free), ph, abort_flag))) break;
          tcgen05_fence_after();
          issue_dp();
        }
      }
    }
  } else if (DH == 64 && warp >= 10) {
    // dQ of every step (fp32 in tensor memory) into the global fp32 dQ: two 32-column boxes through shared memory, TMA reduce-add.
    // Warps of their own, so that the softmax warps go on meanwhile.
    const int quad = warp & 3;
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16, sw = (uint32_t)(lane & 7);
    const uint32_t stg = sdS + PT_BYTES + (uint32_t)quad * 8192u;
    const bool leader = elect_one();
    bool ok = true;
    for (int t = 0; t < n_it && ok; ++t) {
      if (!(ok = mbar_wait_warp(smem_u32(&bar_dq_full), t & 1, abort_flag))) break;
      tcgen05_fence_after();
      uint32_t dq[2][32];
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) tmem_ld32(tdQ + cc * 32 + lane_off, dq[cc]);
      tcgen05_fence_before();
      __syncwarp();
      if (leader) {
        mbar_arrive(smem_u32(&bar_dq_free));
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");                  // the boxes of the step before have left
      }
      __syncwarp();
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        const uint32_t rowaddr = stg + (uint32_t)cc * 4096u + (uint32_t)lane * 128u;
#pragma unroll
        for (int q8 = 0; q8 < 8; ++q8)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(rowaddr + (((uint32_t)q8 ^ sw) << 4)), "r"(dq[cc][4 * q8]),
                       "r"(dq[cc][4 * q8 + 1]), "r"(dq[cc][4 * q8 + 2]), "r"(dq[cc][4 * q8 + 3]) : "memory");
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      const int h = h0 + t / n_i, qrow0 = (j + t % n_i) * BQ + quad * 32;
      if (leader && qrow0 < p.S) {
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) tma_reduce_add_3d(&p.tmDQ, stg + cc * 4096, h * DH + cc * 32, qrow0, b);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
      __syncwarp();
    }
    if (leader) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  } else {
    const int quad = warp & 3;                 // TMEM lane quadrant this warp may access
    const int ch = (warp - 2) >> 2;            // column half (64 columns) this warp works on
    const int r = quad * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    const uint32_t sw = (uint32_t)(lane & 7);
    // two private 4 KB staging buffers: the bytes of this warp's own rows and column half in the P and dS tiles.  Free from
    // the step's last commit on (it covers the products that read them); the reduce-adds have read them before the warp
    // writes its next P and dS.
    const uint32_t stg0 = sP + (uint32_t)ch * (PT_BYTES / 2) + (uint32_t)quad * 4096u;
    const uint32_t stg1 = sdS + (uint32_t)ch * (PT_BYTES / 2) + (uint32_t)quad * 4096u;
    const uint32_t prow = sP + (uint32_t)ch * (PT_BYTES / 2) + (uint32_t)r * 128u;
    const uint32_t drow = sdS + (uint32_t)ch * (PT_BYTES / 2) + (uint32_t)r * 128u;
    // the row statistics of step t; a query row past the end of the sequence has no weight: lse = +inf makes its P zero
    auto stats = [&](int t, float& lse2, float& dl) {
      const int h = h0 + t / n_i, row = (j + t % n_i) * BQ + r;
      const long long at = ((long long)b * p.H + h) * p.S + row;
      const bool live = row < p.S;
      lse2 = live ? p.lse[at] : INFINITY;
      dl = live ? p.delta[at] : 0.f;
    };
    // DH = 128: dQ of step tt (fp32 in tensor memory) into the global fp32 dQ with TMA reduce-add: one group of copies for each box
    auto drain = [&](int tt) -> bool {
      const bool o = mbar_wait(smem_u32(&bar_dq_full), tt & 1, abort_flag);
      if (!__all_sync(0xffffffffu, o)) return false;
      tcgen05_fence_after();
      uint32_t dq[DH / 64][32];
#pragma unroll
      for (int cc = 0; cc < DH / 64; ++cc) tmem_ld32(tdQ + (DH / 64 * ch + cc) * 32 + lane_off, dq[cc]);
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_dq_free));
      const int h = h0 + tt / n_i, qrow0 = (j + tt % n_i) * BQ + quad * 32;
#pragma unroll
      for (int cc = 0; cc < DH / 64; ++cc) {
        const uint32_t stg = cc == 0 ? stg0 : stg1;
        const uint32_t rowaddr = stg + (uint32_t)lane * 128u;
#pragma unroll
        for (int q8 = 0; q8 < 8; ++q8)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(rowaddr + (((uint32_t)q8 ^ sw) << 4)), "r"(dq[cc][4 * q8]),
                       "r"(dq[cc][4 * q8 + 1]), "r"(dq[cc][4 * q8 + 2]), "r"(dq[cc][4 * q8 + 3]) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          if (qrow0 < p.S) tma_reduce_add_3d(&p.tmDQ, stg, h * DH + (DH / 64 * ch + cc) * 32, qrow0, b);
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
      return true;
    };
    float lse_n, dl_n;
    stats(0, lse_n, dl_n);
    bool ok = true;
    for (int t = 0; t < n_it && ok; ++t) {
      const int i = j + t % n_i;
      const float lse2 = lse_n * 1.4426950408889634f, dls = dl_n * p.scale;
      if (t + 1 < n_it) stats(t + 1, lse_n, dl_n);           // in flight during this step
      ok = mbar_wait(smem_u32(&bar_s_full), t & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tcgen05_fence_after();
      // P of this warp's 64 columns, kept in fp32 for dS; the diagonal block runs the variant with the causal mask
      float pv[64];
      auto exp_part = [&](auto DIAG) {
        constexpr bool kDiag = decltype(DIAG)::value;
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          uint32_t sv[32];
          tmem_ld32(tS + ch * 64 + cc * 32 + lane_off, sv);
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            float x = exp2f(fmaf(__uint_as_float(sv[e]), p.scale_log2, -lse2));
            if (kDiag && ch * 64 + cc * 32 + e > r) x = 0.f;
            pv[cc * 32 + e] = x;
          }
        }
      };
      if (i == j) exp_part(cuda::std::true_type{}); else exp_part(cuda::std::false_type{});
      if (t > 0) {
        if constexpr (DH == 128) {
          // dQ of the step before: its products ran while this step's exponentials were taken.  Its last commit covers every
          // product that reads the P and dS tiles, so from here on they may be written.
          if (!(ok = drain(t - 1))) break;
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");    // the box in this warp's bytes of the P tile has left
          __syncwarp();
        } else if (!(ok = mbar_wait_warp(smem_u32(&bar_do_empty), (t - 1) & 1, abort_flag))) {      // dV has read the P tile
          break;
        }
      }
#pragma unroll
      for (int q8 = 0; q8 < 8; ++q8) {
        uint32_t pw[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          __nv_bfloat162 hp = __floats2bfloat162_rn(pv[q8 * 8 + 2 * e], pv[q8 * 8 + 2 * e + 1]);
          pw[e] = *reinterpret_cast<uint32_t*>(&hp);
        }
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(prow + (((uint32_t)q8 ^ sw) << 4)), "r"(pw[0]), "r"(pw[1]),
                     "r"(pw[2]), "r"(pw[3]) : "memory");
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_p_ready));
      if (DH == 64 && t > 0 && !(ok = mbar_wait_warp(smem_u32(&bar_dq_full), (t - 1) & 1, abort_flag))) break;    // dS tile: dK, dQ done
      if (!(ok = mbar_wait_warp(smem_u32(&bar_dp_full), t & 1, abort_flag))) break;
      tcgen05_fence_after();
      // dS carries the softmax scale: d = p * (dp - delta) * scale = p * fma(dp, scale, -delta * scale)
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        uint32_t dv[32];
        tmem_ld32(tdP + ch * 64 + cc * 32 + lane_off, dv);
        if (DH == 128 && cc == 0 && t > 0) {                 // the box staged in this warp's bytes of the dS tile has left them
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          __syncwarp();
        }
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          uint32_t dw[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int k = q4 * 8 + 2 * e;
            const float d0 = pv[cc * 32 + k] * fmaf(__uint_as_float(dv[k]), p.scale, -dls);
            const float d1 = pv[cc * 32 + k + 1] * fmaf(__uint_as_float(dv[k + 1]), p.scale, -dls);
            __nv_bfloat162 hd = __floats2bfloat162_rn(d0, d1);
            dw[e] = *reinterpret_cast<uint32_t*>(&hd);
          }
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(drow + ((((uint32_t)(cc * 4 + q4)) ^ sw) << 4)),
                       "r"(dw[0]), "r"(dw[1]), "r"(dw[2]), "r"(dw[3]) : "memory");
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_ds_ready));
    }
    if (ok && n_it > 0) {                                    // every product done
      if constexpr (DH == 128) ok = drain(n_it - 1);
      else ok = mbar_wait_warp(smem_u32(&bar_dq_full), (n_it - 1) & 1, abort_flag);
    }
    // dV and dK of this kv block.  Whole group in this CTA: TMEM -> bf16 -> staging -> TMA store into the packed gradient;
    // a part of it: stored in fp32 in columns of its own; the pass that rotates dQ back and rounds it adds the parts in order.
    if (ok) {
      tcgen05_fence_after();
      const int orow0 = kvrow0 + quad * 32;
      if (p.split > 1) {
#pragma unroll 1
        for (int x = 0; x < DH / 32; ++x) {      // 32-column boxes of dV, then of dK; this warp takes one column half of each
          const int acc = x / (DH / 64), col = (DH / 64 * ch + x % (DH / 64)) * 32;
          const uint32_t buf = (x & 1) ? stg1 : stg0;
          if (lane == 0) {
            if (x < 2) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            else       asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
          }
          __syncwarp();
          uint32_t v[32];
          tmem_ld32((acc ? tdK : tdV) + col + lane_off, v);
          const uint32_t rowaddr = buf + (uint32_t)lane * 128u;
#pragma unroll
          for (int q8 = 0; q8 < 8; ++q8)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(rowaddr + (((uint32_t)q8 ^ sw) << 4)), "r"(v[4 * q8]),
                         "r"(v[4 * q8 + 1]), "r"(v[4 * q8 + 2]), "r"(v[4 * q8 + 3]) : "memory");
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) {
            if (orow0 < p.S) tma_store_3d(&p.tmPart, buf, (sub * 2 * p.KV + (acc ? g : p.KV + g)) * DH + col, orow0, b);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
      } else {
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();
#pragma unroll
        for (int acc = 0; acc < 2; ++acc) {      // 0 = dV, 1 = dK; at 128 columns this warp stores its half of each, at 64 one of them
          if (DH == 64 && acc != ch) continue;
          const int col = DH == 64 ? 0 : ch * 64;
          const uint32_t tacc = acc ? tdK : tdV;
          const uint32_t buf = acc ? stg1 : stg0;
          const uint32_t rowaddr = buf + (uint32_t)lane * 128u;
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            uint32_t v[32];
            tmem_ld32(tacc + col + hf * 32 + lane_off, v);
            if (acc == 1 && p.rope_cos) {          // dK back through the rotation of this key row: the opposite angle
              const long long tb = (long long)min(orow0 + lane, p.S - 1) * (DH / 2) + (col + hf * 32) / 2;
              const float4* cp = reinterpret_cast<const float4*>(p.rope_cos + tb);
              const float4* sp = reinterpret_cast<const float4*>(p.rope_sin + tb);
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const float4 cv = cp[q], sv = sp[q];
                const float cc[4] = {cv.x, cv.y, cv.z, cv.w}, ss[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const float a = __uint_as_float(v[8 * q + 2 * e]), b2 = __uint_as_float(v[8 * q + 2 * e + 1]);
                  v[8 * q + 2 * e] = __float_as_uint(a * cc[e] + b2 * ss[e]);
                  v[8 * q + 2 * e + 1] = __float_as_uint(b2 * cc[e] - a * ss[e]);
                }
              }
            }
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {
              uint32_t pw[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                __nv_bfloat162 hh = __floats2bfloat162_rn(__uint_as_float(v[8 * q4 + 2 * e]), __uint_as_float(v[8 * q4 + 2 * e + 1]));
                pw[e] = *reinterpret_cast<uint32_t*>(&hh);
              }
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(rowaddr + ((((uint32_t)(hf * 4 + q4)) ^ sw) << 4)),
                           "r"(pw[0]), "r"(pw[1]), "r"(pw[2]), "r"(pw[3]) : "memory");
            }
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0 && orow0 < p.S) {
            tma_store_3d(&p.tmDQKV, buf, (acc ? kcol : vcol) + col, orow0, b);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
  if (threadIdx.x == 0 && s_abort && p.status) atomicOr(p.status, TPLR_ST_WAIT_TIMEOUT);
}

// delta[b, h, s] = sum_d dO * O : DH / 4 lanes per (token, head), 4 elements per lane
template <int DH>
__global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout,
                                                         float* __restrict__ delta, long long tokens, int S, int H,
                                                         long long ld_o) {
  constexpr int LANES = DH / 4;
  const long long w = (long long)blockIdx.x * (256 / LANES) + threadIdx.x / LANES;
  const bool live = w < tokens * H;
  const int lane = threadIdx.x % LANES;
  const long long tok = live ? w / H : 0;
  const int h = live ? (int)(w % H) : 0;
  const uint2 a = *reinterpret_cast<const uint2*>(o + tok * ld_o + h * DH + lane * 4);
  const uint2 d = *reinterpret_cast<const uint2*>(dout + tok * (long long)H * DH + h * DH + lane * 4);
  const float2 a0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a.x));
  const float2 a1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&a.y));
  const float2 d0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&d.x));
  const float2 d1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&d.y));
  float s = a0.x * d0.x + a0.y * d0.y + a1.x * d1.x + a1.y * d1.y;
#pragma unroll
  for (int k = LANES / 2; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
  if (lane == 0 && live) delta[((tok / S) * H + h) * S + tok % S] = s;
}

// dq32 [tokens, q_cols] fp32 -> first q_cols columns (heads of HD) of the packed bf16 gradient, eight values a thread; PARTS: the
// next kv_cols columns (dK | dV of a split walk) are the sums, in order, of `split` parts in part [tokens, split, kv_cols].
// cosb / sinb not null: the pairs are rotated back, in the first rot_cols columns, by the angles of (token % S, pair index in the
// head) on the way.  A pass over memory (4 bytes in and 2 out a value): one 32-bit division for eight values, because with
// four values, 64-bit divisions and a head size of run time it was bound by them (5120 x 4096: 31 us, 19 us here).
template <int HD, bool PARTS>
__global__ void __launch_bounds__(256) attn_dq_cast_kernel(const float* __restrict__ dq32, const float* __restrict__ part, int split,
                                                           __nv_bfloat16* __restrict__ dqkv, long long tokens, int q_cols, int kv_cols,
                                                           int rot_cols, long long ld, const float* __restrict__ cosb,
                                                           const float* __restrict__ sinb, int S) {
  grid_wait();
  grid_release();
  behind_grid_wait(dq32); behind_grid_wait(part); behind_grid_wait(dqkv); behind_grid_wait(cosb); behind_grid_wait(sinb);
  const unsigned w8 = (unsigned)(PARTS ? q_cols + kv_cols : q_cols) / 8;
  const long long n8 = tokens * w8;                     // below 2^32: the scratch would be 137 GB there
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < n8; v += (long long)gridDim.x * blockDim.x) {
    const unsigned tok = (unsigned)v / w8, col = ((unsigned)v - tok * w8) * 8u;
    const bool summed = PARTS && (int)col >= q_cols;
    const float* src = dq32 + 8 * v;                    // without parts the rows lie one behind the other
    if (PARTS) src = summed ? part + (long long)tok * split * kv_cols + (col - q_cols) : dq32 + (long long)tok * q_cols + col;
    const float4 f0 = reinterpret_cast<const float4*>(src)[0], f1 = reinterpret_cast<const float4*>(src)[1];
    float f[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
    if (summed) {
      for (int s = 1; s < split; ++s) {
        const float4* more = reinterpret_cast<const float4*>(src + (long long)s * kv_cols);
        const float4 g0 = more[0], g1 = more[1];
        f[0] += g0.x; f[1] += g0.y; f[2] += g0.z; f[3] += g0.w;
        f[4] += g1.x; f[5] += g1.y; f[6] += g1.z; f[7] += g1.w;
      }
    }
    if (cosb && (int)col < rot_cols) {
      const long long tb = (long long)(tok % (unsigned)S) * (HD / 2) + (col % HD) / 2;
      const float2 c0 = *reinterpret_cast<const float2*>(cosb + tb), c1 = *reinterpret_cast<const float2*>(cosb + tb + 2);
      const float2 s0 = *reinterpret_cast<const float2*>(sinb + tb), s1 = *reinterpret_cast<const float2*>(sinb + tb + 2);
      const float c[4] = {c0.x, c0.y, c1.x, c1.y}, s[4] = {s0.x, s0.y, s1.x, s1.y};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float x = f[2 * e], y = f[2 * e + 1];
        f[2 * e] = x * c[e] + y * s[e];
        f[2 * e + 1] = y * c[e] - x * s[e];
      }
    }
    const __nv_bfloat162 h[4] = {__floats2bfloat162_rn(f[0], f[1]), __floats2bfloat162_rn(f[2], f[3]), __floats2bfloat162_rn(f[4], f[5]),
                                 __floats2bfloat162_rn(f[6], f[7])};
    *reinterpret_cast<uint4*>(dqkv + (long long)tok * ld + col) = *reinterpret_cast<const uint4*>(h);
  }
}

}  // namespace

// ------------------------------------------------------------------------------------------ //
// Pipelined backward.  Same work split as above (CTA = one 128-row key/value block of one kv head), but a
// step covers 64 query rows and everything is computed transposed, with the key/value row as the TMEM lane:
//   S^T = K Q^T, dP^T = V dO^T          (128 x 64 accumulators)
//   P^T, dS^T                            written back over S^T / dP^T as packed bf16 and fed to the next MMAs
//                                        straight from tensor memory (no shared-memory round trip for P)
//   dV += P^T dO, dK += dS^T Q           (A operand from TMEM)
//   dQ^T = K^T dS^T                      (dS^T also stored once in shared memory as the N-contiguous B operand)
// S^T is double buffered and Q / dO / dS^T are two-stage, so the softmax warps work on step t+1 while the
// tensor cores run dV, dK, dQ^T of step t; dQ^T of step t-1 is drained (TMA reduce-add into a [B,H,128,S] fp32
// scratch) between the P and the dS half of step t.  A last kernel transposes that scratch into the packed gradient.
// ------------------------------------------------------------------------------------------ //
namespace {

constexpr int DH = 128, TILE_BYTES = tile_bytes<DH>();     // this variant: head dimension 128, sequences that are multiples of 128
constexpr int B2_BQ = 64;
constexpr int B2_QTILE = B2_BQ * DH * 2;                // 16 KB: 64 x 128 bf16 (two blocks of 64 rows x 128 B)
constexpr int B2_DS_TILE = BKV * B2_BQ * 2;             // 16 KB: 128 kv rows x 64 q
constexpr int B2_STAGE = 8 * 4096;                      // dQ^T drain staging, one 32 x 32 fp32 box per warp
constexpr int B2_SMEM = 2 * TILE_BYTES + 4 * B2_QTILE + 2 * B2_DS_TILE + B2_STAGE + 1024 + 1024;
constexpr int B2_THREADS = 320;

struct AttnBwd2Params {
  CUtensorMap tmKV;     // [B*S, C] bf16, box 64 x 128 (K and V tiles)
  CUtensorMap tmQ;      // [B*S, C] bf16, box 64 x 64  (Q tiles)
  CUtensorMap tmDO;     // [B*S, H*128] bf16, box 64 x 64
  CUtensorMap tmDQT;    // [B*H*128, S] fp32, box 32 x 32 (reduce-add target, transposed dQ)
  CUtensorMap tmDQKV;   // [B*S, C] bf16, box 64 x 32 (dK and dV stores)
  const float* lse;
  const float* delta;
  int B, S, H, KV;
  float scale, scale_log2;
  unsigned int* status;
};

__device__ __forceinline__ void bulk_load_1d(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

__global__ void __launch_bounds__(B2_THREADS, 1)
attn_bwd2_kernel(const __grid_constant__ AttnBwd2Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t bar_kv, bar_q_full[2], bar_q_empty[2], bar_s_full[2], bar_dp_full, bar_p_ready,
      bar_ds_ready, bar_dq_full, bar_dq_free;
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int nQ = p.S / B2_BQ;
  const int gb = p.KV * p.B;
  const int j = (int)(blockIdx.x / gb);
  const int g = (int)(blockIdx.x % gb) % p.KV, b = (int)(blockIdx.x % gb) / p.KV;
  const int group = p.H / p.KV;
  const int iq0 = 2 * j, n_i = nQ - iq0, n_it = group * n_i;
  const int kvrow0 = b * p.S + j * BKV;
  const int kcol = (p.H + g) * DH, vcol = (p.H + p.KV + g) * DH;
  volatile int* abort_flag = &s_abort;

  if (threadIdx.x == 0) {
    s_abort = 0;
    mbar_init(smem_u32(&bar_kv), 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&bar_q_full[s]), 1); mbar_init(smem_u32(&bar_q_empty[s]), 9);
      mbar_init(smem_u32(&bar_s_full[s]), 1);
    }
    mbar_init(smem_u32(&bar_dp_full), 1); mbar_init(smem_u32(&bar_p_ready), 8); mbar_init(smem_u32(&bar_ds_ready), 8);
    mbar_init(smem_u32(&bar_dq_full), 1); mbar_init(smem_u32(&bar_dq_free), 8);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&s_tmem_base)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  grid_wait();
  grid_release();
  const uint32_t tmem_base = s_tmem_base;
  const uint32_t tS0 = tmem_base, tdP = tmem_base + 128, tdQ = tmem_base + 192, tdV = tmem_base + 256, tdK = tmem_base + 384;
  const uint32_t sK = smem_u32(smem), sV = sK + TILE_BYTES, sQ0 = sV + TILE_BYTES, sdO0 = sQ0 + 2 * B2_QTILE,
                 sdS0 = sdO0 + 2 * B2_QTILE, sStage = sdS0 + 2 * B2_DS_TILE, sStat = sStage + B2_STAGE;
  const float* stat = reinterpret_cast<const float*>(smem + (sStat - sK));     // [2][lse 64 | delta 64]

  if (warp == 0) {
    {
      const bool leader = elect_one();
      if (leader) {
        mbar_expect_tx(smem_u32(&bar_kv), 2 * TILE_BYTES);
        tma_load_2d(sK, &p.tmKV, smem_u32(&bar_kv), kcol, kvrow0);
        tma_load_2d(sK + TILE_BYTES / 2, &p.tmKV, smem_u32(&bar_kv), kcol + 64, kvrow0);
        tma_load_2d(sV, &p.tmKV, smem_u32(&bar_kv), vcol, kvrow0);
        tma_load_2d(sV + TILE_BYTES / 2, &p.tmKV, smem_u32(&bar_kv), vcol + 64, kvrow0);
      }
      bool ok = true;
      int n_q = 0;                                           // steps asked for
      for (int t = 0; t < n_it && ok; ++t) {
        const int s = t & 1, k = t >> 1;
        const int h = g * group + t / n_i, iq = iq0 + t % n_i;
        const int qrow0 = b * p.S + iq * B2_BQ, qcol = h * DH;
        if (!(ok = mbar_wait_warp(smem_u32(&bar_q_empty[s]), (uint32_t)((k & 1) ^ 1), abort_flag))) break;
        const uint32_t fb = smem_u32(&bar_q_full[s]);
        if (leader) {
          mbar_expect_tx(fb, 2 * B2_QTILE + 512);
          const uint32_t q_dst = sQ0 + s * B2_QTILE, do_dst = sdO0 + s * B2_QTILE;
          tma_load_2d(q_dst, &p.tmQ, fb, qcol, qrow0);
          tma_load_2d(q_dst + 8192, &p.tmQ, fb, qcol + 64, qrow0);
          tma_load_2d(do_dst, &p.tmDO, fb, qcol, qrow0);
          tma_load_2d(do_dst + 8192, &p.tmDO, fb, qcol + 64, qrow0);
          const long long so = ((long long)b * p.H + h) * p.S + (long long)iq * B2_BQ;
          bulk_load_1d(sStat + s * 512, p.lse + so, 256, fb);
          bulk_load_1d(sStat + s * 512 + 256, p.delta + so, 256, fb);
        }
        ++n_q;
      }
      if (leader) {
        Drain drain;                                         // as in the kernel above
        drain.wait(smem_u32(&bar_kv), 0);
        for (int t = n_q > 2 ? n_q - 2 : 0; t < n_q; ++t) drain.wait(smem_u32(&bar_q_full[t & 1]), (uint32_t)((t >> 1) & 1));
      }
    }
  } else if (warp == 1) {
    {
      const bool leader = elect_one();
      const uint32_t id_st = idesc_mn(64, false, false);     // S^T, dP^T : K-major A and B, N = 64
      const uint32_t id_dv = idesc_mn(128, false, true);     // dV, dK   : A from TMEM, B N-contiguous, N = 128
      const uint32_t id_dq = idesc_mn(64, true, true);       // dQ^T     : A M-contiguous (K^T), B N-contiguous
      // descriptor bases, built once ("k": contraction along the 128-byte rows, "m": along the tile rows)
      const DescBase kK = desc_base(sK, 16, 1024), kV = desc_base(sV, 16, 1024), mK = desc_base(sK, TILE_BYTES / 2, 1024);
      DescBase kQ[2], kdO[2], mQ[2], mdO[2], mdS[2];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        kQ[s] = desc_base(sQ0 + s * B2_QTILE, 16, 1024);    kdO[s] = desc_base(sdO0 + s * B2_QTILE, 16, 1024);
        mQ[s] = desc_base(sQ0 + s * B2_QTILE, 8192, 1024);  mdO[s] = desc_base(sdO0 + s * B2_QTILE, 8192, 1024);
        mdS[s] = desc_base(sdS0 + s * B2_DS_TILE, 8192, 1024);
      }
#define TPLR_K128(kk) ((uint32_t)((kk) >> 2) * (TILE_BYTES / 32) + (uint32_t)((kk) & 3) * 2u)   /* 128-row tile, 16-byte units */
#define TPLR_K64(kk) ((uint32_t)((kk) >> 2) * 512u + (uint32_t)((kk) & 3) * 2u)                /* 64-row tile */
#define TPLR_M(kk) ((uint32_t)(kk) * 128u)
      auto issue_st = [&](int t) {                            // S^T(t) = K Q^T into S buffer t & 1
        if (!leader) return;
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          umma_bf16_b(tS0 + (t & 1) * 64, kK, TPLR_K128(kk), kQ[t & 1], TPLR_K64(kk), id_st, kk > 0 ? 1u : 0u);
        umma_commit(smem_u32(&bar_s_full[t & 1]));
      };
      auto issue_dp = [&](int t) {                            // dP^T(t) = V dO^T
        if (!leader) return;
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) umma_bf16_b(tdP, kV, TPLR_K128(kk), kdO[t & 1], TPLR_K64(kk), id_st, kk > 0 ? 1u : 0u);
        umma_commit(smem_u32(&bar_dp_full));
      };
      bool ok = mbar_wait_warp(smem_u32(&bar_kv), 0, abort_flag);
      if (ok) ok = mbar_wait_warp(smem_u32(&bar_q_full[0]), 0, abort_flag);
      if (ok) {
        tcgen05_fence_after();
        issue_st(0);
        issue_dp(0);
      }
      if (ok && n_it > 1) {
        ok = mbar_wait_warp(smem_u32(&bar_q_full[1]), 0, abort_flag);
        if (ok) { tcgen05_fence_after(); issue_st(1); }
      }
      for (int t = 0; t < n_it && ok; ++t) {
        const int s = t & 1;
        const uint32_t ph = t & 1;
        if (!(ok = mbar_wait_warp(smem_u32(&bar_p_ready), ph, abort_flag))) break;
        tcgen05_fence_after();
        if (leader)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)          // dV += P^T dO ; P^T packed at columns 0-15 and 32-47 of the S buffer
          umma_ts_bf16_b(tdV, tS0 + s * 64 + (kk >> 1) * 32 + (kk & 1) * 8, mdO[s], TPLR_M(kk), id_dv, (t > 0 || kk > 0) ? 1u : 0u);
        if (!(ok = mbar_wait_warp(smem_u32(&bar_ds_ready), ph, abort_flag))) break;
        tcgen05_fence_after();
        if (leader)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)          // dK += dS^T Q
          umma_ts_bf16_b(tdK, tdP + (kk >> 1) * 32 + (kk & 1) * 8, mQ[s], TPLR_M(kk), id_dv, (t > 0 || kk > 0) ? 1u : 0u);
        if (t > 0 && !(ok = mbar_wait_warp(smem_u32(&bar_dq_free), (uint32_t)((t - 1) & 1), abort_flag))) break;
        tcgen05_fence_after();
        if (leader)
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)          // dQ^T = K^T dS^T
          umma_bf16_b(tdQ, mK, TPLR_M(kk), mdS[s], TPLR_M(kk), id_dq, kk > 0 ? 1u : 0u);
        if (leader) {
          umma_commit(smem_u32(&bar_dq_full));
          umma_commit(smem_u32(&bar_q_empty[s]));
        }
        if (t + 1 < n_it) issue_dp(t + 1);
        if (t + 2 < n_it) {
          if (!(ok = mbar_wait_warp(smem_u32(&bar_q_full[s]), (uint32_t)(((t + 2) >> 1) & 1), abort_flag))) break;
          tcgen05_fence_after();
          issue_st(t + 2);
        }
      }
    }
  } else {
    const int quad = warp & 3, ch = (warp - 2) >> 2;
    const int r = quad * 32 + lane;                       // kv row of the block = TMEM lane
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    const uint32_t sw = (uint32_t)(lane & 7);
    const uint32_t stg = sStage + (uint32_t)(warp - 2) * 4096u;
    bool ok = true;
    // drain of dQ^T(tt): this warp's 32 d-rows x 32 q-columns box, reduce-added into the transposed scratch
    auto drain = [&](int tt) -> bool {
      bool o = mbar_wait(smem_u32(&bar_dq_full), (uint32_t)(tt & 1), abort_flag);
      o = __all_sync(0xffffffffu, o);
      if (!o) return false;
      tcgen05_fence_after();
      uint32_t v[32];
      tmem_ld32(tdQ + ch * 32 + lane_off, v);
      tcgen05_fence_before();
      if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_dq_free));
      const uint32_t rowaddr = stg + (uint32_t)lane * 128u;
#pragma unroll
      for (int q8 = 0; q8 < 8; ++q8)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(rowaddr + (((uint32_t)q8 ^ sw) << 4)), "r"(v[4 * q8]),
                     "r"(v[4 * q8 + 1]), "r"(v[4 * q8 + 2]), "r"(v[4 * q8 + 3]) : "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        const int hh = g * group + tt / n_i, iq = iq0 + tt % n_i;
        tma_reduce_add_2d(&p.tmDQT, stg, iq * B2_BQ + ch * 32, (b * p.H + hh) * DH + quad * 32);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
      return true;
    };
    for (int t = 0; t < n_it && ok; ++t) {
      const int s = t & 1;
      const int iq = iq0 + t % n_i;
      const int moff = (iq - iq0) * B2_BQ;                // query column offset of this block relative to the kv block
      const bool diag = iq - iq0 < 2;
      ok = mbar_wait(smem_u32(&bar_q_full[s]), (uint32_t)((t >> 1) & 1), abort_flag);     // lse / delta of this step
      if (ok) ok = mbar_wait(smem_u32(&bar_s_full[s]), (uint32_t)((t >> 1) & 1), abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tcgen05_fence_after();
      const float* st = stat + s * 128 + ch * 32;
      float pv[32];
      {
        uint32_t sv[32], pk[16];
        tmem_ld32(tS0 + s * 64 + ch * 32 + lane_off, sv);
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          float x = exp2f(fmaf(__uint_as_float(sv[e]), p.scale_log2, -st[e] * 1.4426950408889634f));
          if (diag && r > ch * 32 + e + moff) x = 0.f;
          pv[e] = x;
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          __nv_bfloat162 hh = __floats2bfloat162_rn(pv[2 * e], pv[2 * e + 1]);
          pk[e] = *reinterpret_cast<uint32_t*>(&hh);
        }
        tmem_st16(tS0 + s * 64 + ch * 32 + lane_off, pk);   // P^T over this warp's own S^T columns
      }
      tmem_wait_st();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_p_ready));
      if (t > 0 && !(ok = drain(t - 1))) break;
      ok = mbar_wait(smem_u32(&bar_dp_full), (uint32_t)(t & 1), abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tcgen05_fence_after();
      {
        uint32_t dv[32], pk[16];
        tmem_ld32(tdP + ch * 32 + lane_off, dv);
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const float d0 = pv[2 * e] * (__uint_as_float(dv[2 * e]) - st[64 + 2 * e]) * p.scale;
          const float d1 = pv[2 * e + 1] * (__uint_as_float(dv[2 * e + 1]) - st[64 + 2 * e + 1]) * p.scale;
          __nv_bfloat162 hh = __floats2bfloat162_rn(d0, d1);
          pk[e] = *reinterpret_cast<uint32_t*>(&hh);
        }
        tmem_st16(tdP + ch * 32 + lane_off, pk);             // dS^T for the dK MMA
        const uint32_t rowaddr = sdS0 + s * B2_DS_TILE + (uint32_t)r * 128u;      // and as B operand of dQ^T
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(rowaddr + ((((uint32_t)(ch * 4 + q4)) ^ sw) << 4)),
                       "r"(pk[4 * q4]), "r"(pk[4 * q4 + 1]), "r"(pk[4 * q4 + 2]), "r"(pk[4 * q4 + 3]) : "memory");
      }
      tmem_wait_st();
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) { mbar_arrive(smem_u32(&bar_ds_ready)); mbar_arrive(smem_u32(&bar_q_empty[s])); }
    }
    if (ok && n_it > 0) ok = drain(n_it - 1);
    // dV and dK of this kv block: every MMA has completed (the last dQ^T commit covers them)
    if (ok) {
      const int orow0 = kvrow0 + quad * 32;
#pragma unroll
      for (int acc = 0; acc < 2; ++acc) {
        const uint32_t tacc = acc ? tdK : tdV;
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();
        const uint32_t rowaddr = stg + (uint32_t)lane * 128u;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t v[32];
          tmem_ld32(tacc + ch * 64 + hf * 32 + lane_off, v);
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            uint32_t pw[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              __nv_bfloat162 hh = __floats2bfloat162_rn(__uint_as_float(v[8 * q4 + 2 * e]), __uint_as_float(v[8 * q4 + 2 * e + 1]));
              pw[e] = *reinterpret_cast<uint32_t*>(&hh);
            }
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(rowaddr + ((((uint32_t)(hf * 4 + q4)) ^ sw) << 4)),
                         "r"(pw[0]), "r"(pw[1]), "r"(pw[2]), "r"(pw[3]) : "memory");
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          tma_store_2d(&p.tmDQKV, stg, (acc ? kcol : vcol) + ch * 64, orow0);
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
  if (threadIdx.x == 0 && s_abort && p.status) atomicOr(p.status, TPLR_ST_WAIT_TIMEOUT);
}

// dqT [B*H*128, S] fp32 (row = (b, h, d)) -> dqkv[(b*S + s), h*128 + d] bf16, 32 x 32 tiles through shared memory
__global__ void __launch_bounds__(256) attn_dq_transpose_kernel(const float* __restrict__ dqT, __nv_bfloat16* __restrict__ dqkv,
                                                                int S, int H, long long ld) {
  __shared__ float tile[32][33];
  const int s0 = blockIdx.x * 32, row0 = blockIdx.y * 32;      // row0 indexes (b, h, d)
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;      // 32 x 8
#pragma unroll
  for (int i = 0; i < 4; ++i) tile[ty + 8 * i][tx] = dqT[(long long)(row0 + ty + 8 * i) * S + s0 + tx];
  __syncthreads();
  const int bh = row0 / DH, d0 = row0 % DH;
  const int bb = bh / H, hh = bh % H;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int sl = ty + 8 * i;                                  // s within the tile
    dqkv[((long long)bb * S + s0 + sl) * ld + hh * DH + d0 + tx] = __float2bfloat16(tile[tx][sl]);
  }
}

}  // namespace

// Backward variant: 1 = one 128-row query block per step, P / dS through shared memory (default: with the delta and rounding
// passes 0.57 ms against 0.65 to 0.70 at B 8, S 2048, 16 on 8 heads, 0.66 against 0.81 at 16 on 16, 0.09 against 0.15 at B 1, S 1024,
// 32 on 8); 2 = pipelined transposed form, 64 query rows per step, slower at every size tried.
static int g_bwd_variant = [] { const char* e = getenv("TPLR_ATTN_BWD"); return (e && atoi(e) == 2) ? 2 : 1; }();
TPLR_API int tplr_attention_set_bwd_variant(int v) {
  if (v != 1 && v != 2) return -1;
  g_bwd_variant = v;
  return 0;
}

// Gradient of tplr_attention_fwd.  qkv / dqkv: packed [B*S, C] bf16 with row stride ld_qkv; out: the forward's
// output (row stride ld_o); dout: contiguous [B*S, H*head_dim]; lse from the forward; delta: [B,H,S] fp32 scratch;
// dq32: B*S*tplr_attention_bwd_scratch_cols fp32 elements of scratch, of which the caller has zeroed the first
// B*S*H*head_dim.  dqkv receives dq | dk | dv.
extern "C" int tplr_rope(void* buf, const float* cosb, const float* sinb, long long tokens, int S, int n_heads, int Dh,
                         long long row_stride, int inverse, void* stream);

static int bwd_split(int B, int S, int H, int KV, int head_dim);

namespace {
template <int HD>
int launch_bwd(const void* qkv, const void* out, const void* dout, const float* lse, float* delta, float* dq32, void* dqkv, int B,
               int S, int H, int KV, long long ld_qkv, long long ld_o, float scale, const float* cosb, const float* sinb,
               unsigned int* status, cudaStream_t st, bool delta_ready) {
  const long long tokens = (long long)B * S;
  const int C = (H + 2 * KV) * HD;
  if (!delta_ready) {
    constexpr int per_cta = 256 / (HD / 4);
    attn_delta_kernel<HD><<<(unsigned)((tokens * H + per_cta - 1) / per_cta), 256, 0, st>>>(
        (const __nv_bfloat16*)out, (const __nv_bfloat16*)dout, delta, tokens, S, H, ld_o);
  }
  if (HD == 128 && S % 128 == 0 && g_bwd_variant == 2) {
    // pipelined kernel: dq32 is used as the transposed scratch [B*H*128, S]
    AttnBwd2Params p = {};
    if (!make_map(&p.tmKV, qkv, C, tokens, ld_qkv, 64, 128)) return -202;
    if (!make_map(&p.tmQ, qkv, C, tokens, ld_qkv, 64, 64)) return -202;
    if (!make_map(&p.tmDO, dout, (long long)H * DH, tokens, (long long)H * DH, 64, 64)) return -203;
    if (!make_map(&p.tmDQT, dq32, S, (long long)B * H * DH, S, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B, true)) return -204;
    if (!make_map(&p.tmDQKV, dqkv, C, tokens, ld_qkv, 64, 32)) return -205;
    p.lse = lse; p.delta = delta; p.B = B; p.S = S; p.H = H; p.KV = KV;
    p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.status = status;
    cudaError_t e = cudaFuncSetAttribute(attn_bwd2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, B2_SMEM);
    if (e != cudaSuccess) return (int)e;
    attn_bwd2_kernel<<<(unsigned)((S / BKV) * KV * B), B2_THREADS, B2_SMEM, st>>>(p);
    attn_dq_transpose_kernel<<<dim3((unsigned)(S / 32), (unsigned)(B * H * DH / 32)), 256, 0, st>>>(
        dq32, (__nv_bfloat16*)dqkv, S, H, ld_qkv);
    if (cosb) return tplr_rope(dqkv, cosb, sinb, tokens, S, H + KV, DH, ld_qkv, 1, st);   // this variant rotates back in a pass of its own
    return (int)cudaGetLastError();
  }
  AttnBwdParams p = {};
  if (!make_map3(&p.tmQKV, qkv, C, S, B, ld_qkv, 64, 128)) return -202;
  if (!make_map3(&p.tmDO, dout, (long long)H * HD, S, B, (long long)H * HD, 64, 128)) return -203;
  p.split = bwd_split(B, S, H, KV, HD);
  float* part = dq32 + tokens * H * HD;                        // the parts of dK and dV lie behind dQ
  const int kv_cols = p.split > 1 ? 2 * KV * HD : 0;
  if (!make_map3(&p.tmDQ, dq32, (long long)H * HD, S, B, (long long)H * HD, 32, 32, true)) return -204;
  if (kv_cols && !make_map3(&p.tmPart, part, (long long)p.split * kv_cols, S, B, (long long)p.split * kv_cols, 32, 32, true)) return -204;
  if (!make_map3(&p.tmDQKV, dqkv, C, S, B, ld_qkv, 64, 32)) return -205;
  p.lse = lse; p.delta = delta; p.B = B; p.S = S; p.H = H; p.KV = KV;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.status = status;
  p.rope_cos = cosb; p.rope_sin = sinb;
  cudaError_t e = cudaFuncSetAttribute(attn_bwd_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, bwd_smem<HD>());
  if (e != cudaSuccess) return (int)e;
  e = launch_pdl(attn_bwd_kernel<HD>, (unsigned)(((S + BKV - 1) / BKV) * KV * B * p.split), bwd_threads<HD>(), bwd_smem<HD>(), st, p);
  if (e != cudaSuccess) return (int)e;
  auto cast = kv_cols ? attn_dq_cast_kernel<HD, true> : attn_dq_cast_kernel<HD, false>;
  return (int)launch_pdl(cast, tplr_sm_count() * 8, 256, 0, st, dq32, part, p.split, (__nv_bfloat16*)dqkv, tokens, H * HD, kv_cols, (H + KV) * HD, ld_qkv, cosb, sinb, S);
}
}  // namespace

// CTAs that share a group's query heads.  One CTA per (key block, kv head, sequence), one CTA per SM: with few of them the
// longest walk (key block 0 over all n query blocks) takes longer than an even share of the work, (n + 1) / 2 blocks a CTA on
// average, does.  A cut shortens the walk, but each part stores its dK and dV in fp32, a pass over 2 KV heads more, so the
// group is only cut until the walk is within a tenth of the even share.  32 query heads on 8 of 128: B 1, S 1024 155 us whole
// (64 CTAs), 46 us in four parts (256 CTAs; the pass that adds them 2 us more); B 6, S 640 (240 CTAs) 103 us whole, 113 us in
// two parts; B 4, S 1024 (256 CTAs) 151 us whole, 163 us in two.
static int bwd_split(int B, int S, int H, int KV, int head_dim) {
  if (KV <= 0 || H % KV || (head_dim == 128 && S % 128 == 0 && g_bwd_variant == 2)) return 1;
  const int group = H / KV;
  const long long n = (S + BKV - 1) / BKV, ctas = n * KV * B;
  int split = 1;
  for (int s = 1; s <= group && 10 * ctas * split * (n + 1) < 18 * n * tplr_sm_count(); ++s)
    if (group % s == 0) split = s;
  return split;
}

// Fp32 elements per token of the scratch that the backward needs for these sizes: the first B*S*H*head_dim hold dQ (zeroed by
// the caller), what is beyond them the parts of dK and dV.
TPLR_API int tplr_attention_bwd_scratch_cols(int B, int S, int H, int KV, int head_dim) {
  const int split = bwd_split(B, S, H, KV, head_dim);
  return (H + (split > 1 ? 2 * KV * split : 0)) * head_dim;
}

static int attention_bwd_impl(const void* qkv, const void* out, const void* dout, const float* lse, float* delta,
                              float* dq32, void* dqkv, int B, int S, int H, int KV, int head_dim, long long ld_qkv,
                              long long ld_o, float scale, const float* cosb, const float* sinb, unsigned int* status,
                              void* stream, bool delta_ready = false) {
  if (B <= 0 || S <= 0) return 0;
  if ((head_dim != 128 && head_dim != 64) || H % KV || (ld_qkv % 8) || (ld_o % 8) || ((uintptr_t)qkv & 15) ||
      ((uintptr_t)dqkv & 15) || ((uintptr_t)dout & 15) || ((uintptr_t)out & 7) || ((uintptr_t)dq32 & 15))
    return -201;
  auto run = head_dim == 128 ? launch_bwd<128> : launch_bwd<64>;
  return run(qkv, out, dout, lse, delta, dq32, dqkv, B, S, H, KV, ld_qkv, ld_o, scale, cosb, sinb, status, (cudaStream_t)stream,
             delta_ready);
}

TPLR_API int tplr_attention_bwd(const void* qkv, const void* out, const void* dout, const float* lse, float* delta,
                                float* dq32, void* dqkv, int B, int S, int H, int KV, int head_dim, long long ld_qkv, long long ld_o,
                                float scale, unsigned int* status, void* stream) {
  TPLR_ENTER();
  return attention_bwd_impl(qkv, out, dout, lse, delta, dq32, dqkv, B, S, H, KV, head_dim, ld_qkv, ld_o, scale, nullptr, nullptr, status, stream);
}

// tplr_attention_bwd for a qkv whose q and k heads were rotated by the producer (tplr_gemm2_rope): dq and dk are
// returned with respect to the un-rotated projection, i.e. rotated back by the opposite angles where they are written
// (dq in the fp32 -> bf16 pass, dk in the kernel's epilogue), so that no separate pass over the gradient is needed.
// cosb / sinb: [S, head_dim / 2] fp32, 16-byte aligned.
TPLR_API int tplr_attention_bwd_unrope(const void* qkv, const void* out, const void* dout, const float* lse, float* delta,
                                       float* dq32, void* dqkv, int B, int S, int H, int KV, int head_dim, long long ld_qkv, long long ld_o,
                                       float scale, const float* cosb, const float* sinb, unsigned int* status, void* stream) {
  TPLR_ENTER();
  if (!cosb || !sinb || ((uintptr_t)cosb & 15) || ((uintptr_t)sinb & 15)) return -201;
  return attention_bwd_impl(qkv, out, dout, lse, delta, dq32, dqkv, B, S, H, KV, head_dim, ld_qkv, ld_o, scale, cosb, sinb, status, stream);
}

// tplr_attention_bwd_unrope for a caller that has already filled `delta` ([B, H, S] fp32, delta[b, h, s] = sum over the
// head's columns of dout * out): the producer of `dout` (tplr_gemm2_attn_dout, the output projection's data
// gradient) forms it in its epilogue, where a row of dout is in registers anyway.
TPLR_API int tplr_attention_bwd_unrope_delta(const void* qkv, const void* out, const void* dout, const float* lse,
                                             float* delta, float* dq32, void* dqkv, int B, int S, int H, int KV, int head_dim,
                                             long long ld_qkv, long long ld_o, float scale, const float* cosb,
                                             const float* sinb, unsigned int* status, void* stream) {
  TPLR_ENTER();
  if (!cosb || !sinb || ((uintptr_t)cosb & 15) || ((uintptr_t)sinb & 15)) return -201;
  return attention_bwd_impl(qkv, out, dout, lse, delta, dq32, dqkv, B, S, H, KV, head_dim, ld_qkv, ld_o, scale, cosb, sinb, status, stream,
                            true);
}

