// Causal self-attention (head_dim 128) for sm_100a on tcgen05 / TMEM, forward and backward.
//
// Input is the fused projection buffer qkv [T, 3H] (row = b*S + s; q heads, then k heads, then v heads,
// RoPE already applied); output is [T, H] plus the per-row log-sum-exp the backward needs.
//
// Forward for small grids, one CTA per (batch, head, 128-query tile), 320 threads (larger grids: attn_fwd2_kernel):
//   warp 0   : TMA producer (Q once, then K/V tiles of 128 keys through a 2-stage ring)
//   warp 1   : tcgen05.mma issuer.  S_j = Q K_j^T goes to one of two TMEM buffers so that S_{j+1} is
//              computed while the softmax of tile j runs; O += P_j V_j accumulates in TMEM.
//   warps 2-9: softmax.  Two threads own query row r (the 32x32b TMEM load shape gives one row per
//              lane), one per 64-key half; they exchange the half-row maximum through shared memory,
//              write P as bf16 into a 128B-swizzled shared tile (the A operand of the second MMA) and
//              rescale O in TMEM only when the running maximum moved by more than 2^8 (lazy rescaling).
// Every wait is bounded; on a timeout the kernel records a status code and leaves through the normal
// teardown.
//
// The reference calls F.scaled_dot_product_attention in its bench models
// (test/fsdp/bench_fsdp2_compare.py:419,480); this file is that op written for Blackwell.
#include "common.cuh"
#include <cuda.h>
#include <cstdlib>

namespace mfsdp {

int make_tmap_bf16(CUtensorMap* map, const void* base, long long batches, long long rows, long long cols, long long ld,
                   int box_rows, int box_cols);      // defined in gemm_sm100.cu (cached)
void ensure_context_on_this_thread();                // likewise

constexpr int kHd = 128;            // head dim
constexpr int kBq = 128;            // queries per CTA
constexpr int kBk = 128;            // keys per iteration
constexpr int kTileBytes = 128 * 128 * 2;   // one [128 x 128] bf16 tile = two 64-column chunks of 16 KB
constexpr int kHalfTile = kTileBytes / 2;
constexpr int kAttnThreads = 320;          // warp 0 TMA, warp 1 MMA, warps 2-9 softmax (two per TMEM lane quadrant)
constexpr float kLog2e = 1.4426950408889634f;

struct AttnFwdArgs {
  int B, S, nH;
  float scale_log2;          // softmax scale * log2(e)
  __nv_bfloat16* out;        // [T, H]
  long long ld_out;
  float* lse;                // [B, nH, S]  natural-log log-sum-exp of the scaled scores
  int* status;
};

struct AttnFwdSmem {
  // offsets from the 1024-aligned base
  static constexpr int kQ = 0;
  static constexpr int kK = kQ + kTileBytes;            // 2 stages
  static constexpr int kV = kK + 2 * kTileBytes;        // 2 stages
  static constexpr int kP = kV + 2 * kTileBytes;
  static constexpr int kXchg = kP + kTileBytes;          // row max [2 parities][2 halves][128] + row sum [2][128]
  static constexpr int kBars = kXchg + 3 * 1024;
  static constexpr int kBytes = kBars + 256 + 1024;
};

__device__ __forceinline__ void softmax_bar_sync() { asm volatile("bar.sync 2, 256;" ::: "memory"); }
// Barrier over the 256 softmax threads that also ORs a predicate, so that every thread takes the
// same decision about leaving the loop after a wait ran out.
__device__ __forceinline__ bool softmax_bar_or(bool pred) {
  uint32_t out;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 2, 256, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(out) : "r"((uint32_t)pred) : "memory");
  return out != 0;
}

// Issue the 8 k-steps of a 128x128x128 MMA whose operands are [128 x 128] bf16 tiles stored as two
// 64-column swizzled chunks.  A K-major operand advances 32 B per k-step inside a chunk and one chunk
// per 64 k; an MN-major operand advances 16 rows (2048 B) per k-step.
__device__ __forceinline__ void mma_tile_128(uint32_t tmem_d, uint32_t a_base, bool a_mn, uint32_t b_base, bool b_mn,
                                             uint32_t idesc, bool accumulate) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint64_t ad = a_mn ? make_smem_desc_sw128(a_base + k * 2048, kHalfTile, 1024)
                             : make_smem_desc_sw128(a_base + (k >> 2) * kHalfTile + (k & 3) * 32, 16, 1024);
    const uint64_t bd = b_mn ? make_smem_desc_sw128(b_base + k * 2048, kHalfTile, 1024)
                             : make_smem_desc_sw128(b_base + (k >> 2) * kHalfTile + (k & 3) * 32, 16, 1024);
    umma_f16_ss(tmem_d, ad, bd, idesc, (accumulate || k > 0) ? 1u : 0u);
  }
}

// Load a [128 rows x 128 cols] bf16 tile of one sequence, whose top-left corner is (row0, col0), as two 64-column boxes.
// Rows past the end of the sequence are zeros and cost no traffic (they are not the next sequence's: its values, infinities
// among them, have no way into this one's products).
__device__ __forceinline__ void tma_load_tile(uint32_t dst, const CUtensorMap* map, uint32_t bar, int col0, int row0, int batch) {
  tma_load_3d(dst, map, bar, col0, row0, batch);
  tma_load_3d(dst + kHalfTile, map, bar, col0 + 64, row0, batch);
}

__global__ void __launch_bounds__(kAttnThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tma_qkv, const AttnFwdArgs p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + AttnFwdSmem::kBars);
  uint64_t* q_full = bars;             // [1]
  uint64_t* k_full = bars + 1;         // [2]
  uint64_t* k_empty = bars + 3;        // [2]
  uint64_t* v_full = bars + 5;         // [2]
  uint64_t* v_empty = bars + 7;        // [2]
  uint64_t* s_full = bars + 9;         // [2]
  uint64_t* p_full = bars + 11;        // [1]
  uint64_t* pv_done = bars + 12;       // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 13);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qt = (int)gridDim.x - 1 - (int)blockIdx.x;     // heavy (late) query tiles first
  const int h = blockIdx.y, b = blockIdx.z;
  const int H = p.nH * kHd;
  const int q0 = qt * kBq;
  const int row_base = b * p.S;
  int nkv = (q0 + kBq + kBk - 1) / kBk;
  const int max_kv = (p.S + kBk - 1) / kBk;
  if (nkv > max_kv) nkv = max_kv;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < 13; ++i) mbar_init(smem_u32(&bars[i]), (i == 11) ? 256 : 1);
    mbar_fence_init();
    tma_prefetch_desc(&tma_qkv);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_begin();
  const uint32_t tmem_o = tmem_base + 256;
  const uint32_t sQ = smem_u32(smem + AttnFwdSmem::kQ), sK = smem_u32(smem + AttnFwdSmem::kK),
                 sV = smem_u32(smem + AttnFwdSmem::kV), sP = smem_u32(smem + AttnFwdSmem::kP);

  if (warp == 0) {
    if (lane == 0) {
      mbar_arrive_expect_tx(smem_u32(q_full), kTileBytes);
      tma_load_tile(sQ, &tma_qkv, smem_u32(q_full), h * kHd, q0, b);
      for (int j = 0; j < nkv; ++j) {
        const uint32_t s = j & 1, ph = (j >> 1) & 1;
        if (!mbar_wait(smem_u32(&k_empty[s]), ph ^ 1, p.status, abort_flag)) break;
        mbar_arrive_expect_tx(smem_u32(&k_full[s]), kTileBytes);
        tma_load_tile(sK + s * kTileBytes, &tma_qkv, smem_u32(&k_full[s]), H + h * kHd, j * kBk, b);
        if (!mbar_wait(smem_u32(&v_empty[s]), ph ^ 1, p.status, abort_flag)) break;
        mbar_arrive_expect_tx(smem_u32(&v_full[s]), kTileBytes);
        tma_load_tile(sV + s * kTileBytes, &tma_qkv, smem_u32(&v_full[s]), 2 * H + h * kHd, j * kBk, b);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);
      constexpr uint32_t idesc_o = make_idesc_bf16(128, 128, false, true);
      bool ok = mbar_wait(smem_u32(q_full), 0, p.status, abort_flag) &&
                mbar_wait(smem_u32(&k_full[0]), 0, p.status, abort_flag);
      if (ok) {
        tc_fence_after();
        mma_tile_128(tmem_base, sQ, false, sK, false, idesc_s, false);
        umma_commit(smem_u32(&k_empty[0]));
        umma_commit(smem_u32(&s_full[0]));
      }
      for (int j = 0; j < nkv && ok; ++j) {
        if (j + 1 < nkv) {
          const uint32_t s1 = (j + 1) & 1, ph1 = ((j + 1) >> 1) & 1;
          if (!mbar_wait(smem_u32(&k_full[s1]), ph1, p.status, abort_flag)) { ok = false; break; }
          tc_fence_after();
          mma_tile_128(tmem_base + s1 * 128, sQ, false, sK + s1 * kTileBytes, false, idesc_s, false);
          umma_commit(smem_u32(&k_empty[s1]));
          umma_commit(smem_u32(&s_full[s1]));
        }
        const uint32_t s = j & 1, ph = (j >> 1) & 1;
        if (!mbar_wait(smem_u32(p_full), j & 1, p.status, abort_flag)) { ok = false; break; }
        if (!mbar_wait(smem_u32(&v_full[s]), ph, p.status, abort_flag)) { ok = false; break; }
        tc_fence_after();
        mma_tile_128(tmem_o, sP, false, sV + s * kTileBytes, true, idesc_o, j > 0);
        umma_commit(smem_u32(&v_empty[s]));
        umma_commit(smem_u32(pv_done));
      }
    }
  } else {
    // ------------------------------------------------------------ softmax / epilogue (256 threads)
    const int q = warp & 3;                      // TMEM lane quadrant this warp may access
    const int half = (warp - 2) >> 2;            // which 64 keys of the tile / which 64 columns of O
    const int r = q * 32 + lane;                 // query row inside the tile == TMEM lane
    const uint32_t lane_off = (uint32_t)(q * 32) << 16;
    const int qi = q0 + r;
    float* xmax = reinterpret_cast<float*>(smem + AttnFwdSmem::kXchg);     // [parity][half][128]
    float* xsum = xmax + 512;                                              // [half][128]
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < nkv; ++j) {
      mbar_wait(smem_u32(&s_full[j & 1]), (j >> 1) & 1, p.status, abort_flag);
      tc_fence_after();
      float s[64];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t t[32];
        tmem_ld_32x32b_x32(tmem_base + (j & 1) * 128 + lane_off + half * 64 + c * 32, t);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 32; ++e) s[c * 32 + e] = __uint_as_float(t[e]);
      }
      if (j == nkv - 1) {
        const int kv0 = j * kBk + half * 64;
#pragma unroll
        for (int e = 0; e < 64; ++e)
          if (kv0 + e > qi) s[e] = -INFINITY;
      }
      float mx = s[0];
#pragma unroll
      for (int e = 1; e < 64; ++e) mx = fmaxf(mx, s[e]);
      xmax[(j & 1) * 256 + half * 128 + r] = mx;
      if (softmax_bar_or(*abort_flag != 0)) { ok = false; break; }
      mx = fmaxf(mx, xmax[(j & 1) * 256 + (half ^ 1) * 128 + r]) * p.scale_log2;
      if (mx == -INFINITY) mx = 0.f;
      const float m_new = fmaxf(m_used, mx);
      const bool need = (j > 0) && (m_new - m_used > 8.f);
      const bool any_need = __any_sync(0xffffffffu, need);
      const float m_next = (j == 0 || any_need) ? m_new : m_used;
      const float factor = (j == 0) ? 0.f : exp2f(m_used - m_next);
      float sum = 0.f;
      uint32_t pk[32];
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        const float p0 = exp2f(s[2 * e] * p.scale_log2 - m_next);
        const float p1 = exp2f(s[2 * e + 1] * p.scale_log2 - m_next);
        sum += p0 + p1;
        pk[e] = pack_bf16x2(p0, p1);
      }
      l = l * factor + sum;
      m_used = m_next;
      if (j > 0) {
        mbar_wait(smem_u32(pv_done), (j - 1) & 1, p.status, abort_flag);
        tc_fence_after();
        if (any_need) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t t[32];
            tmem_ld_32x32b_x32(tmem_o + lane_off + half * 64 + c * 32, t);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) t[e] = __float_as_uint(__uint_as_float(t[e]) * factor);
            tmem_st_32x32b_x32(tmem_o + lane_off + half * 64 + c * 32, t);
          }
          tmem_st_wait();
        }
      }
      uint8_t* prow = smem + AttnFwdSmem::kP + half * kHalfTile + r * 128;
#pragma unroll
      for (int kc = 0; kc < 8; ++kc) {
        const int phys = kc ^ (r & 7);
        *reinterpret_cast<uint4*>(prow + phys * 16) = make_uint4(pk[kc * 4], pk[kc * 4 + 1], pk[kc * 4 + 2], pk[kc * 4 + 3]);
      }
      fence_proxy_async_smem();
      tc_fence_before();
      mbar_arrive(smem_u32(p_full));
    }
    if (ok) {
      mbar_wait(smem_u32(pv_done), (nkv - 1) & 1, p.status, abort_flag);
      xsum[half * 128 + r] = l;
      ok = !softmax_bar_or(*abort_flag != 0);
    }
    if (ok) {
      tc_fence_after();
      l += xsum[(half ^ 1) * 128 + r];
      const float inv = 1.f / l;
      const bool row_ok = qi < p.S;
      __nv_bfloat16* orow = p.out + (long long)(row_base + qi) * p.ld_out + h * kHd + half * 64;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t t[32];
        tmem_ld_32x32b_x32(tmem_o + lane_off + half * 64 + c * 32, t);
        tmem_ld_wait();
        if (row_ok) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint4 o;
            o.x = pack_bf16x2(__uint_as_float(t[g * 8 + 0]) * inv, __uint_as_float(t[g * 8 + 1]) * inv);
            o.y = pack_bf16x2(__uint_as_float(t[g * 8 + 2]) * inv, __uint_as_float(t[g * 8 + 3]) * inv);
            o.z = pack_bf16x2(__uint_as_float(t[g * 8 + 4]) * inv, __uint_as_float(t[g * 8 + 5]) * inv);
            o.w = pack_bf16x2(__uint_as_float(t[g * 8 + 6]) * inv, __uint_as_float(t[g * 8 + 7]) * inv);
            *reinterpret_cast<uint4*>(orow + c * 32 + g * 8) = o;
          }
        }
      }
      if (half == 0 && row_ok && p.lse) p.lse[((long long)b * p.nH + h) * p.S + qi] = (m_used + log2f(l)) * 0.6931471805599453f;
    }
  }
  if (*abort_flag) __nanosleep(1000000);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// Forward for grids that fill the chip (attn_fwd_two_tiles): one CTA per (batch, head, 256 queries), two 128-query tiles in flight.
// One tile's softmax alone leaves the tensor pipe idle while it runs and waits while the pipe works; with two tiles
// the products of one run beside the softmax of the other.  A thread owns a whole query row (no exchange between
// threads, no block barrier in the loop) and P goes back to tensor memory over the scores it came from, so it
// never touches shared memory.  Tensor memory: S0 | S1 | O0 | O1, 128 columns each; P_t packs into the first 64
// columns of S_t.  Per 128 keys and 2 x 128 queries the tensor pipe needs 2048 cycles and the exponentials as many:
// both bound it.  Measured (one tile per block -> two): 32 heads of 16384 rows 2476 -> 1791 us, 1228 TFLOP/s; 16 heads
// of 2 x 4096 rows 212 -> 141 us; of 4 x 1024 47 -> 33 us; of 3 x 1333 56 -> 41 us.
struct AttnFwd2Smem {
  static constexpr int kQ = 0;                          // 2 query tiles
  static constexpr int kK = kQ + 2 * kTileBytes;        // 2 stages
  static constexpr int kV = kK + 2 * kTileBytes;        // 2 stages
  static constexpr int kBars = kV + 2 * kTileBytes;
  static constexpr int kBytes = kBars + 256 + 1024;
};

constexpr int kFwd2Threads = 384;     // warp 0 TMA, warp 1 MMA, 2 and 3 idle, warps 4-7 and 8-11 the two tiles' softmax
// A row of 128 scores and their packed results need more than the 168 registers per thread of a 384-thread block,
// so the first warpgroup hands registers to the other two: 128 * 56 + 256 * 224 = the launch's 64,512.
constexpr int kRegsIssue = 56, kRegsSoftmax = 224;

// D[128 x 128] (+)= P[128 x 128 (packed bf16 pairs in tensor memory)] * V[128 keys x 128 (N contiguous)]
__device__ __forceinline__ void mma_pv_ts(uint32_t tmem_d, uint32_t tmem_p, uint32_t v_base, bool accumulate) {
  constexpr uint32_t idesc = make_idesc_bf16(128, 128, false, true);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint64_t bd = make_smem_desc_sw128(v_base + k * 2048, kHalfTile, 1024);
    umma_f16_ts(tmem_d, tmem_p + k * 8, bd, idesc, (accumulate || k > 0) ? 1u : 0u);
  }
}

__global__ void __launch_bounds__(kFwd2Threads, 1)
attn_fwd2_kernel(const __grid_constant__ CUtensorMap tma_qkv, const AttnFwdArgs p, const int heads_per_group) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + AttnFwd2Smem::kBars);
  uint64_t* q_full = bars;             // [1]
  uint64_t* k_full = bars + 1;         // [2]
  uint64_t* k_empty = bars + 3;        // [2]
  uint64_t* v_full = bars + 5;         // [2]
  uint64_t* v_empty = bars + 7;        // [2]
  uint64_t* s_full = bars + 9;         // [2] per query tile
  uint64_t* p_full = bars + 11;        // [2] per query tile, count 128
  uint64_t* o_done = bars + 13;        // [2] per query tile: its last product has finished
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Blocks are numbered so that, within a group of heads whose K and V fit the L2 together, the late (long) query
  // tiles of all heads come first and the short ones fill the end of the grid.
  const int nq = (p.S + 2 * kBq - 1) / (2 * kBq), nheads = p.nH * p.B;
  const int grp = (int)blockIdx.x / (heads_per_group * nq);
  const int in_grp = (int)blockIdx.x - grp * heads_per_group * nq;
  const int gheads = min(heads_per_group, nheads - grp * heads_per_group);
  const int qt = nq - 1 - in_grp / gheads;
  const int bh = grp * heads_per_group + in_grp % gheads;
  const int b = bh / p.nH, h = bh - b * p.nH;
  const int H = p.nH * kHd;
  const int q0 = qt * 2 * kBq;
  const int row_base = b * p.S;
  const int n0 = q0 / kBk + 1;                                 // key tiles of query tile 0
  const int n1 = q0 + kBq < p.S ? n0 + 1 : 0;                  // ... and of tile 1, if it has any row
  const int n_max = n1 > 0 ? n1 : n0;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < 15; ++i) mbar_init(smem_u32(&bars[i]), (i == 11 || i == 12) ? 128 : 1);
    mbar_fence_init();
    tma_prefetch_desc(&tma_qkv);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_begin();
  const uint32_t sQ = smem_u32(smem + AttnFwd2Smem::kQ), sK = smem_u32(smem + AttnFwd2Smem::kK),
                 sV = smem_u32(smem + AttnFwd2Smem::kV);

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIssue));
    if (warp == 0 && lane == 0) {
      mbar_arrive_expect_tx(smem_u32(q_full), n1 > 0 ? 2 * kTileBytes : kTileBytes);
      tma_load_tile(sQ, &tma_qkv, smem_u32(q_full), h * kHd, q0, b);
      if (n1 > 0) tma_load_tile(sQ + kTileBytes, &tma_qkv, smem_u32(q_full), h * kHd, q0 + kBq, b);
      for (int j = 0; j < n_max; ++j) {
        const uint32_t s = j & 1, ph = (j >> 1) & 1;
        if (!mbar_wait(smem_u32(&k_empty[s]), ph ^ 1, p.status, abort_flag)) break;
        mbar_arrive_expect_tx(smem_u32(&k_full[s]), kTileBytes);
        tma_load_tile(sK + s * kTileBytes, &tma_qkv, smem_u32(&k_full[s]), H + h * kHd, j * kBk, b);
        if (!mbar_wait(smem_u32(&v_empty[s]), ph ^ 1, p.status, abort_flag)) break;
        mbar_arrive_expect_tx(smem_u32(&v_full[s]), kTileBytes);
        tma_load_tile(sV + s * kTileBytes, &tma_qkv, smem_u32(&v_full[s]), 2 * H + h * kHd, j * kBk, b);
      }
    } else if (warp == 1 && lane == 0) {
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, false, false);
      bool ok = mbar_wait(smem_u32(q_full), 0, p.status, abort_flag) &&
                mbar_wait(smem_u32(&k_full[0]), 0, p.status, abort_flag);
      if (ok) {
        tc_fence_after();
        for (int t = 0; t < (n1 > 0 ? 2 : 1); ++t) {
          mma_tile_128(tmem_base + t * 128, sQ + t * kTileBytes, false, sK, false, idesc_s, false);
          umma_commit(smem_u32(&s_full[t]));
        }
        umma_commit(smem_u32(&k_empty[0]));
      }
      for (int j = 0; j < n_max && ok; ++j) {
        const uint32_t s = j & 1, ph = (j >> 1) & 1, s1 = (j + 1) & 1, ph1 = ((j + 1) >> 1) & 1;
        if (!mbar_wait(smem_u32(&v_full[s]), ph, p.status, abort_flag)) { ok = false; break; }
        if (j + 1 < n_max && !mbar_wait(smem_u32(&k_full[s1]), ph1, p.status, abort_flag)) { ok = false; break; }
        for (int t = 0; t < 2; ++t) {
          const int n = t == 0 ? n0 : n1;
          if (j >= n) continue;
          if (!mbar_wait(smem_u32(&p_full[t]), j & 1, p.status, abort_flag)) { ok = false; break; }
          tc_fence_after();
          // S_t's scores have all been read and P_t lies over them; the next scores may overwrite both because the
          // tensor pipe runs a thread's products in the order they were issued
          mma_pv_ts(tmem_base + 256 + t * 128, tmem_base + t * 128, sV + s * kTileBytes, j > 0);
          if (j + 1 < n) {
            mma_tile_128(tmem_base + t * 128, sQ + t * kTileBytes, false, sK + s1 * kTileBytes, false, idesc_s, false);
            umma_commit(smem_u32(&s_full[t]));
          } else {
            umma_commit(smem_u32(&o_done[t]));
          }
        }
        umma_commit(smem_u32(&v_empty[s]));
        if (j + 1 < n_max) umma_commit(smem_u32(&k_empty[s1]));
      }
    }
  } else {
    // ------------------------------------------------------------ softmax / epilogue: 4 warps per query tile
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoftmax));
    const int t = (warp - 4) >> 2;
    const int q = warp & 3;                      // TMEM lane quadrant this warp may access
    const int r = q * 32 + lane;                 // query row inside the tile == TMEM lane
    const int n = t == 0 ? n0 : n1;
    const uint32_t tmem_s = tmem_base + t * 128 + ((uint32_t)(q * 32) << 16);
    const uint32_t tmem_o = tmem_s + 256;
    const int qi = q0 + t * kBq + r;
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < n; ++j) {
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_full[t]), j & 1, p.status, abort_flag))) { ok = false; break; }
      tc_fence_after();
      uint32_t u[128];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(tmem_s + c * 32, *reinterpret_cast<uint32_t(*)[32]>(u + c * 32));
      tmem_ld_wait();
      if (j == n - 1) {
        const int kv0 = j * kBk;
#pragma unroll
        for (int e = 0; e < 128; ++e)
          if (kv0 + e > qi) u[e] = 0xff800000u;
      }
      float m4[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) m4[e] = fmaxf(__uint_as_float(u[e]), __uint_as_float(u[4 + e]));
#pragma unroll
      for (int e = 8; e < 128; e += 8)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          m4[k] = fmaxf(fmaxf(m4[k], __uint_as_float(u[e + k])), __uint_as_float(u[e + 4 + k]));
      float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * p.scale_log2;
      if (mx == -INFINITY) mx = 0.f;
      const float m_new = fmaxf(m_used, mx);
      const bool need = (j > 0) && (m_new - m_used > 8.f);
      const bool any_need = __any_sync(0xffffffffu, need);
      const float m_next = (j == 0 || any_need) ? m_new : m_used;
      const float factor = (j == 0) ? 0.f : exp2f(m_used - m_next);
      m_used = m_next;
      const uint64_t sc2 = pack_f32x2(p.scale_log2, p.scale_log2), nm2 = pack_f32x2(-m_next, -m_next);
      uint64_t sum2[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t pk[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          float x0, x1;
          unpack_f32x2(fma_f32x2(pack_u32x2(u[half * 64 + 2 * e], u[half * 64 + 2 * e + 1]), sc2, nm2), x0, x1);
          x0 = exp2f(x0);
          x1 = exp2f(x1);
          sum2[e & 3] = add_f32x2(sum2[e & 3], pack_f32x2(x0, x1));
          pk[e] = pack_bf16x2(x0, x1);
        }
        tmem_st_32x32b_x32(tmem_s + half * 32, pk);
      }
      float a0, a1;
      unpack_f32x2(add_f32x2(add_f32x2(sum2[0], sum2[1]), add_f32x2(sum2[2], sum2[3])), a0, a1);
      l = l * factor + (a0 + a1);
      if (any_need) {
        // the scores just read were computed after the previous P V product, so O is complete
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t o[32];
          tmem_ld_32x32b_x32(tmem_o + c * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * factor);
          tmem_st_32x32b_x32(tmem_o + c * 32, o);
        }
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(smem_u32(&p_full[t]));
    }
    if (ok && n > 0) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&o_done[t]), 0, p.status, abort_flag));
    if (ok && n > 0) {
      tc_fence_after();
      const float inv = 1.f / l;
      const bool row_ok = qi < p.S;
      __nv_bfloat16* orow = p.out + (long long)(row_base + qi) * p.ld_out + h * kHd;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t o[32];
        tmem_ld_32x32b_x32(tmem_o + c * 32, o);
        tmem_ld_wait();
        if (row_ok) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(o[g * 8 + 0]) * inv, __uint_as_float(o[g * 8 + 1]) * inv);
            w.y = pack_bf16x2(__uint_as_float(o[g * 8 + 2]) * inv, __uint_as_float(o[g * 8 + 3]) * inv);
            w.z = pack_bf16x2(__uint_as_float(o[g * 8 + 4]) * inv, __uint_as_float(o[g * 8 + 5]) * inv);
            w.w = pack_bf16x2(__uint_as_float(o[g * 8 + 6]) * inv, __uint_as_float(o[g * 8 + 7]) * inv);
            *reinterpret_cast<uint4*>(orow + c * 32 + g * 8) = w;
          }
        }
      }
      if (row_ok && p.lse) p.lse[((long long)b * p.nH + h) * p.S + qi] = (m_used + log2f(l)) * 0.6931471805599453f;
    }
  }
  if (*abort_flag) __nanosleep(1000000);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}


// =============================================================================== backward
// Two kinds of block without atomics (the sums have one order in every run), sharing one body:
//   DQ = false: one CTA per (batch, head, 128-key tile).  K_j and V_j stay in shared memory, the query axis streams
//               in tiles of 128 rows (Q_i, dO_i).  S^T = K_j Q_i^T and dP^T = V_j dO_i^T land in TMEM (thread = key
//               row, four threads per row), P^T and dS^T go back over them as bf16, dV += P^T dO_i and dK += dS^T Q_i
//               accumulate in TMEM.
//   DQ = true : one CTA per (batch, head, 128-query tile).  Q_i and dO_i stay, keys stream (K_j, V_j).
//               S = Q_i K_j^T, dP = dO_i V_j^T, dQ += dS K_j.
// Bound by the tensor pipe (four and three 128 x 128 x 128 products per tile, 512 cycles each).  Its queue never runs
// dry although every buffer is single: while the threads turn dP into dS the pipe adds to dV and computes the next S,
// and while they take exponentials of that S it adds to dK / dQ and computes the next dP.  128-wide streamed tiles,
// because a 64-wide second operand makes the products wait for shared memory (A and B together 192 B per cycle).
// Streamed tiles go through a ring of five 32 KB buffers in the order of their first use (Q_0 dO_0 Q_1 dO_1 Q_2 ... |
// K_0 V_0 K_1 ...), each freed by the last product that reads it: with two buffers per operand a load could only start
// one product before its tile was needed, and the pipe was busy 43 % of the time.  The row statistics of a streamed tile
// arrive with it, in the same barriers, so no thread waits for another.
// Four threads share a row: with two (2 warps per scheduler) the fixed latencies of the element-wise chains showed.
// Measured (64-wide streamed tiles -> 128-wide in pairs of buffers -> this): 16 heads of 2 x 4096 rows 806 -> 547 ->
// 492 us, 16 heads of 3 x 1333 rows 201 -> 157 -> 135 us; 32 heads of 16384 rows 9.9 -> 7.2 -> 6.9 to 7.4 ms back to back,
// where the power cap takes the clock to 1.69 GHz, and 6.6 ms (838 TFLOP/s counting five products per tile) in calls
// apart from one another.
constexpr int kBwdThreads = 640;      // warp 0 TMA, warp 1 MMA, 2 and 3 idle, warps 4-19 P and dS
constexpr int kBwdCols = 32;          // streamed columns per thread
// 640 threads are launched with 96 registers each, 61,440 in all: 128 * 64 + 512 * 104.
constexpr int kBwdRegsIssue = 64, kBwdRegsSoftmax = 104;
constexpr int kStatBytes = 128 * 4;   // one row statistic of a streamed tile

struct AttnBwdArgs {
  int B, S, nH;
  long long Sp;              // row pitch of the statistics: S rounded up to 128
  float scale, scale_log2;
  const float* nlse2;        // [B * nH, Sp] minus log-sum-exp in log2 units
  const float* ndelta;       // [B * nH, Sp] minus rowsum(dO * O)
  __nv_bfloat16* dqkv;       // [T, 3H]
  long long ld_dqkv;
  int* status;
  int heads_per_group;
};

constexpr int kRing = 5;
struct AttnBwdSmem {
  static constexpr int kA0 = 0;
  static constexpr int kA1 = kA0 + kTileBytes;
  static constexpr int kB = kA1 + kTileBytes;             // the ring
  static constexpr int kNlse = kB + kRing * kTileBytes;   // 3 stages: a tile's Q is loaded while two earlier S wait
  static constexpr int kNdelta = kNlse + 3 * kStatBytes;  // 2 stages
  static constexpr int kBars = kNdelta + 2 * kStatBytes;
  static constexpr int kBytes = kBars + 256;              // 232,192 of the 232,448 that a block may have
};


// D[128 x 128] (+)= P[128 x 128] * B[128 rows along K x 128, N contiguous].  The four threads of a row have each packed
// their 32 elements into the first 16 columns of their own quarter.
__device__ __forceinline__ void mma_acc_ts(uint32_t tmem_d, uint32_t tmem_p, uint32_t b_base, bool accumulate) {
  constexpr uint32_t idesc = make_idesc_bf16(128, 128, false, true);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint64_t bd = make_smem_desc_sw128(b_base + k * 2048, kHalfTile, 1024);
    umma_f16_ts(tmem_d, tmem_p + (k >> 1) * 32 + (k & 1) * 8, bd, idesc, (accumulate || k > 0) ? 1u : 0u);
  }
}

template <bool DQ, bool SKIP>
__device__ __forceinline__ void attn_bwd_block(const CUtensorMap& tma_qkv, const CUtensorMap& tma_do, const AttnBwdArgs& p,
                                               const int block) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023) {         // the swizzled tiles need it; nothing has been started yet
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, (int)kErrBadArgument);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + AttnBwdSmem::kBars);
  uint64_t* full = bars;               // [5] ring: tile 2i is Q_i / K_i, tile 2i+1 is dO_i / V_i
  uint64_t* empty = bars + kRing;      // [5] the last product that reads a tile has finished
  uint64_t* stat_full = bars + 10;     // [1]
  uint64_t* s_full = bars + 11;        // [1]
  uint64_t* dp_full = bars + 12;       // [1]
  uint64_t* p_ready = bars + 13;       // [1] count 512: S read, P written
  uint64_t* ds_ready = bars + 14;      // [1] count 512: dP read, dS written
  uint64_t* acc_done = bars + 15;      // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Blocks in the order of attn_fwd2_kernel: per group of heads the long tiles first.
  const int nt = (p.S + 127) / 128, nheads = p.nH * p.B;
  const int grp = block / (p.heads_per_group * nt);
  const int in_grp = block - grp * p.heads_per_group * nt;
  const int gheads = min(p.heads_per_group, nheads - grp * p.heads_per_group);
  const int nth = in_grp / gheads;
  const int bh = grp * p.heads_per_group + in_grp % gheads;
  const int b = bh / p.nH, h = bh - b * p.nH;
  const int H = p.nH * kHd;
  const int row_base = b * p.S;
  // DQ: stationary tile = queries [r0, r0 + 128), streamed = keys up to the diagonal; otherwise stationary = keys,
  // streamed = queries from the diagonal on.
  const int tile = DQ ? nt - 1 - nth : nth;
  const int r0 = tile * 128;
  const int t_begin = DQ ? 0 : tile;
  const int T = DQ ? tile + 1 : nt - tile;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < 16; ++i) mbar_init(smem_u32(&bars[i]), (i == 13 || i == 14) ? 512 : 1);
    mbar_fence_init();
    tma_prefetch_desc(&tma_qkv);
    tma_prefetch_desc(&tma_do);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_begin();
  const uint32_t tmem_dp = tmem_base + 128, tmem_acc0 = tmem_base + 256, tmem_acc1 = tmem_base + 384;
  const uint32_t sA0 = smem_u32(smem + AttnBwdSmem::kA0), sA1 = smem_u32(smem + AttnBwdSmem::kA1),
                 sB = smem_u32(smem + AttnBwdSmem::kB);
  auto slot = [&](int tile_idx) { return sB + (uint32_t)(tile_idx % kRing) * kTileBytes; };
  auto full_bar = [&](int tile_idx) { return smem_u32(&full[tile_idx % kRing]); };
  auto full_phase = [&](int tile_idx) { return (uint32_t)(tile_idx / kRing) & 1u; };

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kBwdRegsIssue));
    if (warp == 0 && lane == 0) {
      mbar_arrive_expect_tx(smem_u32(stat_full), 2 * kTileBytes);
      if (DQ) {
        tma_load_tile(sA0, &tma_qkv, smem_u32(stat_full), h * kHd, r0, b);          // Q_i
        tma_load_tile(sA1, &tma_do, smem_u32(stat_full), h * kHd, r0, b);           // dO_i
      } else {
        tma_load_tile(sA0, &tma_qkv, smem_u32(stat_full), H + h * kHd, r0, b);      // K_j
        tma_load_tile(sA1, &tma_qkv, smem_u32(stat_full), 2 * H + h * kHd, r0, b);  // V_j
      }
      for (int k = 0; k < 2 * T; ++k) {
        if (!mbar_wait(smem_u32(&empty[k % kRing]), full_phase(k) ^ 1, p.status, abort_flag)) break;
        const uint32_t bar = full_bar(k);
        mbar_arrive_expect_tx(bar, kTileBytes + (DQ ? 0 : kStatBytes));
        const int i = k >> 1, t0 = (t_begin + i) * 128;
        const long long stat = (long long)bh * p.Sp + t0;
        if (DQ) {
          tma_load_tile(slot(k), &tma_qkv, bar, ((k & 1) ? 2 * H : H) + h * kHd, t0, b);          // K_t, V_t
        } else if (k & 1) {
          tma_load_tile(slot(k), &tma_do, bar, h * kHd, t0, b);                                   // dO_t
          bulk_load(smem_u32(smem + AttnBwdSmem::kNdelta + (i & 1) * kStatBytes), p.ndelta + stat, kStatBytes, bar);
        } else {
          tma_load_tile(slot(k), &tma_qkv, bar, h * kHd, t0, b);                                  // Q_t
          bulk_load(smem_u32(smem + AttnBwdSmem::kNlse + (i % 3) * kStatBytes), p.nlse2 + stat, kStatBytes, bar);
        }
      }
    } else if (warp == 1 && lane == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(128, 128, false, false);
      bool ok = mbar_wait(smem_u32(stat_full), 0, p.status, abort_flag) && mbar_wait(full_bar(0), 0, p.status, abort_flag);
      if (ok) {
        tc_fence_after();
        mma_tile_128(tmem_base, sA0, false, slot(0), false, idesc, false);
        umma_commit(smem_u32(s_full));
        ok = mbar_wait(full_bar(1), 0, p.status, abort_flag);
      }
      if (ok) {
        tc_fence_after();
        mma_tile_128(tmem_dp, sA1, false, slot(1), false, idesc, false);
        umma_commit(smem_u32(dp_full));
        if (DQ) umma_commit(smem_u32(&empty[1]));                                      // V_0 is not read again
      }
      for (int i = 0; i < T && ok; ++i) {
        const int k = 2 * i;
        const bool more = i + 1 < T;
        if (more && !mbar_wait(full_bar(k + 2), full_phase(k + 2), p.status, abort_flag)) { ok = false; break; }
        if (!mbar_wait(smem_u32(p_ready), i & 1, p.status, abort_flag)) { ok = false; break; }
        tc_fence_after();
        if (!DQ) {
          mma_acc_ts(tmem_acc0, tmem_base, slot(k + 1), i > 0);                        // dV += P^T dO_t
          umma_commit(smem_u32(&empty[(k + 1) % kRing]));
        }
        if (more) {
          // the next S may go over P: the pipe runs one thread's products in the order they were issued
          mma_tile_128(tmem_base, sA0, false, slot(k + 2), false, idesc, false);
          umma_commit(smem_u32(s_full));
        }
        if (!mbar_wait(smem_u32(ds_ready), i & 1, p.status, abort_flag)) { ok = false; break; }
        tc_fence_after();
        mma_acc_ts(tmem_acc1, tmem_dp, slot(k), i > 0);                                // dK += dS^T Q_t  |  dQ += dS K_t
        umma_commit(smem_u32(&empty[k % kRing]));
        if (more) {
          if (!mbar_wait(full_bar(k + 3), full_phase(k + 3), p.status, abort_flag)) { ok = false; break; }
          tc_fence_after();
          mma_tile_128(tmem_dp, sA1, false, slot(k + 3), false, idesc, false);
          umma_commit(smem_u32(dp_full));
          if (DQ) umma_commit(smem_u32(&empty[(k + 3) % kRing]));
        }
      }
      if (ok) umma_commit(smem_u32(acc_done));
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kBwdRegsSoftmax));
    const int q = warp & 3;                      // TMEM lane quadrant this warp may access
    const int part = (warp - 4) >> 2;            // which 32 of the 128 streamed columns this thread handles
    const int r = q * 32 + lane;                 // stationary row inside the tile == TMEM lane
    const uint32_t lane_off = (uint32_t)(q * 32) << 16;
    const uint32_t my_s = tmem_base + lane_off + part * kBwdCols, my_dp = tmem_dp + lane_off + part * kBwdCols;
    const int stat_idx = r0 + r;
    uint64_t own_nlse = 0, own_ndelta = 0;
    if (DQ) {                                    // the pitch covers whole tiles
      const float a = p.nlse2[(long long)bh * p.Sp + stat_idx], d = p.ndelta[(long long)bh * p.Sp + stat_idx];
      own_nlse = pack_f32x2(a, a);
      own_ndelta = pack_f32x2(d, d);
    }
    const uint64_t sc2 = pack_f32x2(p.scale_log2, p.scale_log2);
    // zero the elements above the diagonal and past the end of the sequence; first = index of x[0] along the streamed axis
    auto mask_row = [&](float (&x)[kBwdCols], int first) {
#pragma unroll
      for (int e = 0; e < kBwdCols; ++e)
        if (DQ ? first + e > stat_idx : (first + e < stat_idx || first + e >= p.S)) x[e] = 0.f;
    };
    bool ok = true;
    for (int i = 0; i < T; ++i) {
      bool got = mbar_wait(smem_u32(s_full), i & 1, p.status, abort_flag);
      if (!DQ) got = got && mbar_wait(full_bar(2 * i), full_phase(2 * i), p.status, abort_flag);   // nlse2
      if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
      tc_fence_after();
      const int c0 = (t_begin + i) * 128;        // first streamed index of this tile
      // tiles on the diagonal and at the end of the sequence have elements that do not count
      const bool need_mask = c0 == r0 || (!DQ && c0 + 128 > p.S);
      const uint64_t* nlse = reinterpret_cast<const uint64_t*>(smem + AttnBwdSmem::kNlse + (i % 3) * kStatBytes) + part * (kBwdCols / 2);
      const uint64_t* ndelta = reinterpret_cast<const uint64_t*>(smem + AttnBwdSmem::kNdelta + (i & 1) * kStatBytes) + part * (kBwdCols / 2);
      // a warp none of whose elements counts writes its zeros without computing them
      const int e0 = c0 + part * kBwdCols, w0 = r0 + q * 32;
      const bool skip = SKIP && need_mask && (w0 >= p.S || (DQ ? e0 > w0 + 31 : (e0 + kBwdCols <= w0 || e0 >= p.S)));
      float pe[kBwdCols];
      if (skip) {
#pragma unroll
        for (int e = 0; e < kBwdCols; ++e) pe[e] = 0.f;
      } else {
        uint32_t sv[kBwdCols];
        tmem_ld_32x32b_x32(my_s, sv);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < kBwdCols / 2; ++e) {
          unpack_f32x2(fma_f32x2(pack_u32x2(sv[2 * e], sv[2 * e + 1]), sc2, DQ ? own_nlse : nlse[e]), pe[2 * e], pe[2 * e + 1]);
          pe[2 * e] = exp2f(pe[2 * e]);
          pe[2 * e + 1] = exp2f(pe[2 * e + 1]);
        }
      }
      if (need_mask && !skip) mask_row(pe, e0);
      if (!DQ) {
        uint32_t pk[kBwdCols / 2];
#pragma unroll
        for (int e = 0; e < kBwdCols / 2; ++e) pk[e] = pack_bf16x2(pe[2 * e], pe[2 * e + 1]);
        tmem_st_32x32b_x16(my_s, pk);
        tmem_st_wait();
      }
      // dO_i has to be there for dV now; its buffer, and with it this barrier's phase, may be reused from here on
      if (!DQ && !__all_sync(0xffffffffu, mbar_wait(full_bar(2 * i + 1), full_phase(2 * i + 1), p.status, abort_flag))) { ok = false; break; }
      tc_fence_before();
      mbar_arrive(smem_u32(p_ready));
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(dp_full), i & 1, p.status, abort_flag))) { ok = false; break; }
      tc_fence_after();
      if (skip) {
        uint32_t pk[kBwdCols / 2];
#pragma unroll
        for (int e = 0; e < kBwdCols / 2; ++e) pk[e] = 0u;
        tmem_st_32x32b_x16(my_dp, pk);
        tmem_st_wait();
      } else {
        uint32_t dv[kBwdCols], pk[kBwdCols / 2];
        tmem_ld_32x32b_x32(my_dp, dv);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < kBwdCols / 2; ++e)
          unpack_f32x2(mul_f32x2(pack_f32x2(pe[2 * e], pe[2 * e + 1]),
                                 add_f32x2(pack_u32x2(dv[2 * e], dv[2 * e + 1]), DQ ? own_ndelta : ndelta[e])),
                       pe[2 * e], pe[2 * e + 1]);
        if (need_mask) mask_row(pe, e0);         // 0 * inf from elements that do not count
#pragma unroll
        for (int e = 0; e < kBwdCols / 2; ++e) pk[e] = pack_bf16x2(pe[2 * e], pe[2 * e + 1]);
        tmem_st_32x32b_x16(my_dp, pk);
        tmem_st_wait();
      }
      tc_fence_before();
      mbar_arrive(smem_u32(ds_ready));
    }
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(acc_done), 0, p.status, abort_flag));
    if (ok) {
      // tcgen05.ld is warp-collective: every lane takes part, only the stores depend on the row being valid
      const bool row_ok = stat_idx < p.S;
      tc_fence_after();
      __nv_bfloat16* grow = p.dqkv + (long long)(row_base + stat_idx) * p.ld_dqkv + h * kHd;
#pragma unroll
      for (int a = (DQ ? 1 : 0); a < 2; ++a) {
        // acc0 = dV (columns 2H..); acc1 = dK (columns H..) or dQ (columns 0..), whose factor is applied here, once,
        // to the fp32 sums; each thread stores 32 columns
        __nv_bfloat16* dst = grow + (DQ ? 0 : (a == 0 ? 2 * H : H)) + part * kBwdCols;
        const float f = a == 0 ? 1.f : p.scale;
        uint32_t t4[kBwdCols];
        tmem_ld_32x32b_x32((a == 0 ? tmem_acc0 : tmem_acc1) + lane_off + part * kBwdCols, t4);
        tmem_ld_wait();
        if (!row_ok) continue;
#pragma unroll
        for (int g = 0; g < kBwdCols / 8; ++g) {
          uint4 o;
          o.x = pack_bf16x2(__uint_as_float(t4[g * 8 + 0]) * f, __uint_as_float(t4[g * 8 + 1]) * f);
          o.y = pack_bf16x2(__uint_as_float(t4[g * 8 + 2]) * f, __uint_as_float(t4[g * 8 + 3]) * f);
          o.z = pack_bf16x2(__uint_as_float(t4[g * 8 + 4]) * f, __uint_as_float(t4[g * 8 + 5]) * f);
          o.w = pack_bf16x2(__uint_as_float(t4[g * 8 + 6]) * f, __uint_as_float(t4[g * 8 + 7]) * f);
          *reinterpret_cast<uint4*>(dst + g * 8) = o;
        }
      }
    }
  }
  if (*abort_flag) __nanosleep(1000000);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// Both kinds of block in one grid, dK / dV first, so that the first kind's last wave is filled by the long blocks of the
// second (a head of 1024 rows has 8 blocks of each kind, 1 to 8 tiles long).  Two launches -> one, preparation included:
// 16 heads of 1024 rows 51.5 -> 36.6 us, of 4 x 1024 132 -> 120 us, of 3 x 1333 155 -> 143 us, 8 heads of 8192 rows 478 ->
// 441 us.  Alternating kinds were slower at long rows, where each streams tensors of its own through the L2.
template <bool SKIP>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tma_qkv, const __grid_constant__ CUtensorMap tma_do,
                const __grid_constant__ AttnBwdArgs p) {
  const int n = (int)(gridDim.x >> 1), block = (int)blockIdx.x;
  if (block < n) attn_bwd_block<false, SKIP>(tma_qkv, tma_do, p, block);
  else attn_bwd_block<true, SKIP>(tma_qkv, tma_do, p, block - n);
}

// nlse2 = -lse * log2(e); ndelta = -rowsum(dO * O); both zero for the rows that pad a head to whole tiles.  Half a
// warp per (row, head), 16 bytes of each operand per lane.
__global__ void __launch_bounds__(256)
attn_bwd_prep_kernel(const __nv_bfloat16* __restrict__ dout, long long ld_do, const __nv_bfloat16* __restrict__ out,
                     long long ld_o, const float* __restrict__ lse, float* __restrict__ nlse2, float* __restrict__ ndelta,
                     int B, int S, int nH, int Sp) {
  const long long w = (long long)blockIdx.x * 16 + (threadIdx.x >> 4);
  const int lane = threadIdx.x & 15;
  pdl_begin();
  if (w >= (long long)B * Sp * nH) return;                 // whole half-warps leave
  const int hh = (int)(w % nH);
  const long long row = w / nH;
  const int bb = (int)(row / Sp), ss = (int)(row % Sp);
  float acc = 0.f;
  if (ss < S) {
    const long long t = (long long)bb * S + ss;
    const uint4 a = *reinterpret_cast<const uint4*>(dout + t * ld_do + hh * kHd + lane * 8);
    const uint4 o = *reinterpret_cast<const uint4*>(out + t * ld_o + hh * kHd + lane * 8);
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, ow[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 x = unpack_bf16x2(aw[e]), y = unpack_bf16x2(ow[e]);
      acc += x.x * y.x + x.y * y.y;
    }
  }
  const unsigned mask = 0xffffu << (threadIdx.x & 16);
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) acc += __shfl_xor_sync(mask, acc, off);
  if (lane == 0) {
    const long long head = (long long)bb * nH + hh, idx = head * Sp + ss;
    ndelta[idx] = -acc;
    nlse2[idx] = ss < S ? -lse[head * S + ss] * kLog2e : 0.f;
  }
}
}  // namespace mfsdp

using namespace mfsdp;

// Bytes of K and V that a group of heads may occupy (half of the 126 MB L2, the rest is for Q, O and the other die).
constexpr long long kKvInL2 = 64LL << 20;
static int heads_in_l2(int B, int S, int nH) {
  const long long group = kKvInL2 / ((long long)S * kHd * 2 * 2), heads = (long long)B * nH;
  return (int)(group < 1 ? 1 : group > heads ? heads : group);
}

// One tile per block: its longest block takes 1.31 us per key tile; two: 1.9 us, for twice the queries (0.72 of the time
// where the chip is full).  So two tiles lose where the longest block sets the time: while the heads * (nt + 1) / 2 key
// tiles per query tile, spread over the SMs, leave most of them idle, the more so the longer the rows.  The line is
// measured (1 to 384 heads of 1 to 128 tiles; one / two tiles per block):
//   just below it: 2 heads of 128 tiles 170 / 239 us, 4 of 48 68 / 94, 8 of 24 45.7 / 49.9, 16 of 10 23.2 / 24.5
//   just above:    4 heads of 96 tiles 225 / 186 us, 6 of 48 109 / 98, 8 of 32 74.7 / 68.0, 16 of 12 29.0 / 27.8, 32 of 5 16.8 / 14.6
// Rows of a single tile have no second one to overlap (192 heads: 11.9 / 12.6).  What the line misses: 96 heads of 3 tiles,
// 17.4 / 20.2, whose two-tile blocks just begin a second wave.
static bool attn_fwd_two_tiles(int B, int S, int nH) {
  const long long nt = (S + kBq - 1) / kBq, heads = (long long)nH * B;
  return nt > 1 && nt * heads > 148 && heads * (nt + 1) > 185 + nt;
}

// qkv: [B*S, 3*nH*128] bf16 (row stride ld_qkv elements); out: [B*S, nH*128]; lse: [B, nH, S] fp32.
MFSDP_API int mfsdp_attention_fwd(const void* qkv, void* out, float* lse, int B, int S, int nH, long long ld_qkv,
                                  long long ld_out, float softmax_scale, int* status, cudaStream_t st) {
  if (B <= 0 || S <= 0 || nH <= 0 || (ld_qkv % 8) || (ld_out % 8)) return -2;
  ensure_context_on_this_thread();
  CUtensorMap map;
  int rc = make_tmap_bf16(&map, qkv, B, S, 3LL * nH * kHd, ld_qkv, 128, 64);
  if (rc) return rc;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(attn_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AttnFwdSmem::kBytes);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(attn_fwd2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AttnFwd2Smem::kBytes);
    if (e != cudaSuccess) return (int)e;
    attr = true;
  }
  AttnFwdArgs a{};
  a.B = B; a.S = S; a.nH = nH;
  a.scale_log2 = softmax_scale * kLog2e;
  a.out = (__nv_bfloat16*)out; a.ld_out = ld_out; a.lse = lse; a.status = status;
  if (attn_fwd_two_tiles(B, S, nH)) {
    const int nq = (S + 2 * kBq - 1) / (2 * kBq);
    return launch_pdl(attn_fwd2_kernel, dim3((unsigned)(nq * B * nH)), dim3(kFwd2Threads), AttnFwd2Smem::kBytes, st, map, a,
                      heads_in_l2(B, S, nH));
  }
  dim3 grid((S + kBq - 1) / kBq, nH, B);
  return launch_pdl(attn_fwd_kernel, grid, dim3(kAttnThreads), AttnFwdSmem::kBytes, st, map, a);
}

// dout, out: [B*S, nH*128] bf16; lse: [B, nH, S]; dqkv: [B*S, 3*nH*128] bf16 (written in full);
// scratch: 2 * B * nH * Sp floats, 16-byte aligned, Sp = S rounded up to 128.
MFSDP_API int mfsdp_attention_bwd(const void* dout, const void* qkv, const void* out, const float* lse, void* dqkv,
                                  float* scratch, int B, int S, int nH, long long ld_qkv, long long ld_o,
                                  long long ld_dqkv, float softmax_scale, int* status, cudaStream_t st) {
  if (B <= 0 || S <= 0 || nH <= 0 || (ld_qkv % 8) || (ld_o % 8) || (ld_dqkv % 8) || !scratch || ((uintptr_t)scratch & 15)) return -2;
  ensure_context_on_this_thread();
  CUtensorMap map_qkv, map_do;
  int rc = make_tmap_bf16(&map_qkv, qkv, B, S, 3LL * nH * kHd, ld_qkv, 128, 64);
  if (rc) return rc;
  rc = make_tmap_bf16(&map_do, dout, B, S, (long long)nH * kHd, ld_o, 128, 64);
  if (rc) return rc;
  // Rows of up to a few tiles consist of tiles on the diagonal and at the end, most of whose 32 x 32 parts do not count:
  // leaving those out takes 512 heads of 32 rows from 48.9 to 43.5 us, 256 of 64 30.9 to 28.6, 128 of 300 58.8 to 56.2, 48 of
  // 777 70.8 to 69.2.  From about 1024 rows on whole tiles prevail and lose by it (32 heads of 4096 rows 492 / 504 us).
  const auto kern = S < 1024 ? attn_bwd_kernel<true> : attn_bwd_kernel<false>;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(attn_bwd_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, AttnBwdSmem::kBytes);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(attn_bwd_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, AttnBwdSmem::kBytes);
    if (e != cudaSuccess) return (int)e;
    attr = true;
  }
  const int nt = (S + 127) / 128;
  AttnBwdArgs a{};
  a.B = B; a.S = S; a.nH = nH;
  a.Sp = (long long)nt * 128;
  float* nlse2 = scratch;
  float* ndelta = scratch + (long long)B * nH * a.Sp;
  rc = launch_pdl(attn_bwd_prep_kernel, dim3((unsigned)(((long long)B * nH * a.Sp + 15) / 16)), dim3(256), 0, st,
                  (const __nv_bfloat16*)dout, ld_o, (const __nv_bfloat16*)out, ld_o, lse, nlse2, ndelta, B, S, nH, (int)a.Sp);
  if (rc) return rc;
  a.scale = softmax_scale; a.scale_log2 = softmax_scale * kLog2e;
  a.nlse2 = nlse2; a.ndelta = ndelta;
  a.dqkv = (__nv_bfloat16*)dqkv; a.ld_dqkv = ld_dqkv; a.status = status;
  a.heads_per_group = heads_in_l2(B, S, nH);
  return launch_pdl(kern, dim3(2u * (unsigned)(nt * B * nH)), dim3(kBwdThreads), AttnBwdSmem::kBytes, st, map_qkv,
                    map_do, a);
}
