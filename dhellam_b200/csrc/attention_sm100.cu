// Flash attention forward and backward for sm_100a (head size 128, bf16, grouped KV heads,
// causal or full, strided [S, B, heads, d] operands so a packed QKV buffer needs no copies;
// packed batches of sequences of unequal length in one launch).
//
// What bounds it: per pair of 128-row tiles the tensor cores need 512 cycles per product (two
// forward, seven backward) and the 128 x 128 exponentials 1024 cycles of the special-function
// units, so the kernels are built to keep both busy at once:
//
// Forward, one CTA per two tiles of 128 query rows that share their keys (two query heads of a
// KV group; for groups of odd size two neighbouring row tiles of one head; one tile where that
// leaves no SM with two, fwd_mode):
//   warp 0      TMA producer: Q tiles once, then K_j / V_j through one 5-slot ring
//   warp 1      MMA issuer:   S_t = Q_t K_j^T, O_t += P_t V_j (t = 0, 1) with P read from TMEM
//   warps 4-7, 8-11  softmax of tile 0 / 1: one thread per row, no exchange between threads; P_t
//               overwrites S_t in TMEM as bf16; O_t stays in TMEM and is rescaled when the maximum
//               of one of the warp's rows has grown.  (Two tiles with P over S in TMEM and a rescaling
//               only when the maximum has grown by a factor are the scheme published as
//               FlashAttention-4.  The factor is left out: with it the largest probability of a row
//               is rounded to bf16 where it would be exactly 1.  Error of the output against 64
//               bits, factor 2^8 and without: 0.00201 and 0.00198 for scores of standard deviation
//               1, 0.00207 and 0.00177 for 3; 432 and 473 us on 16384 positions.)
//   While one tile is in softmax the tensor cores work on the other.
//   Measured, causal, 8 query heads on 2 KV heads: 32768 positions inside a training step (power-capped clocks) 3628 -> 2098 us,
//   16384 positions alone 866 -> 478 us (1.15 PFLOP/s);
//   tensor and special-function pipes each ~55 % busy, the rest is the chain softmax -> P V -> S of one tile (two softmax
//   warps per scheduler).  Tried and slower: steps of 64 keys with S double-buffered (an N = 64 product takes as long as an
//   N = 128 one: 2116 against 1550 cycles per tile pair); 1/8 to 1/2 of the exponentials as a polynomial on the FMA pipe
//   (4 to 20 % slower: the warps are bound by instruction latency, not by the special-function pipe).
//
// Backward is two kernels that share delta = rowsum(dO * O):
//   dK/dV: one CTA per (128 keys, batch, KV head) loops over the query heads of the group and
//     the query blocks that see these keys.  Scores are formed transposed (keys on TMEM lanes),
//     so P^T = exp2(S^T - lse) and dS^T = P^T (dP^T - delta) go back to TMEM as they stand and are
//     the A operands of dV += P^T dO and dK += dS^T Q: no shared-memory round trip, and the MMAs
//     read half the shared memory.  The math warps' P phase runs beside dK(i-1), dP(i) and the dS
//     phase beside dV(i), S(i+1), so nothing is double-buffered in TMEM.  When keys x batch x KV
//     heads gives too few CTAs (one KV head per GPU under tensor parallelism), the query heads
//     of a group are split over a power of two of CTAs that write fp32 partials (bwd_head_split);
//     attn_dkv_reduce_kernel adds them in a fixed order.
//   dQ: one CTA per (128 queries, batch, query head) loops over the key blocks, recomputes S
//     and dP and accumulates dQ += dS K in TMEM (dS again as a TMEM operand).  Recomputing two
//     products per tile pair replaces an fp32 atomic accumulation of dQ and keeps dQ reproducible.
//   Measured (32768 positions in the step): dK/dV 7833 -> 3844 us, dQ 5326 -> 2630 us; 16384 alone, both and delta 2856 -> 1455 us.  The forms before
//   ran one phase after the other and applied the mask as predicates (10 ALU instructions per score in dQ).
//
// MMAs are issued under a predicate by a warp whose control flow stays uniform (ptx.cuh, umma_bf16_by): issued inside
// `if (lane == 0)` a 128 x 128 x 16 product took 75-100 cycles to issue, against 64 to execute.
//
// Packed batches: the row offsets of the sequences and a list of (sequence, tile) in descending
// order of work travel as a kernel parameter; tiles are cut by the sequence's own length, and rows
// of the next sequence that a tile load brings in are zeroed where they enter a contraction (zero
// probability times a neighbour's NaN would be NaN).
//
// Role in the reference: the bundled flash-attention 2 sm80 kernels behind
// pymha_varlen_fwd / pymha_varlen_bwd (csrc/operators/flash_atten.cu:220-434, 479-757);
// its fp32 dq_accum and its separate GQA reduction pass (:637-652, 742-745) have no
// counterpart here.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <new>
#include <type_traits>
#include <vector>

#include "api.h"
#include "ptx.cuh"
#include "tmap.h"

namespace dh {
namespace attn {

constexpr int BQ = 128, BKV = 128, D = 128;
constexpr int HALF_BYTES = 128 * 128;        // one [128 rows][64 elems] swizzled box
constexpr int TILE_BYTES = 2 * HALF_BYTES;   // [128][128] bf16
constexpr int THREADS = 384;                 // warp 0 TMA, warp 1 MMA, warps 2-3 helpers, warps 4-11 math
constexpr int MATH_WARP0 = 4;
constexpr float LOG2E = 1.4426950408889634f;

// Sequences and tiles of one packed launch (a kernel parameter: no device table, nothing to copy or keep).
constexpr int MAX_SEQS = 128, MAX_TILES = 768;
constexpr int TILE_BITS = 24;                // tiles of 128 rows of a sequence of up to 2^31 rows
struct Packed {
  int q0[MAX_SEQS], k0[MAX_SEQS];            // first row in the packed tensors
  int nq[MAX_SEQS], nk[MAX_SEQS];            // rows
  int id[MAX_SEQS];                          // position in the batch (row of the statistics)
  uint32_t tile[MAX_TILES];                  // sequence << TILE_BITS | tile
};
struct Dense {};                             // equal lengths: everything follows from the block index

struct Geometry {
  int B, Hq, Hk;                             // batch dimension of the tensors (1 when packed)
  int Sq, Sk;                                // rows per sequence (dense only)
  int Tq, Tk;                                // rows of the tensors' sequence dimension
  int ls;                                    // row stride of the statistics [.., Hq, ls]
  int causal;
  float scale;
  int x0;                                    // first work item of this launch (SM budget: launches in waves)
  int heads;                                 // work items per tile and batch entry
  DeviceStatus* status;
};

// One tile's surroundings: sequence bounds and where its rows start.
struct Work {
  int b, head, tile, sid;                    // batch coordinate, head item, tile, row of the statistics
  int q0, k0, nq, nk;
};

// Heaviest tiles first over ALL heads and sequences: the tile index is the slowest part of the work item.
template <class Table>
__device__ __forceinline__ Work find_work(const Geometry& g, const Table& t, int item) {
  Work w;
  if constexpr (sizeof(Table) > 1) {
    w.head = item % g.heads;
    const uint32_t e = t.tile[item / g.heads];
    const int s = (int)(e >> TILE_BITS);
    w.tile = (int)(e & ((1u << TILE_BITS) - 1));
    w.b = 0;
    w.sid = t.id[s];
    w.q0 = t.q0[s]; w.k0 = t.k0[s]; w.nq = t.nq[s]; w.nk = t.nk[s];
  } else {
    const int per = g.heads * g.B;
    const int i = item % per;
    w.tile = item / per;
    w.head = i % g.heads;
    w.b = i / g.heads;
    w.sid = w.b;
    w.q0 = 0; w.k0 = 0; w.nq = g.Sq; w.nk = g.Sk;
  }
  return w;
}

// K-major operand descriptor for step kk (16 elements of the contraction) of a tile stored
// as two [128][64] swizzled boxes.
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t base, int kk) {
  return umma_smem_desc(base + (kk >> 2) * HALF_BYTES + (kk & 3) * 32, 16, 1024);
}
// MN-major operand descriptor: the contraction runs over the 128 rows of the tile.
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t base, int kk) {
  return umma_smem_desc(base + kk * 2048, HALF_BYTES, 1024);
}
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* m, uint64_t* bar, int head, int b, int row) {
  tma_load_4d(dst, m, bar, 0, head, b, row);
  tma_load_4d(dst + HALF_BYTES, m, bar, 64, head, b, row);
}
// Zeroes rows [first, 128) of a tile in shared memory (whole warp); a row is 128 bytes in each of the two boxes.
__device__ __forceinline__ void zero_tile_rows(uint8_t* tile, int first, int lane) {
  for (int h = 0; h < 2; ++h)
    for (int o = first * 128 + lane * 16; o < HALF_BYTES; o += 512) *reinterpret_cast<uint4*>(tile + h * HALF_BYTES + o) = make_uint4(0, 0, 0, 0);
  fence_proxy_async_smem();
  __syncwarp();
}

// ---- packed fp32 arithmetic: two lanes per instruction, same rounding as the scalar forms
__device__ __forceinline__ uint64_t pk2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void upk2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float ex2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Key j of the tile is visible to a row iff j < limit.
__device__ __forceinline__ int visible_keys(int nk, int causal, int off, int qi, int key0) {
  int limit = nk - key0;
  if (causal) limit = min(limit, qi + off - key0 + 1);
  return limit;
}

// ======================================================================= forward
constexpr int FWD_RING = 5;
struct FwdCtl {
  uint64_t q_full[2];
  uint64_t kv_full[FWD_RING], kv_empty[FWD_RING];
  uint64_t s_full[2], p_ready[2][2], o_done[2];   // [tile], p_ready [tile][half of the keys]
  uint32_t tmem_base;
  int abort_flag;
};
constexpr int FWD_SMEM = TILE_BYTES * (2 + FWD_RING) + 1024 + 512;

struct FwdArgs {
  __nv_bfloat16* out;
  float* lse;
  long long o_s, o_b, o_h;                   // output strides (elements)
  int mode;                                  // what a CTA's two tiles are:
};
enum { ROW_PAIR, HEAD_PAIR, SINGLE };        // row tiles 2i, 2i+1 of one head; query heads 2h, 2h+1; one tile only, the second is empty

// POSITIVE: the scale is; a form of its own for the others, whose masked keys need more than a score of -inf (as one
// kernel 3 % slower for everybody).
template <class Table, bool POSITIVE>
__global__ void __launch_bounds__(THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv,
                const __grid_constant__ Geometry g, const __grid_constant__ FwdArgs a, const __grid_constant__ Table table) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sKV = smem + 2 * TILE_BYTES;
  FwdCtl* ctl = reinterpret_cast<FwdCtl*>(smem + (2 + FWD_RING) * TILE_BYTES);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const Work w = find_work(g, table, g.x0 + (int)blockIdx.x);
  const int off = w.nk - w.nq;                     // key j visible to query i iff j <= i + off
  const int hq_[2] = {a.mode == HEAD_PAIR ? 2 * w.head : w.head, a.mode == HEAD_PAIR ? 2 * w.head + 1 : w.head};
  const int hk = hq_[0] / (g.Hq / g.Hk);
  // dense tiles are counted from the end: the latest queries see most keys
  const int per_cta = a.mode == ROW_PAIR ? 2 * BQ : BQ;
  const int last = (w.nq + per_cta - 1) / per_cta - 1;
  const int tile = sizeof(Table) > 1 ? w.tile : last - w.tile;
  const int qb_[2] = {a.mode == ROW_PAIR ? 2 * tile : tile,
                      a.mode == ROW_PAIR ? 2 * tile + 1 : (a.mode == HEAD_PAIR ? tile : (w.nq + BQ - 1) / BQ)};
  int nblk_[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    int n = (w.nk + BKV - 1) / BKV;
    if (g.causal) {
      const int last_key = min(qb_[t] * BQ + BQ, w.nq) - 1 + off;
      n = last_key < 0 ? 0 : min(n, last_key / BKV + 1);
    }
    nblk_[t] = qb_[t] * BQ < w.nq ? n : 0;
  }
  const int nmax = max(nblk_[0], nblk_[1]);

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&ctl->q_full[i], 1);
      mbar_init(&ctl->s_full[i], 1); mbar_init(&ctl->p_ready[i][0], 4); mbar_init(&ctl->p_ready[i][1], 4); mbar_init(&ctl->o_done[i], 1);
    }
    for (int i = 0; i < FWD_RING; ++i) { mbar_init(&ctl->kv_full[i], 1); mbar_init(&ctl->kv_empty[i], 1); }
    ctl->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(&ctl->tmem_base, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, ctl->tmem_base, 0);
  volatile int* abort_flag = &ctl->abort_flag;
  // TMEM columns: S_0 [0,128) S_1 [128,256), each overwritten by its bf16 P in the first 64; O_0 [256,384) O_1 [384,512)

  if (warp == 0) {
    if (lane == 0 && nmax > 0) {
      tma_prefetch_desc(&tq); tma_prefetch_desc(&tk); tma_prefetch_desc(&tv);
      int slot = 0;
      uint32_t ph = 1;
      for (int i = 0; i < 2 * nmax; ++i) {          // K_0 V_0 K_1 V_1 ...
        if (i < 2 && nblk_[i] > 0) {                // Q_0 goes before K_0, Q_1 before V_0
          mbar_expect_tx(&ctl->q_full[i], TILE_BYTES);
          load_tile(sQ + i * TILE_BYTES, &tq, &ctl->q_full[i], hq_[i], w.b, w.q0 + qb_[i] * BQ);
        }
        if (!mbar_wait(&ctl->kv_empty[slot], ph, abort_flag, g.status, 400)) break;
        mbar_expect_tx(&ctl->kv_full[slot], TILE_BYTES);
        load_tile(sKV + slot * TILE_BYTES, (i & 1) ? &tv : &tk, &ctl->kv_full[slot], hk, w.b, w.k0 + (i >> 1) * BKV);
        if (++slot == FWD_RING) { slot = 0; ph ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t leader = elect_one();
    if (nmax > 0) {
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, 0, 0);
      constexpr uint32_t idesc_pv = umma_idesc_bf16(128, 128, 0, 1);
      // load i of the ring (K of block j: 2 j, V: 2 j + 1)
      auto wait_load = [&](int i, int where) {
        const bool r = warp_wait(&ctl->kv_full[i % FWD_RING], (i / FWD_RING) & 1, abort_flag, g.status, where);
        tc_fence_after();
        return r;
      };
      auto issue_s = [&](int t, int j) {
        const uint32_t q_base = smem_u32(sQ + t * TILE_BYTES), k_base = smem_u32(sKV + (2 * j % FWD_RING) * TILE_BYTES);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) umma_bf16_by(leader, tmem + t * 128, desc_kmajor(q_base, kk), desc_kmajor(k_base, kk), idesc_s, kk > 0);
        umma_commit_by(leader, &ctl->s_full[t]);
      };
      bool ok = wait_load(0, 410);
      for (int t = 0; t < 2 && ok; ++t) {
        if (nblk_[t] == 0) continue;
        ok = warp_wait(&ctl->q_full[t], 0, abort_flag, g.status, 411);
        tc_fence_after();
        if (ok) issue_s(t, 0);
      }
      umma_commit_by(leader, &ctl->kv_empty[0]);
      for (int j = 0; j < nmax && ok; ++j) {
        uint8_t* vtile = sKV + ((2 * j + 1) % FWD_RING) * TILE_BYTES;
        if (!wait_load(2 * j + 1, 412)) { ok = false; break; }
        if (sizeof(Table) > 1 && (j + 1) * BKV > w.nk && w.k0 + w.nk < g.Tk) zero_tile_rows(vtile, w.nk - j * BKV, lane);
        const uint32_t v_base = smem_u32(vtile);
        bool have_k = false;
        for (int t = 0; t < 2 && ok; ++t) {
          if (j >= nblk_[t]) continue;
#pragma unroll
          for (int h = 0; h < 2; ++h) {              // the first half of P V runs beside the exponentials of the second
            if (!warp_wait(&ctl->p_ready[t][h], j & 1, abort_flag, g.status, 413)) ok = false;
            tc_fence_after();
            if (ok) {
#pragma unroll
              for (int kk = 4 * h; kk < 4 * h + 4; ++kk)
                umma_bf16_ts_by(leader, tmem + 256 + t * 128, tmem + t * 128 + kk * 8, desc_mnmajor(v_base, kk), idesc_pv, (j | kk) != 0);
            }
          }
          if (!ok) break;
          if (j + 1 < nblk_[t]) {
            if (!have_k && !wait_load(2 * j + 2, 414)) { ok = false; break; }
            have_k = true;
            issue_s(t, j + 1);                       // in order behind the P V that reads the same columns
          } else {
            umma_commit_by(leader, &ctl->o_done[t]);
          }
        }
        if (!ok) break;
        umma_commit_by(leader, &ctl->kv_empty[(2 * j + 1) % FWD_RING]);
        if (have_k) umma_commit_by(leader, &ctl->kv_empty[(2 * j + 2) % FWD_RING]);
      }
    }
    __syncwarp();
  } else if (warp >= MATH_WARP0) {
    const int t = (warp - MATH_WARP0) >> 2;
    const int quarter = warp & 3;
    const int qi = qb_[t] * BQ + quarter * 32 + lane;
    const bool row_ok = qi < w.nq;
    const int nblk = nblk_[t];
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t ts = tmem + t * 128 + lane_base, to = tmem + 256 + t * 128 + lane_base;
    const float sl2 = g.scale * LOG2E;
    const uint64_t sl2_2 = pk2(sl2, sl2);
    float m = -INFINITY;                             // reference maximum of the row (raw score)
    uint64_t l2 = pk2(0.f, 0.f);                     // row sum in two interleaved parts
    bool ok = nblk > 0;
    for (int j = 0; j < nblk && ok; ++j) {
      if (!warp_wait(&ctl->s_full[t], j & 1, abort_flag, g.status, 420)) { ok = false; break; }
      tc_fence_after();
      const int limit = visible_keys(w.nk, g.causal, off, qi, j * BKV);
      const bool full = __all_sync(0xffffffffu, limit >= BKV);
      uint32_t s[BKV];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(ts + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&s[c * 32]));
      tmem_ld_wait();
      if (!full) {
#pragma unroll
        for (int i = 0; i < BKV; ++i) if (i >= limit) s[i] = __float_as_uint(-INFINITY);
      }
      float mx[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) mx[c] = __uint_as_float(s[c]);
#pragma unroll
      for (int i = 4; i < BKV; i += 4) {
#pragma unroll
        for (int c = 0; c < 4; ++c) mx[c] = fmaxf(mx[c], __uint_as_float(s[i + c]));
      }
      const float bm = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      // every new maximum becomes the reference at once: the largest probability is then exactly 1 and loses nothing in bf16
      const bool grown = j > 0 && __any_sync(0xffffffffu, bm > m);
      float alpha = 1.f;
      if (grown) {
        // a reference of -inf (nothing seen yet) has zero sums: any factor will do, 0 is finite
        const float m_new = fmaxf(m, bm);
        alpha = m == -INFINITY ? 0.f : ex2((m - m_new) * sl2);
        m = m_new;
        l2 = mul2(l2, pk2(alpha, alpha));
      } else if (j == 0) {
        m = bm;
      }
      const float nm = m == -INFINITY ? 0.f : -m * sl2;
      uint64_t mul = sl2_2, add = pk2(nm, nm);
      if (!POSITIVE && !full) {
        // -inf times the scale is -inf only for a positive one: the exponents of masked keys are set here instead
#pragma unroll
        for (int i = 0; i < BKV; ++i) s[i] = __float_as_uint(i < limit ? fmaf(__uint_as_float(s[i]), sl2, nm) : -INFINITY);
        mul = pk2(1.f, 1.f);
        add = 0;
      }
      uint64_t rs[2] = {0, 0};                       // the block's own sum: short chains, then one add to the running sum
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int c = 4 * h; c < 4 * h + 4; ++c) {
          uint32_t p[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int e = c * 16 + 2 * i;
            float x, y;
            upk2(fma2(pk2(__uint_as_float(s[e]), __uint_as_float(s[e + 1])), mul, add), x, y);
            x = ex2(x); y = ex2(y);
            rs[i & 1] = add2(rs[i & 1], pk2(x, y));
            p[i] = pack_bf16x2(x, y);
          }
          tmem_st8(ts + c * 8, p);
        }
        if (h == 0 && grown) {
          // S_t(j) was issued behind P V of block j - 1, so O_t is complete up to that block, and the next P V waits for p_ready.
          // Here half of the scores' registers are free: 32 columns to a round trip (16384 positions, 8 heads on 2: 473 us; in
          // front of the exponentials, 16 to a round trip, 518; 432 if a growth below 2^8 is let pass)
#pragma unroll 1
          for (int c = 0; c < D; c += 32) {
            uint32_t o[2][16];
            tmem_ld16(to + c, o[0]);
            tmem_ld16(to + c + 16, o[1]);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i >> 4][i & 15] = __float_as_uint(__uint_as_float(o[i >> 4][i & 15]) * alpha);
            tmem_st16(to + c, o[0]);
            tmem_st16(to + c + 16, o[1]);
          }
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl->p_ready[t][h]);
      }
      l2 = add2(l2, add2(rs[0], rs[1]));
    }
    float l0, l1;
    upk2(l2, l0, l1);
    const float l = l0 + l1;
    __nv_bfloat16* orow = a.out + (long long)(w.q0 + qi) * a.o_s + (long long)w.b * a.o_b + (long long)hq_[t] * a.o_h;
    float* lrow = a.lse + ((long long)w.sid * g.Hq + hq_[t]) * g.ls + qi;
    if (nblk > 0) {
      if (ok && warp_wait(&ctl->o_done[t], 0, abort_flag, g.status, 422)) {
        tc_fence_after();
        const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t v[32];
          tmem_ld32(to + c * 32, v);
          tmem_ld_wait();
          if (row_ok) {
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {
              uint4 u;
              const int i0 = q4 * 8;
              u.x = pack_bf16x2(__uint_as_float(v[i0 + 0]) * inv, __uint_as_float(v[i0 + 1]) * inv);
              u.y = pack_bf16x2(__uint_as_float(v[i0 + 2]) * inv, __uint_as_float(v[i0 + 3]) * inv);
              u.z = pack_bf16x2(__uint_as_float(v[i0 + 4]) * inv, __uint_as_float(v[i0 + 5]) * inv);
              u.w = pack_bf16x2(__uint_as_float(v[i0 + 6]) * inv, __uint_as_float(v[i0 + 7]) * inv);
              reinterpret_cast<uint4*>(orow + c * 32)[q4] = u;
            }
          }
        }
        if (row_ok) *lrow = l > 0.f ? m * g.scale + logf(l) : -INFINITY;
      }
    } else if (row_ok) {
      for (int i = 0; i < D / 8; ++i) reinterpret_cast<uint4*>(orow)[i] = make_uint4(0, 0, 0, 0);
      *lrow = -INFINITY;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// ======================================================================= backward
// delta[b, h, s] = sum_d dO * O.  Half a warp per row (16 bytes per lane and operand), four rows
// per half warp in flight; one block covers 64 consecutive rows of one head, so the results are
// written as whole lines.
__global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ out,
                                                         float* __restrict__ delta, int Hq, int S, long long do_s, long long do_b,
                                                         long long do_h, long long o_s, long long o_b, long long o_h, int wide) {
  const int hw = threadIdx.x >> 4, l16 = threadIdx.x & 15;
  const int h = blockIdx.x % Hq, b = blockIdx.y;
  const int s0 = (blockIdx.x / Hq) * 64 + hw * 4;
  uint4 x[4], y[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int s = min(s0 + i, S - 1);
    x[i] = ld_nc_v4(dout + s * do_s + b * do_b + h * do_h + l16 * 8);
    const __nv_bfloat16* o = out + s * o_s + b * o_b + h * o_h + l16 * 8;
    if (wide) {
      y[i] = ld_nc_v4(o);
    } else {                              // O with rows that are only 8-byte aligned
      const uint2 u = reinterpret_cast<const uint2*>(o)[0], v = reinterpret_cast<const uint2*>(o)[1];
      y[i] = make_uint4(u.x, u.y, v.x, v.y);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float v = 0.f;
    const uint32_t xs[4] = {x[i].x, x[i].y, x[i].z, x[i].w}, ys[4] = {y[i].x, y[i].y, y[i].z, y[i].w};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float2 p = unpack_bf16x2(xs[c]), q = unpack_bf16x2(ys[c]);
      v += p.x * q.x + p.y * q.y;
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (l16 == 0 && s0 + i < S) delta[((long long)b * Hq + h) * S + s0 + i] = v;
  }
}

// ----------------------------------------------------------------------- dK / dV
constexpr int STAT_RING = 4;
struct DkvCtl {
  uint64_t k_full, v_full;
  uint64_t q_full[2], q_empty[2], do_full[2], do_empty[2];
  uint64_t stat_full[STAT_RING], stat_empty[STAT_RING];
  uint64_t s_full, p_ready[2], dp_full, ds_ready[2], acc_full;      // [half of the query columns]
  uint32_t tmem_base;
  int abort_flag;
};
constexpr int STAT_BYTES = STAT_RING * 2 * BQ * 4;                    // -lse * log2(e) and -delta of the query block
constexpr int DKV_SMEM = TILE_BYTES * 6 + STAT_BYTES + 1024 + 512;    // K, V, Q x2, dO x2

struct DkvArgs {
  const float* lse;
  const float* delta;
  __nv_bfloat16* dk;
  __nv_bfloat16* dv;
  long long dk_s, dk_b, dk_h, dv_s, dv_b, dv_h;
  // Head split: the query heads of one KV head are divided over `hs` CTAs (work heads = Hk * hs) when
  // KV blocks x batch x KV heads alone would leave SMs idle (tensor parallelism leaves one KV head per
  // GPU).  Each CTA then writes fp32 partial dV / dK to `part` ([2][hs][Tk][B][Hk][128]) and
  // attn_dkv_reduce_kernel adds them up.
  int hs;
  float* part;
};

// Columns 32 c .. 32 c + 31 of this thread's accumulator rows of dV and dK -> memory.
__device__ __forceinline__ void store_dkv_cols(const DkvArgs& a, float scale, const uint32_t (&x)[32], const uint32_t (&y)[32], float* pdv, float* pdk,
                                               __nv_bfloat16* dvr, __nv_bfloat16* dkr) {
  if (a.hs > 1) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      reinterpret_cast<float4*>(pdv)[j] = make_float4(__uint_as_float(x[4 * j]), __uint_as_float(x[4 * j + 1]), __uint_as_float(x[4 * j + 2]),
                                                      __uint_as_float(x[4 * j + 3]));
      reinterpret_cast<float4*>(pdk)[j] = make_float4(__uint_as_float(y[4 * j]) * scale, __uint_as_float(y[4 * j + 1]) * scale,
                                                      __uint_as_float(y[4 * j + 2]) * scale, __uint_as_float(y[4 * j + 3]) * scale);
    }
    return;
  }
#pragma unroll
  for (int q4 = 0; q4 < 4; ++q4) {
    uint4 u, w;
    const int i0 = q4 * 8;
    u.x = pack_bf16x2(__uint_as_float(x[i0]), __uint_as_float(x[i0 + 1]));
    u.y = pack_bf16x2(__uint_as_float(x[i0 + 2]), __uint_as_float(x[i0 + 3]));
    u.z = pack_bf16x2(__uint_as_float(x[i0 + 4]), __uint_as_float(x[i0 + 5]));
    u.w = pack_bf16x2(__uint_as_float(x[i0 + 6]), __uint_as_float(x[i0 + 7]));
    w.x = pack_bf16x2(__uint_as_float(y[i0]) * scale, __uint_as_float(y[i0 + 1]) * scale);
    w.y = pack_bf16x2(__uint_as_float(y[i0 + 2]) * scale, __uint_as_float(y[i0 + 3]) * scale);
    w.z = pack_bf16x2(__uint_as_float(y[i0 + 4]) * scale, __uint_as_float(y[i0 + 5]) * scale);
    w.w = pack_bf16x2(__uint_as_float(y[i0 + 6]) * scale, __uint_as_float(y[i0 + 7]) * scale);
    reinterpret_cast<uint4*>(dvr)[q4] = u;
    reinterpret_cast<uint4*>(dkr)[q4] = w;
  }
}

template <class Table>
__global__ void __launch_bounds__(THREADS, 1)
attn_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv,
                    const __grid_constant__ CUtensorMap tdo, const __grid_constant__ Geometry g, const __grid_constant__ DkvArgs a,
                    const __grid_constant__ Table table) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = smem + TILE_BYTES;
  uint8_t* sQ = smem + 2 * TILE_BYTES;
  uint8_t* sDO = smem + 4 * TILE_BYTES;
  float* sStat = reinterpret_cast<float*>(smem + 6 * TILE_BYTES);   // [STAT_RING][2][BQ]
  DkvCtl* ctl = reinterpret_cast<DkvCtl*>(smem + 6 * TILE_BYTES + STAT_BYTES);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const Work w = find_work(g, table, g.x0 + (int)blockIdx.x);
  const int kb = w.tile, hk = w.head / a.hs, hpart = w.head % a.hs;
  const int group = g.Hq / g.Hk;
  const int gpp = group / a.hs;                 // query heads handled by this CTA
  const int hq0 = hk * group + hpart * gpp;
  const int off = w.nk - w.nq;
  const int nqb = (w.nq + BQ - 1) / BQ;
  // first query block that sees any key of this block: i + off >= kb*BKV
  int qb0 = 0;
  if (g.causal) {
    const int first_q = kb * BKV - off;
    qb0 = first_q <= 0 ? 0 : first_q / BQ;
  }
  const int n_iter = qb0 < nqb ? (nqb - qb0) * gpp : 0;

  if (threadIdx.x == 0) {
    mbar_init(&ctl->k_full, 1); mbar_init(&ctl->v_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&ctl->q_full[i], 1); mbar_init(&ctl->q_empty[i], 1);
      mbar_init(&ctl->do_full[i], 1); mbar_init(&ctl->do_empty[i], 1);
    }
    for (int i = 0; i < STAT_RING; ++i) { mbar_init(&ctl->stat_full[i], 1); mbar_init(&ctl->stat_empty[i], 8); }
    mbar_init(&ctl->s_full, 1); mbar_init(&ctl->dp_full, 1); mbar_init(&ctl->acc_full, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&ctl->p_ready[i], 8); mbar_init(&ctl->ds_ready[i], 8); }
    ctl->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(&ctl->tmem_base, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, ctl->tmem_base, 0);
  volatile int* abort_flag = &ctl->abort_flag;
  // TMEM columns: [0,128) S^T, [128,256) dP^T, [256,384) dV, [384,512) dK.  A math warp covers 64 of the 128 query
  // columns and packs its bf16 P^T (dS^T) into the first 32 of the 64 columns it has read.

  if (warp == 0) {
    if (lane == 0 && n_iter > 0) {
      tma_prefetch_desc(&tq); tma_prefetch_desc(&tk); tma_prefetch_desc(&tv); tma_prefetch_desc(&tdo);
      mbar_expect_tx(&ctl->k_full, TILE_BYTES);
      load_tile(sK, &tk, &ctl->k_full, hk, w.b, w.k0 + kb * BKV);
      int hq = hq0, row = w.q0 + qb0 * BQ;
      for (int it = 0; it < n_iter; ++it) {
        const int st = it & 1;
        const uint32_t ph = ((it >> 1) & 1) ^ 1;
        if (!mbar_wait(&ctl->q_empty[st], ph, abort_flag, g.status, 500)) break;
        mbar_expect_tx(&ctl->q_full[st], TILE_BYTES);
        load_tile(sQ + st * TILE_BYTES, &tq, &ctl->q_full[st], hq, w.b, row);
        if (it == 0) {
          mbar_expect_tx(&ctl->v_full, TILE_BYTES);
          load_tile(sV, &tv, &ctl->v_full, hk, w.b, w.k0 + kb * BKV);
        }
        if (!mbar_wait(&ctl->do_empty[st], ph, abort_flag, g.status, 501)) break;
        mbar_expect_tx(&ctl->do_full[st], TILE_BYTES);
        load_tile(sDO + st * TILE_BYTES, &tdo, &ctl->do_full[st], hq, w.b, row);
        if (++hq == hq0 + gpp) { hq = hq0; row += BQ; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t leader = elect_one();
    if (n_iter > 0) {
      constexpr uint32_t id_st = umma_idesc_bf16(128, 128, 0, 0);    // S^T, dP^T: A = K / V, B = Q / dO, both K-major
      constexpr uint32_t id_acc = umma_idesc_bf16(128, 128, 0, 1);   // dV, dK: A = P^T / dS^T in TMEM, B = dO / Q MN-major
      const uint32_t k_base = smem_u32(sK), v_base = smem_u32(sV);
      // scores of iteration j: A = K (V), B = the query block of Q (dO)
      auto issue_scores = [&](int j, bool dp) -> bool {
        const int st = j & 1;
        if (!warp_wait(dp ? &ctl->do_full[st] : &ctl->q_full[st], (j >> 1) & 1, abort_flag, g.status, dp ? 512 : 511)) return false;
        uint8_t* tile = (dp ? sDO : sQ) + st * TILE_BYTES;
        if (sizeof(Table) > 1 && w.q0 + w.nq < g.Tq) {
          const int rows = w.nq - (qb0 + j / gpp) * BQ;
          if (rows < BQ) zero_tile_rows(tile, rows, lane);
        }
        tc_fence_after();
        {
          const uint32_t b_base = smem_u32(tile), a_base = dp ? v_base : k_base, d = tmem + (dp ? 128 : 0);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) umma_bf16_by(leader, d, desc_kmajor(a_base, kk), desc_kmajor(b_base, kk), id_st, kk > 0);
          umma_commit_by(leader, dp ? &ctl->dp_full : &ctl->s_full);
        }
        return true;
      };
      // gradient of iteration j: dV += P^T dO (dK += dS^T Q).  Each math warp delivers its 64 query columns in two parts
      // of 32, so the products of the first parts run beside the math of the second.
      auto issue_grad = [&](int j, bool dk) -> bool {
        const uint32_t b_base = smem_u32((dk ? sQ : sDO) + (j & 1) * TILE_BYTES), src = tmem + (dk ? 128 : 0), d = tmem + (dk ? 384 : 256);
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          if (!warp_wait(dk ? &ctl->ds_ready[part] : &ctl->p_ready[part], j & 1, abort_flag, g.status, dk ? 514 : 513)) return false;
          tc_fence_after();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int half = i >> 1, kk = 4 * half + 2 * part + (i & 1);        // step kk of the contraction = 8 TMEM columns
            umma_bf16_ts_by(leader, d, src + half * 64 + (kk & 3) * 8, desc_mnmajor(b_base, kk), id_acc, (j | part | i) != 0);
          }
        }
        umma_commit_by(leader, dk ? &ctl->q_empty[j & 1] : &ctl->do_empty[j & 1]);
        return true;
      };
      bool ok = warp_wait(&ctl->k_full, 0, abort_flag, g.status, 510) && issue_scores(0, false) &&
                warp_wait(&ctl->v_full, 0, abort_flag, g.status, 510) && issue_scores(0, true);
      for (int it = 0; it < n_iter && ok; ++it) {
        // a score product goes in order behind the gradient product that reads the same TMEM columns
        ok = issue_grad(it, false) && (it + 1 >= n_iter || issue_scores(it + 1, false)) && issue_grad(it, true) &&
             (it + 1 >= n_iter || issue_scores(it + 1, true));
      }
      if (ok) umma_commit_by(leader, &ctl->acc_full);
    }
    __syncwarp();
  } else if (warp == 2) {
    // statistics of the query blocks, ahead of the math warps.  Rows past the end get -inf: exp2(x - inf) = 0.
    int hq = hq0, q0 = qb0 * BQ;
    for (int it = 0; it < n_iter; ++it) {
      const int st = it % STAT_RING;
      const uint32_t ph = ((it / STAT_RING) & 1) ^ 1;
      const float* lp = a.lse + ((long long)w.sid * g.Hq + hq) * g.ls;
      const float* dp = a.delta + ((long long)w.b * g.Hq + hq) * g.Tq + w.q0;
      float L[4], dl[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int q = q0 + i * 32 + lane;
        L[i] = q < w.nq ? -lp[q] * LOG2E : -INFINITY;
        dl[i] = q < w.nq ? -dp[q] : 0.f;
      }
      if (!warp_wait(&ctl->stat_empty[st], ph, abort_flag, g.status, 515)) break;
      float* dst = sStat + st * 2 * BQ;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        dst[i * 32 + lane] = L[i];
        dst[BQ + i * 32 + lane] = dl[i];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->stat_full[st]);
      if (++hq == hq0 + gpp) { hq = hq0; q0 += BQ; }
    }
  } else if (warp >= MATH_WARP0) {
    const int quarter = warp & 3;
    const int half = (warp - MATH_WARP0) >> 2;         // query columns [64 half, 64 half + 64)
    const int kj = kb * BKV + quarter * 32 + lane;     // this thread's key
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t ts = tmem + lane_base + half * 64, tp = ts + 128;
    const float sl2 = g.scale * LOG2E;
    const uint64_t sl2_2 = pk2(sl2, sl2);
    bool ok = n_iter > 0;
    int qb = qb0, head = 0;                            // iterations walk the heads of a query block, then the next block
    for (int it = 0; it < n_iter && ok; ++it) {
      const int sst = it % STAT_RING;
      const uint64_t* nL = reinterpret_cast<const uint64_t*>(sStat + sst * 2 * BQ + half * 64);
      const uint64_t* nD = nL + BQ / 2;
      // query column c of this warp is valid iff lo <= c < hi
      const int qbase = qb * BQ + half * 64;
      const bool edge = (qb + 1) * BQ > w.nq || (kb + 1) * BKV > w.nk || (g.causal && kb * BKV + BKV - 1 > qb * BQ + off);
      const int lo = kj >= w.nk ? BQ : (g.causal ? kj - off - qbase : 0);
      const int hi = w.nq - qbase;
      if (!warp_wait(&ctl->stat_full[sst], (it / STAT_RING) & 1, abort_flag, g.status, 520)) { ok = false; break; }
      if (!warp_wait(&ctl->s_full, it & 1, abort_flag, g.status, 521)) { ok = false; break; }
      tc_fence_after();
      // the mask is a path of its own: as predicates it costs more issue slots than the arithmetic
      uint64_t p[32];
      auto probabilities = [&](auto edge_) {
        constexpr bool masked = decltype(edge_)::value;
        uint32_t s[64];
        tmem_ld32(ts, *reinterpret_cast<uint32_t(*)[32]>(&s[0]));
        tmem_ld32(ts + 32, *reinterpret_cast<uint32_t(*)[32]>(&s[32]));
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            const ulonglong2 L = *reinterpret_cast<const ulonglong2*>(nL + c * 16 + i);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int e = c * 32 + 2 * (i + h);
              float x, y;
              upk2(fma2(pk2(__uint_as_float(s[e]), __uint_as_float(s[e + 1])), sl2_2, h ? L.y : L.x), x, y);
              x = ex2(x); y = ex2(y);
              if (masked) {                            // also rows without statistics (lse = -inf) and neighbours' rows
                if (e < lo || e >= hi) x = 0.f;
                if (e + 1 < lo || e + 1 >= hi) y = 0.f;
              }
              p[c * 16 + i + h] = pk2(x, y);
              pk[i + h] = pack_bf16x2(x, y);
            }
          }
          tmem_st16(ts + c * 16, pk);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->p_ready[c]);
        }
      };
      if (edge) probabilities(std::true_type{});
      else probabilities(std::false_type{});
      if (!warp_wait(&ctl->dp_full, it & 1, abort_flag, g.status, 522)) { ok = false; break; }
      tc_fence_after();
      {
        uint32_t v[64];
        tmem_ld32(tp, *reinterpret_cast<uint32_t(*)[32]>(&v[0]));
        tmem_ld32(tp + 32, *reinterpret_cast<uint32_t(*)[32]>(&v[32]));
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            const ulonglong2 dl = *reinterpret_cast<const ulonglong2*>(nD + c * 16 + i);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int e = c * 32 + 2 * (i + h);
              float x, y;
              upk2(mul2(p[c * 16 + i + h], add2(pk2(__uint_as_float(v[e]), __uint_as_float(v[e + 1])), h ? dl.y : dl.x)), x, y);
              pk[i + h] = pack_bf16x2(x, y);
            }
          }
          tmem_st16(tp + c * 16, pk);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(&ctl->ds_ready[c]);
            if (c == 1) mbar_arrive(&ctl->stat_empty[sst]);
          }
        }
      }
      if (++head == gpp) { head = 0; ++qb; }
    }
    // epilogue: this thread's key row of dV and of dK (times scale), columns [64 half, 64 half + 64)
    const long long part_elems = (long long)g.Tk * g.B * g.Hk * D;
    const long long krow = w.k0 + kj;
    float* pdv = a.hs > 1 ? a.part + (long long)hpart * part_elems + ((krow * g.B + w.b) * g.Hk + hk) * D + half * 64 : nullptr;
    float* pdk = a.hs > 1 ? pdv + (long long)a.hs * part_elems : nullptr;
    __nv_bfloat16* dvr = a.dv + krow * a.dv_s + (long long)w.b * a.dv_b + (long long)hk * a.dv_h + half * 64;
    __nv_bfloat16* dkr = a.dk + krow * a.dk_s + (long long)w.b * a.dk_b + (long long)hk * a.dk_h + half * 64;
    if (n_iter > 0) {
      if (ok && warp_wait(&ctl->acc_full, 0, abort_flag, g.status, 523)) {
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          uint32_t x[32], y[32];
          tmem_ld32(tmem + 256 + lane_base + half * 64 + c * 32, x);      // warp-collective: no per-lane branch around it
          tmem_ld32(tmem + 384 + lane_base + half * 64 + c * 32, y);
          tmem_ld_wait();
          if (kj < w.nk) store_dkv_cols(a, g.scale, x, y, pdv + c * 32, pdk + c * 32, dvr + c * 32, dkr + c * 32);
        }
      }
    } else if (kj < w.nk) {
      // no query sees these keys: zero gradients
      uint32_t z[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) z[i] = 0;
      for (int c = 0; c < 2; ++c) store_dkv_cols(a, g.scale, z, z, pdv + c * 32, pdk + c * 32, dvr + c * 32, dkr + c * 32);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// Sums the `hs` fp32 partials of a head-split backward and writes bf16 dK / dV.
// One thread per 8 consecutive head-dim elements of one (key, batch, KV head) row of dV and of dK.
__global__ void __launch_bounds__(256) attn_dkv_reduce_kernel(const float* __restrict__ part, int hs, __nv_bfloat16* __restrict__ dk,
                                                              __nv_bfloat16* __restrict__ dv, int Sk, int B, int Hk, long long dk_s,
                                                              long long dk_b, long long dk_h, long long dv_s, long long dv_b,
                                                              long long dv_h) {
  const long long nvec = (long long)Sk * B * Hk * (D / 8);
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 2 * nvec) return;
  const int which = i >= nvec;                  // 0: dV, 1: dK
  const long long v = which ? i - nvec : i;
  const int c8 = (int)(v % (D / 8));
  const long long row = v / (D / 8);            // (kj * B + b) * Hk + hk
  const int hk = (int)(row % Hk), b = (int)((row / Hk) % B);
  const long long kj = row / ((long long)Hk * B);
  const long long part_elems = (long long)Sk * B * Hk * D;
  const float* src = part + (long long)which * hs * part_elems + row * D + c8 * 8;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int h = 0; h < hs; ++h) {
    const float4 x = *reinterpret_cast<const float4*>(src + (long long)h * part_elems);
    const float4 y = *reinterpret_cast<const float4*>(src + (long long)h * part_elems + 4);
    acc[0] += x.x; acc[1] += x.y; acc[2] += x.z; acc[3] += x.w;
    acc[4] += y.x; acc[5] += y.y; acc[6] += y.z; acc[7] += y.w;
  }
  __nv_bfloat16* dst = which ? dk + kj * dk_s + b * dk_b + hk * dk_h : dv + kj * dv_s + b * dv_b + hk * dv_h;
  reinterpret_cast<uint4*>(dst)[c8] = make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]),
                                                 pack_bf16x2(acc[6], acc[7]));
}

// ----------------------------------------------------------------------- dQ
constexpr int DQ_KRING = 3, DQ_VRING = 2;
struct DqCtl {
  uint64_t q_full, do_full;
  uint64_t k_full[DQ_KRING], k_empty[DQ_KRING], v_full[DQ_VRING], v_empty[DQ_VRING];
  uint64_t s_full[2], dp_full, ds_ready, dq_full;
  uint32_t tmem_base;
  int abort_flag;
};
constexpr int DQ_SMEM = TILE_BYTES * (2 + DQ_KRING + DQ_VRING) + 1024 + 512;    // Q, dO, K x3, V x2

struct DqArgs {
  const float* lse;
  const float* delta;
  __nv_bfloat16* dq;
  long long dq_s, dq_b, dq_h;
};

template <class Table>
__global__ void __launch_bounds__(THREADS, 1)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv,
                   const __grid_constant__ CUtensorMap tdo, const __grid_constant__ Geometry g, const __grid_constant__ DqArgs a,
                   const __grid_constant__ Table table) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sDO = smem + TILE_BYTES;
  uint8_t* sK = smem + 2 * TILE_BYTES;
  uint8_t* sV = smem + (2 + DQ_KRING) * TILE_BYTES;
  DqCtl* ctl = reinterpret_cast<DqCtl*>(smem + (2 + DQ_KRING + DQ_VRING) * TILE_BYTES);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const Work w = find_work(g, table, g.x0 + (int)blockIdx.x);
  const int hq = w.head, hk = hq / (g.Hq / g.Hk);
  const int qb = sizeof(Table) > 1 ? w.tile : (w.nq + BQ - 1) / BQ - 1 - w.tile;      // dense: latest queries first
  const int off = w.nk - w.nq;
  int nblk = (w.nk + BKV - 1) / BKV;
  if (g.causal) {
    const int last_key = min(qb * BQ + BQ, w.nq) - 1 + off;
    nblk = last_key < 0 ? 0 : min(nblk, last_key / BKV + 1);
  }

  if (threadIdx.x == 0) {
    mbar_init(&ctl->q_full, 1); mbar_init(&ctl->do_full, 1);
    for (int i = 0; i < DQ_KRING; ++i) { mbar_init(&ctl->k_full[i], 1); mbar_init(&ctl->k_empty[i], 1); }
    for (int i = 0; i < DQ_VRING; ++i) { mbar_init(&ctl->v_full[i], 1); mbar_init(&ctl->v_empty[i], 1); }
    mbar_init(&ctl->s_full[0], 1); mbar_init(&ctl->s_full[1], 1);
    mbar_init(&ctl->dp_full, 1); mbar_init(&ctl->ds_ready, 8); mbar_init(&ctl->dq_full, 1);
    ctl->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(&ctl->tmem_base, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, ctl->tmem_base, 0);
  volatile int* abort_flag = &ctl->abort_flag;
  // TMEM columns: S [0,128) and [128,256) in turn, dP [256,384) overwritten by its bf16 dS, dQ [384,512)

  if (warp == 0) {
    if (lane == 0 && nblk > 0) {
      tma_prefetch_desc(&tq); tma_prefetch_desc(&tk); tma_prefetch_desc(&tv); tma_prefetch_desc(&tdo);
      mbar_expect_tx(&ctl->q_full, TILE_BYTES);
      load_tile(sQ, &tq, &ctl->q_full, hq, w.b, w.q0 + qb * BQ);
      int ks = 0, vs = 0;
      uint32_t kph = 1, vph = 1;
      for (int j = 0; j < nblk; ++j) {
        if (!mbar_wait(&ctl->k_empty[ks], kph, abort_flag, g.status, 800)) break;
        mbar_expect_tx(&ctl->k_full[ks], TILE_BYTES);
        load_tile(sK + ks * TILE_BYTES, &tk, &ctl->k_full[ks], hk, w.b, w.k0 + j * BKV);
        if (j == 0) {
          mbar_expect_tx(&ctl->do_full, TILE_BYTES);
          load_tile(sDO, &tdo, &ctl->do_full, hq, w.b, w.q0 + qb * BQ);
        }
        if (!mbar_wait(&ctl->v_empty[vs], vph, abort_flag, g.status, 801)) break;
        mbar_expect_tx(&ctl->v_full[vs], TILE_BYTES);
        load_tile(sV + vs * TILE_BYTES, &tv, &ctl->v_full[vs], hk, w.b, w.k0 + j * BKV);
        if (++ks == DQ_KRING) { ks = 0; kph ^= 1; }
        if (++vs == DQ_VRING) { vs = 0; vph ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t leader = elect_one();
    if (nblk > 0) {
      constexpr uint32_t id_kk = umma_idesc_bf16(128, 128, 0, 0);   // S, dP
      constexpr uint32_t id_km = umma_idesc_bf16(128, 128, 0, 1);   // dQ: A = dS in TMEM, B = K MN-major
      const uint32_t q_base = smem_u32(sQ), do_base = smem_u32(sDO);
      int kslot = 0, vslot = 0;                        // ring slots of the NEXT K (S product) and V (dP product)
      uint32_t kph = 0, vph = 0;
      auto issue_s = [&](int j) -> bool {
        if (!warp_wait(&ctl->k_full[kslot], kph, abort_flag, g.status, 811)) return false;
        tc_fence_after();
        {
          const uint32_t k_base = smem_u32(sK + kslot * TILE_BYTES);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) umma_bf16_by(leader, tmem + (j & 1) * 128, desc_kmajor(q_base, kk), desc_kmajor(k_base, kk), id_kk, kk > 0);
          umma_commit_by(leader, &ctl->s_full[j & 1]);
        }
        if (++kslot == DQ_KRING) { kslot = 0; kph ^= 1; }
        return true;
      };
      auto issue_dp = [&]() -> bool {
        if (!warp_wait(&ctl->v_full[vslot], vph, abort_flag, g.status, 812)) return false;
        tc_fence_after();
        {
          const uint32_t v_base = smem_u32(sV + vslot * TILE_BYTES);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) umma_bf16_by(leader, tmem + 256, desc_kmajor(do_base, kk), desc_kmajor(v_base, kk), id_kk, kk > 0);
          umma_commit_by(leader, &ctl->dp_full);
          umma_commit_by(leader, &ctl->v_empty[vslot]);
        }
        if (++vslot == DQ_VRING) { vslot = 0; vph ^= 1; }
        return true;
      };
      bool ok = warp_wait(&ctl->q_full, 0, abort_flag, g.status, 810) && issue_s(0) &&
                warp_wait(&ctl->do_full, 0, abort_flag, g.status, 810) && issue_dp();
      int dslot = 0;                                   // ring slot of K_j for the dQ product
      for (int j = 0; j < nblk && ok; ++j) {
        // the other S buffer was read before dS(j-1) was announced
        if (j + 1 < nblk && !issue_s(j + 1)) { ok = false; break; }
        if (!warp_wait(&ctl->ds_ready, j & 1, abort_flag, g.status, 813)) { ok = false; break; }
        if (sizeof(Table) > 1 && (j + 1) * BKV > w.nk && w.k0 + w.nk < g.Tk) zero_tile_rows(sK + dslot * TILE_BYTES, w.nk - j * BKV, lane);
        tc_fence_after();
        {
          const uint32_t k_base = smem_u32(sK + dslot * TILE_BYTES);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            umma_bf16_ts_by(leader, tmem + 384, tmem + 256 + (kk >> 2) * 64 + (kk & 3) * 8, desc_mnmajor(k_base, kk), id_km, (j | kk) != 0);
          umma_commit_by(leader, &ctl->k_empty[dslot]);
        }
        if (++dslot == DQ_KRING) dslot = 0;
        if (j + 1 < nblk && !issue_dp()) { ok = false; break; }     // in order behind the product that reads dS
      }
      if (ok) umma_commit_by(leader, &ctl->dq_full);
    }
    __syncwarp();
  } else if (warp >= MATH_WARP0) {
    const int quarter = warp & 3;
    const int half = (warp - MATH_WARP0) >> 2;         // key columns [64 half, 64 half + 64)
    const int qi = qb * BQ + quarter * 32 + lane;
    const bool row_ok = qi < w.nq;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t ts = tmem + lane_base + half * 64, tp = ts + 256;
    const float sl2 = g.scale * LOG2E;
    const uint64_t sl2_2 = pk2(sl2, sl2);
    const float nL = row_ok ? -a.lse[((long long)w.sid * g.Hq + hq) * g.ls + qi] * LOG2E : -INFINITY;
    const float nD = row_ok ? -a.delta[((long long)w.b * g.Hq + hq) * g.Tq + w.q0 + qi] : 0.f;
    const uint64_t nL2 = pk2(nL, nL), nD2 = pk2(nD, nD);
    bool ok = nblk > 0;
    for (int j = 0; j < nblk && ok; ++j) {
      int limit = visible_keys(w.nk, g.causal, off, qi, j * BKV + half * 64);
      if (!row_ok) limit = 0;
      const bool full = __all_sync(0xffffffffu, limit >= 64);
      if (!warp_wait(&ctl->s_full[j & 1], (j >> 1) & 1, abort_flag, g.status, 820)) { ok = false; break; }
      tc_fence_after();
      auto gradients = [&](auto edge_) -> bool {       // as in the dK/dV kernel, the mask is a path of its own
        constexpr bool masked = decltype(edge_)::value;
        uint64_t p[32];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t s[32];
          tmem_ld32(ts + (j & 1) * 128 + c * 32, s);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float x, y;
            upk2(fma2(pk2(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1])), sl2_2, nL2), x, y);
            p[c * 16 + i] = pk2(ex2(x), ex2(y));
          }
        }
        if (!warp_wait(&ctl->dp_full, j & 1, abort_flag, g.status, 821)) return false;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t v[32];
          tmem_ld32(tp + c * 32, v);
          tmem_ld_wait();
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            float x, y;
            upk2(mul2(p[c * 16 + i], add2(pk2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), nD2)), x, y);
            if (masked) {                              // whatever a masked key or a neighbour's row has left in S or dP
              if (c * 32 + 2 * i >= limit) x = 0.f;
              if (c * 32 + 2 * i + 1 >= limit) y = 0.f;
            }
            pk[i] = pack_bf16x2(x, y);
          }
          tmem_st16(tp + c * 16, pk);
        }
        return true;
      };
      ok = full ? gradients(std::false_type{}) : gradients(std::true_type{});
      if (!ok) break;
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->ds_ready);
    }
    __nv_bfloat16* dqr = a.dq + (long long)(w.q0 + qi) * a.dq_s + (long long)w.b * a.dq_b + (long long)hq * a.dq_h + half * 64;
    if (nblk > 0) {
      if (ok && warp_wait(&ctl->dq_full, 0, abort_flag, g.status, 822)) {
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          uint32_t v[32];
          tmem_ld32(tmem + 384 + lane_base + half * 64 + c * 32, v);
          tmem_ld_wait();
          if (row_ok) {
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {
              uint4 u;
              const int i0 = q4 * 8;
              u.x = pack_bf16x2(__uint_as_float(v[i0]) * g.scale, __uint_as_float(v[i0 + 1]) * g.scale);
              u.y = pack_bf16x2(__uint_as_float(v[i0 + 2]) * g.scale, __uint_as_float(v[i0 + 3]) * g.scale);
              u.z = pack_bf16x2(__uint_as_float(v[i0 + 4]) * g.scale, __uint_as_float(v[i0 + 5]) * g.scale);
              u.w = pack_bf16x2(__uint_as_float(v[i0 + 6]) * g.scale, __uint_as_float(v[i0 + 7]) * g.scale);
              reinterpret_cast<uint4*>(dqr + c * 32)[q4] = u;
            }
          }
        }
      }
    } else if (row_ok) {
      for (int i = 0; i < 8; ++i) reinterpret_cast<uint4*>(dqr)[i] = make_uint4(0, 0, 0, 0);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

static const CUtensorMap* tensor_map_sbhd(const void* p, int S, int B, int H, long long s_s, long long s_b, long long s_h) {
  const uint64_t dims[4] = {(uint64_t)D, (uint64_t)H, (uint64_t)B, (uint64_t)S};
  const uint64_t st[3] = {(uint64_t)s_h * 2, (uint64_t)s_b * 2, (uint64_t)s_s * 2};
  const uint32_t box[4] = {64, 1, 1, 128};
  return get_tmap_4d(p, 2, dims, st, box, true);
}

// Shared-memory opt-in, once per kernel and device.
template <class Kernel>
static cudaError_t opt_in(Kernel kern, int bytes, PerDeviceFlags& done_on) {
  bool& done = device_flag(done_on);
  if (done) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) set_last_error("attention: shared memory opt-in failed: %s", cudaGetErrorString(e));
  else done = true;
  return e;
}

// SM budget for kernels whose grid is one CTA per work item (one CTA per SM by shared memory): the items are cut into
// launches of at most `budget` CTAs, which the stream runs one after the other, so at most `budget` SMs are in use at
// any time.  launch(count, x0) starts items x0 .. x0 + count - 1.
template <class F>
static void launch_in_waves(long long items, int sm_budget, F&& launch) {
  const int sms = dh_sm_count();
  const long long wave = (sm_budget <= 0 || sm_budget >= sms) ? items : sm_budget;
  for (long long x0 = 0; x0 < items; x0 += wave) launch((unsigned)std::min(wave, items - x0), (int)x0);
}

// Tiles of a packed batch in descending order of work, cut into launches that fit one kernel parameter: MAX_TILES tiles of at most
// MAX_SEQS sequences.  More sequences are divided by length first (the longest MAX_SEQS, the next, ...): sorted as one, the equal
// tiles of all sequences would stand side by side and every MAX_SEQS of them fill a table (300 causal sequences of 1024 rows: 19
// launches, like this 5).
// rows(nq, nk) = what the tiles cover, `per` rows each; cost(nq, nk, tile) = key (query) blocks of that tile.
struct Sequences {
  int n;
  const int* cu_q;
  const int* cu_k;
  int nq(int s) const { return cu_q[s + 1] - cu_q[s]; }
  int nk(int s) const { return cu_k[s + 1] - cu_k[s]; }
};
template <class Rows, class Cost, class F>
static cudaError_t for_packed_launches(const Sequences& sq, int per, Rows&& rows, Cost&& cost, F&& launch) try {
  struct T { long long cost; int slot, tile; };
  std::vector<int> order(sq.n);
  for (int s = 0; s < sq.n; ++s) order[s] = s;
  if (sq.n > MAX_SEQS) {
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return rows(sq.nq(a), sq.nk(a)) > rows(sq.nq(b), sq.nk(b)); });
  }
  std::vector<T> tiles;
  for (int first = 0; first < sq.n; first += MAX_SEQS) {
    Packed p;
    tiles.clear();
    for (int i = 0; i < MAX_SEQS && first + i < sq.n; ++i) {
      const int s = order[first + i], nq = sq.nq(s), nk = sq.nk(s);
      p.q0[i] = sq.cu_q[s]; p.nq[i] = nq;
      p.k0[i] = sq.cu_k[s]; p.nk[i] = nk;
      p.id[i] = s;
      const int n = (int)(((long long)rows(nq, nk) + per - 1) / per);
      for (int t = 0; t < n; ++t) tiles.push_back({cost(nq, nk, t), i, t});
    }
    std::stable_sort(tiles.begin(), tiles.end(), [](const T& a, const T& b) { return a.cost > b.cost; });
    for (size_t t0 = 0; t0 < tiles.size(); t0 += MAX_TILES) {
      const int nt = (int)std::min(tiles.size() - t0, (size_t)MAX_TILES);
      for (int t = 0; t < nt; ++t) p.tile[t] = (uint32_t)tiles[t0 + t].slot << TILE_BITS | (uint32_t)tiles[t0 + t].tile;
      launch(p, nt);
    }
  }
  return cudaSuccess;
} catch (const std::bad_alloc&) {          // no exception may leave a C entry point
  set_last_error("attention: no host memory for the list of tiles");
  return cudaErrorMemoryAllocation;
}
static bool offsets_ok(const char* who, const Sequences& s, int Tq, int Tk, int max_q) {
  for (int i = 0; i < s.n; ++i) {
    const int nq = s.nq(i), nk = s.nk(i);
    if (s.cu_q[i] < 0 || s.cu_k[i] < 0 || nq < 0 || nk < 0 || nq > max_q || s.cu_q[i + 1] > Tq || s.cu_k[i + 1] > Tk) {
      set_last_error("%s: sequence %d (queries %d..%d, keys %d..%d) does not fit the packed tensors or the longest length %d", who, i,
                     s.cu_q[i], s.cu_q[i + 1], s.cu_k[i], s.cu_k[i + 1], max_q);
      return false;
    }
  }
  return true;
}
// Key blocks that query rows [first, first + rows) see / query blocks that see a key block.
static long long key_blocks(int nq, int nk, int causal, int first, int rows) {
  long long n = (nk + BKV - 1) / BKV;
  if (causal) {
    const long long last_key = (long long)std::min(first + rows, nq) - 1 + nk - nq;
    n = last_key < 0 ? 0 : std::min(n, last_key / BKV + 1);
  }
  return n;
}
static long long query_blocks(int nq, int nk, int causal, int kb) {
  const long long n = (nq + BQ - 1) / BQ;
  const long long first_q = causal ? (long long)kb * BKV - (nk - nq) : 0;
  return std::max(0ll, n - (first_q <= 0 ? 0 : first_q / BQ));
}

struct FwdMaps { const CUtensorMap *q, *k, *v; };
template <class Table>
static void run_fwd(const FwdMaps& m, Geometry& g, const FwdArgs& a, const Table& table, long long items, int sm_budget, cudaStream_t stream) {
  launch_in_waves(items, sm_budget, [&](unsigned n, int x0) {
    g.x0 = x0;
    if (g.scale > 0.f) attn_fwd_kernel<Table, true><<<n, THREADS, FWD_SMEM, stream>>>(*m.q, *m.k, *m.v, g, a, table);
    else attn_fwd_kernel<Table, false><<<n, THREADS, FWD_SMEM, stream>>>(*m.q, *m.k, *m.v, g, a, table);
  });
}

static long long packed_tiles(int nseq, const int* cu) {        // of 128 rows, in all sequences
  long long n = 0;
  for (int s = 0; s < nseq; ++s) n += (cu[s + 1] - cu[s] + BQ - 1) / BQ;
  return n;
}

// What a CTA of the forward takes.  One tile where every tile finds an SM of its own: it then does not wait for another's products and
// exponentials (1000 positions, 8 heads on 1, all keys: 24.7 -> 20.6 us, 2048: 41.5 -> 34.4).  Also where the longest tile alone takes as
// long as all of them spread over the SMs, that is under causal masks (up to twice as many tiles as SMs were measured; 4096
// positions, 8 heads on 1: 71 -> 60 us), unless tiles are so short that a second round of CTAs costs more (384 positions: 14.4 -> 16.5).
// Else two query heads of a KV group where groups are even: both tiles then see the same keys whatever the mask, and
// a sequence of up to 128 rows fills the CTA.  Odd groups (one query head per KV head) take two row tiles instead.
static int fwd_mode(const Sequences& sq, int B, int Hq, int Hk, int causal, int sm_budget) {
  const int sms = dh_sm_count();
  const bool budgeted = sm_budget > 0 && sm_budget < sms;
  const long long room = budgeted ? sm_budget : sms, per_tile = (long long)B * Hq;
  const long long tiles = packed_tiles(sq.n, sq.cu_q) * per_tile;
  if (tiles <= room) return SINGLE;
  if (!budgeted && tiles <= 2 * room) {
    long long work = 0, longest = 0;
    for (int s = 0; s < sq.n; ++s) {
      for (int first = 0; first < sq.nq(s); first += BQ) {
        const long long n = key_blocks(sq.nq(s), sq.nk(s), causal, first, BQ);
        work += n;
        longest = std::max(longest, n);
      }
    }
    if (longest >= 8 && work * per_tile <= room * longest) return SINGLE;
  }
  return (Hq / Hk) % 2 == 0 ? HEAD_PAIR : ROW_PAIR;
}

// Number of CTAs that share the query heads of one KV head in the dK/dV kernel: 1 while
// KV blocks x batch x KV heads already give every SM a few CTAs, else the smallest power of
// two (dividing the group size) that does.
static int bwd_head_split(long long kv_tiles, int Hq, int Hk) {
  static int enabled = -1;
  if (enabled < 0) {
    const char* e = getenv("DHELLAM_ATTN_HEAD_SPLIT");
    enabled = e ? atoi(e) : 1;
  }
  if (!enabled) return 1;
  const int group = Hq / Hk;
  const long long ctas = kv_tiles * Hk;
  int hs = 1;
  while (hs < group && group % (hs * 2) == 0 && ctas * hs < 4LL * dh_sm_count()) hs *= 2;
  return hs;
}
// Scratch of the backward: delta [B*Hq*Tq] fp32 (row dot products of dO and O), rounded up to 256 bytes, then, when
// the dK/dV kernel splits heads, the fp32 partials [2][hs][Tk][B][Hk][128].
static int64_t delta_bytes(int B, int Hq, int Tq) { return ((int64_t)B * Hq * Tq * 4 + 255) / 256 * 256; }
static int64_t scratch_bytes(int B, int Hq, int Hk, int Tq, int Tk, int hs) {
  return delta_bytes(B, Hq, Tq) + (hs > 1 ? (int64_t)2 * hs * Tk * B * Hk * D * 4 : 0);
}

static void launch_delta(const void* dout, const void* out, float* delta, int B, int Hq, int T, const int64_t* sdo, const int64_t* so,
                         cudaStream_t stream) {
  // dO is a TMA operand (16-byte aligned throughout); O need not be
  const int wide = ((reinterpret_cast<uintptr_t>(out) | (uintptr_t)(so[0] * 2) | (uintptr_t)(so[1] * 2) | (uintptr_t)(so[2] * 2)) & 15) == 0;
  attn_delta_kernel<<<dim3((unsigned)((T + 63) / 64 * Hq), B), 256, 0, stream>>>((const __nv_bfloat16*)dout, (const __nv_bfloat16*)out, delta, Hq, T,
                                                                                 sdo[0], sdo[1], sdo[2], so[0], so[1], so[2], wide);
}

struct BwdMaps { const CUtensorMap *q, *k, *v, *dout; };
template <class Table>
static void run_dkv(const BwdMaps& m, Geometry& g, const DkvArgs& a, const Table& table, long long items, int sm_budget, cudaStream_t stream) {
  g.heads = g.Hk * a.hs;
  launch_in_waves(items, sm_budget, [&](unsigned n, int x0) {
    g.x0 = x0;
    attn_bwd_dkv_kernel<Table><<<n, THREADS, DKV_SMEM, stream>>>(*m.q, *m.k, *m.v, *m.dout, g, a, table);
  });
}
template <class Table>
static void run_dq(const BwdMaps& m, Geometry& g, const DqArgs& a, const Table& table, long long items, int sm_budget, cudaStream_t stream) {
  g.heads = g.Hq;
  launch_in_waves(items, sm_budget, [&](unsigned n, int x0) {
    g.x0 = x0;
    attn_bwd_dq_kernel<Table><<<n, THREADS, DQ_SMEM, stream>>>(*m.q, *m.k, *m.v, *m.dout, g, a, table);
  });
}
template <class Table>
static cudaError_t opt_in_fwd() {
  static PerDeviceFlags done, done_other;
  cudaError_t e = opt_in(attn_fwd_kernel<Table, true>, FWD_SMEM, done);
  return e != cudaSuccess ? e : opt_in(attn_fwd_kernel<Table, false>, FWD_SMEM, done_other);
}
template <class Table>
static cudaError_t opt_in_bwd() {
  static PerDeviceFlags done_kv, done_q;
  cudaError_t e = opt_in(attn_bwd_dkv_kernel<Table>, DKV_SMEM, done_kv);
  return e != cudaSuccess ? e : opt_in(attn_bwd_dq_kernel<Table>, DQ_SMEM, done_q);
}

// One backward over either kind of batch; `seqs` null = dense.
static int bwd_common(const void* dout, const void* out, const void* lse, void* dq, void* dk, void* dv, void* scratch, const int64_t* strides,
                      const BwdMaps& maps, Geometry g, int hs, const Sequences* seqs, int sm_budget, cudaStream_t stream) {
  const int64_t* sdo = strides; const int64_t* so = strides + 12;
  const int64_t* sdq = strides + 15; const int64_t* sdk = strides + 18; const int64_t* sdv = strides + 21;
  float* delta = reinterpret_cast<float*>(scratch);
  launch_delta(dout, out, delta, g.B, g.Hq, g.Tq, sdo, so, stream);
  DkvArgs a;
  a.lse = (const float*)lse; a.delta = delta;
  a.dk = (__nv_bfloat16*)dk; a.dv = (__nv_bfloat16*)dv;
  a.dk_s = sdk[0]; a.dk_b = sdk[1]; a.dk_h = sdk[2]; a.dv_s = sdv[0]; a.dv_b = sdv[1]; a.dv_h = sdv[2];
  a.hs = hs;
  a.part = hs > 1 ? reinterpret_cast<float*>(reinterpret_cast<char*>(scratch) + delta_bytes(g.B, g.Hq, g.Tq)) : nullptr;
  DqArgs aq;
  aq.lse = (const float*)lse; aq.delta = delta; aq.dq = (__nv_bfloat16*)dq;
  aq.dq_s = sdq[0]; aq.dq_b = sdq[1]; aq.dq_h = sdq[2];
  cudaError_t e = cudaSuccess;
  if (seqs == nullptr) {
    run_dkv(maps, g, a, Dense{}, (long long)((g.Sk + BKV - 1) / BKV) * g.B * g.Hk * hs, sm_budget, stream);
  } else {
    e = for_packed_launches(*seqs, BKV, [](int, int nk) { return nk; }, [&](int nq, int nk, int t) { return query_blocks(nq, nk, g.causal, t); },
                            [&](const Packed& p, int n) { run_dkv(maps, g, a, p, (long long)n * g.Hk * hs, sm_budget, stream); });
    if (e != cudaSuccess) return (int)e;
  }
  if (hs > 1) {
    const long long n = 2LL * g.Tk * g.B * g.Hk * (D / 8);
    attn_dkv_reduce_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(a.part, hs, a.dk, a.dv, g.Tk, g.B, g.Hk, sdk[0], sdk[1], sdk[2],
                                                                           sdv[0], sdv[1], sdv[2]);
  }
  if (seqs == nullptr) {
    run_dq(maps, g, aq, Dense{}, (long long)((g.Sq + BQ - 1) / BQ) * g.B * g.Hq, sm_budget, stream);
  } else {
    e = for_packed_launches(*seqs, BQ, [](int nq, int) { return nq; },
                            [&](int nq, int nk, int t) { return key_blocks(nq, nk, g.causal, t * BQ, BQ); },
                            [&](const Packed& p, int n) { run_dq(maps, g, aq, p, (long long)n * g.Hq, sm_budget, stream); });
    if (e != cudaSuccess) return (int)e;
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) set_last_error("attention backward launch failed: %s", cudaGetErrorString(e));
  return (int)e;
}

static Geometry geometry(int B, int Hq, int Hk, int Sq, int Sk, int Tq, int Tk, int ls, int causal, float scale) {
  Geometry g;
  g.B = B; g.Hq = Hq; g.Hk = Hk; g.Sq = Sq; g.Sk = Sk; g.Tq = Tq; g.Tk = Tk; g.ls = ls; g.causal = causal; g.scale = scale;
  g.x0 = 0; g.heads = Hq;
  g.status = reinterpret_cast<DeviceStatus*>(dh_status_device_ptr());
  return g;
}
constexpr long long MAX_BWD_ROWS = 1ll << 26;       // query rows x heads (x batch) of one dense backward, or of one sequence

static bool heads_ok(const char* who, int d, int Hq, int Hk) {
  if (d != D) { set_last_error("%s: head size %d is not supported (128 only)", who, d); return false; }
  if (Hk <= 0 || Hq % Hk != 0) { set_last_error("%s: query heads must be a multiple of KV heads", who); return false; }
  return true;
}

}  // namespace attn
}  // namespace dh

using namespace dh;
using namespace dh::attn;

extern "C" {

// There is one dK/dV kernel; callers that used to choose between two forms are accepted.
void dh_attn_set_bwd_mode(int) {}

int dh_attn_fwd(const void* q, const void* k, const void* v, void* out, void* lse, int64_t q_s, int64_t q_b, int64_t q_h, int64_t k_s,
                int64_t k_b, int64_t k_h, int64_t v_s, int64_t v_b, int64_t v_h, int B, int Hq, int Hk, int Sq, int Sk, int d, int causal,
                float scale, int sm_budget, cudaStream_t stream) {
  if (!heads_ok("dh_attn_fwd", d, Hq, Hk)) return (int)cudaErrorInvalidValue;
  if (B <= 0 || Sq <= 0 || Sk <= 0) return 0;
  const FwdMaps m = {tensor_map_sbhd(q, Sq, B, Hq, q_s, q_b, q_h), tensor_map_sbhd(k, Sk, B, Hk, k_s, k_b, k_h),
                     tensor_map_sbhd(v, Sk, B, Hk, v_s, v_b, v_h)};
  if (!m.q || !m.k || !m.v) return (int)cudaErrorInvalidValue;
  cudaError_t e = opt_in_fwd<Dense>();
  if (e != cudaSuccess) return (int)e;
  Geometry g = geometry(B, Hq, Hk, Sq, Sk, Sq, Sk, Sq, causal, scale);
  FwdArgs a;
  a.out = (__nv_bfloat16*)out; a.lse = (float*)lse;
  a.o_h = D; a.o_b = (long long)Hq * D; a.o_s = (long long)B * Hq * D;
  const int cu_q[2] = {0, Sq}, cu_k[2] = {0, Sk};
  a.mode = fwd_mode({1, cu_q, cu_k}, B, Hq, Hk, causal, sm_budget);
  const int per = a.mode == ROW_PAIR ? 2 * BQ : BQ;
  g.heads = a.mode == HEAD_PAIR ? Hq / 2 : Hq;
  run_fwd(m, g, a, Dense{}, (long long)((Sq + per - 1) / per) * g.heads * B, sm_budget, stream);
  e = cudaGetLastError();
  if (e != cudaSuccess) set_last_error("dh_attn_fwd launch failed: %s", cudaGetErrorString(e));
  return (int)e;
}

int dh_attn_fwd_packed(const void* q, const void* k, const void* v, void* out, void* lse, const int64_t* strides /* q,k,v,out x (row,head) */,
                       int nseq, const int* cu_q, const int* cu_k, int Tq, int Tk, int max_q, int Hq, int Hk, int d, int causal, float scale,
                       int sm_budget, cudaStream_t stream) {
  if (!heads_ok("dh_attn_fwd_packed", d, Hq, Hk)) return (int)cudaErrorInvalidValue;
  if (nseq <= 0 || Tq <= 0 || Tk <= 0) return 0;
  const Sequences seqs = {nseq, cu_q, cu_k};
  if (!offsets_ok("dh_attn_fwd_packed", seqs, Tq, Tk, max_q)) return (int)cudaErrorInvalidValue;
  // the batch dimension has one entry: its stride only has to be a valid one
  const FwdMaps m = {tensor_map_sbhd(q, Tq, 1, Hq, strides[0], strides[0], strides[1]), tensor_map_sbhd(k, Tk, 1, Hk, strides[2], strides[2], strides[3]),
                     tensor_map_sbhd(v, Tk, 1, Hk, strides[4], strides[4], strides[5])};
  if (!m.q || !m.k || !m.v) return (int)cudaErrorInvalidValue;
  cudaError_t e = opt_in_fwd<Packed>();
  if (e != cudaSuccess) return (int)e;
  Geometry g = geometry(1, Hq, Hk, 0, 0, Tq, Tk, max_q, causal, scale);
  FwdArgs a;
  a.out = (__nv_bfloat16*)out; a.lse = (float*)lse;
  a.o_s = strides[6]; a.o_h = strides[7]; a.o_b = 0;
  a.mode = fwd_mode(seqs, 1, Hq, Hk, causal, sm_budget);
  const int per = a.mode == ROW_PAIR ? 2 * BQ : BQ;
  g.heads = a.mode == HEAD_PAIR ? Hq / 2 : Hq;
  e = for_packed_launches(seqs, per, [](int nq, int) { return nq; },
                          [&](int nq, int nk, int t) { return key_blocks(nq, nk, causal, t * per, per); },
                          [&](const Packed& p, int n) { run_fwd(m, g, a, p, (long long)n * g.heads, sm_budget, stream); });
  if (e != cudaSuccess) return (int)e;
  e = cudaGetLastError();
  if (e != cudaSuccess) set_last_error("dh_attn_fwd_packed launch failed: %s", cudaGetErrorString(e));
  return (int)e;
}

int dh_attn_packed_launches(int nseq, const int* cu_q, const int* cu_k, int causal) {
  const Sequences seqs = {nseq, cu_q, cu_k};
  int launches = 0;
  const cudaError_t e = for_packed_launches(seqs, BQ, [](int nq, int) { return nq; },
                                            [&](int nq, int nk, int t) { return key_blocks(nq, nk, causal, t * BQ, BQ); },
                                            [&](const Packed&, int) { ++launches; });
  return e == cudaSuccess ? launches : -(int)e;
}

int64_t dh_attn_bwd_scratch_bytes(int B, int Hq, int Hk, int Sq, int Sk) {
  const int hs = Hk > 0 && Hq % Hk == 0 ? bwd_head_split((long long)((Sk + BKV - 1) / BKV) * B, Hq, Hk) : 1;
  return scratch_bytes(B, Hq, Hk, Sq, Sk, hs);
}

int64_t dh_attn_bwd_packed_scratch_bytes(int nseq, const int* cu_k, int Hq, int Hk, int Tq, int Tk) {
  const int hs = Hk > 0 && Hq % Hk == 0 ? bwd_head_split(packed_tiles(nseq, cu_k), Hq, Hk) : 1;
  return scratch_bytes(1, Hq, Hk, Tq, Tk, hs);
}

int dh_attn_bwd(const void* dout, const void* q, const void* k, const void* v, const void* out, const void* lse, void* dq, void* dk,
                void* dv, void* scratch, const int64_t* strides /* 8 tensors x (s,b,h): do,q,k,v,o,dq,dk,dv */, int B, int Hq, int Hk,
                int Sq, int Sk, int d, int causal, float scale, int sm_budget, cudaStream_t stream) {
  if (!heads_ok("dh_attn_bwd", d, Hq, Hk)) return (int)cudaErrorInvalidValue;
  if (B <= 0 || Sq <= 0 || Sk <= 0) return 0;
  const int64_t* sdo = strides; const int64_t* sq = strides + 3; const int64_t* sk = strides + 6; const int64_t* sv = strides + 9;
  const BwdMaps m = {tensor_map_sbhd(q, Sq, B, Hq, sq[0], sq[1], sq[2]), tensor_map_sbhd(k, Sk, B, Hk, sk[0], sk[1], sk[2]),
                     tensor_map_sbhd(v, Sk, B, Hk, sv[0], sv[1], sv[2]), tensor_map_sbhd(dout, Sq, B, Hq, sdo[0], sdo[1], sdo[2])};
  if (!m.q || !m.k || !m.v || !m.dout) return (int)cudaErrorInvalidValue;
  cudaError_t e = opt_in_bwd<Dense>();
  if (e != cudaSuccess) return (int)e;
  const long long rows_ll = (long long)B * Hq * Sq;
  if (rows_ll > MAX_BWD_ROWS) {
    set_last_error("dh_attn_bwd: B*Hq*Sq = %lld rows exceed the supported 2^26", rows_ll);
    return (int)cudaErrorInvalidValue;
  }
  const int hs = bwd_head_split((long long)((Sk + BKV - 1) / BKV) * B, Hq, Hk);
  return bwd_common(dout, out, lse, dq, dk, dv, scratch, strides, m, geometry(B, Hq, Hk, Sq, Sk, Sq, Sk, Sq, causal, scale), hs, nullptr, sm_budget,
                    stream);
}

int dh_attn_bwd_packed(const void* dout, const void* q, const void* k, const void* v, const void* out, const void* lse, void* dq, void* dk,
                       void* dv, void* scratch, const int64_t* strides /* as dh_attn_bwd; the batch strides are not used */, int nseq,
                       const int* cu_q, const int* cu_k, int Tq, int Tk, int lse_rows, int Hq, int Hk, int d, int causal, float scale,
                       int sm_budget, cudaStream_t stream) {
  if (!heads_ok("dh_attn_bwd_packed", d, Hq, Hk)) return (int)cudaErrorInvalidValue;
  if (nseq <= 0 || Tq <= 0 || Tk <= 0) return 0;
  const Sequences seqs = {nseq, cu_q, cu_k};
  if (!offsets_ok("dh_attn_bwd_packed", seqs, Tq, Tk, lse_rows)) return (int)cudaErrorInvalidValue;
  for (int i = 0; i < nseq; ++i) {
    const long long rows = (long long)Hq * (cu_q[i + 1] - cu_q[i]);
    if (rows > MAX_BWD_ROWS) {
      set_last_error("dh_attn_bwd_packed: Hq*Sq = %lld rows of sequence %d exceed the supported 2^26", rows, i);
      return (int)cudaErrorInvalidValue;
    }
  }
  const int64_t* sdo = strides; const int64_t* sq = strides + 3; const int64_t* sk = strides + 6; const int64_t* sv = strides + 9;
  const BwdMaps m = {tensor_map_sbhd(q, Tq, 1, Hq, sq[0], sq[0], sq[2]), tensor_map_sbhd(k, Tk, 1, Hk, sk[0], sk[0], sk[2]),
                     tensor_map_sbhd(v, Tk, 1, Hk, sv[0], sv[0], sv[2]), tensor_map_sbhd(dout, Tq, 1, Hq, sdo[0], sdo[0], sdo[2])};
  if (!m.q || !m.k || !m.v || !m.dout) return (int)cudaErrorInvalidValue;
  cudaError_t e = opt_in_bwd<Packed>();
  if (e != cudaSuccess) return (int)e;
  const int hs = bwd_head_split(packed_tiles(nseq, cu_k), Hq, Hk);
  return bwd_common(dout, out, lse, dq, dk, dv, scratch, strides, m, geometry(1, Hq, Hk, 0, 0, Tq, Tk, lse_rows, causal, scale), hs, &seqs,
                    sm_budget, stream);
}

}  // extern "C"

// =========================================================================== no-allocation entry
#include "attn_noalloc.h"

namespace dh {
bool encode_tmap_4d_into(CUtensorMap* out, const void* base, int elem_bytes, const uint64_t dims[4], const uint64_t strides_bytes[3],
                         const uint32_t box[4], bool swizzle128);
namespace attn {

// Scratch of the no-allocation entry point.  In host code this name is only a handle for
// cudaGetSymbolAddress; kernels receive the resolved device address.
static __device__ __align__(256) unsigned char g_noalloc_scratch[DH_ATTN_NOALLOC_SCRATCH_BYTES];

constexpr int kNoallocMaxDev = 32;
static void* g_noalloc_addr[kNoallocMaxDev] = {nullptr};
static bool g_noalloc_ready[kNoallocMaxDev] = {false};
static std::mutex g_noalloc_mutex;     // two host threads may make the first call on one device at the same time

static bool map_sbhd_into(CUtensorMap* m, const void* p, int S, int B, int H, const int64_t* st) {
  const uint64_t dims[4] = {(uint64_t)D, (uint64_t)H, (uint64_t)B, (uint64_t)S};
  const uint64_t sb[3] = {(uint64_t)st[2] * 2, (uint64_t)st[1] * 2, (uint64_t)st[0] * 2};
  const uint32_t box[4] = {64, 1, 1, 128};
  return encode_tmap_4d_into(m, p, 2, dims, sb, box, true);
}

}  // namespace attn
}  // namespace dh

extern "C" int dh_attn_bwd_noalloc(const void* dout, const void* q, const void* k, const void* v, const void* out, const void* lse,
                                   void* dq, void* dk, void* dv, const int64_t* strides, int B, int Hq, int Hk, int Sq, int Sk, int d,
                                   int causal, float scale, cudaStream_t stream) {
  if (d != D) { set_last_error("dh_attn_bwd_noalloc: head size %d is not supported (128 only)", d); return (int)cudaErrorInvalidValue; }
  if (Hk <= 0 || Hq % Hk != 0) { set_last_error("dh_attn_bwd_noalloc: query heads must be a multiple of KV heads"); return (int)cudaErrorInvalidValue; }
  if (B <= 0 || Sq <= 0 || Sk <= 0) return 0;
  const int64_t rows = (int64_t)B * Hq * Sq;
  const int64_t need = (rows * 4 + 255) / 256 * 256;
  if (need > (int64_t)DH_ATTN_NOALLOC_SCRATCH_BYTES) {
    set_last_error("dh_attn_bwd_noalloc: B*Hq*Sq = %lld rows need %lld bytes of scratch, the built-in array holds %u; "
                   "use dh_attn_bwd with a caller-provided buffer", (long long)rows, (long long)need, DH_ATTN_NOALLOC_SCRATCH_BYTES);
    return (int)cudaErrorInvalidValue;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kNoallocMaxDev) { set_last_error("dh_attn_bwd_noalloc: no usable current device"); return (int)cudaErrorInvalidDevice; }
  {
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_ready[dev]) {
    // once per device, with that device current: resolve the array's device address
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
    if (e != cudaSuccess || ptr == nullptr) { set_last_error("dh_attn_bwd_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e)); return (int)e; }
    e = opt_in_bwd<Dense>();
    if (e != cudaSuccess) return (int)e;
    g_noalloc_addr[dev] = ptr;
    g_noalloc_ready[dev] = true;
  }
  }
  const int64_t* sdo = strides; const int64_t* sq = strides + 3; const int64_t* sk = strides + 6; const int64_t* sv = strides + 9;
  const int64_t* so = strides + 12; const int64_t* sdq = strides + 15; const int64_t* sdk = strides + 18; const int64_t* sdv = strides + 21;
  CUtensorMap tq, tk, tv, tdo;
  if (!map_sbhd_into(&tq, q, Sq, B, Hq, sq) || !map_sbhd_into(&tk, k, Sk, B, Hk, sk) || !map_sbhd_into(&tv, v, Sk, B, Hk, sv) ||
      !map_sbhd_into(&tdo, dout, Sq, B, Hq, sdo))
    return (int)cudaErrorInvalidValue;
  // delta is fully rewritten by every call, so nothing in the shared array needs clearing; the array holds delta only,
  // so the query heads are never split here
  Geometry g = geometry(B, Hq, Hk, Sq, Sk, Sq, Sk, Sq, causal, scale);
  g.status = nullptr;
  return bwd_common(dout, out, lse, dq, dk, dv, g_noalloc_addr[dev], strides, BwdMaps{&tq, &tk, &tv, &tdo}, g, 1, nullptr, 0, stream);
}
