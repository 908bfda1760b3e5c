// Static block-sparse flash attention forward for sm_100a, driven by a CSR list of key
// blocks per query block, plus 2-D rotary embedding.
//
// The reference's static sparse attention
// (src/sparse_wsi_vit/models/static_sparse_attention.py:62-188) materialises a dense
// (N, N*ctx) mask and runs three SDPA calls; the 2-D block pattern the target asks for has
// no reference code at all.  Both are served by one kernel:
//   mode 0  : every listed key block is attended in full (block mask, shared by all heads);
//   mode 1  : inside the listed blocks the reference's token-level pattern applies:
//             query i sees key j iff  i < C  or  j < C  or
//             (|i - j| <= W*d and (i - j) % d == 0)      (C CLS tokens first, window W, dilation d)
//             -- exactly the mask static_sparse_attention.py:159-176 builds.
// A CTA owns (batch, head, one query block) or, of a query block whose list is long, one chunk of
// the list.  The score tile is M = 128 query rows by N = BS keys (BS = 64: the 64 rows behind the
// block are computed by the tensor core and skipped by the softmax).
//   warp 0     : TMA producer (Q once; K, V blocks of the list through rings)
//   warp 1     : UMMA issuer: S(j) = Q K(j)^T, then O += P(j) V(j) with P read from TMEM
//   warps 2..5 : online softmax, one thread per query row: the row's BS scores are read into registers
//                once, their maximum is taken, and P is written as bf16 pairs over the first half of the
//                score columns, in two halves, so that PV starts under the second half's exponentials.
//                The stabiliser is raised (and O in TMEM rescaled) only when a row's maximum exceeds it
//                by 2^8.
// TMEM: S fp32 [0,BS), P (bf16x2) [0,BS/2) over it | O fp32 [BS, BS+D).
// With P on top of S a CTA needs at most 256 columns and 100 KiB of shared memory, so TWO CTAs share
// an SM: one CTA's softmax runs under the other's products.  Bound at 128 x 128 x 128 tiles: the chain
// QK -> softmax -> PV of each CTA (4100 cycles a tile, two tiles in flight; products 1024, exponentials
// 1024 of the SM's time per tile); 32768 tokens, 16 heads, 5 % of the blocks: 0.82 -> 0.79 ms against one
// CTA with two score and two probability buffers and eight softmax warps.  Token patterns are evaluated
// as whole mask words (one arithmetic range per 32 keys; testing every pair took four times the tile's
// time: 2.5 -> 1.0 ms for the 65536-token sliding window), and lists far longer than the mean are divided
// (a CLS block over 33 key blocks, 6 heads: 252 -> 44 us).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"

namespace swv {

struct BsaParams {
  int B, H, Tq, Tk, nQB;
  const int32_t* row_ptr;   // [nQB + 1]
  const int32_t* col_idx;   // [nnz] key block index
  int mode, num_cls, reach, dilation;   // reach = window * dilation, at most Tq + Tk
  int kv_group;             // query heads per key/value head (grouped-query attention), >= 1
  float* lse;               // optional (B,H,Tq): natural-log sum of exponentials per row, -inf for empty rows
  // Optional gated epilogue (the NSA branches): the rows are scaled by sigmoid(gate[b,t,h,gate_idx])
  // (gate (B,Tq,H,3) fp32) and added to `acc_in` (fp32 contiguous (B,H,Tq,D), may be null) before
  // they are written to `o`.
  const float* gate;
  int gate_idx;
  const float* acc_in;
  void* o;
  int64_t osb, osh, ost;
  int o_dtype;
  float scale_log2;
  // Long lists: a query block with more than `chunk` key blocks is divided over ceil(n / chunk) CTAs
  // (chunk = 0: never).  The first `extra` CTAs of every (batch, head) serve the second and later
  // chunks.  Partial rows go to `part_o` / `part_ml`, a later chunk's to the slot of its extra unit, the
  // first chunk's to slot extra + (its list's first extra unit); the CTA that takes the last ticket of the
  // row block adds them up.
  int chunk, extra;
  float* part_o;            // [B*H][2 * extra][BS rows][D] unnormalised fp32 rows
  float2* part_ml;          // [B*H][2 * extra][BS rows] (stabiliser, probability sum)
  uint32_t* tickets;        // [B*H][nQB], zero before the launch
  int* status;
};

constexpr int kBsaThreads = 192;

struct BsaCtl {
  uint64_t q_full;
  uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2];
  uint64_t s_full, p_full[2], pv_done;         // p_full: first and second half of the tile's keys
  uint32_t tmem_base;
  uint32_t abort_flag;
  int unit[3];                                 // query block, chunk, number of extra units before the query block
  uint32_t ticket;
  int scan[kBsaThreads / 32];
};

template <int BS, int D>
struct BsaCfg {
  static constexpr int kStages = BS * D > 8192 ? 1 : 2;   // 128 x 128 blocks: one stage, so that two CTAs fit
  static constexpr int kQBytes = kTile * D * 2;     // 128 query rows
  static constexpr int kKVBytes = BS * D * 2;       // one key / value block
  static constexpr int kOffK = kQBytes;
  static constexpr int kOffV = kOffK + kStages * kKVBytes;
  static constexpr int kOffCtl = kOffV + kStages * kKVBytes;
  static constexpr uint32_t kColO = BS;
  static constexpr uint32_t kTmemCols = (BS + D <= 128) ? 128 : 256;
  static constexpr int kCtas = kTmemCols == 128 ? 3 : 2;  // resident CTAs (registers: 112 and 168 per thread)
  // at least 80 KiB where 256 columns are used so that no third CTA waits for TMEM
  static constexpr size_t kSmemNeed = 1024 + kOffCtl + sizeof(BsaCtl) + 64;
  static constexpr size_t kSmem = (kTmemCols == 256 && kSmemNeed < 80 * 1024) ? 80 * 1024 : kSmemNeed;
};

// bits [0, n) of a word, n clamped to [0, 32]
__device__ __forceinline__ uint32_t low_bits(int n) { return n >= 32 ? 0xFFFFFFFFu : (n <= 0 ? 0u : (1u << n) - 1u); }

// Token-level pattern of the reference's static attention (mode 1) for query `qi` and the 32 keys
// base..base+31 as a bit mask: the CLS keys, and the window's arithmetic progression.  With window 0 a
// patch sees the CLS keys only, not itself (static_sparse_attention.py:92-95).
__device__ __forceinline__ uint32_t static_pattern_word(int qi, int base, int C, int reach, int d) {
  if (qi < C) return 0xFFFFFFFFu;
  uint32_t w = low_bits(C - base);
  if (reach > 0) {
    uint32_t win = low_bits(qi + reach - base + 1) & ~low_bits(qi - reach - base);
    if (d > 1 && win != 0u) {
      int ph = (qi - base) % d;
      if (ph < 0) ph += d;
      uint32_t comb = ph < 32 ? 1u << ph : 0u;
      for (int s = d; s < 32; s <<= 1) comb |= comb << s;
      win &= comb;
    }
    w |= win;
  }
  return w;
}

// max of three / packed pair arithmetic: half the instructions of the scalar forms
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ void fma_pair(float& x, float& y, float a, float b, float sc, float add) {
  asm("{\n\t.reg .b64 v, s, d;\n\tmov.b64 v, {%2, %3};\n\tmov.b64 s, {%4, %4};\n\tmov.b64 d, {%5, %5};\n\t"
      "fma.rn.f32x2 v, v, s, d;\n\tmov.b64 {%0, %1}, v;\n\t}"
      : "=f"(x), "=f"(y)
      : "f"(a), "f"(b), "f"(sc), "f"(add));
}
__device__ __forceinline__ void add_pair(float& x, float& y, float a, float b) {
  asm("{\n\t.reg .b64 v, s;\n\tmov.b64 v, {%0, %1};\n\tmov.b64 s, {%2, %3};\n\tadd.rn.f32x2 v, v, s;\n\tmov.b64 {%0, %1}, v;\n\t}"
      : "+f"(x), "+f"(y)
      : "f"(a), "f"(b));
}

// The (query block, chunk) of extra unit `e`: query block r contributes ceil(len_r / chunk) - 1 extra
// units, in query-block order.  All threads of the CTA take part; returns false past the last unit.
__device__ __forceinline__ bool bsa_find_extra(const BsaParams& p, int e, BsaCtl* ctl) {
  if (threadIdx.x == 0) ctl->unit[0] = -1;
  int before = 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int r0 = 0; r0 < p.nQB; r0 += blockDim.x) {
    const int r = r0 + threadIdx.x;
    int n = 0;
    if (r < p.nQB) n = max(0, (p.row_ptr[r + 1] - p.row_ptr[r] + p.chunk - 1) / p.chunk - 1);
    int inc = n;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= off) inc += t;
    }
    if (lane == 31) ctl->scan[warp] = inc;
    __syncthreads();
    int base = before, total = 0;
    for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) {
      if (w < warp) base += ctl->scan[w];
      total += ctl->scan[w];
    }
    const int first = base + inc - n;
    if (n > 0 && e >= first && e < first + n) {
      ctl->unit[0] = r;
      ctl->unit[1] = e - first + 1;
      ctl->unit[2] = first;
    }
    __syncthreads();
    if (ctl->unit[0] >= 0) return true;
    before += total;
    if (e < before) break;      // (cannot happen: the owner was found above)
  }
  return false;
}

// Number of extra units of the query blocks before `qb` (for the workspace slots of its chunks).
__device__ __forceinline__ int bsa_extra_before(const BsaParams& p, int qb, BsaCtl* ctl) {
  int n = 0;
  for (int r = threadIdx.x; r < qb; r += blockDim.x)
    n += max(0, (p.row_ptr[r + 1] - p.row_ptr[r] + p.chunk - 1) / p.chunk - 1);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) n += __shfl_xor_sync(0xffffffffu, n, off);
  if ((threadIdx.x & 31) == 0) ctl->scan[threadIdx.x >> 5] = n;
  __syncthreads();
  int t = 0;
  for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) t += ctl->scan[w];
  return t;
}

template <int BS, int D>
__global__ void __launch_bounds__(kBsaThreads, BsaCfg<BS, D>::kCtas)
    block_sparse_attn_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                             const __grid_constant__ CUtensorMap tm_v, const BsaParams p) {
  using Cfg = BsaCfg<BS, D>;
  constexpr int NST = Cfg::kStages;
  constexpr uint32_t kIdescQK = make_idesc(/*bf16*/ 1, kTile, BS, 0, 0);
  constexpr uint32_t kIdescPV = make_idesc(/*bf16*/ 1, kTile, D, 0, /*V is MN-major*/ 1);
  constexpr float kStep = 8.0f;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  BsaCtl* ctl = reinterpret_cast<BsaCtl*>(smem + Cfg::kOffCtl);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // the later chunks of long lists first (they are the longest-running units), then query blocks
  // fastest, heads slowest: the CTAs in flight at any time work on one or two heads, whose keys and
  // values stay in L2 (all heads' K/V together can exceed it)
  int qb, bh, ch = 0, nch = 1, ubase = 0;
  const int n_extra = p.extra * p.B * p.H;
  if (static_cast<int>(blockIdx.x) < n_extra) {
    bh = blockIdx.x / p.extra;
    if (!bsa_find_extra(p, blockIdx.x % p.extra, ctl)) return;
    qb = ctl->unit[0];
    ch = ctl->unit[1];
    ubase = ctl->unit[2];
  } else {
    const int u = blockIdx.x - n_extra;
    qb = u % p.nQB;
    bh = u / p.nQB;
  }
  const int h = bh % p.H;
  const int b = bh / p.H;
  int list0 = p.row_ptr[qb];
  int nblk = p.row_ptr[qb + 1] - list0;
  bool peek = false;
  int first_blk = 0;
  if (p.chunk > 0 && nblk > p.chunk) {
    nch = (nblk + p.chunk - 1) / p.chunk;
    if (ch == 0) ubase = bsa_extra_before(p, qb, ctl);
    const int a = static_cast<int>(static_cast<int64_t>(nblk) * ch / nch);
    const int z = static_cast<int>(static_cast<int64_t>(nblk) * (ch + 1) / nch);
    // A later chunk looks at the list's first block before its own: it starts from the same stabiliser
    // as the first chunk, so its probabilities round to bf16 as they would in one sweep unless a block
    // between the two would have raised it.
    peek = ch > 0;
    first_blk = list0;
    list0 += a - (peek ? 1 : 0);
    nblk = z - a + (peek ? 1 : 0);
  }

  if (threadIdx.x == 0) {
    mbar_init(&ctl->q_full, 1);
    for (int s = 0; s < NST; ++s) {
      mbar_init(&ctl->k_full[s], 1);
      mbar_init(&ctl->k_empty[s], 1);
      mbar_init(&ctl->v_full[s], 1);
      mbar_init(&ctl->v_empty[s], 1);
    }
    mbar_init(&ctl->s_full, 1);
    mbar_init(&ctl->p_full[0], 4);
    mbar_init(&ctl->p_full[1], 4);
    mbar_init(&ctl->pv_done, 1);
    ctl->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&ctl->tmem_base, Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;
  volatile uint32_t* abort_flag = &ctl->abort_flag;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0 && nblk > 0) {
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
      mbar_expect_tx(&ctl->q_full, Cfg::kQBytes);
#pragma unroll
      for (int c = 0; c < D / 64; ++c)
        tma_load_4d(smem + c * (kTile * 128), &tm_q, &ctl->q_full, c * 64, qb * BS, h, b);
      const int hk = h / p.kv_group;
      for (int j = 0; j < nblk; ++j) {
        const int s = j % NST;
        const uint32_t par = ((j / NST) & 1) ^ 1;
        const int key0 = checked_index(p.col_idx[peek && j == 0 ? first_blk : list0 + j], (p.Tk + BS - 1) / BS, p.status) * BS;
        if (!mbar_wait_bounded(&ctl->k_empty[s], par, abort_flag)) {
          record_status(p.status, kDevWaitStageEmpty);
          break;
        }
        mbar_expect_tx(&ctl->k_full[s], Cfg::kKVBytes);
#pragma unroll
        for (int c = 0; c < D / 64; ++c)
          tma_load_4d(smem + Cfg::kOffK + s * Cfg::kKVBytes + c * (BS * 128), &tm_k, &ctl->k_full[s], c * 64, key0, hk,
                      b);
        if (!mbar_wait_bounded(&ctl->v_empty[s], par, abort_flag)) {
          record_status(p.status, kDevWaitStageEmpty);
          break;
        }
        mbar_expect_tx(&ctl->v_full[s], Cfg::kKVBytes);
#pragma unroll
        for (int c = 0; c < D / 64; ++c)
          tma_load_4d(smem + Cfg::kOffV + s * Cfg::kKVBytes + c * (BS * 128), &tm_v, &ctl->v_full[s], c * 64, key0, hk,
                      b);
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer
    if (lane == 0 && nblk > 0) {
      const uint32_t q_addr = smem_u32(smem);
      const uint32_t k_addr = smem_u32(smem + Cfg::kOffK);
      const uint32_t v_addr = smem_u32(smem + Cfg::kOffV);
      bool ok = mbar_wait_bounded(&ctl->q_full, 0, abort_flag);
      if (!ok) record_status(p.status, kDevWaitQ);
      for (int j = 0; ok && j < nblk; ++j) {
        const int s = j % NST;
        const uint32_t par = (j / NST) & 1;
        if (!mbar_wait_bounded(&ctl->k_full[s], par, abort_flag)) {
          record_status(p.status, kDevWaitTmaFull);
          break;
        }
        // S(j) overwrites the columns PV(j-1) reads P from
        if (j > 0 && !mbar_wait_bounded(&ctl->pv_done, (j - 1) & 1, abort_flag)) {
          record_status(p.status, kDevWaitPvDone);
          break;
        }
        tc_fence_after();
        const uint64_t da = smem_desc_sw128(q_addr);
        const uint64_t db = smem_desc_sw128(k_addr + s * Cfg::kKVBytes);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          // 64-element halves of the head dimension are separate swizzled tiles
          const uint64_t offa = (ks >> 2) * (kTile * 128 / 16) + (ks & 3) * 2;
          const uint64_t offb = (ks >> 2) * (BS * 128 / 16) + (ks & 3) * 2;
          umma_f16_ss(tmem_base, da + offa, db + offb, kIdescQK, ks > 0);
        }
        umma_commit(&ctl->k_empty[s]);
        umma_commit(&ctl->s_full);
        if (!mbar_wait_bounded(&ctl->v_full[s], par, abort_flag)) {
          record_status(p.status, kDevWaitTmaFull);
          break;
        }
        // V block: rows = keys (128 bytes per 64 head-dim elements), column halves BS*128 bytes apart
        const uint64_t dv = smem_desc_sw128(v_addr + s * Cfg::kKVBytes, BS * 128);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          if (ok && !mbar_wait_bounded(&ctl->p_full[half], j & 1, abort_flag)) {
            record_status(p.status, kDevWaitPReady);
            ok = false;
          }
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int ks = half * (BS / 32); ks < (half + 1) * (BS / 32); ++ks)
            umma_f16_ts(tmem_base + Cfg::kColO, tmem_base + ks * 8, dv + ks * 128, kIdescPV, (j > 0 || ks > 0));
        }
        if (!ok) break;
        umma_commit(&ctl->v_empty[s]);
        umma_commit(&ctl->pv_done);
      }
    }
  } else {
    // ----------------------------------------------------------------- softmax
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const int qrow = qb * BS + row;
    const bool live = quarter * 32 < BS;       // BS = 64: the upper two row quarters hold no query
    const bool row_ok = row < BS && qrow < p.Tq;
    const uint32_t s_col = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t o_col = s_col + Cfg::kColO;
    const float sc = p.scale_log2;
    const float ninf = -__int_as_float(0x7f800000);
    const int reach = p.reach;
    const int dil = p.dilation > 0 ? p.dilation : 1;

    float m_used = ninf;
    float lh[2] = {0.f, 0.f};                  // probability sums of the two halves of the key columns
    bool ok = true;
    int key_next = nblk > 0 ? p.col_idx[peek ? first_blk : list0] : 0;
    for (int j = 0; j < nblk; ++j) {
      const int key0 = checked_index(key_next, (p.Tk + BS - 1) / BS, p.status) * BS;
      if (j + 1 < nblk) key_next = p.col_idx[list0 + j + 1];
      // S(j) computed, which also means that PV(j-1) has retired (the issuer waited for it)
      if (!mbar_wait_bounded(&ctl->s_full, j & 1, abort_flag)) {
        record_status(p.status, kDevWaitAccFull);
        ok = false;
      }
      if (!__all_sync(0xffffffffu, ok)) {        // (the whole warp gives up together)
        ok = false;
        break;
      }
      tc_fence_after();
      if (live) {
        uint32_t s[BS];
#pragma unroll
        for (int c = 0; c < BS / 32; ++c) tmem_ld32(s_col + c * 32, *reinterpret_cast<uint32_t(*)[32]>(s + c * 32));
        tc_wait_ld();
        // Which columns the row attends.  Token-pattern mode: a block whose every (query, key) pair
        // lies inside the window (no CLS row or column involved, dilation 1) needs no mask.
        bool inside = false;
        if (p.mode != 0 && dil == 1 && qb * BS >= p.num_cls && key0 >= p.num_cls) {
          const int q0 = qb * BS, far = max(q0 + BS - 1 - key0, key0 + BS - 1 - q0);
          inside = far <= reach;
        }
        if ((p.mode != 0 && !inside) || key0 + BS > p.Tk) {
#pragma unroll
          for (int c = 0; c < BS / 32; ++c) {
            const int base = key0 + c * 32;
            uint32_t w = low_bits(p.Tk - base);
            if (p.mode != 0 && !inside) w &= static_pattern_word(qrow, base, p.num_cls, reach, dil);
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (!((w >> i) & 1u)) s[c * 32 + i] = __float_as_uint(ninf);
          }
        }
        float m0 = ninf, m1 = ninf, m2 = ninf, m3 = ninf;
#pragma unroll
        for (int i = 0; i < BS; i += 8) {
          m0 = max3(m0, __uint_as_float(s[i]), __uint_as_float(s[i + 1]));
          m1 = max3(m1, __uint_as_float(s[i + 2]), __uint_as_float(s[i + 3]));
          m2 = max3(m2, __uint_as_float(s[i + 4]), __uint_as_float(s[i + 5]));
          m3 = max3(m3, __uint_as_float(s[i + 6]), __uint_as_float(s[i + 7]));
        }
        const float m_new = fmaxf(m_used, fmaxf(max3(m0, m1, m2), m3) * sc);
        if (__any_sync(0xffffffffu, m_new > m_used + kStep)) {
          // raise the stabiliser, rescale what has been accumulated
          const float factor = (m_new == m_used) ? 1.f : ex2_approx(m_used - m_new);
          lh[0] *= factor;
          lh[1] *= factor;
          m_used = m_new;
          if (j > 0) {
#pragma unroll 1
            for (int c = 0; c < D / 16; ++c) {
              uint32_t o[16];
              tmem_ld16(o_col + c * 16, o);
              tc_wait_ld();
#pragma unroll
              for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
              tmem_st16(o_col + c * 16, o);
            }
          }
        }
        // rows that have attended nothing yet have m_used = -inf; their stabiliser is 0 for now
        // (the looked-at block of a later chunk contributes nothing)
        const float neg_m = peek && j == 0 ? ninf : ((m_used == ninf) ? 0.f : -m_used);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float l0 = 0.f, l1 = 0.f;
#pragma unroll
          for (int u = half * (BS / 32); u < (half + 1) * (BS / 32); ++u) {
            uint32_t packed[8];
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
              float x0, x1;
              fma_pair(x0, x1, __uint_as_float(s[u * 16 + i]), __uint_as_float(s[u * 16 + i + 1]), sc, neg_m);
              x0 = ex2_approx(x0);
              x1 = ex2_approx(x1);
              add_pair(l0, l1, x0, x1);
              packed[i >> 1] = pack_bf16x2(x0, x1);
            }
            tmem_st8(s_col + u * 8, packed);
          }
          lh[half] += l0 + l1;
          tc_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->p_full[half]);
        }
      } else if (lane == 0) {
        mbar_arrive(&ctl->p_full[0]);
        mbar_arrive(&ctl->p_full[1]);
      }
    }

    if (nblk > 0 && ok && !mbar_wait_bounded(&ctl->pv_done, (nblk - 1) & 1, abort_flag)) {
      record_status(p.status, kDevWaitPvDone);
      ok = false;
    }
    float l = lh[0] + lh[1];
    tc_fence_after();

    // One chunk of a long list: leave the unnormalised rows, take a ticket; the last CTA of the query
    // block goes on with the sum over all chunks.
    auto slot = [&](int c) { return (bh * 2 + (c == 0)) * static_cast<int64_t>(p.extra) + ubase + (c == 0 ? 0 : c - 1); };
    bool writer = true;
    if (nch > 1) {
      const int64_t u = slot(ch);
      if (ok) {
        if (row_ok) p.part_ml[u * BS + row] = make_float2(m_used, l);
        float* po = p.part_o + (u * BS + row) * D;
#pragma unroll 1
        for (int c = 0; c < D / 16; ++c) {
          uint32_t o[16];
          tmem_ld16(o_col + c * 16, o);
          tc_wait_ld();
          if (!row_ok) continue;
#pragma unroll
          for (int i = 0; i < 16; i += 4)
            *reinterpret_cast<uint4*>(po + c * 16 + i) = make_uint4(o[i], o[i + 1], o[i + 2], o[i + 3]);
        }
      }
      __threadfence();
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (threadIdx.x == 64) ctl->ticket = atomicAdd(p.tickets + static_cast<int64_t>(bh) * p.nQB + qb, 1u);
      asm volatile("bar.sync 1, 128;" ::: "memory");
      writer = ctl->ticket + 1 == static_cast<uint32_t>(nch);
      if (writer) __threadfence();
    }
    if (ok && writer) {
      float wgt_m = m_used;
      if (nch > 1 && row_ok) {
        for (int c = 0; c < nch; ++c) {
          const int64_t u = slot(c);
          wgt_m = fmaxf(wgt_m, __ldcg(p.part_ml + u * BS + row).x);
        }
        l = 0.f;
        for (int c = 0; c < nch; ++c) {
          const int64_t u = slot(c);
          const float2 ml = __ldcg(p.part_ml + u * BS + row);
          l += ml.y * (ml.x == wgt_m ? 1.f : ex2_approx(ml.x - wgt_m));    // (a chunk without keys: 0 * 0)
        }
      }
      const float inv = l > 0.f ? 1.f / l : 0.f;
      if (p.lse != nullptr && row_ok) {
        p.lse[(static_cast<int64_t>(b) * p.H + h) * p.Tq + qrow] =
            l > 0.f ? (wgt_m + log2f(l)) * 0.6931471805599453f : ninf;
      }
#pragma unroll 1
      for (int c = 0; c < D / 16; ++c) {
        uint32_t o[16];
        if (nch > 1) {
          float acc[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) acc[i] = 0.f;
          for (int k = 0; row_ok && k < nch; ++k) {
            const int64_t u = slot(k);
            const float mk = __ldcg(p.part_ml + u * BS + row).x;
            const float f = mk == wgt_m ? 1.f : ex2_approx(mk - wgt_m);    // (no chunk is left out: a NaN stays NaN)
            const float4* po = reinterpret_cast<const float4*>(p.part_o + (u * BS + row) * D + c * 16);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float4 v = __ldcg(po + i);
              acc[4 * i] = fmaf(v.x, f, acc[4 * i]);
              acc[4 * i + 1] = fmaf(v.y, f, acc[4 * i + 1]);
              acc[4 * i + 2] = fmaf(v.z, f, acc[4 * i + 2]);
              acc[4 * i + 3] = fmaf(v.w, f, acc[4 * i + 3]);
            }
          }
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(acc[i]);
        } else if (nblk > 0) {
          tmem_ld16(o_col + c * 16, o);
          tc_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = 0u;
        }
        if (!row_ok) continue;
        if (p.gate != nullptr) {
          // gated accumulate: value = acc_in + sigmoid(g) * (o * inv), the order the stand-alone
          // gate kernel adds the branches in
          const float gl = p.gate[((static_cast<int64_t>(b) * p.Tq + qrow) * p.H + h) * 3 + p.gate_idx];
          const float gs = 1.f / (1.f + __expf(-gl));
          const float* arow = p.acc_in == nullptr ? nullptr
                                                  : p.acc_in + ((static_cast<int64_t>(b) * p.H + h) * p.Tq + qrow) * D + c * 16;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float a = __uint_as_float(o[i]) * inv;
            o[i] = __float_as_uint(arow == nullptr ? gs * a : fmaf(gs, a, arow[i]));
          }
        }
        const float inv_w = p.gate != nullptr ? 1.f : inv;      // (already applied above)
        if (p.o_dtype == SWV_F32) {
          float* orow = static_cast<float*>(p.o) + b * p.osb + h * p.osh + qrow * p.ost + c * 16;
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            *reinterpret_cast<float4*>(orow + i) =
                make_float4(__uint_as_float(o[i]) * inv_w, __uint_as_float(o[i + 1]) * inv_w,
                            __uint_as_float(o[i + 2]) * inv_w, __uint_as_float(o[i + 3]) * inv_w);
          }
        } else {
          uint16_t* orow = static_cast<uint16_t*>(p.o) + b * p.osb + h * p.osh + qrow * p.ost + c * 16;
#pragma unroll
          for (int i = 0; i < 16; i += 8) {
            uint32_t w4[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const float a0 = __uint_as_float(o[i + 2 * q]) * inv_w, a1 = __uint_as_float(o[i + 2 * q + 1]) * inv_w;
              if (p.o_dtype == SWV_BF16) {
                w4[q] = pack_bf16x2(a0, a1);
              } else {
                const __half2 h2 = __floats2half2_rn(a0, a1);
                w4[q] = *reinterpret_cast<const uint32_t*>(&h2);
              }
            }
            *reinterpret_cast<uint4*>(orow + i) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    __syncwarp();
    tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

// ------------------------------------------------------------------ 2-D RoPE
// x (L, H, hd) rotated in place-compatible fashion into y: first half of the head uses
// coords[:,0], second half coords[:,1]; hd/4 frequencies theta^(-2i/(hd/2)), each for two
// adjacent channels; (x0, x1) -> (x0 cos - x1 sin, x1 cos + x0 sin)
// (src/sparse_wsi_vit/models/vit_5/rope.py:33-37, 56-59, 81-97).  Tokens < skip are copied.
// One thread per token and channel pair: the angle is the same for every head (4097 tokens of 6 heads: 8.6 us
// with a sine and cosine per head, 4.1 us).
template <typename T>
__global__ void rope2d_kernel(const T* x, T* y /* may be x */, const float* __restrict__ coords,
                              int64_t L, int H, int hd, int64_t xs_l, int64_t xs_h, int64_t ys_l, int64_t ys_h,
                              float inv_high, float log2_theta, int skip, bool vec) {
  const int64_t gid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int pairs = hd / 2;
  if (gid >= L * pairs) return;
  const int pr = static_cast<int>(gid % pairs);
  const int64_t t = gid / pairs;
  const T* xp = x + t * xs_l + 2 * pr;
  T* yp = y + t * ys_l + 2 * pr;
  if (t < skip) {                                       // copied as they are
    for (int hh = 0; hh < H; ++hh) {
      yp[hh * ys_h] = xp[hh * xs_h];
      yp[hh * ys_h + 1] = xp[hh * xs_h + 1];
    }
    return;
  }
  const int half_pairs = pairs / 2;                     // pairs per coordinate axis
  const int axis = pr >= half_pairs ? 1 : 0;
  const int f = pr - axis * half_pairs;                 // frequency index
  const int dim = hd / 2;
  const float freq = exp2f(-log2_theta * (2.0f * f) / dim);
  const float ang = __fmul_rn(__fmul_rn(coords[t * 2 + axis], inv_high), freq);
  float sn, cs;
  sincosf(ang, &sn, &cs);
  rope_heads(xp, xs_h, yp, ys_h, H, cs, sn, vec);
}

// Mean pooling of overlapping token windows: y[b,h,c,:] = mean_{i < win} x[b,h,c*stride + i,:]
// (the compressed keys / values of the NSA compressed branch).  One thread per output pair of channels.
__global__ void pool_tokens_kernel(const __nv_bfloat16* __restrict__ x, int64_t sb, int64_t sh, int64_t st_,
                                   __nv_bfloat16* __restrict__ y, int B, int H, int T, int D, int nC, int win,
                                   int stride) {
  const int64_t gid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int pairs = D / 2;
  const int64_t total = static_cast<int64_t>(B) * H * nC * pairs;
  if (gid >= total) return;
  const int pr = static_cast<int>(gid % pairs);
  const int c = static_cast<int>((gid / pairs) % nC);
  const int h = static_cast<int>((gid / (static_cast<int64_t>(pairs) * nC)) % H);
  const int b = static_cast<int>(gid / (static_cast<int64_t>(pairs) * nC * H));
  const __nv_bfloat16* xp = x + b * sb + h * sh + static_cast<int64_t>(c) * stride * st_ + 2 * pr;
  float a0 = 0.f, a1 = 0.f;
  for (int i = 0; i < win; ++i) {
    const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(xp + i * st_);
    a0 += __bfloat162float(v.x);
    a1 += __bfloat162float(v.y);
  }
  const float inv = 1.0f / win;
  __nv_bfloat162 o;
  o.x = __float2bfloat16_rn(a0 * inv);
  o.y = __float2bfloat16_rn(a1 * inv);
  *reinterpret_cast<__nv_bfloat162*>(y + ((static_cast<int64_t>(b) * H + h) * nC + c) * D + 2 * pr) = o;
}

// ---------------------------------------------------------------------- host
static bool bsa_aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <int BS, int D>
static int launch_bsa(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const BsaParams& p,
                      cudaStream_t st) {
  using Cfg = BsaCfg<BS, D>;
  SWV_CUDA_OK(cudaFuncSetAttribute(block_sparse_attn_kernel<BS, D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(Cfg::kSmem)));
  const unsigned grid = static_cast<unsigned>(p.B) * (p.nQB + p.extra) * p.H;
  block_sparse_attn_kernel<BS, D><<<grid, kBsaThreads, Cfg::kSmem, st>>>(tq, tk, tv, p);
  SWV_CUDA_OK(cudaGetLastError());
  return SWV_OK;
}

// How long lists are divided, from the sizes the host knows (`nnz` = entries of col_idx).  A chunk is
// never shorter than 8 key blocks (a partial row block costs about one block's time to write and read
// back), than twice the mean list (regular lists stay whole), or than an even share of all work over
// the resident CTAs (a list below that does not reach past the end of the launch).
struct BsaSplit {
  int chunk = 0, extra = 0;
  size_t o_bytes = 0, ml_bytes = 0, ticket_bytes = 0;
};
static BsaSplit bsa_split(int B, int H, int nQB, int nKB, int block, int D, int64_t nnz) {
  BsaSplit s;
  if (nnz <= 0) return s;
  const int64_t slots = static_cast<int64_t>(sm_count()) * (block + D <= 128 ? 3 : 2);
  const int64_t mean2 = (2 * nnz + nQB - 1) / nQB, share = (nnz * B * H + slots - 1) / slots;
  const int64_t chunk = mean2 > share ? (mean2 > 8 ? mean2 : 8) : (share > 8 ? share : 8);
  if (chunk >= nKB) return s;                       // no list can be longer
  s.chunk = static_cast<int>(chunk);
  s.extra = static_cast<int>(nnz / chunk);          // sum over rows of ceil(n / chunk) - 1 <= nnz / chunk
  if (s.extra == 0) s.chunk = 0;
  const size_t rows = static_cast<size_t>(B) * H * 2 * s.extra * block;     // (a divided list has an extra unit or more)
  s.o_bytes = rows * D * sizeof(float);
  s.ml_bytes = rows * sizeof(float2);
  s.ticket_bytes = static_cast<size_t>(B) * H * nQB * sizeof(uint32_t);
  return s;
}

int block_sparse_workspace_bytes_impl(int B, int H, int Tq, int Tk, int D, int block, int64_t nnz, size_t* bytes) {
  if (!bytes) return SWV_ERR_NULL;
  if (B < 1 || H < 1 || Tq < 1 || Tk < 1 || nnz < 0) return SWV_ERR_SHAPE;
  if ((block != 64 && block != 128) || (D != 64 && D != 128)) return SWV_ERR_UNSUPPORTED;
  const BsaSplit s = bsa_split(B, H, (Tq + block - 1) / block, (Tk + block - 1) / block, block, D, nnz);
  *bytes = s.extra > 0 ? s.o_bytes + s.ml_bytes + s.ticket_bytes : 0;
  return SWV_OK;
}

int block_sparse_attn_impl(const void* q, const int64_t* qs, const void* k, const int64_t* ks, const void* v,
                           const int64_t* vs, const int32_t* row_ptr, const int32_t* col_idx, int block, int mode,
                           int num_cls, int window, int dilation, int kv_group, float* lse, void* o,
                           const int64_t* os, int o_dtype, int B, int H, int Tq, int Tk, int D, int* status,
                           cudaStream_t st, const float* gate, int gate_idx, const float* acc_in, int64_t nnz,
                           void* workspace, size_t workspace_bytes) {
  if (!q || !k || !v || !row_ptr || !col_idx || !o || !status || !qs || !ks || !vs || !os) return SWV_ERR_NULL;
  if (B < 1 || H < 1 || Tq < 1 || Tk < 1) return SWV_ERR_SHAPE;
  if (kv_group < 1 || H % kv_group != 0) return SWV_ERR_SHAPE;
  if ((block != 64 && block != 128) || (D != 64 && D != 128)) return SWV_ERR_UNSUPPORTED;
  if (mode != 0 && mode != 1) return SWV_ERR_UNSUPPORTED;
  if (mode == 1 && (num_cls < 0 || window < 0 || dilation < 1)) return SWV_ERR_SHAPE;
  if (o_dtype != SWV_F32 && o_dtype != SWV_BF16 && o_dtype != SWV_F16) return SWV_ERR_DTYPE;
  const int64_t* ss[3] = {qs, ks, vs};
  const void* ps[3] = {q, k, v};
  for (int i = 0; i < 3; ++i) {
    if (ss[i][3] != 1 || !bsa_aligned16(ps[i])) return SWV_ERR_ALIGN;
    if ((ss[i][0] * 2) % 16 || (ss[i][1] * 2) % 16 || (ss[i][2] * 2) % 16) return SWV_ERR_ALIGN;
  }
  const int osz = o_dtype == SWV_F32 ? 4 : 2;
  if (os[3] != 1 || !bsa_aligned16(o) || (os[0] * osz) % 16 || (os[1] * osz) % 16 || (os[2] * osz) % 16)
    return SWV_ERR_ALIGN;

  CUtensorMap tq, tk, tv;
  int rc = make_tmap_4d(&tq, q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, D, Tq, H, B, qs[2] * 2, qs[1] * 2, qs[0] * 2, 64,
                        kTile);
  if (rc != SWV_OK) return rc;
  const int Hkv = H / kv_group;
  rc = make_tmap_4d(&tk, k, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, D, Tk, Hkv, B, ks[2] * 2, ks[1] * 2, ks[0] * 2, 64, block);
  if (rc != SWV_OK) return rc;
  rc = make_tmap_4d(&tv, v, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, D, Tk, Hkv, B, vs[2] * 2, vs[1] * 2, vs[0] * 2, 64, block);
  if (rc != SWV_OK) return rc;

  BsaParams p;
  p.B = B; p.H = H; p.Tq = Tq; p.Tk = Tk;
  p.nQB = (Tq + block - 1) / block;
  p.row_ptr = row_ptr; p.col_idx = col_idx;
  p.mode = mode; p.num_cls = num_cls; p.dilation = dilation;
  // (the bound keeps every sum of a position and the reach within 32 bits)
  p.reach = static_cast<int>(std::min<int64_t>(static_cast<int64_t>(window) * dilation, static_cast<int64_t>(Tq) + Tk));
  p.kv_group = kv_group; p.lse = lse;
  p.gate = gate; p.gate_idx = gate_idx; p.acc_in = acc_in;
  p.o = o; p.osb = os[0]; p.osh = os[1]; p.ost = os[2]; p.o_dtype = o_dtype;
  p.scale_log2 = 1.4426950408889634f / sqrtf(static_cast<float>(D));
  p.status = status;
  p.chunk = 0; p.extra = 0;
  p.part_o = nullptr; p.part_ml = nullptr; p.tickets = nullptr;
  if (workspace != nullptr) {
    const BsaSplit s = bsa_split(B, H, p.nQB, (Tk + block - 1) / block, block, D, nnz);
    if (s.extra > 0) {
      if (workspace_bytes < s.o_bytes + s.ml_bytes + s.ticket_bytes) return SWV_ERR_WORKSPACE;
      if (!bsa_aligned16(workspace)) return SWV_ERR_ALIGN;
      uint8_t* w = static_cast<uint8_t*>(workspace);
      p.chunk = s.chunk; p.extra = s.extra;
      p.part_o = reinterpret_cast<float*>(w);
      p.part_ml = reinterpret_cast<float2*>(w + s.o_bytes);
      p.tickets = reinterpret_cast<uint32_t*>(w + s.o_bytes + s.ml_bytes);
      SWV_CUDA_OK(cudaMemsetAsync(p.tickets, 0, s.ticket_bytes, st));
    }
  }
  if (block == 64 && D == 64) return launch_bsa<64, 64>(tq, tk, tv, p, st);
  if (block == 64 && D == 128) return launch_bsa<64, 128>(tq, tk, tv, p, st);
  if (block == 128 && D == 64) return launch_bsa<128, 64>(tq, tk, tv, p, st);
  return launch_bsa<128, 128>(tq, tk, tv, p, st);
}

int pool_tokens_impl(const void* x, const int64_t* xs, void* y, int B, int H, int T, int D, int win, int stride,
                     cudaStream_t st) {
  if (!x || !y || !xs) return SWV_ERR_NULL;
  if (B < 1 || H < 1 || T < win || win < 1 || stride < 1 || D < 2 || (D & 1)) return SWV_ERR_SHAPE;
  if (xs[3] != 1 || (xs[0] & 1) || (xs[1] & 1) || (xs[2] & 1) || (reinterpret_cast<uintptr_t>(x) & 3)) return SWV_ERR_ALIGN;
  const int nC = (T - win) / stride + 1;
  const int64_t total = static_cast<int64_t>(B) * H * nC * (D / 2);
  pool_tokens_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, st>>>(
      static_cast<const __nv_bfloat16*>(x), xs[0], xs[1], xs[2], static_cast<__nv_bfloat16*>(y), B, H, T, D, nC, win,
      stride);
  SWV_CUDA_OK(cudaGetLastError());
  return SWV_OK;
}

int rope2d_impl(const void* x, const int64_t* xs, void* y, const int64_t* ys, int dtype, const float* coords,
                int64_t L, int H, int hd, float coord_high, float theta, int skip, cudaStream_t st) {
  if (!x || !y || !coords || !xs || !ys) return SWV_ERR_NULL;
  if (L < 1 || H < 1 || hd < 4 || (hd % 4) != 0 || coord_high == 0.f || theta <= 0.f || skip < 0) return SWV_ERR_SHAPE;
  if (xs[2] != 1 || ys[2] != 1) return SWV_ERR_ALIGN;
  if (dtype != SWV_F32 && dtype != SWV_BF16) return SWV_ERR_DTYPE;
  const unsigned grid = static_cast<unsigned>((L * (hd / 2) + 255) / 256);
  const int es = dtype == SWV_F32 ? 4 : 2;
  const bool vec = rope_vec_ok(x, xs[0], xs[1], 0, es) && rope_vec_ok(y, ys[0], ys[1], 0, es);
  if (dtype == SWV_F32) {
    rope2d_kernel<float><<<grid, 256, 0, st>>>(static_cast<const float*>(x), static_cast<float*>(y), coords, L, H, hd,
                                               xs[0], xs[1], ys[0], ys[1], 1.0f / coord_high, log2f(theta), skip, vec);
  } else {
    rope2d_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(static_cast<const __nv_bfloat16*>(x),
                                                       static_cast<__nv_bfloat16*>(y), coords, L, H, hd, xs[0], xs[1],
                                                       ys[0], ys[1], 1.0f / coord_high, log2f(theta), skip, vec);
  }
  SWV_CUDA_OK(cudaGetLastError());
  return SWV_OK;
}

}  // namespace swv
