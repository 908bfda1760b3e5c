// Backward of a DSA layer on the tensor cores, for selections this library's own indexer made
// (ascending key lists; their membership bitmask is rebuilt from them): gradients of the routing-weighted attention
// (src/sparse_wsi_vit/models/deepseek_sparse_attention_kernels/kernels.py:569-762) and of the indexer
// (:128-339), the same formulas as the list kernels in dsa_bwd.cu, which serve every other case.
//
//   sm_ij = exp(logit_ij - m_i) / max(l_i, 1e-6)     P_ij = sm_ij w_ij          (member pairs only)
//   g_ij  = sm_ij (dO_i . v_j - D_i)                 dS_ij = w_ij g_ij
//   dV_j = sum_i P_ij dO_i    dK_j = scale sum_i dS_ij q_i    dQ_i = scale sum_j dS_ij k_j
//   drw_ij = sum_heads g_ij   dq_idx = W sum_j drw_ij k_idx_j   dk_idx = W sum_i drw_ij q_idx_i
//
// Three sweeps over 128 x 64 tiles of (lane side) x (streamed side), one kernel:
//   kStats : lanes = queries, keys streamed: exact row maximum m_i and 1 / max(l_i, 1e-6) in fp32 (kept apart:
//            one log-sum-exp of both would round by 2^-24 of its own size, a factor common to the whole row)
//   kDkv   : lanes = keys, queries streamed: dV, dK; every head's g_ij stored in list order (the slot of a
//            member is its rank in the row's bitmask), summed over the heads afterwards
//   kDq    : lanes = queries, keys streamed: dQ
// Every tile's logits S, routing weights R (TF32, from the collapsed indexer vectors: the forward's own
// products) and dP = dO V^T come from tcgen05 products into one of two TMEM buffers; sixteen warps turn
// them into P and dS, which go back into the very columns they came from, as the A operand (TMEM) of the
// gradient products.  P and dS are fp32 values: each is split into THREE bf16 terms (24 bits) that are
// multiplied one after the other, so no product sees fewer bits than the CUDA-core form.  The tensor cores
// truncate at every accumulation step, always towards zero (2^-27 of the result per step, 9e-6 after the
// 1128 steps of 6009 keys), so an accumulator holds ONE tile's products, those of the smallest terms first:
// the warps add it to fp32 registers (round to nearest) before they hand over the next tile.  Error against
// fp64 (1024 to 16384 tokens): 1.4e-7 to 3.5e-7 of every gradient (dq_idx 7.8e-7 at 1024 tokens with the
// largest terms first), the list kernels 4.1e-7 to 8.4e-7.  q, k, v are bf16; dO must be exact in bf16 as well (it is whenever the next layer ran in bf16) -- where it is not,
// these kernels return at once and the list kernel runs.
//
// A pair that is not a member is multiplied with zero, not skipped: a NaN or an infinity in one row of q, k, v or
// dO can reach every gradient of its head (the list kernels keep it to the selected pairs).
//
// Bound: kDkv by the instructions of the sixteen warps (63 % of the issue slots, tensor pipe 21 % of the time),
// kStats and kDq by the chain products -> terms -> gradient products of two buffers (47 and 42 % of the issue
// slots, tensor pipe 20 and 23 %; ncu at 8192 tokens).  16384 tokens, 8 heads, top-2048: kStats 1.6, kDkv 4.9,
// kDq 3.2 ms; kDkv took 5.8 ms with eight warps, a branch around the list store, and a block barrier per tile
// for the column data, while the accumulators still ran over the whole row.
// The list kernels move 3 rows and reduce 2 per selected pair: 43.7 + 13.4 ms with the indexer's part on the
// same input against 11.4 ms.  They do T * K work, the tiles T^2: the two meet at about one key in 40.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace swv {
namespace {

enum { kStats = 0, kDkv = 1, kDq = 2 };
constexpr int kNW = 64;                 // streamed rows per tile
constexpr int kBwdStages = 4;
constexpr int kHd = 64;                 // head dimension
constexpr int kLBytes = kTile * kHd * 2;            // 16 KiB: lane-side bf16 tile
constexpr int kLRBytes = kTile * kIdxDim * 4;       // 32 KiB: lane-side collapsed indexer vectors
constexpr int kSBytes = kNW * kHd * 2;              // 8 KiB
constexpr int kSRBytes = kNW * kIdxDim * 4;         // 16 KiB
constexpr int kOffL2 = kLBytes;
constexpr int kOffLR = 2 * kLBytes;
constexpr int kOffStage = 2 * kLBytes + kLRBytes;
constexpr int kStageB = 2 * kSBytes + kSRBytes;
constexpr int kOffCols = kOffStage + kBwdStages * kStageB;

// per streamed query (kDkv), double-buffered
struct BwdCols {
  float4 f[kNW];                        // {row maximum, 1 / l, D, -}
  uint2 mem[4][kNW];                    // per 32 keys: {membership word, list position of its first member}
};
struct BwdCtl {
  uint64_t l_full, full[kBwdStages], empty[kBwdStages];
  uint64_t in_full[2], p_ready[2], acc_done;
  uint32_t tmem_base, abort_flag;
  float xm[4][kTile], xl[4][kTile], xe[4][kTile];
};
constexpr int kOffBwdCtl = kOffCols + 2 * static_cast<int>(sizeof(BwdCols));
constexpr size_t kBwdSmem = 1024 + kOffBwdCtl + sizeof(BwdCtl) + 64;
constexpr uint32_t kBufCols = 192;      // S 64 | R 64 | dP 64, two buffers (four narrower ones for kStats gained 1 %)
constexpr uint32_t kColAcc = 384;       // dV (or dQ) 64 | dK 64

struct BwdTileParams {
  int B, H, Tq, Tk, nQT, nKT, top_k;
  int h0, Hn;               // heads of this launch: h0 .. h0 + Hn - 1
  const uint32_t* maskbits;
  const uint16_t* off;      // [B][nKT + 1][Tq] first list slot of row i with a key in tile kt or later
  const float* di;          // (B,H,Tq)
  float *rmax, *linv;       // (B,H,Tq): row maximum of the members' logits (log2 domain), 1 / max(l, 1e-6)
  float *dq, *dk, *dv;
  float* gh;                // [Hn][B*Tq*top_k] the heads' g in list order
  int r_steps;              // 8-channel steps of the routing-weight product (the rest of the 64 channels is zero)
  float scale, c2;          // 1/sqrt(D), and times log2 e
  const int* skip_if;       // non-zero: nothing to do here
  int* status;
};

// A pair of fp32 values as three bf16 pairs whose sum is the pair: each term takes the next 8 of the 24
// bits as they are (byte permutes; rounded conversions cost two issue slots each and gain nothing here).
__device__ __forceinline__ void split3(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
  a -= __uint_as_float(__float_as_uint(a) & 0xffff0000u);
  b -= __uint_as_float(__float_as_uint(b) & 0xffff0000u);
  mid = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
  a -= __uint_as_float(__float_as_uint(a) & 0xffff0000u);
  b -= __uint_as_float(__float_as_uint(b) & 0xffff0000u);
  lo = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}

// *p = x where `on`: one predicated store (a branch around it costs the warp its convergence bookkeeping)
__device__ __forceinline__ void st_global_if(float* p, float x, bool on) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.global.f32 [%0], %1;\n\t}" ::"l"(p), "f"(x),
               "r"(static_cast<uint32_t>(on))
               : "memory");
}

constexpr int kBwdEpi = 16;             // warps that turn a tile's products into its terms, 16 columns each
constexpr int bwd_threads(int mode) { return 64 + 32 * kBwdEpi + (mode == kDkv ? 64 : 0); }

template <int MODE>
__global__ void __launch_bounds__(bwd_threads(MODE), 1)
    dsa_bwd_tiles_kernel(const __grid_constant__ CUtensorMap tm_l1, const __grid_constant__ CUtensorMap tm_l2,
                         const __grid_constant__ CUtensorMap tm_lr, const __grid_constant__ CUtensorMap tm_s1,
                         const __grid_constant__ CUtensorMap tm_s2, const __grid_constant__ CUtensorMap tm_sr,
                         const BwdTileParams p) {
  constexpr uint32_t kIdescQK = make_idesc(/*bf16*/ 1, kTile, kNW, 0, 0);
  constexpr uint32_t kIdescR = make_idesc(/*tf32*/ 2, kTile, kNW, 0, 0);
  constexpr uint32_t kIdescAcc = make_idesc(/*bf16*/ 1, kTile, kHd, 0, /*B is MN-major*/ 1);
  if (p.skip_if != nullptr && *p.skip_if != 0) return;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  BwdCols* cols = reinterpret_cast<BwdCols*>(smem + kOffCols);
  BwdCtl* ctl = reinterpret_cast<BwdCtl*>(smem + kOffBwdCtl);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nLT = MODE == kDkv ? p.nKT : p.nQT;
  const int lt = blockIdx.x % nLT;                       // lane-side tile
  const int h = p.h0 + (blockIdx.x / nLT) % p.Hn;
  const int b = blockIdx.x / (nLT * p.Hn);
  const int nS = ((MODE == kDkv ? p.Tq : p.Tk) + kNW - 1) / kNW;   // streamed tiles

  if (threadIdx.x == 0) {
    mbar_init(&ctl->l_full, 1);
    for (int s = 0; s < kBwdStages; ++s) {
      mbar_init(&ctl->full[s], 1);
      mbar_init(&ctl->empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&ctl->in_full[s], MODE == kDkv ? 3 : 1);    // the products and (kDkv) two warps of column data
      mbar_init(&ctl->p_ready[s], kBwdEpi);
    }
    mbar_init(&ctl->acc_done, 1);
    ctl->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&ctl->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;
  volatile uint32_t* abort_flag = &ctl->abort_flag;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      mbar_expect_tx(&ctl->l_full, kLBytes * (MODE == kStats ? 1 : 2) + kLRBytes);
      tma_load_4d(smem, &tm_l1, &ctl->l_full, 0, lt * kTile, h, b);
      if (MODE != kStats) tma_load_4d(smem + kOffL2, &tm_l2, &ctl->l_full, 0, lt * kTile, h, b);
#pragma unroll
      for (int c = 0; c < 2; ++c)
        tma_load_3d(smem + kOffLR + c * (kLRBytes / 2), &tm_lr, &ctl->l_full, c * 32, lt * kTile, b);
      for (int t = 0; t < nS; ++t) {
        const int s = t % kBwdStages;
        if (!mbar_wait_bounded(&ctl->empty[s], ((t / kBwdStages) & 1) ^ 1, abort_flag)) {
          record_status(p.status, kDevWaitStageEmpty);
          break;
        }
        uint8_t* st = smem + kOffStage + s * kStageB;
        mbar_expect_tx(&ctl->full[s], kSBytes * (MODE == kStats ? 1 : 2) + kSRBytes);
        tma_load_4d(st, &tm_s1, &ctl->full[s], 0, t * kNW, h, b);
        if (MODE != kStats) tma_load_4d(st + kSBytes, &tm_s2, &ctl->full[s], 0, t * kNW, h, b);
#pragma unroll
        for (int c = 0; c < 2; ++c)
          tma_load_3d(st + 2 * kSBytes + c * (kSRBytes / 2), &tm_sr, &ctl->full[s], c * 32, t * kNW, b);
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer
    if (lane == 0) {
      const uint32_t l1 = smem_u32(smem), l2 = l1 + kOffL2, lr = l1 + kOffLR, st0 = l1 + kOffStage;
      bool ok = mbar_wait_bounded(&ctl->l_full, 0, abort_flag);
      if (!ok) record_status(p.status, kDevWaitQ);
      // the gradient products of tile t
      auto accumulate = [&](int t) -> bool {
        if (!mbar_wait_bounded(&ctl->p_ready[t & 1], (t >> 1) & 1, abort_flag)) {
          record_status(p.status, kDevWaitPReady);
          return false;
        }
        tc_fence_after();
        const uint32_t buf = tmem_base + (t & 1) * kBufCols;
        const uint32_t st = st0 + (t % kBwdStages) * kStageB;
        const uint64_t d1 = smem_desc_sw128(st), d2 = smem_desc_sw128(st + kSBytes);
        // Smallest terms first: every accumulation truncates at the size of the sum so far, so only the
        // products of the leading terms (four of the twelve) do it at the size of the result.
#pragma unroll
        for (int term = 2; term >= 0; --term) {
#pragma unroll
          for (int ks = 0; ks < kNW / 16; ++ks) {
            // where the warps left the terms of these 16 streamed rows (see the epilogue): six groups of 8 columns
            const bool acc = term < 2 || ks > 0;
            const uint32_t c1 = buf + 16 * ks + (term == 0 ? 0 : term == 1 ? 8 : 64);
            const uint32_t c2 = buf + 16 * ks + (term == 0 ? 72 : term == 1 ? 128 : 136);
            if (MODE == kDkv) umma_f16_ts(tmem_base + kColAcc, c1, d2 + ks * 128, kIdescAcc, acc);
            umma_f16_ts(tmem_base + kColAcc + (MODE == kDkv ? 64 : 0), c2, d1 + ks * 128, kIdescAcc, acc);
          }
        }
        umma_commit(&ctl->empty[t % kBwdStages]);
        umma_commit(&ctl->acc_done);
        return true;
      };
      for (int t = 0; ok && t < nS; ++t) {
        const int s = t % kBwdStages;
        if (!mbar_wait_bounded(&ctl->full[s], (t / kBwdStages) & 1, abort_flag)) {
          record_status(p.status, kDevWaitTmaFull);
          ok = false;
          break;
        }
        // the buffer's columns are free: tile t - 2 has been multiplied (kStats: read)
        if (t >= 2 && !(MODE == kStats ? mbar_wait_bounded(&ctl->p_ready[t & 1], ((t >> 1) & 1) ^ 1, abort_flag)
                                       : mbar_wait_bounded(&ctl->acc_done, t & 1, abort_flag))) {
          record_status(p.status, kDevWaitAccEmpty);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t st = st0 + s * kStageB;
        const uint32_t buf = tmem_base + (t & 1) * kBufCols;
#pragma unroll
        for (int ks = 0; ks < kHd / 16; ++ks)
          umma_f16_ss(buf, smem_desc_sw128(l1) + ks * 2, smem_desc_sw128(st) + ks * 2, kIdescQK, ks > 0);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          if (ks < p.r_steps) umma_tf32_ss(buf + 64, smem_desc_sw128(lr + (ks >> 2) * (kLRBytes / 2) + (ks & 3) * 32),
                       smem_desc_sw128(st + 2 * kSBytes + (ks >> 2) * (kSRBytes / 2) + (ks & 3) * 32), kIdescR, ks > 0);
        if (MODE != kStats) {
#pragma unroll
          for (int ks = 0; ks < kHd / 16; ++ks)
            umma_f16_ss(buf + 128, smem_desc_sw128(l2) + ks * 2, smem_desc_sw128(st + kSBytes) + ks * 2, kIdescQK, ks > 0);
        } else {
          umma_commit(&ctl->empty[s]);
        }
        umma_commit(&ctl->in_full[t & 1]);
        if (MODE != kStats && t >= 1) ok = accumulate(t - 1);
      }
      if (MODE != kStats && ok) accumulate(nS - 1);
    }
  } else if (MODE == kDkv && warp >= 2 + kBwdEpi) {
    // ------------------------- two warps: the column data of the tiles, one streamed query per thread
    const int cc = (warp & 1) * 32 + lane;
    const int64_t bh = static_cast<int64_t>(b) * p.H + h;
    for (int t = 0; t < nS; ++t) {
      const int i = t * kNW + cc;
      uint4 mw = make_uint4(0u, 0u, 0u, 0u);
      uint32_t pos = 0;
      float4 f = make_float4(__int_as_float(0x7f800000), 0.f, 0.f, 0.f);   // rows behind the end: sm = 2^-inf = 0
      if (i < p.Tq) {
        mw = __ldg(reinterpret_cast<const uint4*>(p.maskbits) +
                   ((static_cast<int64_t>(b) * p.nQT + (i >> 7)) * p.nKT + lt) * kTile + (i & 127));
        const int first = __ldg(p.off + (static_cast<int64_t>(b) * (p.nKT + 1) + lt) * p.Tq + i);
        pos = (static_cast<uint32_t>(b) * p.Tq + i) * p.top_k + first;
        // (a bitmask that does not belong to the list: nothing is stored outside the row)
        if (first + __popc(mw.x) + __popc(mw.y) + __popc(mw.z) + __popc(mw.w) > p.top_k) {
          record_status(p.status, kDevBadIndex);
          mw = make_uint4(0u, 0u, 0u, 0u);
        }
        f.x = __ldg(p.rmax + bh * p.Tq + i);
        f.y = __ldg(p.linv + bh * p.Tq + i);
        f.z = __ldg(p.di + bh * p.Tq + i);
      }
      // tile t - 2 has been turned into its terms: its column data are no longer read
      bool ok = t < 2 || mbar_wait_bounded(&ctl->p_ready[t & 1], ((t >> 1) & 1) ^ 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        record_status(p.status, kDevWaitPReady);
        break;
      }
      BwdCols& c = cols[t & 1];
      c.f[cc] = f;
      const uint32_t w[4] = {mw.x, mw.y, mw.z, mw.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        c.mem[q][cc] = make_uint2(w[q], pos);
        pos += __popc(w[q]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->in_full[t & 1]);
    }
  } else {
    // ------------------------------------------ sixteen warps: (lane quarter, 16 of the 64 columns)
    const int quarter = warp & 3;
    const int grp = (warp - 2) >> 2;
    const int c0 = grp * 16;                              // streamed rows c0 .. c0 + 15 = one k-step of the products
    const int row = quarter * 32 + lane;
    const int lrow = lt * kTile + row;                    // query (kStats, kDq) or key (kDkv)
    const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
    const float ninf = -__int_as_float(0x7f800000);
    const float c2 = p.c2;
    const int64_t bh = static_cast<int64_t>(b) * p.H + h;
    const bool row_ok = lrow < (MODE == kDkv ? p.Tk : p.Tq);
    constexpr int kAcc = MODE == kDkv ? 32 : 16;          // this warp's columns of the accumulators
    const uint32_t acc_col = tmem_base + lane_off + kColAcc + grp * kAcc;
    float acc[kAcc];
#pragma unroll
    for (int i = 0; i < kAcc; ++i) acc[i] = 0.f;
    bool ok = true;
    // adds tile t's products; they are complete before the warps hand over tile t + 1
    auto flush = [&](int t) {
      if (!mbar_wait_bounded(&ctl->acc_done, t & 1, abort_flag)) {
        record_status(p.status, kDevWaitPvDone);
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) return;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < kAcc; c += 16) {
        uint32_t x[16];
        tmem_ld16(acc_col + c, x);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[c + i] += __uint_as_float(x[i]);
      }
    };

    if constexpr (MODE == kDkv) {
      const uint32_t lt_mask = (1u << lane) - 1u;
      float* gh = p.gh + static_cast<size_t>(h - p.h0) * p.B * p.Tq * p.top_k;
      for (int t = 0; t < nS; ++t) {
        const BwdCols& c = cols[t & 1];
        if (!mbar_wait_bounded(&ctl->in_full[t & 1], (t >> 1) & 1, abort_flag)) {
          record_status(p.status, kDevWaitAccFull);
          ok = false;
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t buf = tmem_base + lane_off + (t & 1) * kBufCols;
        uint32_t s[16], r[16], d[16];
        tmem_ld16(buf + c0, s);
        tmem_ld16(buf + 64 + c0, r);
        tmem_ld16(buf + 128 + c0, d);
        tc_wait_ld();
        uint32_t pt[3][8], dt[3][8];
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          float pv[2], dv[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float4 f = c.f[c0 + i + e];
            const uint2 mem = c.mem[quarter][c0 + i + e];
            const bool member = (mem.x >> lane) & 1u;
            const float sm = ex2_approx(fmaf(__uint_as_float(s[i + e]), c2, -f.x)) * f.y;
            const float x = __uint_as_float(d[i + e]) - f.z;
            st_global_if(gh + (mem.y + __popc(mem.x & lt_mask)), sm * x, member);
            // (selected as a product: sm of a pair that is not a member may be infinite)
            pv[e] = member ? sm * fmaxf(__uint_as_float(r[i + e]), 0.f) : 0.f;
            dv[e] = pv[e] * x;
          }
          split3(pv[0], pv[1], pt[0][i >> 1], pt[1][i >> 1], pt[2][i >> 1]);
          split3(dv[0], dv[1], dt[0][i >> 1], dt[1][i >> 1], dt[2][i >> 1]);
        }
        tmem_st8(buf + c0, pt[0]);
        tmem_st8(buf + c0 + 8, pt[1]);
        tmem_st8(buf + 64 + c0, pt[2]);
        tmem_st8(buf + 64 + c0 + 8, dt[0]);
        tmem_st8(buf + 128 + c0, dt[1]);
        tmem_st8(buf + 128 + c0 + 8, dt[2]);
        if (t > 0) flush(t - 1);
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (ok && lane == 0) mbar_arrive(&ctl->p_ready[t & 1]);
      }
    } else {
      float neg_m = ninf, di = 0.f;                       // rows behind the end: sm = 0
      if (MODE == kDq && row_ok) {
        neg_m = -__ldg(p.rmax + bh * p.Tq + lrow);
        di = __ldg(p.di + bh * p.Tq + lrow);
      }
      float m = ninf, mx = ninf, l = 0.f;                 // kStats: stabiliser, exact maximum, sum
      const uint32_t* mrow =
          p.maskbits + ((static_cast<int64_t>(b) * p.nQT + lt) * p.nKT * kTile + row) * 4 + (grp >> 1);
      auto fetch = [&](int t) -> uint32_t {
        return (t < nS && row_ok) ? __ldg(mrow + static_cast<int64_t>(t >> 1) * (kTile * 4) + (t & 1) * 2) >> ((grp & 1) * 16)
                                  : 0u;
      };
      uint32_t next = fetch(0);
      for (int t = 0; t < nS; ++t) {
        const uint32_t word = next;
        next = fetch(t + 1);
        if (!mbar_wait_bounded(&ctl->in_full[t & 1], (t >> 1) & 1, abort_flag)) {
          record_status(p.status, kDevWaitAccFull);
          ok = false;
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t buf = tmem_base + lane_off + (t & 1) * kBufCols;
        uint32_t s[16], r[16];
        tmem_ld16(buf + c0, s);
        tmem_ld16(buf + 64 + c0, r);
        if constexpr (MODE == kStats) {
          tc_wait_ld();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->p_ready[t & 1]);
          float mt = ninf;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            s[i] = ((word >> i) & 1u) ? __float_as_uint(__uint_as_float(s[i]) * c2) : __float_as_uint(ninf);
            mt = fmaxf(mt, __uint_as_float(s[i]));
          }
          mx = fmaxf(mx, mt);
          if (mt > m + 8.f) {                             // raise the stabiliser when it is 2^8 behind
            l *= ex2_approx(m - mt);
            m = mt;
          }
          const float sub = m == ninf ? 0.f : -m;
          float l1 = 0.f;
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            l = fmaf(ex2_approx(__uint_as_float(s[i]) + sub), fmaxf(__uint_as_float(r[i]), 0.f), l);
            l1 = fmaf(ex2_approx(__uint_as_float(s[i + 1]) + sub), fmaxf(__uint_as_float(r[i + 1]), 0.f), l1);
          }
          l += l1;
        } else {
          uint32_t d[16];
          tmem_ld16(buf + 128 + c0, d);
          tc_wait_ld();
          uint32_t dt[3][8];
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            float dv[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float sm = ex2_approx(fmaf(__uint_as_float(s[i + e]), c2, neg_m));   // (1 / l: with the output)
              const float pv = ((word >> (i + e)) & 1u) ? sm * fmaxf(__uint_as_float(r[i + e]), 0.f) : 0.f;
              dv[e] = pv * (__uint_as_float(d[i + e]) - di);
            }
            split3(dv[0], dv[1], dt[0][i >> 1], dt[1][i >> 1], dt[2][i >> 1]);
          }
          tmem_st8(buf + 64 + c0 + 8, dt[0]);
          tmem_st8(buf + 128 + c0, dt[1]);
          tmem_st8(buf + 128 + c0 + 8, dt[2]);
          if (t > 0) flush(t - 1);
          tc_wait_st();
          tc_fence_before();
          __syncwarp();
          if (ok && lane == 0) mbar_arrive(&ctl->p_ready[t & 1]);
        }
      }
      if constexpr (MODE == kStats) {
        ctl->xm[grp][row] = m;
        ctl->xe[grp][row] = mx;
        ctl->xl[grp][row] = l;
        asm volatile("bar.sync 1, 512;" ::: "memory");
        if (grp == 0 && row_ok && ok) {
          const float mm = fmaxf(fmaxf(ctl->xe[0][row], ctl->xe[1][row]), fmaxf(ctl->xe[2][row], ctl->xe[3][row]));
          float lsum = 0.f;
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (ctl->xm[q][row] != ninf) lsum = fmaf(ctl->xl[q][row], exp2f(ctl->xm[q][row] - mm), lsum);
          // a row without members: +inf, all its weights are zero
          p.rmax[bh * p.Tq + lrow] = mm == ninf ? -ninf : mm;
          p.linv[bh * p.Tq + lrow] = 1.f / fmaxf(lsum, 1e-6f);
        }
      }
    }

    if constexpr (MODE != kStats) {
      if (ok) flush(nS - 1);
      if (ok && row_ok) {
        float* dst;
        float f = p.scale;
        if constexpr (MODE == kDkv) {
          dst = (grp < 2 ? p.dv : p.dk) + (bh * p.Tk + lrow) * kHd + (grp & 1) * kAcc;
          if (grp < 2) f = 1.f;
        } else {
          dst = p.dq + (bh * p.Tq + lrow) * kHd + grp * kAcc;
          f *= __ldg(p.linv + bh * p.Tq + lrow);
        }
#pragma unroll
        for (int i = 0; i < kAcc; i += 4)
          *reinterpret_cast<float4*>(dst + i) = make_float4(acc[i] * f, acc[i + 1] * f, acc[i + 2] * f, acc[i + 3] * f);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    __syncwarp();
    tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------ preparation
// Per (batch, head, query) row: D = dO . O in fp32 and dO as bf16 (contiguous); `inexact` is raised when
// some dO has more bits than bf16 holds.  Eight lanes per row.
template <typename TO>
__global__ void __launch_bounds__(256)
    dsa_bwd_prep_kernel(const TO* __restrict__ d_out, int64_t db, int64_t dh, int64_t dt, const TO* __restrict__ o,
                        int64_t ob, int64_t oh, int64_t ot, int B, int H, int T, __nv_bfloat16* __restrict__ do16,
                        float* __restrict__ di, int* __restrict__ inexact) {
  const int64_t r = (static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x) >> 3;
  const int c = (threadIdx.x & 7) * 8;
  const bool in = r < static_cast<int64_t>(B) * H * T;
  float acc = 0.f;
  bool bad = false;
  int64_t row = 0;
  if (in) {
    // rows in token-major order, the order of the caller's strided views
    const int h = static_cast<int>(r % H);
    const int64_t bt = r / H;
    const int t = static_cast<int>(bt % T), b = static_cast<int>(bt / T);
    const TO* x = d_out + b * db + h * dh + t * dt + c;
    const TO* y = o + b * ob + h * oh + t * ot + c;
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      float a[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        a[e] = static_cast<float>(x[i + e]);
        acc = fmaf(a[e], static_cast<float>(y[i + e]), acc);
      }
      w[i >> 1] = pack_bf16x2(a[0], a[1]);
      bad |= __uint_as_float(w[i >> 1] << 16) != a[0] || __uint_as_float(w[i >> 1] & 0xffff0000u) != a[1];
    }
    row = (static_cast<int64_t>(b) * H + h) * T + t;
    *reinterpret_cast<uint4*>(do16 + row * kHd + c) = make_uint4(w[0], w[1], w[2], w[3]);
  }
#pragma unroll
  for (int off = 4; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (in && c == 0) di[row] = acc;
  if (sizeof(TO) != 2 || std::is_same<TO, __half>::value) {
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) *inexact = 1;
  }
}

// off[b][kt][i] = first slot of row i whose key lies in tile kt or later (kt = 0 .. nKT); one warp per row of
// the ascending lists (`n` slots are valid in every row).  With `mask` also the tile-major membership bitmask:
// the CTA's eight rows fill a window of 32 key tiles in shared memory and write it in runs of 128 bytes, so that
// a layer need not keep the T^2 / 8 bytes from its forward to its backward.
__global__ void __launch_bounds__(256)
    dsa_bwd_offsets_kernel(const int32_t* __restrict__ idx, int top_k, int n, int B, int T, int Tk, int nKT,
                           uint16_t* __restrict__ off, uint4* __restrict__ mask, int* status) {
  constexpr int kWin = 32;                               // key tiles per window
  __shared__ __align__(16) uint32_t words[kWin][8][4];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t r0 = static_cast<int64_t>(blockIdx.x) * 8, r = r0 + wib, rows = static_cast<int64_t>(B) * T;
  if (r >= rows) n = 0;
  const int b = static_cast<int>(r / T), t = static_cast<int>(r % T);
  const int32_t* row = idx + r * top_k;
  uint16_t* dst = off + static_cast<int64_t>(b) * (nKT + 1) * T + t;
  int carry = -1;                                        // tile of the slot before this group
  int s0 = -32, key = 0;
  bool placed = true;                                    // this lane's slot has its bit
  constexpr int kAhead = 4;                              // groups of 32 slots in flight (one: 187 us, four: 152 us)
  auto load = [&](int s) { return s < n ? __ldg(row + s) : 0; };
  int ahead[kAhead];
#pragma unroll
  for (int i = 0; i < kAhead; ++i) ahead[i] = load(i * 32 + lane);
  for (int win = 0; win < nKT; win += kWin) {
    reinterpret_cast<uint4*>(words)[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    for (;;) {
      if (!placed && (key >> 7) < win + kWin) {
        if (key >= win * kTile) atomicOr(&words[(key >> 7) - win][wib][(key >> 5) & 3], 1u << (key & 31));
        else record_status(status, kDevBadIndex);        // (not ascending)
        placed = true;
      }
      if (!__all_sync(0xffffffffu, placed) || s0 + 32 >= n) break;     // the rest lies behind the window, or the row is done
      s0 += 32;
      const int s = s0 + lane;
      placed = s >= n;
      key = min(max(ahead[0], 0), Tk - 1);
#pragma unroll
      for (int i = 0; i + 1 < kAhead; ++i) ahead[i] = ahead[i + 1];
      ahead[kAhead - 1] = load(s + 32 * kAhead);
      const int kt = placed ? nKT : key >> 7;
      int before = __shfl_up_sync(0xffffffffu, kt, 1);
      if (lane == 0) before = carry;
      if (!placed)
        for (int q = before + 1; q <= kt; ++q) dst[static_cast<int64_t>(q) * T] = static_cast<uint16_t>(s);
      carry = __shfl_sync(0xffffffffu, kt, min(31, n - 1 - s0));
    }
    __syncthreads();
    const int kt = win + (threadIdx.x >> 3), rr = threadIdx.x & 7;
    if (mask != nullptr && kt < nKT && r0 + rr < rows) {
      const int bb = static_cast<int>((r0 + rr) / T), tt = static_cast<int>((r0 + rr) % T);
      const int nQT = (T + kTile - 1) / kTile;
      mask[((static_cast<int64_t>(bb) * nQT + tt / kTile) * nKT + kt) * kTile + tt % kTile] =
          *reinterpret_cast<const uint4*>(words[threadIdx.x >> 3][rr]);
    }
    __syncthreads();
  }
  if (r < rows)
    for (int q = carry + 1 + lane; q <= nKT; q += 32) dst[static_cast<int64_t>(q) * T] = static_cast<uint16_t>(n);
}

// drw = sum over the heads of their g, heads in ascending order (slots behind the valid ones are zero); `add`:
// the sum goes on from the heads before these
__global__ void __launch_bounds__(256)
    dsa_bwd_sum_heads_kernel(const float* __restrict__ gh, float* __restrict__ drw, int64_t n, int H, int top_k,
                             int n_valid, bool add, const int* __restrict__ skip_if) {
  if (skip_if != nullptr && *skip_if != 0) return;
  const int64_t i = (static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x) * 4;
  if (i >= n) return;
  if (((n | top_k | n_valid) & 3) == 0) {
    float4 a = add ? *reinterpret_cast<const float4*>(drw + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (static_cast<int>(i % top_k) < n_valid)
      for (int h = 0; h < H; ++h) {
        const float4 x = __ldcs(reinterpret_cast<const float4*>(gh + h * n + i));
        a.x += x.x; a.y += x.y; a.z += x.z; a.w += x.w;
      }
    *reinterpret_cast<float4*>(drw + i) = a;
  } else {
    for (int64_t e = i; e < i + 4 && e < n; ++e) {
      float a = add ? drw[e] : 0.f;
      if (static_cast<int>(e % top_k) < n_valid)
        for (int h = 0; h < H; ++h) a += gh[h * n + e];
      drw[e] = a;
    }
  }
}

// ------------------------------------------------------------ indexer gradients
// kLaneQ : lanes = queries of one tile, the key tiles streamed:  dq_idx = W G K_idx, and dW
// kLaneK : lanes = keys of one tile, the query tiles streamed:   dk_idx = W G^T Q_idx
// G is the dense 128 x 128 tile of the list gradients: eight warps clear the tile's three bf16 terms in
// shared memory and scatter the listed pairs into them (two threads per query row), one thread multiplies
// them with the streamed 128 x E tile of the projections (E = IH * ID, N of the instruction).
// Bound: those products, 24 instructions of E/2 cycles per tile; the lists are read twice in all.
struct IdxTileCtl {
  uint64_t full[2], empty[2], g_full, done;
  uint32_t tmem_base, abort_flag;
};
struct IdxTileParams {
  int B, Tq, Tk, nQT, nKT, top_k, IH, ID;
  const int32_t* idx;
  const float* g;           // (B,Tq,top_k)
  const uint16_t* off;
  const float* w;
  const __nv_bfloat16* q_idx;
  int64_t qsb, qst;
  float *dx, *dw;           // dq_idx or dk_idx (parts > 1: [parts] partial sums of it)
  int parts;                // CTAs per lane-side tile, each with its share of the streamed tiles
  int* status;
};
constexpr int kTermBytes = kTile * kTile * 2;           // one bf16 term of G: two 64-column halves of 16 KiB
constexpr int kOffB = 3 * kTermBytes;
constexpr size_t idx_smem(int E, int stages) {
  return 1024 + kOffB + static_cast<size_t>(stages) * kTile * E * 2 + sizeof(IdxTileCtl) + 64;
}
enum { kLaneQ = 0, kLaneK = 1 };

template <int MODE, int E>
__global__ void __launch_bounds__(320, 1)
    dsa_idx_bwd_tiles_kernel(const __grid_constant__ CUtensorMap tm_b, const IdxTileParams p) {
  constexpr int NST = 2;
  constexpr int kBBytes = kTile * E * 2;
  constexpr uint32_t kIdesc = make_idesc(/*bf16*/ 1, kTile, E, 0, /*B is MN-major*/ 1);
  constexpr int kPre = 8;                                // list entries a thread loads ahead
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  IdxTileCtl* ctl = reinterpret_cast<IdxTileCtl*>(smem + kOffB + NST * kBBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nLT = MODE == kLaneQ ? p.nQT : p.nKT, nAll = MODE == kLaneQ ? p.nKT : p.nQT;
  const int lt = blockIdx.x % nLT, b = blockIdx.x / nLT % p.B, part = blockIdx.x / (nLT * p.B);
  const int t_lo = static_cast<int>(static_cast<int64_t>(nAll) * part / p.parts);     // first streamed tile
  const int nS = static_cast<int>(static_cast<int64_t>(nAll) * (part + 1) / p.parts) - t_lo;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NST; ++s) {
      mbar_init(&ctl->full[s], 1);
      mbar_init(&ctl->empty[s], 1);
    }
    mbar_init(&ctl->g_full, 8);
    mbar_init(&ctl->done, 1);
    ctl->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&ctl->tmem_base, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;
  volatile uint32_t* abort_flag = &ctl->abort_flag;

  if (warp == 0) {
    if (lane == 0) {
      for (int t = 0; t < nS; ++t) {
        const int s = t & 1;
        if (!mbar_wait_bounded(&ctl->empty[s], ((t >> 1) & 1) ^ 1, abort_flag)) {
          record_status(p.status, kDevWaitStageEmpty);
          break;
        }
        mbar_expect_tx(&ctl->full[s], kBBytes);
#pragma unroll
        for (int c = 0; c < E / 64; ++c)
          tma_load_3d(smem + kOffB + s * kBBytes + c * (kTile * 128), &tm_b, &ctl->full[s], c * 64, (t_lo + t) * kTile, b);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t a0 = smem_u32(smem), b0 = a0 + kOffB;
      for (int t = 0; t < nS; ++t) {
        const int s = t & 1;
        if (!mbar_wait_bounded(&ctl->full[s], (t >> 1) & 1, abort_flag)) {
          record_status(p.status, kDevWaitTmaFull);
          break;
        }
        if (!mbar_wait_bounded(&ctl->g_full, t & 1, abort_flag)) {
          record_status(p.status, kDevWaitPReady);
          break;
        }
        tc_fence_after();
        const uint64_t db = smem_desc_sw128(b0 + s * kBBytes, kTile * 128);
#pragma unroll
        for (int term = 2; term >= 0; --term) {                // (smallest terms first, see above)
          const uint64_t da = smem_desc_sw128(a0 + term * kTermBytes);
#pragma unroll
          for (int ks = 0; ks < kTile / 16; ++ks)
            umma_f16_ss(tmem_base, da + (ks >> 2) * (kTile * 128 / 16) + (ks & 3) * 2, db + ks * 128, kIdesc,
                        term < 2 || ks > 0);
        }
        umma_commit(&ctl->empty[s]);
        umma_commit(&ctl->done);
      }
    }
  } else {
    const int ct = threadIdx.x - 64;
    const int r = ct >> 1, par = ct & 1;                 // query row of the tile, which half of its entries
    const uint32_t g_addr = smem_u32(smem);
    bool ok = true;
    // the entries of tile t: slots [s0, s1) of the row; this thread takes s0 + par, + 2, ...
    int s0 = 0, s1 = 0, id[kPre];
    float gv[kPre];
    int64_t rowbase = 0;
    auto fetch = [&](int t) {
      const int qt = MODE == kLaneQ ? lt : t_lo + t, kt = MODE == kLaneQ ? t_lo + t : lt;
      const int i = qt * kTile + r;
      s0 = s1 = 0;
      if (t < nS && i < p.Tq) {
        const uint16_t* o = p.off + (static_cast<int64_t>(b) * (p.nKT + 1) + kt) * p.Tq + i;
        rowbase = (static_cast<int64_t>(b) * p.Tq + i) * p.top_k;
        s0 = __ldg(o) + par;
        s1 = __ldg(o + p.Tq);
      }
#pragma unroll
      for (int e = 0; e < kPre; ++e) {
        const bool in = s0 + 2 * e < s1;
        id[e] = in ? __ldg(p.idx + rowbase + s0 + 2 * e) : 0;
        gv[e] = in ? __ldg(p.g + rowbase + s0 + 2 * e) : 0.f;
      }
    };
    auto place = [&](int key, float g) {
      const int j = key & (kTile - 1);
      const int m = MODE == kLaneQ ? r : j, k = MODE == kLaneQ ? j : r;       // lane-side row, streamed index
      const uint32_t a = g_addr + (k >> 6) * (kTile * 128) + m * 128 + ((((k & 63) >> 3) ^ (m & 7)) << 4) + (k & 7) * 2;
      uint32_t hi, mid, lo;
      split3(g, 0.f, hi, mid, lo);
      asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"(static_cast<uint16_t>(hi)) : "memory");
      asm volatile("st.shared.u16 [%0], %1;" ::"r"(a + kTermBytes), "h"(static_cast<uint16_t>(mid)) : "memory");
      asm volatile("st.shared.u16 [%0], %1;" ::"r"(a + 2 * kTermBytes), "h"(static_cast<uint16_t>(lo)) : "memory");
    };
    // this thread's part of the sums, in registers (every accumulation in tensor memory truncates, see above)
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const uint32_t acc_col = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + half * (E / 2);
    float acc[E / 2];
#pragma unroll
    for (int i = 0; i < E / 2; ++i) acc[i] = 0.f;
    auto flush = [&](int t) {
      if (!mbar_wait_bounded(&ctl->done, t & 1, abort_flag)) {
        record_status(p.status, kDevWaitPvDone);
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) return;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < E / 2; c += 16) {
        uint32_t x[16];
        tmem_ld16(acc_col + c, x);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[c + i] += __uint_as_float(x[i]);
      }
      tc_fence_before();
    };
    fetch(0);
    for (int t = 0; t < nS; ++t) {
      if (t > 0 && ok) flush(t - 1);
#pragma unroll
      for (int i = 0; i < 3 * kTermBytes / 16 / 256; ++i) sts128(g_addr + (i * 256 + ct) * 16, 0u, 0u, 0u, 0u);
      asm volatile("bar.sync 1, 256;" ::: "memory");
#pragma unroll
      for (int e = 0; e < kPre; ++e)
        if (s0 + 2 * e < s1) place(id[e], gv[e]);
      for (int s = s0 + 2 * kPre; s < s1; s += 2) place(__ldg(p.idx + rowbase + s), __ldg(p.g + rowbase + s));
      fence_proxy_async_smem();
      __syncwarp();
      ok = __all_sync(0xffffffffu, ok);
      if (ok && lane == 0) mbar_arrive(&ctl->g_full);
      fetch(t + 1);
    }
    if (ok) flush(nS - 1);
    if (ok) {
      const int lrow = lt * kTile + quarter * 32 + lane;
      const int T = MODE == kLaneQ ? p.Tq : p.Tk;
      const bool row_ok = lrow < T;
      float* dst = p.dx + ((static_cast<int64_t>(part) * p.B + b) * T + lrow) * E + half * (E / 2);
      const __nv_bfloat16* qrow = p.q_idx + b * p.qsb + lrow * p.qst + half * (E / 2);
      float dw = 0.f;
      int head = half * (E / 2) / p.ID;
#pragma unroll
      for (int c = 0; c < E / 2; c += 16) {
        uint4 qv[2];
        if (MODE == kLaneQ && row_ok) {
          qv[0] = __ldg(reinterpret_cast<const uint4*>(qrow + c));
          qv[1] = __ldg(reinterpret_cast<const uint4*>(qrow + c) + 1);
        } else {
          qv[0] = qv[1] = make_uint4(0u, 0u, 0u, 0u);
        }
        const uint32_t qw[8] = {qv[0].x, qv[0].y, qv[0].z, qv[0].w, qv[1].x, qv[1].y, qv[1].z, qv[1].w};
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int e = half * (E / 2) + c + i, hh = e / p.ID;
          if (MODE == kLaneQ && hh != head) {            // (uniform) the head's sum is complete
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) dw += __shfl_xor_sync(0xffffffffu, dw, off);
            if (lane == 0) atomicAdd(p.dw + head, dw);
            dw = 0.f;
            head = hh;
          }
          x[i] = acc[c + i];
          if (MODE == kLaneQ) dw = fmaf(x[i], __uint_as_float((i & 1) ? qw[i >> 1] & 0xffff0000u : qw[i >> 1] << 16), dw);
          x[i] *= __ldg(p.w + hh);
        }
        if (row_ok) {
#pragma unroll
          for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(dst + c + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
        }
      }
      if (MODE == kLaneQ) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) dw += __shfl_xor_sync(0xffffffffu, dw, off);
        if (lane == 0) atomicAdd(p.dw + head, dw);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    __syncwarp();
    tmem_dealloc(tmem_base, 256);
  }
}

size_t up256(size_t x) { return (x + 255) / 256 * 256; }
// Room for the heads' list gradients: as many heads as fit go through one dK / dV launch, their sum is added to
// that of the heads before (the same order of additions whatever the number).  16384 tokens, 8 heads, top-2048
// fill it; a sequence whose single head is larger takes one head at a time, the size of drw itself.
constexpr size_t kGhBytes = size_t(1) << 30;
struct BwdLayout {
  int heads;
  size_t do16, di, rmax, linv, wq, wk, off, flag, mask, gh, total;
};
BwdLayout bwd_layout(int B, int H, int Tq, int Tk, int top_k) {
  BwdLayout L;
  const size_t rows = static_cast<size_t>(B) * H * Tq;
  const size_t nKT = (Tk + kTile - 1) / kTile;
  size_t o = 0;
  L.do16 = o; o += up256(rows * kHd * 2);
  L.di = o; o += up256(rows * 4);
  L.rmax = o; o += up256(rows * 4);
  L.linv = o; o += up256(rows * 4);
  L.wq = o; o += up256(static_cast<size_t>(B) * Tq * kIdxDim * 4);
  L.wk = o; o += up256(static_cast<size_t>(B) * Tk * kIdxDim * 4);
  L.off = o; o += up256(static_cast<size_t>(B) * (nKT + 1) * Tq * 2);
  L.flag = o; o += 256;
  L.mask = o; o += up256(static_cast<size_t>(B) * ((Tq + kTile - 1) / kTile) * nKT * kTile * 16);
  const size_t head = static_cast<size_t>(B) * Tq * top_k * 4;
  L.heads = static_cast<int>(std::max<size_t>(1, std::min<size_t>(H, kGhBytes / head)));
  L.gh = o; o += up256(L.heads * head);
  L.total = o;
  return L;
}

template <int MODE>
int launch_bwd(const CUtensorMap& l1, const CUtensorMap& l2, const CUtensorMap& lr, const CUtensorMap& s1,
               const CUtensorMap& s2, const CUtensorMap& sr, const BwdTileParams& p, cudaStream_t st) {
  SWV_CUDA_OK(cudaFuncSetAttribute(dsa_bwd_tiles_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(kBwdSmem)));
  const unsigned grid = static_cast<unsigned>(p.B) * p.Hn * (MODE == kDkv ? p.nKT : p.nQT);
  dsa_bwd_tiles_kernel<MODE><<<grid, bwd_threads(MODE), kBwdSmem, st>>>(l1, l2, lr, s1, s2, sr, p);
  SWV_CUDA_OK(cudaGetLastError());
  return SWV_OK;
}

// out[i] = the parts' sums, added in order (n is a multiple of 4)
__global__ void __launch_bounds__(256)
    dsa_idx_bwd_sum_kernel(const float* __restrict__ partial, int parts, float* __restrict__ out, int64_t n) {
  const int64_t i = (static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x) * 4;
  if (i >= n) return;
  float4 a = __ldcs(reinterpret_cast<const float4*>(partial + i));
  for (int q = 1; q < parts; ++q) {
    const float4 x = __ldcs(reinterpret_cast<const float4*>(partial + q * n + i));
    a.x += x.x; a.y += x.y; a.z += x.z; a.w += x.w;
  }
  *reinterpret_cast<float4*>(out + i) = a;
}

// Short sequences have fewer lane-side tiles than the chip has SMs (6007 tokens: 47): the streamed range is then
// divided over `parts` CTAs, whose partial sums go to `scratch` (128 channels: 143 -> 58 us for dq_idx and
// 128 -> 49 us for dk_idx, plus 4 us of sums).
template <int MODE, int E>
int launch_idx(const CUtensorMap& tb, IdxTileParams p, float* scratch, size_t scratch_floats, cudaStream_t st) {
  constexpr size_t smem = idx_smem(E, 2);
  SWV_CUDA_OK(cudaFuncSetAttribute(dsa_idx_bwd_tiles_kernel<MODE, E>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(smem)));
  const int tiles = p.B * (MODE == kLaneQ ? p.nQT : p.nKT), streamed = MODE == kLaneQ ? p.nKT : p.nQT;
  const int64_t n = static_cast<int64_t>(p.B) * (MODE == kLaneQ ? p.Tq : p.Tk) * E;
  float* out = p.dx;
  p.parts = std::max(1, std::min({sm_count() / tiles, streamed / 4, 8, static_cast<int>(scratch_floats / n)}));
  if (p.parts > 1) p.dx = scratch;
  dsa_idx_bwd_tiles_kernel<MODE, E><<<static_cast<unsigned>(tiles) * p.parts, 320, smem, st>>>(tb, p);
  if (p.parts > 1)
    dsa_idx_bwd_sum_kernel<<<static_cast<unsigned>((n / 4 + 255) / 256), 256, 0, st>>>(scratch, p.parts, out, n);
  SWV_CUDA_OK(cudaGetLastError());
  return SWV_OK;
}

template <typename TO>
int launch_prep(const void* d_out, const int64_t* ds, const void* o, const int64_t* os, int B, int H, int T, void* do16,
                float* di, int* flag, cudaStream_t st) {
  const int64_t threads = static_cast<int64_t>(B) * H * T * 8;
  dsa_bwd_prep_kernel<TO><<<static_cast<unsigned>((threads + 255) / 256), 256, 0, st>>>(
      static_cast<const TO*>(d_out), ds[0], ds[1], ds[2], static_cast<const TO*>(o), os[0], os[1], os[2], B, H, T,
      static_cast<__nv_bfloat16*>(do16), di, flag);
  SWV_CUDA_OK(cudaGetLastError());
  return SWV_OK;
}

bool rows16(const void* p, const int64_t* s, int n) {
  if ((reinterpret_cast<uintptr_t>(p) & 15) || s[n] != 1) return false;
  for (int i = 0; i < n; ++i)
    if ((s[i] * 2) % 16) return false;
  return true;
}

}  // namespace

int dsa_collapse_impl(const void* x, const int64_t* s, int dtype, const float* w, float* out, int B, int Tn, int IH,
                      int ID, cudaStream_t st);
int dsa_attn_bwd_impl(const void* d_out, const int64_t* dos, const void* q, const int64_t* qs, const void* k,
                      const int64_t* ks, const void* v, const int64_t* vs, int dtype, const void* o,
                      const int64_t* os, int o_dtype, const int32_t* idx, const int64_t* is, const float* valid,
                      const int64_t* vls, const float* rw, const int64_t* rs, float* dq, float* dk, float* dv,
                      float* drw, int B, int H, int Tq, int Tk, int D, int top_k, int* status, cudaStream_t st,
                      const int* run_if);
int dsa_indexer_bwd_impl(const float* d_scores, const int64_t* dss, const void* q_idx, const int64_t* qs,
                         const void* k_idx, const int64_t* ks, int dtype, const float* w, const int32_t* idx,
                         const int64_t* is, const float* valid, const int64_t* vls, float* dq, float* dk, float* dw,
                         int B, int Tq, int Tk, int IH, int ID, int top_k, int* status, cudaStream_t st);

int dsa_module_bwd_bytes_impl(int B, int H, int Tq, int Tk, int top_k, size_t* bytes) {
  if (!bytes) return SWV_ERR_NULL;
  if (B < 1 || H < 1 || Tq < 1 || Tk < 1 || top_k < 1) return SWV_ERR_SHAPE;
  *bytes = bwd_layout(B, H, Tq, Tk, top_k).total;
  return SWV_OK;
}

int dsa_module_bwd_impl(const void* d_out, const int64_t* dos, const void* q, const int64_t* qs, const void* k,
                        const int64_t* ks, const void* v, const int64_t* vs, const void* o, const int64_t* os,
                        int o_dtype, const void* q_idx, const int64_t* qis, const void* k_idx, const int64_t* kis,
                        int idx_dtype, const float* w, const int32_t* idx, const float* valid, const float* scores,
                        const uint32_t* maskbits, float* dq, float* dk, float* dv, float* drw, float* dq_idx,
                        float* dk_idx, float* dw, int B, int H, int Tq, int Tk, int D, int IH, int ID, int top_k,
                        void* workspace, size_t workspace_bytes, int* status, cudaStream_t st) {
  if (!d_out || !q || !k || !v || !o || !q_idx || !k_idx || !w || !idx || !valid || !scores || !dq || !dk ||
      !dv || !drw || !dq_idx || !dk_idx || !dw || !workspace || !status)
    return SWV_ERR_NULL;
  if (B < 1 || H < 1 || Tq < 1 || Tk < 1 || top_k < 1 || IH < 1 || ID < 1) return SWV_ERR_SHAPE;
  // list slots are 16-bit offsets, list positions 32-bit
  if (D != kHd || ID > kIdxDim || top_k > 65535 || static_cast<uint64_t>(B) * Tq * top_k >= (1ull << 32))
    return SWV_ERR_UNSUPPORTED;
  if (!rows16(q, qs, 3) || !rows16(k, ks, 3) || !rows16(v, vs, 3) || dos[3] != 1 || os[3] != 1) return SWV_ERR_ALIGN;
  const BwdLayout L = bwd_layout(B, H, Tq, Tk, top_k);
  if (workspace_bytes < L.total) return SWV_ERR_WORKSPACE;
  if (reinterpret_cast<uintptr_t>(workspace) & 255) return SWV_ERR_ALIGN;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  void* do16 = ws + L.do16;
  float* di = reinterpret_cast<float*>(ws + L.di);
  float* wq = reinterpret_cast<float*>(ws + L.wq);
  float* wk = reinterpret_cast<float*>(ws + L.wk);
  uint16_t* off = reinterpret_cast<uint16_t*>(ws + L.off);
  int* flag = reinterpret_cast<int*>(ws + L.flag);
  const int nQT = (Tq + kTile - 1) / kTile, nKT = (Tk + kTile - 1) / kTile;
  const int64_t ls[3] = {static_cast<int64_t>(Tq) * top_k, top_k, 1};

  int rc;
  const bool exact = o_dtype == SWV_BF16;
  if (!exact) SWV_CUDA_OK(cudaMemsetAsync(flag, 0, sizeof(int), st));
  if (o_dtype == SWV_F32) rc = launch_prep<float>(d_out, dos, o, os, B, H, Tq, do16, di, flag, st);
  else if (o_dtype == SWV_BF16) rc = launch_prep<__nv_bfloat16>(d_out, dos, o, os, B, H, Tq, do16, di, flag, st);
  else if (o_dtype == SWV_F16) rc = launch_prep<__half>(d_out, dos, o, os, B, H, Tq, do16, di, flag, st);
  else return SWV_ERR_DTYPE;
  if (rc != SWV_OK) return rc;
  if (!exact) {
    // clears dk, dv, drw and, where some dO does not fit bf16, computes them
    rc = dsa_attn_bwd_impl(d_out, dos, q, qs, k, ks, v, vs, SWV_BF16, o, os, o_dtype, idx, ls, valid, ls, scores, ls, dq,
                           dk, dv, drw, B, H, Tq, Tk, D, top_k, status, st, flag);
    if (rc != SWV_OK) return rc;
  }
  rc = dsa_collapse_impl(q_idx, qis, idx_dtype, w, wq, B, Tq, IH, ID, st);
  if (rc != SWV_OK) return rc;
  rc = dsa_collapse_impl(k_idx, kis, idx_dtype, w, wk, B, Tk, IH, ID, st);
  if (rc != SWV_OK) return rc;
  const int64_t rows = static_cast<int64_t>(B) * Tq;
  uint4* own_mask = maskbits == nullptr ? reinterpret_cast<uint4*>(ws + L.mask) : nullptr;
  if (own_mask != nullptr) maskbits = reinterpret_cast<const uint32_t*>(own_mask);
  dsa_bwd_offsets_kernel<<<static_cast<unsigned>((rows + 7) / 8), 256, 0, st>>>(idx, top_k, top_k < Tk ? top_k : Tk, B, Tq,
                                                                              Tk, nKT, off, own_mask, status);
  SWV_CUDA_OK(cudaGetLastError());

  // maps with 128-row boxes (lane side) and 64-row boxes (streamed side)
  CUtensorMap mq[2], mk[2], mv[2], md[2], mwq[2], mwk[2];
  const CUtensorMapDataType bf = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, f32 = CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  for (int i = 0; i < 2; ++i) {
    const uint32_t box = i == 0 ? kTile : kNW;
    if ((rc = make_tmap_4d(&mq[i], q, bf, D, Tq, H, B, qs[2] * 2, qs[1] * 2, qs[0] * 2, kHd, box)) != SWV_OK) return rc;
    if ((rc = make_tmap_4d(&mk[i], k, bf, D, Tk, H, B, ks[2] * 2, ks[1] * 2, ks[0] * 2, kHd, box)) != SWV_OK) return rc;
    if ((rc = make_tmap_4d(&mv[i], v, bf, D, Tk, H, B, vs[2] * 2, vs[1] * 2, vs[0] * 2, kHd, box)) != SWV_OK) return rc;
    if ((rc = make_tmap_4d(&md[i], do16, bf, D, Tq, H, B, kHd * 2, static_cast<uint64_t>(Tq) * kHd * 2,
                           static_cast<uint64_t>(H) * Tq * kHd * 2, kHd, box)) != SWV_OK) return rc;
    if ((rc = make_tmap_3d(&mwq[i], wq, f32, kIdxDim, Tq, B, kIdxDim * 4, static_cast<uint64_t>(Tq) * kIdxDim * 4, 32,
                           box)) != SWV_OK) return rc;
    if ((rc = make_tmap_3d(&mwk[i], wk, f32, kIdxDim, Tk, B, kIdxDim * 4, static_cast<uint64_t>(Tk) * kIdxDim * 4, 32,
                           box)) != SWV_OK) return rc;
  }
  BwdTileParams p;
  p.B = B; p.H = H; p.Tq = Tq; p.Tk = Tk; p.nQT = nQT; p.nKT = nKT; p.top_k = top_k;
  p.maskbits = maskbits; p.off = off; p.di = di; p.rmax = reinterpret_cast<float*>(ws + L.rmax); p.linv = reinterpret_cast<float*>(ws + L.linv);
  p.h0 = 0; p.Hn = H;
  p.dq = dq; p.dk = dk; p.dv = dv; p.gh = reinterpret_cast<float*>(ws + L.gh);
  p.r_steps = (ID + 7) / 8;
  p.scale = 1.0f / sqrtf(static_cast<float>(D));
  p.c2 = p.scale * 1.4426950408889634f;
  p.skip_if = exact ? nullptr : flag;
  p.status = status;
  if ((rc = launch_bwd<kStats>(mq[0], mq[0], mwq[0], mk[1], mk[1], mwk[1], p, st)) != SWV_OK) return rc;
  if ((rc = launch_bwd<kDq>(mq[0], md[0], mwq[0], mk[1], mv[1], mwk[1], p, st)) != SWV_OK) return rc;
  const int64_t n = rows * top_k;
  for (; p.h0 < H; p.h0 += L.heads) {
    p.Hn = std::min(L.heads, H - p.h0);
    if ((rc = launch_bwd<kDkv>(mk[0], mv[0], mwk[0], mq[1], md[1], mwq[1], p, st)) != SWV_OK) return rc;
    dsa_bwd_sum_heads_kernel<<<static_cast<unsigned>((n + 1023) / 1024), 256, 0, st>>>(
        p.gh, drw, n, p.Hn, top_k, top_k < Tk ? top_k : Tk, p.h0 > 0, p.skip_if);
    SWV_CUDA_OK(cudaGetLastError());
  }

  // indexer: tiles for bf16 projections whose heads lie side by side, else the list kernel
  const int E = IH * ID;
  const int64_t q3[3] = {qis[0], qis[1], qis[3]}, k3[3] = {kis[0], kis[1], kis[3]};
  if (idx_dtype == SWV_BF16 && (E == 64 || E == 128 || E == 256) && qis[2] == ID && kis[2] == ID && rows16(q_idx, q3, 2) &&
      rows16(k_idx, k3, 2)) {
    CUtensorMap tq, tk;
    if ((rc = make_tmap_3d(&tq, q_idx, bf, E, Tq, B, qis[1] * 2, qis[0] * 2, 64, kTile)) != SWV_OK) return rc;
    if ((rc = make_tmap_3d(&tk, k_idx, bf, E, Tk, B, kis[1] * 2, kis[0] * 2, 64, kTile)) != SWV_OK) return rc;
    SWV_CUDA_OK(cudaMemsetAsync(dw, 0, static_cast<size_t>(IH) * sizeof(float), st));
    IdxTileParams ip;
    ip.B = B; ip.Tq = Tq; ip.Tk = Tk; ip.nQT = nQT; ip.nKT = nKT; ip.top_k = top_k; ip.IH = IH; ip.ID = ID;
    ip.idx = idx; ip.g = drw; ip.off = off; ip.w = w;
    ip.q_idx = static_cast<const __nv_bfloat16*>(q_idx); ip.qsb = qis[0]; ip.qst = qis[1];
    ip.dx = dq_idx; ip.dw = dw; ip.status = status;
    // the heads' gradients have been summed: their room takes the partial sums
    float* part = p.gh;
    const size_t nf = static_cast<size_t>(n) * L.heads;
    if (E == 64) rc = launch_idx<kLaneQ, 64>(tk, ip, part, nf, st);
    else if (E == 128) rc = launch_idx<kLaneQ, 128>(tk, ip, part, nf, st);
    else rc = launch_idx<kLaneQ, 256>(tk, ip, part, nf, st);
    if (rc != SWV_OK) return rc;
    ip.dx = dk_idx;
    if (E == 64) return launch_idx<kLaneK, 64>(tq, ip, part, nf, st);
    if (E == 128) return launch_idx<kLaneK, 128>(tq, ip, part, nf, st);
    return launch_idx<kLaneK, 256>(tq, ip, part, nf, st);
  }
  return dsa_indexer_bwd_impl(drw, ls, q_idx, qis, k_idx, kis, idx_dtype, w, idx, ls, valid, ls, dq_idx, dk_idx, dw, B, Tq,
                              Tk, IH, ID, top_k, status, st);
}

}  // namespace swv
