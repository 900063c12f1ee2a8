// Packed variable-length (causal) attention backward for sm_100a, same building blocks as attn_fwd_tcgen05.cu.
//
// Two passes over the (q block, kv block) pairs, each with ONE resident 128-row tile pair and a streamed ring of 64-row tile
// pairs, so that every accumulator lives in tensor memory for the whole CTA and nothing needs atomics or rescaling:
//
//   pass "dKV" (CTA = 128 keys of one kv head): resident K_j, V_j; streams Q_t, dO_t over all q blocks at / below the
//       diagonal and over the q heads of the GQA group.  Transposed orientation -- tensor-memory lanes are KEYS:
//         S^T = K_j Q_t^T      dP^T = V_j dO_t^T                         (two M=128, N=64, K=D products per step)
//         P^T = exp2(S^T * scale*log2e - lse_q * log2e)                  (softmax statistics vary along columns)
//         dS^T = P^T o (dP^T - delta_q) * scale
//         dV_j += P^T dO_t     dK_j += dS^T Q_t                          (two M=128, N=D, K=64 products per step)
//   pass "dQ" (CTA = 128 query rows of one q head): resident Q_i, dO_i; streams K_t, V_t up to the diagonal:
//         S = Q_i K_t^T        dP = dO_i V_t^T      dS = P o (dP - delta) * scale      dQ_i += dS K_t
//
// The streamed tiles are used twice with two different descriptors over the same bytes: as the K-major B operand of the
// S-type products (rows = N) and as the MN-major B operand of the accumulating products (rows = K), exactly the two operand forms of
// the GEMM kernel (forward / wgrad).  P^T and dS^T (or dS) overwrite the front of the S / dP columns they came from, as 16-bit TMEM A operands
// of the accumulating products: they never travel through shared memory, and since the tensor pipe runs in issue order no buffer needs an
// "empty" barrier.  S / dP are double buffered: the pipe runs the S-type products of step t+1 while the threads work on step t.
// Recomputing S and dP in both passes costs 7 instead of 5 products per block pair; in exchange the result is deterministic,
// there is no fp32 dQ scratch tensor to zero / convert, and dK / dV of a GQA group are reduced inside one CTA.
//
// What bounds it: a step is 1024 (dKV) or 768 (dQ) tensor-pipe cycles at D = 128, and its 8192 elements take the CUDA cores about as long when
// eight warps share them (a warp has 32 rows and 32 of the 64 columns).  Four warps, P through shared memory, the streamed rows' statistics
// fetched from global memory inside every step and MMAs issued from a divergent branch kept the tensor pipe 19% busy (32 x 640 tokens x 32
// heads: dKV 613, dQ 506 us, now 322, 240; 8 x 1500..4096, 32 / 8 heads: 2473, 2109 us, now 1553, 1152).
//
// The grid holds one CTA per (row tile, head) (a bound: the lengths are on the device); a running CTA takes the items of CTAs that have not
// started (`clusterlaunchcontrol.try_cancel`), so that the next item's tiles load and its first products run while the last accumulators
// leave.  With a CTA per item 32 x 640 tokens took 17600 cycles an item of which six steps were half.
//
// delta[h, t] = sum_d dO[t, h, d] * O[t, h, d] comes from a small pre-pass; LSE is the forward's ([nq, T], natural log).
#include <type_traits>

#include "attn_common.cuh"

namespace {

constexpr int kR = 128;   // resident rows per CTA (= UMMA M)
constexpr int kX = 64;    // streamed rows per step (= UMMA N of the S-type products, K of the accumulating ones)
constexpr int kXStages = 3;
constexpr int kBwdThreads = 320;   // warp 0: TMA, warp 1: MMA, warps 2-9: elements (two per TMEM quadrant, one per column half)

struct BwdParams {
  const int* cu_seqlens;
  const float* lse;    // [nq, T]
  const float* delta;  // [nq, T]
  void* out1;          // dKV pass: dV;  dQ pass: dQ      ([T, heads, D] views, row pitch ld1)
  void* out2;          // dKV pass: dK
  int64_t ld1, ld2;
  int T, B, nq, nkv, heads;   // heads: of this pass (key heads for dKV, query heads for dQ)
  float scale;
  int causal;
  int* status = nullptr;   // set by the launch: rb_attn_status()
};

template <int kD> struct BCfg {
  static constexpr int kDBlocks = kD / 64;
  static constexpr int kRBytes = kR * kD * 2;     // one resident tile
  static constexpr int kXBytes = kX * kD * 2;     // one streamed tile
  static constexpr int kOut = 2 * kRBytes + kXStages * 2 * kXBytes;   // 4 KB of output staging per element warp
  static constexpr int kBars = kOut + 8 * 4096;
  static constexpr int kStats = kBars + 256;      // [8 element warps][2 buffers][lse | delta][32]
  static constexpr int kSmemBytes = kStats + 8 * 2 * 2 * 32 * 4 + 1024 /*align*/;
};

enum BBar { R_FULL = 0, R_EMPTY = 1, X_FULL = 2, X_EMPTY = X_FULL + kXStages, S_FULL = X_EMPTY + kXStages, P_FULL = S_FULL + 2, ACC_FULL = P_FULL + 2,
            ACC_EMPTY = ACC_FULL + 1, IT_FULL = ACC_EMPTY + 1, IT_EMPTY = IT_FULL + 2, CLC_FULL = IT_EMPTY + 2, B_NUM_BARS = CLC_FULL + 1 };

// One work item: sequence (first token, length), head and first resident row; L < 0 ends the CTA's loop.
struct BItem { int tok0, L, head, r0; };

// tma_r1 / tma_r2: resident operands (box 64 cols x 128 rows); tma_x1 / tma_x2: streamed operands (box 64 x 64).
//   kDKV: r1 = K, r2 = V (kv-head columns), x1 = Q, x2 = dO (q-head columns).   !kDKV: r1 = Q, r2 = dO, x1 = K, x2 = V.
template <int kD, typename T, int kFmt, bool kDKV>
__global__ void __launch_bounds__(kBwdThreads, 1) attn_bwd_kernel(const __grid_constant__ CUtensorMap tma_r1,
                                                                  const __grid_constant__ CUtensorMap tma_r2,
                                                                  const __grid_constant__ CUtensorMap tma_x1,
                                                                  const __grid_constant__ CUtensorMap tma_x2, const __grid_constant__ BwdParams p) {
  using C = BCfg<kD>;
  const int G = p.nq / p.nkv;
  // streamed blocks [blk0, blk0 + nblk) of an item: dKV -> query blocks that can see its keys; dQ -> key blocks its queries can see; dKV also walks
  // the q heads of the group (outer loop)
  auto first_blk = [&](const BItem& it) { return kDKV && p.causal ? it.r0 / kX : 0; };
  auto blocks = [&](const BItem& it) { return RB_CEIL_DIV(!kDKV && p.causal ? min(it.L, it.r0 + kR) : it.L, kX) - first_blk(it); };
  auto steps = [&](const BItem& it) { return blocks(it) * (kDKV ? G : 1); };

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t sR1 = ptx::smem_u32(smem);
  const uint32_t sR2 = sR1 + C::kRBytes;
  const uint32_t sX = sR2 + C::kRBytes;            // stage s: X1 at sX + s * 2 * kXBytes, X2 right after it
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kBars);
  BItem* items = reinterpret_cast<BItem*>(smem + C::kBars + 192);     // two slots of 16 bytes
  const uint32_t clc = sR1 + C::kBars + 224;                          // 16 bytes
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(smem + C::kBars + 240);
  volatile uint32_t* dead = tmem_ptr + 1;
  float* stats = reinterpret_cast<float*>(smem + C::kStats);
  auto bar = [&](int i) { return ptx::smem_u32(&bars[i]); };
  auto wait = [&](int i, uint32_t parity) { bounded_wait(bar(i), parity, dead); };
  // TMEM columns: S buffers [0,64) [64,128); dP buffers [128,192) [192,256); accumulators at 256 (dV / dQ) and 384 (dK)
  constexpr uint32_t kTmS = 0, kTmDP = 128, kTmAcc1 = 256, kTmAcc2 = 384;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0 && lane == 0) {
    *dead = 0;
    ptx::prefetch_tensormap(&tma_r1);
    ptx::prefetch_tensormap(&tma_r2);
    ptx::prefetch_tensormap(&tma_x1);
    ptx::prefetch_tensormap(&tma_x2);
    for (int i = 0; i < B_NUM_BARS; ++i)      // one arrival per element warp; items: the MMA warp too
      ptx::mbar_init(bar(i), i == P_FULL || i == P_FULL + 1 || i == ACC_EMPTY ? 8 : i == IT_EMPTY || i == IT_EMPTY + 1 ? 9 : 1);
    ptx::fence_barrier_init();
  }
  if (warp == 1) {
    ptx::tmem_alloc(ptx::smem_u32(tmem_ptr), 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;

  if (warp == 0) {
    // ===================================================== scheduler + TMA producer
    auto request = [&] {
      if (lane == 0) {
        ptx::mbar_arrive_expect_tx(bar(CLC_FULL), 16);
        ptx::clc_try_cancel(clc, bar(CLC_FULL));
      }
      __syncwarp();
    };
    UnitSearch search;
    int idx = blockIdx.x, n_pub = 0, g = 0;      // g: streamed tiles so far
    uint32_t n_req = 0;
    auto publish = [&](const BItem& it) {
      const int slot = n_pub & 1;
      wait(IT_EMPTY + slot, ((uint32_t)(n_pub >> 1) & 1u) ^ 1u);
      if (lane == 0) {
        items[slot] = it;
        ptx::mbar_arrive(bar(IT_FULL + slot));
      }
      ++n_pub;
    };
    request();
    while (true) {
      BItem it{0, 0, 0, 0};
      int r;
      it.head = idx % p.heads;
      if (search.find(p.cu_seqlens, p.B, kR, idx / p.heads, it.tok0, it.L, r)) {
        it.r0 = (kDKV ? r : RB_CEIL_DIV(it.L, kR) - 1 - r) * kR;       // heaviest tiles first in both passes
        publish(it);
        if (lane == 0) {
          wait(R_EMPTY, (uint32_t)n_pub & 1u);      // (n_pub - 1 items before this one)
          const int nblk = blocks(it), n = steps(it), blk0 = first_blk(it);
          ptx::mbar_arrive_expect_tx(bar(R_FULL), 2 * C::kRBytes);
#pragma unroll
          for (int kb = 0; kb < C::kDBlocks; ++kb) {
            ptx::tma_load_2d(sR1 + kb * (kR * 128), &tma_r1, bar(R_FULL), it.head * kD + kb * 64, it.tok0 + it.r0);
            ptx::tma_load_2d(sR2 + kb * (kR * 128), &tma_r2, bar(R_FULL), it.head * kD + kb * 64, it.tok0 + it.r0);
          }
          int h = kDKV ? it.head * G : it.head / G, blk = 0;           // dQ streams the kv head of its q head
          for (int t = 0; t < n; ++t, ++g) {
            const int st = g % kXStages, row = it.tok0 + (blk0 + blk) * kX;
            wait(X_EMPTY + st, ((uint32_t)(g / kXStages) & 1u) ^ 1u);
            ptx::mbar_arrive_expect_tx(bar(X_FULL + st), 2 * C::kXBytes);
            const uint32_t x1 = sX + st * 2 * C::kXBytes, x2 = x1 + C::kXBytes;
#pragma unroll
            for (int kb = 0; kb < C::kDBlocks; ++kb) {
              ptx::tma_load_2d(x1 + kb * (kX * 128), &tma_x1, bar(X_FULL + st), h * kD + kb * 64, row);
              ptx::tma_load_2d(x2 + kb * (kX * 128), &tma_x2, bar(X_FULL + st), h * kD + kb * 64, row);
            }
            if (++blk == nblk) { blk = 0; ++h; }
          }
        }
        __syncwarp();
      }
      wait(CLC_FULL, n_req & 1u);
      ++n_req;
      if (*dead) break;
      int x;
      const bool got = ptx::clc_query(clc, x);
      __syncwarp();
      if (!got) break;
      idx = x;
      ptx::fence_proxy_async();   // the response was read before it is overwritten
      request();
    }
    publish(BItem{0, -1, 0, 0});
  } else if (warp == 1) {
    // ===================================================== MMA issuer: the whole warp runs the loop, one elected lane issues
    constexpr uint32_t idesc_s = ptx::make_idesc_f16(kFmt, kR, kX, 0, 0);   // resident x streamed^T, both K-major
    constexpr uint32_t idesc_a = ptx::make_idesc_f16(kFmt, kR, kD, 0, 1);   // P-type (TMEM) x streamed (MN-major)
    const uint32_t tm = (uint32_t)ptx::uniform((int)tmem_base);
    const uint64_t r1 = ptx::make_smem_desc_sw128(sR1, 16, 1024), r2 = ptx::make_smem_desc_sw128(sR2, 16, 1024);
    auto issue_sdp = [&](int g, bool last) {      // g: steps of this CTA so far
      const int st = g % kXStages;
      wait(X_FULL + st, (uint32_t)(g / kXStages) & 1u);
      ptx::tc_fence_after();
      const uint32_t d = tm + (g & 1) * 64;
      const uint64_t x1 = ptx::make_smem_desc_sw128(sX + st * 2 * C::kXBytes, 16, 1024);
      const uint64_t x2 = ptx::make_smem_desc_sw128(sX + st * 2 * C::kXBytes + C::kXBytes, 16, 1024);
      if (ptx::elect_one()) {
#pragma unroll
        for (int kk = 0; kk < kD / 16; ++kk)
          ptx::tc_mma_f16(d + kTmS, r1 + (((kk >> 2) * (kR * 128) + (kk & 3) * 32) >> 4), x1 + (((kk >> 2) * (kX * 128) + (kk & 3) * 32) >> 4), idesc_s,
                          kk != 0 ? 1u : 0u);
#pragma unroll
        for (int kk = 0; kk < kD / 16; ++kk)
          ptx::tc_mma_f16(d + kTmDP, r2 + (((kk >> 2) * (kR * 128) + (kk & 3) * 32) >> 4), x2 + (((kk >> 2) * (kX * 128) + (kk & 3) * 32) >> 4), idesc_s,
                          kk != 0 ? 1u : 0u);
        ptx::tc_commit(bar(S_FULL + (g & 1)));
        if (last) ptx::tc_commit(bar(R_EMPTY));
      }
      __syncwarp();
    };
    int g = 0;
    for (int n_it = 0;; ++n_it) {
      const int slot = n_it & 1;
      wait(IT_FULL + slot, (uint32_t)(n_it >> 1) & 1u);
      BItem it = items[slot];
      it.L = ptx::uniform(it.L);
      it.r0 = ptx::uniform(it.r0);
      if (lane == 0) ptx::mbar_arrive(bar(IT_EMPTY + slot));
      __syncwarp();
      if (it.L < 0 || ptx::uniform((int)*dead)) break;
      const int n = steps(it);
      wait(R_FULL, (uint32_t)n_it & 1u);
      issue_sdp(g, n == 1);
      for (int t = 0; t < n; ++t, ++g) {
        if (t + 1 < n) issue_sdp(g + 1, t + 2 == n);       // its S / dP columns: the products that read P of step t-1 there are ahead in the pipe
        const int st = g % kXStages;
        wait(P_FULL + (g & 1), (uint32_t)(g >> 1) & 1u);
        if (t == 0) wait(ACC_EMPTY, ((uint32_t)n_it & 1u) ^ 1u);
        ptx::tc_fence_after();
        const uint32_t a = tm + (g & 1) * 64;
        const uint64_t x1 = ptx::make_smem_desc_sw128(sX + st * 2 * C::kXBytes, kX * 128, 1024);
        const uint64_t x2 = ptx::make_smem_desc_sw128(sX + st * 2 * C::kXBytes + C::kXBytes, kX * 128, 1024);
        const uint32_t keep = t != 0 ? 1u : 0u;
        if (ptx::elect_one()) {
#pragma unroll
          for (int kk = 0; kk < kX / 16; ++kk) {
            // A: 16 streamed rows = 8 columns, the two halves of a row 32 columns apart; B: 16 rows = 2048 B down every 64-wide chunk
            const uint32_t ao = (kk >> 1) * 32 + (kk & 1) * 8;
            if constexpr (kDKV) {
              ptx::tc_mma_f16_ts(tm + kTmAcc1, a + kTmS + ao, x2 + kk * 128, idesc_a, kk != 0 ? 1u : keep);    // dV += P^T dO
              ptx::tc_mma_f16_ts(tm + kTmAcc2, a + kTmDP + ao, x1 + kk * 128, idesc_a, kk != 0 ? 1u : keep);   // dK += dS^T Q
            } else {
              ptx::tc_mma_f16_ts(tm + kTmAcc1, a + kTmDP + ao, x1 + kk * 128, idesc_a, kk != 0 ? 1u : keep);   // dQ += dS K
            }
          }
          ptx::tc_commit(bar(X_EMPTY + st));
          if (t == n - 1) ptx::tc_commit(bar(ACC_FULL));
        }
        __syncwarp();
      }
    }
  } else {
    // ===================================================== element threads (thread = resident row = TMEM lane, and one half of the columns)
    const int quad = warp & 3, half = (warp - 2) >> 2;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
    const float sl2 = p.scale * 1.4426950408889634f;
    float* my_stats = stats + (warp - 2) * 128;
    const uint32_t stage = sR1 + C::kOut + (warp - 2) * 4096;
    int g = 0;       // steps of this CTA so far
    for (int n_it = 0;; ++n_it) {
      const int slot = n_it & 1;
      wait(IT_FULL + slot, (uint32_t)(n_it >> 1) & 1u);
      const BItem it = items[slot];
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(bar(IT_EMPTY + slot));
      if (it.L < 0 || *dead) break;
      const int L = it.L, tok0 = it.tok0, head = it.head, nblk = blocks(it), blk0 = first_blk(it), n_steps = steps(it);
      const int rw = it.r0 + quad * 32, r_pos = rw + lane;  // key (dKV) / query (dQ) position of this thread inside the sequence
      // step t -> (q head, streamed block)
      auto step_head = [&](int t) { return kDKV ? head * G + t / nblk : head; };
      auto step_blk = [&](int t) { return blk0 + (kDKV ? t % nblk : t); };
      float nlse_r = -INFINITY, ndelta_r = 0.f;  // dQ pass: per-row statistics (-lse * log2e, -delta) in registers
      if constexpr (!kDKV) {
        if (r_pos < L) {
          nlse_r = p.lse[(int64_t)head * p.T + tok0 + r_pos] * -1.4426950408889634f;
          ndelta_r = -p.delta[(int64_t)head * p.T + tok0 + r_pos];
        }
      }
      // dKV: statistics of the warp's 32 streamed queries of a step, -lse * log2e and -delta, one per lane, fetched a step ahead and turned through
      // shared memory of the warp; rows past the end of the sequence get lse = +inf, which zeroes their probabilities
      float nlse = -INFINITY, ndelta = 0.f;
      auto fetch_stats = [&](int t) {
        const int qpos = step_blk(t) * kX + half * 32 + lane;
        nlse = -INFINITY;
        ndelta = 0.f;
        if (qpos < L) {
          const int64_t idx = (int64_t)step_head(t) * p.T + tok0 + qpos;
          nlse = p.lse[idx] * -1.4426950408889634f;
          ndelta = -p.delta[idx];
        }
      };
      if constexpr (kDKV) fetch_stats(0);

      for (int t = 0; t < n_steps; ++t, ++g) {
        const int b = g & 1;
        const int x0 = step_blk(t) * kX + half * 32;  // first streamed position of this warp's columns (query for dKV, key for dQ)
        float* st = my_stats + b * 64;
        if constexpr (kDKV) {
          st[lane] = nlse;
          st[32 + lane] = ndelta;
          if (t + 1 < n_steps) fetch_stats(t + 1);
          __syncwarp();
        }
        wait(S_FULL + b, (uint32_t)(g >> 1) & 1u);
        ptx::tc_fence_after();
        const uint32_t tS = lane_addr + kTmS + b * 64 + half * 32, tDP = lane_addr + kTmDP + b * 64 + half * 32;
        bool need_mask, none;         // some / all elements of the warp's block are hidden (uniform)
        if constexpr (kDKV) {
          need_mask = p.causal && rw + 31 > x0;                        // some key > some query
          none = x0 >= L || (p.causal && rw > x0 + 31);
        } else {
          need_mask = x0 + 32 > L || (p.causal && x0 + 31 > rw);        // key past the end / above the diagonal
          none = x0 >= L || (p.causal && x0 > rw + 31);
        }
        // visible columns of the row: dKV those at or behind its key, dQ those below lim
        const int lim = kDKV ? r_pos - x0 : (p.causal ? min(L, r_pos + 1) : L) - x0;
        uint32_t wp[16], wd[16];
        auto form = [&](auto masked) {
          uint32_t rs[32], rd[32];
          ptx::tc_ld_32x32(tS, rs);
          ptx::tc_ld_32x32(tDP, rd);
          ptx::tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            [[maybe_unused]] float l4[4], d4[4];
            if constexpr (kDKV) {
              *reinterpret_cast<float4*>(l4) = *reinterpret_cast<const float4*>(st + i);
              *reinterpret_cast<float4*>(d4) = *reinterpret_cast<const float4*>(st + 32 + i);
            }
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
              float x0_ = __uint_as_float(rs[i + e]), x1_ = __uint_as_float(rs[i + e + 1]), g0 = __uint_as_float(rd[i + e]), g1 = __uint_as_float(rd[i + e + 1]);
              if constexpr (kDKV) {
                fma_pair2(x0_, x1_, sl2, l4[e], l4[e + 1]);
                add_pair(g0, g1, d4[e], d4[e + 1]);
              } else {
                fma_pair(x0_, x1_, sl2, nlse_r);
                add_pair(g0, g1, ndelta_r, ndelta_r);
              }
              float p0 = exp2f(x0_), p1 = exp2f(x1_);
              if constexpr (decltype(masked)::value) {
                if (kDKV ? i + e < lim : i + e >= lim) p0 = 0.f;
                if (kDKV ? i + e + 1 < lim : i + e + 1 >= lim) p1 = 0.f;
              }
              if constexpr (kDKV) wp[(i + e) >> 1] = pack2<T>(p0, p1);
              mul_pair(g0, g1, p0, p1);
              mul_pair(g0, g1, p.scale, p.scale);
              wd[(i + e) >> 1] = pack2<T>(g0, g1);
            }
          }
        };
        if (none) {
#pragma unroll
          for (int i = 0; i < 16; ++i) wp[i] = wd[i] = 0u;
        } else if (need_mask) {
          form(std::true_type{});
        } else {
          form(std::false_type{});
        }
        if constexpr (kDKV) ptx::tc_st_32x16(tS, wp);
        ptx::tc_st_32x16(tDP, wd);
        ptx::tc_wait_st();
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(bar(P_FULL + b));
      }

      // ---- accumulators -> global, 64 columns at a time through the warp's staging rows; dKV: the first four warps store dV, the others dK; dQ:
      // each half of the warps one 64-column block
      wait(ACC_FULL, (uint32_t)n_it & 1u);
      ptx::tc_fence_after();
      auto release = [&] {
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(bar(ACC_EMPTY));
      };
      if (!kDKV && half >= C::kDBlocks) release();
#pragma unroll
      for (int blk = 0; blk < C::kDBlocks; ++blk) {
        if (!kDKV && blk != half) continue;
        const bool second = kDKV && half == 1;
        const int64_t ld = second ? p.ld2 : p.ld1;
        T* dst = reinterpret_cast<T*>(second ? p.out2 : p.out1) + (int64_t)head * kD + blk * 64 + (lane & 7) * 8;
        uint32_t o[64];
        ptx::tc_ld_32x32(lane_addr + (second ? kTmAcc2 : kTmAcc1) + blk * 64, o);
        ptx::tc_ld_32x32(lane_addr + (second ? kTmAcc2 : kTmAcc1) + blk * 64 + 32, o + 32);
        ptx::tc_wait_ld();
        if (!kDKV || blk == C::kDBlocks - 1) release();
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint32_t v[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) v[e] = pack2<T>(__uint_as_float(o[8 * c + 2 * e]), __uint_as_float(o[8 * c + 2 * e + 1]));
          st_shared_v4(stage + lane * 128 + ((c ^ (lane & 7)) << 4), v[0], v[1], v[2], v[3]);
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int rr = i * 4 + (lane >> 3), pos = rw + rr;
          const uint4 v = ld_shared_v4(stage + rr * 128 + (((lane & 7) ^ (rr & 7)) << 4));
          if (pos < L) *reinterpret_cast<uint4*>(dst + (int64_t)(tok0 + pos) * ld) = v;
        }
        __syncwarp();
      }
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  rb::report_given_up(dead, p.status);
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, 512);
  }
}

// delta[h, t] = sum_d dO[t, h, d] * O[t, h, d]: kD / 8 lanes per (t, h) with 16-byte loads, four (t, h) of a lane group in flight (one
// warp per (t, h) with 4-byte loads: 129 us at 20480 tokens x 32 heads x 128, 2.6 TB/s; now 92)
template <typename T, int kD>
__global__ void __launch_bounds__(256) attn_delta_kernel(const T* __restrict__ out, const T* __restrict__ dout, float* __restrict__ delta, int64_t o_ld,
                                                         int64_t do_ld, int Tn, int nq) {
  constexpr int kLanes = kD / 8, kGroups = 256 / kLanes, kUnroll = 4;
  const int sub = threadIdx.x % kLanes, total = Tn * nq;
  const int w0 = blockIdx.x * kGroups * kUnroll + threadIdx.x / kLanes;
  float acc[kUnroll];
  rb::Pack<T, 8> a[kUnroll], g[kUnroll];
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const int w = w0 + u * kGroups, t = w / nq, h = w - t * nq;
    if (w < total) {
      a[u] = *reinterpret_cast<const rb::Pack<T, 8>*>(out + (int64_t)t * o_ld + (int64_t)h * kD + sub * 8);
      g[u] = *reinterpret_cast<const rb::Pack<T, 8>*>(dout + (int64_t)t * do_ld + (int64_t)h * kD + sub * 8);
    }
  }
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const int w = w0 + u * kGroups, t = w / nq, h = w - t * nq;
    acc[u] = 0.f;
    if (w < total) {
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[u] = fmaf(rb::to_f(a[u].v[i]), rb::to_f(g[u].v[i]), acc[u]);
    }
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], o);
    if (sub == 0 && w < total) delta[(int64_t)h * Tn + t] = acc[u];
  }
}

template <int kD, typename T, int kFmt, bool kDKV>
int launch_bwd(const CUtensorMap& r1, const CUtensorMap& r2, const CUtensorMap& x1, const CUtensorMap& x2, BwdParams p, cudaStream_t s) {
  using C = BCfg<kD>;
  static_assert(C::kSmemBytes <= kMaxSmem, "shared memory");
  auto kern = attn_bwd_kernel<kD, T, kFmt, kDKV>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes) != cudaSuccess) return -30;
    attr_set = true;
  }
  p.heads = kDKV ? p.nkv : p.nq;
  if ((p.status = rb_attn_status()) == nullptr) return -34;
  // the sequences' lengths are on the device: sum of ceil(L / kR) is at most (T + (kR - 1) B) / kR
  const int64_t n = (p.T + (int64_t)(kR - 1) * p.B) / kR * p.heads;
  if (n <= 0 || n > 0x7fffffff) return -33;
  kern<<<dim3((unsigned)n), kBwdThreads, C::kSmemBytes, s>>>(r1, r2, x1, x2, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -31;
}

template <int kD, typename T, int kFmt>
int run_bwd(const void* q, const void* k, const void* v, const void* out, const void* dout, const float* lse, float* delta, void* dq,
            void* dk, void* dv, const int* cu, int64_t q_ld, int64_t k_ld, int64_t v_ld, int64_t o_ld, int64_t do_ld, int64_t dq_ld,
            int64_t dk_ld, int64_t dv_ld, int Tn, int B, int nq, int nkv, int max_seqlen, float scale, int causal, cudaStream_t s) {
  const int bf = kFmt == 1;
  {
    const int per_cta = 256 / (kD / 8) * 4;
    attn_delta_kernel<T, kD><<<RB_CEIL_DIV(Tn * nq, per_cta), 256, 0, s>>>(reinterpret_cast<const T*>(out), reinterpret_cast<const T*>(dout), delta, o_ld,
                                                                           do_ld, Tn, nq);
    if (cudaGetLastError() != cudaSuccess) return -20;
  }
  CUtensorMap q128, do128, k128, v128, q64, do64, k64, v64;
  if (!make_tmap(&k128, k, bf, Tn, (uint64_t)nkv * kD, k_ld, 64, kR) || !make_tmap(&v128, v, bf, Tn, (uint64_t)nkv * kD, v_ld, 64, kR) ||
      !make_tmap(&q64, q, bf, Tn, (uint64_t)nq * kD, q_ld, 64, kX) || !make_tmap(&do64, dout, bf, Tn, (uint64_t)nq * kD, do_ld, 64, kX) ||
      !make_tmap(&q128, q, bf, Tn, (uint64_t)nq * kD, q_ld, 64, kR) || !make_tmap(&do128, dout, bf, Tn, (uint64_t)nq * kD, do_ld, 64, kR) ||
      !make_tmap(&k64, k, bf, Tn, (uint64_t)nkv * kD, k_ld, 64, kX) || !make_tmap(&v64, v, bf, Tn, (uint64_t)nkv * kD, v_ld, 64, kX))
    return -10;
  BwdParams pkv{cu, lse, delta, dv, dk, dv_ld, dk_ld, Tn, B, nq, nkv, 0, scale, causal};
  int rc = launch_bwd<kD, T, kFmt, true>(k128, v128, q64, do64, pkv, s);
  if (rc != 0) return rc;
  BwdParams pq{cu, lse, delta, dq, nullptr, dq_ld, 0, Tn, B, nq, nkv, 0, scale, causal};
  return launch_bwd<kD, T, kFmt, false>(q128, do128, k64, v64, pq, s);
}

}  // namespace

// All tensors are [T, heads, hd] views with unit stride over hd and packed heads; `delta` is an [nq, T] fp32 scratch tensor.
// dt: 1 = bf16, 2 = fp16.  Returns 0 or a negative code.
extern "C" int rb_attn_bwd(const void* q, const void* k, const void* v, const void* out, const void* dout, const float* lse,
                           float* delta, void* dq, void* dk, void* dv, const int* cu_seqlens, int64_t q_ld, int64_t k_ld,
                           int64_t v_ld, int64_t o_ld, int64_t do_ld, int64_t dq_ld, int64_t dk_ld, int64_t dv_ld, int T, int B,
                           int nq, int nkv, int hd, int max_seqlen, float scale, int causal, int dt, cudaStream_t s) {
  if (hd != 128 && hd != 64) return -1;
  if (dt != 1 && dt != 2) return -2;
  if (nq % nkv != 0 || T <= 0 || B <= 0 || max_seqlen <= 0) return -3;
  if ((q_ld | k_ld | v_ld | o_ld | do_ld | dq_ld | dk_ld | dv_ld) % 8 != 0) return -4;
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)dout | (uintptr_t)out | (uintptr_t)dq | (uintptr_t)dk | (uintptr_t)dv) & 15) return -5;
#define RB_RUN(D, TT, F)                                                                                                          \
  return run_bwd<D, TT, F>(q, k, v, out, dout, lse, delta, dq, dk, dv, cu_seqlens, q_ld, k_ld, v_ld, o_ld, do_ld, dq_ld, dk_ld, \
                           dv_ld, T, B, nq, nkv, max_seqlen, scale, causal, s)
  if (hd == 128) {
    if (dt == 1) RB_RUN(128, __nv_bfloat16, 1);
    RB_RUN(128, __half, 0);
  }
  if (dt == 1) RB_RUN(64, __nv_bfloat16, 1);
  RB_RUN(64, __half, 0);
#undef RB_RUN
}
