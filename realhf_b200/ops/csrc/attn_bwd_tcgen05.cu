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
// heads: dKV 613, dQ 506 us, now 412, 388; 8 x 1500..4096, 32 / 8 heads: 2473, 2109 us, now 1777, 1662).
//
// delta[h, t] = sum_d dO[t, h, d] * O[t, h, d] comes from a small pre-pass; LSE is the forward's ([nq, T], natural log).
#include "attn_common.cuh"

namespace {

constexpr int kR = 128;   // resident rows per CTA (= UMMA M)
constexpr int kX = 64;    // streamed rows per step (= UMMA N of the S-type products, K of the accumulating ones)
constexpr int kXStages = 4;
constexpr int kBwdThreads = 320;   // warp 0: TMA, warp 1: MMA, warps 2-9: elements (two per TMEM quadrant, one per column half)

struct BwdParams {
  const int* cu_seqlens;
  const float* lse;    // [nq, T]
  const float* delta;  // [nq, T]
  void* out1;          // dKV pass: dV;  dQ pass: dQ      ([T, heads, D] views, row pitch ld1)
  void* out2;          // dKV pass: dK
  int64_t ld1, ld2;
  int T, nq, nkv;
  float scale;
  int causal;
};

template <int kD> struct BCfg {
  static constexpr int kDBlocks = kD / 64;
  static constexpr int kRBytes = kR * kD * 2;     // one resident tile
  static constexpr int kXBytes = kX * kD * 2;     // one streamed tile
  static constexpr int kBars = 2 * kRBytes + kXStages * 2 * kXBytes;
  static constexpr int kStats = kBars + 256;      // [2 buffers][lse | delta][64]
  static constexpr int kSmemBytes = kStats + 2 * 2 * kX * 4 + 1024 /*align*/;
};

enum BBar { R_FULL = 0, X_FULL = 1, X_EMPTY = X_FULL + kXStages, S_FULL = X_EMPTY + kXStages, P_FULL = S_FULL + 2, ACC_FULL = P_FULL + 2,
            B_NUM_BARS = ACC_FULL + 1 };

__device__ int g_wait_error = 0;

RB_DEVICE void element_bar_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// tma_r1 / tma_r2: resident operands (box 64 cols x 128 rows); tma_x1 / tma_x2: streamed operands (box 64 x 64).
//   kDKV: r1 = K, r2 = V (kv-head columns), x1 = Q, x2 = dO (q-head columns).   !kDKV: r1 = Q, r2 = dO, x1 = K, x2 = V.
template <int kD, typename T, int kFmt, bool kDKV>
__global__ void __launch_bounds__(kBwdThreads, 1) attn_bwd_kernel(const __grid_constant__ CUtensorMap tma_r1,
                                                                  const __grid_constant__ CUtensorMap tma_r2,
                                                                  const __grid_constant__ CUtensorMap tma_x1,
                                                                  const __grid_constant__ CUtensorMap tma_x2, const __grid_constant__ BwdParams p) {
  using C = BCfg<kD>;
  const int seq = blockIdx.z, head = blockIdx.y;  // kDKV: kv head; else q head
  const int tile = kDKV ? (int)blockIdx.x : (int)(gridDim.x - 1 - blockIdx.x);  // heaviest tiles first in both passes
  const int tok0 = p.cu_seqlens[seq];
  const int L = p.cu_seqlens[seq + 1] - tok0;
  const int r0 = tile * kR;  // first key (dKV) / first query (dQ) of this CTA inside the sequence
  if (r0 >= L) return;
  const int G = p.nq / p.nkv;
  const int nblk_all = RB_CEIL_DIV(L, kX);
  // streamed block range [blk0, blk1): dKV -> query blocks that can see these keys; dQ -> key blocks these queries can see
  const int blk0 = kDKV ? (p.causal ? r0 / kX : 0) : 0;
  const int blk1 = kDKV ? nblk_all : (p.causal ? RB_CEIL_DIV(min(L, r0 + kR), kX) : nblk_all);
  const int nblk = blk1 - blk0;
  const int n_steps = kDKV ? nblk * G : nblk;  // dKV also walks the q heads of the group (outer loop)

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t sR1 = ptx::smem_u32(smem);
  const uint32_t sR2 = sR1 + C::kRBytes;
  const uint32_t sX = sR2 + C::kRBytes;            // stage s: X1 at sX + s * 2 * kXBytes, X2 right after it
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kBars);
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(bars + B_NUM_BARS);
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
    for (int i = 0; i < B_NUM_BARS; ++i) ptx::mbar_init(bar(i), (i == P_FULL || i == P_FULL + 1) ? 8 : 1);   // one arrival per element warp
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

  // step t -> (q head, streamed block)
  auto step_head = [&](int t) { return kDKV ? head * G + t / nblk : head; };
  auto step_blk = [&](int t) { return blk0 + (kDKV ? t % nblk : t); };

  if (warp == 0) {
    // ===================================================== TMA producer
    if (lane == 0) {
      const int x_kv_head = kDKV ? head : head / G;            // dQ pass streams the kv head of this q head
      ptx::mbar_arrive_expect_tx(bar(R_FULL), 2 * C::kRBytes);
#pragma unroll
      for (int kb = 0; kb < C::kDBlocks; ++kb) {
        ptx::tma_load_2d(sR1 + kb * (kR * 128), &tma_r1, bar(R_FULL), head * kD + kb * 64, tok0 + r0);
        ptx::tma_load_2d(sR2 + kb * (kR * 128), &tma_r2, bar(R_FULL), head * kD + kb * 64, tok0 + r0);
      }
      for (int t = 0; t < n_steps; ++t) {
        const int st = t % kXStages;
        const int row = tok0 + step_blk(t) * kX;
        const int col = (kDKV ? step_head(t) : x_kv_head) * kD;
        wait(X_EMPTY + st, ((uint32_t)(t / kXStages) & 1u) ^ 1u);
        ptx::mbar_arrive_expect_tx(bar(X_FULL + st), 2 * C::kXBytes);
        const uint32_t x1 = sX + st * 2 * C::kXBytes, x2 = x1 + C::kXBytes;
#pragma unroll
        for (int kb = 0; kb < C::kDBlocks; ++kb) {
          ptx::tma_load_2d(x1 + kb * (kX * 128), &tma_x1, bar(X_FULL + st), col + kb * 64, row);
          ptx::tma_load_2d(x2 + kb * (kX * 128), &tma_x2, bar(X_FULL + st), col + kb * 64, row);
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ===================================================== MMA issuer: the whole warp runs the loop, one elected lane issues
    constexpr uint32_t idesc_s = ptx::make_idesc_f16(kFmt, kR, kX, 0, 0);   // resident x streamed^T, both K-major
    constexpr uint32_t idesc_a = ptx::make_idesc_f16(kFmt, kR, kD, 0, 1);   // P-type (TMEM) x streamed (MN-major)
    const uint32_t tm = (uint32_t)ptx::uniform((int)tmem_base);
    const int n = ptx::uniform(n_steps);
    const uint64_t r1 = ptx::make_smem_desc_sw128(sR1, 16, 1024), r2 = ptx::make_smem_desc_sw128(sR2, 16, 1024);
    auto issue_sdp = [&](int t) {
      const int st = t % kXStages;
      wait(X_FULL + st, (uint32_t)(t / kXStages) & 1u);
      ptx::tc_fence_after();
      const uint32_t d = tm + (t & 1) * 64;
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
        ptx::tc_commit(bar(S_FULL + (t & 1)));
      }
      __syncwarp();
    };
    wait(R_FULL, 0);
    issue_sdp(0);
    for (int t = 0; t < n; ++t) {
      if (t + 1 < n) issue_sdp(t + 1);       // its S / dP columns: the products that read P of step t-1 there are ahead in the pipe
      const int st = t % kXStages;
      wait(P_FULL + (t & 1), (uint32_t)(t >> 1) & 1u);
      ptx::tc_fence_after();
      const uint32_t a = tm + (t & 1) * 64;
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
  } else {
    // ===================================================== element threads (thread = resident row = TMEM lane, and one half of the columns)
    const int quad = warp & 3, half = (warp - 2) >> 2;
    const int row = quad * 32 + lane, tid = threadIdx.x - 64;
    const int r_pos = r0 + row;  // key (dKV) / query (dQ) position of this thread inside the sequence
    const int rw = r0 + quad * 32;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
    const float sl2 = p.scale * 1.4426950408889634f;
    float lse_r = INFINITY, delta_r = 0.f;  // dQ pass: per-row statistics in registers
    if constexpr (!kDKV) {
      if (r_pos < L) {
        lse_r = p.lse[(int64_t)head * p.T + tok0 + r_pos] * 1.4426950408889634f;
        delta_r = p.delta[(int64_t)head * p.T + tok0 + r_pos];
      }
    }
    // dKV: statistics of a step's 64 streamed queries, [lse * log2e | delta], fetched a step ahead by the first 128 threads; rows past the end of
    // the sequence get lse = +inf, which zeroes their probabilities
    auto fetch_stat = [&](int t) {
      float v = tid < 64 ? INFINITY : 0.f;
      const int qpos = step_blk(t) * kX + (tid & 63);
      if (tid < 128 && qpos < L) {
        const int64_t idx = (int64_t)step_head(t) * p.T + tok0 + qpos;
        v = tid < 64 ? p.lse[idx] * 1.4426950408889634f : p.delta[idx];
      }
      return v;
    };
    float stat = kDKV ? fetch_stat(0) : 0.f;

    for (int t = 0; t < n_steps; ++t) {
      const int b = t & 1;
      const int x0 = step_blk(t) * kX + half * 32;  // first streamed position of this warp's columns (query for dKV, key for dQ)
      if constexpr (kDKV) {
        if (tid < 128) stats[b * 128 + tid] = stat;
        if (t + 1 < n_steps) stat = fetch_stat(t + 1);
        element_bar_sync();
      }
      wait(S_FULL + b, (uint32_t)(t >> 1) & 1u);
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
      uint32_t wp[16], wd[16];
      if (none) {
#pragma unroll
        for (int i = 0; i < 16; ++i) wp[i] = wd[i] = 0u;
      } else {
        uint32_t rs[32], rd[32];
        ptx::tc_ld_32x32(tS, rs);
        ptx::tc_ld_32x32(tDP, rd);
        ptx::tc_wait_ld();
        float lse4[4], del4[4];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          if constexpr (kDKV) {
            if (i % 4 == 0) {
              *reinterpret_cast<float4*>(lse4) = *reinterpret_cast<const float4*>(stats + b * 128 + half * 32 + i);
              *reinterpret_cast<float4*>(del4) = *reinterpret_cast<const float4*>(stats + b * 128 + 64 + half * 32 + i);
            }
          }
          float pr[2], ds[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float lse_c = kDKV ? lse4[(i + e) & 3] : lse_r, del_c = kDKV ? del4[(i + e) & 3] : delta_r;
            float pv = exp2f(fmaf(__uint_as_float(rs[i + e]), sl2, -lse_c));
            if (need_mask) {
              const int xpos = x0 + i + e;
              const bool vis = kDKV ? (r_pos <= xpos) : (xpos < L && (!p.causal || xpos <= r_pos));
              if (!vis) pv = 0.f;
            }
            pr[e] = pv;
            ds[e] = pv * (__uint_as_float(rd[i + e]) - del_c) * p.scale;
          }
          wp[i >> 1] = pack2<T>(pr[0], pr[1]);
          wd[i >> 1] = pack2<T>(ds[0], ds[1]);
        }
      }
      if constexpr (kDKV) ptx::tc_st_32x16(tS, wp);
      ptx::tc_st_32x16(tDP, wd);
      ptx::tc_wait_st();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(bar(P_FULL + b));
    }

    // ---- accumulators -> global, 64 columns at a time through the warp's staging rows (the streamed ring is done with): dKV: the first four
    // warps store dV, the others dK; dQ: each half of the warps one 64-column block
    wait(ACC_FULL, 0);
    ptx::tc_fence_after();
    const uint32_t stage = sX + (warp - 2) * 4096;
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

  ptx::tc_fence_before();
  __syncthreads();
  if (*dead) {
    if (threadIdx.x == 0) g_wait_error = 1;
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    __syncthreads();
  }
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
int launch_bwd(const CUtensorMap& r1, const CUtensorMap& r2, const CUtensorMap& x1, const CUtensorMap& x2, const BwdParams& p,
               int heads, int B, int max_seqlen, cudaStream_t s) {
  using C = BCfg<kD>;
  auto kern = attn_bwd_kernel<kD, T, kFmt, kDKV>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes) != cudaSuccess) return -30;
    attr_set = true;
  }
  dim3 grid(RB_CEIL_DIV(max_seqlen, kR), heads, B);
  kern<<<grid, kBwdThreads, C::kSmemBytes, s>>>(r1, r2, x1, x2, p);
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
  BwdParams pkv{cu, lse, delta, dv, dk, dv_ld, dk_ld, Tn, nq, nkv, scale, causal};
  int rc = launch_bwd<kD, T, kFmt, true>(k128, v128, q64, do64, pkv, nkv, B, max_seqlen, s);
  if (rc != 0) return rc;
  BwdParams pq{cu, lse, delta, dq, nullptr, dq_ld, 0, Tn, nq, nkv, scale, causal};
  return launch_bwd<kD, T, kFmt, false>(q128, do128, k64, v64, pq, nq, B, max_seqlen, s);
}

}  // namespace

extern "C" int rb_attn_bwd_wait_error() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_wait_error, sizeof(int)) != cudaSuccess) return -1;
  if (v != 0) cudaMemcpyToSymbol(g_wait_error, &zero, sizeof(int));
  return v;
}

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
