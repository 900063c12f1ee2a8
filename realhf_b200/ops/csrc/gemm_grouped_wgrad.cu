// Grouped weight-gradient GEMM for MoE experts in ONE launch:
//
//   dW[g] [M, N] (+)= dY_g^T X_g          dY [T, M], X [T, N] hold the tokens sorted by expert, expert g owns the row range [off[g], off[g+1])
//
// Reference: grouped_gemm's `gmm(..., trans_a=True)` in the experts' backward (impl/model/modules/moe/experts.py); the first
// version here ran one GEMM per expert after a host read of the token counts.  This kernel is the wgrad form of the tile GEMM
// (`gemm_tcgen05.cu`: both operands MN-major, K = tokens) with the K range taken per tile from the device-side offsets:
// tile -> (expert, m-tile, n-tile), persistent CTA pairs (cta_group::2, a 256 x BN tile per pair, see gemm_2cta.cu), TMA producer warp / converged
// tcgen05.mma issuer / eight epilogue warps per CTA, smem ring + double-buffered TMEM accumulators.  The last 64-row K block of an expert may reach into
// the next one's rows: its tiles land on the CTA's own barrier, a warp zeroes the foreign rows of the CTA's share of both operands, and the MMAs
// wait for both CTAs' word instead of the ring's.  (Scattering both operands into buffers padded to 64 rows per expert took
// 720 us of an 8 x 14336 x 4096 feed-forward's backward on 4096 rows.)  An expert without tokens gets zeros (or is left alone when accumulating).
//
// What bounds it: with a few hundred tokens per expert a tile is 4096 tensor-pipe cycles and 64 KB of output per SM, so the output has to leave in
// whole lines and as fast as the next tile's MMAs, and a tile of one SM asks L2 for 96 B per cycle and SM; a pair's for 64.  The two products of that
// backward on 8 x 512 rows: rows stored lane by lane 2281 us, whole lines (store_rows32, four warps) 1905, CTA pairs 1770, eight epilogue warps and 16-bit
// staging (store_rows64) 1480 (1.3 PFLOP/s); row counts that are no multiple of 64 cost 1010 us instead of 840 on the larger one.
#include "cta_pair.cuh"

namespace {

struct WgradParams {
  void* C;          // [G, M, N]
  const int* off;   // [G + 1]
  int G, M, N;
  int accumulate;
};

constexpr int kEpiWarps = 8;         // two per TMEM quadrant, half of the columns each
constexpr int kWgradThreads = 32 * (3 + kEpiWarps);   // warps 0 TMA, 1 MMA (leader), 2-9 epilogue, 10 tail rows

template <int BN> struct WCfg {
  static constexpr int kStages = BN >= 256 ? 6 : 8;
  static constexpr int kABytes = BM * BK * 2;         // [2 chunks of 64 m][64 k rows][128 B]
  static constexpr int kBBytes = BN / 2 * BK * 2;     // [BN / 128 chunks][64 k rows][128 B]: this CTA's half of the columns
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kOut = kStages * kStageBytes, kBars = kOut + kEpiWarps * 4096;   // 4 KB of output staging per epilogue warp
  static constexpr int kSmemBytes = kBars + 1024 + 512;
};

template <int BN, typename OutT>
__global__ void __launch_bounds__(kWgradThreads, 1) grouped_wgrad_kernel(const __grid_constant__ CUtensorMap tma_a,
                                                                         const __grid_constant__ CUtensorMap tma_b, WgradParams p) {
  using C = WCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* smem_a = smem;
  uint8_t* smem_b = smem + C::kStages * C::kABytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kBars);
  uint64_t* full_bar = bars;                       // leader: both CTAs' bytes of an ordinary stage
  uint64_t* empty_bar = bars + C::kStages;         // one per CTA, armed by the leader's multicast commit
  uint64_t* mine_bar = bars + 2 * C::kStages;      // one per CTA: its own bytes of an expert's last, partial stage
  uint64_t* tail_bar = bars + 3 * C::kStages;      // leader: both CTAs' foreign rows of such a stage are zero
  uint64_t* tmem_full = bars + 4 * C::kStages;     // one per CTA
  uint64_t* tmem_empty = tmem_full + 2;            // leader, one arrival per epilogue warp of both CTAs
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(tmem_empty + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int tiles_m = RB_CEIL_DIV(p.M, 2 * BM), tiles_n = RB_CEIL_DIV(p.N, BN);
  const int tpg = tiles_m * tiles_n;
  const int num_tiles = p.G * tpg;
  // tile -> (expert, m0, n0, first token row, number of 64-row K blocks, real rows of the last one); m fastest so neighbouring CTAs share the X panel
  auto coords = [&](int tile, int& g, int& m0, int& n0, int& r0, int& nkb, int& tail) {
    g = tile / tpg;
    const int local = tile - g * tpg;
    m0 = (local % tiles_m) * (2 * BM);
    n0 = (local / tiles_m) * BN;
    r0 = p.off[g];
    const int rows = p.off[g + 1] - r0;
    nkb = RB_CEIL_DIV(rows, BK);
    tail = rows - (nkb - 1) * BK;
  };
  // A partial block is the first of its tile: it is loaded and cleaned while the MMAs are on the previous tile.
  auto block = [](int kb, int nkb, int tail) { return tail == BK ? kb : kb == 0 ? nkb - 1 : kb - 1; };

  if (warp == 0 && lane == 0) {
    ptx::prefetch_tensormap(&tma_a);
    ptx::prefetch_tensormap(&tma_b);
    for (int i = 0; i < C::kStages; ++i) {
      ptx::mbar_init(ptx::smem_u32(&full_bar[i]), 1);
      ptx::mbar_init(ptx::smem_u32(&empty_bar[i]), 1);
      ptx::mbar_init(ptx::smem_u32(&mine_bar[i]), 1);
      ptx::mbar_init(ptx::smem_u32(&tail_bar[i]), 2);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(ptx::smem_u32(&tmem_full[i]), 1);
      ptx::mbar_init(ptx::smem_u32(&tmem_empty[i]), 2 * kEpiWarps);
    }
    ptx::fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc_cg2(ptx::smem_u32(tmem_ptr), 2 * BN);
    tmem_relinquish_cg2();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync();  // the peer's barriers must exist before any remote arrive / multicast commit / cross-CTA TMA completion
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int tile = pair; tile < num_tiles; tile += num_pairs) {
        int g, m0, n0, r0, nkb, tail;
        coords(tile, g, m0, n0, r0, nkb, tail);
        for (int kb = 0; kb < nkb; ++kb) {
          ptx::mbar_wait(ptx::smem_u32(&empty_bar[stage]), phase ^ 1);
          const uint32_t sa = ptx::smem_u32(smem_a + stage * C::kABytes);
          const uint32_t sb = ptx::smem_u32(smem_b + stage * C::kBBytes);
          const int k0 = r0 + block(kb, nkb, tail) * BK, ma = m0 + (int)rank * BM, nb = n0 + (int)rank * (BN / 2);
          if (kb == 0 && tail < BK) {
            const uint32_t fb = ptx::smem_u32(&mine_bar[stage]);
            ptx::mbar_arrive_expect_tx(fb, C::kStageBytes);
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) ptx::tma_load_2d(sa + j * (BK * 128), &tma_a, fb, ma + 64 * j, k0);
#pragma unroll
            for (int j = 0; j < BN / 128; ++j) ptx::tma_load_2d(sb + j * (BK * 128), &tma_b, fb, nb + 64 * j, k0);
          } else {
            const uint32_t fb_local = ptx::smem_u32(&full_bar[stage]);
            if (leader) ptx::mbar_arrive_expect_tx(fb_local, 2 * C::kStageBytes);  // both CTAs' bytes land on this barrier
            const uint32_t fb = mapa_u32(fb_local, 0);
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d_cg2(sa + j * (BK * 128), &tma_a, fb, ma + 64 * j, k0);
#pragma unroll
            for (int j = 0; j < BN / 128; ++j) tma_load_2d_cg2(sb + j * (BK * 128), &tma_b, fb, nb + 64 * j, k0);
          }
          if (++stage == C::kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (leader) {
      constexpr uint32_t idesc = ptx::make_idesc_f16(1, 2 * BM, BN, 1, 1);
      const uint32_t tm = (uint32_t)ptx::uniform((int)tmem_base);
      int stage = 0, as = 0;
      uint32_t aphase = 0, fulls = 0, tails = 0;     // bit s: phase of full_bar[s] / tail_bar[s] (a stage fills by one of the two)
      for (int tile = pair; tile < num_tiles; tile += num_pairs) {
        int g, m0, n0, r0, nkb, tail;
        coords(tile, g, m0, n0, r0, nkb, tail);
        nkb = ptx::uniform(nkb);
        tail = ptx::uniform(tail);
        ptx::mbar_wait(ptx::smem_u32(&tmem_empty[as]), aphase ^ 1);
        ptx::tc_fence_after();
        const uint32_t d_tmem = tm + as * BN;
        for (int kb = 0; kb < nkb; ++kb) {
          if (kb == 0 && tail < BK) {
            mbar_wait_cluster(ptx::smem_u32(&tail_bar[stage]), (tails >> stage) & 1u);
            tails ^= 1u << stage;
          } else {
            ptx::mbar_wait(ptx::smem_u32(&full_bar[stage]), (fulls >> stage) & 1u);
            fulls ^= 1u << stage;
          }
          ptx::tc_fence_after();
          const uint64_t da = ptx::make_smem_desc_sw128(ptx::smem_u32(smem_a + stage * C::kABytes), BK * 128, 1024);
          const uint64_t db = ptx::make_smem_desc_sw128(ptx::smem_u32(smem_b + stage * C::kBBytes), BK * 128, 1024);
          if (ptx::elect_one()) {
#pragma unroll
            for (int k = 0; k < BK / 16; ++k) tc_mma_f16_cg2(d_tmem, da + k * 128, db + k * 128, idesc, (kb | k) != 0 ? 1u : 0u);
            tc_commit_cg2(ptx::smem_u32(&empty_bar[stage]), 0b11);
          }
          __syncwarp();
          if (++stage == C::kStages) stage = 0;
        }
        if (ptx::elect_one()) tc_commit_cg2(ptx::smem_u32(&tmem_full[as]), 0b11);  // with nkb == 0 nothing is pending: arrives at once
        __syncwarp();
        if (++as == 2) { as = 0; aphase ^= 1; }
      }
    }
  } else if (warp == 2 + kEpiWarps) {
    // ===================================================== rows of the next expert (or of nobody) in an expert's last K block: zero in this CTA's share
    int stage = 0;
    uint32_t phases = 0;      // bit s: phase of mine_bar[s], which only such stages use
    for (int tile = pair; tile < num_tiles; tile += num_pairs) {
      int g, m0, n0, r0, nkb, tail;
      coords(tile, g, m0, n0, r0, nkb, tail);
      if (nkb > 0 && tail < BK) {
        const int st = stage;
        ptx::mbar_wait(ptx::smem_u32(&mine_bar[st]), (phases >> st) & 1u);
        phases ^= 1u << st;
        // chunks of 64 columns: [64 token rows][128 B], rows unswizzled among themselves
        for (int c = 0; c < BM / 64 + BN / 128; ++c) {
          uint8_t* base = c < BM / 64 ? smem_a + st * C::kABytes + c * (BK * 128) : smem_b + st * C::kBBytes + (c - BM / 64) * (BK * 128);
          for (int i = tail * 8 + lane; i < BK * 8; i += 32) reinterpret_cast<uint4*>(base)[i] = make_uint4(0u, 0u, 0u, 0u);
        }
        asm volatile("fence.proxy.async;" ::: "memory");      // (the leader's MMAs read both CTAs' shared memory)
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(ptx::smem_u32(&tail_bar[st]), 0);
      }
      stage = (stage + nkb) % C::kStages;
    }
  } else {
    const int quad = warp & 3, half = (warp - 2) >> 2;
    int as = 0;
    uint32_t aphase = 0;
    OutT* Cp = reinterpret_cast<OutT*>(p.C);
    const uint32_t out_stage = ptx::smem_u32(smem + C::kOut + (warp - 2) * 4096);
    const bool vec_ok = (p.N % (16 / sizeof(OutT)) == 0) && ((reinterpret_cast<uintptr_t>(p.C) & 15) == 0);
    for (int tile = pair; tile < num_tiles; tile += num_pairs) {
      int g, m0, n0, r0, nkb, tail;
      coords(tile, g, m0, n0, r0, nkb, tail);
      ptx::mbar_wait(ptx::smem_u32(&tmem_full[as]), aphase);
      ptx::tc_fence_after();
      const int row0 = m0 + (int)rank * BM + quad * 32;
      const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + as * BN + half * (BN / 2);
      n0 += half * (BN / 2);
      OutT* dst = Cp + ((int64_t)g * p.M + row0) * p.N + n0;
      if (sizeof(OutT) == 2 && vec_ok && !p.accumulate && nkb > 0 && n0 + BN / 2 <= p.N && row0 + 32 <= p.M) {
#pragma unroll 1
        for (int c = 0; c < BN / 2; c += 64) {
          uint32_t r[64];
          ptx::tc_ld_32x32(taddr + c, r);
          ptx::tc_ld_32x32(taddr + c + 32, r + 32);
          ptx::tc_wait_ld();
          store_rows64<OutT>(out_stage, r, dst + c, p.N);
        }
      } else {
#pragma unroll 1
        for (int c = 0; c < BN / 2; c += 32) {
          uint32_t r[32];
          ptx::tc_ld_32x32(taddr + c, r);  // warp-collective: executed by every lane whatever its row
          ptx::tc_wait_ld();
          const int n_valid = min(32, p.N - n0 - c);
          if (row0 < p.M && n_valid > 0 && !(nkb == 0 && p.accumulate)) {
            float v[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = nkb == 0 ? 0.f : __uint_as_float(r[i]);  // no tokens: the accumulator is stale
            store_rows32<OutT>(out_stage, v, dst + c, p.N, p.M - row0, n_valid, vec_ok, p.accumulate);
          }
        }
      }
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(ptx::smem_u32(&tmem_empty[as]), 0);
      if (++as == 2) { as = 0; aphase ^= 1; }
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync();  // neither CTA may free TMEM or exit while the pair's MMAs / remote arrivals are in flight
  if (warp == 1) {
    ptx::tc_fence_after();
    tmem_dealloc_cg2(tmem_base, 2 * BN);
  }
}

template <int BN, typename OutT>
int launch_wgrad(const CUtensorMap& ta, const CUtensorMap& tb, const WgradParams& p, int num_sms, cudaStream_t s) {
  using C = WCfg<BN>;
  auto kern = grouped_wgrad_kernel<BN, OutT>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes) != cudaSuccess) return -30;
    attr_set = true;
  }
  const int64_t tiles = (int64_t)p.G * RB_CEIL_DIV(p.M, 2 * BM) * RB_CEIL_DIV(p.N, BN);
  const int pairs = num_sms / 2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(2 * (tiles < pairs ? tiles : pairs)));
  cfg.blockDim = dim3(kWgradThreads);
  cfg.dynamicSmemBytes = C::kSmemBytes;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, kern, ta, tb, p) != cudaSuccess) return -31;
  return cudaGetLastError() == cudaSuccess ? 0 : -31;
}

}  // namespace

// dy [Tp, M], x [Tp, N] bf16 (row pitches ld*), offsets: device int32 [G + 1], nondecreasing, offsets[G] <= Tp; out [G, M, N] contiguous, fp32 (out_dt 0) or bf16 (out_dt 1); accumulate: out += result.
extern "C" int rb_gemm_grouped_wgrad(const void* dy, const void* x, void* out, const int* offsets, int G, int Tp, int M, int N,
                                     int64_t ld_dy, int64_t ld_x, int out_dt, int accumulate, int num_sms, cudaStream_t s) {
  if (G <= 0 || M <= 0 || N <= 0) return 0;
  if (Tp <= 0) return -1;
  if ((ld_dy % 8) || (ld_x % 8) || (reinterpret_cast<uintptr_t>(dy) & 15) || (reinterpret_cast<uintptr_t>(x) & 15)) return -11;
  if (M % 8 || N % 8) return -12;
  if (num_sms <= 0) num_sms = rb::kNumSMs;
  CUtensorMap ta, tb;
  // MN-major operands: the tensor maps address [rows = tokens, cols = features] with 64 x 64 boxes (same as the dense wgrad)
  if (!make_tmap(&ta, dy, 1, (uint64_t)Tp, (uint64_t)M, (uint64_t)ld_dy, 64, BK) ||
      !make_tmap(&tb, x, 1, (uint64_t)Tp, (uint64_t)N, (uint64_t)ld_x, 64, BK))
    return -13;
  WgradParams p{out, offsets, G, M, N, accumulate};
  const bool wide = N % 256 == 0;
  if (out_dt == 0) return wide ? launch_wgrad<256, float>(ta, tb, p, num_sms, s) : launch_wgrad<128, float>(ta, tb, p, num_sms, s);
  if (out_dt == 1) return wide ? launch_wgrad<256, __nv_bfloat16>(ta, tb, p, num_sms, s) : launch_wgrad<128, __nv_bfloat16>(ta, tb, p, num_sms, s);
  return -14;
}
