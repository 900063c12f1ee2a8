// Packed variable-length (causal) attention forward for sm_100a: TMA -> shared (128B swizzle) -> tcgen05.mma -> TMEM.
//
//   O[t, h, :] = softmax(scale * Q[t, h, :] K[seq(t), kv(h), :]^T  (+ causal mask)) V        bf16 / fp16, fp32 softmax
//
// Optional sliding window (causal only): query i sees keys (i - window, i].  Reference: flash-attn's `flash_attn_varlen_func` called
// from `impl/model/modules/attn.py:240-262`.
//
// What bounds it: per 128 x 128 tile the two products take 1024 tensor-pipe cycles at D = 128 and the 16384 exponentials as many cycles
// of the special-function unit, so the tensor pipe is only busy while some other tile's softmax runs beside it.  A work item is therefore
// a PAIR of 128-row query tiles over one K / V stream, each with softmax threads of its own: two query heads of one key head at the same
// rows (grouped heads, even group: both walk the same tiles), else two neighbouring query tiles of a head (counted from the end of
// the sequence, so that a left-over single tile is the shortest one).  Sharing the stream also halves the L2 traffic per product: one
// tile each would ask for 64 B per cycle and SM, more than L2 gives.  With one tile per CTA and four softmax warps the tensor pipe was
// active 19% of the time.
//
// CTA = 16 warps, one CTA per SM.  Warps 0-3 / 4-7: softmax of tile 0 / 1 (thread = query row = TMEM lane).  Warp 8: MMA issue and TMEM
// allocation.  Warp 9: TMA producer and scheduler (10, 11: idle, they complete the warpgroup whose registers go to the softmax).  Warps 12-15 (one per
// TMEM quadrant, both tiles): they scale O and write it out.  With both left to the softmax warps a key tile cost them 470 of 2370 cycles for the scaling, and the
// output, 5000 cycles a pair of tiles, lay between two items: 32 x 640 tokens x 32 heads 232 -> 188 us, 8 x 1500..4096 x 32 / 8 heads
// 839 -> 734 us in short bursts (long ones run into the power limit, 1.7 GHz, and keep a tenth of that), 32 x 1024 tokens with window 512 + 64 kept
// 270 -> 224 us, 300..777 tokens of 12 heads with window 500 114 -> 99 us.  Of that the masks as words and the three-way maximum are 210 -> 201 on 640 tokens
// and 414 -> 263 with a window (masks element by element spill here).  What bounds it
// now, per key tile and query tile: 580 cycles to the maximum, 1500 for the 128 exponentials of a thread (1090 at 8.5 cycles each if nothing else ran), 1360
// from the weights to the next scores (two products, 1024).  Two tiles share the tensor pipe: active 33 % of the time on items of five key tiles, 52 % on 1500..4096
// tokens.  Every second pair of exponentials by a polynomial on the multiply-add units was slower (10.9 cycles each).
//
// The grid holds one CTA per work item (a bound: sequence lengths are on the device); a running CTA takes the items of CTAs that have
// not started (`clusterlaunchcontrol.try_cancel`), so barriers, TMEM and descriptors are set up once per SM, the next item's Q / K / V
// load while the last one's softmax and output run, and ragged batches balance themselves.
//
// Tensor memory (512 columns): S_t at 128 t, O_t at 256 + 128 t.  P_t (16 bit) overwrites the front of S_t and is the TMEM A operand of
// P V, so it never travels through shared memory; S_t of the next tile is issued behind that product on the in-order tensor pipe.  O
// accumulates in TMEM over the whole stream; when a row's maximum grows, its factor goes to the output warp of its quadrant, which scales O while the weights
// are formed: the product before has retired (the scores that showed the growth were issued behind it), and the next one waits for both.  (A maximum
// that only moves when weights exceed it by 2^8 is 2..3 % faster in training, 10 % with a window, but the largest weight is then no longer exactly
// 1 when P is rounded to 16 bits: error against 64 bits 0.0028 instead of 0.0025.)  V_j is the MN-major B operand.
// Issue order: S_0, S_1, then per key tile PV_0, S_0', PV_1, S_1'.  The issuing warp runs converged, the MMAs are predicated on an elected lane: issued from
// `if (lane == 0)` with descriptors built there, eight MMAs took 820-960 cycles of one thread, whatever their size.  (Behind one branch of the elected lane, S alone or all,
// windowed prefill is 3 % faster and 39 of 282 forms by 2 .. 5 %, but items of one key tile without grouped heads are 4 % slower; both in one kernel: most forms slower, up to 14 %.)
//
// Outputs: O [T, nq, DV] through a per-warp staging buffer (whole 128-byte lines), LSE [nq, T] (natural log, scale applied).
//
// Modes (`WindowAttentionConfig`, inference only, no LSE): kGeneral: score = s * scale * temp_h - slope_h * (i - j) with slope_h =
// 2^(-slope_base (h + 1) / nq) (log2 domain, two FMAs per score), a sliding window that also keeps the first `keep` keys (their
// tiles below the window's first tile are walked first).  kSimple: no distance term, temperature or kept keys and a positive scale: the
// maximum is taken over the raw products.  kCap: kSimple with score = softcap * tanh(s * scale / softcap), formed before the
// masks, so that a product that overflowed to -infinity is a visible score of -softcap.  All three: a per-head sink logit starts the running maximum with denominator 1; the output is
// multiplied by sigmoid(gate logit of its head, or of the output element); `chunk` > 0 replaces the window: a query sees the keys of its own
// chunk of positions up to itself.
// Learned distance biases and shared keys / values run in attn_fwd_bias.cu.
#include "attn_common.cuh"

namespace {

constexpr int kTile = 128;          // query rows of a tile (= UMMA M) and keys of a tile (= UMMA N of S, K of P V)
constexpr int kFwdThreads = 512;    // four warpgroups: 128 registers a thread at launch
constexpr int kSoftmaxRegs = 184, kOtherRegs = 64, kOutRegs = 80;   // 128 x (2 x 184 + 64 + 80) = 65536: a softmax thread holds a whole score row
constexpr int kStages = 4;          // K and V tiles share one ring: two key tiles in flight

enum Mode { kPlain = 0, kSimple = 1, kCap = 2, kGeneral = 3 };

template <int kD, int kDV> struct FCfg {
  static constexpr int kQBytes = kTile * kD * 2, kKBytes = kTile * kD * 2, kVBytes = kTile * kDV * 2;
  static constexpr int kStageBytes = kKBytes > kVBytes ? kKBytes : kVBytes;
  static constexpr int kKV = 2 * kQBytes, kOut = kKV + kStages * kStageBytes, kRows = kOut + 4 * 4096, kBars = kRows + 2 * 3 * kTile * 4;
  static constexpr int kSmemBytes = kBars + 512 /*barriers, items*/;
};

enum FBar { Q_FULL = 0, Q_EMPTY = 2, KV_FULL = 4, KV_EMPTY = 8, S_FULL = 12, P_FULL = 14, O_FULL = 16, A_FULL = 18 /* [tile][quadrant] */, L_FULL = 26, L_EMPTY = 28,
            IT_FULL = 30, IT_EMPTY = 32, CLC_FULL = 34, F_NUM_BARS = 35 };
constexpr int kItemReaders = 1 + 8 + 4;      // MMA, softmax and output warps

// One work item: sequence (first token, length), heads and query tiles of the two tiles (tile 1 < 0: absent); L < 0 ends the CTA's loop.
struct Item { int tok0, L, head0, head1, qt0, qt1; };

// The key tiles of an item: the kept first tiles [0, nk), then [lo, end); a tile takes part in key tile j when j < its end and j is at or
// behind its first tile or among the kept ones.  (Plain numbers, no arrays: indexing them by a run-time tile would go through memory.)
struct Walk {
  int first0, end0, first1, end1, keep_tiles, nk, lo, n;
  RB_DEVICE Walk(const Item& it, const AttnParams& p) {
    const int win = (p.causal && p.window > 0) ? p.window : 0;
    keep_tiles = win > 0 ? RB_CEIL_DIV(p.keep, kTile) : 0;
    auto first = [&](int qt) { const int q0 = qt * kTile; return p.chunk > 0 ? (q0 / p.chunk * p.chunk) / kTile : win > 0 ? max(0, q0 - win + 1) / kTile : 0; };
    auto end = [&](int qt) { return qt < 0 ? 0 : RB_CEIL_DIV(p.causal ? min(it.L, qt * kTile + kTile) : it.L, kTile); };
    first0 = first(it.qt0);
    end0 = end(it.qt0);
    end1 = end(it.qt1);
    first1 = it.qt1 < 0 ? first0 : first(it.qt1);
    lo = min(first0, first1);
    nk = min(keep_tiles, lo);
    n = nk + max(end0, end1) - lo;
  }
  RB_DEVICE int tile(int k) const { return k < nk ? k : lo + k - nk; }
  RB_DEVICE bool takes(int t, int j) const { return j < (t ? end1 : end0) && (j >= (t ? first1 : first0) || j < keep_tiles); }
};

template <int kD, int kDV, typename T, int kFmt, int kMode>
__global__ void __launch_bounds__(kFwdThreads, 1) attn_fwd_kernel(const __grid_constant__ CUtensorMap tma_q, const __grid_constant__ CUtensorMap tma_k,
                                                                  const __grid_constant__ CUtensorMap tma_v, const __grid_constant__ AttnParams p) {
  using C = FCfg<kD, kDV>;
  extern __shared__ __align__(1024) uint8_t smem[];      // (addresses are constants then, not registers)
  const uint32_t sQ = ptx::smem_u32(smem), sKV = sQ + C::kKV;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kBars);
  Item* items = reinterpret_cast<Item*>(smem + C::kBars + 288);                // two slots of 24 bytes
  const uint32_t clc = sQ + C::kBars + 288 + 64;                               // 16 bytes
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(smem + C::kBars + 288 + 80);
  static_assert(F_NUM_BARS * 8 <= 288, "barriers");
  volatile uint32_t* dead = tmem_ptr + 1;
  auto bar = [&](int i) { return ptx::smem_u32(&bars[i]); };
  auto wait = [&](int i, uint32_t parity) { bounded_wait(bar(i), parity, dead); };
  if ((sQ & 1023u) != 0u) {                                // (the swizzle wants it; never seen)
    if (threadIdx.x == 0) *reinterpret_cast<volatile int*>(p.status) = rb::kStatusUnaligned;
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* row_alpha = reinterpret_cast<float*>(smem + C::kRows);      // [tile][row]: factor on the row's O, written with every key tile behind the first
  float* row_l = row_alpha + 2 * kTile;                              // [tile][row]: denominator and maximum, written behind the last one
  float* row_m = row_l + 2 * kTile;

  if (warp == 9 && lane == 0) {
    *dead = 0;
    ptx::prefetch_tensormap(&tma_q);
    ptx::prefetch_tensormap(&tma_k);
    ptx::prefetch_tensormap(&tma_v);
    for (int i = 0; i < F_NUM_BARS; ++i) {
      // P_FULL: the four softmax warps of the tile and the four output warps
      ptx::mbar_init(bar(i), i >= P_FULL && i < P_FULL + 2 ? 8 : i >= L_FULL && i < L_EMPTY + 2 ? 4 : i >= IT_EMPTY && i < IT_EMPTY + 2 ? kItemReaders : 1);
    }
    ptx::fence_barrier_init();
  }
  if (warp == 8) {
    ptx::tmem_alloc(ptx::smem_u32(tmem_ptr), 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;

  if (warp >= 8 && warp < 12) {
    ptx::reg_dec<kOtherRegs>();
    if (warp == 9) {
      // ===================================================== scheduler + TMA producer
      auto request = [&] {
        if (lane == 0) {
          ptx::mbar_arrive_expect_tx(bar(CLC_FULL), 16);
          ptx::clc_try_cancel(clc, bar(CLC_FULL));
        }
        __syncwarp();
      };
      UnitSearch search;
      auto find = [&](int idx, Item& it) {
        const int unit = idx / p.n_head_units, hu = idx - unit * p.n_head_units;
        int r;                       // r-th unit of the sequence, longest first
        if (!search.find(p.cu_seqlens, p.B, p.pair_heads ? kTile : 2 * kTile, unit, it.tok0, it.L, r)) return false;
        const int last = RB_CEIL_DIV(it.L, kTile) - 1;
        it.head0 = p.pair_heads ? 2 * hu : hu;
        it.head1 = p.pair_heads ? 2 * hu + 1 : hu;
        it.qt0 = p.pair_heads ? last - r : last - 2 * r;
        it.qt1 = p.pair_heads ? last - r : last - 2 * r - 1;
        return true;
      };

      int idx = blockIdx.x, n_pub = 0;
      uint32_t kvc = 0, qc0 = 0, qc1 = 0, n_req = 0;
      request();
      auto publish = [&](const Item& it) {
        const int slot = n_pub & 1;
        wait(IT_EMPTY + slot, ((uint32_t)(n_pub >> 1) & 1u) ^ 1u);
        if (lane == 0) {
          items[slot] = it;
          ptx::mbar_arrive(bar(IT_FULL + slot));
        }
        ++n_pub;
      };
      while (true) {
        Item it{0, 0, 0, 0, 0, 0};
        if (find(idx, it)) {
          publish(it);
          if (lane == 0) {
            const Walk w(it, p);
            const int hk = it.head0 / (p.nq / p.nkv);
            auto load_q = [&](int t, int head, int qt, uint32_t& count) {
              if (qt < 0) return;
              wait(Q_EMPTY + t, (count & 1u) ^ 1u);
              ++count;
              ptx::mbar_arrive_expect_tx(bar(Q_FULL + t), C::kQBytes);
#pragma unroll
              for (int kb = 0; kb < kD / 64; ++kb)
                ptx::tma_load_2d(sQ + t * C::kQBytes + kb * (kTile * 128), &tma_q, bar(Q_FULL + t), head * kD + kb * 64, it.tok0 + qt * kTile);
            };
            auto load_kv = [&](bool is_v, int j) {
              const int st = kvc & (kStages - 1);
              wait(KV_EMPTY + st, ((kvc / kStages) & 1u) ^ 1u);
              ++kvc;
              ptx::mbar_arrive_expect_tx(bar(KV_FULL + st), is_v ? C::kVBytes : C::kKBytes);
              const int col = is_v ? (hk / p.vshare) * kDV : hk * kD, blocks = is_v ? kDV / 64 : kD / 64;
              for (int kb = 0; kb < blocks; ++kb)
                ptx::tma_load_2d(sKV + st * C::kStageBytes + kb * (kTile * 128), is_v ? &tma_v : &tma_k, bar(KV_FULL + st), col + kb * 64,
                                 it.tok0 + j * kTile);
            };
            load_q(0, it.head0, it.qt0, qc0);
            load_kv(false, w.tile(0));
            load_q(1, it.head1, it.qt1, qc1);
            load_kv(true, w.tile(0));
            for (int k = 1; k < w.n; ++k) {
              load_kv(false, w.tile(k));
              load_kv(true, w.tile(k));
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
      publish(Item{0, -1, 0, 0, -1, -1});
    } else if (warp == 8) {
      // ===================================================== MMA issuer: the whole warp runs the loop, one elected lane issues.  A wait costs the warp 100 to 200 cycles
      // even when there is nothing to wait for, and the pipe holds only some 256 cycles of products: what the tiles' barriers say is asked for ahead of the
      // products in front of them.
      constexpr uint32_t idesc_s = ptx::make_idesc_f16(kFmt, kTile, kTile, 0, 0);   // Q, K both K-major (head-dim contiguous)
      constexpr uint32_t idesc_o = ptx::make_idesc_f16(kFmt, kTile, kDV, 0, 1);     // P (TMEM), V MN-major
      constexpr uint32_t kToMN = (uint32_t)((kTile * 128 - 16) >> 4) << 16;         // from the K-major form of a tile to its MN-major one
      const uint32_t tm = (uint32_t)ptx::uniform((int)tmem_base), el = ptx::elect_one() ? 1u : 0u;
      const uint32_t q_lo = ptx::desc_lo(sQ, 16), kv_lo = ptx::desc_lo(sKV, 16);
      uint32_t kvc = 0, qc[2] = {0, 0}, pc[2] = {0, 0};
      for (int n_it = 0;; ++n_it) {
        const int slot = n_it & 1;
        wait(IT_FULL + slot, (uint32_t)(n_it >> 1) & 1u);
        Item it = items[slot];
        it.L = ptx::uniform(it.L);
        it.qt0 = ptx::uniform(it.qt0);
        it.qt1 = ptx::uniform(it.qt1);
        if (lane == 0) ptx::mbar_arrive(bar(IT_EMPTY + slot));
        __syncwarp();
        if (it.L < 0 || ptx::uniform((int)*dead)) break;
        const Walk w(it, p);
        bool s_open[2] = {false, false}, o_open[2] = {false, false};
        auto last_tile = [&](int t) { return (t ? w.end1 : w.end0) - 1; };
        auto issue_s = [&](int t, int j, uint32_t st) {
          if (!s_open[t]) { wait(Q_FULL + t, qc[t] & 1u); ++qc[t]; s_open[t] = true; }
          ptx::tc_fence_after();
          const uint32_t a = q_lo + t * (C::kQBytes >> 4), b = kv_lo + st * (C::kStageBytes >> 4);
#pragma unroll
          for (int kk = 0; kk < kD / 16; ++kk) {
            const uint32_t off = ((kk >> 2) * (kTile * 128) + (kk & 3) * 32) >> 4;
            ptx::tc_mma_f16_if(el, tm + t * 128, a + off, b + off, idesc_s, kk != 0 ? 1u : 0u);
          }
          ptx::tc_commit_if(el, bar(S_FULL + t));
          if (j == last_tile(t)) ptx::tc_commit_if(el, bar(Q_EMPTY + t));
        };
        auto issue_pv = [&](int t, int j, uint32_t st) {
          wait(P_FULL + t, pc[t] & 1u);
          ++pc[t];
          ptx::tc_fence_after();
          const uint32_t b = kv_lo + kToMN + st * (C::kStageBytes >> 4), keep = o_open[t] ? 1u : 0u;
#pragma unroll
          for (int kk = 0; kk < kTile / 16; ++kk)      // A: 16 keys = 8 TMEM columns; B: 16 key rows = 2048 B down every 64-wide chunk of DV
            ptx::tc_mma_f16_ts_if(el, tm + 256 + t * 128, tm + t * 128 + kk * 8, b + kk * 128, idesc_o, kk != 0 ? 1u : keep);
          if (j == last_tile(t)) ptx::tc_commit_if(el, bar(O_FULL + t));
          o_open[t] = true;
        };
        auto peek_kv = [&](uint32_t c) { return ptx::mbar_try_wait(bar(KV_FULL + (c & (kStages - 1))), (c / kStages) & 1u); };
        auto pass_kv = [&](uint32_t c, bool ready) {
          if (!ready) wait(KV_FULL + (c & (kStages - 1)), (c / kStages) & 1u);
          return c & (kStages - 1);
        };
        auto free_kv = [&](uint32_t st) { ptx::tc_commit_if(el, bar(KV_EMPTY + st)); };
        uint32_t st = pass_kv(kvc, false);
#pragma unroll
        for (int t = 0; t < 2; ++t)
          if (w.takes(t, w.tile(0))) issue_s(t, w.tile(0), st);
        free_kv(st);
        for (int k = 0; k < w.n; ++k) {
          const int j = w.tile(k), jn = w.tile(k + 1);
          const bool more = k + 1 < w.n;
          const uint32_t sv = pass_kv(kvc + 2 * k + 1, peek_kv(kvc + 2 * k + 1));
          const bool k_ready = more && peek_kv(kvc + 2 * k + 2);
          uint32_t sk = kStages;
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (w.takes(t, j)) issue_pv(t, j, sv);
            if (more) {
              if (sk == kStages) sk = pass_kv(kvc + 2 * k + 2, k_ready);
              if (w.takes(t, jn)) issue_s(t, jn, sk);
            }
            if (t == 1) free_kv(sv);
          }
          if (more) free_kv(sk);
        }
        kvc += 2 * w.n;
      }
      __syncwarp();
    }
  } else if (warp < 8) {
    ptx::reg_inc<kSoftmaxRegs>();
    // ===================================================== softmax (4 warps per tile; thread = query row = TMEM lane)
    const int t = warp >> 2, quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
    const uint32_t tS = lane_addr + t * 128;
    auto arrive = [&](int i) {
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(bar(i));
    };
    const float cap_c = kMode == kCap ? 2.f * 1.4426950408889634f * p.scale / p.softcap : 0.f, cap_k = kMode == kCap ? p.softcap * 1.4426950408889634f : 0.f;
    const int win = (p.causal && p.window > 0) ? p.window : 0;
    const bool bounded = win > 0 || p.chunk > 0;
    uint32_t sc = 0, n_l = 0;     // S tiles of this tile / items so far
    for (int n_it = 0;; ++n_it) {
      const int slot = n_it & 1;
      wait(IT_FULL + slot, (uint32_t)(n_it >> 1) & 1u);
      const Item it = items[slot];
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(bar(IT_EMPTY + slot));
      if (it.L < 0 || *dead) break;
      const int qt = t ? it.qt1 : it.qt0;
      if (qt < 0) continue;
      const int L = it.L, q0 = qt * kTile, q_pos = q0 + row;
      [[maybe_unused]] const int head = t ? it.head1 : it.head0;
      // scores live in the log2 domain: weight = exp2(s * c2 [+ distance term] - m_run)
      float c2 = p.scale * 1.4426950408889634f, slope2 = 0.f, m_run = -INFINITY, l_run = 0.f;
      if constexpr (kMode != kPlain) {
        if (p.temp) c2 *= rb::to_f(reinterpret_cast<const T*>(p.temp)[head]);
        if (kMode == kGeneral && p.slope_base >= 0.f) slope2 = exp2f(-p.slope_base * (float)(head + 1) / (float)p.nq) * 1.4426950408889634f;
        if (p.sink) { m_run = rb::to_f(reinterpret_cast<const T*>(p.sink)[head]) * 1.4426950408889634f; l_run = 1.f; }
      }
      // first visible key of the row (used where masks are formed; chunks: formed there again would be a division)
      const int row_lo = p.chunk > 0 ? q_pos / p.chunk * p.chunk : win > 0 ? q_pos - win + 1 : 0;
      const int last_lo = p.chunk > 0 ? (q0 + kTile - 1) / p.chunk * p.chunk : q0 + kTile - win;                  // of the tile's last row
      // this tile's key tiles, in the order of the item's walk
      const int first_tile = p.chunk > 0 ? (q0 / p.chunk * p.chunk) / kTile : win > 0 ? max(0, q0 - win + 1) / kTile : 0;
      const int n_keep = win > 0 ? min(RB_CEIL_DIV(p.keep, kTile), first_tile) : 0;
      const int n_tiles = n_keep + RB_CEIL_DIV(p.causal ? min(L, q0 + kTile) : L, kTile) - first_tile;

      for (int k = 0; k < n_tiles; ++k) {
        const int kv0 = (k < n_keep ? k : first_tile + k - n_keep) * kTile;
        wait(S_FULL + t, sc & 1u);
        ++sc;
        ptx::tc_fence_after();
        uint32_t r[128];
#pragma unroll
        for (int c = 0; c < 4; ++c) ptx::tc_ld_32x32(tS + c * 32, r + c * 32);
        ptx::tc_wait_ld();
        float s[128];
#pragma unroll
        for (int i = 0; i < 128; ++i) s[i] = __uint_as_float(r[i]);
        if constexpr (kMode == kGeneral) {
          const float base = slope2 * (float)(kv0 - q_pos);
#pragma unroll
          for (int i = 0; i < 128; i += 2) {
            float b0 = (float)i, b1 = (float)(i + 1);
            fma_pair(b0, b1, slope2, base);
            fma_pair2(s[i], s[i + 1], c2, b0, b1);
          }
        }
        if constexpr (kMode == kCap) {
#pragma unroll
          for (int i = 0; i < 128; ++i) s[i] = soft_cap2(s[i], cap_c, cap_k, cap_k);
        }
        // only the last tile of the sequence, the diagonal tile and the tiles the window's lower edge crosses need per-element masks
        if ((kv0 + kTile > L) || (p.causal && kv0 + kTile - 1 > q0) || (bounded && last_lo > kv0)) {
          const int lim = (p.causal ? min(L, q_pos + 1) : L) - kv0;   // local key columns [lo, lim) are visible to this row
          const int lo = bounded ? row_lo - kv0 : 0;
          const int kept = kMode == kGeneral ? p.keep - kv0 : 0;      // columns below `kept` stay visible under `lo`
#pragma unroll
          for (int c = 0; c < 4; ++c) {                               // bit i: column 32 c + i is visible
            auto below = [&](int n) { n -= 32 * c; return n <= 0 ? 0u : n >= 32 ? 0xffffffffu : (1u << n) - 1u; };
            const uint32_t vis = below(lim) & (~below(lo) | below(kept));
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if ((vis & (1u << i)) == 0u) s[32 * c + i] = -INFINITY;
          }
        }
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 128; i += 8)
#pragma unroll
          for (int e = 0; e < 4; ++e) mx4[e] = max3(mx4[e], s[i + 2 * e], s[i + 2 * e + 1]);
        float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
        if (kMode != kGeneral && kMode != kCap && mx != -INFINITY) mx *= c2;
        const float m_new = fmaxf(m_run, mx);
        const float alpha = m_new == m_run ? 1.f : exp2f(m_run - m_new);
        l_run = __fmul_rn(l_run, alpha);              // (rounded by itself: contracted with the sum below, the statistics' last bits would depend on the compiler)
        m_run = m_new;
        if (k > 0) {                                  // the output warps scale the row while its weights are formed
          row_alpha[t * kTile + row] = alpha;
          arrive(A_FULL + t * 4 + quad);
        }
        const float neg_m = m_run == -INFINITY ? 0.f : -m_run;      // fully masked so far: keep exp2 arguments finite
        float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 4; ++c) {                 // 32 keys at a time: 16 columns of weights (registers: stored 32 at a time the scores spill)
          uint32_t pw[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float e0 = s[32 * c + i], e1 = s[32 * c + i + 1];
            if constexpr (kMode == kGeneral || kMode == kCap) add_pair(e0, e1, neg_m, neg_m);
            else fma_pair(e0, e1, c2, neg_m);
            e0 = exp2f(e0);
            e1 = exp2f(e1);
            add_pair(sum4[i & 2], sum4[(i & 2) + 1], e0, e1);
            pw[i >> 1] = pack2<T>(e0, e1);
          }
          ptx::tc_st_32x16(tS + 16 * c, pw);
        }
        l_run += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
        ptx::tc_wait_st();
        ptx::tc_fence_before();
        arrive(P_FULL + t);
      }
      wait(L_EMPTY + t, (n_l & 1u) ^ 1u);            // (items of one key tile: the output warps may be two behind)
      ++n_l;
      row_l[t * kTile + row] = l_run;
      row_m[t * kTile + row] = m_run;
      arrive(L_FULL + t);
    }
  } else {
    ptx::reg_dec<kOutRegs>();
    // ===================================================== output (warp = TMEM quadrant, thread = row of both tiles): O of a tile is scaled where a row's maximum has grown (its
    // product in front of the scores that showed it has retired, and the next one waits for these warps too), and leaves when its last product has
    const int quad = warp & 3, row = quad * 32 + lane;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quad * 32) << 16);
    const uint32_t stage = sQ + C::kOut + quad * 4096;
    uint32_t a_par = 0, o_par = 0;                    // parities of A_FULL / O_FULL, a bit a tile
    if (lane == 0) {                                  // O is free for a first product: said again when it has been read out
      ptx::mbar_arrive(bar(P_FULL));
      ptx::mbar_arrive(bar(P_FULL + 1));
    }
    for (int n_it = 0;; ++n_it) {
      const int slot = n_it & 1;
      wait(IT_FULL + slot, (uint32_t)(n_it >> 1) & 1u);
      const Item it = items[slot];
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(bar(IT_EMPTY + slot));
      if (it.L < 0 || *dead) break;
      {
        const Walk w(it, p);
        uint32_t open = 0;
#pragma unroll 1
        for (int k = 0; k < w.n; ++k) {
          const int j = w.tile(k);
#pragma unroll 1
          for (int t = 0; t < 2; ++t) {
            if (!w.takes(t, j)) continue;
            if ((open >> t & 1u) == 0u) {
              open |= 1u << t;
            } else {
              wait(A_FULL + t * 4 + quad, a_par >> t & 1u);
              a_par ^= 1u << t;
              ptx::tc_fence_after();
              const float alpha = row_alpha[t * kTile + row];
              if (__any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll 1
                for (uint32_t tO = lane_addr + 256 + t * 128, end = tO + kDV; tO != end; tO += 32) {
                  uint32_t o[32];
                  ptx::tc_ld_32x32(tO, o);
                  ptx::tc_wait_ld();
#pragma unroll
                  for (int i = 0; i < 32; i += 2) {
                    float x0 = __uint_as_float(o[i]), x1 = __uint_as_float(o[i + 1]);
                    mul_pair(x0, x1, alpha, alpha);
                    o[i] = __float_as_uint(x0);
                    o[i + 1] = __float_as_uint(x1);
                  }
                  ptx::tc_st_32x32(tO, o);
                }
                ptx::tc_wait_st();
                ptx::tc_fence_before();
              }
              __syncwarp();
              if (lane == 0) ptx::mbar_arrive(bar(P_FULL + t));
            }
          }
        }
      }
      // ---- O / l (times the gate), 64 columns at a time through the warp's staging rows
#pragma unroll 1
      for (int t = 0; t < 2; ++t) {
        const int qt = t ? it.qt1 : it.qt0, head = t ? it.head1 : it.head0;
        if (qt < 0) continue;
        const int q_pos = qt * kTile + row;
        float inv = 1.f;
        if constexpr (kMode != kPlain) {
          if (p.gate && p.gate_mode == 1 && q_pos < it.L)
            inv = 1.f / (1.f + __expf(-rb::to_f(reinterpret_cast<const T*>(p.gate)[(int64_t)(it.tok0 + q_pos) * p.gate_ld + head])));
        }
        wait(L_FULL + t, o_par >> t & 1u);
        const float l_run = row_l[t * kTile + row];
        inv *= 1.f / l_run;
        if constexpr (kMode == kPlain) {
          // (the larger product rounded by itself, spelled out: the statistics do not depend on what the compiler contracts)
          if (q_pos < it.L)
            p.lse[(int64_t)head * p.T + it.tok0 + q_pos] = __fmaf_rn(__log2f(l_run), 0.6931471805599453f, __fmul_rn(row_m[t * kTile + row], 0.6931471805599453f));
        }
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(bar(L_EMPTY + t));
        wait(O_FULL + t, o_par >> t & 1u);
        o_par ^= 1u << t;
        ptx::tc_fence_after();
#pragma unroll 1
        for (int half = 0; half < kDV / 64; ++half) {
#pragma unroll 1
          for (int c2 = 0; c2 < 2; ++c2) {
            uint32_t o[32];
            ptx::tc_ld_32x32(lane_addr + 256 + t * 128 + half * 64 + c2 * 32, o);
            ptx::tc_wait_ld();
            if constexpr (kMode != kPlain) {
              if (p.gate && p.gate_mode == 2 && q_pos < it.L) {          // (rows of the gate are 16-byte aligned: checked by the host)
                const T* gr = reinterpret_cast<const T*>(p.gate) + (int64_t)(it.tok0 + q_pos) * p.gate_ld + (int64_t)head * kDV + half * 64 + c2 * 32;
#pragma unroll
                for (int i = 0; i < 32; i += 8) {
                  asm volatile("" ::: "memory");                      // one load after the other: registers
                  const rb::Pack<T, 8> gv = *reinterpret_cast<const rb::Pack<T, 8>*>(gr + i);
#pragma unroll
                  for (int e = 0; e < 8; ++e)
                    o[i + e] = __float_as_uint(__uint_as_float(o[i + e]) * __fdividef(1.f, 1.f + __expf(-rb::to_f(gv.v[e]))));
                }
              }
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              uint32_t v[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) v[e] = pack2<T>(__uint_as_float(o[8 * c + 2 * e]) * inv, __uint_as_float(o[8 * c + 2 * e + 1]) * inv);
              st_shared_v4(stage + lane * 128 + (((c2 * 4 + c) ^ (lane & 7)) << 4), v[0], v[1], v[2], v[3]);
            }
          }
          ptx::tc_fence_before();
          __syncwarp();
          if (half == kDV / 64 - 1 && lane == 0) ptx::mbar_arrive(bar(P_FULL + t));
          T* dst = reinterpret_cast<T*>(p.out) + (int64_t)head * kDV + half * 64 + (lane & 7) * 8;
#pragma unroll 4
          for (int i = 0; i < 8; ++i) {
            const int rr = i * 4 + (lane >> 3), pos = qt * kTile + quad * 32 + rr;
            const uint4 v = ld_shared_v4(stage + rr * 128 + (((lane & 7) ^ (rr & 7)) << 4));
            if (pos < it.L) *reinterpret_cast<uint4*>(dst + (int64_t)(it.tok0 + pos) * p.out_ld) = v;
          }
          __syncwarp();
        }
      }
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  rb::report_given_up(dead, p.status);
  if (warp == 8) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, 512);
  }
}

template <int kD, int kDV, typename T, int kFmt, int kMode>
int launch_attn_fwd(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, AttnParams p, int B, cudaStream_t s) {
  using C = FCfg<kD, kDV>;
  static_assert(C::kSmemBytes <= kMaxSmem, "shared memory");
  auto kern = attn_fwd_kernel<kD, kDV, T, kFmt, kMode>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes) != cudaSuccess) return -30;
    attr_set = true;
  }
  p.B = B;
  if ((p.status = rb_attn_status()) == nullptr) return -34;
  p.pair_heads = (p.nq / p.nkv) % 2 == 0;
  p.n_head_units = p.pair_heads ? p.nq / 2 : p.nq;
  // the sequences' lengths are on the device: sum of ceil(L / rows) is at most (T + (rows - 1) B) / rows
  const int64_t rows = p.pair_heads ? kTile : 2 * kTile;
  const int64_t n = (p.T + (rows - 1) * B) / rows * p.n_head_units;
  if (n <= 0 || n > 0x7fffffff) return -33;
  kern<<<dim3((unsigned)n), kFwdThreads, C::kSmemBytes, s>>>(mq, mk, mv, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -31;
}

}  // namespace

extern "C" int rb_attn_fwd_bias(const CUtensorMap* mq, const CUtensorMap* mk, const CUtensorMap* mv, const AttnParams* p, int B, int hd, int max_seqlen,
                                int kv_shared, int bf, cudaStream_t s);

extern "C" int* rb_attn_status() {
  static int* const word = [] {
    int* w = nullptr;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;      // the first call may come while a graph is being captured
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (cudaHostAlloc(reinterpret_cast<void**>(&w), sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) w = nullptr;
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (w != nullptr) *w = 0;
    return w;
  }();
  return word;
}

// The status word since the last call: not 0 if a kernel left outputs unwritten (synchronises, and clears the word)
extern "C" int rb_attn_wait_error() {
  volatile int* w = rb_attn_status();
  if (w == nullptr || cudaDeviceSynchronize() != cudaSuccess) return -1;
  const int v = *w;
  *w = 0;
  return v;
}

// q / k / v: [T, heads, hd] views (unit stride over hd, `heads * hd` contiguous columns, row pitch *_ld elements) -- e.g. the
// three column ranges of the fused QKV projection.  out [T, nq, hd] with row pitch out_ld, lse [nq, T] fp32.
// dt: 1 = bf16, 2 = fp16.  Returns 0 or a negative code (unsupported shape / descriptor failure).
// window > 0 (causal only): sliding-window attention.
extern "C" int rb_attn_fwd_window(const void* q, const void* k, const void* v, void* out, float* lse, const int* cu_seqlens,
                                  int64_t q_ld, int64_t k_ld, int64_t v_ld, int64_t out_ld, int T, int B, int nq, int nkv, int hd,
                                  int max_seqlen, float scale, int causal, int window, int dt, cudaStream_t s) {
  if (hd != 128 && hd != 64) return -1;
  if (dt != 1 && dt != 2) return -2;
  if (nq % nkv != 0 || T <= 0 || B <= 0 || max_seqlen <= 0) return -3;
  if ((q_ld | k_ld | v_ld | out_ld) % 8 != 0) return -4;
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)out) & 15) return -5;
  CUtensorMap mq, mk, mv;
  const int bf = dt == 1;
  if (!make_tmap(&mq, q, bf, T, (uint64_t)nq * hd, q_ld, 64, kTile)) return -10;
  if (!make_tmap(&mk, k, bf, T, (uint64_t)nkv * hd, k_ld, 64, kTile)) return -11;
  if (!make_tmap(&mv, v, bf, T, (uint64_t)nkv * hd, v_ld, 64, kTile)) return -12;
  if (window > 0 && !causal) return -6;
  AttnParams p{cu_seqlens, out, lse, out_ld, T, nq, nkv, scale, causal, window, 0, nullptr, nullptr, nullptr, 0, -1.f};
  if (hd == 128) {
    return bf ? launch_attn_fwd<128, 128, __nv_bfloat16, 1, kPlain>(mq, mk, mv, p, B, s) : launch_attn_fwd<128, 128, __half, 0, kPlain>(mq, mk, mv, p, B, s);
  }
  return bf ? launch_attn_fwd<64, 64, __nv_bfloat16, 1, kPlain>(mq, mk, mv, p, B, s) : launch_attn_fwd<64, 64, __half, 0, kPlain>(mq, mk, mv, p, B, s);
}

extern "C" int rb_attn_fwd(const void* q, const void* k, const void* v, void* out, float* lse, const int* cu_seqlens,
                           int64_t q_ld, int64_t k_ld, int64_t v_ld, int64_t out_ld, int T, int B, int nq, int nkv, int hd,
                           int max_seqlen, float scale, int causal, int dt, cudaStream_t s) {
  return rb_attn_fwd_window(q, k, v, out, lse, cu_seqlens, q_ld, k_ld, v_ld, out_ld, T, B, nq, nkv, hd, max_seqlen, scale, causal, 0, dt, s);
}

// Window attention with a sink on the tensor cores (see the modes at the top): q / k [T, heads, hd], v [T, heads, vd] as for
// rb_attn_fwd (head sizes of 64 or 128), temp / sink [nq] in the operand type or null, gate logits at gate[t * gate_ld + h] (gate_mode
// 1) or gate[t * gate_ld + h * vd + c] (gate_mode 2) or null, window <= 0 = every earlier key, keep = first keys that stay visible,
// chunk > 0 = chunked instead of windowed, softcap > 0 = capped scores (kSimple cases only), slope_base < 0 = no distance term, bias
// [nq, n_bias] fp32 or null.  kv_shared: the values are the keys (v is not read).  hd != vd takes the kSimple cases; returns a negative
// code for what it does not take.
extern "C" int rb_attn_fwd_sink(const void* q, const void* k, const void* v, void* out, const int* cu_seqlens, int64_t q_ld, int64_t k_ld,
                                int64_t v_ld, int64_t out_ld, int T, int B, int nq, int nkv, int hd, int vd, int max_seqlen, float scale, int window,
                                int keep, const void* temp, const void* sink, const void* gate, int64_t gate_ld, int gate_mode, int chunk,
                                float softcap, float slope_base, const float* bias, int n_bias, int kv_shared, int dt, int vshare, cudaStream_t s) {
  if ((hd != 128 && hd != 64) || (vd != 128 && vd != 64)) return -1;
  if (dt != 1 && dt != 2) return -2;
  if (nq % nkv != 0 || T <= 0 || B <= 0 || max_seqlen <= 0 || vshare < 1 || nkv % vshare) return -3;
  if (kv_shared) { v = k; v_ld = k_ld; if (hd != vd || vshare != 1) return -3; }
  if ((q_ld | k_ld | v_ld | out_ld) % 8 != 0) return -4;
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)out) & 15) return -5;
  if (gate != nullptr && gate_mode == 2 && (gate_ld % 8 != 0 || ((uintptr_t)gate & 15))) return -6;
  const bool plain_mask = slope_base < 0.f && (window <= 0 || keep == 0);
  const bool simple = plain_mask && temp == nullptr && scale > 0.f && bias == nullptr;
  if (softcap > 0.f && !simple) return -7;
  if (chunk > 0 && window > 0) return -8;
  if (bias != nullptr && (!plain_mask || n_bias < 1 || hd != vd)) return -9;
  if (hd != vd && (!simple || softcap > 0.f)) return -9;
  CUtensorMap mq, mk, mv;
  const int bf = dt == 1;
  if (!make_tmap(&mq, q, bf, T, (uint64_t)nq * hd, q_ld, 64, kTile)) return -10;
  if (!make_tmap(&mk, k, bf, T, (uint64_t)nkv * hd, k_ld, 64, kTile)) return -11;
  if (!make_tmap(&mv, v, bf, T, (uint64_t)(nkv / vshare) * vd, v_ld, 64, bias != nullptr ? 64 : kTile)) return -12;
  AttnParams p{cu_seqlens, out, nullptr, out_ld, T, nq, nkv, scale, 1, window > 0 ? window : 0, window > 0 ? keep : 0, temp, sink, gate, gate_ld,
               slope_base, vshare, gate_mode, chunk, softcap, bias, window > 0 && n_bias > window ? window : n_bias, n_bias};
  if (bias != nullptr) return rb_attn_fwd_bias(&mq, &mk, &mv, &p, B, hd, max_seqlen, kv_shared, bf, s);
#define RB_GO2(HD, VD, M)                                                                   \
  return bf ? launch_attn_fwd<HD, VD, __nv_bfloat16, 1, M>(mq, mk, mv, p, B, s)            \
            : launch_attn_fwd<HD, VD, __half, 0, M>(mq, mk, mv, p, B, s)
#define RB_GO(M)                           \
  if (hd == 128) { RB_GO2(128, 128, M); } \
  RB_GO2(64, 64, M)
  if (hd != vd) {
    if (hd == 128) { RB_GO2(128, 64, kSimple); }
    RB_GO2(64, 128, kSimple);
  }
  if (softcap > 0.f) { RB_GO(kCap); }
  if (simple) { RB_GO(kSimple); }
  RB_GO(kGeneral);
#undef RB_GO
#undef RB_GO2
}
