// Fused sampling step for generation: temperature, min-length EOS suppression, top-k, top-p, categorical sample,
// log-prob of the sample, and the bit-packed "filtered" mask — one CTA per sequence, one pass over global memory.
//
// Replaces the eager chain of the reference's `genstep` (fp32 cast, topk, sort, softmax, cumsum, scatter,
// Categorical, gather, mask compare: nn/real_llm_generate.py:26-141, utils/logits_warper.py) — about 1 ms per decode
// step at [128, 32000].  The row is staged once in shared memory as fp32 (V * 4 bytes <= 200 KB).
//
// Nothing here is bound by bytes (8 MB at [128, 32000]): a row's time is the chain of block-wide steps, and a barrier of 1024 threads costs as much
// as 100 .. 200 instructions.  A radix descent over the whole row (4 digits each for top-k and top-p) spends it on shared atomics that pile up on the
// few bins logits fall in: 89 us at [128, 32000], top-k 50, top-p 0.9.  For top_k <= 512 the row is therefore cut down first: the k-th largest of the
// per-thread maxima (of groups of threads where k is small) is a lower bound of the k-th largest logit, as that many elements are at least as large,
// and only k .. 2 k elements reach it.  The threads that hold them append them in any order; one warp finds the exact k-th largest among them bit by
// bit, over the bits in which they differ; a bitmap of the row brings the kept ones back into index order (and is the complement of the mask that is
// returned).  Then the top-p threshold from every kept element summing the mass of the strictly larger ones, and the draw by one warp.
// Counting with block barriers, one a bit, this took 96 of them and 27 us; with one warp in registers it takes 11.7.
// A larger top_k, and a row with more than 1536 candidates or 1024 kept elements (ties), takes the radix descent:
//   * top-k threshold = k-th largest key by a 4 x 8-bit descent over a shared histogram;
//   * top-p threshold = the same descent with probability mass instead of counts (keep x iff the mass of strictly
//     larger logits is < top_p * total).
// The sample is drawn by inverse CDF in index order over the kept set (counter-based RNG).  Ties at a threshold are all kept (same
// rule as `logits < kth` in the PyTorch reference).
#include "common.cuh"

#include <type_traits>

namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kFastTopK = 512;      // the thread maxima bound the k-th logit tightly only while k is well below their number
constexpr int kMaxCand = 1536, kMaxKept = kThreads;   // with 51200 staged logits the block's shared memory is nearly full
constexpr int kMaxV = 51200;

RB_DEVICE uint32_t f2key(float x) {  // order-preserving float -> uint
  const uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
RB_DEVICE uint32_t mix32(uint32_t x) {
  x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
  return x;
}

struct SampleParams {
  const void* logits;
  int64_t row_stride;
  int64_t* next_tok;
  float* logprob;
  uint8_t* mask_bits;
  int64_t mask_stride;
  const bool* unfinished;   // [B] or nullptr: finished rows emit pad / logprob 0
  int V, top_k, eos_id, suppress_eos, greedy, pad_id;
  float inv_temp, top_p;
  uint64_t seed;
  uint32_t step;
  // ---- in-graph mode (step_rows != nullptr): the kernel is the tail of the captured decode step.  The step index lives on the
  // device (one counter per row, advanced here), outputs go to column `step` of [B, n_gen] history buffers, and the kernel
  // also feeds the next replay: next token -> input_ids, cache_lens += 1, unfinished &= (token != eos).
  int* step_rows;
  int64_t* input_ids;
  int* cache_lens;
  bool* unfinished_rw;
  int n_gen, min_new_tokens;
  bool* unfinished_out = nullptr;   // eager mode: unfinished and not eos
  const int64_t* seed_ptr;   // device-resident seed (a replayed graph must not repeat the random stream of the previous call)
};

struct SampleShared {
  float red[32];
  uint32_t redu[32];
  uint32_t u[4];
  float f[4];
  union {
    struct { uint32_t hist[256]; float histm[256]; };                     // radix descent
    uint32_t top[kThreads];                                               // the threads' largest keys
    struct { uint32_t cand[kMaxCand]; uint16_t cand_idx[kMaxCand]; };     // candidates in any order: key and index
  };
  uint32_t kept[kMaxKept];        // elements of the top-k set in index order: key, index, exp(value - max)
  float kept_e[kMaxKept];
  uint16_t kept_idx[kMaxKept];
  uint32_t bitmap[kMaxV / 32];    // a bit an element: kept
};
static_assert(sizeof(SampleShared) + kMaxV * 4 <= 227 * 1024, "shared memory");

// Inclusive prefix over the block of `v`, and the block's total; `red` holds one entry per warp.  Two barriers.
template <typename V> RB_DEVICE V block_inclusive(V v, V* red, V& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  V incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const V x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  __syncthreads();               // protect `red` from a previous use
  if (lane == 31) red[warp] = incl;
  __syncthreads();
  V w = red[lane];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const V x = __shfl_up_sync(0xffffffffu, w, o);
    if (lane >= o) w += x;
  }
  total = __shfl_sync(0xffffffffu, w, 31);
  const V base = __shfl_sync(0xffffffffu, w, warp == 0 ? 0 : warp - 1);
  return (warp == 0 ? V(0) : base) + incl;
}

// The k-th largest of the warp's keys, kPer of them a lane (a lane without one passes 0), or 0 if there are fewer than k: no bound, and every element
// is a candidate.  Bit by bit from the top over the bits in which the keys differ (sign and most of the exponent are common to what competes, and 16-bit
// logits have 16 bits that are not), at most `most` of them: with fewer bits than that left undecided, a lower bound.
template <int kPer> RB_DEVICE uint32_t kth_largest(const uint32_t (&key)[kPer], int k, int most) {
  uint32_t any = 0, all = 0xffffffffu;
  int have = 0;
#pragma unroll
  for (int i = 0; i < kPer; ++i)
    if (key[i] != 0) { any |= key[i]; all &= key[i]; ++have; }
  any = __reduce_or_sync(0xffffffffu, any);
  all = __reduce_and_sync(0xffffffffu, all);
  if ((int)__reduce_add_sync(0xffffffffu, have) < k) return 0;
  uint32_t left = any & ~all, prefix = any & all;       // bits that differ; bits that all keys have
  uint32_t below = 0;                                   // the bits under the last decided one
#pragma unroll 1
  for (; left != 0 && most > 0; --most) {
    const uint32_t bit = 0x80000000u >> __clz(left);
    below = bit - 1;
    const uint32_t c = (prefix & ~below) | bit;
    int n = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i) n += key[i] >= c;
    if ((int)__reduce_add_sync(0xffffffffu, n) >= k) prefix |= bit;
    left ^= bit;
  }
  return left == 0 ? prefix : prefix & ~below;
}

// Largest bin b such that the sum of the bins above it is below `want` and including it reaches it (0 if none does), and that sum above
// it plus `above`: one warp, eight bins a lane, from the top.
template <typename V> RB_DEVICE void find_bin(const V* bins, V above, V want, uint32_t* out_bin, V* out_above) {
  const int lane = threadIdx.x & 31;
  V mine[8], sum = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) { mine[i] = bins[255 - (lane * 8 + i)]; sum += mine[i]; }
  V incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const V x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  V cum = above + incl - sum;
  int bin = -1;
  V at = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (bin < 0 && cum + mine[i] >= want) { bin = 255 - (lane * 8 + i); at = cum; }
    cum += mine[i];
  }
  const unsigned hit = __ballot_sync(0xffffffffu, bin >= 0);
  const int w = hit ? __ffs(hit) - 1 : 31;
  const V all = __shfl_sync(0xffffffffu, cum - mine[7], 31);       // nothing reaches `want`: bin 0, everything above it
  const int b = __shfl_sync(0xffffffffu, bin, w);
  const V a = __shfl_sync(0xffffffffu, at, w);
  if (lane == 0) { *out_bin = hit ? (uint32_t)b : 0u; *out_above = hit ? a : all; }
}

template <typename T>
__global__ void __launch_bounds__(kThreads, 1) sample_kernel(SampleParams p) {
  extern __shared__ float srow[];                       // [V] scaled logits
  __shared__ SampleShared sh;
  const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const T* src = reinterpret_cast<const T*>(p.logits) + (int64_t)row * p.row_stride;
  const int V = p.V;
  const bool in_graph = p.step_rows != nullptr;
  if (in_graph) {
    const int st = min(p.step_rows[row], p.n_gen - 1);
    p.step = (uint32_t)st;
    if (p.seed_ptr != nullptr) p.seed = (uint64_t)*p.seed_ptr;
    p.suppress_eos = (p.eos_id >= 0 && st < p.min_new_tokens) ? 1 : 0;
    p.next_tok += st;                                    // row stride of the history buffers is n_gen (set by the host)
    p.logprob += st;
    if (p.mask_bits != nullptr) p.mask_bits += (int64_t)st * (p.mask_stride / p.n_gen);
    __syncthreads();                                     // everybody has read the counter before thread 0 advances it
  }

  // ---- stage + max
  float mx = -INFINITY;
  uint32_t kmax = 0;
  auto put = [&](int j, float raw) {
    float x = raw * p.inv_temp;
    if (p.suppress_eos && j == p.eos_id) x = -INFINITY;
    mx = fmaxf(mx, x);
    kmax = max(kmax, f2key(x));
    return x;
  };
  constexpr int VEC = 16 / sizeof(T);
  const bool vec = p.row_stride % VEC == 0 && (reinterpret_cast<uintptr_t>(p.logits) & 15) == 0;
  if (vec) {
    const int nvec = V / VEC;
    for (int i0 = tid; i0 < nvec; i0 += 4 * kThreads) {                    // four loads in flight
      rb::Pack<T, VEC> v[4];
#pragma unroll
      for (int n = 0; n < 4; ++n)
        if (i0 + n * kThreads < nvec) v[n] = reinterpret_cast<const rb::Pack<T, VEC>*>(src)[i0 + n * kThreads];
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const int i = i0 + n * kThreads;
        if (i < nvec) {
#pragma unroll
          for (int q = 0; q < VEC / 4; ++q)
            reinterpret_cast<float4*>(srow)[i * (VEC / 4) + q] =
                make_float4(put(i * VEC + 4 * q, rb::to_f(v[n].v[4 * q])), put(i * VEC + 4 * q + 1, rb::to_f(v[n].v[4 * q + 1])),
                            put(i * VEC + 4 * q + 2, rb::to_f(v[n].v[4 * q + 2])), put(i * VEC + 4 * q + 3, rb::to_f(v[n].v[4 * q + 3])));
        }
      }
    }
    for (int j = nvec * VEC + tid; j < V; j += kThreads) srow[j] = put(j, rb::to_f(src[j]));
  } else {
    for (int j = tid; j < V; j += kThreads) srow[j] = put(j, rb::to_f(src[j]));
  }
  mx = rb::warp_max(mx);
  if (lane == 0) sh.red[warp] = mx;
  sh.top[tid] = kmax;
  if (tid == 0) sh.u[1] = 0;
  __syncthreads();
  mx = rb::warp_max(sh.red[lane]);

  bool have_bitmap = false;
  int64_t chosen = 0;
  float chosen_lp = 0.f;
  uint32_t keep_key = 0;  // keep elements with key >= keep_key
  // every warp owns a range of whole 32-element groups: (warp, group, lane) is index order
  const int span = ((V + 31) / 32 + kWarps - 1) / kWarps * 32, w0 = min(V, warp * span), w1 = min(V, w0 + span);

  if (p.greedy) {
    // argmax (lowest index among ties)
    int best = V;
    for (int j = tid; j < V; j += kThreads) if (srow[j] == mx) best = min(best, j);
    __syncthreads();
    for (int o = 16; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
    if (lane == 0) sh.u[0] = 0xffffffffu;
    __syncthreads();
    if (lane == 0) atomicMin(&sh.u[0], (uint32_t)best);
    __syncthreads();
    chosen = sh.u[0];
    float s = 0.f;
    for (int j = tid; j < V; j += kThreads) s += __expf(srow[j] - mx);
    s = rb::block_reduce<false>(s, sh.red);
    chosen_lp = -__logf(s);
    keep_key = 0;
  } else {
    const uint32_t r = mix32((uint32_t)p.seed ^ mix32((uint32_t)(p.seed >> 32) + 0x9e3779b9u * (uint32_t)row) ^ mix32(p.step * 0x85ebca6bu + 1u));
    const float u = ((r >> 8) + 0.5f) * (1.0f / 16777216.0f);
    bool done = false;
    if (p.top_k < V && p.top_k <= kFastTopK) {
      // ---- candidates: elements that reach the k-th largest of 256, 512 or 1024 maxima (at least four times k where there are that many)
      if (warp == 0) {
        uint32_t m[32], t0;
#pragma unroll
        for (int i = 0; i < 32; ++i) m[i] = sh.top[i * 32 + lane];
        if (p.top_k > 128) {
          t0 = kth_largest(m, p.top_k, 14);
        } else {
          uint32_t m2[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) m2[i] = max(m[i], m[i + 16]);
          if (p.top_k > 64) {
            t0 = kth_largest(m2, p.top_k, 14);
          } else {
            uint32_t m4[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) m4[i] = max(m2[i], m2[i + 8]);
            t0 = kth_largest(m4, p.top_k, 14);
          }
        }
        if (lane == 0) sh.u[0] = t0;
      }
      __syncthreads();
      const uint32_t t0 = sh.u[0];
      if (kmax >= t0) {                    // the same elements that this thread staged
        auto offer = [&](int j, float x) {
          const uint32_t key = f2key(x);
          if (key >= t0) {
            const uint32_t at = atomicAdd(&sh.u[1], 1u);
            if (at < (uint32_t)kMaxCand) { sh.cand[at] = key; sh.cand_idx[at] = (uint16_t)j; }
          }
        };
        if (vec) {
          const int nvec = V / VEC;
          for (int i = tid; i < nvec; i += kThreads)
#pragma unroll
            for (int q = 0; q < VEC / 4; ++q) {
              const float4 x = reinterpret_cast<const float4*>(srow)[i * (VEC / 4) + q];
              const int j = i * VEC + 4 * q;
              offer(j, x.x); offer(j + 1, x.y); offer(j + 2, x.z); offer(j + 3, x.w);
            }
          for (int j = nvec * VEC + tid; j < V; j += kThreads) offer(j, srow[j]);
        } else {
          for (int j = tid; j < V; j += kThreads) offer(j, srow[j]);
        }
      }
      const int words = (V + 31) / 32;
      for (int i = tid; i < words; i += kThreads) sh.bitmap[i] = 0;
      __syncthreads();
      const int n_cand = (int)sh.u[1];
      if (n_cand <= kMaxCand) {
        // ---- the exact k-th largest
        if (warp == 0) {
          auto exact = [&](auto per) {
            constexpr int kPer = decltype(per)::value;
            uint32_t key[kPer];
#pragma unroll
            for (int i = 0; i < kPer; ++i) key[i] = i * 32 + lane < n_cand ? sh.cand[i * 32 + lane] : 0u;
            return kth_largest(key, p.top_k, 32);
          };
          const uint32_t t = n_cand <= 128 ? exact(std::integral_constant<int, 4>()) : (n_cand <= 512 ? exact(std::integral_constant<int, 16>()) : exact(std::integral_constant<int, 48>()));
          if (lane == 0) sh.u[0] = t;
        }
        __syncthreads();
        keep_key = sh.u[0];
        for (int i = tid; i < n_cand; i += kThreads)
          if (sh.cand[i] >= keep_key) atomicOr(&sh.bitmap[sh.cand_idx[i] >> 5], 1u << (sh.cand_idx[i] & 31));
        __syncthreads();
        // ---- the top-k set in index order: a thread lists the elements of two words
        uint32_t w2[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) w2[i] = 2 * tid + i < words ? sh.bitmap[2 * tid + i] : 0u;
        uint32_t n_kept;
        const uint32_t n_mine = __popc(w2[0]) + __popc(w2[1]);
        uint32_t at = block_inclusive(n_mine, sh.redu, n_kept) - n_mine;
        if (n_kept <= kMaxKept) {
#pragma unroll
          for (int i = 0; i < 2; ++i)
            for (uint32_t w = w2[i]; w != 0; w &= w - 1, ++at) {
              const int j = (2 * tid + i) * 32 + __ffs(w) - 1;
              sh.kept[at] = f2key(srow[j]);
              sh.kept_idx[at] = (uint16_t)j;
              sh.kept_e[at] = __expf(srow[j] - mx);
            }
          __syncthreads();
          if (p.top_p < 1.f) {
            uint32_t lowest = 0xffffffffu;     // the smallest kept key (a key is kept together with all larger ones)
            if (warp * 32 < (int)n_kept) {
              float total = 0.f;
              for (int j = lane; j < (int)n_kept; j += 32) total += sh.kept_e[j];
              const float P = p.top_p * rb::warp_sum(total);
              const uint32_t k = tid < (int)n_kept ? sh.kept[tid] : 0xffffffffu;
              float larger = 0.f;
#pragma unroll 8
              for (int j = 0; j < (int)n_kept; ++j) larger += sh.kept[j] > k ? sh.kept_e[j] : 0.f;
              lowest = __reduce_min_sync(0xffffffffu, tid < (int)n_kept && larger < P ? k : 0xffffffffu);
            }
            if (lane == 0) sh.redu[warp] = lowest;
            __syncthreads();
            lowest = __reduce_min_sync(0xffffffffu, sh.redu[lane]);
            if (lowest != 0xffffffffu) keep_key = max(keep_key, lowest);
            if (tid < (int)n_kept && sh.kept[tid] < keep_key) atomicAnd(&sh.bitmap[sh.kept_idx[tid] >> 5], ~(1u << (sh.kept_idx[tid] & 31)));
          }
          have_bitmap = done = true;
          // ---- inverse CDF over the kept elements
          if (warp == 0) {
            auto mass = [&](int j) { return j < (int)n_kept && sh.kept[j] >= keep_key ? sh.kept_e[j] : 0.f; };
            auto prefix = [&](float e) {
#pragma unroll
              for (int o = 1; o < 32; o <<= 1) {
                const float x = __shfl_up_sync(0xffffffffu, e, o);
                if (lane >= o) e += x;
              }
              return e;
            };
            float kept = 0.f;
            for (int j0 = 0; j0 < (int)n_kept; j0 += 32) kept += __shfl_sync(0xffffffffu, prefix(mass(j0 + lane)), 31);
            const float target = u * kept;
            float before = 0.f;
            int pick = -1, last = 0;           // `last`: rounding at the very end of the CDF
            for (int j0 = 0; j0 < (int)n_kept && pick < 0; j0 += 32) {
              const float e = mass(j0 + lane), incl = prefix(e);
              const unsigned hit = __ballot_sync(0xffffffffu, e > 0.f && target < before + incl);
              const unsigned in = __ballot_sync(0xffffffffu, j0 + lane < (int)n_kept && sh.kept[j0 + lane] >= keep_key);
              if (hit != 0) pick = j0 + __ffs(hit) - 1;
              if (in != 0) last = j0 + 31 - __clz(in);
              before += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (pick < 0) pick = last;
            chosen = sh.kept_idx[pick];
            chosen_lp = srow[chosen] - mx - __logf(kept);
          }
        }
      }
    }
    if (!done) {
      // ---- top-k: k-th largest key by radix descent
      uint32_t prefix = 0, maskbits = 0;
      keep_key = 0;
      if (p.top_k < V) {
        uint32_t remaining = (uint32_t)p.top_k;
        for (int pass = 0; pass < 4; ++pass) {
          const int shift = 24 - 8 * pass;
          __syncthreads();
          if (tid < 256) sh.hist[tid] = 0;
          __syncthreads();
          for (int j = tid; j < V; j += kThreads) {
            const uint32_t k = f2key(srow[j]);
            if ((k & maskbits) == prefix) atomicAdd(&sh.hist[(k >> shift) & 255u], 1u);
          }
          __syncthreads();
          if (warp == 0) find_bin<uint32_t>(sh.hist, 0u, remaining, &sh.u[0], &sh.u[1]);
          __syncthreads();
          prefix |= sh.u[0] << shift;
          maskbits |= 255u << shift;
          remaining -= sh.u[1];
        }
        keep_key = prefix;
      }
      // ---- top-p: weighted radix descent inside the top-k set
      if (p.top_p < 1.f) {
        float tot = 0.f;                             // softmax mass of the top-k set
        for (int j = tid; j < V; j += kThreads) {
          const float x = srow[j];
          if (f2key(x) >= keep_key) tot += __expf(x - mx);
        }
        tot = rb::block_reduce<false>(tot, sh.red);
        const float P = p.top_p * tot;
        float above = 0.f;
        prefix = 0; maskbits = 0;
        for (int pass = 0; pass < 4; ++pass) {
          const int shift = 24 - 8 * pass;
          __syncthreads();
          if (tid < 256) sh.histm[tid] = 0.f;
          __syncthreads();
          for (int j = tid; j < V; j += kThreads) {
            const float x = srow[j];
            const uint32_t k = f2key(x);
            if (k >= keep_key && (k & maskbits) == prefix) atomicAdd(&sh.histm[(k >> shift) & 255u], __expf(x - mx));
          }
          __syncthreads();
          if (warp == 0) find_bin<float>(sh.histm, above, P, &sh.u[0], &sh.f[0]);
          __syncthreads();
          prefix |= sh.u[0] << shift;
          maskbits |= 255u << shift;
          above = sh.f[0];
        }
        keep_key = max(keep_key, prefix);
      }
      // ---- kept mass per warp range, then inverse-CDF sample in index order: the range that holds the target is searched by its warp
      float local = 0.f;
      for (int j = w0 + lane; j < w1; j += 32) {
        const float x = srow[j];
        if (f2key(x) >= keep_key) local += __expf(x - mx);
      }
      local = rb::warp_sum(local);
      __syncthreads();
      if (lane == 0) sh.red[warp] = local;
      if (tid == 0) { sh.u[2] = 0xffffffffu; sh.u[3] = 0; }
      __syncthreads();
      float upto = sh.red[lane];                     // mass of the ranges up to the lane's
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float x = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += x;
      }
      const float kept = __shfl_sync(0xffffffffu, upto, 31), end = __shfl_sync(0xffffffffu, upto, warp), below = __shfl_sync(0xffffffffu, upto, max(warp - 1, 0));
      const float before = warp == 0 ? 0.f : below, target = u * kept;
      if (target >= before && target < end) {        // (the ranges join without gaps)
        // eight groups of 32 at a time, then inside the one that holds the target
        float c = before;
        int group = -1, tail = -1;
        for (int j0 = w0; j0 < w1 && group < 0; j0 += 256) {
          float sum[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int j = j0 + i * 32 + lane;
            sum[i] = rb::warp_sum(j < w1 && f2key(srow[j]) >= keep_key ? __expf(srow[j] - mx) : 0.f);
          }
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (group < 0) {
              if (target < c + sum[i]) group = j0 + i * 32;
              else { c += sum[i]; if (sum[i] > 0.f) tail = j0 + i * 32; }
            }
        }
        if (group < 0) group = tail;                 // rounding: the groups' sums end below the range's; their last element
        if (group >= 0) {
          const int j = group + lane;
          const bool in = j < w1 && f2key(srow[j]) >= keep_key;
          float incl = in ? __expf(srow[j] - mx) : 0.f;
          const unsigned all = __ballot_sync(0xffffffffu, incl > 0.f);
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const float x = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += x;
          }
          const unsigned hit = __ballot_sync(0xffffffffu, in && target < c + incl);
          if (lane == 0) atomicMin(&sh.u[2], (uint32_t)(group + (hit ? __ffs(hit) - 1 : 31 - __clz(all))));
        }
      }
      __syncthreads();
      chosen = sh.u[2];
      if (sh.u[2] == 0xffffffffu) {                  // rounding at the very end of the CDF, or no mass at all (NaN, infinities alone): the last kept element
        int last = -1;
        if (local > 0.f || !(kept > 0.f))
          for (int j = w0 + lane; j < w1; j += 32)
            if (f2key(srow[j]) >= keep_key) last = j;
        if (last >= 0) atomicMax(&sh.u[3], (uint32_t)last);
        __syncthreads();
        chosen = sh.u[3];
      }
      chosen_lp = srow[chosen] - mx - __logf(kept);
    }
  }

  const bool live = p.unfinished == nullptr || p.unfinished[row];
  const int64_t out_stride = in_graph ? p.n_gen : 1;
  __syncthreads();  // all reads of unfinished[row] precede its update
  if (tid == 0) {
    const int64_t tok = live ? chosen : (int64_t)p.pad_id;
    p.next_tok[row * out_stride] = tok;
    p.logprob[row * out_stride] = live ? chosen_lp : 0.f;
    if (p.unfinished_out != nullptr) p.unfinished_out[row] = live && tok != (int64_t)p.eos_id;
    if (in_graph) {
      p.input_ids[row] = tok;
      p.cache_lens[row] += 1;
      p.step_rows[row] = (int)p.step + 1;
      if (p.eos_id >= 0) p.unfinished_rw[row] = live && tok != (int64_t)p.eos_id;
    }
  }
  if (p.mask_bits != nullptr && have_bitmap) {         // (complete since the barrier above)
    uint8_t* mrow = p.mask_bits + (int64_t)row * p.mask_stride;
    const int nbytes = (V + 7) / 8;
    const bool words = (reinterpret_cast<uintptr_t>(mrow) & 3) == 0;
    for (int i = tid; i * 4 < nbytes; i += kThreads) {
      const uint32_t word = ~sh.bitmap[i] & (V - i * 32 >= 32 ? 0xffffffffu : (1u << (V - i * 32)) - 1u);
      if (words && i * 4 + 4 <= nbytes) {
        *reinterpret_cast<uint32_t*>(mrow + i * 4) = word;
      } else {
        for (int e = 0; e < 4; ++e)
          if (i * 4 + e < nbytes) mrow[i * 4 + e] = (uint8_t)(word >> (8 * e));
      }
    }
  } else if (p.mask_bits != nullptr) {
    // 32 elements a ballot, up to 1024 a warp and round (the words of a short row spread over all warps): lane i ends up with the i-th word of the round
    uint8_t* mrow = p.mask_bits + (int64_t)row * p.mask_stride;
    const int nbytes = (V + 7) / 8, per_warp = min(32, ((V + 31) / 32 + kWarps - 1) / kWarps);
    const bool words = (reinterpret_cast<uintptr_t>(mrow) & 3) == 0;
    for (int j0 = warp * per_warp * 32; j0 < V; j0 += kWarps * per_warp * 32) {
      uint32_t word = 0;
#pragma unroll 8
      for (int i = 0; i < per_warp; ++i) {
        const int j = j0 + i * 32 + lane;
        const unsigned b = __ballot_sync(0xffffffffu, j < V && f2key(srow[j]) < keep_key);
        if (lane == i) word = b;
      }
      const int byte = j0 / 8 + lane * 4;
      if (lane >= per_warp) {
      } else if (words && byte + 4 <= nbytes) {
        *reinterpret_cast<uint32_t*>(mrow + byte) = word;
      } else {
        for (int i = 0; i < 4; ++i)
          if (byte + i < nbytes) mrow[byte + i] = (uint8_t)(word >> (8 * i));
      }
    }
  }
}

int launch_sample(const SampleParams& p, int B, int dt, cudaStream_t s) {
  const size_t smem = (size_t)p.V * sizeof(float);
#define RB_GO(T)                                                                                                  \
  {                                                                                                               \
    static bool cfgd = false;                                                                                     \
    if (!cfgd) {                                                                                                  \
      if (cudaFuncSetAttribute(sample_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess) return -2; \
      cfgd = true;                                                                                                \
    }                                                                                                             \
    sample_kernel<T><<<B, kThreads, smem, s>>>(p);                                                                \
  }
  if (dt == 0) RB_GO(float) else if (dt == 1) RB_GO(__nv_bfloat16) else if (dt == 2) RB_GO(__half) else return -3;
#undef RB_GO
  return 0;
}


}  // namespace

extern "C" int rb_sample(const void* logits, int64_t row_stride, int64_t* next_tok, float* logprob, uint8_t* mask_bits,
                         int64_t mask_stride, const bool* unfinished, int B, int V, int top_k, float top_p, float inv_temp,
                         int eos_id, int suppress_eos, int greedy, int pad_id, uint64_t seed, uint32_t step, bool* unfinished_out, int dt,
                         cudaStream_t s) {
  if (B == 0) return 0;
  const size_t smem = (size_t)V * sizeof(float);
  if (smem > 200 * 1024) return -1;
  SampleParams p{logits, row_stride, next_tok, logprob, mask_bits, mask_stride, unfinished, V, top_k, eos_id, suppress_eos, greedy,
                 pad_id, inv_temp, top_p, seed, step, nullptr, nullptr, nullptr, nullptr, 1, 0, unfinished_out, nullptr};
  return launch_sample(p, B, dt, s);
}

// In-graph variant: see SampleParams.  tok_hist / lp_hist are [B, n_gen], mask_hist [B, n_gen, mask_bytes] (or null).
extern "C" int rb_sample_graph(const void* logits, int64_t row_stride, int64_t* tok_hist, float* lp_hist, uint8_t* mask_hist,
                               int64_t mask_bytes, bool* unfinished, int* step_rows, int64_t* input_ids, int* cache_lens, int n_gen,
                               int min_new_tokens, int B, int V, int top_k, float top_p, float inv_temp, int eos_id, int greedy,
                               int pad_id, const int64_t* seed_ptr, int dt, cudaStream_t s) {
  if (B == 0) return 0;
  if ((size_t)V * sizeof(float) > 200 * 1024) return -1;
  SampleParams p{logits, row_stride, tok_hist, lp_hist, mask_hist, mask_bytes * n_gen, unfinished, V, top_k, eos_id, 0, greedy,
                 pad_id, inv_temp, top_p, 0, 0, step_rows, input_ids, cache_lens, unfinished, n_gen, min_new_tokens, nullptr, seed_ptr};
  return launch_sample(p, B, dt, s);
}

