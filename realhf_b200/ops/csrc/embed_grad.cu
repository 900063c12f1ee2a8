// Rows of an embedding table, out[t, :] = table[ids[t], :]: copies of 16 bytes.  A generation step's 16 rows of 8 KB took 7.5 us through the library, which goes
// through few indices one after the other, now 1.2 (1 / 64 / 1024 rows 1.7 / 1.5 / 3.0, now 1.1 / 1.3 / 2.9; 20480 rows 61, now 48).
// And the table's gradient, added to a dense buffer: dst[v, :] += sum over the tokens t with ids[t] == v, in ascending t, of dy[t, :].
//
// What bounds it: reading dy once and reading and writing the rows that occur, a few dozen MB; everything else is latency.  No sort: a pass chains the tokens
// of an id (atomics, in any order) and counts them, then the warp of one token an id sums the id's rows.  The order within a chain differs from run to run, so
// up to 32 tokens are ranked in registers first and the sums are the same each time.  Ids with more get a list of their tokens, and blocks that own 64 columns each
// put the list in order (by ranks up to 512 tokens, through a bitmap beyond) and sum it.  The sums are fp32 and are rounded once, with the buffer's own value.
// Through the library's dense gradient (sort of the ids, segments, a zeroed [V, H], its sum into the buffer) / so, us, bf16:
//   3790 tokens x 2048, uniform over 32000 ids  349 / 28     20480 x 4096, uniform 1590 / 121     2000 x 768, every id 32 times  105 / 31
//   20480 x 4096, frequencies as 1 / rank      1182 / 191    100000 x 768, as 1 / rank of 50257  669 / 212   20480 x 4096, one id  916 / 111
//   positions 0 .. 1023 of 64 sequences x 1024  255 / 83     0 .. 511 of 128 x 768  228 / 53      32768 tokens of 256 ids x 1024  185 / 54
// (each of those ids scanning all tokens for itself, as it was at first: positions 4374 and 1779, 256 ids 622).  A long list's bitmap is made in windows of 65536 tokens, each of
// which reads the whole list: beyond 2^18 tokens a call goes the library's way (500000 x 768, as 1 / rank: 1554 against 3254; one id of 200000 x 256 still 1689 / 788).
#include <assert.h>

#include "common.cuh"

namespace {

constexpr int kThreads = 256, kWarps = kThreads / 32, kChain = 32, kSlice = 64;
constexpr int kRanked = 512, kWindow = 65536, kStep = 4096;
struct Heavy { int v, at, n; };      // id, first place in the list, tokens

template <typename T> RB_DEVICE void load8(const T* p, rb::Pack<T, 8>& x) {
  constexpr int N = 16 / sizeof(T);
#pragma unroll
  for (int h = 0; h < 8 / N; ++h) reinterpret_cast<rb::Pack<T, N>*>(x.v)[h] = *reinterpret_cast<const rb::Pack<T, N>*>(p + h * N);
}

template <typename T> RB_DEVICE void add8(const T* p, float* acc) {
  constexpr int N = 16 / sizeof(T);
#pragma unroll
  for (int h = 0; h < 8 / N; ++h) {
    const rb::Pack<T, N> v = *reinterpret_cast<const rb::Pack<T, N>*>(p + h * N);
#pragma unroll
    for (int i = 0; i < N; ++i) acc[h * N + i] += rb::to_f(v.v[i]);
  }
}
template <typename T> RB_DEVICE void store8(T* p, const float* acc) {
  constexpr int N = 16 / sizeof(T);
#pragma unroll
  for (int h = 0; h < 8 / N; ++h) {
    rb::Pack<T, N> v;
#pragma unroll
    for (int i = 0; i < N; ++i) v.v[i] = rb::from_f<T>(acc[h * N + i]);
    *reinterpret_cast<rb::Pack<T, N>*>(p + h * N) = v;
  }
}

// A block copies kVec x 128 pieces of one row.  It heads a forward pass, so it lets the next kernels start only behind its own wait: a small-row product two kernels
// on asks for weight tiles in front of ITS wait, and what wrote the weights may be the kernel in front of this one, whose stores nothing but a wait makes visible.
constexpr int kRowThreads = 128;
template <typename I, int kVec>
__global__ void __launch_bounds__(kRowThreads) rows_kernel(const I* __restrict__ ids, const uint4* __restrict__ table, uint4* __restrict__ out, int64_t V, int n) {
  rb::pdl_wait();
  rb::pdl_trigger();
  const int64_t t = blockIdx.x, v = (int64_t)ids[t];
  assert(v >= 0 && v < V);                                // as the library's lookup does
  const int first = blockIdx.y * (kVec * kRowThreads) + threadIdx.x;
  uint4 x[kVec];
#pragma unroll
  for (int i = 0; i < kVec; ++i)
    if (first + i * kRowThreads < n) x[i] = table[v * n + first + i * kRowThreads];
#pragma unroll
  for (int i = 0; i < kVec; ++i)
    if (first + i * kRowThreads < n) out[t * n + first + i * kRowThreads] = x[i];
}

// The same for many rows: a warp a row, four pieces a lane in flight.  A block a row is launched as often as there are rows, whatever is in them.
template <typename I>
__global__ void __launch_bounds__(kThreads) rows_warp_kernel(const I* __restrict__ ids, const uint4* __restrict__ table, uint4* __restrict__ out, int64_t V, int n, int64_t T) {
  constexpr int kAhead = 4;
  rb::pdl_wait();
  rb::pdl_trigger();
  const int64_t t = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
  if (t >= T) return;
  const int64_t v = (int64_t)ids[t];
  assert(v >= 0 && v < V);
  const uint4* from = table + v * n;
  uint4* to = out + t * n;
  for (int c = threadIdx.x & 31; c < n; c += 32 * kAhead) {
    uint4 x[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      if (c + 32 * i < n) x[i] = from[c + 32 * i];
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      if (c + 32 * i < n) to[c + 32 * i] = x[i];
  }
}

// head[v]: last token of the chain plus one (0: none), next[t]: the one before it, in the same form; rank[t]: how many of its id were counted before it
template <typename I>
__global__ void __launch_bounds__(kThreads) chain_kernel(const I* __restrict__ ids, int* __restrict__ head, int* __restrict__ count, int* __restrict__ next,
                                                         int* __restrict__ rank, int T, int V) {
  const int t = blockIdx.x * kThreads + threadIdx.x, lane = threadIdx.x & 31;
  const int64_t v = t < T ? (int64_t)ids[t] : -1;
  const bool in = v >= 0 && v < V;
  // the tokens of a warp with one id are chained among themselves: one pair of atomics for them
  const unsigned same = __match_any_sync(0xffffffffu, in ? (int)v : -1), below = same & ((1u << lane) - 1u);
  if (!in) return;
  int link = 0, before = 0;
  if (below == 0u) {
    link = atomicExch(head + v, t - lane + 32 - __clz(same));
    before = atomicAdd(count + v, __popc(same));
  } else {
    link = t - lane + 32 - __clz(below);
  }
  before = __shfl_sync(same, before, __ffs(same) - 1);
  next[t] = link;
  rank[t] = before + __popc(below);
}

template <typename I, typename G, typename D>
__global__ void __launch_bounds__(kThreads) sum_kernel(const I* __restrict__ ids, int* __restrict__ head, const int* __restrict__ count,
                                                       const int* __restrict__ next, int* __restrict__ totals, Heavy* __restrict__ heavy,
                                                       const G* __restrict__ dy, D* __restrict__ dst, int T, int V, int H) {
  __shared__ int order[kWarps][kChain];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = blockIdx.x * kWarps + warp;
  if (t >= T) return;
  const int64_t v = (int64_t)ids[t];
  if (v < 0 || v >= V || head[v] != t + 1) return;      // the chain's last token speaks for it
  const int c = count[v];
  __syncwarp();                                          // all lanes have read head[v]
  if (c > kChain) {                                      // room in the list of tokens; the place is left where the id's other tokens find it
    if (lane == 0) {
      const int at = atomicAdd(totals + 1, c);
      heavy[atomicAdd(totals, 1)] = Heavy{(int)v, at, c};
      head[v] = -1 - at;
    }
    return;
  }
  int mine = 0, cur = t + 1;
  for (int i = 0; i < c; ++i) {
    if (lane == i) mine = cur;
    cur = next[cur - 1];
  }
  int rank = 0;
  for (int i = 0; i < c; ++i) rank += __shfl_sync(0xffffffffu, mine, i) < mine;
  if (lane < c) order[warp][rank] = mine - 1;
  __syncwarp();
  D* row = dst + v * H;
#pragma unroll 4
  for (int col = lane * 8; col < H; col += 256) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int i = 0; i < c; ++i) add8(dy + (int64_t)order[warp][i] * H + col, acc);
    add8(row + col, acc);
    store8(row + col, acc);
  }
}

// Tokens of the ids with long chains -> the ids' places in the list, in any order.  (The list takes the memory of `next`, which nobody reads any more.)
template <typename I>
__global__ void __launch_bounds__(kThreads) place_kernel(const I* __restrict__ ids, const int* __restrict__ head, const int* __restrict__ count,
                                                         const int* __restrict__ rank, int* __restrict__ list, int T, int V) {
  const int t = blockIdx.x * kThreads + threadIdx.x;
  if (t >= T) return;
  const int64_t v = (int64_t)ids[t];
  if (v < 0 || v >= V || count[v] <= kChain) return;
  list[-1 - head[v] + rank[t]] = t;
}

// Ids with long chains: a block takes an id and some slices of 64 columns, puts the id's tokens in order and lets 32 rows of threads take them by turns; their
// sums are added up in order.
template <typename G, typename D>
__global__ void __launch_bounds__(kThreads, 4) heavy_kernel(const int* __restrict__ totals, const Heavy* __restrict__ heavy, const int* __restrict__ list,
                                                            const G* __restrict__ dy, D* __restrict__ dst, int T, int H) {
  constexpr int kAhead = sizeof(G) == 2 ? 8 : 4;          // rows of a thread on their way
  __shared__ float part[32][kSlice];
  __shared__ __align__(16) unsigned bits[kWindow / 32];   // of a stretch of tokens those of the id; up to kRanked tokens: the tokens, unordered
  __shared__ int sorted[kRanked];
  __shared__ uint16_t hits[kStep];
  __shared__ int per_warp[kWarps];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, group = tid & 7, turn = tid >> 3;
  const int slices = RB_CEIL_DIV(H, kSlice), n_heavy = totals[0];
  // slices of an id that one block takes: several works a block are left, so that they balance
  const int64_t all = (int64_t)n_heavy * slices;
  const int per = (int)min((int64_t)slices, max((int64_t)1, all / (4 * (int64_t)gridDim.x))), parts = RB_CEIL_DIV(slices, per);
  for (int64_t work = blockIdx.x; work < (int64_t)n_heavy * parts; work += gridDim.x) {
    const Heavy h = heavy[work / parts];
    const int* mine = list + h.at;
    const int s0 = (int)(work % parts) * per, s1 = min(slices, s0 + per);
    const bool ranked = h.n <= kRanked;
    if (ranked) {                                         // a token's place is the number of smaller ones
      int* raw = reinterpret_cast<int*>(bits);
      const int n4 = RB_CEIL_DIV(h.n, 4);
      for (int i = tid; i < n4 * 4; i += kThreads) raw[i] = i < h.n ? mine[i] : 0x7fffffff;
      __syncthreads();
      for (int i = tid; i < h.n; i += kThreads) {
        const int x = raw[i];
        int at = 0;
        for (int j = 0; j < n4; ++j) {
          const int4 o = reinterpret_cast<const int4*>(raw)[j];
          at += (o.x < x) + (o.y < x) + (o.z < x) + (o.w < x);
        }
        sorted[at] = x;
      }
      __syncthreads();
    }
    for (int slice = s0; slice < s1; ++slice) {
      const int col = slice * kSlice + group * 8, out = slice * kSlice + tid;
      const bool writes = tid < kSlice && out < H;
      D* const to = dst + (int64_t)h.v * H + out;
      const float old = writes ? rb::to_f(*to) : 0.f;
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      auto sum = [&](auto token, int first, int n) {      // rows token(first), token(first + 32), ..
        if (col >= H) return;
        int i = first;
        for (; i + 32 * (kAhead - 1) < n; i += 32 * kAhead) {
          rb::Pack<G, 8> x[kAhead];
#pragma unroll
          for (int e = 0; e < kAhead; ++e) load8(dy + (int64_t)token(i + 32 * e) * H + col, x[e]);
#pragma unroll
          for (int e = 0; e < kAhead; ++e)
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[k] += rb::to_f(x[e].v[k]);
        }
        for (; i < n; i += 32) add8(dy + (int64_t)token(i) * H + col, acc);
      };
      if (ranked) {
        sum([&](int i) { return sorted[i]; }, turn, h.n);
      } else {
        int seen = 0;                                     // tokens of the id in front of this step
        for (int w0 = 0; w0 < T; w0 += kWindow) {
          for (int i = tid; i < kWindow / 32; i += kThreads) bits[i] = 0u;
          __syncthreads();
#pragma unroll 8
          for (int i = tid; i < h.n; i += kThreads) {
            const unsigned x = (unsigned)(mine[i] - w0);
            if (x < (unsigned)kWindow) atomicOr(bits + (x >> 5), 1u << (x & 31));
          }
          __syncthreads();
          for (int b0 = 0; b0 < kWindow && w0 + b0 < T; b0 += kStep) {
            unsigned m = tid < kStep / 32 ? bits[b0 / 32 + tid] : 0u;
            const int n = __popc(m);
            int upto = n;
#pragma unroll
            for (int d = 1; d < 32; d *= 2) {
              const int y = __shfl_up_sync(0xffffffffu, upto, d);
              if (lane >= d) upto += y;
            }
            if (lane == 31) per_warp[warp] = upto;
            __syncthreads();
            int at = upto - n, total = 0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
              at += w < warp ? per_warp[w] : 0;
              total += per_warp[w];
            }
            for (; m != 0u; m &= m - 1u) hits[at++] = (uint16_t)(tid * 32 + __ffs(m) - 1);
            __syncthreads();
            sum([&](int i) { return w0 + b0 + (int)hits[i]; }, (turn - seen) & 31, total);
            seen += total;
            __syncthreads();
          }
        }
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) part[turn][group * 8 + e] = acc[e];
      __syncthreads();
      if (writes) {
        float s = 0.f;
#pragma unroll
        for (int r = 0; r < 32; ++r) s += part[r][tid];
        *to = rb::from_f<D>(s + old);
      }
      __syncthreads();
    }
  }
}

template <typename I, typename G, typename D>
int run(const void* dy_, const void* ids_, void* dst_, int* scratch, int T, int V, int H, cudaStream_t s) {
  const I* ids = reinterpret_cast<const I*>(ids_);
  const G* dy = reinterpret_cast<const G*>(dy_);
  D* dst = reinterpret_cast<D*>(dst_);
  int *head = scratch, *count = head + V, *totals = count + V, *next = totals + 2, *rank = next + T;
  Heavy* heavy = reinterpret_cast<Heavy*>(rank + T);
  if (cudaMemsetAsync(scratch, 0, sizeof(int) * (2 * (size_t)V + 2), s) != cudaSuccess) return -2;
  chain_kernel<I><<<RB_CEIL_DIV(T, kThreads), kThreads, 0, s>>>(ids, head, count, next, rank, T, V);
  sum_kernel<I, G, D><<<RB_CEIL_DIV(T, kWarps), kThreads, 0, s>>>(ids, head, count, next, totals, heavy, dy, dst, T, V, H);
  if (T > kChain) {                                       // no id can have more otherwise
    place_kernel<I><<<RB_CEIL_DIV(T, kThreads), kThreads, 0, s>>>(ids, head, count, rank, next, T, V);
    const int64_t most = (int64_t)(T / (kChain + 1)) * RB_CEIL_DIV(H, kSlice);
    heavy_kernel<G, D><<<(int)(most < 4 * rb::kNumSMs ? most : 4 * rb::kNumSMs), kThreads, 0, s>>>(totals, heavy, next, dy, dst, T, H);
  }
  return cudaGetLastError() != cudaSuccess ? -3 : T > kChain ? 4 : 2;
}

}  // namespace

// dy [T, H], dst [V, H] (packed, 16-byte aligned, H a multiple of 8); g_dt / d_dt: 0 fp32, 1 bf16, 2 fp16, d_dt = g_dt or 0; ids int64 or int32, those outside
// [0, V) are passed over; scratch: 2 V + 2 + 2 T + 3 (T / 33) words.  Returns the
// number of kernels launched, or a negative code.
extern "C" int rb_embedding_grad(const void* dy, const void* ids, int ids_64, void* dst, int* scratch, int64_t T, int64_t V, int64_t H, int g_dt, int d_dt,
                                 cudaStream_t s) {
  if (T <= 0 || V <= 0 || H <= 0) return 0;
  if (H % 8 != 0 || T > (1 << 30) || V > (1 << 30) || H > (1 << 24) || (((uintptr_t)dy | (uintptr_t)dst) & 15)) return -1;
#define RB_GO(G, D) return ids_64 ? run<int64_t, G, D>(dy, ids, dst, scratch, (int)T, (int)V, (int)H, s) : run<int32_t, G, D>(dy, ids, dst, scratch, (int)T, (int)V, (int)H, s)
  if (g_dt == 1 && d_dt == 1) RB_GO(__nv_bfloat16, __nv_bfloat16);
  if (g_dt == 1 && d_dt == 0) RB_GO(__nv_bfloat16, float);
  if (g_dt == 2 && d_dt == 2) RB_GO(__half, __half);
  if (g_dt == 2 && d_dt == 0) RB_GO(__half, float);
  if (g_dt == 0 && d_dt == 0) RB_GO(float, float);
#undef RB_GO
  return -4;
}

// out [T, row_bytes], table [V, row_bytes] (packed, 16-byte aligned, row_bytes a multiple of 16); ids int64 or int32 below V.  A block a row: a piece a thread while that
// leaves SMs without a block, two otherwise (four: 3.3 us for 1024 rows of 8 KB, two 2.9), four for some thousand rows from 16 KB (1800 of 16 KB two 7.5, four 6.3; 20480 of
// them two 94, four 98).  A warp a row for many rows where blocks would idle for more than a tenth or all stays in L2 (us, the library's lookup / a block / a warp a row:
// 4000 rows of 1.5 KB 3.8 / 4.8 / 3.1, 20480 of them 12.2 / 22.0 / 7.1, 20480 of 6400 bytes 36.1 / 43.3 / 22.6, 4000 of 8 KB 8.4 / 9.1 / 8.2; but 1000 of 1.5 KB
// 2.2 / 1.8 / 2.2, 1300 of 10 KB 4.5 / 4.9 / 5.2, 20480 of 8 KB 61 / 48 / 52).
extern "C" int rb_embedding_rows(const void* table, const void* ids, int ids_64, void* out, int64_t T, int64_t V, int64_t row_bytes, cudaStream_t s) {
  if (T <= 0 || row_bytes <= 0) return 0;
  if (row_bytes % 16 != 0 || T > 0x7fffffff || row_bytes > (1 << 24) || (((uintptr_t)table | (uintptr_t)out) & 15)) return -1;
  const int n = (int)(row_bytes / 16);
  const int64_t slots = (int64_t)RB_CEIL_DIV(n, 2 * kRowThreads) * (2 * kRowThreads);
  if (10 * (slots - n) > slots ? T >= 1536 : n < 1024 && T >= 2048 && T * row_bytes <= (48 << 20)) {
    const dim3 warps((unsigned)RB_CEIL_DIV(T, kWarps));
#define RB_GO(I) rb::launch_pdl(rows_warp_kernel<I>, warps, dim3(kThreads), 0, s, (const I*)ids, (const uint4*)table, (uint4*)out, V, n, T) == cudaSuccess ? 0 : -3
    if (ids_64) return RB_GO(int64_t);
    return RB_GO(int32_t);
#undef RB_GO
  }
  const bool many = T * RB_CEIL_DIV(n, 2 * kRowThreads) >= rb::kNumSMs;
  const int per = many ? (n >= 1024 && T > 1000 && T <= 8192 ? 4 : 2) : 1;
  const dim3 grid((unsigned)T, RB_CEIL_DIV(n, per * kRowThreads));
#define RB_GO(I, N) \
  rb::launch_pdl(rows_kernel<I, N>, grid, dim3(kRowThreads), 0, s, (const I*)ids, (const uint4*)table, (uint4*)out, V, n) == cudaSuccess ? 0 : -3
  if (per == 4) return ids_64 ? RB_GO(int64_t, 4) : RB_GO(int32_t, 4);
  if (ids_64) return many ? RB_GO(int64_t, 2) : RB_GO(int64_t, 1);
  return many ? RB_GO(int32_t, 2) : RB_GO(int32_t, 1);
#undef RB_GO
}

// Tokens of a call up to which the gradient is no slower than the library's.
extern "C" int64_t rb_embedding_grad_tokens() { return 1 << 18; }
