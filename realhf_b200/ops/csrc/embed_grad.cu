// Rows of an embedding table, out[t, :] = table[ids[t], :]: copies of 16 bytes.  A generation step's 16 rows of 8 KB took 7.5 us through the library, which goes
// through few indices one after the other, now 1.2 (1 / 64 / 1024 rows 1.7 / 1.5 / 3.0, now 1.1 / 1.3 / 2.9; 20480 rows 61, now 48).
// And the table's gradient, added to a dense buffer: dst[v, :] += sum over the tokens t with ids[t] == v, in ascending t, of dy[t, :].
//
// What bounds it: reading dy once and reading and writing the rows that occur, a few dozen MB; everything else is latency.  No sort: a pass chains the tokens
// of an id (atomics, in any order) and counts them, then the warp of one token an id sums the id's rows.  The order within a chain differs from run to run, so
// up to 32 tokens are ranked in registers first and the sums are the same each time; ids with more go to a list, and blocks that own 64 columns each scan all ids
// in order for them (20480 equal ids at width 4096: 64 blocks).  The sums are fp32 and are rounded once, with the buffer's own value.
// Through the library's dense gradient (sort of the ids, segments, a zeroed [V, H], its sum into the buffer) 3790 tokens x 2048 of 32000 ids took
// 265 us in a training step, now 17.
#include <assert.h>

#include "common.cuh"

namespace {

constexpr int kThreads = 256, kWarps = kThreads / 32, kChain = 32, kSlice = 64;

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

// head[v]: last token of the chain plus one (0: none), next[t]: the one before it, in the same form
template <typename I>
__global__ void __launch_bounds__(kThreads) chain_kernel(const I* __restrict__ ids, int* __restrict__ head, int* __restrict__ count, int* __restrict__ next, int T,
                                                         int V) {
  const int t = blockIdx.x * kThreads + threadIdx.x;
  if (t >= T) return;
  const int64_t v = (int64_t)ids[t];
  if (v < 0 || v >= V) return;
  next[t] = atomicExch(head + v, t + 1);
  atomicAdd(count + v, 1);
}

template <typename I, typename G, typename D>
__global__ void __launch_bounds__(kThreads) sum_kernel(const I* __restrict__ ids, const int* __restrict__ head, const int* __restrict__ count,
                                                       const int* __restrict__ next, int* __restrict__ n_heavy, int* __restrict__ heavy,
                                                       const G* __restrict__ dy, D* __restrict__ dst, int T, int V, int H) {
  __shared__ int order[kWarps][kChain];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = blockIdx.x * kWarps + warp;
  if (t >= T) return;
  const int64_t v = (int64_t)ids[t];
  if (v < 0 || v >= V || head[v] != t + 1) return;      // the chain's last token speaks for it
  const int c = count[v];
  if (c > kChain) {
    if (lane == 0) heavy[atomicAdd(n_heavy, 1)] = (int)v;
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

// ids with long chains: a block takes (id, slice of 64 columns); 32 rows of threads take its tokens by turns, their sums are added up in order
template <typename I, typename G, typename D>
__global__ void __launch_bounds__(kThreads) heavy_kernel(const I* __restrict__ ids, const int* __restrict__ n_heavy, const int* __restrict__ heavy,
                                                         const G* __restrict__ dy, D* __restrict__ dst, int T, int H) {
  __shared__ int hits[kThreads], per_warp[kWarps];
  __shared__ float part[32][kSlice];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, group = threadIdx.x & 7, turn = threadIdx.x >> 3;
  const int slices = RB_CEIL_DIV(H, kSlice);
  for (int64_t work = blockIdx.x; work < (int64_t)*n_heavy * slices; work += gridDim.x) {
    const int v = heavy[work / slices], col = (int)(work % slices) * kSlice + group * 8;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    int seen = 0;                                         // tokens of the id in front of this stretch of ids
    for (int t0 = 0; t0 < T; t0 += kThreads) {
      const int t = t0 + threadIdx.x;
      const bool hit = t < T && (int64_t)ids[t] == v;
      const unsigned mask = __ballot_sync(0xffffffffu, hit);
      if (lane == 0) per_warp[warp] = __popc(mask);
      __syncthreads();
      int before = 0, total = 0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        before += w < warp ? per_warp[w] : 0;
        total += per_warp[w];
      }
      if (hit) hits[before + __popc(mask & ((1u << lane) - 1u))] = t;
      __syncthreads();
      if (col < H)
        for (int i = (turn - seen) & 31; i < total; i += 32) add8(dy + (int64_t)hits[i] * H + col, acc);
      seen += total;
      __syncthreads();
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) part[turn][group * 8 + e] = acc[e];
    __syncthreads();
    if (turn == 0 && col < H) {
      float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int r = 0; r < 32; ++r)
#pragma unroll
        for (int e = 0; e < 8; ++e) sum[e] += part[r][group * 8 + e];
      D* row = dst + (int64_t)v * H + col;
      add8(row, sum);
      store8(row, sum);
    }
    __syncthreads();
  }
}

template <typename I, typename G, typename D>
int run(const void* dy_, const void* ids_, void* dst_, int* scratch, int T, int V, int H, cudaStream_t s) {
  const I* ids = reinterpret_cast<const I*>(ids_);
  const G* dy = reinterpret_cast<const G*>(dy_);
  D* dst = reinterpret_cast<D*>(dst_);
  int *head = scratch, *count = head + V, *n_heavy = count + V, *heavy = n_heavy + 1, *next = heavy + T / kChain;
  if (cudaMemsetAsync(scratch, 0, sizeof(int) * (2 * (size_t)V + 1), s) != cudaSuccess) return -2;
  chain_kernel<I><<<RB_CEIL_DIV(T, kThreads), kThreads, 0, s>>>(ids, head, count, next, T, V);
  sum_kernel<I, G, D><<<RB_CEIL_DIV(T, kWarps), kThreads, 0, s>>>(ids, head, count, next, n_heavy, heavy, dy, dst, T, V, H);
  if (T > kChain) {                                       // no id can have more otherwise
    const int64_t most = (int64_t)(T / (kChain + 1)) * RB_CEIL_DIV(H, kSlice);
    heavy_kernel<I, G, D><<<(int)(most < 4 * rb::kNumSMs ? most : 4 * rb::kNumSMs), kThreads, 0, s>>>(ids, n_heavy, heavy, dy, dst, T, H);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace

// dy [T, H], dst [V, H] (packed, 16-byte aligned, H a multiple of 8); g_dt / d_dt: 0 fp32, 1 bf16, 2 fp16, d_dt = g_dt or 0; ids int64 or int32, those outside
// [0, V) are passed over; scratch: 2 V + 1 + T / 32 + T words.
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

// out [T, row_bytes], table [V, row_bytes] (packed, 16-byte aligned, row_bytes a multiple of 16); ids int64 or int32 below V.  A piece a thread while that leaves
// SMs without a block, two otherwise (four: 3.3 us for 1024 rows of 8 KB, two 2.9).
extern "C" int rb_embedding_rows(const void* table, const void* ids, int ids_64, void* out, int64_t T, int64_t V, int64_t row_bytes, cudaStream_t s) {
  if (T <= 0 || row_bytes <= 0) return 0;
  if (row_bytes % 16 != 0 || T > 0x7fffffff || row_bytes > (1 << 24) || (((uintptr_t)table | (uintptr_t)out) & 15)) return -1;
  const int n = (int)(row_bytes / 16);
  const bool many = T * RB_CEIL_DIV(n, 2 * kRowThreads) >= rb::kNumSMs;
  const dim3 grid((unsigned)T, RB_CEIL_DIV(n, (many ? 2 : 1) * kRowThreads));
#define RB_GO(I, N) \
  rb::launch_pdl(rows_kernel<I, N>, grid, dim3(kRowThreads), 0, s, (const I*)ids, (const uint4*)table, (uint4*)out, V, n) == cudaSuccess ? 0 : -3
  if (ids_64) return many ? RB_GO(int64_t, 2) : RB_GO(int64_t, 1);
  return many ? RB_GO(int32_t, 2) : RB_GO(int32_t, 1);
#undef RB_GO
}
