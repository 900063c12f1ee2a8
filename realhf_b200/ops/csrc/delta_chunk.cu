// Gated delta rule, packed form, in chunks of 64 tokens on the tensor cores (head size 128 x 128, one decay per head and token; see delta.cu for the
// recurrence and for every other form).  Per (sequence, head) and chunk, from the state S in front of it, with C_i the product of the decays of the
// chunk's tokens up to i and D_ij of those after j up to i (products of decays throughout: no logarithms, so a decay of 0 is one like any other):
//     A_ij = beta_i D_ij (k_i . k_j)  (j < i),   T = (I + A)^-1,   W_ij = D_ij (q_i . k_j)  (j <= i)          [64 x 64], none of them depends on S
//     X = S^T K^T, Y = S^T Q^T,   r_i = beta_i (v_i - C_i X_i),   U^T = R^T T^T                              [128 x 64] each
//     o_i = C_i Y_i + sum_{j <= i} W_ij u_j,   S <- C_last S + sum_j (D_last,j k_j) u_j^T
// The serial chain is one step per 64 tokens instead of one per token, and nearly all of it is matrix products.
//
// Everything is fp32 and stays so: an operand of a product is three bf16 parts (24 bits of a mantissa) and a product of two is the six part products down to
// 2^-16 of the largest, smallest first, in an fp32 accumulator that starts at zero (the update of S too: adding to S inside the tensor core would cut S off
// a little 24 times a chunk).  Decays, the inverse and all sums of products are fp32 on CUDA cores.
//
// One CTA per (sequence, head).  Warps 0 .. 3, thread = row of S^T (lane of tensor memory): S and its parts, r, parts of U, o.  Warps 4 .. 7: A and its inverse
// (blocks of 16, then two of 16 and two of 32 at a time), W.  Warps 8 .. 11: q and k to parts in shared memory, decays.  Warp 12 issues; [K; Q] K^T of the next
// chunk goes ahead of the update of S, so that the inverse is formed while the chain goes on.  Loops are rolled: with the chunk's code unrolled a
// quarter of all stalls were instruction misses.
//
// What bounds it: the chain parts of S -> X, Y -> r -> U -> parts of U -> S of a head, products and element work in turn, which nothing else on the SM
// overlaps.  8 sequences of 700..1024 tokens, 16 heads x 128 x 128: 518 us a token at a time on CUDA cores (shared-memory port and
// latency), 188 this way (20700 cycles a chunk).
#include "attn_common.cuh"

#include <atomic>

namespace {

constexpr int kL = 64, kD = 128;                   // tokens of a chunk; rows and columns of S
// four warpgroups; the registers of the launch (128 a thread) moved to where they are needed: 192 + 104 + 144 + 72 = 4 x 128
constexpr int kChunkThreads = 512, kRegsA = 192, kRegsB = 104, kRegsE = 144, kRegsC = 72;

struct ChunkParams {
  const float* u; float* o;                        // rows of u: q (G x 128) | k (G x 128) | v (H x 128) | beta (H) | g (H)
  const int* cu;
  float* s_state;                                  // [n_slots, H, 128, 128] or null
  const int* slots;
  int H, G;
  int* status;
};

// shared memory
constexpr int kPartBytes = 2 * 128 * 128;          // a part of [K; Q]: two blocks of 64 columns, 128 rows (64 tokens' k, then their q) of 128 bytes
constexpr int kK2Bytes = 2 * kL * 128;             // a part of the rows D_last,j k_j: two blocks of 64 columns, 64 rows
constexpr int kWBytes = kL * 128;                  // a part of W or T: 64 rows i, 64 columns j
constexpr int kLdA = kL + 4;                       // floats a row of A
constexpr int kSK2 = 3 * kPartBytes, kSW = kSK2 + 3 * kK2Bytes, kST = kSW + 3 * kWBytes, kSA = kST + 3 * kWBytes;
constexpr int kSCoef = kSA + kL * kLdA * 4;        // two buffers of beta, g, C, D_last [64] each
constexpr int kSBars = kSCoef + 2 * 4 * kL * 4;
constexpr int kSmemBytes = kSBars + 256 + 1024;
static_assert(kSmemBytes <= kMaxSmem, "shared memory");
// tensor memory columns.  The update of S lies over X and the first third of the parts of S, which are written from the back for that reason.
constexpr uint32_t kTS = 0, kTP = 128, kTY = 192, kTX = 256, kTParts = 320, kTR = 320, kTU = 416, kTD = 256;

enum CBar { KQ_FULL, SP_FULL, R_FULL, T_FULL, U_FULL, K2_FULL, O_READ, P_DONE, X_DONE, Y_DONE, UA_DONE, D_DONE, O_DONE, COEF_FULL, C_NUM_BARS };

RB_DEVICE float2 unpack_bf(uint32_t r) { return make_float2(__uint_as_float(r << 16), __uint_as_float(r & 0xffff0000u)); }
// part 0 .. 2 of a pair of fp32 values: their sum is the value to 24 bits
RB_DEVICE void split3(float a, float b, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
  p0 = pack2<__nv_bfloat16>(a, b);
  float2 x = unpack_bf(p0);
  a -= x.x; b -= x.y;
  p1 = pack2<__nv_bfloat16>(a, b);
  x = unpack_bf(p1);
  p2 = pack2<__nv_bfloat16>(a - x.x, b - x.y);
}
RB_DEVICE void ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
                 "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr)
               : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
RB_DEVICE void st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]),
               "r"(r[6]), "r"(r[7]), "r"(taddr)
               : "memory");
}
// 16 neighbouring columns of a row into the three parts of an operand in tensor memory
RB_DEVICE void store_parts(uint32_t taddr, uint32_t part_cols, const float (&v)[16]) {
  uint32_t part[3][8];
#pragma unroll
  for (int i = 0; i < 8; ++i) split3(v[2 * i], v[2 * i + 1], part[0][i], part[1][i], part[2][i]);
#pragma unroll
  for (int f = 0; f < 3; ++f) st8(taddr + f * part_cols, part[f]);
}

__global__ void __launch_bounds__(kChunkThreads, 1) delta_chunk_kernel(const ChunkParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t sKQ = ptx::smem_u32(smem);
  float* sA = reinterpret_cast<float*>(smem + kSA);
  float* sCoef = reinterpret_cast<float*>(smem + kSCoef);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kSBars);
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(smem + kSBars + 128);
  volatile uint32_t* dead = tmem_ptr + 1;
  auto bar = [&](int i) { return ptx::smem_u32(&bars[i]); };
  auto wait = [&](int i, int chunk) { bounded_wait(bar(i), (uint32_t)chunk & 1u, dead); };     // every barrier completes once a chunk
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int seq = blockIdx.x, h = blockIdx.y, H = p.H, G = p.G;
  const int nqk = G * kD, C = 2 * nqk + H * kD, UW = C + 2 * H;

  if (threadIdx.x == 0) {
    *dead = 0;
    for (int i = 0; i < C_NUM_BARS; ++i) ptx::mbar_init(bar(i), i <= O_READ ? 4 : 1);          // (the first ones: an arrival a warp)
    ptx::fence_barrier_init();
  }
  if (warp == 12) {
    ptx::tmem_alloc(ptx::smem_u32(tmem_ptr), 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr;
  rb::pdl_trigger();
  rb::pdl_wait();
  const int t0 = p.cu[seq], len = max(p.cu[seq + 1] - t0, 0), n_chunks = (len + kL - 1) / kL;
  auto arrive = [&](int i) {
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(bar(i));
  };

  if (warp < 4) {
    ptx::reg_inc<kRegsA>();
    // ===================================================== S, r, U, o: thread = row v of S^T
    const uint32_t tm = tmem_base + ((uint32_t)(warp * 32) << 16);
    const int v = warp * 32 + lane;
    const float* vp = p.u + (int64_t)t0 * UW + 2 * nqk + h * kD + v;
    float* op = p.o + ((int64_t)t0 * H + h) * kD + v;
    float y[kL];                                   // C_i Y_i of the chunk whose second sums are still to come
    auto write_o = [&](int c) {
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        float x[16];
        ld16(tm + kTY + b * 16, x);
        ptx::tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int tok = c * kL + b * 16 + i;
          if (tok < len) op[(int64_t)tok * H * kD] = y[b * 16 + i] + x[i];
        }
      }
      ptx::tc_fence_before();
      arrive(O_READ);
    };
    float c_last = 1.f;
    for (int c = 0; c < n_chunks; ++c) {
      const float* coef = sCoef + (c & 1) * 4 * kL;
      if (c > 0) { wait(D_DONE, c - 1); ptx::tc_fence_after(); }
#pragma unroll 1
      for (int b = 7; b >= 0; --b) {
        float s[16];
        if (c > 0) {
          float d[16];
          ld16(tm + kTS + b * 16, s);
          ld16(tm + kTD + b * 16, d);
          ptx::tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) s[i] = fmaf(c_last, s[i], d[i]);
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) s[i] = 0.f;
        }
        uint32_t raw[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) raw[i] = __float_as_uint(s[i]);
        ptx::tc_st_32x16(tm + kTS + b * 16, raw);
        if (b == 7 && c > 0) { wait(O_DONE, c - 1); ptx::tc_fence_after(); }      // the parts of U, in whose place these go, have been read
        store_parts(tm + kTParts + b * 8, 64, s);
      }
      ptx::tc_wait_st();
      ptx::tc_fence_before();
      arrive(SP_FULL);
      if (c > 0) write_o(c - 1);
      float vv[kL];
#pragma unroll
      for (int i = 0; i < kL; ++i) vv[i] = c * kL + i < len ? vp[(int64_t)(c * kL + i) * UW] : 0.f;
      wait(COEF_FULL, c);
      c_last = coef[2 * kL + kL - 1];
      wait(X_DONE, c);
      ptx::tc_fence_after();
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        float x[16], r[16];
        ld16(tm + kTX + b * 16, x);
        ptx::tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) r[i] = coef[b * 16 + i] * fmaf(-coef[2 * kL + b * 16 + i], x[i], vv[b * 16 + i]);
        if (b == 0) { wait(Y_DONE, c); ptx::tc_fence_after(); }                    // the parts of S have been read
        store_parts(tm + kTR + b * 8, 32, r);
      }
      ptx::tc_wait_st();
      ptx::tc_fence_before();
      arrive(R_FULL);
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        float x[16];
        ld16(tm + kTY + b * 16, x);
        ptx::tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) y[b * 16 + i] = coef[2 * kL + b * 16 + i] * x[i];
      }
      wait(UA_DONE, c);
      ptx::tc_fence_after();
#pragma unroll 1
      for (int b = 0; b < 4; ++b) {
        float x[16];
        ld16(tm + kTX + b * 16, x);
        ptx::tc_wait_ld();
        store_parts(tm + kTU + b * 8, 32, x);
      }
      ptx::tc_wait_st();
      ptx::tc_fence_before();
      arrive(U_FULL);
    }
    if (n_chunks > 0) {
      wait(O_DONE, n_chunks - 1);                  // (behind the update of S)
      ptx::tc_fence_after();
      write_o(n_chunks - 1);
      const int slot = p.s_state == nullptr || p.slots == nullptr ? -1 : p.slots[seq];
      if (slot >= 0) {
        float* S_g = p.s_state + (((int64_t)slot * H + h) * kD) * kD + v;
#pragma unroll 1
        for (int b = 0; b < 8; ++b) {
          float s[16], d[16];
          ld16(tm + kTS + b * 16, s);
          ld16(tm + kTD + b * 16, d);
          ptx::tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) S_g[(int64_t)(b * 16 + i) * kD] = fmaf(c_last, s[i], d[i]);
        }
      }
    }
  } else if (warp < 8) {
    ptx::reg_dec<kRegsB>();
    // ===================================================== A, its inverse, W
    const int w = warp - 4, tid = threadIdx.x - 128;
    const uint32_t tm = tmem_base + ((uint32_t)(w * 32) << 16);
    auto sync = [] { asm volatile("bar.sync 1, 128;" ::: "memory"); };
    // A's block (N rows and columns at `at`, unit lower triangular blocks of N / 2 inverted already on its diagonal): the block below the diagonal becomes
    // -T22 A21 T11.  128 threads, kCols neighbouring outputs each.
    auto join = [&](auto size, int first_of) {
      constexpr int N = decltype(size)::value, kHalf = N / 2, kCols = kHalf * kHalf * (kL / N) / 128, kPerRow = kHalf / kCols;
      const int t = tid % (kHalf * kPerRow), i = t / kPerRow, j0 = t % kPerRow * kCols;
      float* at = sA + (tid / (kHalf * kPerRow)) * N * (kLdA + 1) + first_of;
      float* low = at + kHalf * kLdA;              // A21
#pragma unroll 1
      for (int step = 0; step < 2; ++step) {       // low <- low T11, then low <- -T22 low
        const float* left = step == 0 ? low + i * kLdA : low + i * kLdA + kHalf;
        const float* right = step == 0 ? at : low;
        float a[kCols];
#pragma unroll
        for (int e = 0; e < kCols; ++e) a[e] = 0.f;
#pragma unroll 4
        for (int m = 0; m < kHalf; ++m) {
          const float x = left[m];
#pragma unroll
          for (int e = 0; e < kCols; e += 4) {
            const float4 r = *reinterpret_cast<const float4*>(right + m * kLdA + j0 + e);
            a[e] = fmaf(x, r.x, a[e]); a[e + 1] = fmaf(x, r.y, a[e + 1]); a[e + 2] = fmaf(x, r.z, a[e + 2]); a[e + 3] = fmaf(x, r.w, a[e + 3]);
          }
        }
        const float sign = step == 0 ? 1.f : -1.f;
        sync();
#pragma unroll
        for (int e = 0; e < kCols; e += 4)
          *reinterpret_cast<float4*>(low + i * kLdA + j0 + e) = make_float4(sign * a[e], sign * a[e + 1], sign * a[e + 2], sign * a[e + 3]);
        sync();
      }
    };
    for (int c = 0; c < n_chunks; ++c) {
      const float* coef = sCoef + (c & 1) * 4 * kL;
      wait(COEF_FULL, c);
      wait(P_DONE, c);                             // (T of the chunk in front has been read, too)
      ptx::tc_fence_after();
      // row i of [K; Q] K^T, from the back: lanes 0 .. 63 k_i -> A, 64 .. 127 q_i -> W
      const int i = (w & 1) * 32 + lane;
      const float beta = coef[i];
      float dec = 1.f;
#pragma unroll 1
      for (int b = 3; b >= 0; --b) {
        float x[16];
        ld16(tm + kTP + b * 16, x);
        ptx::tc_wait_ld();
#pragma unroll
        for (int e = 15; e >= 0; --e) {            // D_ij, and nothing ahead of the token
          const int j = b * 16 + e;
          dec = j < i ? dec * coef[kL + j + 1] : 1.f;
          x[e] = j <= i ? dec * x[e] : 0.f;
          if (w < 2) x[e] = j < i ? beta * x[e] : 0.f;
        }
        if (b == 3 && c > 0 && w >= 2) wait(O_DONE, c - 1);    // W of the chunk in front has been read
        if (w < 2) {
#pragma unroll
          for (int e = 0; e < 16; e += 4) *reinterpret_cast<float4*>(sA + i * kLdA + b * 16 + e) = make_float4(x[e], x[e + 1], x[e + 2], x[e + 3]);
        } else {
          uint32_t part[3][8];
#pragma unroll
          for (int e = 0; e < 8; ++e) split3(x[2 * e], x[2 * e + 1], part[0][e], part[1][e], part[2][e]);
#pragma unroll
          for (int f = 0; f < 3; ++f)
#pragma unroll
            for (int q = 0; q < 2; ++q)
              st_shared_v4(sKQ + kSW + f * kWBytes + i * 128 + (((2 * b + q) ^ (i & 7)) << 4), part[f][4 * q], part[f][4 * q + 1], part[f][4 * q + 2], part[f][4 * q + 3]);
        }
      }
      ptx::tc_fence_before();
      sync();
      // ---- T: the diagonal blocks of 16, a column a thread, then joined
      {
        float* at = sA + (tid >> 4) * 16 * (kLdA + 1);
        const int j = tid & 15;
        float x[16];
        if (tid < kL) {
#pragma unroll
          for (int n = 0; n < 16; ++n) {
            float a = n == j ? 1.f : 0.f;
#pragma unroll
            for (int m = 0; m < n; ++m) a = fmaf(-at[n * kLdA + m], x[m], a);
            x[n] = a;
          }
        }
        sync();
        if (tid < kL) {
#pragma unroll
          for (int n = 0; n < 16; ++n) at[n * kLdA + j] = x[n];
        }
        sync();
      }
      join(std::integral_constant<int, 32>(), 0);
      join(std::integral_constant<int, 64>(), 0);
      {
        const int row = tid >> 1, q0 = (tid & 1) * 4;
#pragma unroll 1
        for (int q = q0; q < q0 + 4; ++q) {
          const float4 x = *reinterpret_cast<const float4*>(sA + row * kLdA + q * 8), z = *reinterpret_cast<const float4*>(sA + row * kLdA + q * 8 + 4);
          uint32_t part[3][4];
          split3(x.x, x.y, part[0][0], part[1][0], part[2][0]);
          split3(x.z, x.w, part[0][1], part[1][1], part[2][1]);
          split3(z.x, z.y, part[0][2], part[1][2], part[2][2]);
          split3(z.z, z.w, part[0][3], part[1][3], part[2][3]);
#pragma unroll
          for (int f = 0; f < 3; ++f) st_shared_v4(sKQ + kST + f * kWBytes + row * 128 + ((q ^ (row & 7)) << 4), part[f][0], part[f][1], part[f][2], part[f][3]);
        }
      }
      ptx::fence_proxy_async();
      arrive(T_FULL);
    }
  } else if (warp < 12) {
    ptx::reg_inc<kRegsE>();
    // ===================================================== operands from the inputs
    const int w = warp - 8, g = h / (H / G);
    // Rows of 64 tokens, 16 a warp, four columns a lane: N of them on their way at once, then fours of them to parts.  `row0`: first row of the operand,
    // `scale` (null: none): a factor a token.  (The fours move up in the registers, so that the loop's code is that of four rows.)
    auto load = [&](auto& x, int c, int col, int first) {
#pragma unroll
      for (int i = 0; i < (int)(sizeof(x) / sizeof(float4)); ++i) {
        const int tok = c * kL + w * 16 + first + i;
        x[i] = tok < len ? *reinterpret_cast<const float4*>(p.u + (int64_t)(t0 + tok) * UW + col + g * kD + lane * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    auto rows = [&](auto& x, uint32_t dst, int part_bytes, int row0, int first, const float* scale) {
      constexpr int N = sizeof(x) / sizeof(float4);
      const uint32_t to = dst + (lane >> 4) * (part_bytes / 2) + (lane & 1) * 8;
#pragma unroll 1
      for (int n = 0; n < N; n += 4) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int tok = w * 16 + first + n + i, row = row0 + tok;
          const float f = scale != nullptr ? scale[tok] : 1.f;
          uint32_t part[3][2];
          split3(x[i].x * f, x[i].y * f, part[0][0], part[1][0], part[2][0]);
          split3(x[i].z * f, x[i].w * f, part[0][1], part[1][1], part[2][1]);
          const uint32_t at = to + row * 128 + ((((lane & 15) >> 1) ^ (row & 7)) << 4);
#pragma unroll
          for (int q = 0; q < 3; ++q) asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(at + q * part_bytes), "r"(part[q][0]), "r"(part[q][1]) : "memory");
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {              // around, so that x is whole again at the end
          const float4 front = x[i];
#pragma unroll
          for (int m = i; m + 4 < N; m += 4) x[m] = x[m + 4];
          x[N - 4 + i] = front;
        }
      }
    };
    // beta, g, C, D_last of chunk c into its buffer: one warp, two tokens a lane
    float beta[2], dec[2];
    auto load_coefficients = [&](int c) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int tok = c * kL + 2 * lane + e;
        const float* row = p.u + (int64_t)(t0 + tok) * UW + C + h;
        beta[e] = tok < len ? row[0] : 0.f;
        dec[e] = tok < len ? row[H] : 1.f;
      }
    };
    auto coefficients = [&](int c) {
      if (w != 0) return;
      float* coef = sCoef + (c & 1) * 4 * kL;
      float up = dec[0] * dec[1], down = up;       // products over the lanes up to this one, from this one on
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float a = __shfl_up_sync(0xffffffffu, up, o), b = __shfl_down_sync(0xffffffffu, down, o);
        if (lane >= o) up *= a;
        if (lane + o < 32) down *= b;
      }
      const float prev = __shfl_up_sync(0xffffffffu, up, 1), next = __shfl_down_sync(0xffffffffu, down, 1);
      const float in = lane == 0 ? 1.f : prev, out = lane == 31 ? 1.f : next;
      *reinterpret_cast<float2*>(coef + 2 * lane) = make_float2(beta[0], beta[1]);
      *reinterpret_cast<float2*>(coef + kL + 2 * lane) = make_float2(dec[0], dec[1]);
      *reinterpret_cast<float2*>(coef + 2 * kL + 2 * lane) = make_float2(in * dec[0], up);
      *reinterpret_cast<float2*>(coef + 3 * kL + 2 * lane) = make_float2(dec[1] * out, out);
      arrive(COEF_FULL);
    };
    float4 kx[16], qx[8];
    if (n_chunks > 0) {
      load_coefficients(0);
      load(kx, 0, nqk, 0);
      load(qx, 0, 0, 0);
    }
    for (int c = 0; c < n_chunks; ++c) {
      if (c > 0) wait(Y_DONE, c - 1);              // k and q of the chunk in front have been read
      rows(qx, sKQ, kPartBytes, kL, 0, nullptr);
      load(qx, c, 0, 8);
      rows(kx, sKQ, kPartBytes, 0, 0, nullptr);
      rows(qx, sKQ, kPartBytes, kL, 8, nullptr);
      ptx::fence_proxy_async();
      arrive(KQ_FULL);
      if (c > 0) wait(UA_DONE, c - 1);             // everybody has seen the coefficients of the chunk in front, and nobody needs those before them
      coefficients(c);
      wait(COEF_FULL, c);
      if (c > 0) wait(D_DONE, c - 1);              // the scaled k of the chunk in front has been read
      rows(kx, sKQ + kSK2, kK2Bytes, 0, 0, sCoef + (c & 1) * 4 * kL + 3 * kL);
      ptx::fence_proxy_async();
      arrive(K2_FULL);
      if (c + 1 < n_chunks) {
        load_coefficients(c + 1);
        load(kx, c + 1, nqk, 0);
        load(qx, c + 1, 0, 0);
      }
    }
  } else {
    ptx::reg_dec<kRegsC>();
    // ===================================================== MMA issue: the whole warp runs the loop, one elected lane issues
    constexpr uint32_t idesc64 = ptx::make_idesc_f16(1, 128, kL, 0, 0), idesc_s = ptx::make_idesc_f16(1, 128, kD, 0, 1);
    const uint32_t tm = (uint32_t)ptx::uniform((int)tmem_base);
    // part products, smallest first: (0, 2), (2, 0), (1, 1), (0, 1), (1, 0), (0, 0)
    auto part_a = [](int n) { return (0x010120 >> (4 * n)) & 15; };
    auto part_b = [](int n) { return (0x001102 >> (4 * n)) & 15; };
    const uint64_t kq = ptx::make_smem_desc_sw128(sKQ, 16, 1024), k2 = ptx::make_smem_desc_sw128(sKQ + kSK2, kK2Bytes / 2, 1024),
                   wd = ptx::make_smem_desc_sw128(sKQ + kSW, 16, 1024), td = ptx::make_smem_desc_sw128(sKQ + kST, 16, 1024);
    // D [128 x 64] from parts in tensor memory and 64 rows in shared memory, 64 deep
    auto product64 = [&](uint32_t d, uint32_t a, uint64_t b) {
#pragma unroll 1
      for (int n = 0; n < 6; ++n)
#pragma unroll
        for (int k = 0; k < kL / 16; ++k)
          ptx::tc_mma_f16_ts(tm + d, tm + a + part_a(n) * 32 + k * 8, b + ((part_b(n) * kWBytes + k * 32) >> 4), idesc64, n != 0 || k != 0);
    };
    auto with_s = [&](uint32_t d, int row0) {
#pragma unroll 1
      for (int n = 0; n < 6; ++n)
#pragma unroll
        for (int k = 0; k < kD / 16; ++k)
          ptx::tc_mma_f16_ts(tm + d, tm + kTParts + part_a(n) * 64 + k * 8,
                             kq + ((part_b(n) * kPartBytes + (k >> 2) * (kPartBytes / 2) + (k & 3) * 32 + row0 * 128) >> 4), idesc64, n != 0 || k != 0);
    };
    auto products_of = [&](int c) {                // [K; Q] K^T
      wait(KQ_FULL, c);
      ptx::tc_fence_after();
      if (ptx::elect_one()) {
#pragma unroll 1
        for (int n = 0; n < 6; ++n)
#pragma unroll
          for (int k = 0; k < kD / 16; ++k) {
            const uint32_t off = (k >> 2) * (kPartBytes / 2) + (k & 3) * 32;
            ptx::tc_mma_f16(tm + kTP, kq + ((part_a(n) * kPartBytes + off) >> 4), kq + ((part_b(n) * kPartBytes + off) >> 4), idesc64, n != 0 || k != 0);
          }
        ptx::tc_commit(bar(P_DONE));
      }
      __syncwarp();
    };
    for (int c = 0; warp == 12 && c < n_chunks; ++c) {
      if (c == 0) products_of(0);
      wait(SP_FULL, c);
      ptx::tc_fence_after();
      if (ptx::elect_one()) {
        with_s(kTX, 0);
        ptx::tc_commit(bar(X_DONE));
      }
      __syncwarp();
      if (c > 0) { wait(O_READ, c - 1); ptx::tc_fence_after(); }
      if (ptx::elect_one()) {
        with_s(kTY, kL);
        ptx::tc_commit(bar(Y_DONE));
      }
      __syncwarp();
      wait(R_FULL, c);
      wait(T_FULL, c);
      ptx::tc_fence_after();
      if (ptx::elect_one()) {
        product64(kTX, kTR, td);
        ptx::tc_commit(bar(UA_DONE));
      }
      __syncwarp();
      if (c + 1 < n_chunks) products_of(c + 1);
      wait(U_FULL, c);
      wait(K2_FULL, c);
      ptx::tc_fence_after();
      if (ptx::elect_one()) {
#pragma unroll 1
        for (int n = 0; n < 6; ++n)                // the update of S
#pragma unroll
          for (int k = 0; k < kL / 16; ++k)
            ptx::tc_mma_f16_ts(tm + kTD, tm + kTU + part_a(n) * 32 + k * 8, k2 + ((part_b(n) * kK2Bytes + k * 2048) >> 4), idesc_s, n != 0 || k != 0);
        ptx::tc_commit(bar(D_DONE));
        product64(kTY, kTU, wd);
        ptx::tc_commit(bar(O_DONE));
      }
      __syncwarp();
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  rb::report_given_up(dead, p.status);
  if (warp == 12) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace

// u 16-byte aligned, rows of whole float4s; head size 128 x 128, one decay per head and token (see rb_delta_rule)
extern "C" int rb_delta_chunk(const float* u, float* o, const int* cu, float* s_state, const int* slots, int n_seqs, int H, int G, cudaStream_t s) {
  static std::atomic<uint64_t> opted_in{0};          // the attribute is the kernel's on one device: a bit per device
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -3;
  if (dev >= 64 || !(opted_in.load(std::memory_order_relaxed) >> dev & 1)) {
    if (cudaFuncSetAttribute(delta_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) != cudaSuccess) return -4;
    if (dev < 64) opted_in.fetch_or(uint64_t(1) << dev, std::memory_order_relaxed);
  }
  ChunkParams p{u, o, cu, s_state, slots, H, G, rb_attn_status()};
  if (p.status == nullptr) return -5;
  return rb::launch_pdl(delta_chunk_kernel, dim3(n_seqs, H), dim3(kChunkThreads), kSmemBytes, s, p) == cudaSuccess ? 0 : -3;
}
