// Pieces shared by the tcgen05 GEMM translation units (tile kernel, small-M stream-K kernel, 2-CTA kernel).
#pragma once
#include <cuda.h>
#include <stdio.h>
#include <stdlib.h>

#include "common.cuh"
#include "ptx.cuh"

namespace {

constexpr int BM = 128;
constexpr int BK = 64;  // 64 bf16 = 128 bytes = one swizzle row
constexpr int kThreads = 192;

struct Params {
  void* C;
  const void* bias;
  int64_t ldc;
  int M, N, K;
  int accumulate;  // C += result
  // optional gating of A row-blocks on arrival flags (all-gather -> GEMM: a copy stream fills A chunk by chunk and bumps
  // flag[row / rows_per_flag] to `ready_epoch`); m_rot rotates the m-tile order so the rows that are already local go first
  const uint32_t* ready_flags;
  uint32_t ready_epoch;
  int rows_per_flag;
  int m_rot;
  // optional completion counters (GEMM -> reduce-scatter): every epilogue warp bumps done[row / rows_per_flag] once its 32
  // rows x BN columns of a tile are stored, so a copy stream can ship finished row-blocks while later tiles still compute
  uint32_t* done_counters;
  // optional gated-linear-unit epilogue (2-CTA kernel): B is the fused [gate; up] weight with glu_F rows each, N = glu_F output
  // columns act(gate) * up are written to C, and (when glu_raw != nullptr) the raw gate | up projections to glu_raw [M, 2 glu_F]
  int glu_F;
  int glu_act;       // 0 silu, 1 gelu (tanh approximation), 2 clamped: min(g, L) * sigmoid(alpha min(g, L)) * (clamp(u, -L, L) + 1)
  void* glu_raw;
  int64_t ld_raw;
  float glu_limit;   // L and alpha of the clamped form
  float glu_alpha;
  // optional unary activation on the plain (non-GLU) epilogue of the 2-CTA kernel, after the bias: 0 none, 1 relu(x)^2
  int unary_act;
  int act_cols;            // unary_act applies to output columns below this
};

template <typename T> RB_DEVICE void store_chunk(T* dst, const float* v, int n_valid, bool vec_ok);

template <> RB_DEVICE void store_chunk<float>(float* dst, const float* v, int n_valid, bool vec_ok) {
  if (n_valid == 32 && vec_ok) {
#pragma unroll
    for (int i = 0; i < 8; ++i) reinterpret_cast<float4*>(dst)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
  } else {
    for (int i = 0; i < n_valid; ++i) dst[i] = v[i];
  }
}
template <typename T> RB_DEVICE void store_chunk(T* dst, const float* v, int n_valid, bool vec_ok) {
  if (n_valid == 32 && vec_ok) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      rb::Pack<T, 8> p;
#pragma unroll
      for (int k = 0; k < 8; ++k) p.v[k] = rb::from_f<T>(v[8 * i + k]);
      reinterpret_cast<rb::Pack<T, 8>*>(dst)[i] = p;
    }
  } else {
    for (int i = 0; i < n_valid; ++i) dst[i] = rb::from_f<T>(v[i]);
  }
}

// 32 accumulator columns of a warp's 32 rows (lane = row) to memory, through 4 KB of shared memory of the warp at `stage` (1 KB aligned): a lane holds a
// row, so storing from it writes 32 lines per instruction in 16-byte pieces, and adding to the old value fetched those one element at a time.  Staged as
// fp32, four lines per instruction leave whole, and the old values of an accumulating GEMM come in the same way; the sum is formed in fp32.
// dst: first row and column; rows / cols: how many are real.
template <typename T> RB_DEVICE void store_rows32(uint32_t stage, const float (&v)[32], T* dst, int64_t ldc, int rows, int cols, bool vec_ok, bool accumulate) {
  const int lane = threadIdx.x & 31, q = lane & 7, c = q * 4;
  rb::Pack<T, 4> old[8];
  const bool fetch = accumulate && vec_ok && c + 4 <= cols;
  if (fetch) {                       // all eight in flight while the new values are staged
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = i * 4 + (lane >> 3);
      if (r < rows) old[i] = *reinterpret_cast<const rb::Pack<T, 4>*>(dst + (int64_t)r * ldc + c);
    }
  }
#pragma unroll
  for (int q = 0; q < 8; ++q)
    asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(stage + lane * 128 + ((q ^ (lane & 7)) << 4)), "f"(v[4 * q]), "f"(v[4 * q + 1]), "f"(v[4 * q + 2]),
                 "f"(v[4 * q + 3])
                 : "memory");
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = i * 4 + (lane >> 3);
    float x[4];
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]) : "r"(stage + r * 128 + ((q ^ (r & 7)) << 4)) : "memory");
    if (r < rows && c < cols) {
      T* d = dst + (int64_t)r * ldc + c;
      if (vec_ok && c + 4 <= cols) {
        rb::Pack<T, 4> o;
        if (fetch) {
#pragma unroll
          for (int k = 0; k < 4; ++k) x[k] += rb::to_f(old[i].v[k]);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) o.v[k] = rb::from_f<T>(x[k]);
        *reinterpret_cast<rb::Pack<T, 4>*>(d) = o;
      } else {
        for (int k = 0; k < 4 && c + k < cols; ++k) d[k] = rb::from_f<T>(accumulate ? x[k] + rb::to_f(d[k]) : x[k]);
      }
    }
  }
  __syncwarp();
}

// The same for 64 columns of 16-bit results that are all real, aligned and not added to anything: staged in their own type, eight 16-byte loads and
// stores a lane.
template <typename T> RB_DEVICE void store_rows64(uint32_t stage, const uint32_t (&acc)[64], T* dst, int64_t ldc) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    rb::Pack<T, 8> o;
#pragma unroll
    for (int e = 0; e < 8; ++e) o.v[e] = rb::from_f<T>(__uint_as_float(acc[q * 8 + e]));
    const uint4 w = *reinterpret_cast<const uint4*>(&o);
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(stage + lane * 128 + ((q ^ (lane & 7)) << 4)), "r"(w.x), "r"(w.y), "r"(w.z), "r"(w.w) : "memory");
  }
  __syncwarp();
  uint4 y[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = i * 4 + (lane >> 3);
    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(y[i].x), "=r"(y[i].y), "=r"(y[i].z), "=r"(y[i].w) : "r"(stage + r * 128 + (((lane & 7) ^ (r & 7)) << 4)) : "memory");
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4*>(dst + (int64_t)(i * 4 + (lane >> 3)) * ldc + (lane & 7) * 8) = y[i];
  __syncwarp();
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || p == nullptr) return nullptr;
    fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// 2-D row-major tensor [rows, cols] (cols contiguous, row pitch `ld` elements), 2-byte elements, 128B swizzle.
bool make_tmap(CUtensorMap* m, const void* ptr, int is_bf16, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_cols,
               uint32_t box_rows) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return false;
  // The driver entry point needs a current context in *this* thread; autograd's backward threads only ever
  // called cudaSetDevice, which does not bind the primary context for driver-API calls until a runtime call does.
  static thread_local bool ctx_ready = false;
  if (!ctx_ready) { cudaFree(nullptr); ctx_ready = true; }
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(ptr), dims,
                  strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    fprintf(stderr, "[rb_gemm] cuTensorMapEncodeTiled failed: %d ptr=%p rows=%llu cols=%llu ld=%llu box=(%u,%u)\n", (int)r, ptr,
            (unsigned long long)rows, (unsigned long long)cols, (unsigned long long)ld, box_cols, box_rows);
  }
  return r == CUDA_SUCCESS;
}


// 2-D row-major tensor of BYTES [rows, cols] (fp8 operands), 128B swizzle: a box row is 128 elements = one swizzle row.
bool make_tmap_u8(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_cols, uint32_t box_rows) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return false;
  static thread_local bool ctx_ready = false;
  if (!ctx_ready) { cudaFree(nullptr); ctx_ready = true; }
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) fprintf(stderr, "[rb_gemm] cuTensorMapEncodeTiled(u8) failed: %d rows=%llu cols=%llu ld=%llu\n", (int)r,
                                 (unsigned long long)rows, (unsigned long long)cols, (unsigned long long)ld);
  return r == CUDA_SUCCESS;
}

}  // namespace
