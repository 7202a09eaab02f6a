// Chunks of 64 rows of the requests of a step, for recurrences that take a long request's rows chunk by chunk.
#pragma once

#include "common.cuh"
#include "mma.cuh"

namespace pih {
namespace chunks {

constexpr int kRows = 64;

struct Place { int request, first, rows; };                  // rows first .. first + rows - 1 of the step

// The x-th chunk of the step's requests that have more than small_rows rows (request -1: there is none); for every thread
// of the block.
__device__ __forceinline__ Place find(const int* cu_q, const int* state_slots, int requests, int small_rows, int x, Place* shared) {
  if (threadIdx.x == 0) {
    Place c = {-1, 0, 0};
    int t = x;
    for (int r = 0; r < requests; ++r) {
      const int lo = cu_q[r], n = cu_q[r + 1] - lo;
      if (n <= small_rows || state_slots[r] < 0) continue;
      const int chunks = (n + kRows - 1) / kRows;
      if (t < chunks) {
        c.request = r;
        c.first = lo + t * kRows;
        c.rows = min(kRows, n - t * kRows);
        break;
      }
      t -= chunks;
    }
    *shared = c;
  }
  __syncthreads();
  return *shared;
}

// The index of request r's first chunk.
__device__ __forceinline__ int first_of(const int* cu_q, const int* state_slots, int small_rows, int r) {
  int at = 0;
  for (int o = 0; o < r; ++o) {
    const int n = cu_q[o + 1] - cu_q[o];
    if (n > small_rows && state_slots[o] >= 0) at += (n + kRows - 1) / kRows;
  }
  return at;
}

// The most chunks that a step of `rows` rows can have: every request of more than small_rows rows may end in a part.
inline long long at_most(long long rows, int requests, int small_rows) {
  const long long ends = rows / (small_rows + 1);
  return rows / kRows + (ends < requests ? ends : requests);
}

// `rows` rows of COLS 32-bit numbers (row stride ld) into shared memory [64][LD] by copies (not waited for), zeros beyond.
template <int COLS, int LD>
__device__ __forceinline__ void load_rows(float* dst, const float* src, long long ld, int rows) {
  for (int e = threadIdx.x; e < kRows * (COLS / 4); e += blockDim.x) {
    const int row = e / (COLS / 4), c = (e % (COLS / 4)) * 4;
    if (row < rows) mma::copy_async_16(dst + row * LD + c, src + row * ld + c);
    else *reinterpret_cast<float4*>(dst + row * LD + c) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
}

// The same from bf16, widened on the way (done when the function returns).  Says whether one of this thread's numbers is
// infinite or none.
template <int COLS, int LD>
__device__ __forceinline__ bool load_rows(float* dst, const __nv_bfloat16* src, long long ld, int rows) {
  bool wild = false;
  for (int e = threadIdx.x; e < kRows * (COLS / 8); e += blockDim.x) {
    const int row = e / (COLS / 8), c = (e % (COLS / 8)) * 8;
    const uint4 x = row < rows ? *reinterpret_cast<const uint4*>(src + row * ld + c) : make_uint4(0u, 0u, 0u, 0u);
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
    float f[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[2 * i] = __uint_as_float(w[i] << 16);
      f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
      wild = wild || (w[i] & 0x7f80u) == 0x7f80u || (w[i] & 0x7f800000u) == 0x7f800000u;
    }
    *reinterpret_cast<float4*>(dst + row * LD + c) = make_float4(f[0], f[1], f[2], f[3]);
    *reinterpret_cast<float4*>(dst + row * LD + c + 4) = make_float4(f[4], f[5], f[6], f[7]);
  }
  return wild;
}

// Products of 32-bit numbers in shared memory by 256 threads, (ty, tx) = (thread / 16, thread % 16): rows ty * RM + i.
// acc[i][j] (columns tx + 16 j) += sum over k < K of a[row][k] b[column][k]; both rows of LD = K + 4 words.
template <int RM, int RN, int K, int LD>
__device__ __forceinline__ void multiply_rows(float2 (&acc)[RM][RN], const float* a, const float* b) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll 4
  for (int k = 0; k < K; k += 4) {
    float4 y[RN];
#pragma unroll
    for (int j = 0; j < RN; ++j) y[j] = *reinterpret_cast<const float4*>(b + (tx + 16 * j) * LD + k);
#pragma unroll
    for (int i = 0; i < RM; ++i) {
      const float4 x = *reinterpret_cast<const float4*>(a + (ty * RM + i) * LD + k);
#pragma unroll
      for (int j = 0; j < RN; ++j) {
        acc[i][j] = fma2(make_float2(x.x, x.y), make_float2(y[j].x, y[j].y), acc[i][j]);
        acc[i][j] = fma2(make_float2(x.z, x.w), make_float2(y[j].z, y[j].w), acc[i][j]);
      }
    }
  }
}

template <int R, int C>
__device__ __forceinline__ void clear(float2 (&acc)[R][C]) {
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < C; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
}

// acc[i][2 g + u] (columns 64 g + 4 tx + 2 u, + 1) += sum over k < K (a multiple of 4) of a[row][k] b[k][column].  Chains of
// 16 products, whose sums are added up: the rounding error is that of 16 + K / 16 additions, not of K.  TRIANGLE: without the
// products of k > row, whose a is zero: the same sums, but what b holds there may be anything.
template <int RM, int RN, bool TRIANGLE = false>
__device__ __forceinline__ void multiply_columns(float2 (&acc)[RM][RN / 2], const float* a, int lda, const float* b, int ldb, int K) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll 1
  for (int k0 = 0; k0 < K; k0 += 16) {
    float2 part[RM][RN / 2];
    clear(part);
    const int end = min(K, k0 + 16);
#pragma unroll 1
    for (int k = k0; k < end; k += 4) {
      float4 y[4][RN / 4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int g = 0; g < RN / 4; ++g) y[u][g] = *reinterpret_cast<const float4*>(b + (k + u) * ldb + 64 * g + 4 * tx);
#pragma unroll
      for (int i = 0; i < RM; ++i) {
        const float4 x = *reinterpret_cast<const float4*>(a + (ty * RM + i) * lda + k);
        const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int g = 0; g < RN / 4; ++g) {
            if (TRIANGLE && k + u > ty * RM + i) continue;
            const float2 xx = make_float2(xs[u], xs[u]);
            part[i][2 * g] = fma2(xx, make_float2(y[u][g].x, y[u][g].y), part[i][2 * g]);
            part[i][2 * g + 1] = fma2(xx, make_float2(y[u][g].z, y[u][g].w), part[i][2 * g + 1]);
          }
      }
    }
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
      for (int j = 0; j < RN / 2; ++j) {
        acc[i][j].x += part[i][j].x;
        acc[i][j].y += part[i][j].y;
      }
  }
}

// acc[i][2 g + u] (rows ty * RM + i, columns as above) += sum over k < K of a[k][row] b[k][column].
template <int RM, int RN>
__device__ __forceinline__ void multiply_outer(float2 (&acc)[RM][RN / 2], const float* a, int lda, const float* b, int ldb, int K) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll 4
  for (int k = 0; k < K; ++k) {
    float4 y[RN / 4], x[RM / 4];
#pragma unroll
    for (int g = 0; g < RN / 4; ++g) y[g] = *reinterpret_cast<const float4*>(b + k * ldb + 64 * g + 4 * tx);
#pragma unroll
    for (int g = 0; g < RM / 4; ++g) x[g] = *reinterpret_cast<const float4*>(a + k * lda + ty * RM + 4 * g);
#pragma unroll
    for (int i = 0; i < RM; ++i) {
      const float4 q = x[i / 4];
      const float f = (i & 3) == 0 ? q.x : ((i & 3) == 1 ? q.y : ((i & 3) == 2 ? q.z : q.w));
      const float2 xx = make_float2(f, f);
#pragma unroll
      for (int g = 0; g < RN / 4; ++g) {
        acc[i][2 * g] = fma2(xx, make_float2(y[g].x, y[g].y), acc[i][2 * g]);
        acc[i][2 * g + 1] = fma2(xx, make_float2(y[g].z, y[g].w), acc[i][2 * g + 1]);
      }
    }
  }
}

}  // namespace chunks
}  // namespace pih
