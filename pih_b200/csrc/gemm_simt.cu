// C[M,N] = A[M,K] . W[N,K]^T on CUDA cores with 32-bit FMA accumulation.
//
// This is the matrix product of the true 32-bit path (no tensor cores, no
// TF32, no split tricks) and the plain twin of the tensor-core products.  It
// also takes bf16 inputs and writes bf16 or fp32.  Every output element is
// accumulated in an order that k alone decides — short chains into partial
// sums, the partial sums into the total, which keeps the rounding error of a
// long sum (k of a thousand and more) near that of a short one — so a row's
// result does not depend on how many other rows the call holds: cutting a
// prompt into portions or batching it with other requests cannot change a bit.
//
// The reference runs all products through a library
// (src/backend/cuda/gemm_plan.cpp:83-199: row-major A[m,k], W[n,k] with
// CUBLAS_OP_T, 32-bit compute); it has no kernel of its own for them.
#include "common.cuh"
#include "mma.cuh"

namespace pih {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename TA, typename TC>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TA* __restrict__ A, const TA* __restrict__ W, TC* __restrict__ C, int M, int N,
                 int K, long long lda, long long ldw, long long ldc, long long batch_a, long long batch_w,
                 long long batch_c) {
  wait_for_prior_kernels();
  launch_dependents();                                   // (the next kernel's blocks may become resident and wait)
  // blockIdx.z: one of several products of the same shape (a head, a diagonal block), operands apart by the strides
  A += blockIdx.z * batch_a;
  W += blockIdx.z * batch_w;
  C += blockIdx.z * batch_c;
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid % (BN / TN);        // 0..15 -> columns
  const int ty = tid / (BN / TN);        // 0..15 -> rows
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    // 64x16 elements per operand, 256 threads -> 4 each
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = tid + i * 256;
      const int r = e / BK, c = e % BK;
      const int gm = m0 + r, gn = n0 + r, gk = k0 + c;
      As[c][r] = (gm < M && gk < K) ? to_float<TA>(A[static_cast<long long>(gm) * lda + gk]) : 0.0f;
      Ws[c][r] = (gn < N && gk < K) ? to_float<TA>(W[static_cast<long long>(gn) * ldw + gk]) : 0.0f;
    }
    __syncthreads();
    float part[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) part[i][j] = 0.0f;
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[TM], w[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[k][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = Ws[k][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) part[i][j] = fmaf(a[i], w[j], part[i][j]);
    }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] += part[i][j];
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + ty * TM + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tx * TN + j;
      if (gn < N) C[static_cast<long long>(gm) * ldc + gn] = from_float<TC>(acc[i][j]);
    }
  }
}

// The 32-bit product whose rows start on 16-byte boundaries.  Bound by the FMA units with many rows and by the weights'
// bytes with few; the kernel above reached neither: a block went through all of K alone, four scalar loads and two
// barriers every 16 products, so a prompt of 200 rows (N = 1024: 64 blocks) waited for memory 64 to 192 times in a row.
//   * K is cut into S slices (slices_of_k: by K alone, so that a row's bits do not depend on the other rows), a block of
//     a cluster each; the slices' sums meet in the blocks' shared memory, in the order of the slices.
//   * Operands come by asynchronous copies, kStages - 1 tiles of 32 products ahead, and stay as they lie in memory, k
//     innermost: a 16-byte read of an operand is two pairs of neighbouring k for the two-number FMA.  Rows of 36 words
//     put the 16-byte reads of eight neighbouring rows into different banks.
//   * An output's even and odd products of a tile run in two chains of 16, whose sum joins the slice's: closer to the exact
//     sum than the 16 products and K / 16 partial sums above for short and long k alike.  (Chains of 32 were no
//     faster, and further off for k of a hundred.)
// Tiles of 8 x 64 for at most 8 rows, 32 x 64 up to 32, 64 x 64 beyond: a wider tile would only add rows of padding.
constexpr int kTileK = 32, kTileLd = kTileK + 4, kTileN = 64, kTileThreads = 128;

static int slices_of_k(int K) { return K >= 2048 ? 8 : (K >= 1024 ? 4 : (K >= 512 ? 2 : 1)); }

template <int ROWS, int STAGES>
constexpr size_t tile_bytes() {
  return sizeof(float) * static_cast<size_t>(STAGES) * (ROWS + kTileN) * kTileLd;
}

// ROWS rows of A by 64 rows of W; thread (ty, tx): rows ty * TM .. + TM - 1, columns tx + 16 j.
template <int ROWS, int STAGES>
__global__ void __launch_bounds__(kTileThreads)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                     int slices, int slice_k, long long lda, long long ldw, long long ldc, long long batch_a,
                     long long batch_w, long long batch_c) {
  constexpr int TM = ROWS / 8, TN = 4, kRowsTile = ROWS + kTileN;
  extern __shared__ __align__(16) float tile_smem[];        // [STAGES][ROWS + 64][36]: A's rows, then W's
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int slice = blockIdx.x % slices, n0 = (blockIdx.x / slices) * kTileN, m0 = blockIdx.y * ROWS;
  A += blockIdx.z * batch_a;
  W += blockIdx.z * batch_w;
  C += blockIdx.z * batch_c;
  const int k_lo = slice * slice_k, k_hi = min(K, k_lo + slice_k);
  const int tiles = k_hi > k_lo ? (k_hi - k_lo + kTileK - 1) / kTileK : 0;
  auto fetch = [&](int t, bool weights, bool rows) {
    float* dst = tile_smem + (t % STAGES) * kRowsTile * kTileLd;
    const int piece = (tid & 7) * 4, k = k_lo + t * kTileK + piece;
#pragma unroll
    for (int r = tid >> 3; r < kRowsTile; r += kTileThreads / 8) {
      const bool of_a = r < ROWS;
      if (of_a ? !rows : !weights) continue;
      const int g = of_a ? m0 + r : n0 + r - ROWS;
      const bool there = k < k_hi && g < (of_a ? M : N);
      const float* src = of_a ? A + (there ? g * lda + k : 0) : W + (there ? g * ldw + k : 0);
      mma::copy_async_16_or_zero(dst + r * kTileLd + piece, src, there);
    }
  };
  // the weights are written by no kernel: their first tiles are on the way while the kernel before this one ends
#pragma unroll
  for (int t = 0; t < STAGES - 1; ++t)
    if (t < tiles) fetch(t, true, false);
  wait_for_prior_kernels();
#pragma unroll
  for (int t = 0; t < STAGES - 1; ++t) {
    if (t < tiles) fetch(t, false, true);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  float acc[TM][TN];
  float2 part[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      acc[i][j] = 0.0f;
      part[i][j] = make_float2(0.0f, 0.0f);
    }
  for (int t = 0; t < tiles; ++t) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                                       // tile t is there; tile t - 1's place is free
    if (t + STAGES - 1 < tiles) fetch(t + STAGES - 1, true, true);
    else if (t + STAGES - 1 == tiles) launch_dependents();
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* a_at = tile_smem + (t % STAGES) * kRowsTile * kTileLd + ty * TM * kTileLd;
    const float* w_at = tile_smem + ((t % STAGES) * kRowsTile + ROWS + tx) * kTileLd;
#pragma unroll
    for (int k = 0; k < kTileK; k += 4) {
      float4 w[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(w_at + 16 * j * kTileLd + k);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(a_at + i * kTileLd + k);
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          part[i][j] = fma2(make_float2(a.x, a.y), make_float2(w[j].x, w[j].y), part[i][j]);
          part[i][j] = fma2(make_float2(a.z, a.w), make_float2(w[j].z, w[j].w), part[i][j]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        acc[i][j] += part[i][j].x + part[i][j].y;
        part[i][j] = make_float2(0.0f, 0.0f);
      }
  }
  if (slices == 1) {
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int gm = m0 + ty * TM + i;
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const int gn = n0 + tx + 16 * j;
        if (gm < M && gn < N) C[gm * ldc + gn] = acc[i][j];
      }
    }
    return;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* sums = tile_smem;                                 // [ROWS][64]
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) sums[(ty * TM + i) * kTileN + tx + 16 * j] = acc[i][j];
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const uint32_t local = static_cast<uint32_t>(__cvta_generic_to_shared(sums));
  const int share = ROWS * kTileN / slices;                // this block's outputs of the tile
  for (int e = slice * share + tid; e < (slice + 1) * share; e += kTileThreads) {
    float v[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      v[s] = 0.0f;
      if (s < slices) {
        uint32_t remote;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local + 4u * e), "r"(s));
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[s]) : "r"(remote) : "memory");
      }
    }
    float total = v[0];
#pragma unroll
    for (int s = 1; s < 8; ++s)
      if (s < slices) total += v[s];
    const int gm = m0 + e / kTileN, gn = n0 + e % kTileN;
    if (gm < M && gn < N) C[gm * ldc + gn] = total;
  }
  // nobody leaves while another block may still read its sums
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

}  // namespace pih

using namespace pih;

template <int ROWS, int STAGES>
static void launch_f32_tiles(cudaStream_t s, const float* A, const float* W, float* C, int M, int N, int K, long long lda,
                             long long ldw, long long ldc, int batches, long long batch_a, long long batch_w,
                             long long batch_c) {
  const int slices = slices_of_k(K), slice_k = ((K + slices - 1) / slices + kTileK - 1) / kTileK * kTileK;
  constexpr size_t bytes = tile_bytes<ROWS, STAGES>();
  static_assert(bytes >= sizeof(float) * ROWS * kTileN, "the sums take the tiles' place");
  cudaFuncSetAttribute(gemm_f32_tile_kernel<ROWS, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  launch_kernel_clustered(gemm_f32_tile_kernel<ROWS, STAGES>, dim3((N + kTileN - 1) / kTileN * slices, (M + ROWS - 1) / ROWS, batches),
                          dim3(kTileThreads), bytes, s, static_cast<unsigned>(slices), A, W, C, M, N, K, slices, slice_k, lda,
                          ldw, ldc, batch_a, batch_w, batch_c);
}

// ``batches`` products C_b[M,N] = A_b[M,K] . W_b[N,K]^T in one launch: operand b starts ``batch_*`` elements behind
// operand b-1 (rows of A_b may interleave with those of other batches: lda is free).  The same kernel, hence the same
// rounding, as the single product.
extern "C" int pih_gemm_simt_batched(int in_dtype, int out_dtype, const void* A, const void* W, void* C, int M,
                                     int N, int K, long long lda, long long ldw, long long ldc, int batches,
                                     long long batch_a, long long batch_w, long long batch_c, void* stream) {
  if (M <= 0 || N <= 0 || batches <= 0) return 0;
  if (K <= 0) return PIH_ERR_BAD_ARGUMENT;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batches);
  if (grid.y > 65535 || grid.z > 65535) return PIH_ERR_UNSUPPORTED;
  // whole 16-byte pieces of every row of both operands (views of other widths or offsets: the kernel above)
  const bool pieces = reinterpret_cast<uintptr_t>(A) % 16 == 0 && reinterpret_cast<uintptr_t>(W) % 16 == 0 && K % 4 == 0 &&
                      lda % 4 == 0 && ldw % 4 == 0 && batch_a % 4 == 0 && batch_w % 4 == 0;
  if (in_dtype == PIH_F32 && out_dtype == PIH_F32 && pieces) {
    const float *a = static_cast<const float*>(A), *w = static_cast<const float*>(W);
    float* c = static_cast<float*>(C);
    if (M <= 8) launch_f32_tiles<8, 4>(s, a, w, c, M, N, K, lda, ldw, ldc, batches, batch_a, batch_w, batch_c);
    else if (M <= 32) launch_f32_tiles<32, 3>(s, a, w, c, M, N, K, lda, ldw, ldc, batches, batch_a, batch_w, batch_c);
    else launch_f32_tiles<64, 3>(s, a, w, c, M, N, K, lda, ldw, ldc, batches, batch_a, batch_w, batch_c);
  } else if (in_dtype == PIH_F32 && out_dtype == PIH_F32)
    launch_kernel(gemm_simt_kernel<float, float>, dim3(grid), dim3(256), 0, s, static_cast<const float*>(A),
                                                        static_cast<const float*>(W),
                                                        static_cast<float*>(C), M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c);
  else if (in_dtype == PIH_BF16 && out_dtype == PIH_BF16)
    launch_kernel(gemm_simt_kernel<__nv_bfloat16, __nv_bfloat16>, dim3(grid), dim3(256), 0, s, 
        static_cast<const __nv_bfloat16*>(A), static_cast<const __nv_bfloat16*>(W),
        static_cast<__nv_bfloat16*>(C), M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c);
  else if (in_dtype == PIH_BF16 && out_dtype == PIH_F32)
    launch_kernel(gemm_simt_kernel<__nv_bfloat16, float>, dim3(grid), dim3(256), 0, s, 
        static_cast<const __nv_bfloat16*>(A), static_cast<const __nv_bfloat16*>(W),
        static_cast<float*>(C), M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c);
  else
    return PIH_ERR_BAD_ARGUMENT;
  PIH_LAUNCH_CHECK();
  return 0;
}

extern "C" int pih_gemm_simt(int in_dtype, int out_dtype, const void* A, const void* W, void* C, int M,
                             int N, int K, long long lda, long long ldw, long long ldc, void* stream) {
  return pih_gemm_simt_batched(in_dtype, out_dtype, A, W, C, M, N, K, lda, ldw, ldc, 1, 0, 0, 0, stream);
}
