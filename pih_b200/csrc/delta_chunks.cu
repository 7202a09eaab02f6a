// The gated delta rule by chunks of 64 rows, in 32-bit products on the CUDA cores (the precision of the token loop).
//
// With x_t the log decays (one a key channel, or one a head), S the state in front of a chunk and L_i = x_1 + .. + x_i of the
// chunk's rows, the token loop's u_i = beta_i (v_i - k_i^T diag(g_i) S_{i-1}) are the solution of
//
//   (I + diag(beta) A) U = diag(beta) (V - K~ S),    A_ij = sum_d k_i k_j exp(L_i - L_j), j < i;    K~_i = k_i exp(L_i)
//
// so U = U0 - W S with U0 and W solved once for each chunk, and then o_i = (q_i exp(L_i))^T S + sum_{j <= i} B_ij u_j with
// B_ij = sum_d q_i k_j exp(L_i - L_j), S <- diag(exp(L_end)) S + sum_j (k_j exp(L_end - L_j)) u_j^T.
//
//   delta_chunk_prepare   A, B, W, U0 and the decayed q and k of a chunk; all chunks side by side
//   delta_chunk_states    the chunks in order, a few value columns a block: U and the state in front of each chunk
//   delta_chunk_out       the read-outs; all chunks side by side
//
// Sums of logs are kept for 16 rows at a time, and every exponent is at most zero: between rows of different 16 the factor
// is split at the borders of the 16 in between, between rows of the same 16 it is formed pair by pair.  So no product
// overflows, however fast a channel decays, and an exponent's rounding is that of a sum of 16 numbers.  The log decay is
// formed from decay - 1 (log1p) and cut off at -20: a decay below 2e-9 counts as that, less than half an ulp of one.  Logs are
// kept to the base of two.
#include "chunks.cuh"
#include "common.cuh"
#include "delta_chunks.cuh"

namespace pih {

constexpr int kSub = 16, kSubs = chunks::kRows / kSub;
constexpr float kLowestLog = -20.0f, kLog2E = 1.4426950408889634f;

// A chunk's scratch, one after the other for every (chunk, head).
template <int DIM>
struct DeltaLayout {
  long long q, k, w, b, end, u, state, size;               // decayed q; k decayed to the chunk's end; W; B; exp(L_end); U0, then U; S
  __host__ __device__ explicit DeltaLayout(int vdim) {
    q = 0;
    k = q + chunks::kRows * DIM;
    w = k + chunks::kRows * DIM;
    b = w + chunks::kRows * DIM;
    end = b + chunks::kRows * chunks::kRows;
    u = end + DIM;
    state = u + static_cast<long long>(chunks::kRows) * vdim;
    size = state + static_cast<long long>(DIM) * vdim;
  }
};

// k, q and l; the solution's first 48 rows of 256 columns later take the place of q and l and what else they need
template <int DIM>
constexpr int delta_prepare_rows() {
  constexpr int three = 3 * chunks::kRows * (DIM + 4), solved = chunks::kRows * (DIM + 4) + (chunks::kRows - kSub) * 256;
  return three > solved ? three : solved;
}
template <int DIM>
constexpr size_t delta_prepare_bytes() {
  return sizeof(float) * (delta_prepare_rows<DIM>() + kSubs * (kSubs + 1) / 2 * kSub * kSub + 6 * DIM + chunks::kRows);
}

__device__ __forceinline__ float4 exp4(float4 a, float4 b) {
  return make_float4(exp2f(a.x - b.x), exp2f(a.y - b.y), exp2f(a.z - b.z), exp2f(a.w - b.w));
}

// N neighbouring numbers (16-, 8- or 4-byte aligned as N says)
template <int N>
__device__ __forceinline__ void load_numbers(float (&x)[N], const float* from) {
#pragma unroll
  for (int i = 0; i < N; i += 4) {
    if constexpr (N >= 4) {
      const float4 f = *reinterpret_cast<const float4*>(from + i);
      x[i] = f.x; x[i + 1] = f.y; x[i + 2] = f.z; x[i + 3] = f.w;
    } else if constexpr (N == 2) {
      const float2 f = *reinterpret_cast<const float2*>(from);
      x[0] = f.x; x[1] = f.y;
    } else {
      x[0] = from[0];
    }
  }
}
template <int N>
__device__ __forceinline__ void store_numbers(float* to, const float (&x)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 4) {
    if constexpr (N >= 4) *reinterpret_cast<float4*>(to + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
    else if constexpr (N == 2) *reinterpret_cast<float2*>(to) = make_float2(x[0], x[1]);
    else to[0] = x[0];
  }
}

// Block (chunk, head), 256 threads.  Bound by shared-memory reads and exponentials, in about equal parts.
template <int DIM, bool CHANNELS>
__global__ void __launch_bounds__(256, 2)
delta_chunk_prepare_kernel(const DeltaChunkArgs p) {
  constexpr int LD = DIM + 4, R = chunks::kRows, kParts = 256 / DIM;
  extern __shared__ __align__(16) float smem[];
  float* ks = smem;                                        // [64][LD]: k; then k exp(l), l the sum of logs within the 16 rows
  float* qs = ks + R * LD;                                 // [64][LD]: q; then q exp(l)
  float* ls = qs + R * LD;                                 // [64][LD]: l; then k exp(l_end - l)
  float* as = smem + delta_prepare_rows<DIM>();            // A, its 16 x 16 blocks (i, j <= i) one after the other
  float* between = as + kSubs * (kSubs + 1) / 2 * kSub * kSub;   // [3][DIM]: decay of the 16 rows 1, of 1 and 2, of 2
  float* fronts = between + 3 * DIM;                       // [3][DIM]: decay of the rows in front of the 16 rows 1, 2, 3
  float* betas = fronts + 3 * DIM;                         // [64]
  __shared__ chunks::Place place;
  wait_for_prior_kernels();
  launch_dependents();
  const chunks::Place c = chunks::find(p.cu_q, p.state_slots, p.requests, kDeltaSmallRows, blockIdx.x, &place);
  if (c.request < 0) return;
  const int h = blockIdx.y, kh = h / (p.heads / p.kv_heads), tid = threadIdx.x;
  const DeltaLayout<DIM> at(p.vdim);
  float* mine = p.scratch + (static_cast<long long>(c.index) * p.heads + h) * at.size;
  {
    const long long from = (static_cast<long long>(c.first) * p.kv_heads + kh) * DIM, ld = static_cast<long long>(p.kv_heads) * DIM;
    chunks::load_rows<DIM, LD>(ks, p.k + from, ld, c.rows);
    chunks::load_rows<DIM, LD>(qs, p.q + from, ld, c.rows);
    chunks::copies_commit();
  }
  if (tid < R) betas[tid] = tid < c.rows ? p.beta[static_cast<long long>(c.first + tid) * p.heads + h] : 0.0f;
  const int d = tid % DIM, part = tid / DIM;
  for (int b = part; b < kSubs; b += kParts) {             // a thread a channel and 16 rows
    float x[kSub];
#pragma unroll
    for (int i = 0; i < kSub; ++i) {
      const int row = b * kSub + i;
      const long long item = static_cast<long long>(c.first + row) * p.heads + h;
      x[i] = row < c.rows ? p.decay[CHANNELS ? item * DIM + d : item] : 0.0f;
    }
    float l = 0.0f;
#pragma unroll
    for (int i = 0; i < kSub; ++i) {
      l += fmaxf(log1pf(x[i]), kLowestLog) * kLog2E;
      ls[(b * kSub + i) * LD + d] = l;
    }
  }
  chunks::copies_wait();
  __syncthreads();
  const int pi = tid >> 4, pj = tid & 15;                  // a thread a row and an earlier one of two groups of 16 rows
  float* B = mine + at.b;
  // rows of the same 16, two groups of 16 at a time: (row, earlier row) of the first by the threads below the diagonal, of the
  // second by those above it
  for (int pair = 0; pair < kSubs; pair += 2) {
    const int b = pair + (pj > pi ? 1 : 0), i = max(pi, pj), j = min(pi, pj);
    const int ri = b * kSub + i, rj = b * kSub + j;
    if (pi == pj) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int g = pair + u, row = g * kSub + pi;
        as[(g * (g + 1) / 2 + g) * kSub * kSub + pi * kSub + pi] = 0.0f;
        B[row * R + row] = row < c.rows ? p.qk[static_cast<long long>(c.first + row) * p.kv_heads + kh] : 0.0f;
      }
      continue;
    }
    const float *ki = ks + ri * LD, *kj = ks + rj * LD, *qi = qs + ri * LD, *li = ls + ri * LD, *lj = ls + rj * LD;
    float2 sa[2], sb[2];
    sa[0] = sa[1] = sb[0] = sb[1] = make_float2(0.0f, 0.0f);
#pragma unroll 2
    for (int e = 0; e < DIM; e += 4) {
      const float4 f = exp4(*reinterpret_cast<const float4*>(li + e), *reinterpret_cast<const float4*>(lj + e));
      float4 y = *reinterpret_cast<const float4*>(kj + e);
      const float4 x = *reinterpret_cast<const float4*>(ki + e), q = *reinterpret_cast<const float4*>(qi + e);
      y = make_float4(y.x * f.x, y.y * f.y, y.z * f.z, y.w * f.w);
      sa[0] = fma2(make_float2(x.x, x.y), make_float2(y.x, y.y), sa[0]);
      sa[1] = fma2(make_float2(x.z, x.w), make_float2(y.z, y.w), sa[1]);
      sb[0] = fma2(make_float2(q.x, q.y), make_float2(y.x, y.y), sb[0]);
      sb[1] = fma2(make_float2(q.z, q.w), make_float2(y.z, y.w), sb[1]);
    }
    float* a = as + (b * (b + 1) / 2 + b) * kSub * kSub;
    a[i * kSub + j] = (sa[0].x + sa[1].x) + (sa[0].y + sa[1].y);
    a[j * kSub + i] = 0.0f;
    B[ri * R + rj] = (sb[0].x + sb[1].x) + (sb[0].y + sb[1].y);
    B[rj * R + ri] = 0.0f;
  }
  float E[kSubs], before[kSubs], behind[kSubs];            // of this thread's channel: the decays of the 16 rows, before, behind
#pragma unroll
  for (int b = 0; b < kSubs; ++b) E[b] = ls[(b * kSub + kSub - 1) * LD + d];
  before[0] = 1.0f;
  before[1] = exp2f(E[0]);
  before[2] = exp2f(E[0] + E[1]);
  before[3] = exp2f(E[0] + E[1] + E[2]);
  behind[3] = 1.0f;
  behind[2] = exp2f(E[3]);
  behind[1] = exp2f(E[2] + E[3]);
  behind[0] = exp2f(E[1] + E[2] + E[3]);
  __syncthreads();
  if (part == 0) {
    between[d] = exp2f(E[1]);
    between[DIM + d] = exp2f(E[1] + E[2]);
    between[2 * DIM + d] = exp2f(E[2]);
#pragma unroll
    for (int b = 1; b < kSubs; ++b) fronts[(b - 1) * DIM + d] = before[b];
    mine[at.end + d] = exp2f(E[0] + E[1] + E[2] + E[3]);
  }
#pragma unroll
  for (int b = 0; b < kSubs; ++b) {
#pragma unroll 4
    for (int i = part; i < kSub; i += kParts) {
      const int row = b * kSub + i;
      const float l = ls[row * LD + d], k = ks[row * LD + d], f = exp2f(l);
      const float q = qs[row * LD + d] * f, kj = k * exp2f(E[b] - l);
      ks[row * LD + d] = k * f;
      qs[row * LD + d] = q;
      ls[row * LD + d] = kj;
      mine[at.q + row * DIM + d] = q * before[b];
      mine[at.k + row * DIM + d] = kj * behind[b];
    }
  }
  __syncthreads();
  for (int bi = 1; bi < kSubs; ++bi)
    for (int bj = 0; bj < bi; ++bj) {
      const float *ki = ks + (bi * kSub + pi) * LD, *qi = qs + (bi * kSub + pi) * LD, *kj = ls + (bj * kSub + pj) * LD;
      const float* w = between + (bi == 2 ? 0 : (bj == 0 ? DIM : 2 * DIM));
      const bool apart = bi - bj > 1;
      float2 sa[2], sb[2];
      sa[0] = sa[1] = sb[0] = sb[1] = make_float2(0.0f, 0.0f);
#pragma unroll 4
      for (int e = 0; e < DIM; e += 4) {
        float4 y = *reinterpret_cast<const float4*>(kj + e);
        const float4 x = *reinterpret_cast<const float4*>(ki + e), q = *reinterpret_cast<const float4*>(qi + e);
        if (apart) {
          const float4 f = *reinterpret_cast<const float4*>(w + e);
          y = make_float4(y.x * f.x, y.y * f.y, y.z * f.z, y.w * f.w);
        }
        sa[0] = fma2(make_float2(x.x, x.y), make_float2(y.x, y.y), sa[0]);
        sa[1] = fma2(make_float2(x.z, x.w), make_float2(y.z, y.w), sa[1]);
        sb[0] = fma2(make_float2(q.x, q.y), make_float2(y.x, y.y), sb[0]);
        sb[1] = fma2(make_float2(q.z, q.w), make_float2(y.z, y.w), sb[1]);
      }
      as[(bi * (bi + 1) / 2 + bj) * kSub * kSub + pi * kSub + pj] = (sa[0].x + sa[1].x) + (sa[0].y + sa[1].y);
      B[(bi * kSub + pi) * R + bj * kSub + pj] = (sb[0].x + sb[1].x) + (sb[0].y + sb[1].y);
    }
  __syncthreads();
  // a thread a column of the right-hand sides K~ | V, 16 unknowns at a time in registers, those before in shared memory
  // (where q and the decayed k lay)
  float* xs = qs + tid;                                    // [48][256]
  for (int col = tid; col < DIM + p.vdim; col += 256) {
    const bool of_k = col < DIM;
    const __nv_bfloat16* v = p.v + c.first * p.ldv + static_cast<long long>(h) * p.vdim + (col - DIM);
    float* to = of_k ? mine + at.w + col : mine + at.u + (col - DIM);
    const long long step = of_k ? DIM : p.vdim;
#pragma unroll 1
    for (int b = 0; b < kSubs; ++b) {
      float x[kSub], s[kSub];
      const float front = of_k && b > 0 ? fronts[(b - 1) * DIM + col] : 1.0f;
#pragma unroll
      for (int i = 0; i < kSub; ++i) {
        const int row = b * kSub + i;
        x[i] = of_k ? ks[row * LD + col] * front : (row < c.rows ? __bfloat162float(v[row * p.ldv]) : 0.0f);
        s[i] = 0.0f;
      }
      const float* ab = as + b * (b + 1) / 2 * kSub * kSub;
      for (int j = 0; j < b * kSub; j += 4) {
        const float x0 = xs[j * 256], x1 = xs[(j + 1) * 256], x2 = xs[(j + 2) * 256], x3 = xs[(j + 3) * 256];
        const float* aj = ab + j / kSub * kSub * kSub + j % kSub;
#pragma unroll
        for (int i = 0; i < kSub; ++i) {
          const float4 a = *reinterpret_cast<const float4*>(aj + i * kSub);
          s[i] = fmaf(a.w, x3, fmaf(a.z, x2, fmaf(a.y, x1, fmaf(a.x, x0, s[i]))));
        }
      }
      ab += b * kSub * kSub;
#pragma unroll
      for (int i = 0; i < kSub; ++i) {
        float t0 = s[i], t1 = 0.0f;
#pragma unroll
        for (int j = 0; j < i; j += 4) {
          const float4 a = *reinterpret_cast<const float4*>(ab + i * kSub + j);
          t0 = fmaf(a.x, x[j], t0);
          if (j + 1 < i) t1 = fmaf(a.y, x[j + 1], t1);
          if (j + 2 < i) t0 = fmaf(a.z, x[j + 2], t0);
          if (j + 3 < i) t1 = fmaf(a.w, x[j + 3], t1);
        }
        const int row = b * kSub + i;
        x[i] = betas[row] * (x[i] - (t0 + t1));
        to[row * step] = x[i];
        if (b + 1 < kSubs) xs[row * 256] = x[i];
      }
    }
  }
}

// Sums over LANES neighbouring lanes of N numbers each: lane i of them keeps the N / LANES from i * N / LANES on, in v[0] ...
template <int N, int LANES>
__device__ __forceinline__ void sum_and_share(float (&v)[N]) {
  const int lane = threadIdx.x & 31;
  int n = N;
#pragma unroll
  for (int m = LANES / 2; m > 0; m >>= 1) {
    n >>= 1;
    const bool upper = lane & m;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
      if (i >= n) break;
      const float mine = upper ? v[i + n] : v[i], other = upper ? v[i] : v[i + n];
      v[i] = mine + __shfl_xor_sync(0xffffffffu, other, m);
    }
  }
}

constexpr int kValues = 8;                                 // value columns a block of delta_chunk_states

template <int DIM>
constexpr size_t delta_states_bytes() {
  return sizeof(float) * (4 * chunks::kRows * (DIM + 4) + 2 * chunks::kRows * kValues + chunks::kRows * (kValues + 4) + kValues * (DIM + 4));
}

// Block (request, head, 8 value columns), 256 threads, the request's chunks in order.  A chunk's W, k and U0 are copied
// while the chunk before is computed.  Both products are cut along the sum as well — a thread 4 rows by 8 columns of a
// sixteenth (or eighth) of it, the shares met by shuffles — because a thread with whole sums of two or four outputs reads
// three 16-byte pieces for eight products (80 us for 24 chunks of 8 heads of 128 x 128, bound by those reads; 57 us now).
template <int DIM>
__global__ void __launch_bounds__(256)
delta_chunk_states_kernel(const DeltaChunkArgs p) {
  constexpr int R = chunks::kRows, LD = DIM + 4, VS = kValues, LU = VS + 4, kStage = 2 * R * LD + R * VS;
  constexpr int CU = R * VS / 256, USplit = 16;            // columns of U a thread ends with (of one row); lanes that share a sum
  constexpr int CS = DIM * VS / 256, SSplit = 32 / CS;     // the same of S (of one channel)
  static_assert(CU == 32 / USplit, "32 outputs for every group of lanes");
  extern __shared__ __align__(16) float smem[];            // [2][W [64][LD] | k [64][LD] | U0 [64][VS]]
  float* us = smem + 2 * kStage;                           // [64][LU]
  float* st = us + R * LU;                                 // [VS][LD]: S, a column after the other
  __shared__ int first;
  wait_for_prior_kernels();
  launch_dependents();
  const int r = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * VS, tid = threadIdx.x;
  const int n = p.cu_q[r + 1] - p.cu_q[r], slot = p.state_slots[r];
  if (n <= kDeltaSmallRows || slot < 0) return;
  if (tid == 0) first = chunks::first_of(p.cu_q, p.state_slots, kDeltaSmallRows, r);
  __syncthreads();
  const DeltaLayout<DIM> at(p.vdim);
  float* base = p.scratch + (static_cast<long long>(first) * p.heads + h) * at.size;
  const long long step = p.heads * at.size;
  const int count = (n + R - 1) / R;
  auto fetch = [&](int c) {
    const float* from = base + c * step;
    float* to = smem + (c & 1) * kStage;
    for (int e = tid; e < R * DIM / 4; e += 256) {
      const int row = e / (DIM / 4), col = (e % (DIM / 4)) * 4;
      chunks::copy_async_16(to + row * LD + col, from + at.w + row * DIM + col);
      chunks::copy_async_16(to + (R + row) * LD + col, from + at.k + row * DIM + col);
    }
    for (int e = tid; e < R * VS / 4; e += 256) {
      const int row = e / (VS / 4), col = (e % (VS / 4)) * 4;
      chunks::copy_async_16(to + 2 * R * LD + row * VS + col, from + at.u + static_cast<long long>(row) * p.vdim + v0 + col);
    }
    chunks::copies_commit();
  };
  // what this thread's shares of the sums end as: CS numbers of S (channel sd, columns sc ...), CU of U (row ur, columns uc ...)
  const int sd = tid / (VS / CS), sc = (tid % (VS / CS)) * CS, ur = tid / (VS / CU), uc = (tid % (VS / CU)) * CU;
  float* Sg = p.state + slot * p.state_stride + (static_cast<long long>(h) * DIM + sd) * p.vdim + v0 + sc;
  float S[CS];
#pragma unroll
  for (int i = 0; i < CS; ++i) S[i] = Sg[i];
  const int u_tile = tid / USplit * 4, u_share = tid % USplit, s_tile = tid / SSplit * 4, s_share = tid % SSplit;
  fetch(0);
  for (int c = 0; c < count; ++c) {
#pragma unroll
    for (int i = 0; i < CS; ++i) st[(sc + i) * LD + sd] = S[i];
    const float end = base[c * step + at.end + sd];
    chunks::copies_wait();
    __syncthreads();                                       // the chunk and S are there; the chunk before is done with
    if (c + 1 < count) fetch(c + 1);
    store_numbers<CS>(base + c * step + at.state + static_cast<long long>(sd) * p.vdim + v0 + sc, S);
    const float *ws = smem + (c & 1) * kStage, *ks = ws + R * LD, *u0 = ks + R * LD;
    float sums[32];
    {
      float2 part[4][VS];
      chunks::clear(part);
#pragma unroll
      for (int e = 4 * u_share; e < DIM; e += 4 * USplit) {
        float4 s[VS];
#pragma unroll
        for (int j = 0; j < VS; ++j) s[j] = *reinterpret_cast<const float4*>(st + j * LD + e);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 w = *reinterpret_cast<const float4*>(ws + (u_tile + i) * LD + e);
#pragma unroll
          for (int j = 0; j < VS; ++j) {
            part[i][j] = fma2(make_float2(w.x, w.y), make_float2(s[j].x, s[j].y), part[i][j]);
            part[i][j] = fma2(make_float2(w.z, w.w), make_float2(s[j].z, s[j].w), part[i][j]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < VS; ++j) sums[i * VS + j] = part[i][j].x + part[i][j].y;
    }
    sum_and_share<32, USplit>(sums);
    float u[CU];
    load_numbers<CU>(u, u0 + ur * VS + uc);
#pragma unroll
    for (int i = 0; i < CU; ++i) u[i] -= sums[i];
    store_numbers<CU>(us + ur * LU + uc, u);
    store_numbers<CU>(base + c * step + at.u + static_cast<long long>(ur) * p.vdim + v0 + uc, u);
    __syncthreads();
    {
      float2 part[4][VS / 2];
      chunks::clear(part);
#pragma unroll 4
      for (int j = s_share; j < R; j += SSplit) {
        const float4 k = *reinterpret_cast<const float4*>(ks + j * LD + s_tile);
        const float4 lo = *reinterpret_cast<const float4*>(us + j * LU), hi = *reinterpret_cast<const float4*>(us + j * LU + 4);
        const float kk[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 f = make_float2(kk[i], kk[i]);
          part[i][0] = fma2(f, make_float2(lo.x, lo.y), part[i][0]);
          part[i][1] = fma2(f, make_float2(lo.z, lo.w), part[i][1]);
          part[i][2] = fma2(f, make_float2(hi.x, hi.y), part[i][2]);
          part[i][3] = fma2(f, make_float2(hi.z, hi.w), part[i][3]);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < VS / 2; ++j) {
          sums[i * VS + 2 * j] = part[i][j].x;
          sums[i * VS + 2 * j + 1] = part[i][j].y;
        }
    }
    sum_and_share<32, SSplit>(sums);
#pragma unroll
    for (int i = 0; i < CS; ++i) S[i] = fmaf(end, S[i], sums[i]);
  }
#pragma unroll
  for (int i = 0; i < CS; ++i) Sg[i] = S[i];
}

template <int DIM, int VT>
constexpr size_t delta_out_bytes() {
  return sizeof(float) * chunks::kRows * (DIM + 4 + 68 + VT);
}

// Block (chunk, head, VT value columns), 256 threads: 4 rows by VT / 16 columns of the read-outs a thread.
template <int DIM, int VT>
__global__ void __launch_bounds__(256, 2)
delta_chunk_out_kernel(const DeltaChunkArgs p) {
  constexpr int LD = DIM + 4, LB = 68, R = chunks::kRows;
  extern __shared__ __align__(16) float smem[];
  float* qs = smem;                                        // [64][LD]
  float* bs = qs + R * LD;                                 // [64][LB]
  float* tile = bs + R * LB;                               // 64 rows of the state [64][VT]; then U
  __shared__ chunks::Place place;
  wait_for_prior_kernels();
  launch_dependents();
  const chunks::Place c = chunks::find(p.cu_q, p.state_slots, p.requests, kDeltaSmallRows, blockIdx.x, &place);
  if (c.request < 0) return;
  const int h = blockIdx.y, v0 = blockIdx.z * VT, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const DeltaLayout<DIM> at(p.vdim);
  const float* mine = p.scratch + (static_cast<long long>(c.index) * p.heads + h) * at.size;
  chunks::load_rows<DIM, LD>(qs, mine + at.q, DIM, R);
  chunks::load_rows<R, LB>(bs, mine + at.b, R, R);
  constexpr int RN = VT / 16;
  float2 o[4][RN / 2];
  chunks::clear(o);
#pragma unroll 1
  for (int d0 = 0; d0 < DIM; d0 += R) {
    if (d0 > 0) __syncthreads();                           // (what lay there is done with)
    chunks::load_rows<VT, VT>(tile, mine + at.state + static_cast<long long>(d0) * p.vdim + v0, p.vdim, R);
    chunks::copies_commit();
    chunks::copies_wait();
    __syncthreads();
    chunks::multiply_columns<4, RN>(o, qs + d0, LD, tile, VT, R);
  }
  __syncthreads();
  chunks::load_rows<VT, VT>(tile, mine + at.u + v0, p.vdim, R);
  chunks::copies_commit();
  chunks::copies_wait();
  __syncthreads();
  chunks::multiply_columns<4, RN>(o, bs, LB, tile, VT, (tid >> 5) * 8 + 8);        // (the warp's rows see no later ones)
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = ty * 4 + i;
    if (row >= c.rows) continue;
    float* to = p.out + (static_cast<long long>(c.first + row) * p.heads + h) * p.vdim + v0 + 4 * tx;
#pragma unroll
    for (int g = 0; g < RN / 4; ++g)
      *reinterpret_cast<float4*>(to + 64 * g) = make_float4(o[i][2 * g].x, o[i][2 * g].y, o[i][2 * g + 1].x, o[i][2 * g + 1].y);
  }
}

bool delta_takes_chunks(int heads, int dim, int vdim) {
  return (dim == 64 || dim == 128) && vdim % 64 == 0 && heads <= 65535 && vdim / 8 <= 65535;
}

long long delta_chunk_scratch(int rows, int requests, int heads, int dim, int vdim) {
  const long long each = dim == 128 ? DeltaLayout<128>(vdim).size : DeltaLayout<64>(vdim).size;
  return chunks::at_most(rows, requests, kDeltaSmallRows) * heads * each;
}

template <typename K>
static void allow_shared(K kernel, size_t bytes) {
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
}

template <int DIM>
static void launch_states(cudaStream_t s, const DeltaChunkArgs& p) {
  allow_shared(delta_chunk_states_kernel<DIM>, delta_states_bytes<DIM>());
  launch_kernel(delta_chunk_states_kernel<DIM>, dim3(p.requests, p.heads, p.vdim / kValues), dim3(256), delta_states_bytes<DIM>(), s, p);
}
template <int DIM, int VT>
static void launch_out(cudaStream_t s, const DeltaChunkArgs& p, unsigned count) {
  allow_shared(delta_chunk_out_kernel<DIM, VT>, delta_out_bytes<DIM, VT>());
  launch_kernel(delta_chunk_out_kernel<DIM, VT>, dim3(count, p.heads, p.vdim / VT), dim3(256), delta_out_bytes<DIM, VT>(), s, p);
}
template <int DIM, bool CHANNELS>
static int launch_chunks(cudaStream_t s, const DeltaChunkArgs& p, int rows) {
  const unsigned count = static_cast<unsigned>(chunks::at_most(rows, p.requests, kDeltaSmallRows));
  allow_shared(delta_chunk_prepare_kernel<DIM, CHANNELS>, delta_prepare_bytes<DIM>());
  launch_kernel(delta_chunk_prepare_kernel<DIM, CHANNELS>, dim3(count, p.heads), dim3(256), delta_prepare_bytes<DIM>(), s, p);
  PIH_LAUNCH_CHECK();
  launch_states<DIM>(s, p);
  PIH_LAUNCH_CHECK();
  if (p.vdim % 128 == 0) launch_out<DIM, 128>(s, p, count);
  else launch_out<DIM, 64>(s, p, count);
  PIH_LAUNCH_CHECK();
  return 0;
}

int launch_delta_chunks(cudaStream_t s, DeltaChunkArgs p, int dim, bool channels, int rows) {
  if (dim == 128) return channels ? launch_chunks<128, true>(s, p, rows) : launch_chunks<128, false>(s, p, rows);
  return channels ? launch_chunks<64, true>(s, p, rows) : launch_chunks<64, false>(s, p, rows);
}

}  // namespace pih
