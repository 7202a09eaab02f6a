// Retention: linear attention with a fixed decay a head and a matrix state per (request, head).
//
//   retention_prepare      q and k of every row rotated by the row's position (angles formed in 32-bit from the
//                          frequencies), k then scaled: 32-bit copies [rows, heads, dim]
//   retention_recurrence   per token  S <- S + (decay - 1) S + k v^T,  o = S^T q,  from the request's state slot; S in
//                          shared memory (any key size), or in registers for the key sizes that have an instance
//
// The order of the additions of a read-out is fixed by the kernel and by what its request brings to the step: it does not
// depend on what else the step holds, and with the token loop (32-bit, and bf16 requests of up to ``small_rows`` rows)
// not on how a sequence is cut into steps either.
//
// bf16 requests of more than ``small_rows`` rows go by chunks of 64 rows instead, all chunks side by side, in 32-bit
// products on the CUDA cores (closer to the exact sums than the token loop, which is a chain of 0.27 us a token on 32 of
// the 148 SMs for 8 heads of 128 x 128):
//   retention_chunk_state   U = sum_j decay^(end - j) k_j v_j^T, what a chunk adds to the state
//   retention_state_pass    the chunks in order: the state in front of each takes U's place; S <- decay^rows S + U
//   retention_chunk_out     o_i = decay^(i + 1) S^T q_i + sum_{j <= i} decay^(i - j) (q_i . k_j) v_j
// decay^n is formed as exp(n log1p(decay - 1)).  Steps whose chunks do not fit the scratch go in waves of as many as do, the
// state in the slot in between.
#include "chunks.cuh"
#include "common.cuh"

namespace pih {

// A thread an element of q and of k.  Rotate-half over the first ``rot`` columns: column i < rot / 2 pairs with
// i + rot / 2; (u, v) -> (u cos a - v sin a, v cos a + u sin a), a = position * freq[i].
template <typename T>
__global__ void __launch_bounds__(256)
retention_prepare_kernel(const T* __restrict__ qk, long long ld, const float* __restrict__ freq,
                         const int* __restrict__ positions, float* __restrict__ qf, float* __restrict__ kf, int rows,
                         int heads, int dim, int rot, float key_scale) {
  wait_for_prior_kernels();
  launch_dependents();
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const long long per_row = static_cast<long long>(heads) * dim;
  if (i >= rows * per_row) return;
  const int row = static_cast<int>(i / per_row);
  const int e = static_cast<int>(i % dim);
  const long long head_at = (i - static_cast<long long>(row) * per_row) - e;        // head * dim
  const T* q = qk + row * ld + head_at;
  const T* k = q + per_row;
  float qo, ko;
  const int half = rot >> 1;
  if (e < rot) {
    const int pair = e < half ? e : e - half;
    float sn, cs;
    sincosf(static_cast<float>(positions[row]) * freq[pair], &sn, &cs);
    const float qu = to_float<T>(q[pair]), qv = to_float<T>(q[pair + half]);
    const float ku = to_float<T>(k[pair]), kv = to_float<T>(k[pair + half]);
    if (e < half) {
      qo = qu * cs - qv * sn;
      ko = ku * cs - kv * sn;
    } else {
      qo = qv * cs + qu * sn;
      ko = kv * cs + ku * sn;
    }
  } else {
    qo = to_float<T>(q[e]);
    ko = to_float<T>(k[e]);
  }
  qf[i] = qo;
  kf[i] = ko * key_scale;
}

// Block (request, head, slab of value columns); thread j owns column v0 + j of S (all ``dim`` rows, in shared memory:
// S[i][j]).  The next token's k and q are fetched into registers while this token is computed.  Any dim.
template <typename T>
__global__ void retention_recurrence_kernel(const float* __restrict__ qf, const float* __restrict__ kf,
                                            const T* __restrict__ v, long long ldv, const float* __restrict__ decay_m1,
                                            float* __restrict__ out, float* __restrict__ state, long long state_stride,
                                            const int* __restrict__ cu_q, const int* __restrict__ state_slots, int heads,
                                            int dim, int vdim, int small_rows) {
  extern __shared__ float smem[];
  wait_for_prior_kernels();
  launch_dependents();
  const int r = blockIdx.x, h = blockIdx.y;
  const int cols = blockDim.x;
  const int j = threadIdx.x, col = blockIdx.z * cols + j;
  const int lo = cu_q[r], hi = cu_q[r + 1];
  const int slot = state_slots[r];
  if (hi <= lo || slot < 0 || hi - lo > small_rows) return;
  float* S = smem;                          // [dim][cols]
  float* kq = smem + dim * cols;            // [2 buffers][k: dim | q: dim]
  const bool live = col < vdim;
  float* Sg = state + slot * state_stride + (static_cast<long long>(h) * dim) * vdim;
  for (int i = 0; i < dim; ++i) S[i * cols + j] = live ? Sg[static_cast<long long>(i) * vdim + col] : 0.0f;
  const float dm1 = decay_m1[h];
  const int per = (2 * dim + cols - 1) / cols;                   // numbers of k|q a thread fetches
  auto fetch = [&](int t, int e) -> float {
    const int idx = j + e * cols;
    if (idx >= 2 * dim) return 0.0f;
    const float* src = idx < dim ? kf : qf;
    return src[(static_cast<long long>(t) * heads + h) * dim + (idx < dim ? idx : idx - dim)];
  };
  constexpr int kMaxPer = 32;               // dim <= 16 * cols
  float nxt[kMaxPer];
#pragma unroll
  for (int e = 0; e < kMaxPer; ++e) nxt[e] = e < per ? fetch(lo, e) : 0.0f;
  for (int t = lo; t < hi; ++t) {
    float* cur = kq + (t & 1) * 2 * dim;
#pragma unroll
    for (int e = 0; e < kMaxPer; ++e)
      if (e < per && j + e * cols < 2 * dim) cur[j + e * cols] = nxt[e];
    __syncthreads();
    if (t + 1 < hi) {
#pragma unroll
      for (int e = 0; e < kMaxPer; ++e) nxt[e] = e < per ? fetch(t + 1, e) : 0.0f;
    }
    const float vj = live ? to_float<T>(v[static_cast<long long>(t) * ldv + static_cast<long long>(h) * vdim + col]) : 0.0f;
    const float* k = cur;
    const float* q = cur + dim;
    float o0 = 0.0f, o1 = 0.0f, o2 = 0.0f, o3 = 0.0f;
    int i = 0;
    for (; i + 4 <= dim; i += 4) {
      const float s0 = fmaf(k[i + 0], vj, fmaf(dm1, S[(i + 0) * cols + j], S[(i + 0) * cols + j]));
      const float s1 = fmaf(k[i + 1], vj, fmaf(dm1, S[(i + 1) * cols + j], S[(i + 1) * cols + j]));
      const float s2 = fmaf(k[i + 2], vj, fmaf(dm1, S[(i + 2) * cols + j], S[(i + 2) * cols + j]));
      const float s3 = fmaf(k[i + 3], vj, fmaf(dm1, S[(i + 3) * cols + j], S[(i + 3) * cols + j]));
      S[(i + 0) * cols + j] = s0; S[(i + 1) * cols + j] = s1; S[(i + 2) * cols + j] = s2; S[(i + 3) * cols + j] = s3;
      o0 = fmaf(s0, q[i + 0], o0); o1 = fmaf(s1, q[i + 1], o1); o2 = fmaf(s2, q[i + 2], o2); o3 = fmaf(s3, q[i + 3], o3);
    }
    for (; i < dim; ++i) {
      const float s0 = fmaf(k[i], vj, fmaf(dm1, S[i * cols + j], S[i * cols + j]));
      S[i * cols + j] = s0;
      o0 = fmaf(s0, q[i], o0);
    }
    if (live) out[(static_cast<long long>(t) * heads + h) * vdim + col] = (o0 + o1) + (o2 + o3);
  }
  if (live)
    for (int i = 0; i < dim; ++i) Sg[static_cast<long long>(i) * vdim + col] = S[i * cols + j];
}

// The same recurrence with S in registers, for the key sizes that have an instance.  Block (request, head, 32 value
// columns); a column of S is held by kParts threads (thread (column c = tid / kParts, part p = tid % kParts) the rows
// p * kDim / kParts ...), so the parts of a column sit in neighbouring lanes and meet through shuffles.  What the
// recurrence reads of a token (k, q, the block's 32 values) is staged in shared memory a chunk of tokens at a time, two
// buffers: the next chunk's numbers are copied asynchronously while this chunk is computed, so no load from memory
// and only one barrier a chunk lie on the chain from token to token.  The order of the additions is fixed by the
// kernel, not by the step's make-up or by where a chunk begins.
__device__ __forceinline__ void retention_copy_16(void* smem_dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst))), "l"(src));
}

template <typename T, int kDim>
__global__ void __launch_bounds__(kDim >= 64 ? 256 : (kDim >= 32 ? 128 : 64))
retention_recurrence_reg_kernel(const float* __restrict__ qf, const float* __restrict__ kf, const T* __restrict__ v,
                                long long ldv, const float* __restrict__ decay_m1, float* __restrict__ out,
                                float* __restrict__ state, long long state_stride, const int* __restrict__ cu_q,
                                const int* __restrict__ state_slots, int heads, int vdim, int small_rows) {
  constexpr int kParts = kDim >= 64 ? 8 : (kDim >= 32 ? 4 : 2);   // threads a column of S
  constexpr int kThreads = 32 * kParts;
  constexpr int kRows = kDim / kParts;                    // rows of S a thread holds (a multiple of 4)
  constexpr int kSeg = kRows + 4;                         // a part's stretch of k (or q) in the staging buffer: the parts'
                                                          // 16-byte reads fall into different banks
  constexpr int kChunk = kDim <= 128 ? 16 : 8;            // tokens staged at a time
  constexpr int kVWords = 32 * sizeof(T) / 4;             // the block's 32 values of a token, in 32-bit words
  constexpr int kTok = 2 * kParts * kSeg + kVWords;       // words staged a token: k | q | values
  constexpr int kCopies = 2 * (kDim / 4) + kVWords / 4;   // 16-byte copies a token
  extern __shared__ __align__(16) float stage[];          // [2][kChunk][kTok]
  wait_for_prior_kernels();
  launch_dependents();
  const int r = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * 32;
  const int lo = cu_q[r], hi = cu_q[r + 1];
  const int slot = state_slots[r];
  if (hi <= lo || slot < 0 || hi - lo > small_rows) return;
  const int tid = threadIdx.x, c = tid / kParts, p = tid % kParts;
  float* Sg = state + slot * state_stride + (static_cast<long long>(h) * kDim + p * kRows) * vdim + col0 + c;
  float S[kRows];
#pragma unroll
  for (int i = 0; i < kRows; ++i) S[i] = Sg[static_cast<long long>(i) * vdim];
  const float dm1 = decay_m1[h];
  auto fetch = [&](int buf, int t0) {
    const int n = min(kChunk, hi - t0);
    for (int e = tid; e < n * kCopies; e += kThreads) {
      const int tok = e / kCopies, piece = e % kCopies;
      float* dst = stage + (buf * kChunk + tok) * kTok;
      const long long t = t0 + tok;
      if (piece < 2 * (kDim / 4)) {
        const int which = piece / (kDim / 4), at = (piece % (kDim / 4)) * 4;       // k or q; the element
        const float* src = (which == 0 ? kf : qf) + (t * heads + h) * kDim + at;
        retention_copy_16(dst + which * kParts * kSeg + (at / kRows) * kSeg + at % kRows, src);
      } else {
        const int w = piece - 2 * (kDim / 4);
        retention_copy_16(dst + 2 * kParts * kSeg + w * 4,
                          reinterpret_cast<const float*>(v + t * ldv + static_cast<long long>(h) * vdim + col0) + w * 4);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0, lo);
  int buf = 0;
  for (int t0 = lo; t0 < hi; t0 += kChunk, buf ^= 1) {
    if (t0 + kChunk < hi) {
      fetch(buf ^ 1, t0 + kChunk);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const int n = min(kChunk, hi - t0);
#pragma unroll 4                                           // (a token's shuffles and store run under the next tokens' FMAs)
    for (int tok = 0; tok < n; ++tok) {
      const float* cur = stage + (buf * kChunk + tok) * kTok;
      const float4* k4 = reinterpret_cast<const float4*>(cur + p * kSeg);
      const float4* q4 = reinterpret_cast<const float4*>(cur + kParts * kSeg + p * kSeg);
      const float vj = to_float<T>(reinterpret_cast<const T*>(cur + 2 * kParts * kSeg)[c]);
      float o0 = 0.0f, o1 = 0.0f, o2 = 0.0f, o3 = 0.0f;
#pragma unroll
      for (int i = 0; i < kRows / 4; ++i) {
        const float4 k = k4[i], q = q4[i];
        S[4 * i + 0] = fmaf(k.x, vj, fmaf(dm1, S[4 * i + 0], S[4 * i + 0]));
        S[4 * i + 1] = fmaf(k.y, vj, fmaf(dm1, S[4 * i + 1], S[4 * i + 1]));
        S[4 * i + 2] = fmaf(k.z, vj, fmaf(dm1, S[4 * i + 2], S[4 * i + 2]));
        S[4 * i + 3] = fmaf(k.w, vj, fmaf(dm1, S[4 * i + 3], S[4 * i + 3]));
        o0 = fmaf(S[4 * i + 0], q.x, o0);
        o1 = fmaf(S[4 * i + 1], q.y, o1);
        o2 = fmaf(S[4 * i + 2], q.z, o2);
        o3 = fmaf(S[4 * i + 3], q.w, o3);
      }
      float o = (o0 + o1) + (o2 + o3);
#pragma unroll
      for (int d = 1; d < kParts; d <<= 1) o += __shfl_xor_sync(0xffffffffu, o, d);
      if (p == 0) out[((static_cast<long long>(t0) + tok) * heads + h) * vdim + col0 + c] = o;
    }
    __syncthreads();                                       // the buffer is free for the chunk after the next
  }
#pragma unroll
  for (int i = 0; i < kRows; ++i) Sg[static_cast<long long>(i) * vdim] = S[i];
}

// ---- by chunks ----------------------------------------------------------------------------------------------------------
struct RetentionArgs {
  const float* q;                                          // rotated, [rows, heads, dim]
  const float* k;                                          // rotated and scaled
  const __nv_bfloat16* v;
  long long ldv;
  const float* decay_m1;
  float* out;
  float* state;
  long long state_stride;
  float* chunk_states;                                     // of the wave: [chunks, heads, dim, vdim]
  const int* cu_q;
  const int* state_slots;
  int requests, heads, vdim, small_rows;
  int from, chunks;                                        // the wave: its first chunk of the step's, how many
};

__device__ __forceinline__ float decay_power(float log_decay, int n) { return n == 0 ? 1.0f : expf(log_decay * static_cast<float>(n)); }

// Block (chunk, head, VT value columns), 256 threads: DIM / 16 rows by VT / 16 columns of U a thread.  Bound by the FMA
// units (64 k-steps of 2048 two-number FMAs from 16 KB of shared memory reads).
template <int DIM, int VT>
__global__ void __launch_bounds__(256)
retention_chunk_state_kernel(const RetentionArgs p) {
  extern __shared__ __align__(16) float smem[];
  float* ks = smem;                                        // [64][DIM]
  float* vs = ks + chunks::kRows * DIM;                    // [64][VT]
  __shared__ chunks::Place place;
  __shared__ float power[chunks::kRows];
  wait_for_prior_kernels();
  launch_dependents();
  const chunks::Place c = chunks::find(p.cu_q, p.state_slots, p.requests, p.small_rows, p.from + blockIdx.x, &place);
  if (c.request < 0) return;
  const int h = blockIdx.y, v0 = blockIdx.z * VT, tid = threadIdx.x;
  chunks::load_rows<DIM, DIM>(ks, p.k + (static_cast<long long>(c.first) * p.heads + h) * DIM, static_cast<long long>(p.heads) * DIM, c.rows);
  mma::copy_async_commit();
  if (tid < chunks::kRows) power[tid] = decay_power(log1pf(p.decay_m1[h]), max(0, c.rows - 1 - tid));
  chunks::load_rows<VT, VT>(vs, p.v + c.first * p.ldv + static_cast<long long>(h) * p.vdim + v0, p.ldv, c.rows);
  __syncthreads();
  for (int e = tid; e < chunks::kRows * VT; e += 256) vs[e] *= power[e / VT];
  mma::copy_async_wait<0>();
  __syncthreads();
  constexpr int RM = DIM / 16, RN = VT / 16;
  float2 U[RM][RN / 2];
  chunks::clear(U);
  chunks::multiply_outer<RM, RN>(U, ks, DIM, vs, VT, (c.rows + 3) & ~3);
  const int tx = tid & 15, ty = tid >> 4;
  float* to = p.chunk_states + ((static_cast<long long>(blockIdx.x) * p.heads + h) * DIM + ty * RM) * p.vdim + v0 + 4 * tx;
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int g = 0; g < RN / 4; ++g)
      *reinterpret_cast<float4*>(to + static_cast<long long>(i) * p.vdim + 64 * g) =
          make_float4(U[i][2 * g].x, U[i][2 * g].y, U[i][2 * g + 1].x, U[i][2 * g + 1].y);
}

// Block (request, head, 128 pieces of four numbers of S): a stream over the wave's chunks, eight of them asked for ahead.
__global__ void __launch_bounds__(128)
retention_state_pass_kernel(const RetentionArgs p, int dim) {
  __shared__ int first;
  wait_for_prior_kernels();
  launch_dependents();
  const int r = blockIdx.x, h = blockIdx.y;
  const int n = p.cu_q[r + 1] - p.cu_q[r], slot = p.state_slots[r];
  if (n <= p.small_rows || slot < 0) return;
  if (threadIdx.x == 0) first = chunks::first_of(p.cu_q, p.state_slots, p.small_rows, r);
  __syncthreads();
  const int count = (n + chunks::kRows - 1) / chunks::kRows;
  const int lo = max(0, p.from - first), hi = min(count, p.from + p.chunks - first);     // the request's chunks of this wave
  const long long matrix = static_cast<long long>(dim) * p.vdim, at = (static_cast<long long>(blockIdx.z) * 128 + threadIdx.x) * 4;
  if (lo >= hi || at >= matrix) return;
  float* Sg = p.state + slot * p.state_stride + h * matrix + at;
  float4 S = make_float4(Sg[0], Sg[1], Sg[2], Sg[3]);
  const long long step = p.heads * matrix;
  float* U = p.chunk_states + (static_cast<long long>(first + lo - p.from) * p.heads + h) * matrix + at;
  const float lg = log1pf(p.decay_m1[h]), whole = decay_power(lg, chunks::kRows);
  constexpr int kAhead = 8;
  float4 u[kAhead];
#pragma unroll
  for (int i = 0; i < kAhead; ++i)
    if (lo + i < hi) u[i] = *reinterpret_cast<const float4*>(U + i * step);
  for (int c0 = lo; c0 < hi; c0 += kAhead) {
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const int c = c0 + i;
      if (c >= hi) break;
      const float4 add = u[i];
      if (c + kAhead < hi) u[i] = *reinterpret_cast<const float4*>(U + (c + kAhead - lo) * step);
      *reinterpret_cast<float4*>(U + (c - lo) * step) = S;
      const float f = c + 1 < count ? whole : decay_power(lg, n - c * chunks::kRows);
      S.x = fmaf(f, S.x, add.x);
      S.y = fmaf(f, S.y, add.y);
      S.z = fmaf(f, S.z, add.z);
      S.w = fmaf(f, S.w, add.w);
    }
  }
  Sg[0] = S.x; Sg[1] = S.y; Sg[2] = S.z; Sg[3] = S.w;
}

template <int DIM, int VT>
constexpr size_t retention_out_bytes() {
  return sizeof(float) * chunks::kRows * (2 * (DIM + 4) + (VT > DIM + 4 ? VT - DIM - 4 : 0) + 68);
}

// Block (chunk, head, VT value columns), 256 threads: 4 rows by VT / 16 columns of the read-outs a thread.
template <int DIM, int VT>
__global__ void __launch_bounds__(256, 2)
retention_chunk_out_kernel(const RetentionArgs p) {
  constexpr int LD = DIM + 4, LP = 68;
  extern __shared__ __align__(16) float smem[];
  float* qs = smem;                                        // [64][LD]
  float* P = qs + chunks::kRows * LD;                      // [64][LP]: decayed scores
  float* ks = P + chunks::kRows * LP;                      // [64][LD]; then 64 rows of the state [64][VT]; then the values
  __shared__ chunks::Place place;
  __shared__ float power[chunks::kRows + 1];
  wait_for_prior_kernels();
  launch_dependents();
  const chunks::Place c = chunks::find(p.cu_q, p.state_slots, p.requests, p.small_rows, p.from + blockIdx.x, &place);
  if (c.request < 0) return;
  const int h = blockIdx.y, v0 = blockIdx.z * VT, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const long long at = (static_cast<long long>(c.first) * p.heads + h) * DIM, ld = static_cast<long long>(p.heads) * DIM;
  chunks::load_rows<DIM, LD>(qs, p.q + at, ld, c.rows);
  chunks::load_rows<DIM, LD>(ks, p.k + at, ld, c.rows);
  mma::copy_async_commit();
  if (tid <= chunks::kRows) power[tid] = decay_power(log1pf(p.decay_m1[h]), tid);
  mma::copy_async_wait<0>();
  __syncthreads();
  {
    float2 s[4][4];
    chunks::clear(s);
    chunks::multiply_rows<4, 4, DIM, LD>(s, qs, ks);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int row = ty * 4 + i, col = tx + 16 * j;
        P[row * LP + col] = col <= row ? (s[i][j].x + s[i][j].y) * power[row - col] : 0.0f;
      }
  }
  constexpr int RN = VT / 16;
  float2 o[4][RN / 2];
  chunks::clear(o);
  const float* state = p.chunk_states + (static_cast<long long>(blockIdx.x) * p.heads + h) * DIM * p.vdim + v0;
#pragma unroll 1
  for (int d0 = 0; d0 < DIM; d0 += chunks::kRows) {
    __syncthreads();                                       // (what lay there is done with)
    chunks::load_rows<VT, VT>(ks, state + static_cast<long long>(d0) * p.vdim, p.vdim, chunks::kRows);
    mma::copy_async_commit();
    mma::copy_async_wait<0>();
    __syncthreads();
    chunks::multiply_columns<4, RN>(o, qs + d0, LD, ks, VT, chunks::kRows);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < RN / 2; ++j) {
      o[i][j].x *= power[ty * 4 + i + 1];
      o[i][j].y *= power[ty * 4 + i + 1];
    }
  __syncthreads();
  const bool wild = chunks::load_rows<VT, VT>(ks, p.v + c.first * p.ldv + static_cast<long long>(h) * p.vdim + v0, p.ldv, c.rows);
  const int seen = (tid >> 5) * 8 + 8;                     // (the warp's rows see no later ones)
  if (!__syncthreads_or(wild)) chunks::multiply_columns<4, RN>(o, P, LP, ks, VT, seen);
  else chunks::multiply_columns<4, RN, true>(o, P, LP, ks, VT, seen);          // (zero times infinity is not zero)
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

}  // namespace pih

using namespace pih;
typedef __nv_bfloat16 bf16;

// Steps that may go by chunks: bf16 values that can be read 16 bytes at a time, sizes with an instance.
static bool retention_takes_chunks(int dtype, const void* v, long long ldv, int heads, int dim, int vdim) {
  return dtype == PIH_BF16 && (dim == 64 || dim == 128) && vdim % 64 == 0 && heads <= 65535 && vdim / 64 <= 65535 &&
         reinterpret_cast<uintptr_t>(v) % 16 == 0 && ldv % 8 == 0;
}

// fp32 numbers of chunk scratch for a step of ``rows`` rows whose requests of more than ``small_rows`` rows go by chunks, at most
// ``most`` of them (or one chunk's); 0: its sizes do not go by chunks.
extern "C" long long pih_retention_chunk_scratch(int dtype, const void* v, long long ldv, int rows, int requests, int heads, int dim,
                                                 int vdim, int small_rows, long long most) {
  if (!retention_takes_chunks(dtype, v, ldv, heads, dim, vdim)) return 0;
  const long long each = static_cast<long long>(heads) * dim * vdim, fit = most / each > 1 ? most / each : 1;
  const long long chunks = chunks::at_most(rows, requests, small_rows);
  return (chunks < fit ? chunks : fit) * each;
}

template <int DIM, int VT>
static int launch_retention_chunks(cudaStream_t s, RetentionArgs p, int rows, long long scratch) {
  const unsigned tiles = p.vdim / VT;
  constexpr size_t state_bytes = sizeof(float) * chunks::kRows * (DIM + VT), out_bytes = retention_out_bytes<DIM, VT>();
  cudaFuncSetAttribute(retention_chunk_state_kernel<DIM, VT>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(state_bytes));
  cudaFuncSetAttribute(retention_chunk_out_kernel<DIM, VT>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(out_bytes));
  const long long count = chunks::at_most(rows, p.requests, p.small_rows), fit = scratch / (static_cast<long long>(p.heads) * DIM * p.vdim);
  for (long long from = 0; from < count; from += fit) {
    p.from = static_cast<int>(from);
    p.chunks = static_cast<int>(count - from < fit ? count - from : fit);
    launch_kernel(retention_chunk_state_kernel<DIM, VT>, dim3(p.chunks, p.heads, tiles), dim3(256), state_bytes, s, p);
    PIH_LAUNCH_CHECK();
    launch_kernel(retention_state_pass_kernel, dim3(p.requests, p.heads, (DIM * p.vdim / 4 + 127) / 128), dim3(128), 0, s, p, DIM);
    PIH_LAUNCH_CHECK();
    launch_kernel(retention_chunk_out_kernel<DIM, VT>, dim3(p.chunks, p.heads, tiles), dim3(256), out_bytes, s, p);
    PIH_LAUNCH_CHECK();
  }
  return 0;
}

template <typename T, int D>
static void launch_retention_in_registers(cudaStream_t s, const float* qf, const float* kf, const void* v, long long ldv,
                                          const void* decay_m1, void* out, void* state, long long state_stride,
                                          const void* cu_q, const void* state_slots, int requests, int heads, int vdim, int small_rows) {
  constexpr int parts = D >= 64 ? 8 : (D >= 32 ? 4 : 2);
  constexpr int chunk = D <= 128 ? 16 : 8;
  constexpr size_t needed = 2 * chunk * (2 * parts * (D / parts + 4) + 32 * sizeof(T) / 4) * sizeof(float);
  // The token loop is bound by the SM's shared-memory reads: two blocks on one SM each run at half speed.  With fewer
  // blocks than SMs, every block asks for more than half of an SM's shared memory and so gets an SM alone.
  const bool alone = static_cast<long long>(requests) * heads * (vdim / 32) <= 148;
  const size_t bytes = alone && needed < 116 * 1024 ? 116 * 1024 : needed;
  if (bytes > 48 * 1024)
    cudaFuncSetAttribute(retention_recurrence_reg_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         static_cast<int>(bytes));
  launch_kernel(retention_recurrence_reg_kernel<T, D>, dim3(requests, heads, vdim / 32), dim3(32 * parts), bytes, s, qf, kf,
                static_cast<const T*>(v), ldv, static_cast<const float*>(decay_m1), static_cast<float*>(out),
                static_cast<float*>(state), state_stride, static_cast<const int*>(cu_q),
                static_cast<const int*>(state_slots), heads, vdim, small_rows);
}

// qk [rows, ld]: q heads then k heads ([heads, dim] each); v [rows, ldv]: [heads, vdim]; freq fp32 [rot / 2] (null: no
// rotation); decay_m1 fp32 [heads]: decay - 1; scratch fp32 [2 * rows * heads * dim]; out fp32 [rows, heads, vdim];
// state fp32: S of (slot, head) at state + slot * state_stride + head * dim * vdim, [dim, vdim].  chunk_scratch: null, or
// chunk_numbers of fp32, 16-byte aligned, one chunk's or more (pih_retention_chunk_scratch): requests of more than small_rows
// rows go by chunks.
extern "C" int pih_retention(int dtype, const void* qk, long long ld, const void* v, long long ldv, const void* freq, int rot,
                             const void* positions, const void* decay_m1, float key_scale, void* scratch, void* out,
                             void* state, long long state_stride, const void* cu_q, const void* state_slots, int rows,
                             int requests, int heads, int dim, int vdim, void* chunk_scratch, long long chunk_numbers, int small_rows,
                             void* stream) {
  if (rows <= 0 || requests <= 0) return 0;
  if (chunk_scratch != nullptr && (!retention_takes_chunks(dtype, v, ldv, heads, dim, vdim) ||
                                   reinterpret_cast<uintptr_t>(chunk_scratch) % 16 || reinterpret_cast<uintptr_t>(scratch) % 16))
    return PIH_ERR_UNSUPPORTED;
  if (chunk_scratch != nullptr && (small_rows < 0 || chunk_numbers < static_cast<long long>(heads) * dim * vdim))
    return PIH_ERR_BAD_ARGUMENT;
  if (chunk_scratch == nullptr) small_rows = 0x7fffffff;
  if (rot < 0 || rot > dim || (rot & 1) || (rot > 0 && freq == nullptr)) return PIH_ERR_BAD_ARGUMENT;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int cols = vdim >= 64 ? 64 : 32;
  if (dim > 16 * cols) return PIH_ERR_UNSUPPORTED;
  const size_t smem = (static_cast<size_t>(dim) * cols + 4 * dim) * sizeof(float);
  if (smem > 200 * 1024) return PIH_ERR_UNSUPPORTED;
  float* qf = static_cast<float*>(scratch);
  float* kf = qf + static_cast<long long>(rows) * heads * dim;
  const long long n = static_cast<long long>(rows) * heads * dim;
  const dim3 grid(requests, heads, (vdim + cols - 1) / cols);
  // S in registers: the key sizes with an instance, value columns in whole slabs of 32, and everything that is copied
  // in 16-byte pieces on a 16-byte boundary
  const size_t esize = dtype == PIH_F32 ? 4 : 2;
  const bool in_registers = (dim == 16 || dim == 32 || dim == 64 || dim == 128 || dim == 256) && vdim % 32 == 0 &&
                            (reinterpret_cast<uintptr_t>(v) % 16 == 0) && (ldv * esize) % 16 == 0 &&
                            (vdim * esize) % 16 == 0 && (reinterpret_cast<uintptr_t>(scratch) % 16 == 0);
#define PIH_RET_ARGS s, qf, kf, v, ldv, decay_m1, out, state, state_stride, cu_q, state_slots, requests, heads, vdim, small_rows
#define PIH_RET(T)                                                                                                     \
  do {                                                                                                                 \
    launch_kernel(retention_prepare_kernel<T>, dim3(static_cast<unsigned>((n + 255) / 256)), dim3(256), 0, s,          \
                  static_cast<const T*>(qk), ld, static_cast<const float*>(freq), static_cast<const int*>(positions),  \
                  qf, kf, rows, heads, dim, rot, key_scale);                                                           \
    PIH_LAUNCH_CHECK();                                                                                                \
    if (chunk_scratch != nullptr) {                                                                                    \
      const RetentionArgs p = {qf, kf, static_cast<const bf16*>(v), ldv, static_cast<const float*>(decay_m1),          \
                               static_cast<float*>(out), static_cast<float*>(state), state_stride,                     \
                               static_cast<float*>(chunk_scratch), static_cast<const int*>(cu_q),                      \
                               static_cast<const int*>(state_slots), requests, heads, vdim, small_rows, 0, 0};         \
      const int rc = dim == 128 ? (vdim % 128 ? launch_retention_chunks<128, 64>(s, p, rows, chunk_numbers)            \
                                              : launch_retention_chunks<128, 128>(s, p, rows, chunk_numbers))          \
                                : (vdim % 128 ? launch_retention_chunks<64, 64>(s, p, rows, chunk_numbers)             \
                                              : launch_retention_chunks<64, 128>(s, p, rows, chunk_numbers));          \
      if (rc != 0) return rc;                                                                                          \
    }                                                                                                                  \
    if (in_registers) {                                                                                                \
      switch (dim) {                                                                                                   \
        case 16: launch_retention_in_registers<T, 16>(PIH_RET_ARGS); break;                                           \
        case 32: launch_retention_in_registers<T, 32>(PIH_RET_ARGS); break;                                           \
        case 64: launch_retention_in_registers<T, 64>(PIH_RET_ARGS); break;                                           \
        case 128: launch_retention_in_registers<T, 128>(PIH_RET_ARGS); break;                                         \
        default: launch_retention_in_registers<T, 256>(PIH_RET_ARGS); break;                                          \
      }                                                                                                                \
      break;                                                                                                           \
    }                                                                                                                  \
    if (smem > 48 * 1024)                                                                                              \
      cudaFuncSetAttribute(retention_recurrence_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,                \
                           static_cast<int>(smem));                                                                    \
    launch_kernel(retention_recurrence_kernel<T>, grid, dim3(cols), smem, s, static_cast<const float*>(qf),            \
                  static_cast<const float*>(kf), static_cast<const T*>(v), ldv, static_cast<const float*>(decay_m1),   \
                  static_cast<float*>(out), static_cast<float*>(state), state_stride, static_cast<const int*>(cu_q),   \
                  static_cast<const int*>(state_slots), heads, dim, vdim, small_rows);                                 \
  } while (0)
  if (dtype == PIH_F32) PIH_RET(float);
  else if (dtype == PIH_BF16) PIH_RET(bf16);
  else return PIH_ERR_BAD_ARGUMENT;
#undef PIH_RET
#undef PIH_RET_ARGS
  PIH_LAUNCH_CHECK();
  return 0;
}
