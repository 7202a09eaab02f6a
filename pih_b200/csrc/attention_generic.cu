// Causal grouped-query attention over the paged cache on CUDA cores, 32-bit
// arithmetic, any head size, any number of heads and groups, any page size,
// optional sliding window.  It is the attention of the true 32-bit path and
// the plain twin of the tensor-core kernels.
//
// One warp per (query row, query head).  The row at absolute position p
// reads keys first..p with first = max(0, p - window + 1) (0 without a
// window), in blocks of 32 that start at `first`: the order of every
// reduction depends on p and the window alone, never on how the prompt was
// cut into steps, on the other rows of the batch or on which pages hold the
// keys.  Online softmax as the reference's kernel does it
// (kernels/cuda/qwen_bf16_primitives.cu:660-733): score = (q . k) * scale with
// the scale after the dot product, running maximum, running sum,
// accumulator rescaled when the maximum moves, one rounding of acc / sum.
//
// q is read from the fused projection buffer [rows, row_stride] (head h at
// column h * head_dim); cache layout [page][2][kv_head][page_size][head_dim].
#include "common.cuh"
#include "mma.cuh"

namespace pih {

constexpr int kMaxDimPerLane = 8;   // head_dim <= 256

template <typename T>
__global__ void paged_attention_generic_kernel(
    const T* __restrict__ q, int q_stride, T* __restrict__ out, const T* __restrict__ cache,
    const int* __restrict__ block_table, int table_width, const int* __restrict__ request_of_row,
    const int* __restrict__ positions, int rows, int heads, int kv_heads, int head_dim, int page_size,
    int num_pages, float scale, int window, uint32_t* error) {
  wait_for_prior_kernels();
  launch_dependents();                                   // (the next kernel's blocks may become resident and wait)
  extern __shared__ float smem[];
  const int warps_per_block = blockDim.x >> 5;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long item = static_cast<long long>(blockIdx.x) * warps_per_block + warp;
  if (item >= static_cast<long long>(rows) * heads) return;
  const int t = static_cast<int>(item / heads);
  const int h = static_cast<int>(item % heads);
  const int g = h / (heads / kv_heads);
  const int r = request_of_row[t];
  if (r < 0) return;                                   // a row of padding
  const int p = positions[t];
  const int first = window > 0 ? max(0, p - window + 1) : 0;
  const int* table = block_table + static_cast<size_t>(r) * table_width;

  float* qs = smem + warp * head_dim;
  const T* qrow = q + static_cast<size_t>(t) * q_stride + static_cast<size_t>(h) * head_dim;
  for (int c = lane; c < head_dim; c += 32) qs[c] = to_float<T>(qrow[c]);
  __syncwarp();

  float acc[kMaxDimPerLane];
#pragma unroll
  for (int i = 0; i < kMaxDimPerLane; ++i) acc[i] = 0.0f;
  float m = -INFINITY, l = 0.0f;
  const size_t head_elems = static_cast<size_t>(page_size) * head_dim;

  for (int base = first; base <= p; base += 32) {
    const int j = base + lane;
    const bool valid = j <= p;
    float s = -INFINITY;
    const T* krow = nullptr;
    if (valid) {
      const int page = table[j / page_size];
      if (page < 0 || page >= num_pages) {
        publish_error(error, kRowWithoutPage);
      } else {
        krow = cache + ((static_cast<size_t>(page) * 2 + 0) * kv_heads + g) * head_elems +
               static_cast<size_t>(j % page_size) * head_dim;
        float dot = 0.0f;
        for (int c = 0; c < head_dim; ++c) dot = fmaf(qs[c], to_float<T>(krow[c]), dot);
        s = dot * scale;
      }
    }
    const float block_max = warp_max(s);
    const float m_new = fmaxf(m, block_max);
    const float alpha = (m == -INFINITY) ? 0.0f : expf(m - m_new);
    const float e = (s == -INFINITY) ? 0.0f : expf(s - m_new);
    l = l * alpha + warp_sum(e);
#pragma unroll
    for (int i = 0; i < kMaxDimPerLane; ++i) acc[i] *= alpha;
    const int count = min(32, p - base + 1);
    for (int jj = 0; jj < count; ++jj) {
      const float pj = __shfl_sync(0xffffffffu, e, jj);
      const int kj = base + jj;
      const int page = table[kj / page_size];
      if (page < 0 || page >= num_pages) continue;     // reported above by the lane that owns kj
      const T* vrow = cache + ((static_cast<size_t>(page) * 2 + 1) * kv_heads + g) * head_elems +
                      static_cast<size_t>(kj % page_size) * head_dim;
#pragma unroll
      for (int i = 0; i < kMaxDimPerLane; ++i) {
        const int c = lane + 32 * i;
        if (c < head_dim) acc[i] = fmaf(pj, to_float<T>(vrow[c]), acc[i]);
      }
    }
    m = m_new;
  }
  if (!(l > 0.0f) || !isfinite(l)) {
    if (lane == 0) publish_error(error, kAttentionDenominator);
    l = 1.0f;
  }
  T* orow = out + (static_cast<size_t>(t) * heads + h) * head_dim;
#pragma unroll
  for (int i = 0; i < kMaxDimPerLane; ++i) {
    const int c = lane + 32 * i;
    if (c < head_dim) orow[c] = from_float<T>(acc[i] / l);
  }
}

// The same attention in 32 bits for head sizes 64 and 128.  The kernel above reads a key a lane, 32 cache lines a load:
// 350 us for 200 rows of 16 heads of 128, of which the arithmetic is 10 us.  Here a block takes up to kPairs (row, head)
// pairs of one kv head — neighbouring rows of a request —, so that a key is read once for all of them.  Four warps share
// the keys: warp w takes the tiles of 32 keys whose number is w modulo 4 (numbers of the whole context: what a row adds
// up, and in which order, depends on its position and the window alone), and the four states meet at the end in the order
// of the warps.  A tile's keys lie in shared memory (rows 4 words wider than the head: conflict-free 16-byte reads, a key
// a lane; the next tile's copies run under the softmax and the values), the values come from memory a key a warp.  Bound
// by the shared-memory reads of the scores with many rows, by the latency of a tile with few.
constexpr int kF32Warps = 4, kF32Pairs = 16, kF32FewPairs = 4;
static_assert(kF32Warps * kF32FewPairs == kF32Pairs, "one tile: a few pairs a warp");

template <int HD>
constexpr size_t f32_attention_bytes() {
  return sizeof(float) * (kF32Warps * 32 * (HD + 4) + kF32Pairs * HD + kF32Warps * kF32Pairs * 34);
}

struct F32AttentionArgs {
  const float* q;
  int q_stride;
  float* out;
  const float* cache;
  const int* block_table;
  int table_width;
  const int* request_of_row;
  const int* positions;
  int rows, heads, kv_heads, page_size, num_pages;
  float scale;
  int window;
  uint32_t* error;
};

// The pairs of rows row .. row + pairs / group - 1, whose first one is at position p0 (pair i: row i / group, head i % group).
// ONE_TILE: their keys lie in one tile, of which each warp takes P pairs of its own (else one warp would have them all,
// with the same sums: 16 rows of 8 heads of 64 14.5 us, now 11.4; a row of 16 heads of 64 and 5 keys 11.1 and 7.7).
template <int HD, int P, bool ONE_TILE>
__device__ __forceinline__ void f32_attend(const F32AttentionArgs& a, float* smem, int row, int p0, int pairs, int group, int g,
                                           const int* table) {
  constexpr int C = HD / 32, LD = HD + 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* ks = smem + warp * 32 * LD;                       // this warp's tile of keys; in the end its sums [P][HD]
  float* qs = smem + kF32Warps * 32 * LD;                  // [P][HD]
  float* ps = qs + kF32Pairs * HD + warp * kF32Pairs * 34;   // [P][32] weights of a tile; in the end [P] maxima, [P] sums
  const int own = ONE_TILE ? warp * P : 0;                 // this warp's first pair
  for (int e = threadIdx.x; e < (ONE_TILE ? kF32Warps * P : P) * HD; e += kF32Warps * 32) {
    const int i = e / HD;
    qs[e] = i < pairs ? a.q[static_cast<size_t>(row + i / group) * a.q_stride + static_cast<size_t>(g * group + i % group) * HD + e % HD] : 0.0f;
  }
  __syncthreads();
  const int last = p0 + (pairs - 1) / group;
  const int lowest = a.window > 0 ? max(0, p0 - a.window + 1) : 0;
  const size_t head_elems = static_cast<size_t>(a.page_size) * HD;
  const long long to_values = static_cast<long long>(a.kv_heads) * head_elems;
  auto place = [&](int t) -> long long {                   // of this lane's key of tile t in the cache; -1: none
    const int j = 32 * t + lane;
    if (j < lowest || j > last) return -1;
    const int page = table[j / a.page_size];
    if (page < 0 || page >= a.num_pages) {
      publish_error(a.error, kRowWithoutPage);
      return -1;
    }
    return static_cast<long long>((static_cast<size_t>(page) * 2 * a.kv_heads + g) * head_elems + static_cast<size_t>(j % a.page_size) * HD);
  };
  auto stage = [&](long long at) {
    constexpr int kLanes = HD / 4;                         // 16-byte pieces of a key
#pragma unroll 8
    for (int jj = 0; jj < 32; jj += 32 / kLanes) {
      const int key = jj + lane / kLanes;
      const long long from = __shfl_sync(0xffffffffu, at, key);
      mma::copy_async_16_or_zero(ks + key * LD + (lane % kLanes) * 4, a.cache + (from < 0 ? 0 : from) + (lane % kLanes) * 4, from >= 0);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float m[P], l[P], acc[P][C];
#pragma unroll
  for (int i = 0; i < P; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.0f;
#pragma unroll
    for (int c = 0; c < C; ++c) acc[i][c] = 0.0f;
  }
  const int t_end = last / 32;
  int t = lowest / 32;
  if (!ONE_TILE) t += (warp - t) & (kF32Warps - 1);
  else if (own >= pairs) t = t_end + 1;
  long long at = t <= t_end ? place(t) : -1;
  if (t <= t_end) stage(at);
  for (; t <= t_end; t += kF32Warps) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    float2 dot[P];
#pragma unroll
    for (int i = 0; i < P; ++i) dot[i] = make_float2(0.0f, 0.0f);
#pragma unroll 4
    for (int c = 0; c < HD; c += 4) {
      const float4 k = *reinterpret_cast<const float4*>(ks + lane * LD + c);
#pragma unroll
      for (int i = 0; i < P; ++i) {
        const float4 q = *reinterpret_cast<const float4*>(qs + (own + i) * HD + c);
        dot[i] = fma2(make_float2(q.x, q.y), make_float2(k.x, k.y), dot[i]);
        dot[i] = fma2(make_float2(q.z, q.w), make_float2(k.z, k.w), dot[i]);
      }
    }
    __syncwarp();                                          // every lane is through with the tile and the last weights
    const long long mine = at;
    const int j = 32 * t + lane, tile = t;
    if (t + kF32Warps <= t_end) {
      at = place(t + kF32Warps);
      stage(at);
    }
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const int p = p0 + (own + i) / group;
      const bool seen = own + i < pairs && mine >= 0 && j <= p && (a.window <= 0 || j > p - a.window);
      const float s = seen ? (dot[i].x + dot[i].y) * a.scale : -INFINITY;
      const float m_new = fmaxf(m[i], warp_max(s));
      const float alpha = m[i] == -INFINITY ? 0.0f : expf(m[i] - m_new);
      const float e = s == -INFINITY ? 0.0f : expf(s - m_new);
      l[i] = l[i] * alpha + e;                             // (this lane's keys; the lanes meet at the end)
#pragma unroll
      for (int c = 0; c < C; ++c) acc[i][c] *= alpha;
      ps[i * 32 + lane] = e;
      m[i] = m_new;
    }
    __syncwarp();
    const int count = min(32, last - 32 * tile + 1);
    auto value = [&](int jj, float (&v)[C]) {              // of key jj of the tile, this lane's columns
      const long long from = __shfl_sync(0xffffffffu, mine, jj);
      const float* vrow = a.cache + from + to_values + lane * C;
      if (C == 4) {
        const float4 x = from >= 0 ? *reinterpret_cast<const float4*>(vrow) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        v[0] = x.x; v[1] = x.y; v[C - 2] = x.z; v[C - 1] = x.w;
      } else {
        const float2 x = from >= 0 ? *reinterpret_cast<const float2*>(vrow) : make_float2(0.0f, 0.0f);
        v[0] = x.x; v[1] = x.y;
      }
    };
    // Keys that some of the rows do not see, later rows' or behind a window, enter with a weight of zero, and zero times
    // infinity is not zero: such a tile's values are looked through first, and if not all are finite each row takes its own.
    bool wild = false;
    if (last > p0 && (32 * tile + 31 > p0 || (a.window > 0 && 32 * tile <= last - a.window))) {
      float zeros = 0.0f;
#pragma unroll 8
      for (int jj = 0; jj < count; ++jj) {
        float v[C];
        value(jj, v);
#pragma unroll
        for (int c = 0; c < C; ++c) zeros = fmaf(v[c], 0.0f, zeros);
      }
      wild = __any_sync(0xffffffffu, zeros != 0.0f);
    }
    if (wild) {
#pragma unroll 1
      for (int jj = 0; jj < count; ++jj) {
        const int key = 32 * tile + jj;
        float v[C];
        value(jj, v);
#pragma unroll
        for (int i = 0; i < P; ++i) {
          const int p = p0 + (own + i) / group;
          if (key > p || (a.window > 0 && key <= p - a.window)) continue;
#pragma unroll
          for (int c = 0; c < C; ++c) acc[i][c] = fmaf(ps[i * 32 + jj], v[c], acc[i][c]);
        }
      }
      continue;
    }
#pragma unroll 2
    for (int jj = 0; jj < count; jj += 4) {
      float v[4][C];
#pragma unroll
      for (int u = 0; u < 4; ++u) value(jj + u, v[u]);
#pragma unroll
      for (int i = 0; i < P; ++i) {
        const float4 w = *reinterpret_cast<const float4*>(ps + i * 32 + jj);
#pragma unroll
        for (int c = 0; c < C; ++c)
          acc[i][c] = fmaf(w.w, v[3][c], fmaf(w.z, v[2][c], fmaf(w.y, v[1][c], fmaf(w.x, v[0][c], acc[i][c]))));
      }
    }
  }
  launch_dependents();
  if (ONE_TILE) {
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const int pair = own + i;
      if (pair >= pairs) break;
      float sum = warp_sum(l[i]);
      if (!(sum > 0.0f) || !isfinite(sum)) {
        if (lane == 0) publish_error(a.error, kAttentionDenominator);
        sum = 1.0f;
      }
      float* orow = a.out + (static_cast<size_t>(row + pair / group) * a.heads + g * group + pair % group) * HD + lane * C;
#pragma unroll
      for (int c = 0; c < C; ++c) orow[c] = acc[i][c] / sum;
    }
    return;
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const float total = warp_sum(l[i]);
    if (lane == 0) {
      ps[i] = m[i];
      ps[P + i] = total;
    }
#pragma unroll
    for (int c = 0; c < C; ++c) ks[i * HD + lane * C + c] = acc[i][c];
  }
  __syncthreads();
  for (int i = warp; i < pairs; i += kF32Warps) {
    float top = -INFINITY, sum = 0.0f, o[C];
#pragma unroll
    for (int c = 0; c < C; ++c) o[c] = 0.0f;
    const float* w0 = qs + kF32Pairs * HD;
#pragma unroll
    for (int w = 0; w < kF32Warps; ++w) top = fmaxf(top, w0[w * kF32Pairs * 34 + i]);
#pragma unroll
    for (int w = 0; w < kF32Warps; ++w) {
      const float mw = w0[w * kF32Pairs * 34 + i];
      const float f = mw == -INFINITY ? 0.0f : expf(mw - top);
      sum = fmaf(w0[w * kF32Pairs * 34 + P + i], f, sum);
#pragma unroll
      for (int c = 0; c < C; ++c) o[c] = fmaf(smem[w * 32 * LD + i * HD + lane * C + c], f, o[c]);
    }
    if (!(sum > 0.0f) || !isfinite(sum)) {
      if (lane == 0) publish_error(a.error, kAttentionDenominator);
      sum = 1.0f;
    }
    float* orow = a.out + (static_cast<size_t>(row + i / group) * a.heads + g * group + i % group) * HD + lane * C;
#pragma unroll
    for (int c = 0; c < C; ++c) orow[c] = o[c] / sum;
  }
}

// Block (row, kv head).  Rows that follow one another in a request go together, cut at positions that are multiples of
// the rows a block takes; the block of the first of them works, the others' have nothing to do.
template <int HD>
__global__ void __launch_bounds__(kF32Warps * 32)
paged_attention_f32_kernel(const F32AttentionArgs a) {
  extern __shared__ __align__(16) float smem[];
  wait_for_prior_kernels();
  const int t = blockIdx.x, g = blockIdx.y, group = a.heads / a.kv_heads, most = kF32Pairs / group;
  const int r = a.request_of_row[t];
  if (r < 0) return;                                       // a row of padding
  const int p0 = a.positions[t];
  if (p0 % most != 0 && t > 0 && a.request_of_row[t - 1] == r && a.positions[t - 1] + 1 == p0) return;
  int n = 1;
  while (n < most && (p0 + n) % most != 0 && t + n < a.rows && a.request_of_row[t + n] == r && a.positions[t + n] == p0 + n) ++n;
  const int* table = a.block_table + static_cast<size_t>(r) * a.table_width;
  const int lowest = a.window > 0 ? max(0, p0 - a.window + 1) : 0;
  if ((p0 + n - 1) / 32 == lowest / 32) f32_attend<HD, kF32FewPairs, true>(a, smem, t, p0, n * group, group, g, table);
  else if (n * group <= kF32FewPairs) f32_attend<HD, kF32FewPairs, false>(a, smem, t, p0, n * group, group, g, table);
  else f32_attend<HD, kF32Pairs, false>(a, smem, t, p0, n * group, group, g, table);
}

}  // namespace pih

using namespace pih;

template <int HD>
static void launch_f32_attention(cudaStream_t s, const F32AttentionArgs& a) {
  cudaFuncSetAttribute(paged_attention_f32_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       static_cast<int>(f32_attention_bytes<HD>()));
  launch_kernel(paged_attention_f32_kernel<HD>, dim3(a.rows, a.kv_heads), dim3(kF32Warps * 32), f32_attention_bytes<HD>(), s, a);
}

extern "C" int pih_paged_attention_generic(int dtype, const void* q, int q_stride, void* out,
                                           const void* cache, const int* block_table, int table_width,
                                           const int* request_of_row, const int* positions, int rows,
                                           int heads, int kv_heads, int head_dim, int page_size,
                                           int num_pages, float scale, int window, uint32_t* error,
                                           void* stream) {
  if (rows <= 0) return 0;
  if (heads <= 0 || kv_heads <= 0 || heads % kv_heads || head_dim <= 0 || page_size <= 0 ||
      table_width <= 0 || window < 0)
    return PIH_ERR_BAD_ARGUMENT;
  if (head_dim > 32 * kMaxDimPerLane) return PIH_ERR_UNSUPPORTED;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // 16-byte pieces of keys, up to 16 (row, head) pairs a block, blocks of kv heads along y
  if (dtype == PIH_F32 && (head_dim == 64 || head_dim == 128) && heads / kv_heads <= kF32Pairs && kv_heads <= 65535 &&
      reinterpret_cast<uintptr_t>(cache) % 16 == 0) {
    const F32AttentionArgs a = {static_cast<const float*>(q), q_stride, static_cast<float*>(out), static_cast<const float*>(cache),
                                block_table, table_width, request_of_row, positions, rows, heads, kv_heads, page_size, num_pages,
                                scale, window, error};
    if (head_dim == 64) launch_f32_attention<64>(s, a);
    else launch_f32_attention<128>(s, a);
    PIH_LAUNCH_CHECK();
    return 0;
  }
  const int warps = 4;
  const long long items = static_cast<long long>(rows) * heads;
  const unsigned blocks = static_cast<unsigned>((items + warps - 1) / warps);
  const size_t smem = static_cast<size_t>(warps) * head_dim * sizeof(float);
  if (dtype == PIH_F32)
    launch_kernel(paged_attention_generic_kernel<float>, dim3(blocks), dim3(warps * 32), smem, s, 
        static_cast<const float*>(q), q_stride, static_cast<float*>(out),
        static_cast<const float*>(cache), block_table, table_width, request_of_row, positions, rows,
        heads, kv_heads, head_dim, page_size, num_pages, scale, window, error);
  else if (dtype == PIH_BF16)
    launch_kernel(paged_attention_generic_kernel<__nv_bfloat16>, dim3(blocks), dim3(warps * 32), smem, s, 
        static_cast<const __nv_bfloat16*>(q), q_stride, static_cast<__nv_bfloat16*>(out),
        static_cast<const __nv_bfloat16*>(cache), block_table, table_width, request_of_row, positions,
        rows, heads, kv_heads, head_dim, page_size, num_pages, scale, window, error);
  else
    return PIH_ERR_BAD_ARGUMENT;
  PIH_LAUNCH_CHECK();
  return 0;
}
