// The gated delta rule by chunks of 64 rows (delta_chunks.cu).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace pih {

constexpr int kDeltaSmallRows = 16;                        // requests of at most this many rows go token by token

struct DeltaChunkArgs {
  const float* q;                                          // unit length, scaled: [rows, kv_heads, dim]
  const float* k;
  const float* qk;                                         // q . k: [rows, kv_heads]
  const float* decay;                                      // decay - 1: [rows, heads, dim] (channels) or [rows, heads]
  const float* beta;                                       // [rows, heads]
  const __nv_bfloat16* v;
  long long ldv;
  float* out;                                              // [rows, heads, vdim]
  float* state;
  long long state_stride;
  float* scratch;
  const int* cu_q;
  const int* state_slots;
  int requests, heads, kv_heads, vdim;
};

// Sizes that go by chunks, and the fp32 numbers of scratch that a step of ``rows`` rows needs.
bool delta_takes_chunks(int heads, int dim, int vdim);
long long delta_chunk_scratch(int rows, int requests, int heads, int dim, int vdim);
int launch_delta_chunks(cudaStream_t s, DeltaChunkArgs p, int dim, bool channels, int rows);

}  // namespace pih
