/*
 * kernels_queue.cu - the small kernels between and before the transport
 * phases of both precisions: the order of the tail list and the chunk table.
 * A file of their own, since CUDA loads a file's kernels when the first of
 * them is used: an FP64 run does not load the FP32 transport for them.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "geo_fp32.cuh"
#include "kernels.h"

namespace ptg {

namespace {
/* Hand-over c of the tail list: its slot (front list, then back list). */
__device__ __forceinline__ int tail_slot(int c, int nlong, int tail_cap) {
  return c < nlong ? c : tail_cap - 1 - (c - nlong);
}

/* One thread per hand-over: the bucket offsets from the top bucket down
   (every block from the histogram), then the slot to its bucket's range. */
__global__ void k_order_scatter(const float4* __restrict__ tail, int units, int tail_cap,
                                const int* __restrict__ queue, const int* __restrict__ hist,
                                int* __restrict__ cursor, int* __restrict__ order) {
  __shared__ int h[kOrderBuckets];
  const int nlong = min(queue[2], tail_cap);
  const int ntail = nlong + min(queue[4], tail_cap - nlong);
  if ((int)(blockIdx.x * blockDim.x) >= ntail) return;
  for (int b = threadIdx.x; b < kOrderBuckets; b += blockDim.x) h[b] = hist[b];
  __syncthreads();
  if (threadIdx.x == 0) {
    int run = 0;
    for (int b = kOrderBuckets - 1; b >= 0; --b) {
      const int n = h[b];
      h[b] = run;
      run += n;
    }
  }
  __syncthreads();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ntail) return;
  const int slot = tail_slot(c, nlong, tail_cap);
  const int b = reinterpret_cast<const int*>(tail + (size_t)units * slot + 6)[2];
  order[h[b] + atomicAdd(&cursor[b], 1)] = slot;
}
}  // namespace

/* Chunk table of a run whose kernels read one (kChunkTableExt). */
__global__ void k_expand_chunks(const ChunkQueue q, int nchunk, int4* __restrict__ chunks) {
  for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < nchunk;
       c += (long long)gridDim.x * blockDim.x) {
    const int3 v = queue_chunk(q, (int)c);
    chunks[c] = make_int4(v.x, v.y, v.z, 0);
  }
}

cudaError_t launch_expand_chunks(const ChunkQueue& q, int nchunk, int4* chunks, cudaStream_t st) {
  if (nchunk <= 0) return cudaSuccess;
  const int blocks = (nchunk + 255) / 256;
  k_expand_chunks<<<blocks < 4096 ? blocks : 4096, 256, 0, st>>>(q, nchunk, chunks);
  return cudaGetLastError();
}

cudaError_t launch_tail_order(const float4* tail, int units, int tail_cap, const int* queue,
                              int32_t* order, int32_t* hist, cudaStream_t st) {
  const unsigned blocks = (unsigned)((tail_cap + 255) / 256);
  k_order_scatter<<<blocks, 256, 0, st>>>(tail, units, tail_cap, queue, hist, hist + kOrderBuckets,
                                          order);
  return cudaGetLastError();
}

}  // namespace ptg
