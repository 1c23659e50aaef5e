// A barrier of all blocks of one cooperative launch, for kernels that replace a chain of tiny launches.
// The launch API guarantees that the blocks are resident together; the wait is bounded all the same,
// and a block whose wait runs out raises the flag that ends every other wait.
#pragma once
#include "common.cuh"

namespace hc {

constexpr int kGridSpin = 1 << 24;

struct GridSync {
  unsigned* word;      // [0] arrivals [1] a wait ran out; cleared by the caller in front of the launch
  unsigned round;
  __device__ explicit GridSync(unsigned* w) : word(w), round(0) {}
  // true: every block has arrived, and what it wrote before is visible
  __device__ __forceinline__ bool wait() {
    __shared__ bool ok;
    __syncthreads();
    ++round;
    if (threadIdx.x == 0) {
      __threadfence();      // cumulative: covers what the barrier above ordered before it
      const unsigned want = round * gridDim.x;
      atomicAdd(word, 1u);
      int spins = 0;
      ok = true;
      while (*reinterpret_cast<volatile unsigned*>(word) < want) {
        if (++spins > kGridSpin || *reinterpret_cast<volatile unsigned*>(word + 1) != 0u) {
          *reinterpret_cast<volatile unsigned*>(word + 1) = 1u;
          ok = false;
          break;
        }
      }
      __threadfence();
    }
    __syncthreads();
    return ok;
  }
};

// sum of v[0..n) and of v[0..upto), by the whole block
__device__ __forceinline__ void block_prefix(const int* v, int n, int upto, int* total, int* before) {
  __shared__ int sh[2];
  if (threadIdx.x < 2) sh[threadIdx.x] = 0;
  __syncthreads();
  int t = 0, b = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int x = __ldcg(v + i);
    t += x;
    if (i < upto) b += x;
  }
  t = __reduce_add_sync(kFull, t);
  b = __reduce_add_sync(kFull, b);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&sh[0], t);
    atomicAdd(&sh[1], b);
  }
  __syncthreads();
  *total = sh[0];
  *before = sh[1];
  __syncthreads();
}

// exclusive sum of a small count over the block's threads, and the block's total
template <int THREADS>
__device__ __forceinline__ int block_exclusive(int c, int* total) {
  __shared__ int part[THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = c;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int t = __shfl_up_sync(kFull, x, off);
    if (lane >= off) x += t;
  }
  if (lane == 31) part[warp] = x;
  __syncthreads();
  int before = 0, sum = 0;
#pragma unroll
  for (int w = 0; w < THREADS / 32; ++w) {
    const int v = part[w];
    if (w < warp) before += v;
    sum += v;
  }
  __syncthreads();
  *total = sum;
  return before + x - c;
}

// Cooperative launch behind a clear of the barrier's words.
template <typename... P>
inline int launch_together(void (*kernel)(P...), unsigned blocks, unsigned threads, size_t smem, unsigned* word,
                           cudaStream_t st, P... args) {
  HC_CUDA(cudaMemsetAsync(word, 0, 2 * sizeof(unsigned), st));
  void* list[] = {const_cast<void*>(static_cast<const void*>(&args))...};
  HC_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel), dim3(blocks), dim3(threads), list, smem, st));
  return 0;
}

}  // namespace hc
