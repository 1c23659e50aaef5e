// Adam (Kingma and Ba, "Adam: A Method for Stochastic Optimization", algorithm 1) over all parameters of a
// model in one launch.
//
// torch's fused optimizer step cuts tensors into pieces of 64 K values: the half million parameters of a
// three-layer model keep a handful of blocks busy (38 us), and its host side takes some 100 us of an eager
// step.  Here a block takes 1 024 values, whichever tensor they belong to.  Bias corrections are computed
// in double from the device-side step count, so that a captured step stays right.
#include "common.cuh"

namespace hc {

constexpr int kAdamTensors = 48;
constexpr int kAdamBlock = 256;
constexpr int kAdamChunk = 4 * kAdamBlock;

struct AdamList {
  float* param[kAdamTensors];
  const float* grad[kAdamTensors];
  float* avg[kAdamTensors];
  float* avg_sq[kAdamTensors];
  float* step[kAdamTensors];
  int64_t numel[kAdamTensors];
  int first_block[kAdamTensors + 1];
  int n;
};

__global__ void adam_count_kernel(const AdamList l) {
  const int t = threadIdx.x;
  if (t < l.n) l.step[t][0] += 1.f;
}

__global__ void __launch_bounds__(kAdamBlock)
    adam_kernel(const AdamList l, const double lr, const double beta1, const double beta2, const double eps) {
  int t = 0;
  while (t + 1 < l.n && (int)blockIdx.x >= l.first_block[t + 1]) ++t;
  // fp32 throughout, as torch's step is: 1 - beta and the corrections 1 - beta^t come from the same rounded
  // beta, so that the factors which they share cancel in m / sqrt(v)
  const float b1 = (float)beta1, b2 = (float)beta2, c1 = 1.f - b1, c2 = 1.f - b2, e = (float)eps;
  __shared__ float step_size, root;
  if (threadIdx.x == 0) {
    const double k = (double)l.step[t][0];
    step_size = (float)lr / (1.f - (float)pow((double)b1, k));
    root = sqrtf(1.f - (float)pow((double)b2, k));
  }
  __syncthreads();
  const int64_t base = (int64_t)((int)blockIdx.x - l.first_block[t]) * kAdamChunk;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t i = base + k * kAdamBlock + threadIdx.x;
    if (i >= l.numel[t]) break;
    const float g = l.grad[t][i];
    const float m = fmaf(b1, l.avg[t][i], c1 * g);
    const float v = fmaf(b2, l.avg_sq[t][i], c2 * g * g);
    l.avg[t][i] = m;
    l.avg_sq[t][i] = v;
    l.param[t][i] -= step_size * m / (sqrtf(v) / root + e);
  }
}

}  // namespace hc

using namespace hc;

extern "C" int hc_adam_step(void* const* params, const void* const* grads, void* const* avgs, void* const* avg_sqs,
                            void* const* steps, const int64_t* numels, int32_t n, double lr, double beta1, double beta2,
                            double eps, void* stream) {
  HC_REQUIRE(n >= 0, HC_ERR_SIZE);
  if (n == 0) return 0;
  HC_REQUIRE(params && grads && avgs && avg_sqs && steps && numels, HC_ERR_NULL);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  for (int32_t first = 0; first < n; first += kAdamTensors) {
    AdamList l;
    l.n = n - first < kAdamTensors ? n - first : kAdamTensors;
    int64_t blocks = 0;
    for (int k = 0; k < l.n; ++k) {
      l.param[k] = static_cast<float*>(params[first + k]);
      l.grad[k] = static_cast<const float*>(grads[first + k]);
      l.avg[k] = static_cast<float*>(avgs[first + k]);
      l.avg_sq[k] = static_cast<float*>(avg_sqs[first + k]);
      l.step[k] = static_cast<float*>(steps[first + k]);
      l.numel[k] = numels[first + k];
      HC_REQUIRE(l.param[k] && l.grad[k] && l.avg[k] && l.avg_sq[k] && l.step[k] && l.numel[k] > 0, HC_ERR_NULL);
      l.first_block[k] = (int)blocks;
      blocks += ceil_div(l.numel[k], kAdamChunk);
      HC_REQUIRE(blocks <= 0x7fffffffLL, HC_ERR_SIZE);
    }
    adam_count_kernel<<<1, 64, 0, st>>>(l);
    adam_kernel<<<(unsigned)blocks, kAdamBlock, 0, st>>>(l, lr, beta1, beta2, eps);
  }
  HC_LAUNCH_OK();
  return 0;
}
