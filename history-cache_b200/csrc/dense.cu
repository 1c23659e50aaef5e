// The small work around the dense products of a layer, and the loss.
//
// A layer's products are library calls; around them a step of 16 K rows ran some ten kernels of 2-8 us: two
// copies and a concatenation in front, ones-filled matrix-vector products and sums over slabs behind.  They
// are bound by launches and by latency, so each side is one or two launches here.
#include "common.cuh"

namespace hc {

// ---- [his | x], [wl | wr] and the bias in every row of the result -----------------------------------
// The product then adds onto the bias: as an epilogue the library runs it as a kernel of its own, 7 us a layer.
// One warp per row of either operand; a lane moves four values at a time (one where rows are no multiple of
// 16 bytes), four requests in flight.  Three layers of a step: 36 -> 12 us.
struct PackArgs {
  const float* his; int64_t his_stride;
  const void* x; int x_dtype; int64_t x_stride;
  int64_t n;
  int feat;
  float* rows;               // [n, 2 * feat]
  const float* wl; const float* wr; int hidden;
  float* w;                  // [hidden, 2 * feat]
  const float* bias;
  float* out;                // [n, hidden] = bias, or NULL
  int out_vec;
};

template <typename X, int V>
__global__ void __launch_bounds__(256) sage_pack_kernel(const PackArgs a) {
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
  const int lane = threadIdx.x & 31;
  if (row >= a.n + a.hidden) return;
  const bool weights = row >= a.n;
  const int64_t r = weights ? row - a.n : row;
  const float* left = weights ? a.wl + r * a.feat : a.his + r * a.his_stride;
  float* to = (weights ? a.w : a.rows) + r * 2 * a.feat;
  if (a.out && !weights) {
    if (a.out_vec)
      for (int c = lane; c < a.hidden / 4; c += 32)
        reinterpret_cast<float4*>(a.out + r * a.hidden)[c] = __ldg(reinterpret_cast<const float4*>(a.bias) + c);
    else
      for (int c = lane; c < a.hidden; c += 32) a.out[r * a.hidden + c] = __ldg(a.bias + c);
  }
  const int units = a.feat / V;
  using In = LaneVec<X, V * (int)sizeof(X)>;
  using F32 = LaneVec<float, V * 4>;
#pragma unroll 2
  for (int u = lane; u < units; u += 32) {
    F32 l;
    l.load(left + u * V);
    float lf[V], rf[V];
    l.unpack(lf);
    if (weights) {
      F32 b;
      b.load(a.wr + r * a.feat + u * V);
      b.unpack(rf);
    } else {
      In b;
      b.load(reinterpret_cast<const X*>(a.x) + r * a.x_stride + u * V);
      b.unpack(rf);
    }
    if constexpr (V == 1) {
      to[u] = lf[0];
      to[a.feat + u] = rf[0];
    } else {
      *reinterpret_cast<float4*>(to + u * 4) = make_float4(lf[0], lf[1], lf[2], lf[3]);
      *reinterpret_cast<float4*>(to + a.feat + u * 4) = make_float4(rf[0], rf[1], rf[2], rf[3]);
    }
  }
}

// ---- gradients of weights and bias from slabs ------------------------------------------------
// The weight gradient of tens of thousands of rows is cut into slabs (one batched product, see torch_ops.cpp).
// What is left: the sum over the slabs, the rows that fill no slab, and the column sums of the gradient for
// the bias.  Column sums need every block, so they start in a kernel of their own; its partial sums and the
// slabs are then added up by one launch, both in a fixed order.
constexpr int kColBlock = 1024;
constexpr int kColBlocks = 148;

// V columns a thread (4 where rows are whole 16-byte vectors), eight rows in flight
template <int V>
__global__ void __launch_bounds__(kColBlock)
    column_partials_kernel(const float* __restrict__ g, const int64_t n, const int cols, float* __restrict__ partial) {
  __shared__ float sh[kColBlock * V];
  const int64_t per = ceil_div(n, (int64_t)gridDim.x);
  const int64_t r0 = per * blockIdx.x, r1 = r0 + per < n ? r0 + per : n;
  for (int base = 0; base < cols; base += kColBlock * V) {
    const int width = (cols - base < kColBlock * V ? cols - base : kColBlock * V) / V;
    const int slots = kColBlock / width, slot = threadIdx.x / width, c = threadIdx.x - slot * width;
    float s[V];
#pragma unroll
    for (int q = 0; q < V; ++q) s[q] = 0.f;
    if (slot < slots) {
      constexpr int B = 8;
      for (int64_t r = r0 + slot; r < r1; r += (int64_t)B * slots) {
        LaneVec<float, 4 * V> v[B];
#pragma unroll
        for (int j = 0; j < B; ++j) {
          if (r + j * slots < r1) v[j].load(g + (r + j * slots) * cols + base + c * V);
          else v[j].clear();
        }
#pragma unroll
        for (int j = 0; j < B; ++j) v[j].add_to(s);
      }
    }
#pragma unroll
    for (int q = 0; q < V; ++q) sh[threadIdx.x * V + q] = s[q];
    __syncthreads();
    if (slot == 0) {
      for (int k = 1; k < slots; ++k)
#pragma unroll
        for (int q = 0; q < V; ++q) s[q] += sh[(k * width + c) * V + q];
#pragma unroll
      for (int q = 0; q < V; ++q) partial[(int64_t)blockIdx.x * cols + base + c * V + q] = s[q];
    }
    __syncthreads();
  }
}

struct SlabArgs {
  const float* parts; int slabs;           // [slabs, rows, cols]
  int64_t rows; int cols;
  const float* a; const float* b;          // rows that fill no slab: out[i, j] += sum_k a[k, i] * b[k, j]
  int rest;
  int split;                               // columns [0, split) go to left, the others to right
  float* left; float* right;
  const float* partial; int partials;      // column sums for the bias: [partials, rows]
  float* bias;
  int bias_blocks;
};

// blocks [0, bias_blocks): 32 columns of the bias each, eight threads a column; the others: one value a thread
// (the slabs' values are strided by whole matrices, so consecutive threads read consecutive words)
__global__ void __launch_bounds__(256) slab_sums_kernel(const SlabArgs s) {
  if ((int)blockIdx.x < s.bias_blocks) {
    __shared__ float sh[8][33];
    const int c = blockIdx.x * 32 + (threadIdx.x & 31), part = threadIdx.x / 32;
    float v[20], t = 0.f;
    for (int b0 = part; b0 < s.partials; b0 += 8 * 20) {
#pragma unroll
      for (int j = 0; j < 20; ++j)
        v[j] = c < s.rows && b0 + 8 * j < s.partials ? __ldg(s.partial + (int64_t)(b0 + 8 * j) * s.rows + c) : 0.f;
#pragma unroll
      for (int j = 0; j < 20; ++j) t += v[j];
    }
    sh[part][threadIdx.x & 31] = t;
    __syncthreads();
    if (part == 0 && c < s.rows) {
      for (int k = 1; k < 8; ++k) t += sh[k][threadIdx.x];
      s.bias[c] = t;
    }
    return;
  }
  const int64_t total = s.rows * s.cols, at = ((int64_t)blockIdx.x - s.bias_blocks) * 256 + threadIdx.x;
  if (at >= total) return;
  const int64_t i = at / s.cols;
  const int j = (int)(at - i * s.cols);
  float v[16], t = 0.f;
  for (int k0 = 0; k0 < s.slabs; k0 += 16) {
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = k0 + k < s.slabs ? __ldg(s.parts + (int64_t)(k0 + k) * total + at) : 0.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) t += v[k];
  }
  for (int k = 0; k < s.rest; ++k) t = fmaf(__ldg(s.a + k * s.rows + i), __ldg(s.b + (int64_t)k * s.cols + j), t);
  if (j < s.split) {
    if (s.left) s.left[i * s.split + j] = t;
  } else if (s.right) {
    s.right[i * (s.cols - s.split) + j - s.split] = t;
  }
}

// ---- negative log likelihood -------------------------------------------------------------------
// Mean of -logp[i, y[i]] over the rows whose label is not `ignore`, by one block: 1 000 rows are one round of
// two dependent loads.  torch's kernel takes 32 threads and 16 us for them.  Sums in double, in a fixed
// order.  A label outside the classes makes the loss NaN.
constexpr int kNllBlock = 1024;

__global__ void __launch_bounds__(kNllBlock)
    nll_kernel(const float* __restrict__ logp, const int64_t stride, const int64_t n, const int classes,
               const int64_t* __restrict__ y, const int64_t ignore, float* __restrict__ loss, float* __restrict__ count) {
  __shared__ double sums[32];
  __shared__ double counts[32];
  double s = 0.0, c = 0.0;
  for (int64_t i0 = threadIdx.x; i0 < n; i0 += 4 * kNllBlock) {
    int64_t t[4];
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) t[k] = i0 + k * kNllBlock < n ? y[i0 + k * kNllBlock] : ignore;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      v[k] = t[k] == ignore ? 0.f
             : t[k] >= 0 && t[k] < classes ? __ldg(logp + (i0 + k * kNllBlock) * stride + t[k]) : __int_as_float(0x7fffffff);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      s -= (double)v[k];
      c += t[k] == ignore ? 0.0 : 1.0;
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    s += __shfl_xor_sync(kFull, s, off);
    c += __shfl_xor_sync(kFull, c, off);
  }
  if ((threadIdx.x & 31) == 0) {
    sums[threadIdx.x / 32] = s;
    counts[threadIdx.x / 32] = c;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    s = sums[threadIdx.x];
    c = counts[threadIdx.x];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      s += __shfl_xor_sync(kFull, s, off);
      c += __shfl_xor_sync(kFull, c, off);
    }
    if (threadIdx.x == 0) {
      loss[0] = (float)(s / c);      // no labelled row: 0 / 0 = NaN, as torch's mean is
      count[0] = (float)c;
    }
  }
}

// the whole gradient in one pass: zeros, and -grad / count at the label
__global__ void __launch_bounds__(256)
    nll_bwd_kernel(const float* __restrict__ grad, const int64_t* __restrict__ y, const int64_t ignore,
                   const float* __restrict__ count, const int64_t n, const int classes, float* __restrict__ gx) {
  const int64_t at = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (at >= n * classes) return;
  const int64_t i = at / classes;
  const int c = (int)(at - i * classes);
  const int64_t t = __ldg(y + i);
  gx[at] = t == c && t != ignore ? -__ldg(grad) / __ldg(count) : 0.f;
}

}  // namespace hc

using namespace hc;

extern "C" int hc_sage_pack(const float* his, int64_t his_stride, const void* x, int32_t x_dtype, int64_t x_stride, int64_t n,
                            int32_t feat, float* rows, const float* wl, const float* wr, int32_t hidden, float* w,
                            const float* bias, float* out, void* stream) {
  HC_REQUIRE(n >= 0 && feat > 0 && hidden >= 0 && his_stride >= feat && x_stride >= feat, HC_ERR_SIZE);
  HC_REQUIRE(dtype_size(x_dtype) != 0, HC_ERR_DTYPE);
  HC_REQUIRE((n == 0 || (his && x && rows)) && (hidden == 0 || (wl && wr && w)), HC_ERR_NULL);
  if (n + hidden == 0) return 0;
  const int64_t blocks = ceil_div(n + hidden, 8);
  HC_REQUIRE(blocks <= 0x7fffffffLL, HC_ERR_SIZE);
  HC_REQUIRE(!out || bias, HC_ERR_NULL);
  const PackArgs a{his, his_stride, x, x_dtype, x_stride, n, feat, rows, wl, wr, hidden, w, bias, out,
                   hidden % 4 == 0 && aligned16(bias) && aligned16(out)};
  const bool vec = feat % 4 == 0 && his_stride % 4 == 0 && x_stride % 4 == 0 && aligned16(his) &&
                   aligned_to(x, 4 * dtype_size(x_dtype)) && aligned16(rows) && aligned16(wl) && aligned16(wr) && aligned16(w);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (x_dtype == HC_F16) {
    if (vec) sage_pack_kernel<__half, 4><<<(unsigned)blocks, 256, 0, st>>>(a);
    else sage_pack_kernel<__half, 1><<<(unsigned)blocks, 256, 0, st>>>(a);
  } else {
    if (vec) sage_pack_kernel<float, 4><<<(unsigned)blocks, 256, 0, st>>>(a);
    else sage_pack_kernel<float, 1><<<(unsigned)blocks, 256, 0, st>>>(a);
  }
  HC_LAUNCH_OK();
  return 0;
}

extern "C" int64_t hc_slab_sums_scratch_bytes(int64_t rows) { return kColBlocks * rows * (int64_t)sizeof(float); }

extern "C" int hc_slab_sums(const float* parts, int32_t slabs, int64_t rows, int32_t cols, const float* a, const float* b,
                            int32_t rest, int32_t split, float* left, float* right, const float* g, int64_t n, float* bias,
                            void* scratch, void* stream) {
  HC_REQUIRE(slabs >= 0 && rows > 0 && cols > 0 && rest >= 0 && split >= 0 && split <= cols && n >= 0, HC_ERR_SIZE);
  HC_REQUIRE(rows <= 0x7fffffffLL, HC_ERR_SIZE);
  const bool weights = left || right;
  HC_REQUIRE(!weights || ((slabs == 0 || parts) && (rest == 0 || (a && b))), HC_ERR_NULL);
  HC_REQUIRE(!bias || ((n == 0 || g) && scratch), HC_ERR_NULL);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  SlabArgs s{parts, slabs, rows, cols, a, b, rest, split, left, right, static_cast<float*>(scratch), 0, bias, 0};
  if (bias) {
    const int64_t want = ceil_div(n, 32);      // a block takes at least 32 rows: fewer partial sums for few rows
    s.partials = (int)(want < 1 ? 1 : want < kColBlocks ? want : kColBlocks);
    s.bias_blocks = (int)ceil_div(rows, 32);
    auto* to = static_cast<float*>(scratch);
    if (rows % 4 == 0 && aligned16(g)) column_partials_kernel<4><<<s.partials, kColBlock, 0, st>>>(g, n, (int)rows, to);
    else column_partials_kernel<1><<<s.partials, kColBlock, 0, st>>>(g, n, (int)rows, to);
  }
  const int64_t blocks = s.bias_blocks + (weights ? ceil_div(rows * cols, 256) : 0);
  HC_REQUIRE(blocks <= 0x7fffffffLL, HC_ERR_SIZE);
  if (blocks) slab_sums_kernel<<<(unsigned)blocks, 256, 0, st>>>(s);
  HC_LAUNCH_OK();
  return 0;
}

extern "C" int hc_nll_fwd(const float* logp, int64_t stride, int64_t n, int32_t classes, const int64_t* y, int64_t ignore,
                          float* loss, float* count, void* stream) {
  HC_REQUIRE(n >= 0 && classes > 0 && stride >= classes, HC_ERR_SIZE);
  HC_REQUIRE((n == 0 || (logp && y)) && loss && count, HC_ERR_NULL);
  nll_kernel<<<1, kNllBlock, 0, reinterpret_cast<cudaStream_t>(stream)>>>(logp, stride, n, classes, y, ignore, loss, count);
  HC_LAUNCH_OK();
  return 0;
}

extern "C" int hc_nll_bwd(const float* grad, const int64_t* y, int64_t ignore, const float* count, int64_t n, int32_t classes,
                          float* grad_logp, void* stream) {
  HC_REQUIRE(n >= 0 && classes > 0, HC_ERR_SIZE);
  if (n == 0) return 0;
  HC_REQUIRE(grad && y && count && grad_logp, HC_ERR_NULL);
  const int64_t blocks = ceil_div(n * classes, 256);
  HC_REQUIRE(blocks <= 0x7fffffffLL, HC_ERR_SIZE);
  nll_bwd_kernel<<<(unsigned)blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(grad, y, ignore, count, n, classes,
                                                                                     grad_logp);
  HC_LAUNCH_OK();
  return 0;
}
