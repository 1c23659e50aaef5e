// fp32 product C[m, n] = sum_k A[m, k] * B[n, k] (+ bias[n]), both operands with k contiguous: the forward
// product of a layer, and with transposed weights the gradient of its input.
//
// These shapes (thousands of rows, 256 to 512 columns, k of 256 to 512) are bound by the fp32 pipes, and the
// library's tiles for them reach 28-46 of the 74 TFLOP/s.  Here:
//   * k runs in pairs: fma.rn.f32x2 on the two halves of a 64-bit register, even k in one half and odd k in
//     the other, added at the end.  Operands are pairs as they lie in shared memory, so nothing is packed or
//     duplicated, and a multiply-add of two values takes one issue slot of the two cycles that the pipe is
//     busy: the loads from shared memory fit in between.
//   * tiles enter through cp.async (three stages of 16 k, rows padded to 20 words: the eight rows that a warp
//     reads of A, and the four of B, fall into different banks);
//   * B's rows are permuted on the way in, so that a thread owns four neighbouring columns and stores 16 bytes.
// Tiles of 128 x 128 (8 x 8 a thread) where they fill the chip, 64 x 64 (8 x 4 a thread) below; products too
// small for one tile per SM stay with the library.
#include "common.cuh"

namespace hc {

constexpr int kGemmK = 16, kGemmLd = 20, kGemmStages = 3;

struct GemmArgs {
  const float* a; int64_t lda; int64_t m;
  const float* b; int64_t ldb; int n;
  int k;
  const float* bias;
  float* c; int64_t ldc;
  int wide;        // 16-byte stores
};

__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
// 16 bytes, or zeros where the source is past the end of k
__device__ __forceinline__ void cp_async_or_zero(uint32_t dst, const float* src, bool take) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(take ? 16 : 0) : "memory");
}

template <int BM, int BN, int TM, int TN, int MIN_BLOCKS>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), MIN_BLOCKS) gemm_pairs_kernel(const GemmArgs g) {
  constexpr int TY = BM / TM, TX = BN / TN, kThreads = TY * TX, kStage = (BM + BN) * kGemmLd;
  constexpr int kChunks = (BM + BN) * (kGemmK / 4) / kThreads;
  static_assert((BM + BN) * (kGemmK / 4) % kThreads == 0 && TY % 8 == 0 && TX % 4 == 0 && TN % 4 == 0, "tile");
  extern __shared__ __align__(16) float sh[];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  // a warp covers 8 x 4 threads of the tile
  const int ty = warp / (TX / 4) * 8 + lane / 4, tx = warp % (TX / 4) * 4 + lane % 4;
  const int64_t m0 = (int64_t)blockIdx.y * BM;
  const int n0 = blockIdx.x * BN;

  const float* src[kChunks];
  uint32_t dst[kChunks];
  const int q = threadIdx.x % 4;        // the same k chunk in every row (kThreads is a multiple of 4)
#pragma unroll
  for (int i = 0; i < kChunks; ++i) {
    const int row = (threadIdx.x + i * kThreads) / 4;
    int slot = row;
    if (row < BM) {
      const int64_t r = m0 + row < g.m ? m0 + row : g.m - 1;
      src[i] = g.a + r * g.lda + 4 * q;
    } else {
      const int r = row - BM, c = n0 + r < g.n ? n0 + r : g.n - 1;
      src[i] = g.b + (int64_t)c * g.ldb + 4 * q;
      slot = BM + r / (4 * TX) * (4 * TX) + r % 4 * TX + r % (4 * TX) / 4;
    }
    dst[i] = (uint32_t)__cvta_generic_to_shared(sh + slot * kGemmLd + 4 * q);
  }
  const int tiles = (g.k + kGemmK - 1) / kGemmK;
  auto fetch = [&](int t) {
    if (t < tiles) {
      const bool take = t * kGemmK + 4 * q < g.k;
      const uint32_t to = (uint32_t)(t % kGemmStages * kStage * (int)sizeof(float));
#pragma unroll
      for (int i = 0; i < kChunks; ++i) cp_async_or_zero(dst[i] + to, src[i] + (take ? t * kGemmK : 0), take);
    }
    cp_async_commit();
  };
  unsigned long long acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
#pragma unroll
  for (int t = 0; t < kGemmStages - 1; ++t) fetch(t);
  for (int t = 0; t < tiles; ++t) {
    cp_async_wait<kGemmStages - 2>();
    __syncthreads();      // tile t has landed, and nobody reads the stage that is filled next
    fetch(t + kGemmStages - 1);
    const float* as = sh + t % kGemmStages * kStage + ty * kGemmLd;
    const float* bs = sh + t % kGemmStages * kStage + (BM + tx) * kGemmLd;
#pragma unroll
    for (int kk = 0; kk < kGemmK; kk += 4) {
      ulonglong2 av[TM], bv[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const ulonglong2*>(as + i * TY * kGemmLd + kk);
#pragma unroll
      for (int j = 0; j < TN; ++j)
        bv[j] = *reinterpret_cast<const ulonglong2*>(bs + (j / 4 * (4 * TX) + j % 4 * TX) * kGemmLd + kk);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) fma2(acc[i][j], av[i].x, bv[j].x);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) fma2(acc[i][j], av[i].y, bv[j].y);
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int h = 0; h < TN / 4; ++h) {
    const int col = n0 + h * 4 * TX + 4 * tx;
    float bias[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) bias[j] = g.bias && col + j < g.n ? __ldg(g.bias + col + j) : 0.f;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int64_t row = m0 + ty + i * TY;
      if (row >= g.m) continue;
      float v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const unsigned long long s = acc[i][h * 4 + j];
        v[j] = __uint_as_float((unsigned)s) + __uint_as_float((unsigned)(s >> 32)) + bias[j];
      }
      float* to = g.c + row * g.ldc + col;
      if (g.wide && col + 3 < g.n) {
        *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (col + j < g.n) to[j] = v[j];
      }
    }
  }
}

template <int BM, int BN, int TM, int TN, int MIN_BLOCKS>
static int run_gemm(const GemmArgs& g, cudaStream_t st) {
  static std::atomic<uint64_t> raised{0};
  constexpr int kBytes = kGemmStages * (BM + BN) * kGemmLd * (int)sizeof(float);
  auto kernel = gemm_pairs_kernel<BM, BN, TM, TN, MIN_BLOCKS>;
  raise_smem(kernel, kBytes, raised);
  const int64_t rows = ceil_div(g.m, BM);
  HC_REQUIRE(rows <= 65535, HC_ERR_UNSUPPORTED);
  kernel<<<dim3((unsigned)ceil_div(g.n, BN), (unsigned)rows), (BM / TM) * (BN / TN), kBytes, st>>>(g);
  HC_LAUNCH_OK();
  return 0;
}

}  // namespace hc

using namespace hc;

extern "C" int hc_gemm_fits(int64_t m, int32_t n, int32_t k) {
  if (m < 1 || n < 1 || k < 4 || k % 4) return 0;
  if (ceil_div(m, 128) * ceil_div(n, 128) >= 148) return ceil_div(m, 128) <= 65535 ? 2 : 0;
  return ceil_div(m, 64) * ceil_div(n, 64) >= 148 ? 1 : 0;
}

extern "C" int hc_gemm(const float* a, int64_t lda, int64_t m, const float* b, int64_t ldb, int32_t n, int32_t k,
                       const float* bias, float* c, int64_t ldc, void* stream) {
  const int fits = hc_gemm_fits(m, n, k);
  HC_REQUIRE(fits, HC_ERR_UNSUPPORTED);
  HC_REQUIRE(a && b && c, HC_ERR_NULL);
  HC_REQUIRE(lda >= k && ldb >= k && ldc >= n, HC_ERR_SIZE);
  HC_REQUIRE(lda % 4 == 0 && ldb % 4 == 0 && aligned16(a) && aligned16(b), HC_ERR_UNSUPPORTED);
  const GemmArgs g{a, lda, m, b, ldb, n, k, bias, c, ldc, ldc % 4 == 0 && aligned16(c)};
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return fits == 2 ? run_gemm<128, 128, 8, 8, 1>(g, st) : run_gemm<64, 64, 8, 4, 3>(g, st);
}
