// Shared device/host helpers for libhiscache_b200 (sm_100a only).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "hiscache_b200.h"

#define HC_CUDA(call)                        \
  do {                                       \
    cudaError_t hc_e_ = (call);              \
    if (hc_e_ != cudaSuccess) return (int)hc_e_; \
  } while (0)

// Launch errors are read with cudaPeekAtLastError so that a sticky error left
// by somebody else's kernel is reported, not swallowed.
#define HC_LAUNCH_OK()                           \
  do {                                           \
    cudaError_t hc_e_ = cudaPeekAtLastError();   \
    if (hc_e_ != cudaSuccess) return (int)hc_e_; \
  } while (0)

#define HC_REQUIRE(cond, err) \
  do {                        \
    if (!(cond)) return -(err); \
  } while (0)

namespace hc {

constexpr int kWarp = 32;
constexpr unsigned kFull = 0xffffffffu;

__host__ __device__ inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline bool aligned_to(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }
inline int dtype_size(int dt) { return dt == HC_F32 ? 4 : (dt == HC_F16 ? 2 : 0); }

// Raises a kernel's shared-memory limit, once per kernel (`done` is its own) and device; not a stream
// operation, so it may happen during a capture.
template <typename K>
inline void raise_smem(K kernel, int bytes, std::atomic<uint64_t>& done) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev > 63) dev = 63;
  if (done.load(std::memory_order_relaxed) >> dev & 1) return;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess)
    done.fetch_or(1ull << dev, std::memory_order_relaxed);
}

// 64-bit shuffle (two 32-bit shuffles).
__device__ __forceinline__ int64_t shfl64(int64_t v, int src) {
  return __shfl_sync(kFull, (long long)v, src);
}

// Element load with run-time dtype, converted to fp32.
__device__ __forceinline__ float load_as_f32(const void* base, int dt, int64_t off) {
  return dt == HC_F16 ? __half2float(reinterpret_cast<const __half*>(base)[off])
                      : reinterpret_cast<const float*>(base)[off];
}
__device__ __forceinline__ void store_from_f32(void* base, int dt, int64_t off, float v) {
  if (dt == HC_F16)
    reinterpret_cast<__half*>(base)[off] = __float2half_rn(v);
  else
    reinterpret_cast<float*>(base)[off] = v;
}

// 16-byte read-only load.
__device__ __forceinline__ uint4 ldg16(const void* p) {
  return __ldg(reinterpret_cast<const uint4*>(p));
}

// Unpack a 16-byte vector of T into fp32 values.
template <typename T>
struct Vec16;
template <>
struct Vec16<float> {
  static constexpr int kElems = 4;
  __device__ __forceinline__ static void unpack(const uint4& v, float* f) {
    f[0] = __uint_as_float(v.x);
    f[1] = __uint_as_float(v.y);
    f[2] = __uint_as_float(v.z);
    f[3] = __uint_as_float(v.w);
  }
};
template <>
struct Vec16<__half> {
  static constexpr int kElems = 8;
  __device__ __forceinline__ static void unpack(const uint4& v, float* f) {
    const __half2* h = reinterpret_cast<const __half2*>(&v);
    float2 a = __half22float2(h[0]), b = __half22float2(h[1]);
    float2 c = __half22float2(h[2]), d = __half22float2(h[3]);
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
    f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
  }
};

// acc0 += low half of the word, acc1 += high half, with the mixed-precision add of sm_100 (f32 += f16
// in one instruction; the widening is exact, so the result equals convert-then-add).
#define HC_MIXED_ADD2(a0, a1, word)                                                   \
  asm("{.reg .b16 lo, hi; mov.b32 {lo, hi}, %2; add.f32.f16 %0, lo, %0; "             \
      "add.f32.f16 %1, hi, %1;}"                                                      \
      : "+f"(a0), "+f"(a1)                                                            \
      : "r"(word))

// What one lane moves of a row per request: VB bytes (16, 8, 4 or 2) of elements of type T.  Rows
// whose length or address is no multiple of 16 bytes are moved in the widest unit that divides both.
template <typename T, int VB>
struct LaneVec {
  static constexpr int kElems = VB / (int)sizeof(T);
  static constexpr int kWords = VB >= 4 ? VB / 4 : 1;
  uint32_t w[kWords];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < kWords; ++i) w[i] = 0u;
  }
  __device__ __forceinline__ void load(const void* p) {
    if constexpr (VB == 16) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
      w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    } else if constexpr (VB == 8) {
      const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
      w[0] = v.x; w[1] = v.y;
    } else if constexpr (VB == 4) {
      w[0] = __ldg(reinterpret_cast<const uint32_t*>(p));
    } else {
      w[0] = __ldg(reinterpret_cast<const uint16_t*>(p));
    }
  }
  // read once: not kept in the L1, first to leave the L2 (`policy` from l2_policy(true))
  __device__ __forceinline__ void load_once(const void* p, uint64_t policy) {
    static_assert(VB == 16, "wide units only");
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "l"(p), "l"(policy));
  }
  __device__ __forceinline__ void load_shared(const void* p) {
    if constexpr (VB == 16) {
      const uint4 v = *reinterpret_cast<const uint4*>(p);
      w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    } else if constexpr (VB == 8) {
      const uint2 v = *reinterpret_cast<const uint2*>(p);
      w[0] = v.x; w[1] = v.y;
    } else {
      w[0] = *reinterpret_cast<const uint32_t*>(p);
    }
  }
  __device__ __forceinline__ void unpack(float* f) const {
    if constexpr (sizeof(T) == 4) {
#pragma unroll
      for (int i = 0; i < kWords; ++i) f[i] = __uint_as_float(w[i]);
    } else if constexpr (VB == 2) {
      f[0] = __half2float(__ushort_as_half((unsigned short)w[0]));
    } else {
#pragma unroll
      for (int i = 0; i < kWords; ++i) {
        const float2 p = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
        f[2 * i] = p.x;
        f[2 * i + 1] = p.y;
      }
    }
  }
  __device__ __forceinline__ void add_to(float* acc) const {
    if constexpr (sizeof(T) == 4) {
#pragma unroll
      for (int i = 0; i < kWords; ++i) acc[i] += __uint_as_float(w[i]);
    } else if constexpr (VB == 2) {
      acc[0] += __half2float(__ushort_as_half((unsigned short)w[0]));
    } else {
#pragma unroll
      for (int i = 0; i < kWords; ++i) HC_MIXED_ADD2(acc[2 * i], acc[2 * i + 1], w[i]);
    }
  }
};

// 4-, 8- or 16-byte asynchronous copy of one lane into shared memory (past the L1 where it can)
template <int VB>
__device__ __forceinline__ void cp_async(uint32_t dst_smem, const void* src) {
  if constexpr (VB == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst_smem), "l"(src), "n"(VB) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Store of N consecutive fp32 values (N * 4 bytes aligned, at most 16) under an L2 policy.
template <int N>
__device__ __forceinline__ void store_f32(float* p, const float* f, uint64_t policy) {
  if constexpr (N >= 4) {
#pragma unroll
    for (int i = 0; i < N; i += 4)
      asm volatile("st.global.L2::cache_hint.v4.f32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(p + i), "f"(f[i]), "f"(f[i + 1]),
                   "f"(f[i + 2]), "f"(f[i + 3]), "l"(policy) : "memory");
  } else if constexpr (N == 2) {
    asm volatile("st.global.L2::cache_hint.v2.f32 [%0], {%1, %2}, %3;" ::"l"(p), "f"(f[0]), "f"(f[1]), "l"(policy)
                 : "memory");
  } else {
    asm volatile("st.global.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(p), "f"(f[0]), "l"(policy) : "memory");
  }
}
// evict-first for results that will not stay in the L2 anyway, so that they do not push out the rows
// the kernel still gathers; the default otherwise
__device__ __forceinline__ uint64_t l2_policy(bool stream) {
  uint64_t p;
  if (stream)
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  else
    asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// Vectorised fp32 reduction into global memory (one 16-byte transaction).
__device__ __forceinline__ void red_add_v4(float* addr, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b),
               "f"(c), "f"(d)
               : "memory");
}

// fp32 reductions of N = 1, 2 or 4 consecutive values
template <int N>
__device__ __forceinline__ void red_add(float* p, const float* f) {
  if constexpr (N == 4)
    red_add_v4(p, f[0], f[1], f[2], f[3]);
  else if constexpr (N == 2)
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(f[0]), "f"(f[1]) : "memory");
  else
    asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(f[0]) : "memory");
}

// ---- bulk-copy engine (TMA, untiled cp.async.bulk) and mbarrier helpers -----
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void bulk_load(uint32_t dst_smem, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst_smem),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void bulk_store(void* dst, uint32_t src_smem, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src_smem),
               "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}


// ---- the library's fixed score reduction --------------------------------
// Element e of a row belongs to lane (e/4) mod 32; a lane adds its terms in
// increasing e with separately rounded multiply and add; partial sums are
// combined by an xor butterfly; L2 ends with a correctly rounded sqrt.
__device__ __forceinline__ float score_term(float acc, float x, int kind) {
  return kind == HC_SCORE_L2 ? __fadd_rn(acc, __fmul_rn(x, x)) : __fadd_rn(acc, fabsf(x));
}
__device__ __forceinline__ float score_finish(float partial, int kind) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) partial = __fadd_rn(partial, __shfl_xor_sync(kFull, partial, off));
  return kind == HC_SCORE_L2 ? __fsqrt_rn(partial) : partial;
}
__device__ __forceinline__ float row_score(const float* row, int feat, int kind, int lane) {
  float acc = 0.f;
  for (int c0 = 0; c0 < feat; c0 += 128) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      int e = c0 + 4 * lane + k;
      if (e < feat) acc = score_term(acc, row[e], kind);
    }
  }
  return score_finish(acc, kind);
}

// splitmix64 finaliser: the owner hash of the sharded table.
__host__ __device__ inline uint64_t mix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

}  // namespace hc
