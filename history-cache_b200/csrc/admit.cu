// Admission scores, quantile threshold, deterministic admission with history
// writeback, and eviction.
//
// Replaces record_history_kernel_used_mask (src/cpp/src/grad_check.cu:6-68)
// and the torch arithmetic of HistoryCache.update_history
// (hiscache/history_cache.py:180-254) and HistoryTable.record_history /
// evict_by_* (hiscache/history_table.py:128-254).  The reference takes ring
// slots with atomicInc in warp-scheduling order; here slots follow an
// exclusive scan of the admission mask, so the remaps are reproducible.
#include "grid_sync.cuh"

namespace hc {

// ---------------------------------------------------------------------------
// scores
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
    score_rows_kernel(const float* __restrict__ x, int64_t n, int feat, int64_t stride, int kind,
                      float* __restrict__ score) {
  const int lane = threadIdx.x & 31;
  const int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (r >= n) return;
  const float s = row_score(x + r * stride, feat, kind, lane);
  if (lane == 0) score[r] = s;
}

// ---------------------------------------------------------------------------
// quantile threshold: exact radix select of two order statistics + lerp
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t order_key(float x) {
  if (x != x) return 0xFFFFFFFFu;  // NaN sorts last
  const uint32_t b = __float_as_uint(x);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_to_float(uint32_t k) {
  const uint32_t b = (k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k;
  return __uint_as_float(b);
}

// rank = q * (n - 1) in fp32 and the two order statistics around it (torch.quantile)
struct Ranks {
  int64_t n, k_lo, k_hi;
  float w;
};
__device__ __forceinline__ Ranks quantile_ranks(int64_t n_all, const int64_t* n_dev, float q) {
  // with n_dev the quantile is taken over the *n_dev smallest of the n_all scores: the caller
  // sets the scores of padding rows to +inf, which sorts them last
  Ranks r;
  r.n = n_all;
  if (n_dev) {
    r.n = n_dev[0];
    if (r.n > n_all) r.n = n_all;
  }
  if (r.n < 1) {
    r.k_lo = r.k_hi = 0;
    r.w = 0.f;
    return r;
  }
  const float pos = __fmul_rn(q, (float)(r.n - 1));
  r.k_lo = (int64_t)pos;  // truncation, pos >= 0
  if (r.k_lo > r.n - 1) r.k_lo = r.n - 1;
  if (r.k_lo < 0) r.k_lo = 0;
  r.k_hi = (int64_t)ceilf(pos);
  if (r.k_hi > r.n - 1) r.k_hi = r.n - 1;
  if (r.k_hi < 0) r.k_hi = 0;
  r.w = __fsub_rn(pos, (float)r.k_lo);
  return r;
}
__device__ __forceinline__ float quantile_lerp(uint32_t key_lo, uint32_t key_hi, float w) {
  const float lo = key_to_float(key_lo), hi = key_to_float(key_hi);
  const float diff = __fsub_rn(hi, lo);
  // torch's lerp with its fused multiply-add (CPU AVX2+ and CUDA builds)
  return fabsf(w) < 0.5f ? __fmaf_rn(w, diff, lo) : __fmaf_rn(-diff, __fsub_rn(1.f, w), hi);
}

// ---- up to kSelSmall scores: one block, keys staged once in shared memory ----------------
// One global read brings the keys into shared memory and finds the bits in which they differ (scores of
// a batch have nearly the same exponent).  A histogram of the highest 11 of those bits leaves a bin of
// a few dozen keys around the wanted rank; these are collected and ranked against each other.  A bin of
// more than 1 024 keys (ties) is cut by another histogram.  16 K scores: 8.2 us with four 8-bit passes.
// With `valid`, rows whose byte is 0 count as +inf and the quantile is over the others.
constexpr int kSelSmall = 48 * 1024;
constexpr int kSelThreads = 1024;
constexpr int kSelBins = 2048;
constexpr uint32_t kInfKey = 0xFF800000u;

__global__ void __launch_bounds__(kSelThreads)
    select_small_kernel(const float* __restrict__ score, int64_t n_all, const int64_t* n_dev,
                        const uint8_t* __restrict__ valid, float q, float* __restrict__ thres) {
  extern __shared__ uint32_t keys[];   // [n_all]
  __shared__ uint32_t hist[kSelBins];
  __shared__ uint32_t picked[kSelThreads];
  __shared__ uint32_t bcast[3];
  __shared__ uint32_t range[2];
  __shared__ uint32_t answer[2];
  __shared__ unsigned n_picked;
  __shared__ int counted;
  __shared__ int64_t n_valid;
  const int n = (int)n_all;
  if (threadIdx.x == 0) {
    range[0] = 0xFFFFFFFFu;
    range[1] = 0u;
    counted = 0;
  }
  __syncthreads();
  int has_nan = 0, mine = 0;
  uint32_t low = 0xFFFFFFFFu, high = 0u;
  constexpr int B = 8;      // loads in flight: the read is most of the call
  for (int i0 = threadIdx.x; i0 < n; i0 += B * kSelThreads) {
    float v[B];
    bool ok[B];
#pragma unroll
    for (int j = 0; j < B; ++j) {
      const int i = i0 + j * kSelThreads;
      ok[j] = i < n && (!valid || valid[i] != 0);
      v[j] = i < n ? score[i] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < B; ++j) {
      const int i = i0 + j * kSelThreads;
      if (i >= n) break;
      has_nan |= ok[j] && (v[j] != v[j]);
      const uint32_t key = ok[j] ? order_key(v[j]) : kInfKey;
      keys[i] = key;
      if (ok[j]) {      // the ranks asked for lie among these keys
        low = key < low ? key : low;
        high = key > high ? key : high;
      }
      mine += ok[j];
    }
  }
  low = __reduce_min_sync(kFull, low);
  high = __reduce_max_sync(kFull, high);
  mine = __reduce_add_sync(kFull, mine);
  if ((threadIdx.x & 31) == 0) {
    atomicMin(&range[0], low);
    atomicMax(&range[1], high);
    atomicAdd(&counted, mine);
  }
  has_nan = __syncthreads_or(has_nan);
  if (valid) {
    if (threadIdx.x == 0) n_valid = counted;
    n_dev = &n_valid;
    __syncthreads();
  }
  const Ranks rk = quantile_ranks(n_all, n_dev, q);
  if (rk.n < 1) {
    if (threadIdx.x == 0) thres[0] = __int_as_float(0x7fc00000);
    return;
  }
  uint32_t k = (uint32_t)rk.k_lo;      // rank among the keys of the current prefix
  // a caller's n_dev may reach into its padding: then the full range counts
  const bool all_in = valid != nullptr || n_dev == nullptr;
  const uint32_t top = all_in ? range[1] : 0xFFFFFFFFu;
  const uint32_t base = range[0] < top ? range[0] : top;
  int bits = 32 - __clz(base ^ top);           // low bits in which keys differ
  if (!all_in) bits = 32;
  uint32_t mask = bits >= 32 ? 0u : ~((1u << bits) - 1u);
  uint32_t prefix = base & mask;
  uint32_t inside = (uint32_t)n;      // keys that carry the current prefix
  while (bits > 0 && inside > kSelThreads) {
    const int take = bits < 11 ? bits : 11, shift = bits - take;
    const uint32_t digits = (1u << take) - 1u;
    for (int i = threadIdx.x; i < kSelBins; i += kSelThreads) hist[i] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += kSelThreads) {
      const uint32_t key = keys[i];
      if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & digits], 1u);
    }
    __syncthreads();
    const uint32_t c0 = hist[2 * threadIdx.x], c1 = hist[2 * threadIdx.x + 1];
    int all;
    const uint32_t run = (uint32_t)block_exclusive<kSelThreads>((int)(c0 + c1), &all);
    if (k >= run && k < run + c0 + c1) {      // the wanted key is in one of this thread's two bins
      const bool second = k >= run + c0;
      bcast[0] = 2 * threadIdx.x + (second ? 1u : 0u);
      bcast[1] = run + (second ? c0 : 0u);
      bcast[2] = second ? c1 : c0;
    }
    __syncthreads();
    prefix |= bcast[0] << shift;
    mask |= digits << shift;
    k -= bcast[1];
    inside = bcast[2];
    bits = shift;
    __syncthreads();
  }
  // the keys of the last bin against each other; the smallest key above the bin for the second statistic
  if (threadIdx.x == 0) {
    n_picked = 0;
    answer[0] = prefix;        // bits == 0: every key of the bin is this one
    answer[1] = prefix;
    range[1] = 0xFFFFFFFFu;
  }
  __syncthreads();
  uint32_t above = 0xFFFFFFFFu;
  for (int i = threadIdx.x; i < n; i += kSelThreads) {
    const uint32_t key = keys[i];
    if ((key & mask) == prefix) {
      if (bits > 0) picked[atomicAdd(&n_picked, 1u)] = key;
    } else if (key > prefix && key < above) {
      above = key;
    }
  }
  above = __reduce_min_sync(kFull, above);
  if ((threadIdx.x & 31) == 0) atomicMin(&range[1], above);
  __syncthreads();
  const uint32_t k_hi = k + (uint32_t)(rk.k_hi - rk.k_lo);
  if (bits > 0 && threadIdx.x < n_picked) {
    const uint32_t key = picked[threadIdx.x];
    uint32_t rank = 0;
    for (unsigned j = 0; j < n_picked; ++j) {
      const uint32_t o = picked[j];
      rank += o < key || (o == key && j < threadIdx.x);
    }
    if (rank == k) answer[0] = key;
    if (rank == k_hi) answer[1] = key;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t key_lo = answer[0], key_hi = k_hi < inside ? answer[1] : range[1];
    thres[0] = has_nan ? __int_as_float(0x7fc00000) : quantile_lerp(key_lo, key_hi, rk.w);
  }
}

// ---- any size: histograms by many blocks, digit choice by one ----------------------------
// Both order statistics descend together (two prefixes); four passes of
//   sel_hist (grid over the scores) -> sel_pick (one block), state in caller scratch.
struct SelState {
  long long n_valid;     // rows of a masked call
  uint32_t prefix[2];
  uint32_t mask;
  int has_nan;
  long long k[2];
  uint32_t hist[2][256];
};

__global__ void __launch_bounds__(256)
    sel_count_kernel(SelState* st, const uint8_t* __restrict__ valid, int64_t n) {
  int c = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    c += valid[i] != 0;
  c = __reduce_add_sync(kFull, c);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(reinterpret_cast<unsigned long long*>(&st->n_valid), (unsigned long long)c);
}

__global__ void __launch_bounds__(256) sel_init_kernel(SelState* st, int64_t n_all, const int64_t* n_dev, float q) {
  const Ranks rk = quantile_ranks(n_all, n_dev, q);
  if (threadIdx.x == 0) {
    st->prefix[0] = st->prefix[1] = 0;
    st->mask = 0;
    st->has_nan = rk.n < 1 ? 1 : 0;   // no valid score: NaN
    st->k[0] = rk.k_lo;
    st->k[1] = rk.k_hi;
  }
  for (int i = threadIdx.x; i < 512; i += blockDim.x) (&st->hist[0][0])[i] = 0;
}

__global__ void __launch_bounds__(256)
    sel_hist_kernel(const float* __restrict__ score, const uint8_t* __restrict__ valid, int64_t n, int shift,
                    SelState* st) {
  __shared__ uint32_t h[2][256];
  for (int i = threadIdx.x; i < 512; i += blockDim.x) (&h[0][0])[i] = 0;
  __syncthreads();
  const uint32_t p0 = st->prefix[0], p1 = st->prefix[1], mask = st->mask;
  int nan = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const bool ok = !valid || valid[i] != 0;
    const float v = score[i];
    nan |= ok && (v != v);
    const uint32_t key = ok ? order_key(v) : kInfKey;
    const uint32_t d = (key >> shift) & 255u;
    if ((key & mask) == p0) atomicAdd(&h[0][d], 1u);
    if ((key & mask) == p1) atomicAdd(&h[1][d], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 512; i += blockDim.x) {
    const uint32_t c = (&h[0][0])[i];
    if (c) atomicAdd(&(&st->hist[0][0])[i], c);
  }
  if (shift == 24 && __syncthreads_or(nan) && threadIdx.x == 0) atomicOr(&st->has_nan, 1);
}

__global__ void __launch_bounds__(64) sel_pick_kernel(SelState* st, int shift, float q, int64_t n_all,
                                                      const int64_t* n_dev, float* __restrict__ thres) {
  const int s = threadIdx.x >> 5, lane = threadIdx.x & 31;   // warp s handles order statistic s
  uint32_t c[8];
  unsigned long long tot = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) { c[j] = st->hist[s][lane * 8 + j]; tot += c[j]; }
  unsigned long long inc = tot;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned long long t = __shfl_up_sync(kFull, inc, off);
    if (lane >= off) inc += t;
  }
  unsigned long long run = inc - tot;
  const unsigned long long k = (unsigned long long)st->k[s];
  uint32_t digit = 0xFFFFFFFFu;
  long long rem = 0;
  if (k >= run && k < inc) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (digit == 0xFFFFFFFFu && k < run + c[j]) { digit = lane * 8 + j; rem = (long long)(k - run); }
      run += c[j];
    }
  }
  // exactly one lane found it (or none when there is no valid score)
  const unsigned who = __ballot_sync(kFull, digit != 0xFFFFFFFFu);
  const int src = who ? __ffs(who) - 1 : 0;
  digit = __shfl_sync(kFull, digit, src);
  rem = __shfl_sync(kFull, rem, src);
  if (!who) { digit = 0; rem = 0; }
  __syncthreads();    // all reads of hist are done
  if (lane == 0) {
    st->prefix[s] |= digit << shift;
    st->k[s] = rem;
  }
  for (int i = lane; i < 256; i += 32) st->hist[s][i] = 0;
  __syncthreads();
  if (threadIdx.x == 0) {
    st->mask |= 255u << shift;
    if (shift == 0) {
      const Ranks rk = quantile_ranks(n_all, n_dev, q);
      thres[0] = st->has_nan ? __int_as_float(0x7fc00000) : quantile_lerp(st->prefix[0], st->prefix[1], rk.w);
    }
  }
}

// ---------------------------------------------------------------------------
// admission
// ---------------------------------------------------------------------------
// One launch: count the admitted rows of every block | number them and unmap what they displace | copy
// the rows and set the maps, with a barrier of all blocks at each bar.  As four launches whose blocks
// covered 1 024 rows each, a table of 16 K candidates kept 16 SMs busy with the copies (18 us of a
// 36 us admission).  Phases are kept apart so that the result equals applying the rows one by one.
constexpr int kAdmitThreads = 512;
constexpr int kAdmitBlocks = 148;

struct AdmitArgs {
  int mode;  // 0 = per-layer table ring (grad_check.cu:6-46), 1 = unified cache buffer
  int64_t n;
  const float* rows; int64_t row_stride;   // candidate rows, fp32
  void* buffer; int buf_dtype; int width;  // destination rows
  int64_t capacity;
  const uint8_t* used; const uint8_t* valid;
  const int64_t* sub_to_full;
  const int64_t* sub_map;   // sub_to_history / sub2embed
  const float* score; const float* thres;
  int64_t* slot_to_full;    // history_to_full / embed2full
  int64_t* full_to_slot;    // full_to_history / full2embed
  int64_t* header;
  int64_t* checkin; int64_t glb_iter;
  // cache mode only
  int in_feat; int64_t total_num_node; const int64_t* feat2full; int64_t feat2full_len;
  int reset_header;
  int64_t* n_admitted;
  // scratch
  unsigned* word;          // barrier
  int* block_counts;       // [blocks]
  int vec_ok;
};

// The loads do not wait for each other: one latency per row.
__device__ __forceinline__ bool admit_flag(const AdmitArgs& a, int64_t i, float thres) {
  const bool absent = a.sub_map[i] == -1;
  const bool used = a.used == nullptr || a.used[i] != 0;
  const bool valid = a.valid == nullptr || a.valid[i] != 0;
  const float score = a.mode == 0 && thres == 0.f ? 0.f : a.score[i];
  const bool pass = a.mode == 0 ? !(thres != 0.f && score > thres) : score < thres;
  return absent & used & valid & pass;
}

__global__ void __launch_bounds__(kAdmitThreads) admit_kernel(const AdmitArgs a) {
  __shared__ int list_row[kAdmitThreads];
  __shared__ int64_t list_slot[kAdmitThreads];
  GridSync grid(a.word);
  const float thres = a.thres[0];
  // consecutive rows per block, so that ranks follow the row order
  const int64_t per = ceil_div(a.n, (int64_t)gridDim.x);
  const int64_t r0 = per * blockIdx.x < a.n ? per * blockIdx.x : a.n;
  const int64_t r1 = r0 + per < a.n ? r0 + per : a.n;
  // a thread remembers the flag of its first row (nearly always its only one)
  const bool flag0 = r0 + threadIdx.x < r1 && admit_flag(a, r0 + threadIdx.x, thres);
  auto flag_of = [&](int64_t t0) {
    const int64_t i = t0 + threadIdx.x;
    return t0 == r0 ? flag0 : (i < r1 && admit_flag(a, i, thres));
  };
  int mine = 0;
  for (int64_t t0 = r0; t0 < r1; t0 += blockDim.x) mine += flag_of(t0);
  int count;
  block_exclusive<kAdmitThreads>(mine, &count);
  if (threadIdx.x == 0) a.block_counts[blockIdx.x] = count;
  if (!grid.wait()) return;

  int total, first;
  block_prefix(a.block_counts, gridDim.x, blockIdx.x, &total, &first);
  int64_t h0 = a.header[0], eff = total;
  if (a.mode == 0) {
    h0 %= a.capacity;
    if (h0 < 0) h0 += a.capacity;
  } else {
    if (a.reset_header || h0 < 0) h0 = 0;
    const int64_t room = a.capacity > h0 ? a.capacity - h0 : 0;
    if (eff > room) eff = room;
  }
  // slot of an admitted row by its rank; -1: displaced again by a later row, or out of room
  auto slot_of = [&](int64_t rank) -> int64_t {
    if (a.mode == 0) return rank >= (int64_t)total - a.capacity ? (h0 + rank) % a.capacity : -1;
    return rank < eff ? h0 + rank : -1;
  };
  // everything that must be unmapped is unmapped before anything is set; the rows themselves can move now
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t rank0 = first;
  for (int64_t t0 = r0; t0 < r1; t0 += blockDim.x) {
    const bool f = flag_of(t0);
    int here;
    const int local = block_exclusive<kAdmitThreads>(f, &here);
    if (f) {
      const int64_t rank = rank0 + local;
      list_row[local] = threadIdx.x;
      list_slot[local] = slot_of(rank);
      if (a.mode == 0) {
        const int64_t slot = (h0 + rank) % a.capacity;
        const int64_t old = a.slot_to_full[slot];
        if (old != -1 && a.full_to_slot[old] == slot) a.full_to_slot[old] = -1;
      } else if (rank < eff) {
        const int64_t old = a.slot_to_full[h0 + rank];
        if (old != -1) {
          const int64_t cur = a.full_to_slot[old];
          if (cur >= h0 && cur < h0 + eff) a.full_to_slot[old] = -1;
        }
      }
    }
    rank0 += here;
    __syncthreads();
    for (int k = warp; k < here; k += kAdmitThreads / 32) {
      const int64_t row = t0 + list_row[k], slot = list_slot[k];
      if (slot < 0) continue;
      const float* __restrict__ src = a.rows + row * a.row_stride;
      if (a.buf_dtype == HC_F32) {
        float* dst = reinterpret_cast<float*>(a.buffer) + slot * a.width;
        if (a.vec_ok)
          for (int v = lane; v < (a.width >> 2); v += kWarp)
            reinterpret_cast<uint4*>(dst)[v] = ldg16(src + 4 * v);
        else
          for (int c = lane; c < a.width; c += kWarp) dst[c] = src[c];
      } else {
        __half* dst = reinterpret_cast<__half*>(a.buffer) + slot * a.width;
        if (a.vec_ok)
          for (int v = lane; v < (a.width >> 2); v += kWarp) {
            float f4[4];
            Vec16<float>::unpack(ldg16(src + 4 * v), f4);
            __half2 lo = __floats2half2_rn(f4[0], f4[1]), hi = __floats2half2_rn(f4[2], f4[3]);
            uint2 pk;
            pk.x = *reinterpret_cast<uint32_t*>(&lo);
            pk.y = *reinterpret_cast<uint32_t*>(&hi);
            reinterpret_cast<uint2*>(dst)[v] = pk;
          }
        else
          for (int c = lane; c < a.width; c += kWarp) dst[c] = __float2half_rn(src[c]);
      }
    }
    __syncthreads();
  }
  if (a.mode == 1 && a.feat2full) {      // raw-feature slots overlapped by embedding slots [h0, h0 + eff)
    const int64_t fb = h0 * a.width / a.in_feat;
    int64_t fe = ((h0 + eff) * a.width + a.in_feat - 1) / a.in_feat;
    if (fe > a.feat2full_len) fe = a.feat2full_len;
    for (int64_t k = fb + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < fe; k += (int64_t)gridDim.x * blockDim.x)
      a.full_to_slot[a.feat2full[k]] = -1;
  }
  if (!grid.wait()) return;

  if (blockIdx.x == 0 && threadIdx.x == 0) {      // every block has read the header
    a.header[0] = a.mode == 0 ? (h0 + total) % a.capacity : h0 + eff;
    if (a.n_admitted) a.n_admitted[0] = eff;
  }
  rank0 = first;
  for (int64_t t0 = r0; t0 < r1; t0 += blockDim.x) {
    const bool f = flag_of(t0);
    int here;
    const int64_t rank = rank0 + block_exclusive<kAdmitThreads>(f, &here);
    rank0 += here;
    if (!f) continue;
    const int64_t slot = slot_of(rank), full = a.sub_to_full[t0 + threadIdx.x];
    if (slot >= 0) {
      a.full_to_slot[full] = slot;
      a.slot_to_full[slot] = full;
      if (a.checkin) a.checkin[slot] = a.glb_iter;
    } else if (a.mode == 0) {
      // more admissions than slots: applied one by one, this row was written and then displaced, which
      // leaves it unmapped
      a.full_to_slot[full] = -1;
    }
  }
}

static int run_admit(AdmitArgs& a, void* scratch, cudaStream_t st) {
  if (a.n == 0 && !(a.mode == 1 && a.reset_header)) {
    if (a.n_admitted) HC_CUDA(cudaMemsetAsync(a.n_admitted, 0, sizeof(int64_t), st));
    return 0;
  }
  HC_REQUIRE(scratch != nullptr, HC_ERR_NULL);
  HC_REQUIRE(aligned_to(scratch, 8), HC_ERR_ALIGN);
  HC_REQUIRE(a.n < 0x7fffffffLL, HC_ERR_SIZE);
  a.word = reinterpret_cast<unsigned*>(scratch);
  a.block_counts = reinterpret_cast<int*>(scratch) + 4;
  const int es = dtype_size(a.buf_dtype);
  a.vec_ok = a.width % 4 == 0 && aligned16(a.rows) && (a.row_stride % 4) == 0 &&
             aligned_to(a.buffer, a.buf_dtype == HC_F32 ? 16 : 8) && es != 0;
  const int64_t blocks = ceil_div(a.n > 0 ? a.n : 1, 32);      // a warp of rows each, up to one block per SM
  return launch_together(admit_kernel, (unsigned)(blocks < kAdmitBlocks ? blocks : kAdmitBlocks),
                                          kAdmitThreads, 0, a.word, st, a);
}

// ---------------------------------------------------------------------------
// eviction
// ---------------------------------------------------------------------------
__global__ void evict_stale_kernel(int64_t* checkin, int64_t* h2f, int64_t* f2h, int64_t cap,
                                   int64_t stale_iter) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= cap) return;
  const int64_t c = checkin[s];
  if (c > -1 && c <= stale_iter) {
    const int64_t full = h2f[s];
    checkin[s] = -1;
    h2f[s] = -1;
    if (full != -1) f2h[full] = -1;
  }
}

// the same with the iteration number read from device memory (steps replayed from a CUDA graph
// cannot carry it as a launch argument)
__global__ void evict_stale_dev_kernel(int64_t* checkin, int64_t* h2f, int64_t* f2h, int64_t cap,
                                       const int64_t* __restrict__ iter_dev, int64_t limit) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= cap) return;
  const int64_t c = checkin[s];
  if (c > -1 && c <= iter_dev[0] - limit) {
    const int64_t full = h2f[s];
    checkin[s] = -1;
    h2f[s] = -1;
    if (full != -1) f2h[full] = -1;
  }
}
__global__ void stamp_checkin_kernel(int64_t* checkin, int64_t cap, int64_t marker,
                                     const int64_t* __restrict__ iter_dev) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s < cap && checkin[s] == marker) checkin[s] = iter_dev[0];
}

__global__ void evict_by_score_kernel(const int64_t* __restrict__ sub_to_history,
                                      const float* __restrict__ score,
                                      const float* __restrict__ thres, int64_t n, int64_t* checkin,
                                      int64_t* h2f, int64_t* f2h) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const int64_t slot = sub_to_history[r];
  if (slot == -1 || !(score[r] >= thres[0])) return;
  const int64_t full = h2f[slot];
  if (full != -1) f2h[full] = -1;
  h2f[slot] = -1;
  checkin[slot] = -1;
}

// Both evictions of a table in one launch: thread k < n looks at row k's score, the others at a slot's
// check-in time.  A slot that both drop ends up the same whichever comes first.
__global__ void __launch_bounds__(256)
    evict_both_kernel(const int64_t* __restrict__ sub_to_history, const float* __restrict__ score,
                      const float* __restrict__ thres, int64_t n, int64_t* checkin, int64_t* h2f, int64_t* f2h,
                      int64_t cap, int64_t glb_iter, const int64_t* __restrict__ iter_dev, int64_t limit) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t slot;
  if (t < n) {
    slot = sub_to_history[t];
    if (slot == -1 || !(score[t] >= thres[0])) return;
  } else {
    slot = t - n;
    if (slot >= cap) return;
    const int64_t c = checkin[slot];
    if (!(c > -1 && c <= (iter_dev ? iter_dev[0] : glb_iter) - limit)) return;
  }
  const int64_t full = h2f[slot];
  if (full != -1) f2h[full] = -1;
  h2f[slot] = -1;
  checkin[slot] = -1;
}

}  // namespace hc

using namespace hc;

extern "C" int hc_evict_both(const int64_t* sub_to_history, const float* score, const float* thres, int64_t n,
                             int64_t* checkin_iter, int64_t* history_to_full, int64_t* full_to_history,
                             int64_t capacity, int64_t glb_iter, const int64_t* glb_iter_dev, int64_t limit,
                             void* stream) {
  HC_REQUIRE(n >= 0 && capacity >= 0, HC_ERR_SIZE);
  if (n + capacity == 0) return 0;
  HC_REQUIRE(checkin_iter && history_to_full && full_to_history, HC_ERR_NULL);
  HC_REQUIRE(n == 0 || (sub_to_history && score && thres), HC_ERR_NULL);
  const int64_t blocks = ceil_div(n + capacity, 256);
  HC_REQUIRE(blocks <= 0x7fffffffLL, HC_ERR_SIZE);
  evict_both_kernel<<<(unsigned)blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      sub_to_history, score, thres, n, checkin_iter, history_to_full, full_to_history, capacity, glb_iter, glb_iter_dev,
      limit);
  HC_LAUNCH_OK();
  return 0;
}

extern "C" int hc_score_rows(const float* x, int64_t n, int32_t feat, int64_t stride, int32_t kind,
                             float* score, void* stream) {
  HC_REQUIRE(n >= 0 && feat > 0, HC_ERR_SIZE);
  HC_REQUIRE(kind == HC_SCORE_L2 || kind == HC_SCORE_L1, HC_ERR_SIZE);
  if (n == 0) return 0;
  HC_REQUIRE(x && score, HC_ERR_NULL);
  if (stride == 0) stride = feat;
  HC_REQUIRE(stride >= feat, HC_ERR_SIZE);
  const int64_t blocks = ceil_div(n, 8);
  HC_REQUIRE(blocks <= 0x7fffffffLL, HC_ERR_SIZE);
  score_rows_kernel<<<(unsigned)blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      x, n, feat, stride, kind, score);
  HC_LAUNCH_OK();
  return 0;
}

extern "C" int64_t hc_select_scratch_bytes(int64_t n) {
  return n > kSelSmall ? (int64_t)sizeof(SelState) + 64 : 0;
}

static int select_launch(const float* score, int64_t n, const int64_t* n_valid, const uint8_t* valid, float q,
                         float* thres, void* scratch, cudaStream_t st) {
  if (n <= kSelSmall) {
    const size_t smem = (size_t)n * sizeof(uint32_t);
    if (smem > 32 * 1024) {      // static arrays come on top
      // raised once per device (not a stream operation, so keep it out of stream captures)
      static bool raised[64] = {};
      int devno = 0;
      HC_CUDA(cudaGetDevice(&devno));
      if (devno >= 0 && devno < 64 && !raised[devno]) {
        HC_CUDA(cudaFuncSetAttribute(select_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     kSelSmall * (int)sizeof(uint32_t)));
        raised[devno] = true;
      }
    }
    select_small_kernel<<<1, kSelThreads, smem, st>>>(score, n, n_valid, valid, q, thres);
    HC_LAUNCH_OK();
    return 0;
  }
  HC_REQUIRE(scratch != nullptr && aligned_to(scratch, 8), HC_ERR_NULL);
  HC_REQUIRE(n < 0xffffffffLL, HC_ERR_SIZE);
  SelState* state = reinterpret_cast<SelState*>(scratch);
  int64_t blocks = ceil_div(n, 256 * 8);
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (valid) {
    HC_CUDA(cudaMemsetAsync(&state->n_valid, 0, sizeof(state->n_valid), st));
    sel_count_kernel<<<(unsigned)blocks, 256, 0, st>>>(state, valid, n);
    n_valid = reinterpret_cast<const int64_t*>(&state->n_valid);
  }
  sel_init_kernel<<<1, 256, 0, st>>>(state, n, n_valid, q);
  for (int shift = 24; shift >= 0; shift -= 8) {
    sel_hist_kernel<<<(unsigned)blocks, 256, 0, st>>>(score, valid, n, shift, state);
    sel_pick_kernel<<<1, 64, 0, st>>>(state, shift, q, n, n_valid, thres);
  }
  HC_LAUNCH_OK();
  return 0;
}

extern "C" int hc_select_threshold(const float* score, int64_t n, float q, float* thres,
                                   void* scratch, void* stream) {
  HC_REQUIRE(n > 0, HC_ERR_SIZE);
  HC_REQUIRE(score && thres, HC_ERR_NULL);
  HC_REQUIRE(q >= 0.f && q <= 1.f, HC_ERR_SIZE);
  return select_launch(score, n, nullptr, nullptr, q, thres, scratch, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int hc_select_threshold_counted(const float* score, int64_t n, const int64_t* n_valid,
                                           float q, float* thres, void* scratch, void* stream) {
  HC_REQUIRE(n > 0, HC_ERR_SIZE);
  HC_REQUIRE(score && thres && n_valid, HC_ERR_NULL);
  HC_REQUIRE(q >= 0.f && q <= 1.f, HC_ERR_SIZE);
  return select_launch(score, n, n_valid, nullptr, q, thres, scratch, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int hc_select_threshold_masked(const float* score, const uint8_t* valid, int64_t n, float q, float* thres,
                                          void* scratch, void* stream) {
  HC_REQUIRE(n > 0, HC_ERR_SIZE);
  HC_REQUIRE(score && thres && valid, HC_ERR_NULL);
  HC_REQUIRE(q >= 0.f && q <= 1.f, HC_ERR_SIZE);
  return select_launch(score, n, nullptr, valid, q, thres, scratch, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int64_t hc_admit_scratch_bytes(int64_t n) {
  (void)n;
  return 16 + kAdmitBlocks * (int64_t)sizeof(int);
}

extern "C" int hc_record_history_masked(const float* buffer_new, int64_t new_stride, int64_t n,
                                 void* buffer_all, int32_t table_dtype, int64_t capacity,
                                 int32_t history_size, const uint8_t* used_mask, const uint8_t* valid,
                                 const int64_t* sub_to_full, const int64_t* sub_to_history,
                                 int64_t* history_to_full, int64_t* full_to_history,
                                 int64_t* header, const float* score, const float* thres,
                                 int64_t* checkin_iter, int64_t glb_iter, int64_t* n_admitted,
                                 void* scratch, void* stream) {
  HC_REQUIRE(n >= 0 && capacity >= 0 && history_size > 0, HC_ERR_SIZE);
  HC_REQUIRE(dtype_size(table_dtype) != 0, HC_ERR_DTYPE);
  if (n > 0) {
    HC_REQUIRE(buffer_new && sub_to_full && sub_to_history && history_to_full && full_to_history &&
                   header && score && thres && checkin_iter,
               HC_ERR_NULL);
    HC_REQUIRE(capacity == 0 || buffer_all != nullptr, HC_ERR_NULL);
  }
  if (new_stride == 0) new_stride = history_size;
  HC_REQUIRE(new_stride >= history_size, HC_ERR_SIZE);
  AdmitArgs a{};
  a.mode = 0; a.n = n; a.rows = buffer_new; a.row_stride = new_stride;
  a.buffer = buffer_all; a.buf_dtype = table_dtype; a.width = history_size;
  a.capacity = capacity; a.used = used_mask; a.valid = valid; a.sub_to_full = sub_to_full;
  a.sub_map = sub_to_history; a.score = score; a.thres = thres;
  a.slot_to_full = history_to_full; a.full_to_slot = full_to_history; a.header = header;
  a.checkin = checkin_iter; a.glb_iter = glb_iter; a.n_admitted = n_admitted;
  if (capacity == 0) {
    // an empty table admits nothing (history_table.py:130-131 skips such layers)
    if (n_admitted)
      HC_CUDA(cudaMemsetAsync(n_admitted, 0, sizeof(int64_t), reinterpret_cast<cudaStream_t>(stream)));
    return 0;
  }
  return run_admit(a, scratch, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int hc_record_history(const float* buffer_new, int64_t new_stride, int64_t n,
                                 void* buffer_all, int32_t table_dtype, int64_t capacity,
                                 int32_t history_size, const uint8_t* used_mask,
                                 const int64_t* sub_to_full, const int64_t* sub_to_history,
                                 int64_t* history_to_full, int64_t* full_to_history,
                                 int64_t* header, const float* score, const float* thres,
                                 int64_t* checkin_iter, int64_t glb_iter, int64_t* n_admitted,
                                 void* scratch, void* stream) {
  return hc_record_history_masked(buffer_new, new_stride, n, buffer_all, table_dtype, capacity, history_size, used_mask,
                                  nullptr, sub_to_full, sub_to_history, history_to_full, full_to_history, header, score,
                                  thres, checkin_iter, glb_iter, n_admitted, scratch, stream);
}

extern "C" int hc_cache_admit(const float* produced, int64_t prod_stride, int64_t n, void* buffer,
                              int32_t buf_dtype, int32_t hidden, int32_t in_feat,
                              int64_t embed_capacity, const int64_t* sub_to_full,
                              const int64_t* sub2embed, const float* score, const float* thres,
                              int64_t* full2embed, int64_t total_num_node, int64_t* embed2full,
                              const int64_t* feat2full, int64_t feat2full_len, int64_t* header,
                              int32_t reset_header, const uint8_t* valid, int64_t* n_admitted,
                              void* scratch, void* stream) {
  HC_REQUIRE(n >= 0 && embed_capacity >= 0 && hidden > 0 && in_feat > 0 && total_num_node >= 0 &&
                 feat2full_len >= 0,
             HC_ERR_SIZE);
  HC_REQUIRE(dtype_size(buf_dtype) != 0, HC_ERR_DTYPE);
  HC_REQUIRE(header != nullptr, HC_ERR_NULL);
  if (n > 0)
    HC_REQUIRE(produced && buffer && sub_to_full && sub2embed && score && thres && full2embed &&
                   embed2full,
               HC_ERR_NULL);
  if (prod_stride == 0) prod_stride = hidden;
  HC_REQUIRE(prod_stride >= hidden, HC_ERR_SIZE);
  AdmitArgs a{};
  a.mode = 1; a.n = n; a.rows = produced; a.row_stride = prod_stride;
  a.buffer = buffer; a.buf_dtype = buf_dtype; a.width = hidden; a.capacity = embed_capacity;
  a.sub_to_full = sub_to_full; a.sub_map = sub2embed; a.score = score; a.thres = thres;
  a.slot_to_full = embed2full; a.full_to_slot = full2embed; a.header = header;
  a.in_feat = in_feat; a.total_num_node = total_num_node;
  a.feat2full = feat2full_len > 0 ? feat2full : nullptr; a.feat2full_len = feat2full_len;
  a.reset_header = reset_header; a.n_admitted = n_admitted; a.used = valid;
  if (n == 0 && reset_header) {
    // nothing to admit, but the ring still restarts
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    HC_CUDA(cudaMemsetAsync(header, 0, sizeof(int64_t), st));
    if (n_admitted) HC_CUDA(cudaMemsetAsync(n_admitted, 0, sizeof(int64_t), st));
    return 0;
  }
  return run_admit(a, scratch, reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int hc_evict_stale(int64_t* checkin_iter, int64_t* history_to_full,
                              int64_t* full_to_history, int64_t capacity, int64_t glb_iter,
                              int64_t limit, void* stream) {
  HC_REQUIRE(capacity >= 0, HC_ERR_SIZE);
  if (capacity == 0) return 0;
  HC_REQUIRE(checkin_iter && history_to_full && full_to_history, HC_ERR_NULL);
  const int64_t blocks = ceil_div(capacity, 256);
  HC_REQUIRE(blocks <= 0x7fffffffLL, HC_ERR_SIZE);
  evict_stale_kernel<<<(unsigned)blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      checkin_iter, history_to_full, full_to_history, capacity, glb_iter - limit);
  HC_LAUNCH_OK();
  return 0;
}

extern "C" int hc_evict_stale_dev(int64_t* checkin_iter, int64_t* history_to_full,
                                  int64_t* full_to_history, int64_t capacity,
                                  const int64_t* glb_iter_dev, int64_t limit, void* stream) {
  HC_REQUIRE(capacity >= 0, HC_ERR_SIZE);
  if (capacity == 0) return 0;
  HC_REQUIRE(checkin_iter && history_to_full && full_to_history && glb_iter_dev, HC_ERR_NULL);
  const int64_t blocks = ceil_div(capacity, 256);
  HC_REQUIRE(blocks <= 0x7fffffffLL, HC_ERR_SIZE);
  evict_stale_dev_kernel<<<(unsigned)blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      checkin_iter, history_to_full, full_to_history, capacity, glb_iter_dev, limit);
  HC_LAUNCH_OK();
  return 0;
}

extern "C" int hc_stamp_checkin(int64_t* checkin_iter, int64_t capacity, int64_t marker,
                                const int64_t* glb_iter_dev, void* stream) {
  HC_REQUIRE(capacity >= 0, HC_ERR_SIZE);
  if (capacity == 0) return 0;
  HC_REQUIRE(checkin_iter && glb_iter_dev, HC_ERR_NULL);
  const int64_t blocks = ceil_div(capacity, 256);
  HC_REQUIRE(blocks <= 0x7fffffffLL, HC_ERR_SIZE);
  stamp_checkin_kernel<<<(unsigned)blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      checkin_iter, capacity, marker, glb_iter_dev);
  HC_LAUNCH_OK();
  return 0;
}

extern "C" int hc_evict_by_score(const int64_t* sub_to_history, const float* score,
                                 const float* thres, int64_t n, int64_t* checkin_iter,
                                 int64_t* history_to_full, int64_t* full_to_history, void* stream) {
  HC_REQUIRE(n >= 0, HC_ERR_SIZE);
  if (n == 0) return 0;
  HC_REQUIRE(sub_to_history && score && thres && checkin_iter && history_to_full && full_to_history,
             HC_ERR_NULL);
  const int64_t blocks = ceil_div(n, 256);
  HC_REQUIRE(blocks <= 0x7fffffffLL, HC_ERR_SIZE);
  evict_by_score_kernel<<<(unsigned)blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      sub_to_history, score, thres, n, checkin_iter, history_to_full, full_to_history);
  HC_LAUNCH_OK();
  return 0;
}


// ---------------------------------------------------------------------------
// Ring admission with built-in scratch (no allocation by anybody)
// ---------------------------------------------------------------------------
// hc_record_history needs a few KB of device scratch that the caller allocates.  Some
// callers have nothing to allocate with: a plain-C, cgo or JNI host that was only handed the
// input and output buffers and holds no handle to the framework's device allocator, or a
// training loop whose memory is entirely owned by a caching allocator and in which a raw
// cudaMalloc / cudaFree would stall the device.  For them the scratch lives in this
// file-scope array, which every GPU that loads the library carries until the process exits.
namespace hc {

constexpr int64_t kNoAllocMaxRows = 1 << 20;  // HC_NOALLOC_MAX_ROWS
constexpr int64_t kNoAllocBytes = 16 + kAdmitBlocks * (int64_t)sizeof(int);
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

constexpr int kNoAllocMaxDevices = 64;
// Device address of g_noalloc_scratch per device ordinal.  In host code the array's name is
// only a handle for the runtime, never an address a kernel may be given; the address comes
// from cudaGetSymbolAddress, asked once per device with that device current.
static void* g_noalloc_addr[kNoAllocMaxDevices];

static int noalloc_scratch(void** out) {
  int dev = -1;
  HC_CUDA(cudaGetDevice(&dev));
  HC_REQUIRE(dev >= 0 && dev < kNoAllocMaxDevices, HC_ERR_SIZE);
  void* p = __atomic_load_n(&g_noalloc_addr[dev], __ATOMIC_ACQUIRE);
  if (p == nullptr) {
    HC_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    HC_REQUIRE(p != nullptr, HC_ERR_NULL);
    __atomic_store_n(&g_noalloc_addr[dev], p, __ATOMIC_RELEASE);
  }
  *out = p;
  return 0;
}

}  // namespace hc

extern "C" int64_t hc_noalloc_max_rows(void) { return hc::kNoAllocMaxRows; }

extern "C" int hc_record_history_noalloc(const float* buffer_new, int64_t new_stride, int64_t n,
                                         void* buffer_all, int32_t table_dtype, int64_t capacity,
                                         int32_t history_size, const uint8_t* used_mask,
                                         const int64_t* sub_to_full,
                                         const int64_t* sub_to_history, int64_t* history_to_full,
                                         int64_t* full_to_history, int64_t* header,
                                         const float* score, const float* thres,
                                         int64_t* checkin_iter, int64_t glb_iter,
                                         int64_t* n_admitted, void* stream) {
  if (n > hc::kNoAllocMaxRows) return -HC_ERR_LIMIT;
  void* scratch = nullptr;
  const int rc = hc::noalloc_scratch(&scratch);
  if (rc != 0) return rc;
  // every scratch word that is read was written earlier in the same call, so the contents
  // left by the previous call need no clearing
  return hc_record_history(buffer_new, new_stride, n, buffer_all, table_dtype, capacity,
                           history_size, used_mask, sub_to_full, sub_to_history, history_to_full,
                           full_to_history, header, score, thres, checkin_iter, glb_iter,
                           n_admitted, scratch, stream);
}
