// History-aware CSR gather-reduce (forward) and transposed scatter (backward).
//
// Replaces the eight kernels of the reference's src/cpp/src/history_aggr.cu
// (:7-397) and their launchers (:399-596).  The reference splits one row over
// F/32 warps of scalar 4-byte lanes, each re-reading ptr / idx / hmap; here
// one warp owns a whole destination row, every lane moves 16 bytes per
// request, narrow rows are shared by several edges per request, and the
// choice between a fresh source row, an alternative (cached) source row and a
// history row is made inside the gather.  Memory bound: no tensor cores.
#include <atomic>

#include "common.cuh"

namespace hc {

// ---------------------------------------------------------------------------
// index checks of the HC_CHECK_BOUNDS build: a validation pass over the block records the first
// index that lies outside its table; while the status word is set the operator kernels return at
// once, so no out-of-range access is ever made and nothing traps.
// ---------------------------------------------------------------------------
#ifdef HC_CHECK_BOUNDS
static __device__ unsigned long long g_status[4];   // code, which array, position, value

__device__ __forceinline__ void status_set(int which, int64_t pos, int64_t value) {
  if (atomicCAS(&g_status[0], 0ull, (unsigned long long)HC_ERR_RANGE) == 0ull) {
    g_status[1] = (unsigned long long)which;
    g_status[2] = (unsigned long long)pos;
    g_status[3] = (unsigned long long)value;
  }
}

__global__ void __launch_bounds__(256) aggr_check_kernel(const hc_aggr_args a) {
  constexpr int G = 8;
  const int gl = threadIdx.x & (G - 1);
  const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
  if (r >= a.num_node) return;
  const int64_t b = a.ptr[r], e_end = a.ptr[r + 1];
  if (gl == 0) {
    if (b < 0 || e_end < b) status_set(1, r, e_end < b ? e_end : b);
    if (a.hmap) {
      const int64_t h = a.hmap[r];
      const int64_t rows = a.h_rows;
      if (h < -1 || (a.h_indexed && rows > 0 && h >= rows) || (!a.h_indexed && h != -1 && rows > 0 && r >= rows))
        status_set(4, r, h);
    }
  }
  if (b < 0 || e_end < b) return;
  for (int64_t e = b + gl; e < e_end; e += G) {
    const int64_t s = a.idx[e];
    if (s < 0 || s >= a.n_src) {
      status_set(2, e, s);
      continue;
    }
    if (a.src_map) {
      const int64_t m = a.src_map[s];
      if (m < -1 || (a.alt_rows > 0 && m >= a.alt_rows)) status_set(3, s, m);
    }
  }
}
#define HC_BAIL_IF_BAD() \
  if (g_status[0] != 0ull) return;
#else
#define HC_BAIL_IF_BAD()
#endif

// history row -> columns [v0 * EL, ...) of the fp32 output row
template <int EL>
__device__ __forceinline__ void copy_history_part(const hc_aggr_args& a, int64_t hrow, float* __restrict__ orow,
                                                  int width, int v0, int v1, int lane, int h_vec) {
  const int F = a.feat;
  const bool shared_row = a.hsize == F;      // one history row for all heads
  const int c0 = v0 * EL, c1 = v1 * EL < width ? v1 * EL : width;
  const int64_t base = hrow * a.hsize;
  if (h_vec) {
    for (int c = c0 + 4 * lane; c < c1; c += 4 * kWarp) {
      const int64_t off = base + (shared_row ? c % F : c);
      float4 o;
      if (a.h_dtype == HC_F32) {
        o = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(a.hbuf) + off);
      } else {
        LaneVec<__half, 8> h;
        h.load(reinterpret_cast<const __half*>(a.hbuf) + off);
        float f[4];
        h.unpack(f);
        o = make_float4(f[0], f[1], f[2], f[3]);
      }
      *reinterpret_cast<float4*>(orow + c) = o;
    }
  } else {
    for (int c = c0 + lane; c < c1; c += kWarp)
      orow[c] = load_as_f32(a.hbuf, a.h_dtype, base + (shared_row ? c % F : c));
  }
}

// ---------------------------------------------------------------------------
// forward, rows of at least 4-byte units: a stream of edges through shared memory
//   T    storage type of source rows
//   VB   bytes per lane and request: 16 where rows allow it, else 8 or 4
//   G    lanes that share one source row (G < 32: 32/G edges per request)
//   V    vectors per lane; a row of more than G*V vectors is cut into column parts (gridDim.y)
//   EV   0 mean, 1 sum weighted per edge, 2 sum weighted per edge and head
//   MAP  per-source select between input and src_alt
// ---------------------------------------------------------------------------
// A destination row costs three dependent memory latencies: ptr -> idx -> source rows.  A warp per
// row has its bytes in flight during the last of them only, and more unrolling did not help (ragged
// rows of 10 edges of 256 B: 370 us with 6 loads in flight per lane and 40 warps, 415 with 8 and 32:
// the time followed the number of warps).  Here a warp owns a run of consecutive rows, whose edges
// are one contiguous slice of idx, and walks them as a stream: asynchronous copies keep D requests in
// flight at all times, across row boundaries, while the oldest is added up; idx comes in chunks of 32,
// one chunk ahead.  A lane copies and reads back only its own bytes, so the ring needs no barrier.
// Measured, start -> now: 500 K ragged rows, 5 M edges of 256 B (fp16) out of 2 M rows 370 -> 231 us
// (1.58 GB gathered, read and written: 6.8 TB/s, a tenth of the gathers hit the L2); 200 K rows, 1.8 M
// skewed edges of 1 KB 294 -> 243 us; 100 K rows, 1 M edges with weights for 4 heads of 64 285 -> 175 us;
// 60 K rows, 720 K edges of 75 fp32 columns 112 -> 62 us (was the scalar kernel).
// Two requests per slot halve the walking (row switches, ring, commit) per edge: with one the issue
// slots were 84 % busy at 5.5 TB/s.  Ring size and blocks per SM are what the sweep over U = 1..4,
// 4 / 6 / 8 KB per warp and 3..5 blocks left (weighted sums, which also load weights through the L1,
// want the fourth block).
template <int VB, int V, int EV>
struct StreamShape {
  static constexpr int U = 2;                                             // requests per slot
  static constexpr int kReq = V * VB * kWarp;                             // bytes of one request of the warp
  static constexpr int kSlot = U * kReq;
  static constexpr int kRing = EV ? 6144 : 8192;
  static constexpr int D = kRing / kSlot < 3 ? 3 : (kRing / kSlot > 8 ? 8 : kRing / kSlot);   // slots in flight
  static constexpr int kWarpBytes = D * kSlot + 64 * 8;                   // + ring of row addresses
  static constexpr int kSmem = 8 * kWarpBytes;
  static constexpr int kFit = 220 * 1024 / (kSmem + 1024);
  static constexpr int kMinBlocks = kFit < (EV ? 4 : 3) ? kFit : (EV ? 4 : 3);
};
constexpr int kMaxRun = 31;      // rows of a run: one ptr entry per lane

template <typename T, int VB, int G, int V, int EV, bool MAP>
__global__ void __launch_bounds__(256, (StreamShape<VB, V, EV>::kMinBlocks))
    aggr_fwd_stream_kernel(const hc_aggr_args a, float* __restrict__ out, const int nvec, const int part_vec,
                           const int h_vec, const int stream_out, const int run_rows) {
  HC_BAIL_IF_BAD()
  using Vec = LaneVec<T, VB>;
  using Shape = StreamShape<VB, V, EV>;
  constexpr int EL = Vec::kElems;
  constexpr int EPW = kWarp / G;
  constexpr int D = Shape::D, U = Shape::U;
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned char* mine = smem + (size_t)warp * Shape::kWarpBytes + lane * VB;
  const uint32_t mine_s = smem_u32(mine);
  unsigned long long* ring = reinterpret_cast<unsigned long long*>(smem + (size_t)warp * Shape::kWarpBytes + D * Shape::kSlot);
  const int H = a.num_head;
  const int width = H * a.feat;
  const int v0 = blockIdx.y * part_vec;                       // this block's columns of the row
  const int v1 = v0 + part_vec < nvec ? v0 + part_vec : nvec;
  const int sub = lane / G, gl = lane % G;
  const char* __restrict__ in = reinterpret_cast<const char*>(a.input);
  const char* __restrict__ alt = reinterpret_cast<const char*>(a.src_alt);
  const int64_t in_bytes = a.in_stride * (int64_t)sizeof(T), alt_bytes = a.alt_stride * (int64_t)sizeof(T);
  const uint64_t policy = l2_policy(stream_out != 0);
  int head[V];
#pragma unroll
  for (int k = 0; k < V; ++k) head[k] = EV == 2 ? (v0 + gl + k * G) * EL / a.feat : 0;

  const int64_t runs = ceil_div(a.num_node, run_rows);
  const int64_t step = (int64_t)gridDim.x * 8;
  int64_t run = (int64_t)blockIdx.x * 8 + warp;
  int64_t my_p = 0, my_h = -1;      // lane l: ptr and history entry of row l of the run
  auto fetch_run = [&](int64_t q) {
    const int64_t row = q * run_rows + lane;
    my_p = 0;
    my_h = -1;
    if (q < runs && lane <= run_rows && row <= a.num_node) {
      my_p = a.ptr[row];
      if (a.hmap && lane < run_rows && row < a.num_node) my_h = a.hmap[row];
    }
  };
  fetch_run(run);
  for (; run < runs; run += step) {
    const int64_t r0 = run * run_rows;
    const int nr = (int)(a.num_node - r0 < run_rows ? a.num_node - r0 : run_rows);
    const int64_t e0 = shfl64(my_p, 0);
    const int off = (int)(my_p - e0);                // lane l <= nr: first edge of row l of the run
    const int64_t hrow = my_h;
    const unsigned miss = __ballot_sync(kFull, lane < nr && my_h == -1);
    const unsigned hits = __ballot_sync(kFull, lane < nr && my_h != -1);
    const int total = __shfl_sync(kFull, off, nr);
    int64_t next_i = lane < total ? a.idx[e0 + lane] : 0;      // chunk [loaded, loaded + 32) of the run's edges
    fetch_run(run + step);                                     // in flight during this run
    int loaded = 0;
    // producer: edge pe of a row that ends at pend, rows left in pm
    unsigned pm = miss;
    int pe = 0, pend = 0;
    auto produce = [&](int slot) {
      while (pe >= pend && pm) {
        const int row = __ffs(pm) - 1;
        pm &= pm - 1;
        pe = __shfl_sync(kFull, off, row);
        pend = __shfl_sync(kFull, off, row + 1);
      }
      if (pe < pend) {
        const int need = pe + U * EPW < pend ? pe + U * EPW : pend;
        if (pe >= loaded + kWarp) {      // rows served from history were skipped
          loaded = pe & ~31;
          next_i = loaded + lane < total ? a.idx[e0 + loaded + lane] : 0;
        }
        while (need > loaded) {
          const char* p = in + next_i * in_bytes;
          if (MAP && loaded + lane < total) {
            const int64_t m = a.src_map[next_i];
            if (m != -1) p = alt + m * alt_bytes;
          }
          __syncwarp();
          ring[(loaded + lane) & 63] = reinterpret_cast<unsigned long long>(p);
          __syncwarp();
          loaded += kWarp;
          next_i = loaded + lane < total ? a.idx[e0 + loaded + lane] : 0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int e = pe + u * EPW + sub;
          if (e < pend) {
            const char* p = reinterpret_cast<const char*>(ring[e & 63]);
            const uint32_t dst = mine_s + slot * Shape::kSlot + u * Shape::kReq;
#pragma unroll
            for (int k = 0; k < V; ++k) {
              const int v = v0 + gl + k * G;
              if (v < v1) cp_async<VB>(dst + k * VB * kWarp, p + v * VB);
            }
          }
        }
        pe += U * EPW;
      }
      cp_async_commit();
    };
#pragma unroll 1
    for (int d = 0; d < D; ++d) produce(d);
    for (unsigned h = hits; h; h &= h - 1) {
      const int row = __ffs(h) - 1;
      const int64_t hr = shfl64(hrow, row);
      copy_history_part<EL>(a, a.h_indexed ? hr : r0 + row, out + (r0 + row) * width, width, v0, v1, lane, h_vec);
    }
    // weights of the next slot, one slot ahead: a slot is a new sector of them
    float w_next[U][EV == 2 ? V : 1];
    int w_at = -1;
    auto load_weights = [&](int from) {
      w_at = from;
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int k = 0; k < (EV == 2 ? V : 1); ++k) {
          const int ee = from + u * EPW + sub;
          w_next[u][k] = ee < total ? __ldg(a.edge_value + (EV == 2 ? (e0 + ee) * H + head[k] : e0 + ee)) : 0.f;
        }
    };
    int slot = 0;
    for (unsigned m = miss; m; m &= m - 1) {
      const int row = __ffs(m) - 1;
      const int b = __shfl_sync(kFull, off, row), end = __shfl_sync(kFull, off, row + 1);
      float acc[V][EL];
#pragma unroll
      for (int k = 0; k < V; ++k)
#pragma unroll
        for (int q = 0; q < EL; ++q) acc[k][q] = 0.f;
#pragma unroll 1
      for (int e = b; e < end; e += U * EPW) {
        float w[U][EV == 2 ? V : 1];
        if (EV) {
          if (e != w_at) load_weights(e);      // rows served from history were skipped
#pragma unroll
          for (int u = 0; u < U; ++u)
#pragma unroll
            for (int k = 0; k < (EV == 2 ? V : 1); ++k) w[u][k] = w_next[u][k];
          load_weights(e + U * EPW < end ? e + U * EPW : end);
        }
        cp_async_wait<D - 1>();
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (e + u * EPW + sub < end) {
            const int at = slot * Shape::kSlot + u * Shape::kReq;
#pragma unroll
            for (int k = 0; k < V; ++k) {
              if (v0 + gl + k * G < v1) {
                Vec x;
                x.load_shared(mine + at + k * VB * kWarp);
                if (EV) {
                  float f[EL];
                  x.unpack(f);
#pragma unroll
                  for (int q = 0; q < EL; ++q) acc[k][q] = fmaf(w[u][EV == 2 ? k : 0], f[q], acc[k][q]);
                } else {
                  x.add_to(acc[k]);
                }
              }
            }
          }
        }
        produce(slot);
        slot = slot + 1 == D ? 0 : slot + 1;
      }
      if (EPW > 1) {
#pragma unroll
        for (int o = G; o < kWarp; o <<= 1)
#pragma unroll
          for (int k = 0; k < V; ++k)
#pragma unroll
            for (int q = 0; q < EL; ++q) acc[k][q] += __shfl_xor_sync(kFull, acc[k][q], o);
      }
      if (sub == 0) {
        float* orow = out + (r0 + row) * width;
        if (!EV && end > b) {
          const float inv = __frcp_rn((float)(end - b));  // one correctly rounded reciprocal per row
#pragma unroll
          for (int k = 0; k < V; ++k)
#pragma unroll
            for (int q = 0; q < EL; ++q) acc[k][q] *= inv;
        }
#pragma unroll
        for (int k = 0; k < V; ++k) {
          const int v = v0 + gl + k * G;
          if (v < v1) store_f32<EL>(orow + v * EL, acc[k], policy);
        }
      }
    }
    cp_async_wait<0>();
  }
}

// ---------------------------------------------------------------------------
// forward, fp16 rows on odd 2-byte addresses: no asynchronous copy is that narrow, so the rows come
// through registers, U requests at a time; while they are on their way the warp loads the indices of
// its next row and the ptr / history entries of the one after.
// ---------------------------------------------------------------------------
template <int VB, int V>
struct FwdShape {
  static constexpr int words = (VB >= 4 ? VB / 4 : 1) * V;            // registers of one row per lane
  static constexpr int U = words >= 8 ? 4 : 8;                        // rows in flight per lane group
  static constexpr int kMinBlocks = words * U >= 32 ? 4 : 5;
};

template <typename T, int VB, int G, int V, int EV, bool MAP>
__global__ void __launch_bounds__(256, (FwdShape<VB, V>::kMinBlocks))
    aggr_fwd_kernel(const hc_aggr_args a, float* __restrict__ out, const int nvec, const int part_vec,
                    const int h_vec, const int stream_out) {
  HC_BAIL_IF_BAD()
  using Vec = LaneVec<T, VB>;
  constexpr int EL = Vec::kElems;
  constexpr int EPW = kWarp / G;
  constexpr int U = FwdShape<VB, V>::U;
  const int lane = threadIdx.x & 31;
  const int64_t step = (int64_t)gridDim.x * (blockDim.x >> 5);
  int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (r >= a.num_node) return;
  const int H = a.num_head;
  const int width = H * a.feat;
  const int v0 = blockIdx.y * part_vec;                       // this block's columns of the row
  const int v1 = v0 + part_vec < nvec ? v0 + part_vec : nvec;
  const int sub = lane / G, gl = lane % G;
  const T* __restrict__ in = reinterpret_cast<const T*>(a.input);
  const T* __restrict__ alt = reinterpret_cast<const T*>(a.src_alt);
  const uint64_t policy = l2_policy(stream_out != 0);
  int head[V];
#pragma unroll
  for (int k = 0; k < V; ++k) head[k] = EV == 2 ? (v0 + gl + k * G) * EL / a.feat : 0;

  // what is known of a row ahead of time, one value per lane: ptr[r], ptr[r + 1], hmap[r]
  auto row_meta = [&](int64_t row) -> int64_t {
    if (row < a.num_node) {
      if (lane < 2) return a.ptr[row + lane];
      if (lane == 2 && a.hmap) return a.hmap[row];
    }
    return lane < 2 ? 0 : -1;
  };
  int64_t meta = row_meta(r), meta_n = row_meta(r + step);
  uint32_t my_s = 0u;
  {   // the shuffles stand outside the condition: every lane takes part in them
    const int64_t at = shfl64(meta, 0) + lane, end = shfl64(meta, 1), hit = shfl64(meta, 2);
    if (at < end && hit == -1) my_s = (uint32_t)a.idx[at];
  }
  while (true) {
    const int64_t b = shfl64(meta, 0), e = shfl64(meta, 1), hid = shfl64(meta, 2);
    float acc[V][EL];
#pragma unroll
    for (int k = 0; k < V; ++k)
#pragma unroll
      for (int q = 0; q < EL; ++q) acc[k][q] = 0.f;
    uint32_t next_s = 0u;
    int64_t meta_2 = -1;
    bool fetched = false;
    // what the following rows need, issued behind the first batch of this row's loads
    auto fetch_next = [&]() {
      if (fetched) return;
      fetched = true;
      const int64_t at = shfl64(meta_n, 0) + lane, end = shfl64(meta_n, 1), hit = shfl64(meta_n, 2);
      if (at < end && hit == -1) next_s = (uint32_t)a.idx[at];
      meta_2 = row_meta(r + 2 * step);
    };
    float* __restrict__ orow = out + r * width;
    if (hid == -1) {
      for (int64_t i = b; i < e; i += kWarp) {
        const int cnt = (int)((e - i) < (int64_t)kWarp ? (e - i) : (int64_t)kWarp);
        if (i != b) my_s = i + lane < e ? (uint32_t)a.idx[i + lane] : 0u;
        bool my_alt = false;
        if (MAP && lane < cnt) {
          const int64_t m = a.src_map[my_s];
          my_alt = m != -1;
          if (my_alt) my_s = (uint32_t)m;
        }
        float my_w = 0.f;
        if (EV == 1 && lane < cnt) my_w = a.edge_value[i + lane];
        const unsigned alts = MAP ? __ballot_sync(kFull, my_alt) : 0u;
        for (int j = 0; j < cnt; j += EPW * U) {
          Vec buf[U][V];
          float w[U][EV == 2 ? V : 1];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (j + u * EPW < cnt) {  // warp-uniform
              const int jj = j + u * EPW + sub;
              const bool ok = jj < cnt;
              const uint32_t s = __shfl_sync(kFull, my_s, jj & 31);
              if (EV == 1) w[u][0] = __shfl_sync(kFull, my_w, jj & 31);   // lanes behind cnt hold 0
              const T* row = (MAP && ((alts >> (jj & 31)) & 1u)) ? alt + (int64_t)s * a.alt_stride
                                                                 : in + (int64_t)s * a.in_stride;
#pragma unroll
              for (int k = 0; k < V; ++k) {
                const int v = v0 + gl + k * G;
                buf[u][k].clear();
                if (EV == 2) w[u][k] = 0.f;
                if (ok && v < v1) {
                  buf[u][k].load(row + v * EL);
                  if (EV == 2) w[u][k] = __ldg(a.edge_value + (i + jj) * H + head[k]);
                }
              }
            }
          }
          fetch_next();
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (j + u * EPW < cnt) {
#pragma unroll
              for (int k = 0; k < V; ++k) {
                if (EV) {
                  float f[EL];
                  buf[u][k].unpack(f);
#pragma unroll
                  for (int q = 0; q < EL; ++q) acc[k][q] = fmaf(w[u][EV == 2 ? k : 0], f[q], acc[k][q]);
                } else {
                  buf[u][k].add_to(acc[k]);
                }
              }
            }
          }
        }
      }
      fetch_next();      // a row without edges
      if (EPW > 1) {
#pragma unroll
        for (int off = G; off < kWarp; off <<= 1)
#pragma unroll
          for (int k = 0; k < V; ++k)
#pragma unroll
            for (int q = 0; q < EL; ++q) acc[k][q] += __shfl_xor_sync(kFull, acc[k][q], off);
      }
      if (sub == 0) {
        if (!EV && e > b) {
          const float inv = __frcp_rn((float)(e - b));  // one correctly rounded reciprocal per row
#pragma unroll
          for (int k = 0; k < V; ++k)
#pragma unroll
            for (int q = 0; q < EL; ++q) acc[k][q] *= inv;
        }
#pragma unroll
        for (int k = 0; k < V; ++k) {
          const int v = v0 + gl + k * G;
          if (v < v1) store_f32<EL>(orow + v * EL, acc[k], policy);
        }
      }
    } else {
      fetch_next();
      copy_history_part<EL>(a, a.h_indexed ? hid : r, orow, width, v0, v1, lane, h_vec);
    }
    r += step;
    if (r >= a.num_node) return;
    meta = meta_n;
    meta_n = meta_2;
    my_s = next_s;
  }
}

// ---------------------------------------------------------------------------
// forward, generic path: any dtype mix, source ids beyond 32 bits, odd widths with weights per head
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
    aggr_fwd_generic_kernel(const hc_aggr_args a, float* __restrict__ out) {
  HC_BAIL_IF_BAD()
  const int lane = threadIdx.x & 31;
  const int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int H = a.num_head, F = a.feat;
  if (t >= a.num_node * H) return;
  const int64_t r = t / H;
  const int h = (int)(t % H);
  float* __restrict__ orow = out + t * F;
  const int64_t hid = a.hmap ? a.hmap[r] : -1;
  if (hid != -1) {
    const int64_t off = (a.h_indexed ? hid : r) * a.hsize + (a.hsize == F ? 0 : (int64_t)h * F);
    for (int c = lane; c < F; c += kWarp) orow[c] = load_as_f32(a.hbuf, a.h_dtype, off + c);
    return;
  }
  const int64_t begin = a.ptr[r], end = a.ptr[r + 1];
  const int64_t deg = end - begin;
  const bool ev = a.edge_value != nullptr;
  for (int c0 = 0; c0 < F; c0 += 128) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int64_t e = begin; e < end; ++e) {
      const int64_t s = a.idx[e];
      const int64_t al = a.src_map ? a.src_map[s] : -1;
      const float w = ev ? a.edge_value[e * H + h] : 1.f;
      const void* base = al != -1 ? a.src_alt : a.input;
      const int dt = al != -1 ? a.alt_dtype : a.in_dtype;
      const int64_t off = (al != -1 ? al * a.alt_stride : s * a.in_stride) + (int64_t)h * F;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int c = c0 + lane + 32 * k;
        if (c < F) acc[k] = fmaf(w, load_as_f32(base, dt, off + c), acc[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = c0 + lane + 32 * k;
      if (c < F) orow[c] = (!ev && deg > 0) ? __fdiv_rn(acc[k], (float)deg) : acc[k];
    }
  }
}

// ---------------------------------------------------------------------------
// backward, 16-byte vector path
//   MH  several heads (one warp per (row, head) target; fp32 source rows)
//   EG  also the gradient of the edge values: edge_grad[e(, h)] = <grad_out[t], source row>, the
//       dot product taken by the G lanes that share the row and written once (every edge of every
//       head belongs to exactly one target, so no atomics)
// ---------------------------------------------------------------------------
template <int G, int V, bool EV, bool MH = false, bool EG = false>
__global__ void __launch_bounds__(256)
    aggr_bwd_vec_kernel(const hc_aggr_args a, const float* __restrict__ grad_out,
                        float* __restrict__ grad_input, float* __restrict__ grad_history,
                        float* __restrict__ row_score_out, const int score_kind, const int nvec,
                        const int64_t gi_stride, float* __restrict__ edge_grad, const int64_t go_stride) {
  HC_BAIL_IF_BAD()
  constexpr int EPW = kWarp / G;
  const int lane = threadIdx.x & 31;
  const int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int H = MH ? a.num_head : 1;
  if (t >= a.num_node * H) return;
  const int64_t r = MH ? t / H : t;
  const int h = MH ? (int)(t - r * H) : 0;
  const int F = a.feat;
  const int sub = lane / G, gl = lane % G;

  float4 g[V];
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int v = gl + k * G;
    g[k] = v < nvec ? __ldg(reinterpret_cast<const float4*>(grad_out + t * go_stride) + v)
                    : make_float4(0.f, 0.f, 0.f, 0.f);
  }

  if (!MH && row_score_out) {
    float p = 0.f;
    if (sub == 0) {
#pragma unroll
      for (int k = 0; k < V; ++k) {
        p = score_term(p, g[k].x, score_kind);
        p = score_term(p, g[k].y, score_kind);
        p = score_term(p, g[k].z, score_kind);
        p = score_term(p, g[k].w, score_kind);
      }
    }
    p = score_finish(p, score_kind);
    if (lane == 0) row_score_out[r] = p;
  }

  const int64_t hid = a.hmap ? a.hmap[r] : -1;
  if (grad_history && sub == 0) {
    // per-head history rows (hsize == num_head * feat) or a single head
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    float* hrow = grad_history + r * a.hsize + (MH ? (int64_t)h * F : 0);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int v = gl + k * G;
      if (v < nvec) reinterpret_cast<float4*>(hrow)[v] = hid != -1 ? g[k] : z;
    }
  }
  const int64_t begin = a.ptr[r], end = a.ptr[r + 1];
  if (hid != -1) {
    // edges of a history row carry no gradient (zeros_like in the reference, :536)
    if (EG)
      for (int64_t e = begin + lane; e < end; e += kWarp) edge_grad[MH ? e * H + h : e] = 0.f;
    return;
  }
  if (grad_input == nullptr && !EG) return;
  const int64_t deg = end - begin;
  if (deg == 0) return;
  if (!EV) {
    const float inv = __frcp_rn((float)deg);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      g[k].x *= inv;
      g[k].y *= inv;
      g[k].z *= inv;
      g[k].w *= inv;
    }
  }
  const bool has_map = a.src_map != nullptr;
  const float* __restrict__ in = reinterpret_cast<const float*>(a.input) + (MH ? (int64_t)h * F : 0);
  const float* __restrict__ alt = reinterpret_cast<const float*>(a.src_alt) + (MH ? (int64_t)h * F : 0);
  for (int64_t i = begin; i < end; i += kWarp) {
    int64_t my_s = 0, my_alt = -1;
    float my_w = 0.f;
    if (i + lane < end) {
      my_s = a.idx[i + lane];
      if (has_map) my_alt = a.src_map[my_s];
      if (EV) my_w = MH ? a.edge_value[(i + lane) * H + h] : a.edge_value[i + lane];
    }
    const int cnt = (int)((end - i) < (int64_t)kWarp ? (end - i) : (int64_t)kWarp);
    for (int j = 0; j < cnt; j += EPW) {
      const int jj = j + sub;
      const int from = jj & 31;
      const int64_t s = shfl64(my_s, from);
      const int64_t al = has_map ? shfl64(my_alt, from) : -1;
      const float w = EV ? __shfl_sync(kFull, my_w, from) : 1.f;
      const bool ok = jj < cnt;
      if (EG) {
        float dot = 0.f;
        if (ok) {
          const float* row = al != -1 ? alt + al * a.alt_stride : in + s * a.in_stride;
#pragma unroll
          for (int k = 0; k < V; ++k) {
            const int v = gl + k * G;
            if (v < nvec) {
              const float4 x = __ldg(reinterpret_cast<const float4*>(row) + v);
              dot = fmaf(g[k].x, x.x, dot);
              dot = fmaf(g[k].y, x.y, dot);
              dot = fmaf(g[k].z, x.z, dot);
              dot = fmaf(g[k].w, x.w, dot);
            }
          }
        }
#pragma unroll
        for (int off = 1; off < G; off <<= 1) dot += __shfl_xor_sync(kFull, dot, off);
        if (ok && gl == 0) edge_grad[MH ? (i + jj) * H + h : (i + jj)] = dot;
      }
      if (ok && al == -1 && grad_input != nullptr) {
        float* dst = grad_input + s * gi_stride + (MH ? (int64_t)h * F : 0);
#pragma unroll
        for (int k = 0; k < V; ++k) {
          const int v = gl + k * G;
          if (v < nvec) {
            if (EV)
              red_add_v4(dst + 4 * v, g[k].x * w, g[k].y * w, g[k].z * w, g[k].w * w);
            else
              red_add_v4(dst + 4 * v, g[k].x, g[k].y, g[k].z, g[k].w);
          }
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// backward, rows of any width (one head, no edge gradients)
// ---------------------------------------------------------------------------
// What bounds the scatter is the number of reductions, not their bytes: 16-byte ones move about 2.2 times
// as many values per second as 4-byte ones.  Rows whose width is no multiple of four start anywhere, so
// the warp keeps its (scaled) gradient row in shared memory four times, shifted by 0..3 values: for a
// source row that starts `shift` values behind a 16-byte boundary, word w of the copy `shift` is what the
// w-th aligned word of that row gets.  The first and the last word reach into the neighbouring rows, which
// get zeros added.  60 K rows, 720 K edges of 75 columns: 123 us with 4-byte reductions.
__host__ __device__ inline int shift_words(int feat) { return (feat + 6) / 4; }   // of a shifted row, at most

template <bool EV>
__global__ void __launch_bounds__(256)
    aggr_bwd_shift_kernel(const hc_aggr_args a, const float* __restrict__ grad_out, float* __restrict__ grad_input,
                          float* __restrict__ grad_history, float* __restrict__ row_score_out, const int score_kind) {
  HC_BAIL_IF_BAD()
  extern __shared__ __align__(16) float sh[];
  const int lane = threadIdx.x & 31;
  const int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (r >= a.num_node) return;
  const int F = a.feat, words = shift_words(F);
  float* copies = sh + (size_t)(threadIdx.x >> 5) * 16 * words;     // [4][words * 4]
  const float* __restrict__ grow = grad_out + r * F;
  if (row_score_out) {
    const float s = row_score(grow, F, score_kind, lane);
    if (lane == 0) row_score_out[r] = s;
  }
  const int64_t hid = a.hmap ? a.hmap[r] : -1;
  if (grad_history)
    for (int c = lane; c < F; c += kWarp) grad_history[r * a.hsize + c] = hid != -1 ? grow[c] : 0.f;
  if (hid != -1 || grad_input == nullptr) return;
  const int64_t begin = a.ptr[r], end = a.ptr[r + 1];
  if (begin == end) return;
  const float scale = EV ? 1.f : __frcp_rn((float)(end - begin));
  const int64_t values = a.n_src * F;
  for (int c = lane; c < 4 * words; c += kWarp) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int col = c - k;
      copies[k * 4 * words + c] = col >= 0 && col < F ? grow[col] * scale : 0.f;
    }
  }
  __syncwarp();
  for (int64_t i = begin; i < end; i += kWarp) {
    int64_t my_s = -1;      // < 0: no gradient (read from the alternative table)
    float my_w = 0.f;
    if (i + lane < end) {
      my_s = a.idx[i + lane];
      if (a.src_map && a.src_map[my_s] != -1) my_s = -1;
      if (EV) my_w = a.edge_value[i + lane];
    }
    const int cnt = (int)((end - i) < (int64_t)kWarp ? (end - i) : (int64_t)kWarp);
    for (int j = 0; j < cnt; ++j) {
      const int64_t s = shfl64(my_s, j);
      const float w = EV ? __shfl_sync(kFull, my_w, j) : 1.f;
      if (s < 0) continue;
      const int64_t o = s * F;
      const int shift = (int)(o & 3);
      const int n = (shift + F + 3) >> 2;
      const float4* copy = reinterpret_cast<const float4*>(copies + shift * 4 * words);
      float* dst = grad_input + (o - shift);
      for (int v = lane; v < n; v += kWarp) {
        float4 g = copy[v];
        if (EV) {
          g.x *= w; g.y *= w; g.z *= w; g.w *= w;
        }
        if (EV && (v == 0 || 4 * v + 4 - shift > F)) {      // 0 * w may be NaN
          const int c = 4 * v - shift;
          if (c < 0 || c >= F) g.x = 0.f;
          if (c + 1 < 0 || c + 1 >= F) g.y = 0.f;
          if (c + 2 < 0 || c + 2 >= F) g.z = 0.f;
          if (c + 3 >= F) g.w = 0.f;
        }
        if (o - shift + 4 * v + 4 <= values) {
          red_add_v4(dst + 4 * v, g.x, g.y, g.z, g.w);
        } else {      // the array ends inside this word
          const float f[3] = {g.x, g.y, g.z};
          for (int k = 0; k < 3; ++k)
            if (o - shift + 4 * v + k < values) red_add<1>(dst + 4 * v + k, f + k);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// backward, generic path: any F, multi-head, edge_grad
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
    aggr_bwd_generic_kernel(const hc_aggr_args a, const float* __restrict__ grad_out,
                            float* __restrict__ grad_input, float* __restrict__ grad_history,
                            float* __restrict__ edge_grad, float* __restrict__ row_score_out,
                            const int score_kind, const int64_t gi_stride) {
  HC_BAIL_IF_BAD()
  const int lane = threadIdx.x & 31;
  const int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int H = a.num_head, F = a.feat;
  if (t >= a.num_node * H) return;
  const int64_t r = t / H;
  const int h = (int)(t % H);
  const float* __restrict__ grow = grad_out + t * F;
  if (row_score_out && H == 1) {
    const float s = row_score(grow, F, score_kind, lane);
    if (lane == 0) row_score_out[r] = s;
  }
  const int64_t hid = a.hmap ? a.hmap[r] : -1;
  const bool heads_share_history = H > 1 && a.hsize == F;
  if (grad_history) {
    float* dst = grad_history + r * a.hsize + (a.hsize == F ? 0 : (int64_t)h * F);
    if (heads_share_history) {
      // all heads of a hit row add into one row; the launcher cleared it
      if (hid != -1)
        for (int c = lane; c < F; c += kWarp) atomicAdd(dst + c, grow[c]);
    } else {
      for (int c = lane; c < F; c += kWarp) dst[c] = hid != -1 ? grow[c] : 0.f;
    }
  }
  const int64_t begin = a.ptr[r], end = a.ptr[r + 1];
  if (hid != -1) {
    // edges of a history row carry no gradient (zeros_like in the reference, :536)
    if (edge_grad)
      for (int64_t e = begin + lane; e < end; e += kWarp) edge_grad[e * H + h] = 0.f;
    return;
  }
  if (grad_input == nullptr && edge_grad == nullptr) return;
  const int64_t deg = end - begin;
  const bool ev = a.edge_value != nullptr;
  for (int64_t e = begin; e < end; ++e) {
    const int64_t s = a.idx[e];
    const int64_t al = a.src_map ? a.src_map[s] : -1;
    const float w = ev ? a.edge_value[e * H + h] : 1.f;
    float dot = 0.f;
    for (int c = lane; c < F; c += kWarp) {
      const float gv = grow[c];
      if (grad_input && al == -1) {
        const float val = ev ? gv * w : __fdiv_rn(gv, (float)deg);
        atomicAdd(grad_input + s * gi_stride + (int64_t)h * F + c, val);
      }
      if (edge_grad) {
        const void* base = al != -1 ? a.src_alt : a.input;
        const int dt = al != -1 ? a.alt_dtype : a.in_dtype;
        const int64_t off = (al != -1 ? al * a.alt_stride : s * a.in_stride) + (int64_t)h * F;
        dot = fmaf(gv, load_as_f32(base, dt, off + c), dot);
      }
    }
    if (edge_grad) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) dot += __shfl_xor_sync(kFull, dot, off);
      if (lane == 0) edge_grad[e * H + h] = dot;
    }
  }
}

// grad_input before the scatter: row r < rooted starts from root[r], the others from zero
__global__ void __launch_bounds__(256)
    start_rows_kernel(float* __restrict__ grad_input, const int64_t rows, const int64_t nvec,
                      const float* __restrict__ root, const int64_t root_stride, const int64_t rooted) {
  const int64_t total = rows * nvec;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / nvec;
    reinterpret_cast<float4*>(grad_input)[i] =
        r < rooted ? *reinterpret_cast<const float4*>(root + r * root_stride + 4 * (i - r * nvec)) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static int validate(const hc_aggr_args* a, hc_aggr_args* n) {
  HC_REQUIRE(a != nullptr, HC_ERR_NULL);
  HC_REQUIRE(a->struct_size == sizeof(hc_aggr_args), HC_ERR_STRUCT);
  *n = *a;
  HC_REQUIRE(n->num_node >= 0 && n->feat > 0 && n->num_head >= 1 && n->n_src >= 0, HC_ERR_SIZE);
  if (n->num_node == 0) return 0;
  HC_REQUIRE(n->ptr && n->idx && n->input, HC_ERR_NULL);
  HC_REQUIRE(dtype_size(n->in_dtype) != 0, HC_ERR_DTYPE);
  const int64_t row = (int64_t)n->num_head * n->feat;
  if (n->in_stride == 0) n->in_stride = row;
  HC_REQUIRE(n->in_stride >= row, HC_ERR_SIZE);
  HC_REQUIRE(aligned_to(n->ptr, 8) && aligned_to(n->idx, 8), HC_ERR_ALIGN);
  HC_REQUIRE(aligned_to(n->input, dtype_size(n->in_dtype)), HC_ERR_ALIGN);
  if (n->src_map) {
    HC_REQUIRE(n->src_alt != nullptr, HC_ERR_NULL);
    HC_REQUIRE(dtype_size(n->alt_dtype) != 0, HC_ERR_DTYPE);
    if (n->alt_stride == 0) n->alt_stride = row;
    HC_REQUIRE(n->alt_stride >= row, HC_ERR_SIZE);
  }
  if (n->hmap) {
    HC_REQUIRE(n->hbuf != nullptr, HC_ERR_NULL);
    HC_REQUIRE(dtype_size(n->h_dtype) != 0, HC_ERR_DTYPE);
    // history rows are either shared by the heads or one segment per head
    // (the reference asserts on the device: history_aggr.cu:97-106)
    HC_REQUIRE(n->hsize >= n->feat, HC_ERR_SIZE);
    HC_REQUIRE(n->num_head == 1 || n->hsize == n->feat || n->hsize == row, HC_ERR_SIZE);
  }
  return 0;
}

static int vec_shape(int nvec, int* G, int* V) {
  if (nvec <= 8) { *G = 8; *V = 1; }
  else if (nvec <= 16) { *G = 16; *V = 1; }
  else if (nvec <= 32) { *G = 32; *V = 1; }
  else if (nvec <= 64) { *G = 32; *V = 2; }
  else if (nvec <= 96) { *G = 32; *V = 3; }
  else if (nvec <= 128) { *G = 32; *V = 4; }
  else if (nvec <= 192) { *G = 32; *V = 6; }
  else if (nvec <= 256) { *G = 32; *V = 8; }
  else return 0;
  return 1;
}

// Widest unit (16, 8, 4 or 2 bytes) that divides every given address or length; never below `es`.
static int lane_bytes(uintptr_t bits, int es) {
  for (int vb = 16; vb > es; vb >>= 1)
    if (bits % vb == 0) return vb;
  return es;
}

struct FwdLaunch {
  hc_aggr_args a;
  float* out;
  int nvec, h_vec, stream_out;
  cudaStream_t st;
};

struct FwdGrid {
  dim3 grid;
  int part_vec, run_rows;
};
// column parts of about equal width that start on a float4 of the output row, and one wave of blocks
static FwdGrid fwd_grid(const FwdLaunch& l, int el, int most_vec, int min_blocks, int max_run) {
  FwdGrid g;
  const int parts = (int)ceil_div(l.nvec, most_vec);
  const int unit = el < 4 ? 4 / el : 1;
  g.part_vec = (int)ceil_div(ceil_div(l.nvec, parts), unit) * unit;
  if (g.part_vec > most_vec) g.part_vec = most_vec;           // most_vec is a multiple of 4
  g.grid.y = (unsigned)ceil_div(l.nvec, g.part_vec);
  int64_t most = 148 * min_blocks / g.grid.y;
  if (most < 1) most = 1;
  // every warp gets the same number of runs, as long as they may be: a short run leaves the start of its
  // pipeline uncovered
  const int64_t per_warp = ceil_div(l.a.num_node, most * 8);
  const int64_t run = ceil_div(per_warp, ceil_div(per_warp, max_run));
  const int64_t blocks = ceil_div(ceil_div(l.a.num_node, run), 8);
  g.run_rows = (int)run;
  g.grid.x = (unsigned)(blocks < most ? blocks : most);
  return g;
}

template <typename T, int VB, int G, int V, int EV, bool MAP>
static void launch_fwd_one(const FwdLaunch& l) {
  if constexpr (VB == 2) {
    const FwdGrid g = fwd_grid(l, 1, G * V, FwdShape<VB, V>::kMinBlocks, 1);
    aggr_fwd_kernel<T, VB, G, V, EV, MAP><<<g.grid, 256, 0, l.st>>>(l.a, l.out, l.nvec, g.part_vec, l.h_vec, l.stream_out);
  } else {
    using Shape = StreamShape<VB, V, EV>;
    auto kernel = aggr_fwd_stream_kernel<T, VB, G, V, EV, MAP>;
    static std::atomic<uint64_t> raised{0};
    if (Shape::kSmem > 48 * 1024) raise_smem(kernel, Shape::kSmem, raised);
    const FwdGrid g = fwd_grid(l, LaneVec<T, VB>::kElems, G * V, Shape::kMinBlocks, kMaxRun);
    kernel<<<g.grid, 256, Shape::kSmem, l.st>>>(l.a, l.out, l.nvec, g.part_vec, l.h_vec, l.stream_out, g.run_rows);
  }
}

template <typename T, int EV, bool MAP>
static void launch_fwd_wide(const FwdLaunch& l) {
  if (l.nvec <= 8) launch_fwd_one<T, 16, 8, 1, EV, MAP>(l);
  else if (l.nvec <= 16) launch_fwd_one<T, 16, 16, 1, EV, MAP>(l);
  else if (l.nvec <= 32) launch_fwd_one<T, 16, 32, 1, EV, MAP>(l);
  else launch_fwd_one<T, 16, 32, 2, EV, MAP>(l);
}
template <typename T, int VB, int EV>
static void launch_fwd_narrow(const FwdLaunch& l) {
  if (l.nvec <= 16) launch_fwd_one<T, VB, 16, 1, EV, false>(l);
  else if (l.nvec <= 32) launch_fwd_one<T, VB, 32, 1, EV, false>(l);
  else if (l.nvec <= 64) launch_fwd_one<T, VB, 32, 2, EV, false>(l);
  else if (l.nvec <= 96) launch_fwd_one<T, VB, 32, 3, EV, false>(l);
  else launch_fwd_one<T, VB, 32, 4, EV, false>(l);
}
template <typename T, int EV>
static bool launch_fwd_any(const FwdLaunch& l, int vb) {
  if (vb == 16) {
    if (l.a.src_map) launch_fwd_wide<T, EV, true>(l);
    else launch_fwd_wide<T, EV, false>(l);
    return true;
  }
  if constexpr (EV != 2) {
    if (l.a.src_map) return false;
    if (vb == 8) launch_fwd_narrow<T, 8, EV>(l);
    else if (vb == 4) launch_fwd_narrow<T, 4, EV>(l);
    else if constexpr (sizeof(T) == 2) launch_fwd_narrow<T, 2, EV>(l);
    return true;
  }
  return false;
}
template <typename T>
static bool launch_fwd(const FwdLaunch& l, int vb) {
  if (!l.a.edge_value) return launch_fwd_any<T, 0>(l, vb);
  return l.a.num_head == 1 ? launch_fwd_any<T, 1>(l, vb) : launch_fwd_any<T, 2>(l, vb);
}

template <bool EV>
static void launch_bwd_vec(int G, int V, dim3 grid, cudaStream_t st, const hc_aggr_args& a,
                           const float* grad_out, float* grad_input, float* grad_history,
                           float* row_score, int score_kind, int nvec, int64_t gi_stride, int64_t go_stride) {
#define HC_BWD_CASE(g, v)                                                                  \
  if (G == g && V == v) {                                                                  \
    aggr_bwd_vec_kernel<g, v, EV><<<grid, 256, 0, st>>>(a, grad_out, grad_input,           \
                                                        grad_history, row_score,           \
                                                        score_kind, nvec, gi_stride, nullptr, go_stride); \
    return;                                                                                \
  }
  HC_BWD_CASE(8, 1) HC_BWD_CASE(16, 1) HC_BWD_CASE(32, 1) HC_BWD_CASE(32, 2)
  HC_BWD_CASE(32, 3) HC_BWD_CASE(32, 4) HC_BWD_CASE(32, 6) HC_BWD_CASE(32, 8)
#undef HC_BWD_CASE
}

// edge-weighted backward with several heads and / or the gradient of the edge values (fp32 rows)
template <bool MH, bool EG>
static void launch_bwd_heads(int G, int V, dim3 grid, cudaStream_t st, const hc_aggr_args& a,
                             const float* grad_out, float* grad_input, float* grad_history,
                             float* row_score, int score_kind, int nvec, int64_t gi_stride,
                             float* edge_grad) {
#define HC_BWD_CASE(g, v)                                                                          \
  if (G == g && V == v) {                                                                          \
    aggr_bwd_vec_kernel<g, v, true, MH, EG><<<grid, 256, 0, st>>>(a, grad_out, grad_input,         \
                                                                  grad_history, row_score,         \
                                                                  score_kind, nvec, gi_stride,     \
                                                                  edge_grad, a.feat);              \
    return;                                                                                        \
  }
  HC_BWD_CASE(8, 1) HC_BWD_CASE(16, 1) HC_BWD_CASE(32, 1) HC_BWD_CASE(32, 2)
  HC_BWD_CASE(32, 3) HC_BWD_CASE(32, 4) HC_BWD_CASE(32, 6) HC_BWD_CASE(32, 8)
#undef HC_BWD_CASE
}

}  // namespace hc

using namespace hc;

#ifdef HC_CHECK_BOUNDS
#define HC_CHECK_BLOCK(a, st)                                                                 \
  do {                                                                                        \
    const int64_t cb_ = ceil_div((a).num_node * 8, 256);                                      \
    HC_REQUIRE(cb_ <= 0x7fffffffLL, HC_ERR_SIZE);                                             \
    aggr_check_kernel<<<(unsigned)cb_, 256, 0, st>>>(a);                                      \
  } while (0)
#else
#define HC_CHECK_BLOCK(a, st)
#endif

extern "C" int hc_last_status(int64_t out[4], int32_t clear, void* stream) {
#ifdef HC_CHECK_BOUNDS
  HC_REQUIRE(out != nullptr, HC_ERR_NULL);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  HC_CUDA(cudaStreamSynchronize(st));
  unsigned long long h[4];
  HC_CUDA(cudaMemcpyFromSymbol(h, g_status, sizeof(h)));
  for (int i = 0; i < 4; ++i) out[i] = (int64_t)h[i];
  if (clear) {
    const unsigned long long z[4] = {0, 0, 0, 0};
    HC_CUDA(cudaMemcpyToSymbol(g_status, z, sizeof(z)));
  }
  return 0;
#else
  (void)out; (void)clear; (void)stream;
  return -HC_ERR_UNSUPPORTED;
#endif
}

extern "C" int hc_aggr_fwd(const hc_aggr_args* args, float* out, void* stream) {
  hc_aggr_args a;
  int rc = validate(args, &a);
  if (rc) return rc;
  if (a.num_node == 0) return 0;
  HC_REQUIRE(out != nullptr, HC_ERR_NULL);
  HC_REQUIRE(aligned_to(out, 4), HC_ERR_ALIGN);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  HC_CHECK_BLOCK(a, st);
  const int s = dtype_size(a.in_dtype);
  // The vector kernels take rows of one storage type and source ids of 32 bits.  The unit that a lane
  // moves has to divide a row's length and every row's address, and with weights per head it may not
  // straddle two heads.
  const int64_t width = (int64_t)a.num_head * a.feat;
  const bool per_head = a.edge_value != nullptr && a.num_head > 1;
  uintptr_t bits = reinterpret_cast<uintptr_t>(a.input) | (uintptr_t)(a.in_stride * s) |
                   (uintptr_t)((per_head ? a.feat : width) * s);
  bool vec = width * s <= (1 << 20) && a.n_src <= 0xffffffffLL;
  if (a.src_map) {
    vec = vec && a.alt_dtype == a.in_dtype;
    bits |= reinterpret_cast<uintptr_t>(a.src_alt) | (uintptr_t)(a.alt_stride * s);
  }
  int vb = lane_bytes(bits, s);
  while (vb > s && !aligned_to(out, (size_t)(vb / s * 4 < 16 ? vb / s * 4 : 16))) vb >>= 1;
  FwdLaunch l;
  l.a = a;
  l.out = out;
  l.st = st;
  l.nvec = (int)(width * s / vb);
  // results of more than half the L2 are not read from it again
  l.stream_out = a.num_node * width * 4 > (64 << 20);
  l.h_vec = 0;
  if (a.hmap) {
    const int hs = dtype_size(a.h_dtype);
    l.h_vec = aligned16(out) && a.feat % 4 == 0 && aligned_to(a.hbuf, 4 * hs) && a.hsize % 4 == 0;
  }
  if (!(vec && (a.in_dtype == HC_F32 ? launch_fwd<float>(l, vb) : launch_fwd<__half>(l, vb)))) {
    const int64_t blocks = ceil_div(a.num_node * a.num_head, 8);
    HC_REQUIRE(blocks <= 0x7fffffffLL, HC_ERR_SIZE);
    aggr_fwd_generic_kernel<<<(unsigned)blocks, 256, 0, st>>>(a, out);
  }
  HC_LAUNCH_OK();
  return 0;
}

extern "C" int hc_aggr_bwd_rooted(const hc_aggr_args* args, const float* grad_out, int64_t go_stride, const float* root,
                                  int64_t root_stride, float* grad_input, int32_t zero_grad_input,
                                  float* grad_history, float* edge_grad, float* row_score, int32_t score_kind,
                                  void* stream) {
  hc_aggr_args a;
  int rc = validate(args, &a);
  if (rc) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int64_t row = (int64_t)a.num_head * a.feat;
  const int64_t gi_stride = row;  // grad_input is dense [n_src, num_head, feat]
  if (go_stride == 0) go_stride = row;
  if (root && root_stride == 0) root_stride = row;
  HC_REQUIRE(go_stride >= row && (!root || root_stride >= row), HC_ERR_SIZE);
  HC_REQUIRE(!root || (grad_input && a.num_node <= a.n_src), HC_ERR_UNSUPPORTED);
  if (grad_input && zero_grad_input && a.n_src > 0) {
    if (root) {
      HC_REQUIRE(row % 4 == 0 && root_stride % 4 == 0 && aligned16(root) && aligned16(grad_input), HC_ERR_UNSUPPORTED);
      const int64_t blocks = ceil_div(a.n_src * row / 4, 256 * 4);
      start_rows_kernel<<<(unsigned)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, st>>>(grad_input, a.n_src, row / 4, root,
                                                                                         root_stride, a.num_node);
    } else {
      HC_CUDA(cudaMemsetAsync(grad_input, 0, (size_t)a.n_src * row * sizeof(float), st));
    }
  }
  if (a.num_node == 0) return 0;
  HC_REQUIRE(grad_out != nullptr, HC_ERR_NULL);
  HC_REQUIRE(score_kind == HC_SCORE_L2 || score_kind == HC_SCORE_L1, HC_ERR_SIZE);
  HC_CHECK_BLOCK(a, st);
  HC_REQUIRE(!(row_score && a.num_head != 1), HC_ERR_UNSUPPORTED);
  HC_REQUIRE(!(edge_grad && !a.edge_value), HC_ERR_UNSUPPORTED);
  HC_REQUIRE(!(grad_history && !a.hmap), HC_ERR_NULL);
  if (grad_history && a.num_head > 1 && a.hsize == a.feat)
    HC_CUDA(cudaMemsetAsync(grad_history, 0, (size_t)a.num_node * a.hsize * sizeof(float), st));

  const bool heads = a.num_head > 1;
  bool vec = a.feat % 4 == 0 && aligned16(grad_out) && go_stride % 4 == 0 && (grad_input == nullptr || aligned16(grad_input)) &&
             (grad_history == nullptr || (aligned16(grad_history) && a.hsize % 4 == 0));
  // several heads / the gradient of the edge values: vector path for edge-weighted sums over fp32
  // rows, with per-head (or single-head) history rows
  const bool special = heads || edge_grad != nullptr;
  if (vec && special) {
    vec = a.edge_value != nullptr && a.in_dtype == HC_F32 && aligned16(a.input) && a.in_stride % 4 == 0 &&
          (!a.src_map || (a.alt_dtype == HC_F32 && aligned16(a.src_alt) && a.alt_stride % 4 == 0)) &&
          (grad_history == nullptr || !heads || a.hsize == row) &&
          (edge_grad == nullptr || aligned_to(edge_grad, 4));
  }
  int G = 0, V = 0;
  const int nvec = a.feat / 4;
  if (vec) vec = vec_shape(nvec, &G, &V) != 0;
  HC_REQUIRE(go_stride == row || (vec && !special), HC_ERR_UNSUPPORTED);
  const int64_t targets = a.num_node * a.num_head;
  const int64_t blocks = ceil_div(targets, 8);
  HC_REQUIRE(blocks <= 0x7fffffffLL, HC_ERR_SIZE);
  dim3 grid((unsigned)blocks);
  if (vec && special) {
    if (heads && edge_grad)
      launch_bwd_heads<true, true>(G, V, grid, st, a, grad_out, grad_input, grad_history, row_score,
                                   score_kind, nvec, gi_stride, edge_grad);
    else if (heads)
      launch_bwd_heads<true, false>(G, V, grid, st, a, grad_out, grad_input, grad_history, row_score,
                                    score_kind, nvec, gi_stride, nullptr);
    else
      launch_bwd_heads<false, true>(G, V, grid, st, a, grad_out, grad_input, grad_history, row_score,
                                    score_kind, nvec, gi_stride, edge_grad);
  } else if (vec) {
    if (a.edge_value)
      launch_bwd_vec<true>(G, V, grid, st, a, grad_out, grad_input, grad_history, row_score,
                           score_kind, nvec, gi_stride, go_stride);
    else
      launch_bwd_vec<false>(G, V, grid, st, a, grad_out, grad_input, grad_history, row_score,
                            score_kind, nvec, gi_stride, go_stride);
  } else if (!special && a.feat <= 512 && (grad_input == nullptr || aligned16(grad_input))) {
    // four copies of a row per warp: up to 66 KB of shared memory at 512 columns
    const int smem = 8 * 16 * shift_words(a.feat) * 4;
    static std::atomic<uint64_t> raised[2];
    if (smem > 48 * 1024) {
      const int most = 8 * 16 * shift_words(512) * 4;
      if (a.edge_value) raise_smem(aggr_bwd_shift_kernel<true>, most, raised[1]);
      else raise_smem(aggr_bwd_shift_kernel<false>, most, raised[0]);
    }
    if (a.edge_value)
      aggr_bwd_shift_kernel<true><<<grid, 256, smem, st>>>(a, grad_out, grad_input, grad_history, row_score, score_kind);
    else
      aggr_bwd_shift_kernel<false><<<grid, 256, smem, st>>>(a, grad_out, grad_input, grad_history, row_score, score_kind);
  } else {
    aggr_bwd_generic_kernel<<<grid, 256, 0, st>>>(a, grad_out, grad_input, grad_history, edge_grad,
                                                  row_score, score_kind, gi_stride);
  }
  HC_LAUNCH_OK();
  return 0;
}

extern "C" int hc_aggr_bwd(const hc_aggr_args* args, const float* grad_out, float* grad_input,
                           int32_t zero_grad_input, float* grad_history, float* edge_grad,
                           float* row_score, int32_t score_kind, void* stream) {
  return hc_aggr_bwd_rooted(args, grad_out, 0, nullptr, 0, grad_input, zero_grad_input, grad_history, edge_grad, row_score,
                            score_kind, stream);
}
