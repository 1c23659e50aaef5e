// Aggregation backward by source (hc_aggr_bwd_source): every grad_input row is written once, as the
// weighted sum of the gradient rows of the destinations that read it, and the gradient of the edge
// weights is taken in the same pass.
//
// The scatter of hc_aggr_bwd moves a line DRAM -> L2 -> DRAM for every reduction once grad_input no
// longer fits the L2, needs a zero-fill first, and with edge weights gathers the source rows a second
// time (100 K rows, 1 M edges, 4 heads of 64: 621 us, of which the reductions and the gathers are
// 1 GB each).  Turned round, the source row is read once from where it lies, its gradient is written
// once, and what is gathered is grad_out, which is the smaller side of a sampled block and usually
// stays in the L2.
//
// The price is a transposition of the block.  hc_transpose_block sorts, so that sums have a fixed
// order; this one only counts: an atomic per edge gives the edge its rank among its source's edges,
// a scan gives the lists their places, and a second walk over the edges writes them there (2 M edges
// into 800 K sources: about 30 us against 150 us for the three radix passes).  List order, and with it
// the last bits of the sums, differ from call to call, as they do with the scatter; the reproducible
// mode keeps the sort.
#include <atomic>

#include "common.cuh"

namespace hc {

constexpr int kSrcLong = 64;       // entries of a list that one warp takes; longer lists are cut
constexpr int kSrcItem = 64;       // into items of this many entries, each added to the row atomically
constexpr int kSrcScan = 4096;     // sources per scan block
constexpr int kSrcRows = 31;       // most sources of a unit (one list start per lane)
constexpr int kSrcCounters = 1028; // words of counters in front of the scratch: 1 + at most 2^18 / 256 parts
constexpr int kSrcRowCost = 4;     // what a source costs beside its entries, in entries
constexpr int kSrcUnit = kSrcRows * kSrcRowCost;     // cost of a unit: at most kSrcRows sources

struct SourceLists {
  uint32_t* count;       // [4][n_src] entries per source, counted by row number mod 4; then where each of
                         // these quarters of the list starts
  uint32_t* rank;        // [n_edges] rank of an edge among its source's edges
  uint32_t* sums;        // [scan blocks]
  int64_t* t_ptr;        // [n_src + 1]
  uint32_t* t_dst;       // [n_edges] destination rows; with one weight per edge (destination, weight) pairs
  uint32_t* t_edge;      // [n_edges] edge numbers (only for the gradient of the weights)
  float* t_w;            // [n_edges(, H)] 1 / degree, or the edge's weights: in list order they are read
                         // next to each other
  unsigned int* n_units; // [1 + column parts] units, then per part the units handed out
  int2* units;           // [max_units] (first source, sources), or (source, -1 - chunk) of a long list
  int64_t max_units;
};

// Rank of every edge among its source's edges of rows with the same number mod 4: a popular source's
// atomics follow each other at the L2 (2 M skewed edges, 21 K of them to one source: 64 us with one
// counter per source), so they are spread over four,
// in different lines.  Edges without gradient (rows served from history,
// sources read from the alternative table) get no rank.
__global__ void __launch_bounds__(256)
    src_count_kernel(const hc_aggr_args a, const int64_t n_edges, const SourceLists l, float* __restrict__ edge_grad) {
  constexpr int G = 8;
  const int gl = threadIdx.x & (G - 1);
  const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
  if (r >= a.num_node) return;
  const bool row_counts = !(a.hmap && a.hmap[r] != -1);
  int64_t end = a.ptr[r + 1];
  if (end > n_edges) end = n_edges;
  for (int64_t e = a.ptr[r] + gl; e < end; e += G) {
    uint32_t k = 0xffffffffu;
    if (row_counts) {
      const int64_t s = a.idx[e];
      if (s >= 0 && s < a.n_src && !(a.src_map && a.src_map[s] != -1)) k = atomicAdd(l.count + (r & 3) * a.n_src + s, 1u);
    }
    l.rank[e] = k;
    if (edge_grad && k == 0xffffffffu)
      for (int h = 0; h < a.num_head; ++h) edge_grad[e * a.num_head + h] = 0.f;
  }
}

__device__ __forceinline__ uint4 source_counts(const SourceLists& l, int64_t s, int64_t n_src) {
  if (s >= n_src) return make_uint4(0u, 0u, 0u, 0u);
  const uint32_t* c = l.count + s;
  return make_uint4(c[0], c[n_src], c[2 * n_src], c[3 * n_src]);
}
__device__ __forceinline__ uint32_t sum4(const uint4& v) { return v.x + v.y + v.z + v.w; }

__global__ void __launch_bounds__(1024) src_sums_kernel(const int64_t n_src, const SourceLists l) {
  __shared__ uint32_t part[32];
  uint32_t x = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) x += sum4(source_counts(l, (int64_t)blockIdx.x * kSrcScan + k * 1024 + threadIdx.x, n_src));
  x = __reduce_add_sync(kFull, x);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x < 32) {
    x = __reduce_add_sync(kFull, part[threadIdx.x]);
    if (threadIdx.x == 0) l.sums[blockIdx.x] = x;
  }
}

// List starts, and the units of work of the gather: runs of consecutive short lists of about equal
// size, so that popular sources (which sit together in a degree-ordered graph) do not end up in a few
// warps, and the items of long lists.  Every block adds up the sums of the blocks in front of it.
__global__ void __launch_bounds__(1024) src_starts_kernel(const int64_t n_src, const SourceLists l) {
  __shared__ uint32_t part[32];
  __shared__ uint32_t front, base, n_ends;
  __shared__ uint16_t ends[kSrcScan];      // last source of every unit, block-local
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t before = 0;
  for (unsigned b = threadIdx.x; b < blockIdx.x; b += 1024) before += l.sums[b];
  before = __reduce_add_sync(kFull, before);
  if (lane == 0) part[warp] = before;
  __syncthreads();
  if (warp == 0) {
    before = __reduce_add_sync(kFull, part[lane]);
    if (lane == 0) front = before;
  }
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * kSrcScan + 4 * threadIdx.x;
  // counts come in coalesced, go through shared memory to the thread that owns four sources
  __shared__ uint32_t counts[kSrcScan + 1];
  uint4 quarter[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    quarter[k] = source_counts(l, (int64_t)blockIdx.x * kSrcScan + k * 1024 + threadIdx.x, n_src);
    counts[k * 1024 + threadIdx.x] = sum4(quarter[k]);
  }
  if (threadIdx.x == 0) counts[kSrcScan] = 0u;      // the first source of the next block ends a unit anyway
  __syncthreads();
  uint32_t c[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) c[k] = counts[4 * threadIdx.x + k];
  const uint32_t mine = c[0] + c[1] + c[2] + c[3];
  uint32_t x = mine;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, x, off);
    if (lane >= off) x += t;
  }
  if (lane == 31) part[warp] = x;
  __syncthreads();
  uint32_t at = front + x - mine;
  for (int w = 0; w < warp; ++w) at += part[w];
  __shared__ uint32_t starts[kSrcScan];
  unsigned is_end = 0;      // bit k: source i + k is the last of its unit
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (i + k < n_src) {
      starts[4 * threadIdx.x + k] = at;
      const uint32_t next = at + c[k];
      if (i + k == n_src - 1) l.t_ptr[n_src] = next;
      const bool is_long = c[k] > kSrcLong;
      if (is_long) {
        const unsigned chunks = (c[k] + kSrcItem - 1) / kSrcItem;
        const unsigned first = atomicAdd(l.n_units, chunks);
        for (unsigned q = 0; q < chunks && first + q < l.max_units; ++q)
          l.units[first + q] = make_int2((int)(i + k), -1 - (int)q);
      }
      const int64_t cost = at + (i + k) * kSrcRowCost;
      if (is_long || c[k + 1] > kSrcLong || cost / kSrcUnit != (cost + c[k] + kSrcRowCost) / kSrcUnit ||
          i + k == n_src - 1 || 4 * threadIdx.x + k == kSrcScan - 1)
        is_end |= 1u << k;
      at = next;
    }
  }
  // positions of the unit ends, in order
  uint32_t y = __popc(is_end);
  const uint32_t own = y;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, y, off);
    if (lane >= off) y += t;
  }
  __syncthreads();
  if (lane == 31) part[warp] = y;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t s = (int64_t)blockIdx.x * kSrcScan + k * 1024 + threadIdx.x;
    if (s < n_src) {
      uint32_t to = starts[k * 1024 + threadIdx.x];
      l.t_ptr[s] = to;
      uint32_t* c = l.count + s;
      c[0] = to;
      c[n_src] = to += quarter[k].x;
      c[2 * n_src] = to += quarter[k].y;
      c[3 * n_src] = to += quarter[k].z;
    }
  }
  __syncthreads();
  uint32_t pos = y - own;
  for (int w = 0; w < warp; ++w) pos += part[w];
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (is_end >> k & 1u) ends[pos++] = (uint16_t)(4 * threadIdx.x + k);
  if (threadIdx.x == 1023) {
    n_ends = pos;
    base = atomicAdd(l.n_units, pos);
  }
  __syncthreads();
  for (uint32_t u = threadIdx.x; u < n_ends; u += 1024) {
    const int first = u ? ends[u - 1] + 1 : 0, nr = ends[u] + 1 - first;
    const int64_t s = (int64_t)blockIdx.x * kSrcScan + first;
    // the unit of a long list is its items: here it is a run of no sources
    const bool is_long = nr == 1 && counts[first] > kSrcLong;
    if (base + u < l.max_units) l.units[base + u] = make_int2((int)s, is_long ? 0 : nr);
  }
}

// the lists; the rows of cut lists are cleared for the items that add to them
__global__ void __launch_bounds__(256)
    src_place_kernel(const hc_aggr_args a, const int64_t n_edges, const SourceLists l,
                     float* __restrict__ grad_input, const int width, const int heads) {
  constexpr int G = 8;
  const int gl = threadIdx.x & (G - 1);
  const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t r = gtid / G;
  if (r < a.num_node) {
    const int64_t b = a.ptr[r];
    int64_t end = a.ptr[r + 1];
    const float inv = __frcp_rn((float)(end - b));
    if (end > n_edges) end = n_edges;
    for (int64_t e = b + gl; e < end; e += G) {
      const uint32_t k = l.rank[e];
      if (k == 0xffffffffu) continue;
      const int64_t at = l.count[(r & 3) * a.n_src + a.idx[e]] + k;
      if (l.t_edge) l.t_edge[at] = (uint32_t)e;
      if (heads) {
        l.t_dst[at] = (uint32_t)r;
        for (int h = 0; h < a.num_head; ++h) l.t_w[at * a.num_head + h] = a.edge_value[e * a.num_head + h];
      } else {      // destination and weight side by side: one write
        reinterpret_cast<uint2*>(l.t_dst)[at] = make_uint2((uint32_t)r, __float_as_uint(a.edge_value ? a.edge_value[e] : inv));
      }
    }
  }
  if (grad_input) {
    unsigned n = *l.n_units;
    if (n > l.max_units) n = (unsigned)l.max_units;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t q = gtid >> 5; q < n; q += warps) {
      const int2 it = l.units[q];
      if (it.y != -1) continue;      // the first item of a long list
      for (int c = threadIdx.x & 31; c < width; c += kWarp) grad_input[(int64_t)it.x * width + c] = 0.f;
    }
  }
}

// ---------------------------------------------------------------------------
// the gather: the stream of aggr_fwd_stream_kernel over the lists
//   VB, G, V   unit of a lane, lanes per row, units per lane, as there (rows are fp32)
//   MODE       0 mean, 1 weighted, one head, 2 weighted per head
//   EG         also edge_grad[e(, h)] = <grad_out row of e's destination, source row>
// Units keep lists whole, so a list's sum is added up in registers and stored once; only the items of
// long lists are added atomically.  With EG a head's `seg` units lie on neighbouring lanes (lanes [0, lanes) of the warp are used, a
// multiple of seg), so that its dot product is a segmented warp sum.
// ---------------------------------------------------------------------------
struct SourceGather {
  const float* grad_out;   // [num_node, width]
  float* grad_input;       // [n_src, width] or NULL (EG only)
  const float* x;          // source rows (EG)
  int64_t x_stride;
  float* edge_grad;
  int64_t n_src;
  int width, heads, feat, nvec, part_vec, lanes, seg, stream_out;
};

template <int VB, int V, bool EG>
struct SourceShape {
  static constexpr int U = 2;
  static constexpr int kReq = V * VB * kWarp;
  static constexpr int kSlot = U * kReq;
  static constexpr int D = 6144 / kSlot < 3 ? 3 : (6144 / kSlot > 8 ? 8 : 6144 / kSlot);
  static constexpr int kWarpBytes = D * kSlot + 64 * 4;     // + ring of destination rows
  static constexpr int kSmem = 8 * kWarpBytes;
  static constexpr int kFit = 220 * 1024 / (kSmem + 1024);
  static constexpr int kMost = EG ? 3 : 4;
  static constexpr int kMinBlocks = kFit < kMost ? kFit : kMost;
};

// Sums over S = seg neighbouring lanes of N values per lane (N = 2 or 4, S a power of two >= N), N shuffles
// and log2(S / N) more instead of N log2(S): lane p of a segment, p < N, ends up with the sum of value p.
template <int N>
__device__ __forceinline__ float packed_sum(const float* d, int lane, int seg) {
  float t[N];
#pragma unroll
  for (int i = 0; i < N; ++i) t[i] = d[i];
#pragma unroll
  for (int n = N, bit = 1; n > 1; n >>= 1, bit <<= 1) {
    const bool hi = lane & bit;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const float keep = hi ? t[2 * i + 1] : t[2 * i], send = hi ? t[2 * i] : t[2 * i + 1];
      t[i] = keep + __shfl_xor_sync(kFull, send, bit);
    }
  }
  for (int o = N; o < seg; o <<= 1) t[0] += __shfl_xor_sync(kFull, t[0], o);
  return t[0];
}

template <int VB, int G, int V, bool HEADS, bool EG>
__global__ void __launch_bounds__(256, (SourceShape<VB, V, EG>::kMinBlocks))
    aggr_bwd_source_kernel(const SourceGather a, const SourceLists l) {
  using Vec = LaneVec<float, VB>;
  using Shape = SourceShape<VB, V, EG>;
  constexpr int EL = Vec::kElems;
  constexpr int EPW = kWarp / G;
  constexpr int D = Shape::D, U = Shape::U;
  static_assert(!EG || G == 32, "the edge gradients take whole warps");
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned char* mine = smem + (size_t)warp * Shape::kWarpBytes + lane * VB;
  const uint32_t mine_s = smem_u32(mine);
  uint32_t* ring = reinterpret_cast<uint32_t*>(smem + (size_t)warp * Shape::kWarpBytes + D * Shape::kSlot);
  const int H = HEADS ? a.heads : 1;
  const int lanes = EG ? a.lanes : G;
  const int v0 = blockIdx.y * a.part_vec;                     // this block's columns of the row
  const int v1 = v0 + a.part_vec < a.nvec ? v0 + a.part_vec : a.nvec;
  const int sub = lane / G, gl = lane % G;
  const char* __restrict__ in = reinterpret_cast<const char*>(a.grad_out);
  const int64_t row_bytes = (int64_t)a.width * 4;
  const uint64_t policy = l2_policy(a.stream_out != 0);
  int vk[V], head[V];                                         // this lane's units; < 0: none
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const int v = v0 + gl + k * lanes;
    vk[k] = (!EG || lane < lanes) && v < v1 ? v : -1;
    head[k] = HEADS && vk[k] >= 0 ? v * EL / a.feat : 0;
  }

  // Units are handed out by a counter: the number of rounds is small and their lengths differ.  What a
  // unit needs is fetched ahead: its number two units before, its place one before that it starts.
  unsigned n_units = *l.n_units;
  if (n_units > l.max_units) n_units = (unsigned)l.max_units;
  const unsigned warps = gridDim.x * 8;
  unsigned q = blockIdx.x * 8 + warp, q_next = 0;
  auto take = [&]() {
    unsigned t = 0;
    if (lane == 0) t = atomicAdd(l.n_units + 1 + blockIdx.y, 1u) + warps;
    return t;       // lane 0's value counts
  };
  int2 unit = make_int2(0, 0);
  int my_p = 0;                                               // lane l: first entry of source l of the next unit
  auto fetch_ptr = [&]() {
    my_p = 0;
    if (unit.y < 0) {
      const int b = (int)l.t_ptr[unit.x] + (-1 - unit.y) * kSrcItem, end = (int)l.t_ptr[unit.x + 1];
      my_p = lane == 0 ? b : (b + kSrcItem < end ? b + kSrcItem : end);
    } else if (lane <= unit.y) {
      my_p = (int)l.t_ptr[unit.x + lane];
    }
  };
  if (q >= n_units) return;
  unit = l.units[q];
  fetch_ptr();
  q_next = take();
  q_next = __shfl_sync(kFull, q_next, 0);
  int2 unit_2 = q_next < n_units ? l.units[q_next] : make_int2(0, 0);
  unsigned q_2 = take();
  while (q < n_units) {
    const bool item = unit.y < 0;
    const int64_t s0 = unit.x;
    const int nr = item ? 1 : unit.y;
    const int off = my_p;
    const int next_off = __shfl_down_sync(kFull, off, 1);
    const int first = __shfl_sync(kFull, off, 0), last = __shfl_sync(kFull, off, nr);
    int loaded = first;
    uint32_t next_i = loaded + lane < last ? l.t_dst[(HEADS ? 1 : 2) * (int64_t)(loaded + lane)] : 0u;   // chunk [loaded, loaded + 32)
    q = q_next;
    unit = unit_2;
    fetch_ptr();                                                            // in flight during this unit
    q_next = __shfl_sync(kFull, q_2, 0);
    unit_2 = q_next < n_units ? l.units[q_next] : make_int2(0, 0);
    q_2 = take();
    if (nr == 0) continue;
    // producer: the unit's lists are one slice of entries; requests of a single row (G == 32) follow
    // each other across list ends, those of several rows (G < 32) stay within a list
    int pe = first, prow = 0;
    int pend = EPW == 1 ? last : __shfl_sync(kFull, next_off, 0);
    auto produce = [&](int slot) {
      if (EPW > 1) {
        while (pe >= pend && prow + 1 < nr) {
          pe = pend;
          pend = __shfl_sync(kFull, next_off, ++prow);
        }
      }
      if (pe < pend) {
        const int need = pe + U * EPW < pend ? pe + U * EPW : pend;
        if (need > loaded) {
          __syncwarp();
          ring[(loaded + lane) & 63] = next_i;
          __syncwarp();
          loaded += kWarp;
          next_i = loaded + lane < last ? l.t_dst[(HEADS ? 1 : 2) * (int64_t)(loaded + lane)] : 0u;
        }
        const uint32_t dst = mine_s + slot * Shape::kSlot;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int e = pe + u * EPW + sub;
          if (e < pend) {
            const char* p = in + (int64_t)ring[e & 63] * row_bytes;
#pragma unroll
            for (int k = 0; k < V; ++k)
              if (vk[k] >= 0) cp_async<VB>(dst + u * Shape::kReq + k * VB * kWarp, p + vk[k] * VB);
          }
        }
        pe += U * EPW;
      }
      cp_async_commit();
    };
#pragma unroll 1
    for (int d = 0; d < D; ++d) produce(d);
    int slot = 0, row = 0, end = __shfl_sync(kFull, next_off, 0);
    float acc[V][EL], xs[EG ? V : 1][EL];
    Vec xn[EG ? V : 1];      // the next source's own row
    auto fetch_x = [&](int r) {
#pragma unroll
      for (int k = 0; k < V; ++k) {
        xn[k].clear();
        if constexpr (EG)
          if (r < nr && vk[k] >= 0) xn[k].load_once(a.x + (s0 + r) * a.x_stride + vk[k] * EL, policy);
      }
    };
    auto begin_row = [&](int r) {
#pragma unroll
      for (int k = 0; k < V; ++k)
#pragma unroll
        for (int i = 0; i < EL; ++i) acc[k][i] = 0.f;
      if constexpr (EG) {
#pragma unroll
        for (int k = 0; k < V; ++k) xn[k].unpack(xs[k]);
        fetch_x(r + 1);
      }
    };
    auto end_row = [&]() {
      if (EPW > 1) {
#pragma unroll
        for (int o = G; o < kWarp; o <<= 1)
#pragma unroll
          for (int k = 0; k < V; ++k)
#pragma unroll
            for (int i = 0; i < EL; ++i) acc[k][i] += __shfl_xor_sync(kFull, acc[k][i], o);
      }
      if (sub == 0 && (!EG || a.grad_input)) {
        float* orow = a.grad_input + (s0 + row) * a.width;
#pragma unroll
        for (int k = 0; k < V; ++k) {
          if (vk[k] >= 0) {
            if (item) red_add<EL>(orow + vk[k] * EL, acc[k]);
            else store_f32<EL>(orow + vk[k] * EL, acc[k], policy);
          }
        }
      }
      ++row;
    };
    if constexpr (EG) fetch_x(0);
    begin_row(0);
    // weights (and edge numbers) of the next slot, one slot ahead: a slot is a new sector of them
    float w_next[U][HEADS ? V : 1];
    uint32_t edge_next[EG ? U : 1];
    auto load_weights = [&](int from) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int ee = from + u * EPW + sub;
#pragma unroll
        for (int k = 0; k < (HEADS ? V : 1); ++k)
          w_next[u][k] = ee < last ? __ldg(l.t_w + (HEADS ? (int64_t)ee * H + head[k] : 2 * (int64_t)ee)) : 0.f;
        if (EG) edge_next[u] = ee < last ? __ldg(l.t_edge + ee) : 0u;
      }
    };
    load_weights(first);
    // one pass over the slots; with G == 32 a slot may hold the end of one list and the start of the next
    int e = first;
    while (true) {
      const int stop = EPW == 1 ? last : end;
      if (e >= stop) {
        end_row();
        if (row >= nr) break;
        end = __shfl_sync(kFull, next_off, row);
        begin_row(row);
        continue;
      }
      float w[U][HEADS ? V : 1];
      uint32_t edge[EG ? U : 1];
#pragma unroll
      for (int u = 0; u < U; ++u) {
#pragma unroll
        for (int k = 0; k < (HEADS ? V : 1); ++k) w[u][k] = w_next[u][k];
        if (EG) edge[u] = edge_next[u];
      }
      load_weights(EPW == 1 ? e + U : (e + U * EPW < end ? e + U * EPW : end));
      cp_async_wait<D - 1>();
      float dot[EG ? U * V : 1];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (EG) {
#pragma unroll
          for (int k = 0; k < V; ++k) dot[u * V + k] = 0.f;
        }
        if (e + u * EPW + sub < stop) {
          if (EPW == 1) {
            while (e + u == end) {
              end_row();
              end = __shfl_sync(kFull, next_off, row);
              begin_row(row);
            }
          }
          const unsigned char* src = mine + slot * Shape::kSlot + u * Shape::kReq;
#pragma unroll
          for (int k = 0; k < V; ++k) {
            if (vk[k] >= 0) {
              Vec x;
              x.load_shared(src + k * VB * kWarp);
              float f[EL];
              x.unpack(f);
#pragma unroll
              for (int i = 0; i < EL; ++i) {
                acc[k][i] = fmaf(w[u][HEADS ? k : 0], f[i], acc[k][i]);
                if (EG) dot[u * V + k] = fmaf(f[i], xs[k][i], dot[u * V + k]);
              }
            }
          }
        }
      }
      if constexpr (EG) {
        if constexpr (!HEADS) {
          float d[2];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            d[u] = dot[u * V];
#pragma unroll
            for (int k = 1; k < V; ++k) d[u] += dot[u * V + k];
          }
          const float t = packed_sum<2>(d, lane, 32);
          if (lane < 2 && e + lane < stop) a.edge_grad[lane ? edge[U - 1] : edge[0]] = t;
        } else if ((a.seg & (a.seg - 1)) == 0 && a.seg >= U * V) {
          const int pos = lane & (a.seg - 1);
          const float t = packed_sum<U * V>(dot, lane, a.seg);
          if (pos < U * V) {
            const int u = pos / V, k = pos % V;
            const int h = k ? head[V - 1] : head[0];
            if (e + u < stop && (k ? vk[V - 1] : vk[0]) >= 0) a.edge_grad[(int64_t)(u ? edge[U - 1] : edge[0]) * H + h] = t;
          }
        } else {
          const int pos = lane % a.seg;
#pragma unroll
          for (int u = 0; u < U; ++u)
#pragma unroll
            for (int k = 0; k < V; ++k) {
              float t = dot[u * V + k];
#pragma unroll
              for (int o = 16; o > 0; o >>= 1) {
                const float other = __shfl_down_sync(kFull, t, o);
                if (pos + o < a.seg) t += other;
              }
              if (pos == 0 && vk[k] >= 0 && e + u < stop) a.edge_grad[(int64_t)edge[u] * H + head[k]] = t;
            }
        }
      }
      produce(slot);
      slot = slot + 1 == D ? 0 : slot + 1;
      e += U * EPW;
      if (EPW > 1 && e > end) e = end;
    }
    cp_async_wait<0>();
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
struct SourcePlan {
  int vb, nvec, heads, seg, lanes;
  bool per_head;
};

// which form of the gather a block takes; false: none (odd widths with weights per head or with the
// gradient of the weights, fp16 rows with the latter)
static bool source_plan(const hc_aggr_args* a, bool want_edge_grad, SourcePlan* p) {
  const int64_t width = (int64_t)a->num_head * a->feat;
  p->per_head = a->edge_value != nullptr && a->num_head > 1;
  p->vb = width % 4 == 0 ? 16 : (width % 2 == 0 ? 8 : 4);
  p->heads = a->num_head;
  p->nvec = (int)(width * 4 / p->vb);
  p->lanes = 32;
  p->seg = 0;
  if (p->per_head && a->feat % 4 != 0) return false;
  if (!want_edge_grad) return true;
  const int64_t xs = a->in_stride ? a->in_stride : width;
  if (!a->edge_value || a->in_dtype != HC_F32 || a->src_map || a->feat % 4 != 0 || xs % 4 != 0 || !aligned16(a->input))
    return false;
  if (!p->per_head) return p->nvec <= 128;
  p->seg = a->feat / 4;
  if (p->seg > 32) return false;
  p->lanes = 32 / p->seg * p->seg;
  return true;
}

static int64_t up16(int64_t v) { return (v + 15) / 16 * 16; }
static int64_t source_units(int64_t n_src, int64_t n_edges) {
  // ends by cost and around long lists, one per scan block; items of long lists
  return n_src / kSrcRows + n_edges / kSrcUnit + 2 * (n_edges / kSrcLong) + ceil_div(n_src, kSrcScan) +
         n_edges / (kSrcItem / 2) + 16;
}

static int64_t source_scratch(int64_t n_src, int64_t n_edges, int heads, bool per_head, bool want_edge_grad, char* base,
                              SourceLists* l) {
  int64_t at = 0;
  auto take = [&](int64_t bytes) {
    char* p = base + at;
    at += up16(bytes);
    return p;
  };
  // counters first: one clear covers them
  l->n_units = reinterpret_cast<unsigned int*>(take(kSrcCounters * 4));
  l->count = reinterpret_cast<uint32_t*>(take(16 * n_src));
  l->sums = reinterpret_cast<uint32_t*>(take(4 * ceil_div(n_src, kSrcScan)));
  l->rank = reinterpret_cast<uint32_t*>(take(4 * n_edges));
  l->t_ptr = reinterpret_cast<int64_t*>(take(8 * (n_src + 1)));
  l->t_dst = reinterpret_cast<uint32_t*>(take(per_head ? 4 * n_edges : 8 * n_edges));
  l->t_edge = want_edge_grad ? reinterpret_cast<uint32_t*>(take(4 * n_edges)) : nullptr;
  l->t_w = per_head ? reinterpret_cast<float*>(take(4 * n_edges * heads)) : reinterpret_cast<float*>(l->t_dst) + 1;
  l->max_units = source_units(n_src, n_edges);
  l->units = reinterpret_cast<int2*>(take(8 * l->max_units));
  return at;
}

template <int VB, int G, int V, bool HEADS, bool EG>
static int launch_source(SourceGather g, const SourceLists& l, cudaStream_t st) {
  using Shape = SourceShape<VB, V, EG>;
  auto kernel = aggr_bwd_source_kernel<VB, G, V, HEADS, EG>;
  static std::atomic<uint64_t> raised{0};
  if (Shape::kSmem > 48 * 1024) raise_smem(kernel, Shape::kSmem, raised);
  const int lanes = EG ? g.lanes : G, most_vec = lanes * V;
  const int parts = (int)ceil_div(g.nvec, most_vec);
  const int unit = EG && HEADS ? g.seg : 1;                      // a head stays in one part
  g.part_vec = (int)(ceil_div(ceil_div(g.nvec, parts), unit) * unit);
  dim3 grid(1, (unsigned)ceil_div(g.nvec, g.part_vec));
  int64_t most = 148 * Shape::kMinBlocks / grid.y;
  if (most < 1) most = 1;
  const int64_t blocks = ceil_div(ceil_div(g.n_src, 4), 8);
  grid.x = (unsigned)(blocks < most ? blocks : most);
  kernel<<<grid, 256, Shape::kSmem, st>>>(g, l);
  return 0;
}

static int launch_source_any(const SourcePlan& p, const SourceGather& g, const SourceLists& l, cudaStream_t st) {
  const int n = p.nvec;
  if (g.edge_grad) {
    if (p.per_head) {
      if (n <= p.lanes) return launch_source<16, 32, 1, true, true>(g, l, st);
      return launch_source<16, 32, 2, true, true>(g, l, st);
    }
    if (n <= 32) return launch_source<16, 32, 1, false, true>(g, l, st);
    if (n <= 64) return launch_source<16, 32, 2, false, true>(g, l, st);
    return launch_source<16, 32, 4, false, true>(g, l, st);
  }
  if (p.per_head) {
    if (n <= 16) return launch_source<16, 16, 1, true, false>(g, l, st);
    if (n <= 32) return launch_source<16, 32, 1, true, false>(g, l, st);
    return launch_source<16, 32, 2, true, false>(g, l, st);
  }
  if (p.vb == 16) {
    if (n <= 8) return launch_source<16, 8, 1, false, false>(g, l, st);
    if (n <= 16) return launch_source<16, 16, 1, false, false>(g, l, st);
    if (n <= 32) return launch_source<16, 32, 1, false, false>(g, l, st);
    return launch_source<16, 32, 2, false, false>(g, l, st);
  }
  if (p.vb == 8) {
    if (n <= 32) return launch_source<8, 32, 1, false, false>(g, l, st);
    if (n <= 64) return launch_source<8, 32, 2, false, false>(g, l, st);
    if (n <= 96) return launch_source<8, 32, 3, false, false>(g, l, st);
    return launch_source<8, 32, 4, false, false>(g, l, st);
  }
  if (n <= 32) return launch_source<4, 32, 1, false, false>(g, l, st);
  if (n <= 64) return launch_source<4, 32, 2, false, false>(g, l, st);
  if (n <= 96) return launch_source<4, 32, 3, false, false>(g, l, st);
  return launch_source<4, 32, 4, false, false>(g, l, st);
}

}  // namespace hc

using namespace hc;

extern "C" int64_t hc_aggr_bwd_source_scratch_bytes(const hc_aggr_args* a, int64_t n_edges, int32_t want_edge_grad) {
  if (!a || a->struct_size != sizeof(hc_aggr_args) || a->num_node < 1 || a->n_src < 1 || a->feat < 1 ||
      a->num_head < 1 || n_edges < 1)
    return -1;
  if (n_edges >= 0x7fffffffLL || a->n_src >= 0x7fffffffLL || a->num_node >= 0x7fffffffLL) return -1;
  if ((int64_t)a->num_head * a->feat > (1 << 18)) return -1;
  SourcePlan p;
  if (!source_plan(a, want_edge_grad != 0, &p)) return -1;
  SourceLists l;
  return source_scratch(a->n_src, n_edges, p.heads, p.per_head, want_edge_grad != 0, nullptr, &l);
}

extern "C" int hc_aggr_bwd_source(const hc_aggr_args* a, int64_t n_edges, const float* grad_out, float* grad_input,
                                  float* edge_grad, void* scratch, void* stream) {
  HC_REQUIRE(a != nullptr, HC_ERR_NULL);
  HC_REQUIRE(a->struct_size == sizeof(hc_aggr_args), HC_ERR_STRUCT);
  HC_REQUIRE(hc_aggr_bwd_source_scratch_bytes(a, n_edges, edge_grad != nullptr) >= 0, HC_ERR_UNSUPPORTED);
  HC_REQUIRE(a->ptr && a->idx && grad_out && (grad_input || edge_grad) && scratch, HC_ERR_NULL);
  HC_REQUIRE(aligned16(scratch) && aligned16(grad_out) && (!grad_input || aligned16(grad_input)), HC_ERR_ALIGN);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  SourcePlan p;
  source_plan(a, edge_grad != nullptr, &p);
  SourceLists l;
  source_scratch(a->n_src, n_edges, p.heads, p.per_head, edge_grad != nullptr, reinterpret_cast<char*>(scratch), &l);
  const int width = a->num_head * a->feat;
  const int64_t rows8 = ceil_div(a->num_node * 8, 256), tiles = ceil_div(a->n_src, kSrcScan);
  HC_REQUIRE(rows8 <= 0x7fffffffLL, HC_ERR_SIZE);
  HC_CUDA(cudaMemsetAsync(l.n_units, 0, kSrcCounters * 4 + 16 * a->n_src, st));
  src_count_kernel<<<(unsigned)rows8, 256, 0, st>>>(*a, n_edges, l, edge_grad);
  src_sums_kernel<<<(unsigned)tiles, 1024, 0, st>>>(a->n_src, l);
  src_starts_kernel<<<(unsigned)tiles, 1024, 0, st>>>(a->n_src, l);
  src_place_kernel<<<(unsigned)rows8, 256, 0, st>>>(*a, n_edges, l, grad_input, width, p.per_head);
  SourceGather g{};
  g.grad_out = grad_out;
  g.grad_input = grad_input;
  g.x = reinterpret_cast<const float*>(a->input);
  g.x_stride = a->in_stride ? a->in_stride : width;
  g.edge_grad = edge_grad;
  g.n_src = a->n_src;
  g.width = width;
  g.heads = a->num_head;
  g.feat = a->feat;
  g.nvec = p.nvec;
  g.lanes = p.lanes;
  g.seg = p.seg;
  // a gradient of more than half the L2 would push out the rows that are gathered
  g.stream_out = a->n_src * (int64_t)width * 4 > (64 << 20);
  launch_source_any(p, g, l, st);
  HC_LAUNCH_OK();
  return 0;
}
