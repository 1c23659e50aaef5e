// A whole sampled batch in a FIXED shape, built without one device->host read.
//
// hc_sample_counts / hc_sample_picks / hc_relabel (sampler.cu) build a batch hop by hop, and the
// host reads two sizes back per hop to allocate the next arrays.  With the layer sizes fixed
// in advance (caps) nothing depends on those sizes on the host any more: every array has its
// capacity, the real counts stay on the device, rows behind them are padding (no neighbours,
// node 0, mask 0).  The whole batch is then a fixed sequence of launches, so it can run on a
// second stream behind the training step or be captured in the step's CUDA graph.
//
// Layout (the one NeighborSampler.sample_padded produces): layer k owns rows [0, caps[k]); the new
// nodes of hop h start at row caps[h-1]; ptr has caps[L-1] + 1 entries, idx edge_cap entries.
// Draws are the ones of hc_sample_picks: a function of (batch seed, frontier position, draw), the
// position counted over the REAL frontier nodes, so a batch that fits its caps is bit-identical to
// the host-driven one.  What does not fit is cut in a memory-safe way and counted: a new node beyond
// its layer's capacity is not added and the edges to it become self loops of their destination row;
// edges beyond edge_cap are dropped.
#include "grid_sync.cuh"

namespace hc {

constexpr int kAbsentF = (int)0x80000000;
constexpr int kMaxHops = 8;

// ---------------------------------------------------------------------------
// One kernel draws the whole batch.
//
// A hop is: draw and claim, count what is new, number it, translate the edges; each stage needs the
// stage before it from every block.  As separate launches (35 for three hops of some thousands of
// rows) a batch took 172 us, 166 of them the host's launches and 113 the GPU's, nearly all of it the
// start and end of tiny kernels.  Here the stages are separated by a barrier of all blocks of one
// cooperative launch, three per hop:
//   A  draw, claim (the lowest position of a node wins), sum up the draws per block        | barrier
//   B  count per block the positions that won their node                                   | barrier
//   C  number the new nodes, give them rows                                                | barrier
//   D  edges of the hop into idx, ptr entries
// Positions are row * fanout + draw, so their order needs no scan; a block owns the same rows through
// all stages and keeps their draw counts in shared memory and most draws in registers.  The others are
// kept in two buffers, because a fast block is already drawing hop h + 1 while a slow one still
// translates hop h.  A cluster of 16 blocks with the hardware's barrier took 61 us against 50: hashing
// and the memory latencies of a hop want more SMs.
// ---------------------------------------------------------------------------
constexpr int kSampleThreads = 512;
constexpr int kSampleKeep = 2;           // draws per thread that stay in registers
constexpr int kSampleBlocks = 96;        // leaves SMs to the kernels it runs beside; 64..148 blocks: 50..53 us

struct FixedPlan {
  int num_hops;
  int fanout[kMaxHops];
  int64_t caps[kMaxHops + 1];
  int64_t edge_cap;
  int64_t* ptr;
  int64_t* idx;
  int64_t* sub_to_full;
  uint8_t* mask;
  int64_t* counters;     // [0] real nodes [1] real edges [2] new nodes cut [3] edges cut
  // inputs
  const int64_t* gptr;
  const int64_t* gidx;
  const int64_t* seeds;
  int64_t n_seeds;
  int* local_map;
  uint64_t seed;
  int64_t* batch_no;
  const int64_t* labels;   // with y [caps[0]]: y = labels[seed], -100 in padding rows
  int64_t* y;
  // scratch
  unsigned* barrier;
  int* draws;              // [blocks] draws per block of the current hop
  int* firsts;             // [blocks] new nodes per block
  int64_t* nbr[2];         // [max rows * fanout] drawn neighbours, -1: none
  int* row_at;             // [blocks][rows_cap] when a block's rows do not fit its shared memory
};

__global__ void __launch_bounds__(kSampleThreads) sample_fixed_kernel(const FixedPlan p, const int rows_cap) {
  extern __shared__ int sh_rows[];
  // [rows_cap] draws of a row, then where its edges start in the hop
  int* row_at = p.row_at ? p.row_at + (int64_t)blockIdx.x * rows_cap : sh_rows;
  const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, threads = (int64_t)gridDim.x * blockDim.x;
  GridSync grid(p.barrier);
  const int64_t total = p.caps[p.num_hops];
  const uint64_t batch_seed = mix64(p.seed * 1000003ull + (uint64_t)p.batch_no[0]);
  for (int64_t i = gtid; i < total; i += threads) {
    const bool s = i < p.n_seeds;
    const int64_t v = s ? p.seeds[i] : 0;
    p.sub_to_full[i] = v;
    p.mask[i] = s ? 1 : 0;
    if (s) p.local_map[v] = (int)i;
    if (p.y && i < p.caps[0]) p.y[i] = s ? p.labels[v] : -100;
  }
  for (int64_t e = gtid; e < p.edge_cap; e += threads) p.idx[e] = 0;
  if (!grid.wait()) return;

  int64_t base = 0;                    // real frontier rows of the earlier hops
  int64_t frontier = p.n_seeds;        // real rows of this hop's frontier
  int64_t e_off = 0, nodes = p.n_seeds, cut_nodes = 0, cut_edges = 0;
  for (int h = 0; h < p.num_hops; ++h) {
    const int64_t fs = h == 0 ? 0 : p.caps[h - 1];
    const int64_t nf = p.caps[h] - fs;                // frontier capacity (rows [fs, caps[h]))
    const int64_t row0 = p.caps[h];                   // the new nodes' first row
    const int64_t cap_new = p.caps[h + 1] - p.caps[h];
    const int fan = p.fanout[h];
    if (nf == 0) continue;
    int64_t* nbr = p.nbr[h & 1];
    // rows of this block; real rows come first, so they are cut evenly
    const int64_t per = ceil_div(frontier, (int64_t)gridDim.x);
    const int64_t r0 = per * blockIdx.x < frontier ? per * blockIdx.x : frontier;
    const int rows = (int)(r0 + per < frontier ? per : frontier - r0);
    const int slots = rows * fan;
    // a thread keeps its first draws, and whether they won, in registers; the rest is read again
    int64_t kept_d[kSampleKeep];
    bool kept_won[kSampleKeep];
    auto won_at = [&](int t, int64_t d) { return d >= 0 && __ldcg(p.local_map + d) == -(int)(r0 * fan + t + 2); };
    // A
    int mine = 0;
    for (int i = threadIdx.x; i < rows; i += blockDim.x) {
      const int64_t v = __ldcg(p.sub_to_full + fs + r0 + i);
      const int64_t deg = p.gptr[v + 1] - p.gptr[v];
      const int c = (int)(deg < fan ? deg : fan);
      row_at[i] = c;
      mine += c;
    }
    auto pick = [&](int i, int j, int64_t first, int64_t deg) {
      const uint64_t u = mix64(batch_seed ^ mix64((uint64_t)(base + r0 + i) * (uint64_t)fan + (uint64_t)j));
      return first + (int64_t)(u % (uint64_t)deg);
    };
    {
      // the draws of a thread side by side: three latencies for all of them
      int64_t v[kSampleKeep], first[kSampleKeep], deg[kSampleKeep];
#pragma unroll
      for (int k = 0; k < kSampleKeep; ++k) {
        const int t = threadIdx.x + k * kSampleThreads;
        v[k] = t < slots ? __ldcg(p.sub_to_full + fs + r0 + t / fan) : -1;
      }
#pragma unroll
      for (int k = 0; k < kSampleKeep; ++k) {
        first[k] = v[k] >= 0 ? p.gptr[v[k]] : 0;
        deg[k] = v[k] >= 0 ? p.gptr[v[k] + 1] : 0;
      }
#pragma unroll
      for (int k = 0; k < kSampleKeep; ++k) {
        const int t = threadIdx.x + k * kSampleThreads, i = t / fan, j = t - i * fan;
        deg[k] -= first[k];
        kept_d[k] = j < deg[k] ? p.gidx[pick(i, j, first[k], deg[k])] : -1;
      }
#pragma unroll
      for (int k = 0; k < kSampleKeep; ++k)
        if (kept_d[k] >= 0) atomicMax(p.local_map + kept_d[k], -(int)(r0 * fan + threadIdx.x + k * kSampleThreads + 2));
      for (int t = threadIdx.x + kSampleKeep * kSampleThreads; t < slots; t += kSampleThreads) {
        const int i = t / fan, j = t - i * fan;
        const int64_t w = __ldcg(p.sub_to_full + fs + r0 + i);
        const int64_t b = p.gptr[w], n = p.gptr[w + 1] - b;
        int64_t d = -1;
        if (j < n) {
          d = p.gidx[pick(i, j, b, n)];
          atomicMax(p.local_map + d, -(int)(r0 * fan + t + 2));
        }
        nbr[r0 * fan + t] = d;
      }
    }
    int block_draws;
    block_exclusive<kSampleThreads>(mine, &block_draws);
    if (threadIdx.x == 0) p.draws[blockIdx.x] = block_draws;
    if (!grid.wait()) return;
    // B
    int won = 0;
    {
#pragma unroll
      for (int k = 0; k < kSampleKeep; ++k) {
        const int t = threadIdx.x + k * kSampleThreads;
        const int64_t d = kept_d[k];
        kept_won[k] = won_at(t, d);
        won += kept_won[k];
      }
      for (int t = threadIdx.x + kSampleKeep * kSampleThreads; t < slots; t += blockDim.x)
        won += won_at(t, nbr[r0 * fan + t]);
    }
    int block_new;
    block_exclusive<kSampleThreads>(won, &block_new);
    if (threadIdx.x == 0) p.firsts[blockIdx.x] = block_new;
    int hop_draws, first_edge;
    block_prefix(p.draws, gridDim.x, blockIdx.x, &hop_draws, &first_edge);
    // where each row's edges start
    for (int i0 = 0; i0 < rows; i0 += blockDim.x) {
      const int i = i0 + threadIdx.x;
      const int c = i < rows ? row_at[i] : 0;
      int n_here;
      const int at = first_edge + block_exclusive<kSampleThreads>(c, &n_here);
      if (i < rows) row_at[i] = at;
      first_edge += n_here;
    }
    if (!grid.wait()) return;
    // C
    int hop_new, first_new;
    block_prefix(p.firsts, gridDim.x, blockIdx.x, &hop_new, &first_new);
    {
      int n = 0;
      for (int t0 = 0; t0 < slots; t0 += blockDim.x, ++n) {
        const int t = t0 + threadIdx.x;
        int64_t d = -1;
        bool f = false;
        if (t < slots) {
#pragma unroll
          for (int k = 0; k < kSampleKeep; ++k)
            if (n == k) { d = kept_d[k]; f = kept_won[k]; }
          if (n >= kSampleKeep) { d = nbr[r0 * fan + t]; f = won_at(t, d); }
        }
        int n_here;
        const int64_t rank = first_new + block_exclusive<kSampleThreads>(f ? 1 : 0, &n_here);
        first_new += n_here;
        if (f && rank < cap_new) {       // those beyond the layer's capacity keep their claim: they are cut
          p.sub_to_full[row0 + rank] = d;
          p.mask[row0 + rank] = 1;
          p.local_map[d] = (int)(row0 + rank);
        }
      }
    }
    if (!grid.wait()) return;
    // D
    for (int i = threadIdx.x; i < rows; i += blockDim.x) {
      const int64_t at = e_off + row_at[i];
      p.ptr[fs + r0 + i] = at < p.edge_cap ? at : p.edge_cap;
    }
    for (int64_t i = frontier + gtid; i < nf; i += threads) {      // padding rows have no edges
      const int64_t at = e_off + hop_draws;
      p.ptr[fs + i] = at < p.edge_cap ? at : p.edge_cap;
    }
    auto put_edge = [&](int t, int loc) {
      const int i = t / fan, j = t - i * fan;
      const int64_t e = e_off + row_at[i] + j;
      // a node that was cut has no row: the edge becomes a self loop of its destination row
      if (e < p.edge_cap) p.idx[e] = loc >= 0 ? (int64_t)loc : fs + r0 + i;
    };
    {
      int loc[kSampleKeep];
#pragma unroll
      for (int k = 0; k < kSampleKeep; ++k) loc[k] = kept_d[k] >= 0 ? __ldcg(p.local_map + kept_d[k]) : 0;
#pragma unroll
      for (int k = 0; k < kSampleKeep; ++k)
        if (kept_d[k] >= 0) put_edge(threadIdx.x + k * kSampleThreads, loc[k]);
      for (int t = threadIdx.x + kSampleKeep * kSampleThreads; t < slots; t += kSampleThreads) {
        const int64_t d = nbr[r0 * fan + t];
        if (d >= 0) put_edge(t, __ldcg(p.local_map + d));
      }
    }
    if (hop_new > cap_new) {           // the claims of cut nodes are withdrawn once every block has read them
      if (!grid.wait()) return;
      int n = 0;
      for (int t = threadIdx.x; t < slots; t += blockDim.x, ++n) {
        int64_t d = -1;
#pragma unroll
        for (int k = 0; k < kSampleKeep; ++k)
          if (n == k) d = kept_d[k];
        if (n >= kSampleKeep) d = nbr[r0 * fan + t];
        if (d >= 0 && __ldcg(p.local_map + d) == -(int)(r0 * fan + t + 2)) p.local_map[d] = kAbsentF;
      }
      cut_nodes += hop_new - cap_new;
      if (!grid.wait()) return;
    }
    const int64_t kept = hop_new < cap_new ? hop_new : cap_new;
    base += frontier;
    frontier = kept;
    nodes += kept;
    const int64_t e_end = e_off + hop_draws;
    if (e_end > p.edge_cap) cut_edges += e_end - (e_off > p.edge_cap ? e_off : p.edge_cap);
    e_off = e_end;
    __syncthreads();                   // row_at is reused
  }
  if (!grid.wait()) return;
  for (int64_t i = gtid; i < total; i += threads)
    if (__ldcg(p.mask + i)) p.local_map[__ldcg(p.sub_to_full + i)] = kAbsentF;
  if (gtid == 0) {
    p.ptr[p.caps[p.num_hops - 1]] = e_off < p.edge_cap ? e_off : p.edge_cap;
    p.counters[0] = nodes;
    p.counters[1] = e_off < p.edge_cap ? e_off : p.edge_cap;
    p.counters[2] = cut_nodes;
    p.counters[3] = cut_edges;
    p.batch_no[0] += 1;
  }
}

}  // namespace hc

using namespace hc;

static int64_t max_frontier(const hc_fixed_batch* b) {
  int64_t m = b->caps[0];
  for (int h = 1; h < b->num_hops; ++h) {
    const int64_t f = b->caps[h] - b->caps[h - 1];
    if (f > m) m = f;
  }
  return m;
}
static int64_t max_draws(const hc_fixed_batch* b) {
  int64_t m = 0;
  for (int h = 0; h < b->num_hops; ++h) {
    const int64_t f = (h == 0 ? b->caps[0] : b->caps[h] - b->caps[h - 1]) * (int64_t)b->fanout[h];
    if (f > m) m = f;
  }
  return m;
}

// rows of a block, and whether they need memory behind the draws
static int sample_rows(const hc_fixed_batch* b) { return (int)ceil_div(max_frontier(b), kSampleBlocks); }
static constexpr int kSampleSharedRows = 8 * 1024;

extern "C" int64_t hc_sample_fixed_scratch_bytes(const hc_fixed_batch* b) {
  if (!b || b->num_hops < 1 || b->num_hops > kMaxHops) return 0;
  const int64_t rows = sample_rows(b);
  return 64 + 2 * kSampleBlocks * (int64_t)sizeof(int) + 2 * (max_draws(b) + 1) * (int64_t)sizeof(int64_t) +
         (rows > kSampleSharedRows ? rows * kSampleBlocks * (int64_t)sizeof(int) : 0);
}

extern "C" int hc_sample_batch(const int64_t* gptr, const int64_t* gidx, const int64_t* seeds, int64_t n_seeds,
                               int32_t* local_map, uint64_t seed, int64_t* batch_no, const int64_t* labels, int64_t* y,
                               const hc_fixed_batch* b, void* scratch, void* stream) {
  HC_REQUIRE(b != nullptr, HC_ERR_NULL);
  HC_REQUIRE(b->struct_size == sizeof(hc_fixed_batch), HC_ERR_STRUCT);
  HC_REQUIRE(b->num_hops >= 1 && b->num_hops <= kMaxHops, HC_ERR_SIZE);
  HC_REQUIRE(n_seeds >= 0 && n_seeds <= b->caps[0] && b->edge_cap >= 0, HC_ERR_SIZE);
  for (int h = 0; h < b->num_hops; ++h)
    HC_REQUIRE(b->fanout[h] >= 1 && b->caps[h + 1] >= b->caps[h] && b->caps[h] >= 0, HC_ERR_SIZE);
  HC_REQUIRE(b->caps[b->num_hops] < 0x7fffffffLL && max_draws(b) < 0x7ffffff0LL, HC_ERR_SIZE);
  HC_REQUIRE(gptr && gidx && local_map && batch_no && scratch && b->ptr && b->idx && b->sub_to_full && b->mask &&
                 b->counters && (seeds || n_seeds == 0) && (!y || labels),
             HC_ERR_NULL);
  HC_REQUIRE(aligned_to(scratch, 8), HC_ERR_ALIGN);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  FixedPlan p{};
  p.num_hops = b->num_hops;
  for (int h = 0; h < b->num_hops; ++h) p.fanout[h] = b->fanout[h];
  for (int h = 0; h <= b->num_hops; ++h) p.caps[h] = b->caps[h];
  p.edge_cap = b->edge_cap;
  p.ptr = b->ptr; p.idx = b->idx; p.sub_to_full = b->sub_to_full; p.mask = b->mask; p.counters = b->counters;
  p.gptr = gptr; p.gidx = gidx; p.seeds = seeds; p.n_seeds = n_seeds; p.local_map = local_map;
  p.seed = seed; p.batch_no = batch_no; p.labels = labels; p.y = y;
  char* w = reinterpret_cast<char*>(scratch);
  const int64_t draws = max_draws(b);
  p.barrier = reinterpret_cast<unsigned*>(w); w += 64;
  p.nbr[0] = reinterpret_cast<int64_t*>(w); w += (draws + 1) * sizeof(int64_t);
  p.nbr[1] = reinterpret_cast<int64_t*>(w); w += (draws + 1) * sizeof(int64_t);
  p.draws = reinterpret_cast<int*>(w); w += kSampleBlocks * sizeof(int);
  p.firsts = reinterpret_cast<int*>(w); w += kSampleBlocks * sizeof(int);
  const int rows = sample_rows(b);
  size_t smem = (size_t)rows * sizeof(int);
  if (rows > kSampleSharedRows) {
    p.row_at = reinterpret_cast<int*>(w);
    smem = 0;
  }
  return launch_together(sample_fixed_kernel, kSampleBlocks, kSampleThreads, smem, p.barrier, st, p, rows);
}

extern "C" int hc_sample_fixed(const int64_t* gptr, const int64_t* gidx, const int64_t* seeds, int64_t n_seeds,
                               int32_t* local_map, uint64_t seed, int64_t* batch_no,
                               const hc_fixed_batch* b, void* scratch, void* stream) {
  return hc_sample_batch(gptr, gidx, seeds, n_seeds, local_map, seed, batch_no, nullptr, nullptr, b, scratch, stream);
}
