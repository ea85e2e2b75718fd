// Candidate filter and compaction.
//
// Same predicate as the reference's LDfilterSSM_kernel
// (in-core/lib/filter/src/filter_kernel.cu:122-283) and the CPU filterSSM
// (out-of-core/lib/filter/src/filter.cu:160-240): label equality, query degree
// <= data degree + T, and a neighbour-label-count deficit <= T over the labels
// that occur in the query.  The degree test follows from the deficit (a
// query vertex's needs sum to its degree, so a deficit <= T leaves at least
// degree - T neighbours) and is not made apart.  Each (row, 32 data vertices)
// result is one word; the compaction turns the words into sorted candidate
// lists and rank words, so that the same row answers "is v in C(u)" and
// "where is v in C(u)" with one 8-byte load.
#include "device_common.cuh"
#include "kernels.h"

namespace gem {

// One warp per (set of TS tiles of 32 vertices, group of up to 32 rows of one
// label): a lane per row (and per tile, several side by side for a group of
// few rows).  Only a tile's vertices of that label, a few of the
// 32, can be the rows' candidates: one ballot finds them, and the lanes test
// their rows' needs (label, count) on those vertices alone, all on the same
// one, so that a ballot of the answers is the vertex's membership column.
// The rows' words are turned in shared memory so that a row's TS words leave
// in one coalesced store.
//
// What bounds it is instruction issue, then the words written.  A lane per
// vertex instead, every row tested on all 32 of them against a descriptor of
// up to 32 labels (the counts copied to local memory), took 6 ms for the
// 2,880 query vertices of 180 mixed-size queries on 1,048,576 vertices with
// 32 labels, and transposing the columns out of the rows' words 2.2 ms; the
// whole filter phase, host and compaction included, is 2.4 ms now (8.1).
template <uint32_t TS>
__global__ void __launch_bounds__(256) filter_kernel(const uint32_t *__restrict__ lab, uint32_t nv,
                                                     const uint8_t *__restrict__ nlc, uint32_t stride,
                                                     const FilterRow *__restrict__ rows,
                                                     const uint32_t *__restrict__ more,
                                                     const FilterGroup *__restrict__ groups, uint32_t ngroups,
                                                     uint32_t T, uint32_t nwords,
                                                     uint32_t *__restrict__ bits, uint32_t *__restrict__ cnt,
                                                     uint32_t *__restrict__ cols, uint32_t W) {
  __shared__ uint32_t turn[8][32][TS + 1];
  const uint32_t lane = dev::lane_id(), warp = threadIdx.x >> 5;
  const uint32_t nsets = (nwords + TS - 1) / TS;
  const uint64_t items = (uint64_t)ngroups * nsets;
  for (uint64_t it = blockIdx.x * 8ull + warp; it < items; it += gridDim.x * 8ull) {
    const uint32_t set = (uint32_t)(it / ngroups);
    const FilterGroup g = groups[it % ngroups];
    // lanes per tile: the group's rows rounded up to a power of two (no more
    // tiles side by side than a set has)
    uint32_t lg = g.n > 1 ? 32 - __clz(g.n - 1) : 0;
    if (32u >> lg > TS) lg = 31 - __clz(32u / TS);
    const uint32_t R = 1u << lg, rl = lane & (R - 1), sub = lane >> lg, nsub = 32u >> lg;
    const uint32_t mine = R == 32 ? dev::FULL : (1u << R) - 1u;
    const bool have = rl < g.n;
    FilterRow row = {};
    if (have) row = rows[g.row0 + rl];
    const bool live = have && row.need <= T;
    uint32_t n = 0;
    for (uint32_t t0 = 0; t0 < TS; t0 += nsub) {
      uint32_t m = 0;
      const uint64_t v0 = ((uint64_t)set * TS + t0) * 32 + lane;
      for (uint32_t j = 0; nsub < 8 && j < nsub; ++j) {
        const uint32_t b = __ballot_sync(dev::FULL, v0 + j * 32 < nv && __ldg(lab + v0 + j * 32) == g.lab);
        if (sub == j) m = b;
      }
      for (uint32_t j0 = 0; nsub >= 8 && j0 < nsub; j0 += 8) {  // eight tiles' labels in flight (nsub: a power of two)
        uint32_t l[8];
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) l[j] = v0 + (j0 + j) * 32 < nv ? __ldg(lab + v0 + (j0 + j) * 32) : 0u;
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
          const uint32_t b = __ballot_sync(dev::FULL, v0 + (j0 + j) * 32 < nv && l[j] == g.lab);
          if (sub == j0 + j) m = b;
        }
      }
      const uint64_t vb = ((uint64_t)set * TS + t0 + sub) * 32;
      uint32_t word = 0;
      while (__ballot_sync(dev::FULL, m != 0)) {  // two vertices a step: their loads overlap
        const bool a0 = m != 0;
        const uint32_t b0 = a0 ? __ffs(m) - 1 : 0u;
        m &= m - 1;  // 0 stays 0
        const bool a1 = m != 0;
        const uint32_t b1 = a1 ? __ffs(m) - 1 : b0;
        m &= m - 1;
        uint32_t d0 = row.need, d1 = row.need;
        if (live && a0) {
          const uint8_t *r0 = nlc + (vb + b0) * stride, *r1 = nlc + (vb + b1) * stride;
#pragma unroll
          for (uint32_t i = 0; i < FILTER_NEEDS; ++i) {
            const uint32_t k = row.needs[i] >> 8, q = row.needs[i] & 0xFFu;  // unused entries need 0
            const uint32_t c0 = q ? __ldg(r0 + k) : 0u, c1 = q ? __ldg(r1 + k) : 0u;
            d0 += q > c0 ? q - c0 : 0u;
            d1 += q > c1 ? q - c1 : 0u;
          }
          for (uint32_t i = 0; i < row.n_more; ++i) {
            const uint32_t e = __ldg(more + row.more + i), k = e >> 8, q = e & 0xFFu;
            const uint32_t c0 = __ldg(r0 + k), c1 = __ldg(r1 + k);
            d0 += q > c0 ? q - c0 : 0u;
            d1 += q > c1 ? q - c1 : 0u;
          }
        }
        const bool in0 = live && a0 && d0 <= T, in1 = live && a1 && d1 <= T;
        word |= (in0 ? 1u << b0 : 0u) | (in1 ? 1u << b1 : 0u);
        const uint32_t c0 = __ballot_sync(dev::FULL, in0), c1 = __ballot_sync(dev::FULL, in1);
        if (cols && rl == 0) {
          if (a0) cols[(vb + b0) * W + g.word] = ((c0 >> lane) & mine) << g.shift;
          if (a1) cols[(vb + b1) * W + g.word] = ((c1 >> lane) & mine) << g.shift;
        }
      }
      n += __popc(word);
      turn[warp][rl][t0 + sub] = word;
    }
    for (uint32_t o = R; o < 32; o <<= 1) n += __shfl_xor_sync(dev::FULL, n, o);
    if (have && sub == 0) cnt[(uint64_t)row.row * nsets + set] = n;
    __syncwarp();
    constexpr uint32_t RP = 32 / TS;  // rows per store
    for (uint32_t r0 = 0; r0 < g.n; r0 += RP) {
      const uint32_t r = r0 + lane / TS, w = set * TS + lane % TS;
      const uint32_t rr = __shfl_sync(dev::FULL, row.row, r & 31u);
      if (r < g.n && w < nwords) bits[(uint64_t)rr * nwords + w] = turn[warp][r][lane % TS];
    }
    __syncwarp();  // the words are read before the next item's are written
  }
}

// Adds one to the count of label l if it is one of want[0, n) (sorted).
__device__ __forceinline__ void count_label(uint32_t l, const FilterLabel *want, uint32_t n, uint32_t *found) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (want[mid].lab < l) lo = mid + 1; else hi = mid;
  }
  if (lo < n && want[lo].lab == l) atomicAdd(found + lo, 1u);
}

// Counts the rest [a0, a1) of a list, 128 arcs a step, until found[i] is at
// least want[i].most for every label or the list ends.
__device__ __forceinline__ void count_rest(const DevGraph &G, uint64_t a0, uint64_t a1, const FilterLabel *want,
                                           uint32_t n, uint32_t *found) {
  const uint32_t lane = dev::lane_id();
  for (uint64_t b = a0; b < a1; b += 128) {
    bool open = false;
    for (uint32_t i = lane; i < n; i += 32) open |= found[i] < want[i].most;
    if (!__any_sync(dev::FULL, open)) break;
    uint32_t x[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) x[k] = b + 32 * k + lane < a1 ? __ldg(G.nbr + b + 32 * k + lane) : 0u;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) x[k] = b + 32 * k + lane < a1 ? __ldg(G.lab + x[k]) : 0u;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k)
      if (b + 32 * k + lane < a1) count_label(x[k], want, n, found);
    __syncwarp();
  }
}

// One tile on graphs of too many labels for resident counts: v0 its first
// vertex, m its vertices of the group's label, row the lane's.  The warp counts
// the group's labels among a vertex's neighbours itself, all lanes on its list,
// until every label has reached the most that a row wants (a hub's first few
// hundred arcs) or the list ends; vertices with too few neighbours are not
// read.  Returns the lane's row's word; the vertices' columns go to cols.
constexpr uint32_t FV = 2;  // vertices a step: their loads overlap
__device__ __forceinline__ uint32_t count_tile(const DevGraph &G, uint64_t v0, uint32_t m, const FilterGroup &g,
                                               const FilterRow &row, bool live, const uint32_t *__restrict__ more,
                                               const FilterLabel *want, uint32_t (*found)[FILTER_LABELS], uint32_t T,
                                               uint32_t *__restrict__ cols, uint32_t W) {
  const uint32_t lane = dev::lane_id();
  uint32_t word = 0;
  while (m) {
    uint32_t b[FV], x[FV];
    uint64_t a0[FV], a1[FV];
#pragma unroll
    for (uint32_t k = 0; k < FV; ++k) {
      b[k] = m ? __ffs(m) - 1 : 32u;
      m &= m - 1;  // 0 stays 0
      a0[k] = b[k] < 32 ? __ldg(G.off + v0 + b[k]) : 0ull;
      a1[k] = b[k] < 32 ? __ldg(G.off + v0 + b[k] + 1) : 0ull;
    }
    __syncwarp();  // the previous step's counts are read
    for (uint32_t i = lane; i < FILTER_LABELS; i += 32)
#pragma unroll
      for (uint32_t k = 0; k < FV; ++k) found[k][i] = 0;
    __syncwarp();
#pragma unroll
    for (uint32_t k = 0; k < FV; ++k) {
      if (a1[k] - a0[k] + T < g.min_deg) a1[k] = a0[k];  // too few neighbours: a row's needs add up to its degree
      x[k] = a0[k] + lane < a1[k] ? __ldg(G.nbr + a0[k] + lane) : 0u;
    }
#pragma unroll
    for (uint32_t k = 0; k < FV; ++k) x[k] = a0[k] + lane < a1[k] ? __ldg(G.lab + x[k]) : 0u;
#pragma unroll
    for (uint32_t k = 0; k < FV; ++k)
      if (a0[k] + lane < a1[k]) count_label(x[k], want, g.nlab, found[k]);
    __syncwarp();
#pragma unroll
    for (uint32_t k = 0; k < FV; ++k) {
      if (b[k] == 32) break;
      count_rest(G, a0[k] + 32, a1[k], want, g.nlab, found[k]);
      uint32_t d = row.need;
#pragma unroll
      for (uint32_t i = 0; i < FILTER_NEEDS; ++i) {
        const uint32_t q = row.needs[i] & 0xFFu, c = q ? found[k][row.needs[i] >> 8] : 0u;
        d += q > c ? q - c : 0u;
      }
      for (uint32_t i = 0; i < row.n_more; ++i) {
        const uint32_t e = __ldg(more + row.more + i), q = e & 0xFFu, c = found[k][e >> 8];
        d += q > c ? q - c : 0u;
      }
      const bool in = live && d <= T;
      word |= in ? 1u << b[k] : 0u;
      const uint32_t c = __ballot_sync(dev::FULL, in);
      if (cols && lane == 0) cols[(v0 + b[k]) * W + g.word] = c << g.shift;
    }
  }
  return word;
}

// filter_kernel on those graphs: a list is read at most once per group, only
// for vertices of a row's label, and no memory is taken.  A warp per (set of TS
// tiles, group), or a block (BLOCK), a tile per warp at a time.  Latency bounds
// it.  Four plain queries on 4.2 M vertices of 1,000 labels, equal degrees: 1.4
// ms, and 1.7 ms with the adjacency in host memory.  A thread per list took 3.6
// and 4.4 ms, a table of the wave's labels for every vertex 4.7 and 66 ms.  100
// queries of four vertices on 2.1 M vertices of 200 labels with hubs: 2.6 ms, 527
// and 10.2 ms in those forms.
template <uint32_t TS, bool BLOCK>
__global__ void __launch_bounds__(256) filter_count_kernel(DevGraph G, const FilterRow *__restrict__ rows,
                                                           const uint32_t *__restrict__ more,
                                                           const FilterGroup *__restrict__ groups, uint32_t ngroups,
                                                           const FilterLabel *__restrict__ glabels, uint32_t T,
                                                           uint32_t nwords, uint32_t *__restrict__ bits,
                                                           uint32_t *__restrict__ cnt, uint32_t *__restrict__ cols,
                                                           uint32_t W) {
  constexpr uint32_t WPB = BLOCK ? 1 : 8;  // items in flight per block
  __shared__ uint32_t turn[WPB][32][TS + 1], total[32];
  __shared__ uint32_t found[8][FV][FILTER_LABELS];  // per warp and vertex: its neighbours of each label of the group
  __shared__ FilterLabel want[WPB][FILTER_LABELS];
  const uint32_t lane = dev::lane_id(), warp = threadIdx.x >> 5;
  const uint32_t at = BLOCK ? 0 : warp;
  const uint32_t nsets = (nwords + TS - 1) / TS;
  const uint64_t items = (uint64_t)ngroups * nsets;
  for (uint64_t it = blockIdx.x * (uint64_t)WPB + at; it < items; it += (uint64_t)gridDim.x * WPB) {
    const uint32_t set = (uint32_t)(it / ngroups);
    const FilterGroup g = groups[it % ngroups];
    FilterRow row = {};
    if (lane < g.n) row = rows[g.row0 + lane];
    const bool live = lane < g.n && row.need <= T;
    auto tile = [&](uint32_t t, bool mine) {
      const uint64_t v0 = ((uint64_t)set * TS + t) * 32;
      return count_tile(G, v0, __ballot_sync(dev::FULL, mine), g, row, live, more, want[at], found[warp], T, cols, W);
    };
    if (BLOCK) {
      if (threadIdx.x < g.nlab) want[0][threadIdx.x] = glabels[g.lab0 + threadIdx.x];
      if (threadIdx.x < 32) total[threadIdx.x] = 0;
      __syncthreads();
      uint32_t n = 0, mine = 0;
#pragma unroll
      for (uint32_t j = 0; j < TS / 8; ++j) {
        const uint64_t v = ((uint64_t)set * TS + warp + 8 * j) * 32 + lane;
        mine |= (v < G.nv && __ldg(G.lab + v) == g.lab ? 1u : 0u) << j;
      }
      for (uint32_t j = 0; j < TS / 8; ++j) {
        const uint32_t word = tile(warp + 8 * j, mine >> j & 1u);
        turn[0][lane][warp + 8 * j] = word;
        n += __popc(word);
      }
      if (n) atomicAdd(total + lane, n);
      __syncthreads();
      for (uint32_t i = threadIdx.x; i < g.n * TS; i += 256)
        if (set * TS + i % TS < nwords)
          bits[(uint64_t)rows[g.row0 + i / TS].row * nwords + set * TS + i % TS] = turn[0][i / TS][i % TS];
      if (threadIdx.x < g.n) cnt[(uint64_t)row.row * nsets + set] = total[threadIdx.x];
      __syncthreads();  // read before the next item's are written
    } else {
      for (uint32_t i = lane; i < g.nlab; i += 32) want[at][i] = glabels[g.lab0 + i];
      __syncwarp();
      uint32_t n = 0;
      for (uint32_t t0 = 0; t0 < TS; t0 += 8) {  // eight tiles' labels in flight
        const uint64_t v = ((uint64_t)set * TS + t0) * 32 + lane;
        uint32_t mine = 0;
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) mine |= (v + j * 32 < G.nv && __ldg(G.lab + v + j * 32) == g.lab ? 1u : 0u) << j;
        for (uint32_t j = 0; j < 8; ++j) {
          const uint32_t word = tile(t0 + j, mine >> j & 1u);
          turn[at][lane][t0 + j] = word;
          n += __popc(word);
        }
      }
      if (lane < g.n) cnt[(uint64_t)row.row * nsets + set] = n;
      __syncwarp();
      for (uint32_t r = 0; r < g.n; ++r) {
        const uint32_t rr = __shfl_sync(dev::FULL, row.row, r);
        if (set * TS + lane < nwords) bits[(uint64_t)rr * nwords + set * TS + lane] = turn[at][r][lane];
      }
      __syncwarp();  // read before the next item's are written
    }
  }
}

uint32_t filter_set_tiles(uint32_t ngroups, uint32_t nwords) {
  // sets of 32 tiles (128-byte stores) once they make two warps per
  // scheduler, else sets of 8, so that a small graph's rows still spread
  return (uint64_t)ngroups * ((nwords + 31) / 32) >= 148 * 8 ? 32u : 8u;
}

template <uint32_t TS, bool BLOCK>
static void launch_count(const DevGraph &g, const FilterRow *rows, const uint32_t *more, const FilterGroup *groups,
                         uint32_t ngroups, const FilterLabel *glabels, uint32_t threshold, uint32_t *bits,
                         uint32_t *cnt, uint32_t *cols, uint32_t W, uint32_t nwords, cudaStream_t s) {
  const uint64_t items = (uint64_t)ngroups * ((nwords + TS - 1) / TS);
  uint64_t blocks = BLOCK ? items : (items + 7) / 8;
  if (blocks > 148ull * 48) blocks = 148ull * 48;
  filter_count_kernel<TS, BLOCK><<<(uint32_t)blocks, 256, 0, s>>>(g, rows, more, groups, ngroups, glabels, threshold,
                                                                  nwords, bits, cnt, cols, W);
}

void launch_filter(const DevGraph &g, const FilterRow *rows, const uint32_t *more, const FilterGroup *groups,
                   uint32_t ngroups, const FilterLabel *glabels, uint64_t held, uint32_t TS, uint32_t threshold,
                   uint32_t *bits, uint32_t *cnt, uint32_t *cols, uint32_t W, uint32_t nwords, cudaStream_t s) {
  if (nwords == 0 || ngroups == 0) return;
  const uint64_t items = (uint64_t)ngroups * ((nwords + TS - 1) / TS);
  count_launch();
  if (!g.nlc_stride) {
    // A block per item where the sets are few, or hold many vertices of a
    // group's label, whose lists one warp would read one after the other: 32
    // rows on 65,536 vertices of 80 Zipf labels with hubs, 0.37 ms for 0.90.
    // Where few, the block's barriers cost more: 100 queries on 2.1 M vertices of
    // 300 equally frequent labels (3 a set) 6.0 ms, a warp per item 2.7; at 15 a
    // set still 0.67 and 0.49.
    const auto fn = TS == 8 ? launch_count<8, true> : held >= 24 * items ? launch_count<32, true> : launch_count<32, false>;
    return fn(g, rows, more, groups, ngroups, glabels, threshold, bits, cnt, cols, W, nwords, s);
  }
  uint64_t blocks = (items + 7) / 8;
  if (blocks > 148ull * 48) blocks = 148ull * 48;
  if (TS == 32)
    filter_kernel<32><<<(uint32_t)blocks, 256, 0, s>>>(g.lab, g.nv, g.nlc, g.nlc_stride, rows, more, groups, ngroups,
                                                       threshold, nwords, bits, cnt, cols, W);
  else
    filter_kernel<8><<<(uint32_t)blocks, 256, 0, s>>>(g.lab, g.nv, g.nlc, g.nlc_stride, rows, more, groups, ngroups,
                                                      threshold, nwords, bits, cnt, cols, W);
}

// One warp per 32 words of a row (a row per grid line: a 64-bit division per
// 32 words to find them cost as much as the rest): their ranks into the rank words, their
// candidates to the row's list.  ex: exclusive scan of the filter's counts
// (all rows' sets of TS words in order), which is where a set's candidates
// start in the lists laid back to back.
__global__ void __launch_bounds__(256) rank_rows_kernel(const uint32_t *__restrict__ bits, uint32_t nrows,
                                                        uint32_t nwords, const uint64_t *__restrict__ ex,
                                                        uint32_t TS, uint64_t *__restrict__ rb,
                                                        uint32_t *__restrict__ cand) {
  const uint32_t lane = dev::lane_id();
  const uint32_t G = (nwords + 31) / 32, nsets = (nwords + TS - 1) / TS, per = 32 / TS;  // TS: 8 or 32
  for (uint32_t r = blockIdx.y; r < nrows; r += gridDim.y)
  for (uint32_t g = blockIdx.x * 8 + (threadIdx.x >> 5); g < G; g += gridDim.x * 8) {
    const uint32_t w0 = g * 32, w = w0 + lane;
    const uint64_t at = __ldg(ex + (uint64_t)r * nsets + g * per), row0 = __ldg(ex + (uint64_t)r * nsets);
    const uint64_t i = (uint64_t)r * nwords + w;
    const uint32_t word = w < nwords ? __ldg(bits + i) : 0u, c = __popc(word);
    uint32_t incl = c;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(dev::FULL, incl, d);
      if (lane >= d) incl += y;
    }
    if (w < nwords) rb[i] = ((at - row0 + incl - c) << 32) | word;
    const uint32_t total = __shfl_sync(dev::FULL, incl, 31);
    if (__reduce_max_sync(dev::FULL, c) <= 4) {  // sparse words: every lane its own
      uint32_t *to = cand + at + incl - c;
      for (uint32_t m = word; m; m &= m - 1) *to++ = w * 32u + __ffs(m) - 1;
      continue;
    }
    for (uint32_t b = 0; b < total; b += 32) {  // a candidate per lane: the first word whose count passes it
      const uint32_t q = b + lane;
      uint32_t j = 0;
#pragma unroll
      for (uint32_t step = 16; step >= 1; step >>= 1)
        if (__shfl_sync(dev::FULL, incl, j + step - 1) <= q) j += step;
      const uint32_t wj = __shfl_sync(dev::FULL, word, j), before = __shfl_sync(dev::FULL, incl - c, j);
      if (q < total) cand[at + q] = (w0 + j) * 32u + dev::nth_set_bit(wj, q - before);
    }
  }
}

void launch_rank_rows(const uint32_t *bits, uint32_t nrows, uint32_t nwords, const uint64_t *ex, uint32_t TS,
                      uint64_t *rb, uint32_t *cand, cudaStream_t s) {
  const uint32_t G = (nwords + 31) / 32;
  if (nrows == 0 || G == 0) return;
  // all of the row's words in flight for a few rows, a few blocks each for many
  uint32_t bx = (G + 7) / 8, share = 148 * 48 / nrows;
  if (share < 8) share = 8;
  if (bx > share) bx = share;
  count_launch();
  rank_rows_kernel<<<dim3(bx, nrows < 65535 ? nrows : 65535), 256, 0, s>>>(bits, nrows, nwords, ex, TS, rb, cand);
}

// Compaction of bit rows kept in the low halves of rank words
// (gem_filter_static, whose scratch is fixed).
__global__ void compact_kernel(uint64_t *__restrict__ rb, const uint64_t *__restrict__ ex, uint32_t nrows,
                               uint32_t nwords, const uint64_t *__restrict__ c_base, uint32_t *__restrict__ cand) {
  const uint64_t n = (uint64_t)nrows * nwords;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t r = (uint32_t)(i / nwords), w = (uint32_t)(i % nwords);
    const uint32_t bits = (uint32_t)rb[i];
    const uint64_t rank = ex[i] - ex[(uint64_t)r * nwords];
    rb[i] = (rank << 32) | bits;
    uint32_t m = bits, j = 0;
    uint32_t *dst = cand + c_base[r] + rank;
    while (m) {
      uint32_t b = __ffs(m) - 1;
      m &= m - 1;
      dst[j++] = w * 32u + b;
    }
  }
}

void launch_compact(uint64_t *rb, const uint64_t *ex, uint32_t nrows, uint32_t nwords, const uint64_t *c_base,
                    uint32_t *cand, cudaStream_t s) {
  uint64_t n = (uint64_t)nrows * nwords;
  if (n == 0) return;
  uint64_t blocks = (n + 255) / 256;
  if (blocks > 148ull * 32) blocks = 148ull * 32;
  count_launch();
  compact_kernel<<<(uint32_t)blocks, 256, 0, s>>>(rb, ex, nrows, nwords, c_base, cand);
}

}  // namespace gem
