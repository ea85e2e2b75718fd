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

// found[i] = neighbours with label want[i].lab (sorted) in the list [a0, a1),
// at least want[i].most where the list holds that many.
__device__ __forceinline__ void count_labels(const DevGraph &G, uint64_t a0, uint64_t a1, const FilterLabel *want,
                                             uint32_t n, uint32_t *found) {
  const uint32_t lane = dev::lane_id();
  __syncwarp();  // the previous vertex's counts are read
  for (uint32_t i = lane; i < n; i += 32) found[i] = 0;
  __syncwarp();
  for (uint64_t b = a0; b < a1; b += 128) {
    uint32_t l[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      const uint64_t i = b + 32 * k + lane;
      l[k] = i < a1 ? __ldg(G.nbr + i) : dev::FULL;
    }
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k)
      if (l[k] != dev::FULL) l[k] = __ldg(G.lab + l[k]);
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      uint32_t lo = 0, hi = n;
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (want[mid].lab < l[k]) lo = mid + 1; else hi = mid;
      }
      if (lo < n && want[lo].lab == l[k] && b + 32 * k + lane < a1) atomicAdd(found + lo, 1u);
    }
    __syncwarp();
    bool open = false;
    for (uint32_t i = lane; i < n; i += 32) open |= found[i] < want[i].most;
    if (!__any_sync(dev::FULL, open)) break;
  }
}

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
//
// COUNT: a graph of too many labels for resident counts.  The warp counts the
// group's labels among a vertex's neighbours itself, all lanes on its list,
// 128 arcs a step, until every label has reached the most that a row wants (a
// hub's first few hundred arcs) or the list ends; vertices with too few
// neighbours are not read.  So a list is read at most once per group, only for
// vertices of a row's label, and no memory is taken.  Latency bounds it.  Four
// plain queries on 4.2 M vertices of 1,000 labels, equal degrees: 1.4 ms, and
// 1.7 ms with the adjacency in host memory.  A thread per list took 3.6 and 4.4
// ms, a table of the wave's labels for every vertex 4.7 and 69 ms.  100 queries
// of four vertices on 2.1 M vertices of 200 labels with hubs: 2.9 ms, 527 and
// 10.2 ms in those forms.
template <uint32_t TS, bool COUNT>
__global__ void __launch_bounds__(256) filter_kernel(DevGraph G, const FilterRow *__restrict__ rows,
                                                     const uint32_t *__restrict__ more,
                                                     const FilterGroup *__restrict__ groups, uint32_t ngroups,
                                                     const FilterLabel *__restrict__ glabels, uint32_t T,
                                                     uint32_t nwords, uint32_t *__restrict__ bits,
                                                     uint32_t *__restrict__ cnt, uint32_t *__restrict__ cols,
                                                     uint32_t W) {
  __shared__ uint32_t turn[8][32][TS + 1];
  __shared__ uint32_t found[COUNT ? 8 : 1][FILTER_LABELS];  // neighbours of the vertex, per label of the group
  __shared__ FilterLabel want[COUNT ? 8 : 1][FILTER_LABELS];
  const uint32_t lane = dev::lane_id(), warp = threadIdx.x >> 5;
  const uint32_t *__restrict__ lab = G.lab;
  const uint32_t nv = G.nv, stride = G.nlc_stride;
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
    if (COUNT) {
      for (uint32_t i = lane; i < g.nlab; i += 32) want[warp][i] = glabels[g.lab0 + i];
      __syncwarp();
    }
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
      for (uint32_t j = 0; COUNT && j < nsub; ++j) {  // the warp's tiles one by one, a vertex a step
        for (uint32_t mj = __shfl_sync(dev::FULL, m, j << lg); mj; mj &= mj - 1) {
          const uint32_t b = __ffs(mj) - 1;
          const uint64_t v = ((uint64_t)set * TS + t0 + j) * 32 + b;
          const uint64_t a0 = __ldg(G.off + v), a1 = __ldg(G.off + v + 1);
          bool in = false;
          if (a1 - a0 + T >= g.min_deg) {  // a row's needs add up to its degree
            count_labels(G, a0, a1, want[warp], g.nlab, found[warp]);
            if (live && sub == j) {
              uint32_t d = row.need;
#pragma unroll
              for (uint32_t i = 0; i < FILTER_NEEDS; ++i) {
                const uint32_t q = row.needs[i] & 0xFFu, c = q ? found[warp][row.needs[i] >> 8] : 0u;
                d += q > c ? q - c : 0u;
              }
              for (uint32_t i = 0; i < row.n_more; ++i) {
                const uint32_t e = __ldg(more + row.more + i), q = e & 0xFFu, c = found[warp][e >> 8];
                d += q > c ? q - c : 0u;
              }
              in = d <= T;
            }
          }
          word |= in ? 1u << b : 0u;
          const uint32_t c = __ballot_sync(dev::FULL, in);
          if (cols && lane == 0) cols[v * W + g.word] = ((c >> (j << lg)) & mine) << g.shift;
        }
      }
      while (!COUNT && __ballot_sync(dev::FULL, m != 0)) {  // two vertices a step: their loads overlap
        const bool a0 = m != 0;
        const uint32_t b0 = a0 ? __ffs(m) - 1 : 0u;
        m &= m - 1;  // 0 stays 0
        const bool a1 = m != 0;
        const uint32_t b1 = a1 ? __ffs(m) - 1 : b0;
        m &= m - 1;
        uint32_t d0 = row.need, d1 = row.need;
        if (live && a0) {
          const uint8_t *r0 = G.nlc + (vb + b0) * stride, *r1 = G.nlc + (vb + b1) * stride;
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

uint32_t filter_set_tiles(uint32_t ngroups, uint32_t nwords) {
  // sets of 32 tiles (128-byte stores) once they make two warps per
  // scheduler, else sets of 8, so that a small graph's rows still spread
  return (uint64_t)ngroups * ((nwords + 31) / 32) >= 148 * 8 ? 32u : 8u;
}

template <uint32_t TS, bool COUNT>
static void launch_sets(const DevGraph &g, const FilterRow *rows, const uint32_t *more, const FilterGroup *groups,
                        uint32_t ngroups, const FilterLabel *glabels, uint32_t threshold, uint32_t *bits, uint32_t *cnt,
                        uint32_t *cols, uint32_t W, uint32_t nwords, cudaStream_t s) {
  const uint64_t items = (uint64_t)ngroups * ((nwords + TS - 1) / TS);
  uint64_t blocks = (items + 7) / 8;
  if (blocks > 148ull * 48) blocks = 148ull * 48;
  count_launch();
  filter_kernel<TS, COUNT><<<(uint32_t)blocks, 256, 0, s>>>(g, rows, more, groups, ngroups, glabels, threshold, nwords,
                                                            bits, cnt, cols, W);
}

void launch_filter(const DevGraph &g, const FilterRow *rows, const uint32_t *more, const FilterGroup *groups,
                   uint32_t ngroups, const FilterLabel *glabels, uint32_t TS, uint32_t threshold, uint32_t *bits,
                   uint32_t *cnt, uint32_t *cols, uint32_t W, uint32_t nwords, cudaStream_t s) {
  if (nwords == 0 || ngroups == 0) return;
  const auto fn = g.nlc_stride ? (TS == 32 ? launch_sets<32, false> : launch_sets<8, false>)
                               : (TS == 32 ? launch_sets<32, true> : launch_sets<8, true>);
  fn(g, rows, more, groups, ngroups, glabels, threshold, bits, cnt, cols, W, nwords, s);
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
