// Edge-candidate tables T(u -> w): for the i-th candidate v of C(u), the
// neighbours of v that are candidates of w, in adjacency order.
//
// The reference (in-core/lib/structure/src/unifiedTrie.cu:1093-1240 with the
// kernels of construct_kernel.cu:1183-1340) runs, per directed query edge, a
// count kernel over 32-neighbour tiles, a CUB scan over the tiles of the
// *whole* data graph, a max kernel and a write kernel, with host syncs in
// between.  Here all tables of a wave share each launch, and the passes walk
// the data graph's vertex tiles (32 arcs of one vertex) once: each tile
// serves every source row whose candidates hold its vertex (in a batch of
// queries a vertex is a candidate of many rows), and membership of an arc's
// target in every target row is one word of that target's membership
// column, staged in shared memory.  The tables keep the per-source layout
// (a key's values at the key's tiles of its source), so the offsets, the
// scans and the join see the same tables as a pass over each source would
// write.
#include "device_common.cuh"
#include "kernels.h"

namespace gem {

// A grid line per source (or table): finding each key's source by binary
// search cost more than its work (180 mixed-size queries: 117 us; offsets
// 143 us).  Blocks per line for lines of at most `most` items.
static dim3 lines_grid(uint64_t lines, uint64_t most) {
  uint64_t bx = (most + 2047) / 2048;
  if (bx > 148 * 8) bx = 148 * 8;
  return dim3((uint32_t)(bx ? bx : 1), (uint32_t)(lines < 65535 ? lines : 65535));
}

__global__ void __launch_bounds__(256) key_tiles_kernel(DevGraph g, const TabSource *__restrict__ src, uint32_t nsrc,
                                                        uint32_t *__restrict__ tiles) {
  for (uint32_t s = blockIdx.y; s < nsrc; s += gridDim.y) {
    const TabSource S = src[s];
    for (uint64_t k = blockIdx.x * 256 + threadIdx.x; k < S.nkeys; k += gridDim.x * 256)
      tiles[S.key_base + k] = (__ldg(g.deg + __ldg(S.keys + k)) + 31u) >> 5;
  }
}

void launch_key_tiles(const DevGraph &g, const TabSource *d_src, uint32_t nsrc, uint64_t most_keys, uint32_t *tiles,
                      cudaStream_t s) {
  if (most_keys == 0 || nsrc == 0) return;
  count_launch();
  key_tiles_kernel<<<lines_grid(nsrc, most_keys), 256, 0, s>>>(g, d_src, nsrc, tiles);
}

__global__ void source_tile_bases_kernel(const TabSource *__restrict__ src, uint32_t nsrc, uint64_t nkeys,
                                         const uint64_t *__restrict__ tp, const uint64_t *__restrict__ vtg,
                                         uint32_t nv, uint64_t *__restrict__ out, VSrc *__restrict__ vsrc,
                                         unsigned long long *__restrict__ counters) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 2) counters[i] = 0;
  if (i <= nsrc) out[i] = tp[i < nsrc ? src[i].key_base : nkeys];
  if (i < nsrc) vsrc[src[i].pos].stb = out[i];
  if (i == nsrc + 1) out[i] = vtg[nv];
}

void launch_source_tile_bases(const TabSource *d_src, uint32_t nsrc, uint64_t nkeys, const uint64_t *tp,
                              const uint64_t *vtg, uint32_t nv, uint64_t *out, VSrc *vsrc,
                              unsigned long long *counters, cudaStream_t s) {
  count_launch();
  source_tile_bases_kernel<<<(nsrc + 2 + 255) / 256, 256, 0, s>>>(d_src, nsrc, nkeys, tp, vtg, nv, out, vsrc, counters);
}

// The entry of a vertex's label: its own index in a list of all the graph's
// labels, else found by binary search, or none (words = 0).
__device__ __forceinline__ RowLabel find_label(const RowLabel *__restrict__ labels, uint32_t n, uint32_t nlabels,
                                               uint32_t lab) {
  if (n == nlabels) {
    const uint4 r = __ldg(reinterpret_cast<const uint4 *>(labels + lab));
    return RowLabel{r.x, r.y, r.z, 0};
  }
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(&labels[mid].lab) < lab) lo = mid + 1; else hi = mid;
  }
  if (lo < n) {
    const RowLabel r = labels[lo];
    if (r.lab == lab) return r;
  }
  return RowLabel{lab, 0, 0, 0};
}

__global__ void vertex_tiles_kernel(DevGraph g, const RowLabel *__restrict__ labels, uint32_t nlab,
                                    const uint32_t *__restrict__ cols, uint32_t W,
                                    const uint32_t *__restrict__ smask, uint32_t *__restrict__ vtiles) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < g.nv; v += (uint64_t)gridDim.x * blockDim.x) {
    const RowLabel l = nlab ? find_label(labels, nlab, g.nlabels, __ldg(g.lab + v)) : RowLabel{0, 0, 1, 0};
    uint32_t any = 0;
    for (uint32_t c = 0; c < l.words && !any; ++c) any = __ldg(cols + v * W + c) & __ldg(smask + l.word0 + c);
    vtiles[v] = any ? (__ldg(g.deg + v) + 31u) >> 5 : 0u;
  }
}

void launch_vertex_tiles(const DevGraph &g, const RowLabel *labels, uint32_t nlab, const uint32_t *cols, uint32_t W,
                         const uint32_t *smask, uint32_t *vtiles, cudaStream_t s) {
  if (g.nv == 0) return;
  uint32_t blocks = (g.nv + 255) / 256;
  if (blocks > 148u * 32) blocks = 148u * 32;
  count_launch();
  vertex_tiles_kernel<<<blocks, 256, 0, s>>>(g, labels, nlab, cols, W, smask, vtiles);
}

// map[i] = the vertex of the warp's 32 whose range holds i, for the warp's
// whole range [b, e) of items; end: the lane's vertex's end.
__device__ __forceinline__ void fill_map(uint32_t b, uint32_t e, uint32_t end, uint32_t v0, uint32_t *__restrict__ map) {
  for (uint32_t i0 = b; i0 < e; i0 += 32) {
    const uint32_t i = i0 + dev::lane_id();
    uint32_t j = 0;  // the first lane whose end passes i
#pragma unroll
    for (uint32_t step = 16; step >= 1; step >>= 1)
      if (__shfl_sync(dev::FULL, end, j + step - 1) <= i) j += step;
    if (i < e) map[i] = v0 + j;
  }
}

// One warp per 32 vertices, whose tiles (and units) are one range: stores are
// coalesced and a hub's thousands of tiles are 32 to a step (a thread per
// vertex wrote them one by one, and the two maps apart).
__global__ void __launch_bounds__(256) vertex_maps_kernel(const uint64_t *__restrict__ vtg, uint32_t nv,
                                                          uint32_t *__restrict__ vt, uint32_t *__restrict__ vg) {
  const uint32_t lane = dev::lane_id();
  const uint64_t nwarps = (uint64_t)gridDim.x * 8;
  for (uint64_t w = blockIdx.x * 8ull + (threadIdx.x >> 5); w * 32 < nv; w += nwarps) {
    const uint64_t v = w * 32 + lane;
    const uint64_t end = __ldg(vtg + (v < nv ? v + 1 : nv)), first = __ldg(vtg + w * 32);
    const uint64_t last = __shfl_sync(dev::FULL, end, 31);
    fill_map((uint32_t)first, (uint32_t)last, (uint32_t)end, (uint32_t)(w * 32), vt);
    fill_map((uint32_t)(first >> 32), (uint32_t)(last >> 32), (uint32_t)(end >> 32), (uint32_t)(w * 32), vg);
  }
}

void launch_vertex_maps(const uint64_t *vtg, uint32_t nv, uint32_t *vt, uint32_t *vg, cudaStream_t s) {
  if (nv == 0) return;
  uint32_t blocks = (nv + 255) / 256;
  if (blocks > 148u * 16) blocks = 148u * 16;
  count_launch();
  vertex_maps_kernel<<<blocks, 256, 0, s>>>(vtg, nv, vt, vg);
}

__global__ void gather_u64_kernel(const uint64_t *__restrict__ a, const uint32_t *__restrict__ idx, uint32_t n,
                                  uint64_t *__restrict__ out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = __ldg(a + __ldg(idx + i));
}

void launch_gather_u64(const uint64_t *a, const uint32_t *idx, uint32_t n, uint64_t *out, cudaStream_t s) {
  if (n == 0) return;
  count_launch();
  gather_u64_kernel<<<(n + 255) / 256, 256, 0, s>>>(a, idx, n, out);
}

// 16-byte asynchronous copy global -> shared (both 16-byte aligned),
// bypassing L1; cp_async_wait_all waits for this thread's copies.
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const uint32_t sa = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
// The same for one word.
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
  const uint32_t sa = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// The table passes over vertex tiles.  One warp per unit (G tiles of 32 arcs of one
// vertex v): the arcs are read once for every source whose candidates hold
// v.  Those sources are the set bits of v's source column; the warp takes
// them 32 at a time, one per lane, and each lane computes its source's key
// position of v (rank bitmap) and tile index (tp).  The tables of those
// sources are then flattened into (source, table) pairs, again one per
// lane, 32 at a time:
//   count: each lane tests its table's target column bit (tcol) for the
//          arcs of the tile whose target has the target row's label (a few
//          of the 32; the warp stages the arcs' columns in shared memory) and
//          writes the tile's mask;
//   write: each lane reads its pair's mask and value position into a
//          per-warp record (records of empty masks dropped); then for each
//          record the lanes, one per arc, write the arcs whose bit is set
//          (and the key position) at the value position plus their rank in
//          the mask.
// The mask and value positions are those of the source's own tile order
// (mask[tile_base + lt], lt = the tile's index among the source's tiles), so
// both passes lay out every table exactly as a pass over the sources would.
struct VRec {
  uint64_t vb;  // first value position of the pair's tile
  uint32_t m;   // the tile's mask
  uint32_t kf;  // key position to record, or 0xFFFFFFFF (no key map)
};

// ONE: waves of at most 32 rows (a plain query): one column word for all of
// them, zero for other vertices, so an arc-lane holds its target's whole
// column and a table's mask is one ballot; nothing is staged.
//
// A unit is a chain of dependent loads (counter, vertex, offsets, arcs,
// columns, rank word, tile base), which bounds the passes of few rows; the
// count pass fetches the next unit's counter, vertex and offsets while this
// one's are used (the count passes of four plain queries on the scale-22 graph:
// 2.55 ms staged and without the prefetch, 2.10 ms).  The write pass does not: a
// unit held ahead by every warp doubles the window of vertices in flight, whose
// partly written value sectors L2 must then hold (993 rows on 524,288 vertices
// of 5 labels: 29.4 ms with, 24.2 without).
//
// Columns hold a vertex's bits for the rows of its own label only: a few
// words per vertex where one bit per target row of the wave was 80 words (320
// bytes staged per arc) for 180 mixed-size queries, count pass 4.2 -> 1.0 ms.
// The count pass stages them up to the word of the last row that some table
// targets (WT): rows that only key tables, as the centres of stars do, cost
// nothing there (720 star centres of one label: staged whole 4.4 ms, 3.8).
template <bool WRITE, bool ONE, uint32_t G>
__global__ void __launch_bounds__(256) table_vtx_kernel(VPass P) {
  extern __shared__ uint32_t stage[];  // count: 32 columns per tile and warp
  __shared__ VRec rec[WRITE ? 8 : 1][32 * G];  // write: the records of one round
  __shared__ uint32_t larcs[WRITE || ONE ? 1 : 8][G][NLC_MAX_LABELS];  // count: a tile's arcs to each label
  const uint32_t lane = dev::lane_id(), warp = threadIdx.x >> 5;
  const uint32_t *vmap = G > 1 ? P.vg : P.vt;
  constexpr bool AHEAD = !WRITE;
  constexpr uint32_t half = G > 1 ? 32 : 0;  // a vertex's first unit in its word of vtg
  // units are taken in order from one counter, so the units in flight
  // stay a narrow window of consecutive vertices
  unsigned long long got = 0;
  if (lane == 0) got = atomicAdd(P.next, 1ull);
  uint64_t t = P.t0 + __shfl_sync(dev::FULL, got, 0);
  const uint64_t t1 = P.end ? (uint64_t)(uint32_t)(__ldg(P.end) >> half) : P.t1;
  if (t >= t1) return;
  uint32_t v = __ldg(vmap + t);
  uint64_t a0 = __ldg(P.off + v), a1 = __ldg(P.off + v + 1);
  uint64_t c = (t - (uint32_t)(__ldg(P.vtg + v) >> half)) * G;  // the unit: tiles c .. c + nt - 1 of vertex v
  for (;;) {
    if (AHEAD && lane == 0) got = atomicAdd(P.next, 1ull);  // the next unit's number, looked at below
    const uint64_t tiles = (a1 - a0 + 31) >> 5;
    const uint32_t nt = tiles - c < G ? (uint32_t)(tiles - c) : G;
    uint32_t xs[G];
#pragma unroll
    for (uint32_t i = 0; i < G; ++i) {
      const uint64_t arc = a0 + (c + i) * 32u + lane;
      xs[i] = i < nt && arc < a1 ? __ldg(P.nbr + (arc - P.arc_shift)) : 0u;
    }
    // the valid lanes of tile i are a prefix of nvalid(i)
    const uint64_t left = a1 - a0 - c * 32u;
    auto nvalid = [&](uint32_t i) -> uint32_t {
      return left <= i * 32u ? 0u : left - i * 32u < 32u ? (uint32_t)(left - i * 32u) : 32u;
    };
    const RowLabel vl = ONE ? RowLabel{0, 0, 1, 0} : find_label(P.labels, P.nlab, P.nlabels, __ldg(P.lab + v));
    uint32_t *wst = stage + (uint64_t)warp * G * 32u * P.WT;
    uint32_t xl[G], xc[G];
    if (!WRITE && ONE) {
#pragma unroll
      for (uint32_t i = 0; i < G; ++i) xc[i] = lane < nvalid(i) ? __ldg(P.cols + xs[i]) : 0u;
    } else if (!WRITE) {
      // stage the columns of the tiles' arcs with asynchronous copies, all in
      // flight at once: of 16 bytes when they are whole 16-byte chunks
#pragma unroll
      for (uint32_t i = 0; i < G; ++i) xl[i] = lane < nvalid(i) ? __ldg(P.lab + xs[i]) : 0xFFFFFFFFu;
      __syncwarp();  // the previous unit's reads of the stage are done
#pragma unroll
      for (uint32_t i = 0; i < G; ++i) {
        const uint32_t nv = nvalid(i), x = xs[i];
        if (nv == 0) break;
        uint32_t *st = wst + i * 32u * P.WT;
        if (P.WT >= 4) {
          const uint32_t ch = P.WT >> 2;  // chunks per column
          for (uint32_t g = lane; g < ((nv * ch + 31u) & ~31u); g += 32) {
            const uint32_t l = g / ch, q = g - l * ch;
            const uint32_t xa = __shfl_sync(dev::FULL, x, l & 31u);
            if (l < nv) cp_async16(st + l * P.WT + q * 4u, P.cols + (uint64_t)xa * P.W + q * 4u);
          }
        } else if (lane < nv) {
          for (uint32_t q = 0; q < P.WT; ++q) cp_async4(st + lane * P.WT + q, P.cols + (uint64_t)x * P.W + q);
        }
        if (P.nlabels <= NLC_MAX_LABELS) {
#pragma unroll
          for (uint32_t l = 0; l < NLC_MAX_LABELS; l += 32) larcs[warp][i][l + lane] = 0;
          __syncwarp();
          const uint32_t peers = __match_any_sync(dev::FULL, xl[i]);
          if (lane < nv && lane == (uint32_t)__ffs(peers) - 1) larcs[warp][i][xl[i]] = peers;
        }
      }
      cp_async_wait_all();
      __syncwarp();
    }
    uint64_t tn = 0;
    uint32_t vn = 0;
    if (AHEAD) {
      tn = P.t0 + __shfl_sync(dev::FULL, got, 0);
      if (tn < t1) vn = __ldg(vmap + tn);
    }
    const uint32_t *sv = P.cols + (uint64_t)v * P.W;
    for (uint32_t wb = 0; wb < vl.words; wb += 32) {
      const uint32_t word = wb + lane < vl.words ? __ldg(sv + wb + lane) & __ldg(P.smask + vl.word0 + wb + lane) : 0u;
      const uint32_t cnt = __popc(word);
      uint32_t incl = cnt;
#pragma unroll
      for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(dev::FULL, incl, d);
        if (lane >= d) incl += y;
      }
      const uint32_t total = __shfl_sync(dev::FULL, incl, 31);
      for (uint32_t b = 0; b < total; b += 32) {
        // lane i takes the (b + i)-th source of this word range: the first
        // lane j whose inclusive count exceeds it holds it
        const uint32_t q = b + lane;
        uint32_t j = 0;
#pragma unroll
        for (uint32_t step = 16; step >= 1; step >>= 1)
          if (__shfl_sync(dev::FULL, incl, j + step - 1) <= q) j += step;
        const uint32_t wj = __shfl_sync(dev::FULL, word, j);
        const uint32_t exj = __shfl_sync(dev::FULL, incl - cnt, j);
        uint32_t k = 0, e0 = 0, ne = 0;
        uint64_t lt = 0;
        if (q < total) {
          const VSrc &src = P.vsrc[(vl.word0 + wb + j) * 32u + dev::nth_set_bit(wj, q - exj)];
          const uint64_t rw = __ldg(src.rb + (v >> 5));
          k = (uint32_t)(rw >> 32) + __popc((uint32_t)rw & ((1u << (v & 31u)) - 1u));
          lt = __ldg(P.tp + src.key_base + k) - src.stb + c;
          e0 = src.e0;
          ne = src.ne;
        }
        // the (source, table) pairs of these sources, one per lane
        uint32_t pin = ne;
#pragma unroll
        for (uint32_t d = 1; d < 32; d <<= 1) {
          const uint32_t y = __shfl_up_sync(dev::FULL, pin, d);
          if (lane >= d) pin += y;
        }
        const uint32_t npairs = __shfl_sync(dev::FULL, pin, 31);
        for (uint32_t pb = 0; pb < npairs; pb += 32) {
          const uint32_t p = pb + lane;
          uint32_t o = 0;  // the source lane of pair p
#pragma unroll
          for (uint32_t step = 16; step >= 1; step >>= 1)
            if (__shfl_sync(dev::FULL, pin, o + step - 1) <= p) o += step;
          const uint32_t u = p - (__shfl_sync(dev::FULL, pin, o) - __shfl_sync(dev::FULL, ne, o));
          const uint32_t pe = __shfl_sync(dev::FULL, e0, o) + u;
          const uint64_t plt = __shfl_sync(dev::FULL, lt, o);
          const uint32_t pk = __shfl_sync(dev::FULL, k, o);
          const bool have = p < npairs;
          const VEdge E = have ? P.vedge[pe] : VEdge{0, 0, 0};
          const uint64_t maddr = E.tile_base + plt;
          if (!WRITE) {
            uint32_t m[G];
#pragma unroll
            for (uint32_t g = 0; g < G; ++g) m[g] = 0;
            if (ONE) {  // one ballot per pair and tile
              const uint32_t np = npairs - pb < 32u ? npairs - pb : 32u;
              for (uint32_t i = 0; i < np; ++i) {
                const uint32_t tc = __shfl_sync(dev::FULL, E.tcol, i) & 31u;
#pragma unroll
                for (uint32_t g = 0; g < G; ++g) {
                  const uint32_t bal = __ballot_sync(dev::FULL, (xc[g] >> tc) & 1u);
                  if (lane == i) m[g] = bal;
                }
              }
            } else {
              const uint32_t sh = E.tcol & 31u;
#pragma unroll
              for (uint32_t g = 0; g < G; ++g) {
                const uint32_t nv = nvalid(g);
                if (nv == 0) break;
                // the tile's arcs whose target has the pair's target label
                uint32_t am = 0;
                if (P.nlabels <= NLC_MAX_LABELS) {
                  am = larcs[warp][g][E.tlab & (NLC_MAX_LABELS - 1)];
                } else {  // one ballot per distinct label among them
                  for (uint32_t rest = nv == 32u ? dev::FULL : (1u << nv) - 1u; rest;) {
                    const uint32_t ll = __shfl_sync(dev::FULL, xl[g], __ffs(rest) - 1);
                    const uint32_t bal = __ballot_sync(dev::FULL, xl[g] == ll) & rest;
                    if (ll == E.tlab) am = bal;
                    rest &= ~bal;
                  }
                }
                const uint32_t *col = wst + g * 32u * P.WT + ((E.tcol & 0x7FFFFFFFu) >> 5);
                while (am) {  // two arcs a step
                  const uint32_t l0 = __ffs(am) - 1;
                  am &= am - 1;
                  const uint32_t l1 = am ? __ffs(am) - 1 : l0;
                  am &= am - 1;
                  m[g] |= ((col[l0 * P.WT] >> sh) & 1u) << l0 | ((col[l1 * P.WT] >> sh) & 1u) << l1;
                }
              }
            }
#pragma unroll
            for (uint32_t g = 0; g < G; ++g)
              if (have && g < nt) P.mask[maddr + g] = m[g];
          } else {
            // records of the pair's tiles that have values, packed to the
            // front; the tile's index in the unit rides in the top byte of
            // the value position.  A key's tiles are consecutive in its
            // source's tile order, so the unit's masks and positions are
            // consecutive words.
            const uint32_t kf = have && P.vkey && (E.tcol >> 31) ? pk : 0xFFFFFFFFu;
            const uint32_t below = (1u << lane) - 1u;
            uint32_t m[G];
            uint64_t vb[G];
#pragma unroll
            for (uint32_t i = 0; i < G; ++i) {
              m[i] = have && i < nt ? __ldg(P.mask + maddr + i) : 0u;
              vb[i] = have && i < nt ? __ldg(P.vp + maddr + i) : 0ull;
            }
            __syncwarp();  // the previous round's records are read
            uint32_t nr = 0;
#pragma unroll
            for (uint32_t i = 0; i < G; ++i) {
              const uint32_t nz = __ballot_sync(dev::FULL, m[i] != 0u);
              if (m[i]) rec[warp][nr + __popc(nz & below)] = VRec{vb[i] | ((uint64_t)i << 56), m[i], kf};
              nr += __popc(nz);
            }
            __syncwarp();
            for (uint32_t i = 0; i < nr; ++i) {
              const VRec r0 = rec[warp][i];
              if ((r0.m >> lane) & 1u) {
                const uint32_t ti = (uint32_t)(r0.vb >> 56);
                uint32_t xi = xs[0];
#pragma unroll
                for (uint32_t j = 1; j < G; ++j) xi = ti == j ? xs[j] : xi;
                const uint64_t pos = (r0.vb & ((1ull << 56) - 1)) + __popc(r0.m & below);
                P.values[pos] = xi;
                if (r0.kf != 0xFFFFFFFFu) P.vkey[pos] = r0.kf;
              }
            }
          }
        }
      }
    }
    if (!AHEAD) {
      if (lane == 0) got = atomicAdd(P.next, 1ull);
      tn = P.t0 + __shfl_sync(dev::FULL, got, 0);
      if (tn < t1) vn = __ldg(vmap + tn);
    }
    if (tn >= t1) return;
    v = vn;
    a0 = __ldg(P.off + v);
    a1 = __ldg(P.off + v + 1);
    c = (tn - (uint32_t)(__ldg(P.vtg + v) >> half)) * G;
  }
}

// Tiles per unit of the count pass.  Four, as in the write pass, let a hub's
// chain of loads serve four tiles: four plain queries on the scale-22 graph
// 2.09 -> 0.81 ms, 100 at once 5.4 -> 3.7 ms.  With few hubs the units hold
// one tile and only the larger kernel shows (mixed sizes on equal degrees 1.01
// -> 1.12 ms), so there one.  For wide columns one too: where a vertex is in
// hundreds of rows the pairs bound the pass, and more resident warps win (720
// star centres, W = 24: 3.8 ms, in units of four 4.5), though queries whose rows
// are targets as well would gain (140 mixed-size queries at scale 22, W = 16: 40.6
// and 23.4 ms).
uint32_t table_count_tiles(uint32_t W, uint32_t nlab, uint64_t vtiles, uint64_t vunits) {
  return nlab == 0 || (W <= 8 && vtiles >= vunits + vunits / 4) ? TAB_WGROUP : 1u;
}

// Dynamic shared memory of a count block, at most (count_warps keeps to it: a
// warp's stage is 16 KB for the widest columns).
constexpr uint32_t COUNT_SMEM = 96u << 10;

// Warps per block of the count pass: each warp stages 32 columns of WT words
// per tile; blocks stay within COUNT_SMEM so that two fit an SM.
static uint32_t count_warps(uint32_t WT, uint32_t G) {
  const uint64_t per_warp = 32ull * G * WT * 4;
  const uint64_t w = COUNT_SMEM / per_warp;
  return w > 8 ? 8u : w < 1 ? 1u : (uint32_t)w;
}

uint32_t table_col_words(uint32_t words) {
  return words <= 1 ? 1u : words == 2 ? 2u : (words + 3) / 4 * 4;
}

bool table_vtx_fits(uint32_t W) { return W == 1 || W == 2 || (W % 4 == 0 && W <= 128); }

// Persistent grid: what the SMs hold at once (blocks per SM by occupancy).
// Its warps take tiles in order from the launch's counter, so the tiles in
// flight are a window of consecutive vertices, and the rank words, tile
// bases, masks and positions they read are the same few lines per source
// and table, which stay in L2 while the window passes (a static stride lets
// the warps drift apart until they touch the whole order at once).
static uint32_t resident_blocks(const void *fn, int threads, size_t smem, uint64_t want) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem);
  uint64_t b = (uint64_t)(sms > 0 ? sms : 148) * (uint64_t)(per_sm > 0 ? per_sm : 1);
  if (b > want) b = want;
  return (uint32_t)(b ? b : 1);
}

template <bool WRITE, bool ONE, uint32_t G>
static void launch_vtx(const VPass &P, uint32_t warps, size_t smem, cudaStream_t s) {
  const void *fn = (const void *)table_vtx_kernel<WRITE, ONE, G>;
  // A limit above the default (48 KB with the static part) belongs to the
  // kernel, not to the launch, and lanes launch from threads of their own: always
  // the most that any wave takes (the wave's own size let one lane lower it
  // between another lane's two calls, whose launch then failed).
  if (smem > 32u << 10) cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)COUNT_SMEM);
  const uint32_t blocks = resident_blocks(fn, (int)warps * 32, smem, (P.t1 - P.t0 + warps - 1) / warps);
  table_vtx_kernel<WRITE, ONE, G><<<blocks, warps * 32, smem, s>>>(P);
}

void launch_table_vtx(const VPass &P, bool write, cudaStream_t s) {
  if (P.t1 <= P.t0) return;
  count_launch();
  if (write && P.nlab == 0) return launch_vtx<true, true, TAB_WGROUP>(P, 8, 0, s);
  if (write) return launch_vtx<true, false, TAB_WGROUP>(P, 8, 0, s);
  if (P.nlab == 0) return launch_vtx<false, true, TAB_WGROUP>(P, 8, 0, s);
  const uint32_t G = P.units ? TAB_WGROUP : 1u, warps = count_warps(P.WT, G);
  const size_t smem = (size_t)warps * 32 * G * P.WT * 4;
  if (G > 1) launch_vtx<false, false, TAB_WGROUP>(P, warps, smem, s);
  else launch_vtx<false, false, 1>(P, warps, smem, s);
}

__global__ void edge_value_bases_kernel(const TabEdge *__restrict__ edges, uint32_t nedge,
                                       const uint64_t *__restrict__ vp, uint64_t tiles, uint64_t *__restrict__ out) {
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e <= nedge; e += gridDim.x * blockDim.x)
    out[e] = vp[e < nedge ? edges[e].tile_base : tiles];
}

void launch_edge_value_bases(const TabEdge *d_edge, uint32_t nedge, const uint64_t *vp, uint64_t tiles,
                             uint64_t *out, cudaStream_t s) {
  count_launch();
  edge_value_bases_kernel<<<(nedge + 256) / 256, 256, 0, s>>>(d_edge, nedge, vp, tiles, out);
}

__global__ void __launch_bounds__(256) table_offsets_kernel(const TabSource *__restrict__ srcs,
                                                            const TabEdge *__restrict__ edges, uint32_t nedge,
                                                            const uint64_t *__restrict__ tp,
                                                            const uint64_t *__restrict__ vp) {
  for (uint32_t e = blockIdx.y; e < nedge; e += gridDim.y) {
    const TabEdge E = edges[e];
    const TabSource S = srcs[E.src];
    const uint64_t first = __ldg(tp + S.key_base);
    for (uint64_t key = blockIdx.x * 256 + threadIdx.x; key <= S.nkeys; key += gridDim.x * 256)
      E.offsets[key] = __ldg(vp + E.tile_base + (__ldg(tp + S.key_base + key) - first));
  }
}

void launch_table_offsets(const TabSource *d_src, const TabEdge *d_edge, uint32_t nedge, const uint64_t *tp,
                          const uint64_t *vp, uint64_t most_keys, cudaStream_t s) {
  if (nedge == 0) return;
  count_launch();
  table_offsets_kernel<<<lines_grid(nedge, most_keys + 1), 256, 0, s>>>(d_src, d_edge, nedge, tp, vp);
}

}  // namespace gem
