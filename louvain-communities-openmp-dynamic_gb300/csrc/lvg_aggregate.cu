// lvg_aggregate.cu — aggregation phase (replaces louvainAggregateEdgesOmpW
// and louvainAggregateOmpW, inc/louvain.hxx:897-912, 987-992).
//
// Input: a level, its renumbered membership, the community -> member CSR and
// the row capacity offsets yoff (exclusive scan of each community's total
// degree, as louvainCommunityTotalDegreeOmpW + scan do, inc/louvain.hxx:989-990).
// Each community merges the neighbour communities of all its members'
// edges, self-loops included (louvainScanCommunitiesW<true>), into a hash
// table sized by the community's total degree, then writes the distinct
// (community, summed weight) pairs to its row at yoff[c] and the row's degree
// to ydeg[c] (the reference's gapped DiGraphCsr). The super-vertex's weight
// (louvainVertexWeightsOmpW on the new level, :1209: the row sum, self-loop
// included) equals the community's total and is taken from the FP64 totals
// by the driver (launch_next_vertex_weights), not re-summed here.
//
// Communities are binned by total degree like vertices in the move kernels:
// sub-warp tiles / warps with shared tables for total degrees up to 128, where
// the members' edge lists are flattened with a tile prefix scan over member
// degrees, so lanes stay busy whatever the member degrees are; blocks of 64 to
// 1024 threads with shared tables up to 8192, where a few lanes take a member
// and warps the pieces of a long row; chunks on many blocks above. Internal
// edges (into the community itself, the hottest key) are summed privately per
// lane and added once.
#include <type_traits>

#include "lvg_internal.cuh"

namespace lvg {
namespace {

__host__ __device__ constexpr int ilog2c(int x) { return x <= 1 ? 0 : 1 + ilog2c(x >> 1); }

template <int T>
__device__ __forceinline__ unsigned tile_mask() {
  if (T == 32) return 0xffffffffu;
  const int lane = threadIdx.x & 31;
  return ((1u << T) - 1u) << (lane & ~(T - 1));
}

template <class KP, class VP>
__device__ __forceinline__ bool table_add(KP keys, VP vals, int log2cap, uint32_t c, float w) {
  const uint32_t mask = (1u << log2cap) - 1u;
  uint32_t s = hash_hi(c, log2cap);
  for (uint32_t probe = 0; probe <= mask; ++probe) {
    uint32_t k = keys[s];
    if (k == c) { atomicAdd(&vals[s], w); return true; }
    if (k == EMPTY) {
      uint32_t prev = atomicCAS(&keys[s], EMPTY, c);
      if (prev == EMPTY || prev == c) { atomicAdd(&vals[s], w); return true; }
    }
    s = (s + 1u) & mask;
  }
  return false;
}

// Warp-aggregated insert (the lanes holding the same key sum their weights
// in lane order; the lowest of them calls ins).
template <class Ins>
__device__ __forceinline__ bool agg_warp_insert(uint32_t c, float w, Ins ins) {
  const unsigned grp = __match_any_sync(0xffffffffu, c);
  const int lane = threadIdx.x & 31;
  const unsigned cnt = c == EMPTY ? 0u : unsigned(__popc(grp));
  const unsigned most = __reduce_max_sync(0xffffffffu, cnt);
  float sum = 0.f;
  unsigned rem = grp;
  for (unsigned it = 0; it < most; ++it) {
    const int src = rem ? __ffs(rem) - 1 : lane;
    rem &= rem - 1u;
    const float x = __shfl_sync(0xffffffffu, w, src);
    if (it < cnt) sum += x;
  }
  if (c != EMPTY && (grp & ((1u << lane) - 1u)) == 0u) return ins(c, sum);
  return true;
}

// Visit all edges of members cmem[m0..m1), T lanes cooperating (tile mask
// m). Edges into the community itself (`self`, the hottest key: every
// internal edge) are summed in the lane-private `self_w`; the others go to
// `add(key, weight)`, which returns false to stop early. Returns edges read.
template <int T, class Add>
__device__ __forceinline__ uint64_t visit_members(const AggArgs &a, uint32_t m0, uint32_t m1, int tl, unsigned m,
                                                  uint32_t self, float &self_w, Add add) {
  uint64_t nread = 0;
  bool go = true;
  for (uint32_t base = m0; base < m1; base += T) {
    const uint32_t mm = base + tl;
    uint32_t dg = 0;
    uint64_t o = 0;
    if (mm < m1) {
      const uint32_t u = a.cmem[mm];
      dg = a.deg[u];
      o = a.off[u];
    }
    uint32_t incl = dg;
#pragma unroll
    for (int sh = 1; sh < T; sh <<= 1) {
      uint32_t t = __shfl_up_sync(m, incl, sh, T);
      if (tl >= sh) incl += t;
    }
    const uint32_t total = __shfl_sync(m, incl, T - 1, T);
    nread += total;
    for (uint32_t k0 = 0; k0 < total; k0 += T) {
      const uint32_t k = k0 + tl;
      // owner lane: first lane whose inclusive prefix exceeds k
      int lo = 0, hi = T - 1;
#pragma unroll
      for (int step = 0; step < ilog2c(T); ++step) {
        const int mid = (lo + hi) >> 1;
        const uint32_t x = __shfl_sync(m, incl, mid, T);
        if (x <= k) lo = mid + 1; else hi = mid;
      }
      const uint32_t oincl = __shfl_sync(m, incl, lo, T);
      const uint32_t odeg = __shfl_sync(m, dg, lo, T);
      const uint64_t oo = __shfl_sync(m, o, lo, T);
      uint32_t c = EMPTY;
      float w = 0.f;
      if (go && k < total) {
        const uint64_t e = oo + (k - (oincl - odeg));
        c = a.vcom[a.key[e]];
        w = a.w[e];
        if (c == self) { self_w += w; c = EMPTY; }
      }
      if constexpr (T == 32) {
        // a whole warp: lanes holding the same community add once
        go = __all_sync(0xffffffffu, agg_warp_insert(c, w, add)) && go;
      } else {
        if (c != EMPTY) go = add(c, w);
      }
    }
  }
  return nread;
}

constexpr int TILE_BLOCK = 256;

template <int T, int C>
__global__ void __launch_bounds__(TILE_BLOCK) agg_tile_kernel(AggArgs a) {
  constexpr int LOGC = ilog2c(C);
  constexpr int TPB = TILE_BLOCK / T;
  extern __shared__ __align__(16) uint8_t smem[];
  const int tib = threadIdx.x / T;
  const int tl = threadIdx.x & (T - 1);
  const int lane = threadIdx.x & 31;
  uint32_t *keys = reinterpret_cast<uint32_t *>(smem) + tib * C;
  float *vals = reinterpret_cast<float *>(smem + size_t(TPB) * C * sizeof(uint32_t)) + tib * C;
  const unsigned m = tile_mask<T>();
  const uint32_t ntiles = gridDim.x * TPB;
  unsigned long long nread = 0;
  bool ok = true;
  for (uint32_t i = blockIdx.x * TPB + tib; i < a.count; i += ntiles) {
    const uint32_t c = a.list[i];
    const uint32_t m0 = a.coff[c], m1 = a.coff[c + 1];
#pragma unroll
    for (int s = tl; s < C; s += T) { keys[s] = EMPTY; vals[s] = 0.f; }
    __syncwarp(m);
    float self_w = 0.f;
    nread += visit_members<T>(a, m0, m1, tl, m, c, self_w, [&](uint32_t k, float w) {
      ok &= table_add(keys, vals, LOGC, k, w);
      return true;
    });
#pragma unroll
    for (int sh = T / 2; sh > 0; sh >>= 1) self_w += __shfl_xor_sync(m, self_w, sh, T);
    __syncwarp(m);
    if (tl == 0 && self_w != 0.f) ok &= table_add(keys, vals, LOGC, c, self_w);
    __syncwarp(m);
    const uint64_t y0 = a.yoff[c];
    uint32_t cnt = 0;
#pragma unroll
    for (int s0 = 0; s0 < C; s0 += T) {
      const int s = s0 + tl;
      const uint32_t k = keys[s];
      const bool has = k != EMPTY;
      const unsigned bal = (__ballot_sync(m, has) >> (lane & ~(T - 1))) & (T == 32 ? 0xffffffffu : ((1u << T) - 1u));
      if (has) {
        const uint32_t r = __popc(bal & ((1u << tl) - 1u));
        const float v = vals[s];
        a.ykey[y0 + cnt + r] = k;
        a.yw[y0 + cnt + r] = v;
      }
      cnt += __popc(bal);
    }
    if (tl == 0) a.ydeg[c] = cnt;
    __syncwarp(m);
  }
  if (tl != 0) nread = 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) nread += __shfl_xor_sync(0xffffffffu, nread, o);
  const bool bad = __any_sync(0xffffffffu, !ok);
  if (lane == 0) {
    if (nread) atomicAdd(&a.ctr->agg_edges, nread);
    if (bad) atomicOr(&a.ctr->err, ERR_TABLE_FULL);
  }
}

// ------------------------------------------------------------ groups of warps

// How a level's weights add up: any FP32, all 1, or whole numbers whose total
// is below 2^31 (integer shared-memory atomics are native, FP32 ones are a
// compare-and-swap loop; the integer sums are exact and rounded to FP32 once).
enum Weights { FLOATS, UNIT, WHOLE };
template <int MODE>
using Sum = typename std::conditional<MODE == FLOATS, float, uint32_t>::type;
template <int MODE>
__device__ __forceinline__ Sum<MODE> weight(const AggArgs &a, uint64_t i) {
  if constexpr (MODE == FLOATS) return __ldcs(a.w + i);
  else if constexpr (MODE == WHOLE) return __float2uint_rn(__ldcs(a.w + i));
  else return 1u;
}
template <int MODE>
__device__ __forceinline__ float value(uint32_t bits) {
  if constexpr (MODE == FLOATS) return __uint_as_float(bits);
  else return float(bits);
}

// Add w to community c's slot of a table (linear probing from slot s). False
// when every slot holds another community. `claims` counts the slots taken.
template <class V>
__device__ __forceinline__ bool sum_add(uint32_t *keys, uint32_t *vals, uint32_t slots, uint32_t s, uint32_t c, V w,
                                        uint32_t &claims) {
  for (uint32_t p = 0; p < slots; ++p) {
    uint32_t k = keys[s];
    if (k == EMPTY) {
      k = atomicCAS(&keys[s], EMPTY, c);
      if (k == EMPTY) {
        k = c;
        ++claims;
      }
    }
    if (k == c) {
      atomicAdd(reinterpret_cast<V *>(&vals[s]), w);
      return true;
    }
    s = (s + 1u) & (slots - 1u);
  }
  return false;
}
template <class V>
__device__ __forceinline__ bool sum_add(uint32_t *keys, uint32_t *vals, uint32_t slots, uint32_t s, uint32_t c, V w) {
  uint32_t claims = 0;
  return sum_add(keys, vals, slots, s, c, w, claims);
}

// Visit the edges [e0, e1) of the members cmem[m0..m1), counted along the
// members in order (mpre; nullptr: every edge; `total` edges in all), by the
// whole block: one to eight lanes per member by the members' mean degree, rows
// of more than LONG_ROW edges put aside (long_o, long_n; at most MAXLONG of
// them, the others visited by their own lanes) and then taken in pieces of 128
// edges, a warp each. Edges into `self` are summed in self_w,
// the others go to add(community, weight). Ends without a barrier.
constexpr uint32_t LONG_ROW = 64;
template <int MODE, int B, int MAXLONG, class Add>
__device__ __forceinline__ void visit(const AggArgs &a, const uint64_t *mpre, uint64_t e0, uint64_t e1, uint32_t total, uint32_t m0,
                                      uint32_t m1, uint32_t self, Sum<MODE> &self_w, uint64_t *long_o, uint32_t *long_n,
                                      uint32_t *nlong, Add add) {
  constexpr int U = 4;  // edges of a lane in flight
  auto run = [&](uint64_t o, uint32_t n, uint32_t t, uint32_t step) {
    for (uint32_t j = t; j < n; j += U * step) {
      uint32_t c[U];
      Sum<MODE> w[U];
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const bool in = j + k * step < n;
        c[k] = in ? __ldcs(a.key + o + j + k * step) : EMPTY;
        w[k] = in ? weight<MODE>(a, o + j + k * step) : Sum<MODE>(0);
      }
#pragma unroll
      for (int k = 0; k < U; ++k) c[k] = c[k] != EMPTY ? a.vcom[c[k]] : EMPTY;
#pragma unroll
      for (int k = 0; k < U; ++k) {
        if (c[k] == self) self_w += w[k];
        else if (c[k] != EMPTY) add(c[k], MODE == UNIT ? Sum<MODE>(1) : w[k]);  // (the constant 1: counted per address)
      }
    }
  };
  const uint32_t mean = total / (m1 - m0);
  const uint32_t lgl = mean >= 8 ? 3u : mean >= 4 ? 2u : mean >= 2 ? 1u : 0u, L = 1u << lgl;
  const uint32_t sl = threadIdx.x & (L - 1u), lead = threadIdx.x & 31u & ~(L - 1u);
  for (uint32_t m = m0 + (threadIdx.x >> lgl); m < m1; m += B >> lgl) {
    const uint32_t u = a.cmem[m];
    uint64_t o = a.off[u];
    uint32_t n = a.deg[u];
    if (mpre) {  // only the part of the row inside [e0, e1)
      const uint64_t f = mpre[m], l = f + n;
      const uint64_t lo = f > e0 ? f : e0, hi = l < e1 ? l : e1;
      o += lo - f;
      n = hi > lo ? uint32_t(hi - lo) : 0u;
    }
    uint32_t at = MAXLONG;
    if (n > LONG_ROW) {
      if (sl == 0) at = atomicAdd(nlong, 1u);
      at = __shfl_sync(((1u << L) - 1u) << lead, at, lead);
    }
    if (at < MAXLONG) {
      if (sl == 0) { long_o[at] = o; long_n[at] = n; }
    } else {
      run(o, n, sl, L);
    }
  }
  __syncthreads();
  const uint32_t nl = min(*nlong, uint32_t(MAXLONG));
  constexpr uint32_t W = B / 32;
  for (uint32_t i = 0; i < nl; ++i) {
    const uint32_t n = long_n[i];
    for (uint32_t p = ((threadIdx.x >> 5) + W - i % W) % W; p * 128u < n; p += W)
      run(long_o[i] + p * 128u, min(128u, n - p * 128u), threadIdx.x & 31u, 32);
  }
}

// One block per community of total degree 129-8192: its members' edges summed
// per neighbour community in a shared table of twice its total degree (at most
// 2^LOGS slots, or twice the community count where that is less), then written
// out as the row. Each of the three steps is a chain of gathers, so the blocks
// are small where the communities are (64 threads up to total degree 256):
// several communities per SM at different steps. Measured on level 0 of an
// R-MAT scale-23 run against one warp per 32 members, a claim counter and an
// HBM fallback table: total degree 129-512 1.5 -> 0.9 ms, 513-2048 8.7 -> 1.1
// ms, 2049-8192 7.0 -> 0.9 ms. (Long rows in pieces, not a row per warp: 5.6 ->
// 1.0 ms for the last.)
template <int MODE, int B, int LOGS>
__global__ void __launch_bounds__(B) agg_group_kernel(AggArgs a) {
  extern __shared__ __align__(16) uint32_t tab[];
  constexpr int MAXLONG = (1 << LOGS) / (2 * int(LONG_ROW)) + 1;
  __shared__ uint64_t long_o[MAXLONG];
  __shared__ uint32_t long_n[MAXLONG];
  __shared__ uint32_t s_cnt, s_nlong;
  const int lane = threadIdx.x & 31;
  unsigned long long nread = 0;
  bool ok = true;
  for (uint32_t i = blockIdx.x; i < a.count; i += gridDim.x) {
    const uint32_t c = a.list[i];
    const uint32_t m0 = a.coff[c], m1 = a.coff[c + 1];
    const uint64_t y0 = a.yoff[c], tdeg = a.yoff[c + 1] - y0;
    const int lg = min(LOGS, max(5, ceil_log2(2ull * (tdeg < a.cn ? tdeg : a.cn))));
    const uint32_t slots = 1u << lg;
    uint32_t *keys = tab, *vals = tab + slots;
    for (uint32_t s = threadIdx.x; s < slots; s += B) { keys[s] = EMPTY; vals[s] = 0u; }
    if (threadIdx.x == 0) { s_cnt = 0; s_nlong = 0; }
    __syncthreads();
    Sum<MODE> self_w = 0;
    visit<MODE, B, MAXLONG>(a, nullptr, 0, 0, uint32_t(tdeg), m0, m1, c, self_w, long_o, long_n, &s_nlong,
                            [&](uint32_t k, Sum<MODE> w) { ok &= sum_add(keys, vals, slots, hash_hi(k, lg), k, w); });
    if (threadIdx.x == 0) nread += tdeg;
    // internal weight: one insertion per warp
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) self_w += __shfl_xor_sync(0xffffffffu, self_w, o);
    if (lane == 0 && self_w != Sum<MODE>(0)) ok &= sum_add(keys, vals, slots, hash_hi(c, lg), c, self_w);
    __syncthreads();
    for (uint32_t s = threadIdx.x; s - lane < slots; s += B) {
      const uint32_t k = s < slots ? keys[s] : EMPTY;
      const unsigned bal = __ballot_sync(0xffffffffu, k != EMPTY);
      uint32_t base = 0;
      if (lane == 0 && bal) base = atomicAdd(&s_cnt, uint32_t(__popc(bal)));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (k != EMPTY) {
        const uint64_t y = y0 + base + __popc(bal & ((1u << lane) - 1u));
        a.ykey[y] = k;
        a.yw[y] = value<MODE>(vals[s]);
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) a.ydeg[c] = s_cnt;
  }
  if (threadIdx.x == 0 && nread) atomicAdd(&a.ctr->agg_edges, nread);
  if (!ok) atomicOr(&a.ctr->err, ERR_TABLE_FULL);
}

// ------------------------------------------------------------ communities above total degree 8192
//
// A community's members' edges, counted along the members in order, are the
// range [mpre[m0], mpre[m1]) of the member-degree prefix mpre. The largest
// communities (after the first pass of a power-law graph, a handful hold most
// of the edges) are cut into AGG_CHUNK-edge chunks, a run of consecutive ones
// per block. A block sums its chunks per neighbour community in a shared table,
// as many as leave room for the next chunk's communities, and writes the
// (community, weight) pairs out as a list grouped by the community's hash
// partition (parts: as many as leave about AGG_PART distinct communities each;
// seg: the groups' bounds). A second kernel, a block per (community,
// partition), sums a partition's pairs of all lists the same way and appends
// them to the community's merged row. The lists lie in the row's own place (a
// list has at most as many pairs as its chunks edges, and the row has room for
// them all), so a third kernel copies the merged row there: lists of their own
// took 8 bytes per edge of these communities. No table in global memory: its
// atomics (two per pair) took longer than both kernels. Measured on an R-MAT scale-23 run against such
// tables: level 0 4.7 -> 2.9 ms, scale 18 2.4 -> 0.1 ms (too few chunks to hide
// the atomics); a fixed eight lanes per list in the merge took 11 ms where a
// community has two partitions.
// Partitions take every bit of the id (two multiply-and-shift rounds: lowbias32,
// published by Chris Wellons), unlike the tables' slots (chunk_slot: the high bits
// after one multiplication by MurmurHash3's 0x85EBCA6B).
__device__ __forceinline__ uint32_t part_of(uint32_t c, uint32_t R) {
  c = (c ^ (c >> 16)) * 0x7FEB352Du;
  c = (c ^ (c >> 15)) * 0x846CA68Bu;
  return __umulhi(c ^ (c >> 16), R);
}
// Table slots by a hash that is not the rows' order: the rows of an aggregated
// level are stored in the order of hash_hi, and a chunk of one would crowd
// into one stretch of slots.
constexpr int CHUNK_LOGS = 13, MERGE_LOGS = 14;
static_assert((1u << CHUNK_LOGS) == 2 * AGG_CHUNK, "a chunk's communities fill half its table");
static_assert((1u << MERGE_LOGS) == 2 * AGG_PART, "a partition's communities fill about half its table");
__device__ __forceinline__ uint32_t chunk_slot(uint32_t c) { return (c * 0x85EBCA6Bu) >> (32 - CHUNK_LOGS); }

// A warp finds the last m in [lo, hi) with mpre[m] <= e, 32 probes a step.
__device__ __forceinline__ uint32_t member_of(const uint64_t *mpre, uint32_t lo, uint32_t hi, uint64_t e) {
  const uint32_t lane = threadIdx.x & 31u;
  while (hi - lo > 1) {
    const uint32_t step = (hi - lo + 31) / 32;
    const uint64_t x = uint64_t(lo) + uint64_t(lane + 1) * step;
    const unsigned m = __ballot_sync(0xffffffffu, x < hi && mpre[x] <= e);
    lo += __popc(m) * step;
    hi = min(hi, lo + step);
  }
  return lo;
}

template <int MODE, int B>
__global__ void __launch_bounds__(B) agg_chunk_kernel(AggArgs a, AggChunks ch) {
  extern __shared__ __align__(16) uint32_t tab[];  // keys, values, partition counters
  constexpr uint32_t CS = 1u << CHUNK_LOGS;
  constexpr int MAXLONG = int(AGG_CHUNK / LONG_ROW) + 1;
  __shared__ uint64_t long_o[MAXLONG];
  __shared__ uint32_t long_n[MAXLONG];
  __shared__ uint32_t s_nlong, s_m[2], s_used, s_list;
  uint32_t *keys = tab, *vals = tab + CS, *pc = tab + 2 * CS;
  const int lane = threadIdx.x & 31;
  const uint4 cr = ch.run[blockIdx.x];  // (community slot, first chunk, chunks)
  const uint32_t j = cr.x, R = ch.parts[j];
  const uint32_t c = ch.comm[j];
  const uint32_t m0 = a.coff[c], m1 = a.coff[c + 1];
  const uint64_t ebeg = ch.mpre[m0], eend = ch.mpre[m1];
  uint32_t from = cr.y;  // the first chunk in the table
  bool ok = true;
  for (uint32_t k = cr.y; k < cr.y + cr.z; ++k) {
    const uint64_t e0 = ebeg + uint64_t(k) * AGG_CHUNK;
    const uint64_t e1 = min(eend, e0 + AGG_CHUNK);
    if (from == k) {
      for (uint32_t s = threadIdx.x; s < CS; s += B) { keys[s] = EMPTY; vals[s] = 0u; }
      for (uint32_t r = threadIdx.x; r < R; r += B) pc[r] = 0;
      if (threadIdx.x == 0) s_used = 0;
    }
    if (threadIdx.x == 0) s_nlong = 0;
    if (threadIdx.x < 64) {  // the members holding the chunk's first and last edge
      const uint32_t m = member_of(ch.mpre, m0, m1, threadIdx.x < 32 ? e0 : e1 - 1);
      if (lane == 0) s_m[threadIdx.x >> 5] = m;
    }
    __syncthreads();
    Sum<MODE> self_w = 0;
    uint32_t claims = 0;
    visit<MODE, B, MAXLONG>(a, ch.mpre, e0, e1, uint32_t(e1 - e0), s_m[0], s_m[1] + 1, c, self_w, long_o, long_n, &s_nlong,
                            [&](uint32_t x, Sum<MODE> w) { ok &= sum_add(keys, vals, CS, chunk_slot(x), x, w, claims); });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) self_w += __shfl_xor_sync(0xffffffffu, self_w, o);
    if (lane == 0 && self_w != Sum<MODE>(0)) ok &= sum_add(keys, vals, CS, chunk_slot(c), c, self_w, claims);
    claims = __reduce_add_sync(0xffffffffu, claims);
    if (lane == 0 && claims) atomicAdd(&s_used, claims);
    __syncthreads();
    // room for another chunk: at most 5/8 of the slots taken after it
    if (k + 1 < cr.y + cr.z && s_used <= CS / 8) {
      __syncthreads();
      continue;
    }
    // the pairs, grouped by partition: counts, their prefix, places (lanes of
    // one partition take theirs together)
    for (uint32_t s = threadIdx.x; s < CS; s += B) {  // (whole warps)
      const uint32_t r = keys[s] != EMPTY ? part_of(keys[s], R) : EMPTY;
      const unsigned grp = __match_any_sync(0xffffffffu, r);
      if (r != EMPTY && (grp & ((1u << lane) - 1u)) == 0u) atomicAdd(&pc[r], uint32_t(__popc(grp)));
    }
    if (threadIdx.x == 0) {
      s_list = atomicAdd(&ch.nlist[j], 1u);
      ch.list_at[ch.list_off[j] + s_list] = from;
    }
    __syncthreads();
    uint32_t *seg = ch.seg + ch.seg_off[j] + uint64_t(s_list) * (R + 1);
    if (threadIdx.x < 32) {
      uint32_t carry = 0;
      for (uint32_t r0 = 0; r0 < R; r0 += 32) {
        const uint32_t r = r0 + lane, x = r < R ? pc[r] : 0u;
        uint32_t inc = x;
#pragma unroll
        for (int sh = 1; sh < 32; sh <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, inc, sh);
          if (lane >= sh) inc += y;
        }
        if (r < R) { pc[r] = carry + inc - x; seg[r] = carry + inc - x; }
        carry += __shfl_sync(0xffffffffu, inc, 31);
      }
      if (lane == 0) seg[R] = carry;
    }
    __syncthreads();
    const uint64_t p0 = a.yoff[c] + uint64_t(from) * AGG_CHUNK;
    uint32_t *yv = reinterpret_cast<uint32_t *>(a.yw);
    for (uint32_t s = threadIdx.x; s < CS; s += B) {
      const uint32_t x = keys[s];
      const uint32_t r = x != EMPTY ? part_of(x, R) : EMPTY;
      const unsigned grp = __match_any_sync(0xffffffffu, r);
      const int leader = __ffs(grp) - 1;
      uint32_t at = 0;
      if (r != EMPTY && lane == leader) at = atomicAdd(&pc[r], uint32_t(__popc(grp)));
      at = __shfl_sync(0xffffffffu, at, leader) + __popc(grp & ((1u << lane) - 1u));
      if (r != EMPTY) { a.ykey[p0 + at] = x; yv[p0 + at] = vals[s]; }
    }
    __syncthreads();
    from = k + 1;
  }
  if (threadIdx.x == 0) {
    const uint64_t e0 = ebeg + uint64_t(cr.y) * AGG_CHUNK;
    atomicAdd(&a.ctr->agg_edges, (unsigned long long)(min(eend, e0 + uint64_t(cr.z) * AGG_CHUNK) - e0));
  }
  if (!ok) atomicOr(&a.ctr->err, ERR_TABLE_FULL);
}

template <int MODE, int B>
__global__ void __launch_bounds__(B) agg_merge_kernel(AggArgs a, AggChunks ch) {
  extern __shared__ __align__(16) uint32_t tab[];
  constexpr uint32_t CS = 1u << MERGE_LOGS;
  __shared__ uint32_t s_n, s_at;
  uint32_t *keys = tab, *vals = tab + CS;
  const int lane = threadIdx.x & 31;
  const uint2 task = ch.merge[blockIdx.x];  // (community slot, partition)
  const uint32_t j = task.x, r = task.y, R = ch.parts[j];
  const uint32_t c = ch.comm[j];
  const uint32_t nc = ch.nlist[j];
  const uint32_t *list_at = ch.list_at + ch.list_off[j];
  for (uint32_t s = threadIdx.x; s < CS; s += B) { keys[s] = EMPTY; vals[s] = 0u; }
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  bool ok = true;
  // L lanes per list's group of pairs, about a quarter of the pairs a group
  // has where every community of a chunk differs (a community of two
  // partitions has few large groups, one of hundreds thousands of small ones),
  // the next group's bounds loaded ahead
  const uint32_t want = AGG_CHUNK / (4u * R);
  const uint32_t L = min(256u, max(8u, want ? 1u << (31 - __clz(want)) : 0u));
  const uint32_t sl = threadIdx.x & (L - 1u), step = B / L;
  const uint32_t *seg = ch.seg + ch.seg_off[j] + r;
  const uint32_t *pk = a.ykey + a.yoff[c], *pv = reinterpret_cast<const uint32_t *>(a.yw) + a.yoff[c];
  uint32_t k = threadIdx.x / L;
  uint32_t b = 0, e = 0, f = 0;
  if (k < nc) { b = seg[uint64_t(k) * (R + 1)]; e = seg[uint64_t(k) * (R + 1) + 1]; f = list_at[k]; }
  for (; k < nc; k += step) {
    uint32_t nb = 0, ne = 0, nf = 0;
    if (k + step < nc) {
      nb = seg[uint64_t(k + step) * (R + 1)];
      ne = seg[uint64_t(k + step) * (R + 1) + 1];
      nf = list_at[k + step];
    }
    const uint64_t g = uint64_t(f) * AGG_CHUNK;
    for (uint32_t q = b + sl; q < e; q += 4 * L) {  // four pairs of a lane in flight
      uint32_t x[4], v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool in = q + u * L < e;
        x[u] = in ? __ldcs(pk + g + q + u * L) : EMPTY;
        v[u] = in ? __ldcs(pv + g + q + u * L) : 0u;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (x[u] == EMPTY) continue;
        Sum<MODE> w;
        if constexpr (MODE == FLOATS) w = __uint_as_float(v[u]);
        else w = v[u];
        ok &= sum_add(keys, vals, CS, hash_hi(x[u], MERGE_LOGS), x[u], w);
      }
    }
    b = nb;
    e = ne;
    f = nf;
  }
  __syncthreads();
  uint32_t mine = 0;
  for (uint32_t s = threadIdx.x; s < CS; s += B) mine += keys[s] != EMPTY;
  mine = __reduce_add_sync(0xffffffffu, mine);
  if (lane == 0 && mine) atomicAdd(&s_n, mine);
  __syncthreads();
  if (threadIdx.x == 0) s_at = s_n ? atomicAdd(&a.ydeg[c], s_n) : 0u;  // the partition's place in the row
  __syncthreads();
  uint2 *out = ch.merged + ch.merged_off[j];
  for (uint32_t s = threadIdx.x; s < CS; s += B) {
    const uint32_t k = keys[s];
    const unsigned bal = __ballot_sync(0xffffffffu, k != EMPTY);
    uint32_t at = 0;
    if (lane == 0 && bal) at = atomicAdd(&s_at, uint32_t(__popc(bal)));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(bal & ((1u << lane) - 1u));
    if (k != EMPTY) out[at] = make_uint2(k, __float_as_uint(value<MODE>(vals[s])));
  }
  if (!ok) atomicOr(&a.ctr->err, ERR_TABLE_FULL);
}

// The merged rows to their places: a block per (community, partition) as
// above, each a stretch of AGG_PART entries (and those that many partitions on).
__global__ void __launch_bounds__(256) agg_place_kernel(AggArgs a, AggChunks ch) {
  const uint2 task = ch.merge[blockIdx.x];
  const uint32_t j = task.x, c = ch.comm[j], n = a.ydeg[c];
  const uint64_t y0 = a.yoff[c];
  const uint2 *in = ch.merged + ch.merged_off[j];
  for (uint64_t b = uint64_t(task.y) * AGG_PART; b < n; b += uint64_t(ch.parts[j]) * AGG_PART)
    for (uint64_t i = b + threadIdx.x; i < min(uint64_t(n), b + AGG_PART); i += 256) {
      const uint2 x = __ldcs(in + i);
      a.ykey[y0 + i] = x.x;
      a.yw[y0 + i] = __uint_as_float(x.y);
    }
}

__global__ void comm_tdeg_kernel(const uint32_t *list, size_t n, const uint64_t *yoff, uint64_t *out) {
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
    out[i] = yoff[list[i] + 1] - yoff[list[i]];
}

__global__ void member_degrees_kernel(const uint32_t *cmem, const uint32_t *deg, size_t n, uint64_t *dst) {
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
    dst[i] = deg[cmem[i]];
}

template <class K>
void set_smem(K kernel, size_t bytes) {
  if (bytes > 48 * 1024) LVG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)));
}

template <int T, int C>
void launch_tile(const AggArgs &a, cudaStream_t s) {
  constexpr int TPB = TILE_BLOCK / T;
  const size_t smem = size_t(TPB) * C * 8;
  auto k = agg_tile_kernel<T, C>;
  static PerDevice<bool> configured;
  configured.get([&] { set_smem(k, smem); return true; });
  size_t want = (a.count + TPB - 1) / TPB;
  size_t cap = size_t(device_sms()) * (smem > 32 * 1024 ? 3 : 8);
  unsigned grid = unsigned(want < cap ? want : cap);
  if (!grid) return;
  k<<<grid, TILE_BLOCK, smem, s>>>(a);
  LVG_CHECK_LAUNCH();
}

template <int MODE, int B, int LOGS>
void launch_group(const AggArgs &a, cudaStream_t s) {
  const size_t smem = (size_t(1) << LOGS) * 8;
  auto k = agg_group_kernel<MODE, B, LOGS>;
  // as many blocks as fit the device
  static PerDevice<unsigned> fit;
  const unsigned resident = fit.get([&] {
    set_smem(k, smem);
    int per_sm = 0;
    LVG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, B, smem));
    return unsigned(per_sm > 0 ? per_sm : 1) * unsigned(device_sms());
  });
  const unsigned grid = a.count < resident ? a.count : resident;
  if (!grid) return;
  k<<<grid, B, smem, s>>>(a);
  LVG_CHECK_LAUNCH();
}

template <int MODE>
void launch_groups(int b, const AggArgs &a, cudaStream_t s) {
  switch (b) {
    case 7: launch_group<MODE, 64, 9>(a, s); break;
    case 8: launch_group<MODE, 128, 10>(a, s); break;
    case 9: launch_group<MODE, 256, 12>(a, s); break;
    case 10: launch_group<MODE, 1024, 14>(a, s); break;
    default: break;
  }
}

constexpr int AGG_CHUNK_B = 512, AGG_MERGE_B = 1024;
template <int MODE>
void launch_chunks(const AggArgs &a, const AggChunks &ch, size_t runs, size_t merges, uint32_t max_parts,
                   cudaStream_t s) {
  const size_t smem1 = (size_t(1) << CHUNK_LOGS) * 8, smem2 = (size_t(1) << MERGE_LOGS) * 8;
  auto k1 = agg_chunk_kernel<MODE, AGG_CHUNK_B>;
  auto k2 = agg_merge_kernel<MODE, AGG_MERGE_B>;
  static PerDevice<bool> configured;
  configured.get([&] {
    set_smem(k1, smem1 + size_t(AGG_MAX_PARTS) * 4);
    set_smem(k2, smem2);
    return true;
  });
  k1<<<unsigned(runs), AGG_CHUNK_B, smem1 + size_t(max_parts) * 4, s>>>(a, ch);  // (the partitions' counters behind)
  LVG_CHECK_LAUNCH();
  k2<<<unsigned(merges), AGG_MERGE_B, smem2, s>>>(a, ch);
  LVG_CHECK_LAUNCH();
  agg_place_kernel<<<unsigned(merges), 256, 0, s>>>(a, ch);
  LVG_CHECK_LAUNCH();
}

}  // namespace

void launch_comm_tdeg(const uint32_t *list, size_t n, const uint64_t *yoff, uint64_t *out, cudaStream_t s) {
  if (!n) return;
  comm_tdeg_kernel<<<grid_for(n, 256), 256, 0, s>>>(list, n, yoff, out);
  LVG_CHECK_LAUNCH();
}

void launch_member_degrees(const uint32_t *cmem, const uint32_t *deg, size_t n, uint64_t *dst, cudaStream_t s) {
  if (!n) return;
  member_degrees_kernel<<<grid_for(n, 256), 256, 0, s>>>(cmem, deg, n, dst);
  LVG_CHECK_LAUNCH();
}

void launch_aggregate_chunks(const AggArgs &a, const AggChunks &ch, size_t runs, size_t merges, uint32_t max_parts,
                             cudaStream_t s) {
  if (!runs) return;
  if (a.unit) launch_chunks<UNIT>(a, ch, runs, merges, max_parts, s);
  else if (a.whole) launch_chunks<WHOLE>(a, ch, runs, merges, max_parts, s);
  else launch_chunks<FLOATS>(a, ch, runs, merges, max_parts, s);
}

void launch_aggregate_bin(int b, const AggArgs &a, cudaStream_t s) {
  switch (b) {
    case 1: launch_tile<4, 8>(a, s); break;
    case 2: launch_tile<8, 16>(a, s); break;
    case 3: launch_tile<16, 32>(a, s); break;
    case 4: launch_tile<32, 64>(a, s); break;
    case 5: launch_tile<32, 128>(a, s); break;
    case 6: launch_tile<32, 256>(a, s); break;
    default:
      if (a.unit) launch_groups<UNIT>(b, a, s);
      else if (a.whole) launch_groups<WHOLE>(b, a, s);
      else launch_groups<FLOATS>(b, a, s);
      break;
  }
}

}  // namespace lvg
