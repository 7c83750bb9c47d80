// lvg_phase.cu — a level's whole local-moving phase in one kernel
// (louvainMoveOmpW, inc/louvain.hxx:588-609: every iteration, every colour
// class, the stop test).
//
// What bounds a level of up to a few million edges is not its work but the
// chain of steps: 16 colour classes an iteration, each of them a compaction,
// a fork onto five streams, a kernel per degree bin, a join and (deterministic
// mode) two more kernels, at 3-8 us a launch even inside a CUDA graph. Here
// one cooperative launch of at most a block per SM stays on the GPU for the
// phase; a class is two grid barriers (one in asynchronous mode), and every
// block serves all degree bins of its share of the class.
//
// A class's vertices (Level::bins, grouped by degree bin) are dealt to the
// blocks in small chunks, heaviest bins first. Per class a block
//   1. lists the active ones among its vertices per bin (the flags as they
//      are when the class starts);
//   2. decides them: hubs (degree above 8192) chunk by chunk on many blocks,
//      merged behind a further barrier; degree <= 32 by a tile of 4/8/16/32
//      lanes that groups equal communities with warp matches and needs no
//      table; degree 33-128 by a warp, 129-512 by four warps (by one where the
//      weights' order counts, ORDERED), 513-2048 by eight, above by the whole
//      block, each with an open-addressing table of twice the degree in shared
//      memory;
//   3. deterministic mode: waits until every block has decided, then commits
//      its own decisions (community, totals) and marks the movers' neighbours.
//      Asynchronous mode commits at once, on sparse uploaded levels; dense and
//      aggregated ones are decided as in deterministic mode.
// Where every weight is 1, or a whole number (the aggregated levels of a
// unit-weight graph), the tables add with integer shared-memory atomics
// (native) instead of FP32 ones (a compare-and-swap loop); the sums are exact,
// so the gains are those of exact FP32 sums.
//
// Measured on a GB300, deterministic static runs, launches -> this kernel with
// the aggregation beside it: 2K vertices 4.3 -> 1.7 ms, 131K-vertex planted
// partition 17.5 -> 3.7 ms, R-MAT scale 20 21.7 -> 8.9 ms, scale 23 129 -> 51 ms
// (its two large levels' moving 44 + 37 -> 17 + 17 ms). A class of a small level
// takes about 9 us: 1 to list, 3-4 to decide, 1 to commit, 2 a barrier; of a
// large one, what its gathers take (ncu, scale 20: warps wait at the groups'
// barriers and on gathers, 22 % of issue slots busy).
// Tried and dropped: tables of 1.5x instead of 2x to 4x the degree on half
// blocks (the longest probe of a warp decides: 21 -> 29 ms), one code copy for
// all group sizes (20.7 -> 21.6 ms), the next vertex's offset and degree
// fetched ahead (no gain).
#include <algorithm>
#include <type_traits>

#include "lvg_internal.cuh"

namespace lvg {
namespace {

constexpr int PB = 1024;                  // threads per block
constexpr int PW = PB / 32;               // warps per block
constexpr uint32_t LOG_BLOCK = 14;        // shared slots of a block's vertex (log2)
constexpr uint32_t TABLE_WORDS = 2u << LOG_BLOCK;  // keys and values
constexpr uint32_t LIST_CAP = 1920;       // listed vertices a block keeps in shared memory
constexpr uint32_t PIECE = 1024;          // edges of a large mover's row marked at once
constexpr uint32_t TODO = 256;            // hub chunks a block looks through at a time
constexpr uint32_t MERGE_FULL = 8192;     // partial entries of a hub that one block merges at once

// The level's weights: any FP32, all 1, or whole numbers whose total is below 2^31.
enum Weights { FLOATS, UNIT, WHOLE };
// With UNIT or WHOLE: the vertices' and communities' totals are known to be
// whole numbers below 2^31 too (static runs: sums of such weights), so gains
// are computed from their integers. The SM issues an FP64 instruction of a warp
// in 16 cycles, and a gain takes three of them (two additions and the rounding
// to FP32): with tables a quarter full that was two thirds of a large vertex's
// time (16.6 of 26 us above degree 2048, 5.7 of 12.8 at 257-512). The sum wu +
// tc - td is exact either way and rounded once, so the gains are the same bits.
constexpr int TOTALS = 4;
template <int MODE>
using Tot = typename std::conditional<(MODE & TOTALS) != 0, uint32_t, double>::type;
// A whole number below 2^32 out of its FP64 bits (an FP64-to-integer
// conversion would be as slow as the additions).
__device__ __forceinline__ uint32_t whole_of(double x) {
  const uint32_t hi = uint32_t(__double2hiint(x)), lo = uint32_t(__double2loint(x));
  const uint32_t top = __funnelshift_l(lo, hi, 11) | 0x80000000u;  // the mantissa's first 32 bits
  return __funnelshift_rc(top, 0u, 1054u - (hi >> 20));            // (0: shifted out)
}
template <int MODE>
__device__ __forceinline__ Tot<MODE> total(double x) {
  if constexpr ((MODE & TOTALS) != 0) return whole_of(x);
  else return x;
}
__device__ __forceinline__ float rounded(double x) { return __double2float_rn(x); }
__device__ __forceinline__ float rounded(uint32_t x) { return __uint2float_rn(x); }
// gain_of() of whole totals, beside the one of FP64 totals.
using lvg::gain_of;
__device__ __forceinline__ float gain_of(float kc, float kd, uint32_t wu, float wuf, uint32_t tc, uint32_t td, float kr) {
  const float c = __int2float_rn(int(wu + tc - td));
  return __fsub_rn(__fsub_rn(kc, kd), __fmul_rn(__fmul_rn(wuf, c), kr));
}
template <int MODE>
using Sum = typename std::conditional<(MODE & 3) == FLOATS, float, uint32_t>::type;
__device__ __forceinline__ uint32_t bits(float x) { return __float_as_uint(x); }
__device__ __forceinline__ uint32_t bits(uint32_t x) { return x; }
template <int MODE>
__device__ __forceinline__ Sum<MODE> of_bits(uint32_t x) {
  if constexpr ((MODE & 3) == FLOATS) return __uint_as_float(x);
  else return x;
}
// Weight of edge i.
template <int MODE>
__device__ __forceinline__ Sum<MODE> weight(const PhaseArgs &a, uint64_t i) {
  if constexpr ((MODE & 3) == FLOATS) return __ldcs(a.w + i);
  else if constexpr ((MODE & 3) == WHOLE) return __float2uint_rn(__ldcs(a.w + i));
  else return 1u;
}

// Deterministic runs that are not static ones of whole weights: a few marked
// vertices a class, most of the work in large ones. Their blocks share the
// vertices of degree bins 9 and 10 of a class through one list and the rows of
// large movers in pieces; dealt out beforehand, the unluckiest block of a class
// took 1.6 times the average to decide and 4 times to mark. (Two runs of a 1e-4
// |E| batch on R-MAT scale 24: 5.7 -> 3.7 ms.) Static runs keep their own
// shares: every block has many vertices, and the shared words cost small levels
// 2-5 %.
template <bool SYNC, int MODE>
constexpr bool SHARES = SYNC && (MODE & TOTALS) == 0;

// Deterministic runs of any FP32 weights: the order of a sum is part of its
// value, so up to degree 512 a vertex's weights are summed by one warp in one
// order (equal communities of 32 neighbours in lane order, then the 32s in
// turn), the same in every run and the one of the launch-by-launch kernels.
// (Four warps adding to one table at degree 129-512 let two runs of one call
// differ wherever two communities' weights are equal but for their order. First
// pass of a planted partition with fractional weights, mean degree 48 / 100 /
// 200 / 400: 2.08 / 2.43 / 1.44 / 2.58 ms, with four warps and no order 2.01 /
// 2.07 / 1.50 / 2.08, launch by launch 4.88 / 4.25 / 2.13 / 2.86.)
template <bool SYNC, int MODE>
constexpr bool ORDERED = SYNC && (MODE & 3) == FLOATS;

struct Shared {
  uint32_t off[MAX_BUCKETS];   // [class][bin]: the block's first list slot of the bin
  uint32_t pos[MAX_BUCKETS];   // [class][bin]: the bin's first position dealt to the block
  uint32_t tot[MAX_COLORS];    // the block's list slots of a class
  uint32_t cnt[NUM_BINS];      // listed vertices per bin of the current class
  uint32_t edges[NUM_BINS];    // scanned edges of the current iteration
  unsigned long long sv[NUM_BINS], se[NUM_BINS];  // the phase's vertices and edges
  unsigned long long moves;
  uint32_t redk[PW], redg[PW], redc[PW];
  uint32_t next;               // next warp-sized unit of work of the class
  uint32_t nmv, nbig;          // moves of the class; those with long rows
  uint32_t hubmv;              // hubs moved by the block's merges
  uint32_t over, bad, stop;
  uint32_t ntodo, todo[TODO];  // hub chunks that have work
  uint32_t turn;               // of the class step: the words of PhaseCtl's triples
  uint32_t unit[2];            // the block's units of the shared queue
  uint32_t any;                // some block moved a vertex before the last barrier that counts moves
  unsigned long long sum;      // the iteration's gain sum, or the union's graphs still moving
};

__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// Barrier number n of the grid (the launch is cooperative, so all blocks are
// resident). A barrier's word counts the arrivals below and `moves` above, so
// the waiting poll also tells whether any block moved a vertex (S.any); three
// words take turns, block 0 clearing the next one (whose last readers have all
// arrived at the barrier before this one). `sum` (optional) is read behind the
// barrier into S.sum. False when a wait was given up (PhaseArgs::polls), here
// or in another block: every thread of the block then returns. The other
// blocks get past this barrier at most (their next one never completes), so
// every block ends, with the class's work in whatever state it was: the host
// restores what a phase leaves zero for the next (reset_hub_scratch).
__device__ __forceinline__ bool grid_barrier(const PhaseArgs &a, Shared &S, uint32_t n, uint32_t moves,
                                             const unsigned long long *sum) {
  __syncthreads();
  if (threadIdx.x == 0) {
    if (gridDim.x == 1) {
      S.any = moves;
    } else {
      if (blockIdx.x == 0) a.ctl->bar[(n + 1) % 3] = 0;
      __threadfence();
      unsigned long long *word = &a.ctl->bar[n % 3];
      atomicAdd(word, 1ull + (static_cast<unsigned long long>(moves) << 32));
      unsigned long long v;
      uint32_t polls = 0;
      while (uint32_t(v = ld_acquire(word)) < gridDim.x) {
        ++polls;
        if (polls >= a.polls || ((polls & 255u) == 0 && ld_acquire(&a.ctl->aborted))) {
          atomicExch(&a.ctl->aborted, 1ull);
          atomicOr(&a.ctr->err, ERR_BARRIER);
          S.stop = 1;
          break;
        }
      }
      __threadfence();
      S.any = uint32_t(v >> 32);
    }
    if (sum) S.sum = *reinterpret_cast<const volatile unsigned long long *>(sum);
  }
  __syncthreads();
  return !S.stop;
}

// A barrier over the n threads (whole warps) of group `id`.
__device__ __forceinline__ void group_sync(uint32_t id, uint32_t n) {
  if (n == 32) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// The lanes of a warp holding the same key (grp) sum their weights in lane
// order; every one of them gets the sum.
template <class V>
__device__ __forceinline__ V match_sum(unsigned grp, bool some, V w, int lane) {
  const unsigned most = __reduce_max_sync(0xffffffffu, some ? unsigned(__popc(grp)) : 0u);
  V sum = 0;
  unsigned rem = some ? grp : 0u;
  for (unsigned it = 0; it < most; ++it) {
    const int src = rem ? __ffs(rem) - 1 : lane;
    const V x = __shfl_sync(0xffffffffu, w, src);
    if (rem) sum += x;
    rem &= rem - 1u;
  }
  return sum;
}

template <class V>
__device__ __forceinline__ V warp_sum(V x) {
  if constexpr (std::is_same<V, uint32_t>::value) {
    return __reduce_add_sync(0xffffffffu, x);
  } else {
#pragma unroll
    for (int sh = 16; sh > 0; sh >>= 1) x += __shfl_xor_sync(0xffffffffu, x, sh);
    return x;
  }
}

// Add w to community c's slot of a table of 2^lg slots (linear probing).
// False when every slot holds another key. Not the aggregation tables' hash
// (hash_hi): an aggregated row is stored in the order of that one, so a chunk
// of a hub's row would crowd into one stretch of slots (40 us of probing a
// chunk, against 3).
template <class V>
__device__ __forceinline__ bool add(uint32_t *keys, uint32_t *vals, uint32_t lg, uint32_t c, V w) {
  const uint32_t mask = (1u << lg) - 1u;
  uint32_t s = (c * 0x85EBCA6Bu) >> (32u - lg);
  for (uint32_t p = 0; p <= mask; ++p) {
    uint32_t k = keys[s];
    if (k == EMPTY) {
      k = atomicCAS(&keys[s], EMPTY, c);
      if (k == EMPTY) k = c;
    }
    if (k == c) {
      atomicAdd(reinterpret_cast<V *>(&vals[s]), w);
      return true;
    }
    s = (s + 1u) & mask;
  }
  return false;
}

// add() of FP32 weights by the lanes of a converged warp (c == EMPTY: nothing
// to add). An FP32 shared-memory atomic retries while other lanes use its
// address, and the neighbours of a large vertex share few communities: up to
// three communities that four lanes or more hold are summed over the warp
// first. (Whole weights need none of this: the hardware adds integers.)
__device__ __forceinline__ bool add_warp(uint32_t *keys, uint32_t *vals, uint32_t lg, uint32_t c, float w, int lane) {
  bool fine = true;
  unsigned todo = __ballot_sync(0xffffffffu, c != EMPTY);
  for (int r = 0; r < 3 && __popc(todo) >= 8; ++r) {
    const int src = __ffs(todo) - 1;
    const uint32_t key = __shfl_sync(0xffffffffu, c, src);
    const unsigned same = __ballot_sync(0xffffffffu, c == key);
    todo &= ~same;
    if (__popc(same) < 4) continue;
    const float sum = warp_sum<float>(c == key ? w : 0.f);
    if (lane == src) fine &= add<float>(keys, vals, lg, c, sum);
    if (c == key) c = EMPTY;
  }
  if (c != EMPTY) fine &= add<float>(keys, vals, lg, c, w);
  return fine;
}
// The same in one order: each community's weights summed in lane order and
// added once (ORDERED).
__device__ __forceinline__ bool add_ordered(uint32_t *keys, uint32_t *vals, uint32_t lg, uint32_t c, float w, int lane) {
  const unsigned grp = __match_any_sync(0xffffffffu, c);
  const float sum = match_sum<float>(grp, c != EMPTY, w, lane);
  return c == EMPTY || (grp & ((1u << lane) - 1u)) != 0u || add<float>(keys, vals, lg, c, sum);
}

// A community or a total that other blocks change within the class: in
// asynchronous mode read past L1, which would keep the values of the class's
// start (every vertex of a class joining the same small total).
template <bool SYNC, class T>
__device__ __forceinline__ T live(const T *p) {
  if constexpr (SYNC) return *p;
  else return __ldcg(p);
}

// R/(2M), the community that is never a target, and the graph of vertex u.
struct Of {
  float kr;
  uint32_t zero, g;
  __device__ __forceinline__ Of(const PhaseArgs &a, uint32_t u) : kr(a.kr), zero(0), g(0) {
    if (a.gid) {
      g = a.gid[u];
      kr = a.gkr[g];
      zero = a.gzero[g];
    }
  }
};

// The hash partition (of R) of a hub's community. Every bit of the id takes
// part (two multiply-and-shift rounds), so that no pattern of ids gathers in
// one partition; unlike the tables' slots, which are the high bits of one
// multiplication. (The mixer is lowbias32, published by Chris Wellons; the slots'
// factor is MurmurHash3's 0x85EBCA6B.)
__device__ __forceinline__ uint32_t hub_part(uint32_t c, uint32_t R) {
  c = (c ^ (c >> 16)) * 0x7FEB352Du;
  c = (c ^ (c >> 15)) * 0x846CA68Bu;
  return __umulhi(c ^ (c >> 16), R);
}

// A vertex's best gain into its iteration's sum: the thread's for one graph
// (flushed once an iteration), the graph's for a union.
__device__ __forceinline__ void add_gain(const PhaseArgs &a, unsigned long long &fix, const Of &G, float bg) {
  if (a.gfix) atomicAdd(&a.gfix[G.g], gain_to_fix(bg));
  else fix += gain_to_fix(bg);
}

// Graph unions, once an iteration: graph i's own stop test (as
// iter_control_kernel).
__device__ __forceinline__ void phase_control(const PhaseArgs &a, uint32_t i, uint32_t slot) {
  if (!a.gact[i]) return;
  const double el = double(a.gfix[i]) / GAIN_FIX / a.gM[i];
  a.gfix[i] = 0;
  GraphCtl &c = a.gctl[i];
  c.el = el;
  c.it += 1;
  if (el <= a.E || c.it >= uint32_t(a.itcap)) a.gact[i] = 0;
  else atomicAdd(&a.ctl->gactive[slot], 1ull);
}

// Mark the neighbours row[0..m) of u (thread t of n), four in flight; with
// resident hub tables (tabs), u's move from community d to c into the tables
// of those that are hubs.
__device__ __forceinline__ void mark_row(const PhaseArgs &a, uint32_t u, uint64_t o, uint32_t m, uint32_t t, uint32_t n,
                                         bool tabs = false, uint32_t d = 0, uint32_t c = 0) {
  for (uint32_t j = t; j < m; j += 4 * n) {
    uint32_t v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = j + k * n < m ? __ldcs(a.key + o + j + k * n) : u;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (v[k] != u) a.vaff[v[k]] = 1;
    if (tabs) {
      uint32_t h[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) h[k] = v[k] != u ? a.ht.slot[v[k]] : NO_HUB;
      for (int k = 0; k < 4; ++k)
        if (h[k] != NO_HUB) ht_move_at(a.ht, h[k], d, c, a.ctr);
    }
  }
}
// The same by whole warps (thread t of n, both multiples of 32 for lane 0): the
// hubs among a warp's 128 neighbours are dealt to its lanes, since the
// neighbours of a large vertex are often hubs and a lane with four of them
// would update their tables one after the other.
__device__ __forceinline__ void mark_row_warp(const PhaseArgs &a, uint32_t u, uint64_t o, uint32_t m, uint32_t t,
                                              uint32_t n, bool tabs, uint32_t d, uint32_t c) {
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t j = t; j - lane < m; j += 4 * n) {
    uint32_t v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = j + k * n < m ? __ldcs(a.key + o + j + k * n) : u;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (v[k] != u) a.vaff[v[k]] = 1;
    if (tabs) {
      uint32_t h[4], has[4], hits = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) h[k] = v[k] != u ? a.ht.slot[v[k]] : NO_HUB;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        has[k] = __ballot_sync(0xffffffffu, h[k] != NO_HUB);
        hits += __popc(has[k]);
      }
      for (uint32_t i = lane; i - lane < hits; i += 32) {
        uint32_t mine = NO_HUB, before = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t cnt = __popc(has[k]);
          const bool in = i >= before && i < before + cnt;
          const uint32_t x = __shfl_sync(0xffffffffu, h[k], in ? __fns(has[k], 0, int(i - before) + 1) : lane);
          if (in) mine = x;
          before += cnt;
        }
        if (mine != NO_HUB) ht_move_at(a.ht, mine, d, c, a.ctr);
        __syncwarp();
      }
    }
  }
}


// One thread: vertex u of community d leaves for c.
template <bool SYNC>
__device__ __forceinline__ void commit(const PhaseArgs &a, Shared &S, uint2 *mv, uint32_t u, uint32_t d, uint32_t c) {
  const uint32_t i = atomicAdd(&S.nmv, 1u);
  if constexpr (SYNC) {
    mv[i] = make_uint2(u, c);
  } else {
    const double wu = a.vtot[u];
    atomicAdd(&a.ctot[d], -wu);
    atomicAdd(&a.ctot[c], wu);
    a.vcom[u] = c;
  }
}

// Two rounds of 32/T vertices of degree <= T (T = 4, 8, 16, 32), one per tile
// of the warp: list[first ..), those at `n` and beyond idle; both rounds'
// loads are in flight together (a vertex is a chain of five dependent
// gathers). Each lane holds one neighbour; equal communities of a tile are
// grouped by a warp match.
constexpr int TILE_ROUNDS = 2;
template <bool SYNC, int MODE>
__device__ __forceinline__ void tile_vertices(const PhaseArgs &a, Shared &S, uint2 *mv, const uint32_t *list,
                                              uint32_t first, uint32_t n, uint32_t T, int bin,
                                              unsigned long long &fix) {
  constexpr int N = TILE_ROUNDS;
  using V = Sum<MODE>;
  const int lane = threadIdx.x & 31;
  const uint32_t tl = lane & (T - 1);
  const unsigned tmask = (T == 32 ? 0xffffffffu : ((1u << T) - 1u) << (lane & ~(T - 1)));
  uint32_t u[N], dg[N], d[N], v[N], c[N];
  Tot<MODE> wu[N], td[N];
  V w[N];
#pragma unroll
  for (int r = 0; r < N; ++r) {
    const uint32_t i = first + r * (32 / T) + lane / T;
    u[r] = i < n ? list[i] : EMPTY;
  }
#pragma unroll
  for (int r = 0; r < N; ++r) {
    dg[r] = 0;
    d[r] = EMPTY;
    wu[r] = 0;
    v[r] = u[r];
    w[r] = 0;
    if (u[r] != EMPTY) {
      const uint64_t o = a.off[u[r]];
      dg[r] = a.deg[u[r]];
      d[r] = a.vcom[u[r]];
      wu[r] = total<MODE>(a.vtot[u[r]]);
      if (tl < dg[r]) {
        v[r] = __ldcs(a.key + o + tl);
        w[r] = weight<MODE>(a, o + tl);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < N; ++r) {
    c[r] = v[r] != u[r] ? live<SYNC>(a.vcom + v[r]) : EMPTY;
    td[r] = total<MODE>(u[r] != EMPTY ? live<SYNC>(a.ctot + d[r]) : 0.0);
  }
  V kc[N], kd[N];
  Tot<MODE> tc[N];
  unsigned lead = 0;
#pragma unroll
  for (int r = 0; r < N; ++r) {
    kd[r] = 0;
    if (c[r] == d[r]) {
      kd[r] = w[r];
      c[r] = EMPTY;
    }
    const unsigned grp = __match_any_sync(0xffffffffu, c[r]) & tmask;
    const bool is = c[r] != EMPTY && (grp & ((1u << lane) - 1u)) == 0u;
    lead |= unsigned(is) << r;
    tc[r] = total<MODE>(is ? live<SYNC>(a.ctot + c[r]) : 0.0);
    if constexpr ((MODE & 3) == UNIT) {
      kc[r] = __popc(grp);
      kd[r] = __popc(__ballot_sync(0xffffffffu, kd[r] != 0u) & tmask);
    } else {
      kc[r] = match_sum<V>(grp, c[r] != EMPTY, w[r], lane);
      for (uint32_t sh = T >> 1; sh; sh >>= 1) kd[r] += __shfl_xor_sync(0xffffffffu, kd[r], sh);
    }
  }
#pragma unroll
  for (int r = 0; r < N; ++r) {
    const Of G(a, u[r] != EMPTY ? u[r] : 0u);
    float bg = 0.f;
    uint32_t bc = EMPTY;
    if ((lead >> r) & 1u) {
      const float g = gain_of(float(kc[r]), float(kd[r]), wu[r], rounded(wu[r]), tc[r], td[r], G.kr);
      if (g > 0.f) { bg = g; bc = c[r]; }
    }
    for (uint32_t sh = T >> 1; sh; sh >>= 1) {
      const float og = __shfl_xor_sync(0xffffffffu, bg, sh);
      const uint32_t oc = __shfl_xor_sync(0xffffffffu, bc, sh);
      if (better(og, oc, bg, bc)) { bg = og; bc = oc; }
    }
    const bool moved = bc != EMPTY && bc != G.zero;
    if (u[r] != EMPTY && tl == 0) {
      if (bc != EMPTY) add_gain(a, fix, G, bg);
      if (moved) commit<SYNC>(a, S, mv, u[r], d[r], bc);
      atomicAdd(&S.edges[bin], dg[r]);
    }
    if constexpr (!SYNC) {
      if (moved && v[r] != u[r]) a.vaff[v[r]] = 1;
      if (u[r] != EMPTY && tl == 0) a.vaff[u[r]] = 0;
    }
  }
}

// Sum the weights of the neighbours row[0..m) of u per community into a table
// of 2^lg slots by the n threads of a group (thread t); those in u's own
// community d are summed in the return value (each thread its share).
template <bool SYNC, int MODE>
__device__ __forceinline__ Sum<MODE> scan_row(const PhaseArgs &a, Shared &S, uint32_t u, uint64_t o, uint32_t m,
                                              uint32_t d, uint32_t t, uint32_t n, uint32_t *keys, uint32_t *vals,
                                              uint32_t lg) {
  using V = Sum<MODE>;
  const int lane = threadIdx.x & 31;
  V kd = 0;
  bool fine = true;
  constexpr int U = 4;  // edges of a lane in flight
  for (uint32_t base = t - lane; base < m; base += U * n) {
    uint32_t v[U], c[U];
    V w[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const uint32_t j = base + k * n + lane;
      v[k] = j < m ? __ldcs(a.key + o + j) : u;
      w[k] = j < m ? weight<MODE>(a, o + j) : V(0);
    }
#pragma unroll
    for (int k = 0; k < U; ++k) c[k] = v[k] != u ? live<SYNC>(a.vcom + v[k]) : EMPTY;
#pragma unroll
    for (int k = 0; k < U; ++k) {
      if (c[k] == d) { kd += w[k]; c[k] = EMPTY; }
      if constexpr ((MODE & 3) == FLOATS)
        fine &= ORDERED<SYNC, MODE> && n == 32 ? add_ordered(keys, vals, lg, c[k], w[k], lane)
                                               : add_warp(keys, vals, lg, c[k], w[k], lane);
      else if (c[k] != EMPTY) fine &= add<V>(keys, vals, lg, c[k], (MODE & 3) == UNIT ? 1u : w[k]);
    }
  }
  if (!fine) S.bad = 1;  // (a table has twice as many slots as neighbours)
  return kd;
}

// The group's best of its threads' moves (gain bg, community bc): the largest
// gain (positive, so its bits order as the floats), then the lowest id.
__device__ __forceinline__ void group_best(Shared &S, float bg, uint32_t n, uint32_t id, int w0, uint32_t &gb,
                                           uint32_t &bc) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  gb = __reduce_max_sync(0xffffffffu, __float_as_uint(bg));
  bc = __reduce_min_sync(0xffffffffu, __float_as_uint(bg) == gb ? bc : EMPTY);
  if (n > 32) {
    if (lane == 0) { S.redg[wid] = gb; S.redc[wid] = bc; }
    group_sync(id, n);
    gb = 0;
    bc = EMPTY;
    for (uint32_t k = 0; k < (n >> 5); ++k) {
      const uint32_t og = S.redg[w0 + k], oc = S.redc[w0 + k];
      if (og > gb || (og == gb && oc < bc)) { gb = og; bc = oc; }
    }
  } else {
    __syncwarp();
  }
}

// The best move of u over the communities of a table (kd: the weight to its
// own community), by the n threads of a group whose first warp is w0. Four
// slots of a thread in flight: their communities' totals are gathers.
template <bool SYNC, int MODE>
__device__ __forceinline__ void best_of_table(const PhaseArgs &a, Shared &S, const uint32_t *keys, const uint32_t *vals,
                                              uint32_t slots, uint32_t t, uint32_t n, uint32_t id, int w0, float kd,
                                              Tot<MODE> wu, Tot<MODE> td, float kr, uint32_t &gb, uint32_t &bc) {
  const float wuf = rounded(wu);
  float bg = 0.f;
  bc = EMPTY;
  constexpr int U = 4;
  for (uint32_t s = t; s < slots; s += U * n) {
    uint32_t c[U];
    Tot<MODE> tc[U];
#pragma unroll
    for (int k = 0; k < U; ++k) c[k] = s + k * n < slots ? keys[s + k * n] : EMPTY;
#pragma unroll
    for (int k = 0; k < U; ++k) tc[k] = total<MODE>(c[k] != EMPTY ? live<SYNC>(a.ctot + c[k]) : 0.0);
#pragma unroll
    for (int k = 0; k < U; ++k) {
      if (c[k] == EMPTY) continue;
      const float kc = float(of_bits<MODE>(vals[s + k * n]));
      const float g = gain_of(kc, kd, wu, wuf, tc[k], td, kr);
      if (g > 0.f && better(g, c[k], bg, bc)) { bg = g; bc = c[k]; }
    }
  }
  group_best(S, bg, n, id, w0, gb, bc);
}
// One vertex by the n threads (1, 4, 8 or 32 warps, thread t) of a group, with
// a table of twice its degree (at most 2^lgmax slots).
template <bool SYNC, int MODE>
__device__ __forceinline__ void group_vertex(const PhaseArgs &a, Shared &S, uint2 *mv, uint32_t u, uint32_t t,
                                             uint32_t n, uint32_t id, uint32_t *table, uint32_t lgmax, int bin,
                                             unsigned long long &fix) {
  using V = Sum<MODE>;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int w0 = wid - int(t >> 5);  // the group's first warp
  const uint64_t o = a.off[u];
  const uint32_t dg = a.deg[u];
  const uint32_t d = a.vcom[u];
  const Tot<MODE> wu = total<MODE>(a.vtot[u]), td = total<MODE>(live<SYNC>(a.ctot + d));
  const Of G(a, u);
  const uint32_t lg = min(lgmax, uint32_t(ceil_log2(2ull * dg)));
  uint32_t *keys = table, *vals = table + (1u << lg);
  for (uint32_t s = t; s < (1u << lg); s += n) { keys[s] = EMPTY; vals[s] = 0u; }
  group_sync(id, n);
  V kd = warp_sum<V>(scan_row<SYNC, MODE>(a, S, u, o, dg, d, t, n, keys, vals, lg));
  if (lane == 0) S.redk[wid] = bits(kd);
  group_sync(id, n);  // the table and the sums are complete
  kd = 0;
  for (uint32_t k = 0; k < (n >> 5); ++k) kd += of_bits<MODE>(S.redk[w0 + k]);
  uint32_t gb, bc;
  best_of_table<SYNC, MODE>(a, S, keys, vals, 1u << lg, t, n, id, w0, float(kd), wu, td, G.kr, gb, bc);
  const bool moved = bc != EMPTY && bc != G.zero;
  if (t == 0) {
    if (bc != EMPTY) add_gain(a, fix, G, __uint_as_float(gb));
    if (moved) {
      if (SHARES<SYNC, MODE> && bin >= 9) {  // its row is marked in pieces, by whichever blocks
        const uint32_t n = (dg + PIECE - 1) / PIECE, at = atomicAdd(&a.ctl->pieces[S.turn], n);
        for (uint32_t p = 0; p < n; ++p) a.big[at + p] = make_uint4(u, d, bc, p);
        atomicAdd(&S.hubmv, 1u);
      } else {
        commit<SYNC>(a, S, mv, u, d, bc);
      }
    }
    atomicAdd(&S.edges[bin], dg);
  }
  if constexpr (!SYNC) {
    if (moved) mark_row(a, u, o, dg, t, n);
    if (t == 0) a.vaff[u] = 0;
  }
}

// Hub h of the plan by the n threads of a group from its resident table, which
// describes the state of the class's start: the community it goes to into
// hub_move (EMPTY: it stays, or is not active) and the one it leaves into
// hub_from. A hub whose table is bad is left to its chunks. 256 threads a hub:
// a table has 64 to 65536 slots, and a class a hub or two for each block; what
// it costs is the chain of loads, not the slots. The tables are brought up to
// date where the movers' neighbours are marked (mark_row), which looks at those
// rows anyway; as a kernel of its own per class it took 156 us, reading every
// vertex's decision.
__device__ __forceinline__ bool table_good(const PhaseArgs &a, uint32_t u) {
  const uint32_t h = a.ht.key ? a.ht.slot[u] : NO_HUB;
  return h != NO_HUB && !a.ht.bad[h];
}

__device__ __forceinline__ void table_hub(const PhaseArgs &a, Shared &S, uint32_t h, uint32_t t, uint32_t n,
                                          uint32_t id, unsigned long long &fix, unsigned long long &slots) {
  const int w0 = int(threadIdx.x >> 5) - int(t >> 5);
  const uint32_t u = a.hub_vertex[h], ti = a.ht.slot[u];
  if (ti == NO_HUB || a.ht.bad[ti]) return;
  if (!a.vaff[u] || (a.fa && !a.fa[u])) {
    if (t == 0) a.hub_move[h] = EMPTY;
    return;
  }
  const uint64_t o = a.ht.off[ti];
  const int lg = a.ht.lg[ti];
  const uint32_t m = 1u << lg, d = a.vcom[u];
  const uint32_t *keys = a.ht.key + o, *cnt = a.ht.cnt + o;
  const double wu = a.vtot[u], td = a.ctot[d];
  const float wuf = __double2float_rn(wu);
  float kd = 0.f;
  for (uint32_t s = hash_hi(d, lg), p = 0; p < m; ++p, s = (s + 1u) & (m - 1u)) {
    const uint32_t c = keys[s];
    if (c == d) kd = float(cnt[s]);
    if (c == d || c == EMPTY) break;
  }
  float bg = 0.f;
  uint32_t bc = EMPTY, gb;
  constexpr int U = 4;
  for (uint32_t s = t; s < m; s += U * n) {
    uint32_t c[U], k[U];
    double tc[U];
#pragma unroll
    for (int x = 0; x < U; ++x) c[x] = s + x * n < m ? keys[s + x * n] : EMPTY;
#pragma unroll
    for (int x = 0; x < U; ++x) {
      if (c[x] == d) c[x] = EMPTY;
      k[x] = c[x] != EMPTY ? cnt[s + x * n] : 0u;
      tc[x] = c[x] != EMPTY ? a.ctot[c[x]] : 0.0;
    }
#pragma unroll
    for (int x = 0; x < U; ++x) {
      if (!k[x]) continue;
      const float g = gain_of(float(k[x]), kd, wu, wuf, tc[x], td, a.kr);
      if (g > 0.f && better(g, c[x], bg, bc)) { bg = g; bc = c[x]; }
    }
  }
  group_best(S, bg, n, id, w0, gb, bc);
  if (t == 0) {
    const bool moved = bc != EMPTY && bc != 0u;  // (community 0 is never a target)
    if (bc != EMPTY) fix += gain_to_fix(__uint_as_float(gb));
    a.hub_move[h] = moved ? bc : EMPTY;
    a.hub_from[h] = d;
    a.vaff[u] = 0;
    atomicAdd(&S.cnt[NUM_BINS - 1], 1u);
    if (moved) atomicAdd(&S.hubmv, 1u);
    slots += m;
  }
  group_sync(id, n);  // (the group's sums are read until here)
}

// ---- hubs (degree above 8192), in two steps with a grid barrier between.
// Step 1, a block per chunk of a hub's edges: the chunk's communities are
// counted in the block's table and written out as (community, weight) pairs,
// grouped by the hub's `parts` hash partitions of the communities (segs: the
// groups' bounds), so that step 2 splits a hub of many communities over
// blocks. chunk_cnt is EMPTY for a hub that is not active.
__device__ __forceinline__ bool hub_active(const PhaseArgs &a, uint32_t u) {
  return a.vaff[u] && (!a.fa || a.fa[u]) && (!a.gact || a.gact[a.gid[u]]) && !table_good(a, u);
}

template <bool SYNC, int MODE>
__device__ __forceinline__ void hub_chunk(const PhaseArgs &a, Shared &S, uint32_t ci, uint32_t *table) {
  using V = Sum<MODE>;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint4 ch = a.chunk[ci];
  const uint32_t u = ch.w, h = ch.x;
  if (threadIdx.x == 0) {
    S.over = hub_active(a, u);
    S.next = 0;
  }
  __syncthreads();
  if (!S.over) {  // (block-uniform)
    __syncthreads();
    if (threadIdx.x == 0) a.chunk_cnt[ci] = EMPTY;
    return;
  }
  const uint32_t m = ch.z - ch.y, d = a.vcom[u];
  const uint32_t lg = max(1u, uint32_t(ceil_log2(2ull * m))), slots = 1u << lg;
  uint32_t *keys = table, *vals = table + slots, *pc = table + 2 * slots;
  const uint32_t R = a.hub_parts[h];
  for (uint32_t s = threadIdx.x; s < slots; s += PB) { keys[s] = EMPTY; vals[s] = 0u; }
  for (uint32_t r = threadIdx.x; r < R; r += PB) pc[r] = 0;
  __syncthreads();
  const V kd = warp_sum<V>(scan_row<SYNC, MODE>(a, S, u, a.off[u] + ch.y, m, d, threadIdx.x, PB, keys, vals, lg));
  if (lane == 0) S.redk[wid] = bits(kd);
  __syncthreads();
  uint32_t *pk = a.part_key + a.chunk_part[ci];
  uint32_t *pv = a.part_val + a.chunk_part[ci];
  // (lanes of one partition take their places together: the counters are few
  // and hot)
  if (R > 1) {
    for (uint32_t s = threadIdx.x; s - lane < slots; s += PB) {
      const uint32_t c = s < slots ? keys[s] : EMPTY;
      const uint32_t r = c != EMPTY ? hub_part(c, R) : EMPTY;
      const unsigned grp = __match_any_sync(0xffffffffu, r);
      if (r != EMPTY && (grp & ((1u << lane) - 1u)) == 0u) atomicAdd(&pc[r], uint32_t(__popc(grp)));
    }
    __syncthreads();
    uint32_t *seg = a.segs + a.seg_off[h] + size_t(ci - a.hub_first[h]) * (R + 1);
    if (wid == 0) {  // exclusive prefix of the partitions' counts
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
      if (lane == 0) { seg[R] = carry; S.next = carry; }
    }
    __syncthreads();
  }
  for (uint32_t s = threadIdx.x; s - lane < slots; s += PB) {
    const uint32_t c = s < slots ? keys[s] : EMPTY;
    const uint32_t r = c == EMPTY ? EMPTY : R > 1 ? hub_part(c, R) : 0u;
    const unsigned grp = __match_any_sync(0xffffffffu, r);
    const int leader = __ffs(grp) - 1;
    uint32_t at = 0;
    if (r != EMPTY && lane == leader) at = atomicAdd(R > 1 ? &pc[r] : &S.next, uint32_t(__popc(grp)));
    at = __shfl_sync(0xffffffffu, at, leader) + __popc(grp & ((1u << lane) - 1u));
    if (r != EMPTY) { pk[at] = c; pv[at] = vals[s]; }
  }
  if (threadIdx.x == 0) {
    V k = 0;
    for (int x = 0; x < PW; ++x) k += of_bits<MODE>(S.redk[x]);
    if (k != V(0)) atomicAdd(reinterpret_cast<V *>(&a.hub_kd[u]), k);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    a.chunk_cnt[ci] = S.next;
    S.next = 0;
  }
}

// Step 2, a block per (hub, partition): the partition's pairs of all chunks
// are merged in the block's table and its best move goes to hub_best; the
// block that completes the hub takes its decision (hub_move: the community it
// goes to, EMPTY if it stays). A hub whose pairs all fit one table is merged
// by the block of partition 0 alone. A hub that was marked while its chunks
// ran (asynchronous mode: some chunks skipped it) waits for the next
// iteration.
template <bool SYNC, int MODE>
__device__ __forceinline__ void hub_merge(const PhaseArgs &a, Shared &S, uint2 task, uint32_t *table,
                                          unsigned long long &fix) {
  using V = Sum<MODE>;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t h = task.x, r = task.y, R = a.hub_parts[h];
  const uint32_t u = a.hub_vertex[h];
  if (table_good(a, u)) return;  // (decided from its table; block-uniform)
  const uint32_t c0 = a.hub_first[h], nc = a.hub_first[h + 1] - c0;
  if (threadIdx.x == 0) { S.next = 0; S.over = 0; }
  __syncthreads();
  {
    uint32_t sum = 0;
    bool stale = false;
    for (uint32_t c = threadIdx.x; c < nc; c += PB) {
      const uint32_t x = a.chunk_cnt[c0 + c];
      stale |= x == EMPTY;
      sum += x == EMPTY ? 0u : x;
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0 && sum) atomicAdd(&S.next, sum);
    if (stale) S.over = 1;
  }
  __syncthreads();
  const uint32_t P = S.next;
  const bool stale = S.over != 0, single = R == 1 || P <= MERGE_FULL;
  __syncthreads();
  if (stale || (single && r > 0)) {  // (block-uniform)
    if (stale && r == 0 && threadIdx.x == 0) {
      a.hub_move[h] = EMPTY;
      a.hub_kd[u] = 0.f;
    }
    if (threadIdx.x == 0) S.next = 0;
    return;
  }
  const uint32_t lg = single ? max(1u, uint32_t(ceil_log2(2ull * P))) : LOG_BLOCK, slots = 1u << lg;
  uint32_t *keys = table, *vals = table + slots;
  for (uint32_t s = threadIdx.x; s < slots; s += PB) { keys[s] = EMPTY; vals[s] = 0u; }
  const uint32_t d = a.vcom[u];
  const Tot<MODE> wu = total<MODE>(a.vtot[u]), td = total<MODE>(live<SYNC>(a.ctot + d));
  const V kd = of_bits<MODE>(__float_as_uint(a.hub_kd[u]));
  const Of G(a, u);
  __syncthreads();
  bool fine = true;
  // a warp per (chunk, piece of its pairs): 128 pairs at a time, `pieces`
  // warps to a chunk (as many as its pairs are likely to need)
  const uint32_t pieces = single ? min(32u, max(1u, P / (nc * 128u) + 1)) : min(32u, 32u / R + 1);
  for (uint32_t x = wid; x < nc * pieces; x += PW) {
    const uint32_t c = x / pieces, piece = x - c * pieces;
    const uint64_t p = a.chunk_part[c0 + c];
    uint32_t b = 0, e = 0;
    if (single) {
      e = a.chunk_cnt[c0 + c];
    } else {
      const uint32_t *seg = a.segs + a.seg_off[h] + size_t(c) * (R + 1);
      b = seg[r];
      e = seg[r + 1];
    }
    for (uint32_t q = b + piece * 128u + lane; q - lane < e; q += pieces * 128u) {
      uint32_t k4[4], v4[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool in = q + 32 * k < e;
        k4[k] = in ? a.part_key[p + q + 32 * k] : EMPTY;
        v4[k] = in ? a.part_val[p + q + 32 * k] : 0u;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k4[k] != EMPTY) fine &= add<V>(keys, vals, lg, k4[k], of_bits<MODE>(v4[k]));
    }
  }
  if (!fine) S.bad = 1;
  __syncthreads();
  uint32_t gb, bc;
  best_of_table<SYNC, MODE>(a, S, keys, vals, slots, threadIdx.x, PB, 0, 0, float(kd), wu, td, G.kr, gb, bc);
  if (threadIdx.x == 0) {
    bool last = true;
    if (!single) {
      if (bc != EMPTY) atomicMax(&a.hub_best[h], (static_cast<unsigned long long>(gb) << 32) | (0xFFFFFFFFu - bc));
      __threadfence();
      last = atomicAdd(&a.hub_done[h], 1u) == R - 1;
      if (last) {
        __threadfence();
        const unsigned long long best = atomicExch(&a.hub_best[h], 0ull);
        gb = uint32_t(best >> 32);
        bc = best ? 0xFFFFFFFFu - uint32_t(best) : EMPTY;
        a.hub_done[h] = 0;
      }
    }
    if (last) {
      const bool moved = bc != EMPTY && bc != G.zero;
      if (bc != EMPTY) add_gain(a, fix, G, __uint_as_float(gb));
      a.hub_move[h] = moved ? bc : EMPTY;
      a.hub_kd[u] = 0.f;
      a.vaff[u] = 0;
      S.cnt[NUM_BINS - 1] += 1;
      S.edges[NUM_BINS - 1] += a.deg[u];
      if (moved) {
        S.hubmv += 1;
        if constexpr (SYNC) {
          a.hub_from[h] = d;
        } else {
          const double x = a.vtot[u];
          atomicAdd(&a.ctot[d], -x);
          atomicAdd(&a.ctot[bc], x);
          a.vcom[u] = bc;
        }
      }
    }
    S.next = 0;
  }
}

// log2 of the vertices a block takes of a bin at a time (dealt in turn).
__host__ __device__ constexpr uint32_t chunk_log(int b) { return b <= 2 ? 5 : b == 3 ? 4 : b == 4 ? 3 : b <= 6 ? 2 : 0; }

template <bool SYNC, int MODE>
__global__ void __launch_bounds__(PB, 1) phase_kernel(const __grid_constant__ PhaseArgs a) {
  extern __shared__ __align__(16) uint32_t table[];  // TABLE_WORDS, then the moves, then the list
  __shared__ Shared S;
  const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const uint32_t G = gridDim.x, bid = blockIdx.x;
  const int K = a.colors;
  const bool in_smem = a.cap <= LIST_CAP;
  uint2 *mv = in_smem ? reinterpret_cast<uint2 *>(table + TABLE_WORDS) : a.gmv + size_t(bid) * a.cap;
  uint32_t *list = in_smem ? table + TABLE_WORDS + 2 * LIST_CAP : a.glist + size_t(bid) * a.cap;
  // the block's share of every class: bins in descending order, the chunks of
  // all of them dealt to the blocks in turn
  for (int k = int(tid); k < K; k += PB) {
    uint32_t q = 0, items = 0;  // chunks of the bins before, the block's list slots of them
    for (int b = NUM_BINS - 2; b >= 1; --b) {
      const uint32_t n = a.start[k * NUM_BINS + b + 1] - a.start[k * NUM_BINS + b];
      const uint32_t chunks = (n + (1u << chunk_log(b)) - 1) >> chunk_log(b);
      const uint32_t r = q % G;
      const uint32_t first = bid >= r ? bid - r : bid + G - r;  // the block's first chunk of the bin
      S.off[k * NUM_BINS + b] = items;
      S.pos[k * NUM_BINS + b] = first << chunk_log(b);
      if (first < chunks) items += ((chunks - first + G - 1) / G) << chunk_log(b);
      q += chunks;
    }
    S.tot[k] = items;
  }
  if (tid < NUM_BINS) { S.sv[tid] = 0; S.se[tid] = 0; S.edges[tid] = 0; S.cnt[tid] = 0; }
  if (tid == 0) { S.moves = 0; S.nmv = 0; S.nbig = 0; S.hubmv = 0; S.bad = 0; S.stop = 0; S.next = 0; }
  __syncthreads();
  uint32_t nbar = 0;  // barriers so far
  double el = 0.0;
  unsigned long long fix = 0;  // the thread's share of the iteration's gain sum
  unsigned long long sum = 0, slots = 0;
  const bool tabs = SYNC && MODE == UNIT && a.ht.key;  // the hubs are decided from resident tables
  constexpr bool SHARE = SHARES<SYNC, MODE>;
  uint32_t l = 0, step = 0;
  while (l < uint32_t(a.L)) {
    // what ends an iteration: its gain sum, or the graphs of the union still moving
    const unsigned long long *total = a.gfix ? &a.ctl->gactive[l % 3] : &a.ctl->fix[l % 3];
    for (int k = 0; k < K; ++k) {
      const bool last = k == K - 1;
      // ---- 1. the block's active vertices of the class, per bin
      const uint32_t turn = SHARE ? step++ % 3 : 0u;
      const bool shared = SHARE && a.heavy;  // bins 9 and 10 through a list of all blocks
      if (SHARE && tid == 0) S.turn = turn;
      const uint32_t tot = S.tot[k];
      const uint32_t *off = S.off + k * NUM_BINS;
      for (uint32_t t0 = tid - lane; t0 < tot; t0 += PB) {
        const uint32_t t = t0 + lane;
        int b = -1;
        uint32_t u = 0, rank = 0;
        if (t < tot) {
          b = 1;
#pragma unroll
          for (int x = 2; x < NUM_BINS - 1; ++x)
            if (t < off[x - 1]) b = x;
          const uint32_t j = t - off[b], lgc = chunk_log(b);
          const uint32_t p = S.pos[k * NUM_BINS + b] + (((j >> lgc) * G) << lgc) + (j & ((1u << lgc) - 1u));
          const uint32_t s0 = a.start[k * NUM_BINS + b];
          if (p < a.start[k * NUM_BINS + b + 1] - s0) {
            u = a.bins[s0 + p];
            if (!a.vaff[u] || (a.fa && !a.fa[u]) || (a.gact && !a.gact[a.gid[u]])) b = -1;
            else if (SYNC) a.vaff[u] = 0;  // (marks of this class come after every block has decided)
          } else {
            b = -1;
          }
        }
        const unsigned grp = __match_any_sync(0xffffffffu, b);
        const int leader = __ffs(grp) - 1;
        if (b >= 0 && int(lane) == leader) rank = atomicAdd(&S.cnt[b], uint32_t(__popc(grp)));
        rank = __shfl_sync(0xffffffffu, rank, leader);
        if (shared) {
          uint32_t at = 0;
          if (b >= 9 && int(lane) == leader) at = atomicAdd(&a.ctl->heavy[turn][10 - b], uint32_t(__popc(grp)));
          at = __shfl_sync(0xffffffffu, at, leader);
          if (b >= 9) a.heavy[(b == 9 ? a.heavy9 : 0u) + at + __popc(grp & ((1u << lane) - 1u))] = u;
        }
        if (b >= 0 && !(shared && b >= 9)) list[off[b] + rank + __popc(grp & ((1u << lane) - 1u))] = u;
      }
      __syncthreads();
      // ---- 2. decide them
      const uint32_t ch0 = a.chunk_begin[k], nch = a.chunk_begin[k + 1] - ch0;
      // the block's chunks of the class that pred holds for, to work(); 256 are
      // asked at once: most are of hubs with nothing to do, and one after the
      // other each would cost the latency of two loads. (From the last block:
      // the first ones have the heaviest lists.)
      auto each_chunk = [&](auto pred, auto work) {
        for (uint32_t t0 = G - 1 - bid; t0 < nch; t0 += TODO * G) {
          if (tid == 0) S.ntodo = 0;
          __syncthreads();
          const uint32_t t = t0 + tid * G;
          if (tid < TODO && t < nch && pred(t)) S.todo[atomicAdd(&S.ntodo, 1u)] = t;
          __syncthreads();
          const uint32_t n = S.ntodo;
          for (uint32_t i = 0; i < n; ++i) {
            work(S.todo[i]);
            __syncthreads();
          }
          __syncthreads();
        }
      };
      bool scan = nch != 0;  // some hub of the class is counted from its edges
      if constexpr (SYNC && MODE == UNIT) {
        if (tabs && nch) {
          scan = ld_relaxed(a.ht.nbad) != 0;  // (raised between decisions only: the same for every block)
          const uint32_t g = wid >> 3, h1 = a.hub_begin[k + 1];
          for (uint32_t h = a.hub_begin[k] + (G - 1 - bid) * 4 + g; h < h1; h += G * 4)
            table_hub(a, S, h, tid & 255u, 256, 9 + g, fix, slots);
          __syncthreads();
        }
      }
      if (scan)
        each_chunk(
            [&](uint32_t t) {
              const bool act = hub_active(a, a.chunk[ch0 + t].w);
              if (!act) a.chunk_cnt[ch0 + t] = EMPTY;
              return act;
            },
            [&](uint32_t t) { hub_chunk<SYNC, MODE>(a, S, ch0 + t, table); });
      auto blocks = [&] {  // degree above 512: the whole block, then eight warps each
        const uint32_t c10 = S.cnt[10], c9 = S.cnt[9];
        for (uint32_t i = 0; i < c10; ++i) {
          group_vertex<SYNC, MODE>(a, S, mv, list[off[10] + i], tid, PB, 0, table, LOG_BLOCK, 10, fix);
          __syncthreads();
        }
        if (c9) {
          const uint32_t g = wid >> 3;
          for (uint32_t i = g; i < c9; i += 4)
            group_vertex<SYNC, MODE>(a, S, mv, list[off[9] + i], tid & 255u, 256, 9 + g, table + g * 8192u, 12, 9, fix);
          __syncthreads();
        }
      };
      auto fours = [&] {  // degree 129-512, tables in the first half of the area
        const uint32_t c8 = S.cnt[8], c7 = S.cnt[7];
        if constexpr (ORDERED<SYNC, MODE>) {  // a warp each, tables in the whole area
          if (wid < PW / 2)
            for (uint32_t i = wid; i < c8; i += PW / 2)
              group_vertex<SYNC, MODE>(a, S, mv, list[off[8] + i], lane, 32, 0, table + wid * 2048u, 10, 8, fix);
          __syncthreads();
          for (uint32_t i = wid; i < c7; i += PW)
            group_vertex<SYNC, MODE>(a, S, mv, list[off[7] + i], lane, 32, 0, table + wid * 1024u, 9, 7, fix);
          __syncthreads();
          return;
        }
        for (uint32_t i = wid >> 2; i < c8 + c7; i += PW / 4) {
          const int b = i < c8 ? 8 : 7;
          const uint32_t u = i < c8 ? list[off[8] + i] : list[off[7] + i - c8];
          group_vertex<SYNC, MODE>(a, S, mv, u, tid & 127u, 128, 1 + (wid >> 2), table + (wid >> 2) * 2048u, 10, b, fix);
        }
      };
      // warp-sized units, by whichever warp is free: degree 33-128 (tables in
      // the second half), then tiles
      auto units = [&] {
        constexpr uint32_t N = TILE_ROUNDS;
        const uint32_t n6 = S.cnt[6], n5 = n6 + S.cnt[5], n4 = n5 + (S.cnt[4] + N - 1) / N,
                       n3 = n4 + (S.cnt[3] + 2 * N - 1) / (2 * N), n2 = n3 + (S.cnt[2] + 4 * N - 1) / (4 * N),
                       n1 = n2 + (S.cnt[1] + 8 * N - 1) / (8 * N);
        for (;;) {
          uint32_t x = 0;
          if (lane == 0) x = atomicAdd(&S.next, 1u);
          x = __shfl_sync(0xffffffffu, x, 0);
          if (x >= n1) break;
          if (x < n5) {
            const int b = x < n6 ? 6 : 5;
            const uint32_t u = x < n6 ? list[off[6] + x] : list[off[5] + x - n6];
            group_vertex<SYNC, MODE>(a, S, mv, u, lane, 32, 0, table + TABLE_WORDS / 2 + wid * 512u, 8, b, fix);
          } else {
            const int b = x < n4 ? 4 : x < n3 ? 3 : x < n2 ? 2 : 1;
            const uint32_t x0 = x < n4 ? n5 : x < n3 ? n4 : x < n2 ? n3 : n2;
            const uint32_t T = 2u << b;
            tile_vertices<SYNC, MODE>(a, S, mv, list + off[b], (x - x0) * (N * 32 / T), S.cnt[b], T, b, fix);
          }
        }
      };
      if constexpr (SYNC) {  // the order changes nothing but the time: long work first
        if (!shared) blocks();
        fours();
        units();
      } else {
        // light vertices first: they see a class's heavy moves an iteration
        // later and the heavy ones see theirs at once, as in the reference's
        // sweep most vertices do. (Static runs of R-MAT scale 24, this level
        // alone asynchronous: modularity 0.0602 on average of 8 and 0.0594 at
        // worst; every level so 0.0594 and 0.0576, the launches 0.0596 and
        // 0.0584; on another graph of the scale heavy first and totals through
        // L1 0.0586 on average of 65, light first and past L1 0.0598.)
        units();
        fours();
        __syncthreads();
        blocks();
      }
      __syncthreads();
      if (scan || shared) {  // (the same for every block)
        if (tid == 0) S.next = 0;
        if (!grid_barrier(a, S, nbar++, 0, nullptr)) return;
      }
      if (scan) {
        const uint32_t m0 = a.merge_begin[k], m1 = a.merge_begin[k + 1];
        for (uint32_t t = m0 + bid; t < m1; t += G) {
          hub_merge<SYNC, MODE>(a, S, a.merge[t], table, fix);
          __syncthreads();
        }
      }
      if (shared) {
        // the class's listed vertices of bin 10, one to a block at a time, and
        // of bin 9, four (the next unit is fetched while one is decided)
        const uint32_t n10 = __ldcg(&a.ctl->heavy[turn][0]), n9 = __ldcg(&a.ctl->heavy[turn][1]);
        const uint32_t nu = n10 + (n9 + 3) / 4, g = wid >> 3;
        uint32_t x = bid;
        for (uint32_t r = 0; x < nu; ++r) {
          if (tid == 0) S.unit[r & 1] = G + atomicAdd(&a.ctl->queue[turn], 1u);
          if (x < n10) {
            group_vertex<SYNC, MODE>(a, S, mv, __ldcg(a.heavy + x), tid, PB, 0, table, LOG_BLOCK, 10, fix);
          } else if ((x - n10) * 4 + g < n9) {
            group_vertex<SYNC, MODE>(a, S, mv, __ldcg(a.heavy + a.heavy9 + (x - n10) * 4 + g), tid & 255u, 256, 9 + g,
                                     table + g * 8192u, 12, 9, fix);
          }
          __syncthreads();
          x = S.unit[r & 1];
        }
        __syncthreads();
      }
      const uint32_t nmv = S.nmv, moves = nmv + S.hubmv;
      if (tid == 0) {
        S.next = 0;
        if (SHARE && a.big && bid == 0) {  // (last used two steps ago)
          const uint32_t t = (turn + 1) % 3;
          a.ctl->pieces[t] = 0; a.ctl->heavy[t][0] = 0; a.ctl->heavy[t][1] = 0; a.ctl->queue[t] = 0;
        }
        S.moves += moves;
        if (last && bid == 0) { a.ctl->fix[(l + 1) % 3] = 0; a.ctl->gactive[(l + 1) % 3] = 0; }
      }
      if (last && !a.gfix) {
#pragma unroll
        for (int sh = 16; sh > 0; sh >>= 1) fix += __shfl_xor_sync(0xffffffffu, fix, sh);
        if (lane == 0 && fix) atomicAdd(&a.ctl->fix[l % 3], fix);
        fix = 0;
      }
      if (tid < NUM_BINS) {
        S.sv[tid] += S.cnt[tid];
        S.cnt[tid] = 0;
        if (last) { S.se[tid] += S.edges[tid]; S.edges[tid] = 0; }
      }
      if (!grid_barrier(a, S, nbar++, moves, last ? total : nullptr)) return;
      const bool any = S.any != 0;  // some block moved a vertex (the same for every block)
      // ---- 3. commit the decisions, mark the movers' neighbours
      if constexpr (SYNC) {
        if (any) {
          // Eight lanes per move, longer rows by 256 threads; where the blocks
          // share, by a warp, and those of degree bins 9 and 10 in pieces. With
          // few moves a row is long above 32 entries there: eight lanes take
          // eight rounds for one of 256, each with up to four hub tables to
          // update one after the other, and the block that had one kept the
          // others waiting (40 us a class of a 1e-4 |E| batch on R-MAT scale
          // 24).
          uint32_t *big = table;  // (vertex, its old and new community)
          constexpr uint32_t BIG_CAP = TABLE_WORDS / 3;
          const uint32_t wide = SHARE && nmv <= 8 * PW ? 32u : 256u;
          const bool cut = SHARE && a.big && a.start[k * NUM_BINS + NUM_BINS - 1] > a.start[k * NUM_BINS + 9];
          const uint32_t np = cut ? __ldcg(&a.ctl->pieces[turn]) : 0u;
          const uint32_t sl = tid & 7u;
          for (uint32_t i = tid >> 3; i < nmv; i += PB / 8) {
            const uint2 m = mv[i];
            const uint64_t o = a.off[m.x];
            const uint32_t dg = a.deg[m.x];
            uint32_t d = 0, late = 0;
            if (sl == 0) {
              d = a.vcom[m.x];
              const double wu = a.vtot[m.x];
              atomicAdd(&a.ctot[d], -wu);
              atomicAdd(&a.ctot[m.y], wu);
              a.vcom[m.x] = m.y;
              if (dg > wide) {
                const uint32_t j = atomicAdd(&S.nbig, 1u);
                if (j < BIG_CAP) {
                  big[3 * j] = m.x;
                  big[3 * j + 1] = d;
                  big[3 * j + 2] = m.y;
                  late = 1;
                }
              }
            }
            d = __shfl_sync(0xffu << (lane & 24u), d, 0, 8);
            if (!__shfl_sync(0xffu << (lane & 24u), late, 0, 8)) mark_row(a, m.x, o, dg, sl, 8, tabs, d, m.y);
          }
          __syncthreads();
          const uint32_t nbig = min(S.nbig, BIG_CAP);
          for (uint32_t i = SHARE ? wid : wid >> 3; i < nbig; i += SHARE ? PW : PW / 8) {
            const uint32_t u = big[3 * i];
            if constexpr (SHARE) mark_row_warp(a, u, a.off[u], a.deg[u], lane, 32, tabs, big[3 * i + 1], big[3 * i + 2]);
            else mark_row(a, u, a.off[u], a.deg[u], tid & 255u, 256);
          }
          if constexpr (SHARE) {  // the pieces of the class's large movers, 256 threads each
            for (uint32_t i = bid * 4 + (wid >> 3); i < np; i += G * 4) {
              const uint4 e = __ldcg(a.big + i);
              const uint32_t dg = a.deg[e.x], p = e.w * PIECE;
              if (p == 0 && (tid & 255u) == 0) {
                const double wu = a.vtot[e.x];
                atomicAdd(&a.ctot[e.y], -wu);
                atomicAdd(&a.ctot[e.z], wu);
                a.vcom[e.x] = e.z;
              }
              mark_row_warp(a, e.x, a.off[e.x] + p, min(PIECE, dg - p), tid & 255u, 256, tabs, e.y, e.z);
            }
          }
          each_chunk([&](uint32_t t) { return a.hub_move[a.chunk[ch0 + t].x] != EMPTY; },  // the moved hubs' chunks
                     [&](uint32_t t) {
                       const uint4 ch = a.chunk[ch0 + t];
                       const uint32_t c = a.hub_move[ch.x], d = a.hub_from[ch.x], u = ch.w;
                       if (ch.y == 0 && tid == 0) {
                         const double wu = a.vtot[u];
                         atomicAdd(&a.ctot[d], -wu);
                         atomicAdd(&a.ctot[c], wu);
                         a.vcom[u] = c;
                       }
                       mark_row_warp(a, u, a.off[u] + ch.y, ch.z - ch.y, tid, PB, tabs, d, c);
                     });
        }
      } else {
        // the moved hubs' neighbours, by the blocks of their chunks
        each_chunk([&](uint32_t t) { return a.hub_move[a.chunk[ch0 + t].x] != EMPTY; },
                   [&](uint32_t t) {
                     const uint4 ch = a.chunk[ch0 + t];
                     mark_row(a, ch.w, a.off[ch.w] + ch.y, ch.z - ch.y, tid, PB);
                   });
      }
      if (last && a.gfix)  // graph unions: each graph's own stop test
        for (uint32_t i = bid * PB + tid; i < a.graphs; i += G * PB) phase_control(a, i, l % 3);
      __syncthreads();
      if (tid == 0) { S.nbig = 0; S.nmv = 0; S.hubmv = 0; }
      if ((SYNC && any) || (last && a.gfix)) {
        if (!grid_barrier(a, S, nbar++, 0, last && a.gfix ? total : nullptr)) return;
      } else {
        __syncthreads();
      }
    }
    // ---- the stop test (el <= E), the same value in every block
    sum = S.sum;
    __syncthreads();
    ++l;
    if (a.gfix) {
      if (sum == 0ull) break;
    } else {
      el = double(sum) / GAIN_FIX / a.M;
      if (el <= a.E) break;
    }
  }
  if (bid == 0 && tid == 0) {
    a.ctr->dev_iters = l;
    a.ctr->dev_el = el;
    if (a.gfix) a.ctr->gactive = uint32_t(sum);
  }
  if (tid < NUM_BINS && S.sv[tid]) {
    atomicAdd(&a.ctr->bin_vertices[tid], S.sv[tid]);
    atomicAdd(&a.ctr->bin_edges[tid], S.se[tid]);
  }
  if (SYNC && MODE == UNIT && slots) atomicAdd(&a.ctr->ht_slots, slots);
  if (tid == 0) {
    if (S.moves) atomicAdd(&a.ctr->moves, S.moves);
    if (S.bad) atomicOr(&a.ctr->err, ERR_TABLE_FULL);
  }
}

constexpr size_t SMEM = (size_t(TABLE_WORDS) + 3 * LIST_CAP) * sizeof(uint32_t);

// The device's blocks that can be resident at once, with the kernel's attribute
// set (0: the device launches none cooperatively).
template <bool SYNC, int MODE>
uint32_t most_blocks() {
  static PerDevice<uint32_t> most;
  return most.get([] {
    int dev = 0, coop = 0, per_sm = 0;
    LVG_CUDA(cudaGetDevice(&dev));
    LVG_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) return 0u;
    auto k = phase_kernel<SYNC, MODE>;
    LVG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(SMEM)));
    LVG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, PB, SMEM));
    return uint32_t(per_sm) * uint32_t(device_sms());
  });
}

template <bool SYNC, int MODE>
void launch(uint32_t grid, const PhaseArgs &a, cudaStream_t s) {
  void *args[] = {const_cast<PhaseArgs *>(&a)};
  LVG_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void *>(phase_kernel<SYNC, MODE>), dim3(grid), dim3(PB), args,
                                       SMEM, s));
  ++launch_counter();
}

// f(SYNC, MODE) of the kernel that serves a phase.
template <class F>
void variant(bool sync, bool unit, bool whole, bool totals, F f) {
  auto mode = [&](auto S) {
    const bool t = totals && (unit || whole);
    if (unit) t ? f(S, std::integral_constant<int, UNIT | TOTALS>()) : f(S, std::integral_constant<int, UNIT>());
    else if (whole) t ? f(S, std::integral_constant<int, WHOLE | TOTALS>()) : f(S, std::integral_constant<int, WHOLE>());
    else f(S, std::integral_constant<int, FLOATS>());
  };
  if (sync) mode(std::true_type());
  else mode(std::false_type());
}

}  // namespace

bool phase_lists_fit(uint32_t cap) { return cap <= LIST_CAP; }

// Enough blocks for the largest class's warps of work (a block's vertex
// counts 32 of them, a tile-sized one its share of a warp) to be about one per
// warp, at most those that are resident at once: fewer blocks make the barriers
// cheaper.
uint32_t phase_grid(const Level &lv, bool sync, bool unit, bool whole, bool totals) {
  uint32_t blocks = 0;
  variant(sync, unit, whole, totals, [&](auto S, auto M) { blocks = most_blocks<S.value, M.value>(); });
  if (!blocks) return 0;
  static const uint32_t share[NUM_BINS] = {0, 4, 8, 16, 32, 32, 32, 128, 128, 256, 1024, 1024};  // 1/32 warps
  uint64_t most = 0;
  for (int k = 0; k < lv.colors; ++k) {
    uint64_t units = 0;
    for (int b = 1; b < NUM_BINS - 1; ++b) units += uint64_t(lv.bucket_size(k, b)) * share[b];
    units += uint64_t(lv.hub.chunk_begin[k + 1] - lv.hub.chunk_begin[k]) * share[NUM_BINS - 1];  // (a block per chunk)
    most = std::max(most, units / 32);
  }
  return uint32_t(std::max<uint64_t>(1, std::min<uint64_t>(blocks, (most + PW / 2 - 1) / (PW / 2))));
}

uint32_t phase_list_cap(const Level &lv, uint32_t grid) {
  uint64_t cap = 1;
  for (int k = 0; k < lv.colors; ++k) {
    uint64_t items = 0;
    for (int b = 1; b < NUM_BINS - 1; ++b) {
      const uint64_t chunks = (lv.bucket_size(k, b) + (size_t(1) << chunk_log(b)) - 1) >> chunk_log(b);
      items += ((chunks + grid - 1) / grid) << chunk_log(b);
    }
    cap = std::max(cap, items);
  }
  return uint32_t(cap);
}

void launch_phase(bool sync, bool unit, bool whole, bool totals, uint32_t grid, const PhaseArgs &a, cudaStream_t s) {
  variant(sync, unit, whole, totals, [&](auto S, auto M) { launch<S.value, M.value>(grid, a, s); });
}

}  // namespace lvg
