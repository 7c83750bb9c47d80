// lvg_update.cu — applying a batch update to a graph resident in HBM.
//
// The reference prepares each batch on the host, outside its timed section:
// tidyBatchUpdateU (inc/batch.hxx:202-209) keeps the deletions whose edge is
// present and the insertions whose edge is absent, sorted by (source,
// target) without duplicates; applyBatchUpdateOmpU (inc/batch.hxx:241-248)
// then removes and adds them on LazyBitset rows that stay sorted
// (inc/_bitset.hxx:227-261), and an added edge makes both endpoints present
// (DiGraph::addEdge, inc/Graph.hxx:318-334). main.cxx:108-109 runs the two
// back to back, and hands the tidied batch to the dynamic methods.
//
// Here the uploaded graph is a gapped CSR: row u holds deg[u] sorted entries
// at off[u] with room for cap[u]; gaps and unused pool entries hold (0, 0.0).
// Only the rows the batch touches are rewritten, one warp per row:
//   merge:  the warp tests every deletion and insertion of its row against
//           the row (the tidy filter), keeping running counts of the kept
//           ones; every surviving entry and every kept insertion then finds
//           its output position with binary searches, so the row is
//           rewritten into scratch without a sequential merge;
//   commit: the row is copied back in place when it fits its capacity, or to
//           a fresh stretch of the overflow pool (bump allocation) when it
//           outgrows it; what the row no longer uses is zeroed.
// The host hands the batch over sorted by (source, target) with duplicates
// removed, and one UpdRow per touched source vertex. The kept flags are left
// in keep[] (deletions, then insertions) for the tidied batch.
#include "lvg_internal.cuh"

namespace lvg {
namespace {

// Number of entries of sorted a[0..n) that are < x.
__device__ __forceinline__ uint32_t count_less(const uint32_t *a, uint32_t n, uint32_t x) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (a[mid] < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ double warp_sum_f64(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Step 1, one warp per touched row: the tidy filter and the row's plan.
//   ikeep/dkeep: the insertion is absent / the deletion is present in the row;
//   ipre[j] / dpre[j]: kept insertions / deletions before j in the row;
//   P.n1: new degree; P.f0: first old index whose position changes (0 when
//   the row moves to the pool); P.len: entries to rewrite (n1 - f0);
//   P.src: source items (old entries from f0, then every insertion);
//   P.grow: pool entries the row takes (0 unless it outgrows its capacity).
// Also the change of the edge count and of the total weight (FP64), and the
// endpoints of kept insertions marked present in ex (when given).
__global__ void row_plan_kernel(const uint64_t *off, const uint32_t *deg, const uint32_t *cap, const uint32_t *key,
                                const float *w, const UpdRow *rows, size_t nrows, const uint32_t *dd,
                                const uint32_t *id, const float *iw, size_t nd_all, uint32_t *pre, uint32_t *keep,
                                RowPlan *plan, uint64_t *len, uint64_t *src, uint64_t *grow, uint8_t *ex,
                                unsigned long long *upd, double *wdelta) {
  const size_t warps = size_t(gridDim.x) * blockDim.x / 32;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1;
  long long edges = 0;
  double dw = 0;
  for (size_t r = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32; r < nrows; r += warps) {
    const UpdRow R = rows[r];
    const uint64_t o = off[R.u];
    const uint32_t n = deg[R.u];
    const uint32_t *row = key + o;
    const uint32_t *dl = dd + R.d0, nd = R.d1 - R.d0;
    const uint32_t *il = id + R.i0, ni = R.i1 - R.i0;
    uint32_t *dpre = pre + R.d0, *ipre = pre + nd_all + R.i0;
    uint32_t *dkeep = keep + R.d0, *ikeep = keep + nd_all + R.i0;
    uint32_t icarry = 0, dcarry = 0, first = n;
    for (uint32_t b = 0; b < ni; b += 32) {  // warp-uniform bound
      const uint32_t j = b + lane;
      bool k = false;
      if (j < ni) {
        const uint32_t p = count_less(row, n, il[j]);
        k = !(p < n && row[p] == il[j]);
        if (k) {
          first = min(first, p);
          dw += double(iw[R.i0 + j]);
          if (ex) ex[il[j]] = 1;
        }
      }
      const uint32_t m = __ballot_sync(0xffffffffu, k);
      if (j < ni) {
        ipre[j] = icarry + __popc(m & lt);
        ikeep[j] = k;
      }
      icarry += __popc(m);
    }
    for (uint32_t b = 0; b < nd; b += 32) {
      const uint32_t j = b + lane;
      bool k = false;
      if (j < nd) {
        const uint32_t p = count_less(row, n, dl[j]);
        k = p < n && row[p] == dl[j];
        if (k) {
          first = min(first, p);
          dw -= double(w[o + p]);
        }
      }
      const uint32_t m = __ballot_sync(0xffffffffu, k);
      if (j < nd) {
        dpre[j] = dcarry + __popc(m & lt);
        dkeep[j] = k;
      }
      dcarry += __popc(m);
    }
    first = __reduce_min_sync(0xffffffffu, first);
    if (lane == 0) {
      const uint32_t n1 = n - dcarry + icarry;
      const bool moved = n1 > cap[R.u];
      const uint32_t f0 = moved ? 0 : first;
      RowPlan P;
      P.n1 = n1;
      P.f0 = f0;
      P.dcarry = dcarry;
      P.icarry = icarry;
      plan[r] = P;
      len[r] = n1 - f0;
      src[r] = uint64_t(n - f0) + ni;
      grow[r] = moved ? row_capacity(n1) : 0;
      edges += (long long)n1 - (long long)n;
      if (icarry && ex) ex[R.u] = 1;
    }
  }
  dw = warp_sum_f64(dw);
  if (lane == 0) {
    if (edges) atomicAdd(&upd[UPD_EDGES], (unsigned long long)edges);
    if (dw != 0.0) atomicAdd(wdelta, dw);
  }
}

// The row an item of a flat range belongs to: the last r with start[r] <= x.
__device__ __forceinline__ uint32_t row_of(const uint64_t *start, uint32_t nrows, uint64_t x) {
  uint32_t lo = 0, hi = nrows;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (start[mid] <= x) lo = mid; else hi = mid;
  }
  return lo;
}

// The rows of a stretch [x0, x1) of a flat range, for a converged warp: r0 and
// r1, the rows of its ends, found by 32 probes at a time (a search of 17 steps
// per item was most of the time of the passes below), and the starts of the
// 32 rows from r0 on, one a lane.
struct WarpRows {
  uint32_t r0, r1;
  uint64_t st;
  __device__ __forceinline__ WarpRows(const uint64_t *start, uint32_t nrows, uint64_t x0, uint64_t x1) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t lo = 0, hi = nrows;  // start[lo] <= x0 < start[hi]
    while (hi - lo > 1) {
      const uint32_t step = (hi - lo + 31u) >> 5, at = lo + lane * step;
      const uint32_t n = __popc(__ballot_sync(0xffffffffu, at < hi && start[at] <= x0));  // (a prefix; at least lane 0)
      lo += (n - 1) * step;
      hi = min(hi, lo + step);
    }
    r0 = lo;
    st = r0 + lane < nrows ? start[r0 + lane] : ~0ull;
    const uint32_t n = __popc(__ballot_sync(0xffffffffu, st < x1));
    r1 = n < 32 ? r0 + n - 1 : r0 + 31 + row_of(start + r0 + 31, nrows - r0 - 31, x1 - 1);
  }
  // The row of item x (of this stretch), by all lanes.
  __device__ __forceinline__ uint32_t find(const uint64_t *start, uint64_t x) const {
    if (r1 == r0) return r0;
    if (r1 - r0 >= 32) return r0 + row_of(start + r0, r1 - r0 + 1, x);
    uint32_t at = 0;
#pragma unroll
    for (uint32_t step = 16; step > 0; step >>= 1)
      if (__shfl_sync(0xffffffffu, st, at + step) <= x) at += step;
    return r0 + at;
  }
};

// Items a warp takes at once: enough stretches for every warp of the device,
// at most 1024 items (the ends' searches and a row's plan are paid once).
uint32_t items_per_warp(uint64_t total) {
  uint32_t per = 32;
  while (per < 1024 && total / (2 * per) >= 16384) per *= 2;
  return per;
}

// Step 2, over the source items (old entries from f0, then insertions) of all
// touched rows: the item's place in the rewritten row, into scratch. An old
// entry at i goes to i - (kept deletions before it) + (kept insertions before
// it); a kept insertion j to j's kept rank + (old entries before it) - (kept
// deletions before it). Where a stretch of old entries lies between two
// neighbouring batch entries of its row, it is copied by a constant shift: the
// bulk of the items are those of a few long rows. (A 1e-4 |E| batch on R-MAT
// scale 24: 269 us, 446 with a search of the rows and the row's lists per
// item.)
__global__ void merge_items_kernel(const uint64_t *off, const uint32_t *deg, const uint32_t *key, const float *w,
                                   const UpdRow *rows, uint32_t nrows, const uint32_t *dd, const uint32_t *id,
                                   const float *iw, size_t nd_all, const uint32_t *pre, const uint32_t *keep,
                                   const RowPlan *plan, const uint64_t *src, uint64_t total, uint32_t per,
                                   const uint64_t *spos, uint32_t *skey, float *sw) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t warps = uint64_t(gridDim.x) * blockDim.x / 32;
  for (uint64_t x0 = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32 * per; x0 < total; x0 += warps * per) {
    const uint64_t x1 = min(x0 + per, total);
    const WarpRows W(src, nrows, x0, x1);
    if (W.r0 == W.r1) {
      const uint32_t r = W.r0;
      const UpdRow R = rows[r];
      const RowPlan P = plan[r];
      const uint64_t o = off[R.u];
      const uint32_t n = deg[R.u], i0 = P.f0 + uint32_t(x0 - src[r]), i1 = P.f0 + uint32_t(x1 - src[r]);
      if (i1 <= n) {  // old entries only
        const uint32_t *dl = dd + R.d0, nd = R.d1 - R.d0;
        const uint32_t *il = id + R.i0, ni = R.i1 - R.i0;
        // lanes 0-3: the batch entries before the stretch's ends
        const uint32_t k = key[o + (lane & 1u ? i1 - 1 : i0)];
        const uint32_t c = lane & 2u ? count_less(il, ni, k) : count_less(dl, nd, k);
        const uint32_t a0 = __shfl_sync(0xffffffffu, c, 0), a1 = __shfl_sync(0xffffffffu, c, 1);
        const uint32_t b0 = __shfl_sync(0xffffffffu, c, 2), b1 = __shfl_sync(0xffffffffu, c, 3);
        const uint32_t last = __shfl_sync(0xffffffffu, k, 1);
        const bool shift = a0 == a1 && b0 == b1 && !(a1 < nd && dl[a1] == last);
        const uint32_t *dpre = pre + R.d0, *ipre = pre + nd_all + R.i0;
        const uint64_t base = spos[r] - P.f0;
        const uint32_t by = (b0 < ni ? ipre[b0] : P.icarry) - (a0 < nd ? dpre[a0] : P.dcarry);
        for (uint32_t i = i0 + lane; i < i1; i += 128) {
          uint32_t kk[4];
          float ww[4];
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (i + 32 * q < i1) { kk[q] = key[o + i + 32 * q]; ww[q] = w[o + i + 32 * q]; }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint32_t ii = i + 32 * q;
            if (ii >= i1) continue;
            uint32_t at = ii + by;
            if (!shift) {
              const uint32_t aa = a0 + count_less(dl + a0, a1 - a0, kk[q]);
              if (aa < nd && dl[aa] == kk[q]) continue;  // deleted (present, so kept)
              const uint32_t bb = b0 + count_less(il + b0, b1 - b0, kk[q]);
              at = ii - (aa < nd ? dpre[aa] : P.dcarry) + (bb < ni ? ipre[bb] : P.icarry);
            }
            skey[base + at] = kk[q];
            sw[base + at] = ww[q];
          }
        }
        continue;
      }
    }
    for (uint64_t x = x0 + lane; x - lane < x1; x += 32) {  // any rows, any items
      const uint32_t r = W.find(src, min(x, x1 - 1));
      if (x >= x1) continue;
      const UpdRow R = rows[r];
      const RowPlan P = plan[r];
      const uint64_t o = off[R.u];
      const uint32_t n = deg[R.u];
      const uint32_t *row = key + o;
      const uint32_t *dl = dd + R.d0, nd = R.d1 - R.d0;
      const uint32_t *il = id + R.i0, ni = R.i1 - R.i0;
      const uint32_t *dpre = pre + R.d0, *ipre = pre + nd_all + R.i0;
      const uint32_t j = uint32_t(x - src[r]);
      const uint64_t base = spos[r];
      if (j < n - P.f0) {
        const uint32_t i = P.f0 + j;
        const uint32_t k = row[i];
        const uint32_t a = count_less(dl, nd, k);
        if (a < nd && dl[a] == k) continue;  // deleted (present, so kept)
        const uint32_t b = count_less(il, ni, k);
        const uint32_t at = i - (a < nd ? dpre[a] : P.dcarry) + (b < ni ? ipre[b] : P.icarry) - P.f0;
        skey[base + at] = k;
        sw[base + at] = w[o + i];
      } else {
        const uint32_t jj = j - (n - P.f0);
        if (!keep[nd_all + R.i0 + jj]) continue;  // already present: tidied away
        const uint32_t k = il[jj];
        const uint32_t a = count_less(dl, nd, k);
        const uint32_t at = ipre[jj] + count_less(row, n, k) - (a < nd ? dpre[a] : P.dcarry) - P.f0;
        skey[base + at] = k;
        sw[base + at] = iw[R.i0 + jj];
      }
    }
  }
}

// Step 3, over the rewritten entries: scratch -> the row's place (in place
// from f0, or the row's new stretch in the pool at pool + gpos[r]). A lane
// keeps the place of each of the stretch's 32 first rows. (The same batch:
// 146 us, 417 with a search per entry, 232 with the
// places of a stretch of several rows looked up per entry.)
__global__ void copy_items_kernel(const uint64_t *off, const UpdRow *rows, uint32_t nrows, const RowPlan *plan,
                                  const uint64_t *spos, uint64_t total, uint32_t per, const uint64_t *grow,
                                  const uint64_t *gpos, uint64_t pool, const uint32_t *skey, const float *sw,
                                  uint32_t *key, float *w) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t warps = uint64_t(gridDim.x) * blockDim.x / 32;
  auto place = [&](uint32_t r) {  // of entry 0 of the flat range, were it the row's
    return (grow[r] ? pool + gpos[r] : off[rows[r].u]) + plan[r].f0 - spos[r];
  };
  for (uint64_t x0 = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32 * per; x0 < total; x0 += warps * per) {
    const uint64_t x1 = min(x0 + per, total);
    const WarpRows W(spos, nrows, x0, x1);
    const bool few = W.r1 - W.r0 < 32;
    const uint64_t mine = few && W.r0 + lane <= W.r1 ? place(W.r0 + lane) : 0;
    for (uint64_t x = x0 + lane; x - lane < x1; x += 128) {
      uint32_t kk[4];
      float ww[4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (x + 32 * q < x1) { kk[q] = skey[x + 32 * q]; ww[q] = sw[x + 32 * q]; }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint64_t y = x + 32 * q;
        const uint32_t r = W.find(spos, min(y, x1 - 1));
        const uint64_t to = few ? __shfl_sync(0xffffffffu, mine, r - W.r0) : place(r);
        if (y < x1) { key[to + y] = kk[q]; w[to + y] = ww[q]; }
      }
    }
  }
}

// Step 4, one warp per touched row: zero what the row no longer uses (the
// tail in place; the old stretch and the new stretch's slack when it moved)
// and set its offset, capacity and degree.
__global__ void finish_rows_kernel(uint64_t *off, uint32_t *deg, uint32_t *cap, uint32_t *key, float *w,
                                   const UpdRow *rows, size_t nrows, const RowPlan *plan, const uint64_t *grow,
                                   const uint64_t *gpos, uint64_t pool) {
  const size_t warps = size_t(gridDim.x) * blockDim.x / 32;
  const uint32_t lane = threadIdx.x & 31;
  for (size_t r = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32; r < nrows; r += warps) {
    const uint32_t u = rows[r].u;
    const uint32_t n0 = deg[u], n1 = plan[r].n1;
    const uint64_t o = off[u];
    if (grow[r]) {
      const uint64_t no = pool + gpos[r];
      const uint32_t nc = uint32_t(grow[r]);
      for (uint32_t i = lane; i < n0; i += 32) { key[o + i] = 0; w[o + i] = 0.f; }
      for (uint32_t i = n1 + lane; i < nc; i += 32) { key[no + i] = 0; w[no + i] = 0.f; }
      __syncwarp();  // every lane has read the row's old extent
      if (lane == 0) { off[u] = no; cap[u] = nc; deg[u] = n1; }
    } else {
      for (uint32_t i = n1 + lane; i < n0; i += 32) { key[o + i] = 0; w[o + i] = 0.f; }
      __syncwarp();
      if (lane == 0) deg[u] = n1;
    }
  }
}

// Present vertices, counted into *dst, sixteen flags per load (ex is a device
// allocation, so aligned; a byte per load took 30 us on R-MAT scale 24).
__global__ void count_present_kernel(const uint8_t *ex, size_t n, unsigned long long *dst) {
  unsigned int c = 0;
  const size_t n16 = n / 16, t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const uint4 *e16 = reinterpret_cast<const uint4 *>(ex);
  auto some = [](uint32_t v) { return __popc(__vcmpne4(v, 0u)) / 8; };
  for (size_t i = t; i < n16; i += size_t(gridDim.x) * blockDim.x) {
    const uint4 v = e16[i];
    c += some(v.x) + some(v.y) + some(v.z) + some(v.w);
  }
  if (t < n % 16) c += ex[16 * n16 + t] != 0;
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(dst, (unsigned long long)c);
}

// Spread a compact CSR into the gapped layout (one warp per row; gaps zero).
__global__ void spread_rows_kernel(const uint64_t *coff, const uint32_t *ckey, const float *cw, size_t n,
                                   const uint64_t *off, const uint32_t *cap, uint32_t *key, float *w) {
  const size_t warps = size_t(gridDim.x) * blockDim.x / 32;
  const uint32_t lane = threadIdx.x & 31;
  for (size_t u = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32; u < n; u += warps) {
    const uint64_t s = coff[u], d = coff[u + 1] - coff[u], o = off[u];
    for (uint32_t i = lane; i < cap[u]; i += 32) {
      key[o + i] = i < d ? ckey[s + i] : 0;
      w[o + i] = i < d ? cw[s + i] : 0.f;
    }
  }
}

// Degrees and capacities of a compact CSR.
__global__ void row_caps_kernel(const uint64_t *coff, size_t n, uint32_t *deg, uint32_t *cap, uint64_t *cap64) {
  for (size_t u = size_t(blockIdx.x) * blockDim.x + threadIdx.x; u < n; u += size_t(gridDim.x) * blockDim.x) {
    const uint32_t d = uint32_t(coff[u + 1] - coff[u]);
    const uint32_t c = row_capacity(d);
    deg[u] = d;
    cap[u] = c;
    cap64[u] = c;
  }
}

// Fresh capacities from the current degrees.
__global__ void fresh_caps_kernel(const uint32_t *deg, size_t n, uint32_t *cap, uint64_t *cap64) {
  for (size_t u = size_t(blockIdx.x) * blockDim.x + threadIdx.x; u < n; u += size_t(gridDim.x) * blockDim.x) {
    const uint32_t c = row_capacity(deg[u]);
    cap[u] = c;
    cap64[u] = c;
  }
}

// ---------------------------------------------------------------- plan

// The entries of two lists as packed (list, src, dst) keys with their indices
// (list: the bit above 2b, set for the second where both have entries).
__global__ void pack_keys_kernel(const uint32_t *ds, const uint32_t *dd, size_t nd, const uint32_t *is,
                                 const uint32_t *id, size_t ni, int b, uint64_t *key, uint32_t *val) {
  const uint64_t second = nd ? uint64_t(1) << (2 * b & 63) : 0u;
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < nd + ni; i += size_t(gridDim.x) * blockDim.x) {
    key[i] = i < nd ? uint64_t(ds[i]) << b | dd[i] : second | uint64_t(is[i - nd]) << b | id[i - nd];
    val[i] = uint32_t(i);
  }
}

// First of each run of equal keys; the sort is stable, so that is the first
// occurrence in batch order.
__global__ void first_flags_kernel(const uint64_t *key, size_t n, uint32_t *flag) {
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
    flag[i] = i == 0 || key[i] != key[i - 1];
}

// The first of each run back into its list (the first list's keys are sorted
// before the second's; pos: the flags' exclusive prefix, their sum at pos[nd +
// ni]); the lists' lengths into *cd and *ci (where given).
__global__ void unpack_keys_kernel(const uint64_t *key, const uint32_t *val, const uint32_t *flag,
                                   const uint32_t *pos, size_t nd, size_t ni, int b, const float *dw, const float *iw,
                                   uint32_t *ods, uint32_t *odd, float *odw, uint32_t *ois, uint32_t *oid, float *oiw,
                                   uint32_t *cd, uint32_t *ci) {
  const uint64_t mask = (uint64_t(1) << b) - 1;
  const uint32_t kept = pos[nd], all = pos[nd + ni];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (cd) *cd = kept;
    if (ci) *ci = all - kept;
  }
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < nd + ni; i += size_t(gridDim.x) * blockDim.x) {
    if (!flag[i]) continue;
    const uint32_t u = uint32_t(key[i] >> b & mask), v = uint32_t(key[i] & mask);
    if (i < nd) {
      const uint32_t o = pos[i];
      ods[o] = u;
      odd[o] = v;
      odw[o] = dw[val[i]];
    } else {
      const uint32_t o = pos[i] - kept;
      ois[o] = u;
      oid[o] = v;
      oiw[o] = iw[val[i] - nd];
    }
  }
}

__device__ __forceinline__ uint32_t lower_bound_u32(const uint32_t *a, uint32_t n, uint32_t x) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (a[mid] < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// The touched vertices are the sources of the two sorted lists (their lengths
// are read from the device: *nd, *ni; room for cap entries each): flag[i] = 1
// for the first deletion of a source, flag[cap + j] = 1 for the first
// insertion of a source without deletions.
__global__ void row_flags_kernel(const uint32_t *ds, const uint32_t *nd, const uint32_t *is, const uint32_t *ni,
                                 size_t cap, uint32_t *flag) {
  const uint32_t a = *nd, c = *ni;
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < cap; i += size_t(gridDim.x) * blockDim.x) {
    flag[i] = i < a && (i == 0 || ds[i] != ds[i - 1]);
    bool f = i < c && (i == 0 || is[i] != is[i - 1]);
    if (f) {
      const uint32_t p = lower_bound_u32(ds, a, is[i]);
      f = !(p < a && ds[p] == is[i]);
    }
    flag[cap + i] = f;
  }
}

// One UpdRow per touched vertex, in id order (pos: the flags' exclusive prefix;
// a row's place is its rank in its own list plus the other list's flagged
// sources below it); the longest insertion run into upd[UPD_MAXG]. (A pass over
// all vertices for the batch's few sources took 0.25 ms with its scan on R-MAT
// scale 24.)
__global__ void plan_rows_kernel(const uint32_t *flag, const uint32_t *pos, size_t cap, const uint32_t *ds,
                                 const uint32_t *nd, const uint32_t *is, const uint32_t *ni, UpdRow *rows,
                                 unsigned long long *upd, uint32_t *nrows) {
  const uint32_t a = *nd, c = *ni;
  const uint32_t deletions = pos[cap], total = pos[2 * cap];  // flagged
  if (blockIdx.x == 0 && threadIdx.x == 0) *nrows = total;
  for (size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x; t < 2 * cap; t += size_t(gridDim.x) * blockDim.x) {
    if (!flag[t]) continue;
    const bool del = t < cap;
    UpdRow R;
    R.u = del ? ds[t] : is[t - cap];
    R.d0 = del ? uint32_t(t) : lower_bound_u32(ds, a, R.u);
    R.d1 = del ? lower_bound_u32(ds, a, R.u + 1) : R.d0;
    R.i0 = del ? lower_bound_u32(is, c, R.u) : uint32_t(t - cap);
    R.i1 = lower_bound_u32(is, c, R.u + 1);
    rows[del ? pos[t] + (pos[cap + R.i0] - deletions) : pos[t] - deletions + pos[R.d0]] = R;
    if (R.i1 > R.i0) atomicMax(&upd[UPD_MAXG], (unsigned long long)(R.i1 - R.i0));
  }
}

// Compaction of a sorted batch list by its kept flags (the tidied batch):
// entry i goes to pos[i] - *pos_base when keep[i].
__global__ void tidy_compact_kernel(const uint32_t *src, const uint32_t *dst, const float *w, size_t n,
                                    const uint32_t *keep, const uint32_t *pos, const uint32_t *pos_base,
                                    uint32_t *osrc, uint32_t *odst, float *ow) {
  const uint32_t b = pos_base ? *pos_base : 0;
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
    if (!keep[i]) continue;
    const uint32_t o = pos[i] - b;
    osrc[o] = src[i];
    odst[o] = dst[i];
    ow[o] = w[i];
  }
}

// ---- the steps of a small batch, one block each

constexpr int SB = 1024;  // threads
constexpr int SI = 4;     // consecutive items a thread holds
static_assert(SB * SI == 2 * PLAN_SMALL && SB * SI == ROWS_SMALL, "");

// Exclusive prefix of x over the block's threads; the sum into *total. (All
// threads; `part` holds 33 values and is free again after the call's barrier.)
template <class T>
__device__ __forceinline__ T block_prefix(T x, T *part, T *total) {
  const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
  T inc = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= uint32_t(o)) inc += y;
  }
  if (lane == 31) part[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    T p = part[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T y = __shfl_up_sync(0xffffffffu, p, o);
      if (lane >= uint32_t(o)) p += y;
    }
    part[lane] = p;
  }
  __syncthreads();
  const T before = wid ? part[wid - 1] : T(0);
  *total = part[31];
  __syncthreads();
  return before + inc - x;
}

// Both lists packed as (list, source, target, index) keys and sorted at once in
// shared memory (a bitonic network), the first of each equal (list, source,
// target) kept in batch order, and a row per source: what the passes above do
// for large batches in thirteen launches (22 us for 1280 entries against 60 and
// the gaps between them; with the two kernels below, half the host's waits and
// fewer copies an applied and answered batch of 640 edges on a 1M-vertex graph
// takes 367 us instead of 443). A list above PLAN_SMALL would leave the chip
// idle behind one block for longer than the passes take. cnt: kept deletions and insertions,
// rows, the longest insertion run.
__global__ void __launch_bounds__(SB) plan_small_kernel(const uint32_t *ds, const uint32_t *dd, const float *dw,
                                                        uint32_t nd, const uint32_t *is, const uint32_t *id,
                                                        const float *iw, uint32_t ni, uint32_t n2, uint32_t *ods,
                                                        uint32_t *odd, float *odw, uint32_t *ois, uint32_t *oid,
                                                        float *oiw, UpdRow *rows, uint32_t *cnt) {
  constexpr int IB = 11, KB = PLAN_SMALL_ID;  // bits of an index and of an id
  static_assert((1u << IB) == PLAN_SMALL && 1 + 2 * KB + IB <= 64, "");
  __shared__ __align__(16) unsigned long long key[SB * SI];
  __shared__ uint32_t part[33];
  __shared__ uint32_t run;
  const uint32_t tid = threadIdx.x, n = nd + ni;
  for (uint32_t e = tid; e < n2; e += SB) {
    unsigned long long k = ~0ull;
    if (e < nd) k = ((unsigned long long)ds[e] << KB | dd[e]) << IB | e;
    else if (e < n) k = 1ull << (2 * KB + IB) | ((unsigned long long)is[e - nd] << KB | id[e - nd]) << IB | (e - nd);
    key[e] = k;
  }
  if (tid == 0) run = 0;
  __syncthreads();
  for (uint32_t size = 2; size <= n2; size <<= 1)
    for (uint32_t step = size >> 1; step > 0; step >>= 1) {
      for (uint32_t t = tid; t < n2 / 2; t += SB) {
        const uint32_t i = (t & ~(step - 1)) * 2 + (t & (step - 1)), j = i + step;
        const unsigned long long a = key[i], b = key[j];
        if ((a > b) == ((i & size) == 0)) { key[i] = b; key[j] = a; }
      }
      // (a warp's 32 pairs of a step up to 32 lie in its own 64 keys)
      if (step > 32 || (step == 1 && size > 32)) __syncthreads();
      else __syncwarp();
    }
  __syncthreads();
  // the first of each run, four consecutive keys a thread
  unsigned long long k[SI];
  uint32_t first = 0, tot;
#pragma unroll
  for (int x = 0; x < SI; ++x) {
    const uint32_t e = tid * SI + x;
    k[x] = e < n ? key[e] : ~0ull;
    if (e < n && (e == 0 || key[e - 1] >> IB != k[x] >> IB)) first |= 1u << x;
  }
  uint32_t at = block_prefix<uint32_t>(uint32_t(__popc(first)), part, &tot);  // (and key[] is read)
  // kept deletions: those of list 0 (sorted first)
  uint32_t dels = 0;
#pragma unroll
  for (int x = 0; x < SI; ++x) dels += (first >> x & 1u) && k[x] >> (2 * KB + IB) == 0;
  uint32_t a;
  block_prefix<uint32_t>(dels, part, &a);
  uint32_t *src = reinterpret_cast<uint32_t *>(key), *pos = src + SB * SI;  // kept sources; the rows before each
#pragma unroll
  for (int x = 0; x < SI; ++x) {
    if (!(first >> x & 1u)) continue;
    const uint32_t u = uint32_t(k[x] >> (KB + IB)) & ((1u << KB) - 1u), v = uint32_t(k[x] >> IB) & ((1u << KB) - 1u);
    const uint32_t i = uint32_t(k[x]) & ((1u << IB) - 1u);
    src[at] = u;
    if (at < a) { ods[at] = u; odd[at] = v; odw[at] = dw[i]; }
    else { ois[at - a] = u; oid[at - a] = v; oiw[at - a] = iw[i]; }
    ++at;
  }
  __syncthreads();
  const uint32_t c = tot - a;
  const uint32_t *us = src + a;  // the insertions' sources
  uint32_t head = 0;
#pragma unroll
  for (int x = 0; x < SI; ++x) {
    const uint32_t e = tid * SI + x;
    if (e >= tot) continue;
    bool h = e == 0 || e == a || src[e] != src[e - 1];
    if (h && e >= a) {
      const uint32_t p = lower_bound_u32(src, a, src[e]);
      h = !(p < a && src[p] == src[e]);
    }
    if (h) head |= 1u << x;
  }
  uint32_t nrows;
  uint32_t before = block_prefix<uint32_t>(uint32_t(__popc(head)), part, &nrows);
  uint32_t b = before;
#pragma unroll
  for (int x = 0; x < SI; ++x) {
    const uint32_t e = tid * SI + x;
    if (e < tot) pos[e] = b;
    b += head >> x & 1u;
  }
  __syncthreads();
  const uint32_t drows = a < tot ? pos[a] : nrows;  // rows of sources with deletions
#pragma unroll
  for (int x = 0; x < SI; ++x) {
    if (!(head >> x & 1u)) continue;
    const uint32_t e = tid * SI + x;
    const bool del = e < a;
    UpdRow R;
    R.u = src[e];
    R.d0 = del ? e : lower_bound_u32(src, a, R.u);
    R.d1 = del ? lower_bound_u32(src, a, R.u + 1) : R.d0;
    R.i0 = del ? lower_bound_u32(us, c, R.u) : e - a;
    R.i1 = lower_bound_u32(us, c, R.u + 1);
    const uint32_t o = del ? R.i0 + a : R.d0;  // the other list's rows below
    const uint32_t p = o < tot ? pos[o] : nrows;
    rows[del ? pos[e] + (p - drows) : pos[e] - drows + p] = R;
    if (R.i1 > R.i0) atomicMax(&run, R.i1 - R.i0);
  }
  __syncthreads();
  if (tid == 0) { cnt[0] = a; cnt[1] = c; cnt[2] = nrows; cnt[3] = run; }
}

// The exclusive prefixes of the rows' rewritten entries, source items and pool
// entries, and their sums.
__global__ void __launch_bounds__(SB) row_scans_small_kernel(const uint64_t *len, const uint64_t *src,
                                                             const uint64_t *grow, uint32_t nrows, uint64_t *spos,
                                                             uint64_t *srcpos, uint64_t *gpos,
                                                             unsigned long long *upd) {
  __shared__ unsigned long long part[33];
  const uint64_t *in[3] = {len, src, grow};
  uint64_t *out[3] = {spos, srcpos, gpos};
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    unsigned long long x[SI], sum = 0, total;
#pragma unroll
    for (int i = 0; i < SI; ++i) {
      const uint32_t e = threadIdx.x * SI + i;
      x[i] = e < nrows ? in[q][e] : 0ull;
      sum += x[i];
    }
    unsigned long long at = block_prefix<unsigned long long>(sum, part, &total);
#pragma unroll
    for (int i = 0; i < SI; ++i) {
      const uint32_t e = threadIdx.x * SI + i;
      if (e < nrows) out[q][e] = at;
      at += x[i];
    }
    if (threadIdx.x == 0) upd[UPD_ENTRIES + q] = total;
  }
}

// The kept entries of both lists, in order; cnt: kept deletions, kept entries.
__global__ void __launch_bounds__(SB) tidy_small_kernel(const uint32_t *ds, const uint32_t *dd, const float *dw,
                                                        uint32_t nd, const uint32_t *is, const uint32_t *id,
                                                        const float *iw, uint32_t ni, const uint32_t *keep,
                                                        uint32_t *tds, uint32_t *tdd, float *tdw, uint32_t *tis,
                                                        uint32_t *tid, float *tiw, uint32_t *cnt) {
  __shared__ uint32_t part[33];
  uint32_t kept = 0, dels = 0, total, a;
#pragma unroll
  for (int i = 0; i < SI; ++i) {
    const uint32_t e = threadIdx.x * SI + i;
    if (e < nd + ni && keep[e]) {
      kept |= 1u << i;
      dels += e < nd;
    }
  }
  uint32_t at = block_prefix<uint32_t>(uint32_t(__popc(kept)), part, &total);
  block_prefix<uint32_t>(dels, part, &a);
#pragma unroll
  for (int i = 0; i < SI; ++i) {
    if (!(kept >> i & 1u)) continue;
    const uint32_t e = threadIdx.x * SI + i;
    if (e < nd) { tds[at] = ds[e]; tdd[at] = dd[e]; tdw[at] = dw[e]; }
    else { tis[at - a] = is[e - nd]; tid[at - a] = id[e - nd]; tiw[at - a] = iw[e - nd]; }
    ++at;
  }
  if (threadIdx.x == 0) { cnt[0] = a; cnt[1] = total; }
}

// Copy every row into a new gapped layout (one warp per row; gaps zero).
__global__ void relayout_kernel(const uint64_t *old_off, const uint32_t *deg, const uint32_t *old_key,
                                const float *old_w, size_t n, const uint64_t *off, const uint32_t *cap,
                                uint32_t *key, float *w) {
  const size_t warps = size_t(gridDim.x) * blockDim.x / 32;
  const uint32_t lane = threadIdx.x & 31;
  for (size_t u = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32; u < n; u += warps) {
    const uint64_t s = old_off[u], o = off[u];
    const uint32_t d = deg[u];
    for (uint32_t i = lane; i < cap[u]; i += 32) {
      key[o + i] = i < d ? old_key[s + i] : 0;
      w[o + i] = i < d ? old_w[s + i] : 0.f;
    }
  }
}

}  // namespace

void launch_row_caps(const uint64_t *coff, size_t n, uint32_t *deg, uint32_t *cap, uint64_t *cap64, cudaStream_t s) {
  if (!n) return;
  row_caps_kernel<<<grid_for(n, 256), 256, 0, s>>>(coff, n, deg, cap, cap64);
  LVG_CHECK_LAUNCH();
}

void launch_spread_rows(const uint64_t *coff, const uint32_t *ckey, const float *cw, size_t n, const uint64_t *off,
                        const uint32_t *cap, uint32_t *key, float *w, cudaStream_t s) {
  if (!n) return;
  spread_rows_kernel<<<grid_for(n * 32, 256), 256, 0, s>>>(coff, ckey, cw, n, off, cap, key, w);
  LVG_CHECK_LAUNCH();
}

void launch_row_plan(const uint64_t *off, const uint32_t *deg, const uint32_t *cap, const uint32_t *key,
                     const float *w, const UpdRow *rows, size_t nrows, const uint32_t *dd, const uint32_t *id,
                     const float *iw, size_t nd_all, uint32_t *pre, uint32_t *keep, RowPlan *plan, uint64_t *len,
                     uint64_t *src, uint64_t *grow, uint8_t *ex, unsigned long long *upd, double *wdelta,
                     cudaStream_t s) {
  if (!nrows) return;
  row_plan_kernel<<<grid_for(nrows * 32, 256), 256, 0, s>>>(off, deg, cap, key, w, rows, nrows, dd, id, iw, nd_all,
                                                              pre, keep, plan, len, src, grow, ex, upd, wdelta);
  LVG_CHECK_LAUNCH();
}

void launch_merge_items(const uint64_t *off, const uint32_t *deg, const uint32_t *key, const float *w,
                        const UpdRow *rows, size_t nrows, const uint32_t *dd, const uint32_t *id, const float *iw,
                        size_t nd_all, const uint32_t *pre, const uint32_t *keep, const RowPlan *plan,
                        const uint64_t *src, uint64_t total, const uint64_t *spos, uint32_t *skey, float *sw,
                        cudaStream_t s) {
  if (!total) return;
  const uint32_t per = items_per_warp(total);
  merge_items_kernel<<<grid_for((total + per - 1) / per * 32, 256), 256, 0, s>>>(
      off, deg, key, w, rows, uint32_t(nrows), dd, id, iw, nd_all, pre, keep, plan, src, total, per, spos, skey, sw);
  LVG_CHECK_LAUNCH();
}

void launch_copy_items(const uint64_t *off, const UpdRow *rows, size_t nrows, const RowPlan *plan,
                       const uint64_t *spos, uint64_t total, const uint64_t *grow, const uint64_t *gpos,
                       uint64_t pool, const uint32_t *skey, const float *sw, uint32_t *key, float *w,
                       cudaStream_t s) {
  if (!total) return;
  const uint32_t per = items_per_warp(total);
  copy_items_kernel<<<grid_for((total + per - 1) / per * 32, 256), 256, 0, s>>>(
      off, rows, uint32_t(nrows), plan, spos, total, per, grow, gpos, pool, skey, sw, key, w);
  LVG_CHECK_LAUNCH();
}

void launch_finish_rows(uint64_t *off, uint32_t *deg, uint32_t *cap, uint32_t *key, float *w, const UpdRow *rows,
                        size_t nrows, const RowPlan *plan, const uint64_t *grow, const uint64_t *gpos,
                        uint64_t pool, cudaStream_t s) {
  if (!nrows) return;
  finish_rows_kernel<<<grid_for(nrows * 32, 256), 256, 0, s>>>(off, deg, cap, key, w, rows, nrows, plan, grow, gpos,
                                                                 pool);
  LVG_CHECK_LAUNCH();
}

void launch_count_present(const uint8_t *ex, size_t span, unsigned long long *upd, cudaStream_t s) {
  if (!span) return;
  count_present_kernel<<<grid_for(span / 16, 256), 256, 0, s>>>(ex, span, &upd[UPD_ORDER]);
  LVG_CHECK_LAUNCH();
}

void launch_tidy_compact(const uint32_t *src, const uint32_t *dst, const float *w, size_t n, const uint32_t *keep,
                         const uint32_t *pos, const uint32_t *pos_base, uint32_t *osrc, uint32_t *odst, float *ow,
                         cudaStream_t s) {
  if (!n) return;
  tidy_compact_kernel<<<grid_for(n, 256), 256, 0, s>>>(src, dst, w, n, keep, pos, pos_base, osrc, odst, ow);
  LVG_CHECK_LAUNCH();
}

void launch_pack_keys(const uint32_t *ds, const uint32_t *dd, size_t nd, const uint32_t *is, const uint32_t *id,
                      size_t ni, int b, uint64_t *key, uint32_t *val, cudaStream_t s) {
  if (!(nd + ni)) return;
  pack_keys_kernel<<<grid_for(nd + ni, 256), 256, 0, s>>>(ds, dd, nd, is, id, ni, b, key, val);
  LVG_CHECK_LAUNCH();
}

void launch_first_flags(const uint64_t *key, size_t n, uint32_t *flag, cudaStream_t s) {
  if (!n) return;
  first_flags_kernel<<<grid_for(n, 256), 256, 0, s>>>(key, n, flag);
  LVG_CHECK_LAUNCH();
}

void launch_unpack_keys(const uint64_t *key, const uint32_t *val, const uint32_t *flag, const uint32_t *pos, size_t nd,
                        size_t ni, int b, const float *dw, const float *iw, uint32_t *ods, uint32_t *odd, float *odw,
                        uint32_t *ois, uint32_t *oid, float *oiw, uint32_t *cd, uint32_t *ci, cudaStream_t s) {
  if (!(nd + ni)) return;
  unpack_keys_kernel<<<grid_for(nd + ni, 256), 256, 0, s>>>(key, val, flag, pos, nd, ni, b, dw, iw, ods, odd, odw, ois,
                                                            oid, oiw, cd, ci);
  LVG_CHECK_LAUNCH();
}

void launch_plan_rows(const uint32_t *ds, const uint32_t *nd, const uint32_t *is, const uint32_t *ni, size_t cap,
                      uint32_t *flag, uint32_t *pos, uint32_t *scan, UpdRow *rows, unsigned long long *upd,
                      uint32_t *nrows, cudaStream_t s) {
  if (!cap) return;
  row_flags_kernel<<<grid_for(cap, 256), 256, 0, s>>>(ds, nd, is, ni, cap, flag);
  LVG_CHECK_LAUNCH();
  exclusive_scan_u32(flag, pos, 2 * cap, pos + 2 * cap, scan, s);
  plan_rows_kernel<<<grid_for(2 * cap, 256), 256, 0, s>>>(flag, pos, cap, ds, nd, is, ni, rows, upd, nrows);
  LVG_CHECK_LAUNCH();
}

void launch_plan_small(const uint32_t *ds, const uint32_t *dd, const float *dw, size_t nd, const uint32_t *is,
                       const uint32_t *id, const float *iw, size_t ni, uint32_t *ods, uint32_t *odd, float *odw,
                       uint32_t *ois, uint32_t *oid, float *oiw, UpdRow *rows, uint32_t *cnt, cudaStream_t s) {
  uint32_t n2 = 64;
  while (n2 < nd + ni) n2 *= 2;
  plan_small_kernel<<<1, SB, 0, s>>>(ds, dd, dw, uint32_t(nd), is, id, iw, uint32_t(ni), n2, ods, odd, odw, ois, oid,
                                     oiw, rows, cnt);
  LVG_CHECK_LAUNCH();
}

void launch_row_scans_small(const uint64_t *len, const uint64_t *src, const uint64_t *grow, size_t nrows,
                            uint64_t *spos, uint64_t *srcpos, uint64_t *gpos, unsigned long long *upd,
                            cudaStream_t s) {
  row_scans_small_kernel<<<1, SB, 0, s>>>(len, src, grow, uint32_t(nrows), spos, srcpos, gpos, upd);
  LVG_CHECK_LAUNCH();
}

void launch_tidy_small(const uint32_t *ds, const uint32_t *dd, const float *dw, size_t nd, const uint32_t *is,
                       const uint32_t *id, const float *iw, size_t ni, const uint32_t *keep, uint32_t *tds,
                       uint32_t *tdd, float *tdw, uint32_t *tis, uint32_t *tid, float *tiw, uint32_t *cnt,
                       cudaStream_t s) {
  tidy_small_kernel<<<1, SB, 0, s>>>(ds, dd, dw, uint32_t(nd), is, id, iw, uint32_t(ni), keep, tds, tdd, tdw, tis, tid,
                                     tiw, cnt);
  LVG_CHECK_LAUNCH();
}

void launch_fresh_caps(const uint32_t *deg, size_t n, uint32_t *cap, uint64_t *cap64, cudaStream_t s) {
  if (!n) return;
  fresh_caps_kernel<<<grid_for(n, 256), 256, 0, s>>>(deg, n, cap, cap64);
  LVG_CHECK_LAUNCH();
}

void launch_relayout_rows(const uint64_t *old_off, const uint32_t *deg, const uint32_t *old_key, const float *old_w,
                          size_t n, const uint64_t *off, const uint32_t *cap, uint32_t *key, float *w,
                          cudaStream_t s) {
  if (!n) return;
  relayout_kernel<<<grid_for(n * 32, 256), 256, 0, s>>>(old_off, deg, old_key, old_w, n, off, cap, key, w);
  LVG_CHECK_LAUNCH();
}

}  // namespace lvg
