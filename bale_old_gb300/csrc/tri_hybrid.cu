// tri_hybrid.cu -- triangle counting, bitmap/search hybrid over rows i (tri.mode 1;
// also the path for matrices beyond the wedge kernels' 32-bit limits).
//
// Same count as apps/triangle_src/triangle_agi.upc:69-99 (alg 0): for every
// nonzero L[i][j] after the first of row i, |row_i and row_j|.  The rows of a
// degree-ordered L are long exactly where the work is (a hub's row holds its
// higher-degree neighbours, hundreds of them), so the two sides of each
// intersection are handled by size (tri_device.cuh):
//
//  * heavy rows (label below 2^19 and at least 64 nonzeros): one CTA per row.
//    Row i becomes a bitmap over [0,i) in shared memory; each warp streams
//    whole rows j (16-byte loads from a u32 copy of the column array) and
//    tests every element against the bitmap -- one shared-memory load per
//    element instead of a binary search.  The bits are cleared by row i's own
//    columns before the next row, so the bitmap is never swept;
//  * light rows: one warp per row, row i staged in shared memory.  For each
//    neighbour j the cheaper side is searched: either row j is streamed and
//    each element is binary-searched in the part of row i before j, or each
//    element of that part of row i is binary-searched in row j.
//
//  * short rows (at most 63 nonzeros, matrices below 2^32 nonzeros): eight rows
//    per warp, each row a small hashed bit set, their neighbours' rows streamed
//    together (tri_short_kernel); the light kernel then takes only the rows
//    from a list that are neither heavy nor short.
//
// Launch sequence: convert (int64 columns -> u32), classify (row records, the
// lists of heavy and long rows), heavy kernel, short kernel, light kernel.
// The work tally counts row-j elements streamed plus binary-search probes.
// Validation: bad offsets, columns outside [0,i) or non-ascending rows are
// counted in *bad and the row is skipped.
#include <algorithm>

#include "tri_device.cuh"

namespace bale {

namespace {

using tri::kBadCol;
using tri::kFull;
constexpr int kHeavyThreads = 512;
constexpr int kLightThreads = 256;
constexpr int kLightWarps = kLightThreads / 32;

__global__ void __launch_bounds__(256)
    tri_convert_kernel(const int64_t *__restrict__ col, int64_t nnz, uint32_t *__restrict__ col32, const unsigned *__restrict__ run_if) {
  if (tri::skipped(run_if, 0u)) return;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; k < nnz; k += stride) {
    const int64_t c = ld_stream(col + k);
    col32[k] = (c < 0 || c >= static_cast<int64_t>(kBadCol)) ? kBadCol : static_cast<uint32_t>(c);
  }
}

__global__ void __launch_bounds__(256)
    tri_classify_kernel(const int64_t *__restrict__ off, int64_t n, int64_t bits,
                        uint32_t *__restrict__ heavy, unsigned long long *__restrict__ nheavy, const unsigned *__restrict__ run_if) {
  if (tri::skipped(run_if, 0u)) return;
  const int64_t lim = n < bits ? n : bits;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t base = static_cast<int64_t>(blockIdx.x) * blockDim.x; base < lim; base += stride) {
    const int64_t i = base + threadIdx.x;
    const bool h = i < lim && tri::is_heavy(i, off[i], off[i + 1], bits);
    const unsigned m = __ballot_sync(kFull, h);
    unsigned long long slot = 0;
    if (lane_id() == 0 && m) slot = atomicAdd(nheavy, static_cast<unsigned long long>(__popc(m)));
    slot = __shfl_sync(kFull, slot, 0);
    if (h) heavy[slot + __popc(m & ((1u << lane_id()) - 1u))] = static_cast<uint32_t>(i);
  }
}

__device__ __forceinline__ void flush_tally(tri::Tally t, unsigned long long *count, unsigned long long *work,
                                            unsigned long long *bad) {
  t.cnt = warp_sum_u64(t.cnt);
  t.work = warp_sum_u64(t.work);
  t.bad = warp_sum_u64(t.bad);
  if (lane_id() == 0) {
    if (t.cnt) atomicAdd(count, t.cnt);
    if (t.work && work) atomicAdd(work, t.work);
    if (t.bad) atomicAdd(bad, t.bad);
  }
}

__global__ void __launch_bounds__(kHeavyThreads, 3)
    tri_heavy_kernel(const int64_t *__restrict__ off, const uint32_t *__restrict__ col, int64_t nnz,
                     const uint32_t *__restrict__ heavy, const unsigned long long *__restrict__ nheavy_p,
                     int64_t bits, unsigned long long *__restrict__ count, unsigned long long *__restrict__ work,
                     unsigned long long *__restrict__ bad, unsigned long long *__restrict__ cursor, const unsigned *__restrict__ run_if) {
  if (tri::skipped(run_if, 0u)) return;
  extern __shared__ uint32_t bm[];
  __shared__ long long sel;
  const int64_t nwords = bits >> 5;  // bits is a power of two >= 32
  const uint32_t wmask = static_cast<uint32_t>(nwords - 1);
  const unsigned long long nheavy = *nheavy_p;
  if (nheavy == 0) return;
  for (int64_t w = threadIdx.x; w < nwords; w += kHeavyThreads) bm[w] = 0;
  tri::Tally t;
  for (;;) {
    __syncthreads();  // sel may be rewritten
    if (threadIdx.x == 0) {
      const unsigned long long r = atomicAdd(cursor, 1ull);
      sel = r < nheavy ? static_cast<long long>(heavy[r]) : -1ll;
    }
    __syncthreads();
    const long long i = sel;
    if (i < 0) break;
    tri::heavy_row<uint32_t, kHeavyThreads>(off, col, i, nnz, bm, wmask, t);
  }
  flush_tally(t, count, work, bad);
}

__global__ void __launch_bounds__(kLightThreads)
    tri_light_kernel(const int64_t *__restrict__ off, const uint32_t *__restrict__ col, int64_t n, int64_t nnz,
                     int64_t bits, unsigned long long *__restrict__ count, unsigned long long *__restrict__ work,
                     unsigned long long *__restrict__ bad, unsigned long long *__restrict__ cursor,
                     int rows_per_fetch, const uint32_t *__restrict__ list,
                     const unsigned long long *__restrict__ nlist, const unsigned *__restrict__ run_if) {
  if (tri::skipped(run_if, 0u)) return;
  if (list) n = min(n, static_cast<int64_t>(*nlist));  // the rows of the list (at most n) instead of all
  if (n == 0) return;  // before thousands of warps ask the one cursor
  __shared__ uint32_t rowbuf[kLightWarps][tri::kLightCap];
  uint32_t *rb = rowbuf[threadIdx.x >> 5];
  tri::Tally t;
  for (;;) {
    unsigned long long r0 = 0;
    if (lane_id() == 0) r0 = atomicAdd(cursor, static_cast<unsigned long long>(rows_per_fetch));
    r0 = __shfl_sync(kFull, r0, 0);
    if (r0 >= static_cast<unsigned long long>(n)) break;
    const int64_t r1 = static_cast<int64_t>(r0) + rows_per_fetch < n ? static_cast<int64_t>(r0) + rows_per_fetch : n;
    for (int64_t r = static_cast<int64_t>(r0); r < r1; r++)
      tri::light_row(off, col, list ? static_cast<int64_t>(list[r]) : r, nnz, bits, rb, t);
  }
  flush_tally(t, count, work, bad);
}

// ---------------------------------------------------------------- short rows
constexpr uint32_t kShortMax = 63;  // a valid row above this is heavy or long
static_assert(kShortMax + 1 == tri::kHeavyMinDeg, "a row is short, or long enough to be heavy");
constexpr uint32_t kRecBad = 0xffffffffu;       // record of a row with bad offsets
constexpr uint32_t kRecBadHeavy = 0xfffffffeu;  // ... which the heavy kernel counts
constexpr int kShortThreads = 256;
constexpr int kShortWarps = kShortThreads / 32;
constexpr int kGroup = 8;           // rows a warp takes at once
constexpr int kPlaces = 512;        // of a row's hash table
constexpr int kStreamLen = 64;      // longer neighbours are searched where that is the cheaper side
constexpr int kShortFlight = 2;     // 16-byte vectors in flight per lane

struct __align__(16) ShortRows {
  uint32_t col[kGroup * kShortMax];  // the rows' columns, one after another
  uint4 slot[32];
  uint8_t row[kGroup * kShortMax];   // the row (0..7) of each entry of col
};
struct __align__(512) ShortSmem {
  uint8_t table[kShortWarps][kGroup][kPlaces];  // 4 * a column's position in its row, by the column's low 9 bits
  ShortRows rows[kShortWarps];
};
constexpr uint32_t kShared = 1;       // a place that two columns of the row fall on

__device__ __forceinline__ uint32_t lds_u8(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}

// One warp-aggregated entry per flagged lane: list[k] = value while k < most.
__device__ __forceinline__ void append(bool flag, uint32_t value, uint32_t *__restrict__ list, int64_t most,
                                       unsigned long long *__restrict__ size) {
  const unsigned m = __ballot_sync(kFull, flag);
  unsigned long long at = 0;
  if (lane_id() == 0 && m) at = atomicAdd(size, static_cast<unsigned long long>(__popc(m)));
  at = __shfl_sync(kFull, at, 0) + __popc(m & ((1u << lane_id()) - 1u));
  if (flag && at < static_cast<unsigned long long>(most)) list[at] = value;
}

// rec[i] = {start, length} of row i, and the lists of heavy rows and of long
// ones (neither short nor heavy).  Offsets that do not ascend could make more
// long rows than the list holds; some row is then bad and the count with it.
__global__ void __launch_bounds__(256)
    tri_record_kernel(const int64_t *__restrict__ off, int64_t n, int64_t nnz, int64_t bits, uint2 *__restrict__ rec,
                      uint32_t *__restrict__ heavy, unsigned long long *__restrict__ nheavy,
                      uint32_t *__restrict__ longs, int64_t most_longs, unsigned long long *__restrict__ nlongs,
                      const unsigned *__restrict__ run_if) {
  if (tri::skipped(run_if, 0u)) return;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t base = static_cast<int64_t>(blockIdx.x) * blockDim.x; base < n; base += stride) {
    const int64_t i = base + threadIdx.x;
    bool h = false, lg = false;
    if (i < n) {
      const int64_t b = off[i], e = off[i + 1];
      h = tri::is_heavy(i, b, e, bits);
      if (b < 0 || e < b || e > nnz) {
        rec[i] = make_uint2(0u, h ? kRecBadHeavy : kRecBad);
      } else {
        rec[i] = make_uint2(static_cast<uint32_t>(b), static_cast<uint32_t>(e - b));
        lg = !h && e - b > kShortMax;
      }
    }
    append(h, static_cast<uint32_t>(i), heavy, n < bits ? n : bits, nheavy);
    append(lg, static_cast<uint32_t>(i), longs, most_longs, nlongs);
  }
}

// The lane owning position bb + lane of a sequence flattened over the warp
// (lane r covers [inc_r - len_r, inc_r), the prefixes strictly increasing over
// the lanes that cover anything): the lanes that end at or before bb plus
// those that end inside (bb, bb + lane].
__device__ __forceinline__ int flat_owner(uint32_t inc, uint32_t bb) {
  const unsigned lane = lane_id();
  const uint32_t a = __popc(__ballot_sync(kFull, inc <= bb));
  const uint32_t x = inc - bb;
  const uint32_t ends = __reduce_or_sync(kFull, (inc > bb && x < 32u) ? (1u << x) : 0u);
  const uint32_t o = a + __popc(ends & ((2u << lane) - 1u));
  return o < 32u ? static_cast<int>(o) : 31;
}

__device__ __forceinline__ uint32_t incl_scan_u32(uint32_t v) {
  const unsigned lane = lane_id();
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, v, o);
    if (static_cast<int>(lane) >= o) v += y;
  }
  return v;
}

// Is w in the ascending run r[0,len)?
__device__ __forceinline__ bool search_u32(const uint32_t *__restrict__ r, uint32_t len, uint32_t w) {
  uint32_t lo = 0, hi = len;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (r[mid] < w) lo = mid + 1; else hi = mid;
  }
  return lo < len && r[lo] == w;
}

// Eight consecutive rows per warp.  Their columns are staged in shared memory,
// checked, and hashed: a byte table per row gives the position in the row of
// the column with the same low 9 bits.  Then the rows of all their neighbours
// are streamed, as 16-byte vectors flattened over the lanes, and each element
// is compared with the one column it can equal: two shared-memory loads.  An
// empty place says position 0, which is harmless: a column equal to the row's
// first would have that column's own place.  Places that two columns share
// are marked and their elements looked up by a binary search.  A neighbour so
// long that searching it is far cheaper is searched instead.
//
// A row of a graph without hubs has 16 neighbours of 16 elements each, and the
// work is finding and testing them, not memory: the kernel is bound by its
// shared-memory accesses (73% of the LSU data pipe) and instruction issue
// (63%).  On the Erdos-Renyi graph of 2^20 rows and degree 32 it takes 436 us
// (the light kernel, row by row with a prefix sum and a binary search per
// element, 1354).  Measured against it: a 4096-bit filter per row and a search
// for what passes 485, a 1024-bit filter of one word per bank before the table
// 480, tables of 256 places 474 (more shared places, so more searches).
__global__ void __launch_bounds__(kShortThreads, 4)
    tri_short_kernel(const uint2 *__restrict__ rec, const uint32_t *__restrict__ col, int64_t n, uint32_t nvec_all,
                     unsigned long long *__restrict__ count, unsigned long long *__restrict__ work,
                     unsigned long long *__restrict__ bad, const unsigned *__restrict__ run_if) {
  if (tri::skipped(run_if, 0u)) return;
  extern __shared__ __align__(512) unsigned char short_smem[];
  const unsigned lane = lane_id();
  ShortRows &sm = reinterpret_cast<ShortSmem *>(short_smem)->rows[threadIdx.x >> 5];
  uint8_t(*tables)[kPlaces] = reinterpret_cast<ShortSmem *>(short_smem)->table[threadIdx.x >> 5];
  const uint32_t table_at = static_cast<uint32_t>(__cvta_generic_to_shared(tables));
  const uint32_t col_at = static_cast<uint32_t>(__cvta_generic_to_shared(sm.col));
  if (table_at & (kPlaces - 1)) {  // the addresses below are put together with an OR
    if (threadIdx.x == 0) atomicAdd(bad, 1ull);
    return;
  }
  const uint4 *__restrict__ col4 = reinterpret_cast<const uint4 *>(col);  // col is 256-byte aligned
  unsigned long long wk, nbad = 0, cnt = 0;
  // a lane's share of at most 2^32 neighbours over a full grid stays far below 2^21
  uint32_t cnt32 = 0, wk32 = 0;
  const int64_t groups = (n + kGroup - 1) / kGroup, warps = static_cast<int64_t>(gridDim.x) * kShortWarps;
  for (int64_t g = static_cast<int64_t>(blockIdx.x) * kShortWarps + (threadIdx.x >> 5); g < groups; g += warps) {
    const uint32_t r0 = static_cast<uint32_t>(g * kGroup);
    uint2 rc = make_uint2(0u, 0u);
    if (lane < kGroup && g * kGroup + lane < n) rc = rec[r0 + lane];
    if (rc.y == kRecBad) nbad++;
    const uint32_t len = rc.y <= kShortMax ? rc.y : 0u;
    const uint32_t inc = incl_scan_u32(len), ex = inc - len, tot = __shfl_sync(kFull, inc, 31);
    if (tot == 0) continue;
#pragma unroll
    for (int z = 0; z < kGroup * kPlaces / 512; z++)
      reinterpret_cast<uint4 *>(tables)[z * 32 + lane] = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    // stage, check and hash: 8 lanes per row, 4 rows at a time
    uint32_t badrows = 0;
#pragma unroll
    for (int h = 0; h < kGroup; h += 4) {
      const uint32_t r = h + (lane >> 3);
      const uint32_t s = __shfl_sync(kFull, rc.x, r), l = __shfl_sync(kFull, len, r), x = __shfl_sync(kFull, ex, r);
      for (uint32_t k = lane & 7u; k < l; k += 8) {
        const uint32_t c = col[s + k];
        const uint32_t prev = k ? col[s + k - 1] : 0u;
        if (c >= r0 + r || (k && prev >= c)) badrows |= 1u << r;
        sm.col[x + k] = c;
        sm.row[x + k] = static_cast<uint8_t>(r);
        tables[r][c & (kPlaces - 1)] = static_cast<uint8_t>(4 * k);
      }
    }
    badrows = __reduce_or_sync(kFull, badrows);
    if (lane == 0) nbad += __popc(badrows);
    __syncwarp();
    for (uint32_t p0 = 0; p0 < tot; p0 += 32) {
      const uint32_t p = p0 + lane, r = p < tot ? sm.row[p] : 0u, q = p - __shfl_sync(kFull, ex, r);
      if (p < tot) {
        uint8_t *place = &tables[r][sm.col[p] & (kPlaces - 1)];
        if (*place != 4 * q) *place = kShared;  // another column of the row wrote its position here
      }
    }
    __syncwarp();
    for (uint32_t p0 = 0; p0 < tot; p0 += 32) {
      // one neighbour per lane: position q of row r, row j = {s, l}
      const uint32_t p = p0 + lane;
      const uint32_t r = p < tot ? sm.row[p] : 0u, j = p < tot ? sm.col[p] : 0u;
      uint32_t q = p - __shfl_sync(kFull, ex, r);
      if (p >= tot) q = 0;
      uint2 rj = make_uint2(0u, 0u);
      if (q > 0 && !(badrows >> r & 1u)) rj = rec[j];
      if (rj.y >= kRecBadHeavy) {
        nbad++;
        rj.y = 0;
      }
      const uint32_t steps = 32u - __clz(rj.y + 1u);  // of a binary search in row j
      const bool search = q * steps < rj.y;           // q < 64
      wk32 += search ? q : rj.y;                      // below 2^11
      const bool far = search && rj.y > kStreamLen;
      const uint32_t nv = rj.y && !far ? ((rj.x + rj.y + 3u) >> 2) - (rj.x >> 2) : 0u;
      // the streamed neighbours to the low lanes, so their ends are distinct
      // (lengths below 2^10: q * steps >= l)
      const unsigned m = __ballot_sync(kFull, nv > 0);
      if (nv) sm.slot[__popc(m & ((1u << lane) - 1u))] = make_uint4(rj.x, rj.y | q << 16, table_at + r * kPlaces | (p - q) << 18, nv);
      __syncwarp();
      uint4 sl = make_uint4(0u, 0u, 0u, 0u);
      if (lane < static_cast<unsigned>(__popc(m))) sl = sm.slot[lane];
      __syncwarp();
      const uint32_t vinc = incl_scan_u32(sl.w), vtot = __shfl_sync(kFull, vinc, 31);
      const uint32_t rel = (sl.x >> 2) - (vinc - sl.w);  // vector index - flattened place
      for (uint32_t base = 0; base < vtot; base += 32 * kShortFlight) {
        uint4 xv[kShortFlight];
        uint32_t off[kShortFlight], len2[kShortFlight], info[kShortFlight];
#pragma unroll
        for (int u = 0; u < kShortFlight; u++) {
          const uint32_t bb = base + 32u * u;
          if (u && bb >= vtot) break;  // the same in all lanes
          const int o = flat_owner(vinc, bb);
          const uint32_t vi = __shfl_sync(kFull, rel, o) + bb + lane;
          off[u] = (vi << 2) - __shfl_sync(kFull, sl.x, o);  // wraps for elements before the row
          len2[u] = __shfl_sync(kFull, sl.y, o);
          info[u] = __shfl_sync(kFull, sl.z, o);
          const bool act = bb + lane < vtot && vi < nvec_all;
          if (!act) {  // no element of length 0 counts, but the lane still reads: row 0's table and columns
            len2[u] = 0;
            info[u] = table_at;
          }
          xv[u] = col4[act ? vi : 0u];
        }
#pragma unroll
        for (int u = 0; u < kShortFlight; u++) {
          if (u && base + 32u * u >= vtot) break;
          const uint32_t table = info[u] & 0x3ffffu, mine = col_at + (info[u] >> 18) * 4u, l = len2[u] & 0xffffu;
          uint32_t w[4] = {xv[u].x, xv[u].y, xv[u].z, xv[u].w}, at[4];
#pragma unroll
          for (int k = 0; k < 4; k++) at[k] = lds_u8(table | (w[k] & (kPlaces - 1)));
          if ((at[0] | at[1] | at[2] | at[3]) & kShared) {  // rare
#pragma unroll
            for (int k = 0; k < 4; k++)
              if (at[k] == kShared) {
                if (off[u] + k < l && search_u32(sm.col + (info[u] >> 18), len2[u] >> 16, w[k])) cnt32++;
                at[k] = 0;
                w[k] = kBadCol;  // no column
              }
          }
#pragma unroll
          for (int k = 0; k < 4; k++) {
            const uint32_t v = lds_u32(mine + at[k]);
            if (off[u] + k < l && v == w[k]) cnt32++;
          }
        }
      }
      // searched neighbours: the first q columns of the row, each in row j
      unsigned mf = __ballot_sync(kFull, far);
      while (mf) {
        const int o = __ffs(mf) - 1;
        mf &= mf - 1;
        const uint32_t fs = __shfl_sync(kFull, rj.x, o), fl = __shfl_sync(kFull, rj.y, o);
        const uint32_t fq = __shfl_sync(kFull, q, o), fx = __shfl_sync(kFull, p - q, o);
        for (uint32_t k = lane; k < fq; k += 32)
          if (search_u32(col + fs, fl, sm.col[fx + k])) cnt++;
      }
      __syncwarp();
    }
  }
  cnt = warp_sum_u64(cnt + cnt32);
  wk = warp_sum_u64(wk32);
  nbad = warp_sum_u64(nbad);
  if (lane == 0) {
    if (cnt) atomicAdd(count, cnt);
    if (wk && work) atomicAdd(work, wk);
    if (nbad) atomicAdd(bad, nbad);
  }
}

bool g_heavy_attr[64];

// Workspace: columns, heavy rows, then (short rows) the records and long rows.
struct Layout {
  size_t heavy, rec, longs, total;
  bool shorts;  // the records' starts are 32 bits
};

Layout layout(int64_t numrows, int64_t nnz) {
  auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
  const int64_t lim = numrows < tri::kHeavyBits ? numrows : tri::kHeavyBits;
  Layout l;
  l.shorts = nnz < 0xffffff00ll;
  l.heavy = up(static_cast<size_t>(nnz > 0 ? nnz : 1) * sizeof(uint32_t));
  l.rec = l.heavy + static_cast<size_t>(lim > 0 ? lim : 1) * sizeof(uint32_t);
  if (!l.shorts) {
    l.longs = l.total = l.rec;
    return l;
  }
  l.rec = up(l.rec);
  l.longs = l.rec + up(static_cast<size_t>(numrows) * sizeof(uint2));
  l.total = l.longs + (static_cast<size_t>(nnz) / (kShortMax + 1) + 1) * sizeof(uint32_t);
  return l;
}

}  // namespace

size_t tri_hybrid_workspace_bytes(int64_t numrows, int64_t nnz) { return layout(numrows, nnz).total; }

static int launch_convert(const int64_t *nonzero, int64_t nnz, uint32_t *col32, cudaStream_t stream,
                          const unsigned *run_if) {
  if (nnz <= 0) return BALE_OK;
  const int64_t blocks = std::min<int64_t>((nnz + 255) / 256, static_cast<int64_t>(num_sms()) * 8);
  tri_convert_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(nonzero, nnz, col32, run_if);
  BALE_CUDA_OK(cudaGetLastError());
  return BALE_OK;
}

int tri_hybrid_prepare(const int64_t *offset, const int64_t *nonzero, int64_t numrows, int64_t nnz,
                       uint32_t *col32, uint32_t *heavy, unsigned long long *nheavy, cudaStream_t stream,
                       const unsigned *run_if) {
  const int64_t bits = tri::bitmap_bits(numrows);
  BALE_CUDA_OK(cudaMemsetAsync(nheavy, 0, sizeof(unsigned long long), stream));
  const int rc = launch_convert(nonzero, nnz, col32, stream, run_if);
  if (rc != BALE_OK) return rc;
  const int64_t lim = numrows < bits ? numrows : bits;
  int64_t blocks = (lim + 255) / 256, cap = static_cast<int64_t>(num_sms()) * 8;
  if (blocks < 1) blocks = 1;
  tri_classify_kernel<<<static_cast<unsigned>(blocks < cap ? blocks : cap), 256, 0, stream>>>(
      offset, numrows, bits, heavy, nheavy, run_if);
  BALE_CUDA_OK(cudaGetLastError());
  return BALE_OK;
}

// The heavy kernel, then the light kernel over the list's rows (at most
// `most` of them) or, without a list, over all rows.
static int launch_heavy_light(const int64_t *offset, const uint32_t *col32, const uint32_t *heavy,
                              const unsigned long long *nheavy, int64_t numrows, int64_t nnz,
                              unsigned long long *count, unsigned long long *work, unsigned long long *bad,
                              unsigned long long *cursors, int rows_per_fetch, const uint32_t *list,
                              const unsigned long long *nlist, int64_t most, cudaStream_t stream,
                              const unsigned *run_if) {
  const int sms = num_sms();
  const int64_t bits = tri::bitmap_bits(numrows);
  {
    const size_t smem = static_cast<size_t>(bits / 32) * sizeof(uint32_t);
    const int dev = current_device();
    if (dev >= 0 && dev < 64 && !g_heavy_attr[dev]) {
      BALE_CUDA_OK(cudaFuncSetAttribute(tri_heavy_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>((tri::kHeavyBits / 32) * sizeof(uint32_t))));
      g_heavy_attr[dev] = true;
    }
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, tri_heavy_kernel, kHeavyThreads, smem) != cudaSuccess ||
        occ < 1)
      occ = 1;
    tri_heavy_kernel<<<static_cast<unsigned>(sms * occ), kHeavyThreads, smem, stream>>>(
        offset, col32, nnz, heavy, nheavy, bits, count, work, bad, cursors, run_if);
    BALE_CUDA_OK(cudaGetLastError());
  }
  if (most <= 0) return BALE_OK;
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, tri_light_kernel, kLightThreads, 0) != cudaSuccess ||
      occ < 1)
    occ = 1;
  int64_t blocks = static_cast<int64_t>(sms) * occ;
  const int64_t need = ((most + rows_per_fetch - 1) / rows_per_fetch + kLightWarps - 1) / kLightWarps;
  if (blocks > need) blocks = need > 0 ? need : 1;
  tri_light_kernel<<<static_cast<unsigned>(blocks), kLightThreads, 0, stream>>>(
      offset, col32, list ? most : numrows, nnz, bits, count, work, bad, cursors + 1, rows_per_fetch, list, nlist,
      run_if);
  BALE_CUDA_OK(cudaGetLastError());
  return BALE_OK;
}

int tri_hybrid_run(const int64_t *offset, const uint32_t *col32, const uint32_t *heavy,
                   const unsigned long long *nheavy, int64_t numrows, int64_t nnz, unsigned long long *count,
                   unsigned long long *work, unsigned long long *bad, unsigned long long *cursors,
                   int rows_per_fetch, cudaStream_t stream, const unsigned *run_if) {
  BALE_CUDA_OK(cudaMemsetAsync(cursors, 0, 2 * sizeof(unsigned long long), stream));
  return launch_heavy_light(offset, col32, heavy, nheavy, numrows, nnz, count, work, bad, cursors, rows_per_fetch,
                            nullptr, nullptr, numrows, stream, run_if);
}

int launch_triangle_hybrid(const int64_t *offset, const int64_t *nonzero, int64_t numrows, int64_t nnz,
                           unsigned long long *count, unsigned long long *work, unsigned long long *bad,
                           void *ws, unsigned long long *words, int rows_per_fetch, cudaStream_t stream,
                           const unsigned *run_if) {
  // words: [0] heavy-list length, [1] heavy cursor, [2] light cursor, [3] long-list length
  const Layout l = layout(numrows, nnz);
  char *p = static_cast<char *>(ws);
  uint32_t *col32 = reinterpret_cast<uint32_t *>(p), *heavy = reinterpret_cast<uint32_t *>(p + l.heavy);
  if (!l.shorts) {
    int rc = tri_hybrid_prepare(offset, nonzero, numrows, nnz, col32, heavy, words, stream, run_if);
    if (rc != BALE_OK) return rc;
    return tri_hybrid_run(offset, col32, heavy, words, numrows, nnz, count, work, bad, words + 1, rows_per_fetch,
                          stream, run_if);
  }
  uint2 *rec = reinterpret_cast<uint2 *>(p + l.rec);
  uint32_t *longs = reinterpret_cast<uint32_t *>(p + l.longs);
  const int64_t sms = num_sms(), bits = tri::bitmap_bits(numrows);
  BALE_CUDA_OK(cudaMemsetAsync(words, 0, 4 * sizeof(unsigned long long), stream));
  int rc = launch_convert(nonzero, nnz, col32, stream, run_if);
  if (rc != BALE_OK) return rc;
  tri_record_kernel<<<static_cast<unsigned>(std::min<int64_t>((numrows + 255) / 256, sms * 8)), 256, 0, stream>>>(
      offset, numrows, nnz, bits, rec, heavy, words, longs, nnz / (kShortMax + 1) + 1, words + 3, run_if);
  BALE_CUDA_OK(cudaGetLastError());
  const int smem = static_cast<int>(sizeof(ShortSmem));
  BALE_CUDA_OK(cudaFuncSetAttribute(tri_short_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const int64_t groups = (numrows + kGroup - 1) / kGroup;
  tri_short_kernel<<<static_cast<unsigned>(std::min<int64_t>((groups + kShortWarps - 1) / kShortWarps, sms * 4)),
                     kShortThreads, smem, stream>>>(rec, col32, numrows, static_cast<uint32_t>((nnz + 3) / 4), count,
                                                    work, bad, run_if);
  BALE_CUDA_OK(cudaGetLastError());
  return launch_heavy_light(offset, col32, heavy, words, numrows, nnz, count, work, bad, words + 1, rows_per_fetch,
                            longs, words + 3, nnz / (kShortMax + 1) + 1, stream, run_if);
}

}  // namespace bale
