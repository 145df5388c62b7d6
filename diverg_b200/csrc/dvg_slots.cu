// dvg_slots.cu -- chains of range products in the row-slot format.
//
// An index build or a power is a chain of up to 24 products whose intermediate
// matrices nobody sees, and on a sequence graph nearly every row of every one
// of them is a single run of columns.  In range CRS such a row costs a row
// pointer and a range to write, two row pointers and a range to read, and the
// order in which rows are stored makes each product wait for the sizes of the
// rows before.  Here an intermediate matrix is one 8-byte slot (x, y) a row
// instead:
//   x <= y               the run of columns x .. y
//   (1, 0)               no column
//   y + 1 < x < kMulti   the two columns y and x
//   x >= kMulti          x - kMulti ranges from place y of an arena that the
//                        whole chain shares
// A row is then one load to read, one store to write, its position is its
// number, and no product needs a prefix, a look-back or another block's
// result.  Only the last pass counts its ranges, and k_slots_to_crs turns it
// into range CRS.
//
// Rows are canonical (sorted, disjoint, non-adjacent runs), as the reference's
// accumulators emit them (range_sparse.hpp:487-678, 1132-1442 in
// cartoonist/diverg: merge rule start <= hi + 1), so the chain's result is the
// matrix that the reference's sequence of range_spgemm / range_spadd gives.
//
// Measured on a B200 against the same builds product by product in range CRS:
// 5.0e7 loci, window [400, 600]: 23.05 -> 2.62 ms; 1e6 loci, [0, 250]: 1.26 ->
// 0.21 ms; 1e5 loci of a variant-dense graph, [100, 300]: 1.01 -> 0.145 ms.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "dvg_device.cuh"
#include "dvg_slots.h"

namespace dvg {
namespace {

constexpr int kSThreads = 256;  // streaming kernels
constexpr int kSWarps = kSThreads / 32;
constexpr int kWThreads = 128;  // kernels that walk rows
constexpr int kWWarps = kWThreads / 32;
constexpr int kWBlocks = 7;     // of them an SM holds at once (72 registers a thread)
constexpr int kSRows = 4;       // rows a lane of k_chain_rows takes
constexpr int kSRuns = 8;       // runs of a lane's list
constexpr int kSWin = 256;      // window words of a warp (8,192 columns)
// A run of a lane's list has at most so many columns; the 32 lanes of a warp share the
// columns of a row with a longer one.
constexpr uint32_t kLaneColumns = 256;
constexpr uint32_t kMulti = kSlotMulti;
constexpr uint32_t kMultiMax = 0xFFFFFFFFu - kMulti - 1;  // ranges of one row
constexpr unsigned long long kArenaFull = 1, kLongRow = 2, kWideRows = 4;  // why a chain is given up
// Unions by windows cost a warp about 1 us for every 32 rows that they name and window
// that they fill, twice.  A chain may spend kWideCost and a sixteenth of its rows on
// them, and one union name kWideColumns: a few rows that reach far cost little, but with
// one range of 20,000 columns in 2e5 rows a build for [100, 300] took 364 ms, in range
// CRS 58.
constexpr uint64_t kWideCost = 1u << 14;
constexpr uint32_t kWideColumns = 1u << 12;
constexpr uint32_t kCountRows = 32 * kSRows;  // rows whose ranges the last pass counts together
constexpr uint32_t kSmallRows = 1u << 17;     // rows up to which a pass is one kernel
constexpr double kChainReach = 1.28;          // branching * steps of a pass's left factors
// A result of up to so many rows gets room for two ranges a row and is written
// before its size is known, so that the host waits once.  A second wait and the
// gap before it are 20 us: from 2^24 rows on, under 3 % of a product.  An index, which
// its holder keeps, gets room for an eighth more ranges a row than the context's last
// one had, and kEarlySpare: rows of windows that a graph's runs fill are one range.
constexpr uint32_t kEarlyRows = 1u << 24;
constexpr double kEarlySlack = 1.125;
constexpr uint64_t kEarlySpare = 1u << 16;
constexpr uint32_t kQueueRows = 1u << 15;  // places of a queue (rows past them are walked at once)
constexpr size_t kQueueBytes = kQueueRows * sizeof(unsigned long long);
// Ranges a row that an arena is made for at most (4 at first: the builds of 1e6 bases of a
// variant-dense graph take up to 0.3, up to [1000, 1300] 1.1, A^300 1.1 and A^1000 4.3;
// those of a chromosome 0.05).
constexpr double kSlotGrowthMax = 8.0;
// Up to so many rows, and for single products as long as their results are written
// early, the chain's kernels are launched close behind one another: the next one's
// blocks are placed while the kernel before ends, 2 us a kernel.  Builds of
// 2e3 nodes 96 -> 82 us, 1e5 158 -> 143, 1.5e6 233 -> 208, 3e6 344 -> 330, but 6e6 511
// -> 523 and 5e7 2.64 -> 2.94 ms: blocks that wait take places of blocks that work.
// A^2 at 1.5e6 rows 64 -> 56 us, 6e6 119 -> 114, 1.2e7 193 -> 185.  Kernels of a
// batch, in a CUDA graph, gained nothing.
constexpr uint32_t kCloseRows = 1u << 22;
// A single product goes through slots from so many rows on.  The conversions are
// launches of their own, 3 to 7 us more than the row kernel's one at 1e4 rows, equal
// at 2e4; A^2 of a sequence graph's A takes 39 in place of 62 us at 1e5 rows, 54 of
// 83 at 1e6, 166 of 223 at 1e7 and 546 of 785 at 4e7.  With two different factors,
// both converted: 41, 58, 218 and 732 us against 63, 83, 233 and 823.
constexpr uint32_t kProductRows = 3u << 13;
constexpr int kCrsRows = kSlotPartRows;        // rows of a block of the conversions
constexpr uint32_t kSuperGroups = 512;        // counts that k_slot_sums adds up

__device__ __forceinline__ uint2 empty_slot() { return make_uint2(1u, 0u); }
__device__ __forceinline__ bool is_multi(uint2 s) { return s.x >= kMulti; }
// Every load of what a kernel of the same chain wrote is an ordinary one: a close
// chain's kernels (kCloseRows) start while the one before still writes, and the
// read-only path is for memory that nothing writes from a kernel's start on.  After
// follow() an ordinary load sees all that the kernels before wrote.  (Read-only loads
// in a chain that is not close: 170 against 153 us for a build of 1e5 bases, 231
// against 217 for A^100 of 1e6; ordinary loads by __ldca: 186 and 276.)
__device__ __forceinline__ uint2 ld_slot(const uint2* p, size_t i) { return p[i]; }
__device__ __forceinline__ bool is_run(uint2 s) { return s.x <= s.y; }
__device__ __forceinline__ uint32_t slot_count(uint2 s) {
  return is_run(s) ? 1u : is_multi(s) ? s.x - kMulti : s.x == s.y + 1 ? 0u : 2u;
}
// Range t of a slot that has it.
__device__ __forceinline__ uint2 slot_range(const uint2* arena, uint2 s, uint32_t t) {
  if (is_multi(s)) return arena[s.y + t];
  if (is_run(s)) return s;
  return t ? make_uint2(s.x, s.x) : make_uint2(s.y, s.y);
}
// The slot of the two columns or equal columns c and d.
__device__ __forceinline__ uint2 pair_slot(uint32_t c, uint32_t d) {
  const uint32_t lo = min(c, d), hi = max(c, d);
  return hi - lo <= 1 ? make_uint2(lo, hi) : make_uint2(hi, lo);
}

// v |= w for two runs that overlap or touch; false, v unchanged, for any other
// two slots.  Columns are below kMulti, so y + 1 does not wrap.
__device__ __forceinline__ bool unite(uint2& v, uint2 w) {
  if (!is_run(v) || !is_run(w) || w.x > v.y + 1 || v.x > w.y + 1) return false;
  v.x = min(v.x, w.x);
  v.y = max(v.y, w.y);
  return true;
}

// One pass: with S_0 = I and S_(j+1) = S_j M_j,
//   s = S_k                         (where s is not null)
//   c = union of S_j B over bits j  (where c is not null; B null: the identity)
struct ChainArgs {
  const uint2* m[kChainMax];
  const uint2* b;
  uint2* s;
  uint2* c;
  uint32_t k, bits;
  uint2* arena;
  unsigned long long* top;    // ranges taken from the arena
  uint64_t arena_cap;
  DeviceControl* ctl;
  // Why the chain is given up (kArenaFull, ...), 0: it is not.  The host drops the result;
  // until then rows that did not fit, and those that a warp would have to walk, are left
  // empty, so that later passes stay in bounds and are over soon.  (Lanes' walks do not
  // look: that took up to 4 % of a small chain, A^129 of 2.7e5 bases 163 -> 169 us.)
  unsigned long long* abort;
  unsigned long long* wide;   // what unions by windows have cost, and may
  unsigned long long wide_max;
  uint32_t* masks;            // bit r % 32 of word r / 32: k_chain_rows left row r to k_chain_walk
  unsigned long long* queue;  // rows that a warp walks, and of this pass how many places
  uint32_t* taken;            // were taken (taken[0]) and filled (taken[1])
  uint32_t epoch;             // the pass's: what it puts into the queue has it in the upper half
  uint32_t queue_cap;
  uint32_t* group_cnt;        // last pass: ranges and columns of c per kCountRows rows
  unsigned long long* group_nnz;
  bool add_counts;            // the last pass's blocks add to them (from zero)
  uint32_t n;
};

// U * 32 rows from r0, all of them rows of the matrix: those that are one or
// two columns in every S_j on the way, as nearly all rows of a sequence graph's
// powers are.  A row of one column takes the next factor's row (at the end: B's)
// as it is -- a row of several ranges keeps its place in the arena, rows are
// never rewritten; a row of two takes two rows of one column each.  Returns the
// rows that do not go through (bit u: row r0 + u * 32 + lane).
template <bool OUTS, bool OUTC, bool COUNT, int U>
__device__ __forceinline__ uint32_t chain_rows(const ChainArgs& p, uint32_t r0, uint32_t& cnt,
                                               unsigned long long& nnz) {
  const uint32_t r = r0 + lane_id();
  uint32_t at[U], at2[U], bad = 0, two = 0;  // a row's column or two (bit u of two); of a bad row, its own number
  uint2 acc[U];
  bool pairs = false;                        // some row of the warp has two
  bool have = OUTC && (p.bits & 1u) != 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    at[u] = at2[u] = r + u * 32;
    acc[u] = have && p.b ? ld_slot(p.b, at[u]) : make_uint2(at[u], at[u]);
  }
  if (have && (p.bits & ~1u)) {  // only runs are united below
#pragma unroll
    for (int u = 0; u < U; ++u) bad |= (is_run(acc[u]) ? 0u : 1u) << u;
  }
#pragma unroll 1
  for (uint32_t j = 0; j < p.k; ++j) {
    const uint2* mat = p.m[j];
    const bool last = j + 1 == p.k, gather = OUTC && ((p.bits >> (j + 1)) & 1u);
    uint2 s[U];
#pragma unroll
    for (int u = 0; u < U; ++u) s[u] = ld_slot(mat, at[u]);
    if (pairs) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!((two >> u) & 1u)) continue;
        const uint2 t = ld_slot(mat, at2[u]);
        if (s[u].x == s[u].y && t.x == t.y) {
          s[u] = pair_slot(s[u].x, t.x);
        } else {  // (a marker is no column: never followed)
          bad |= 1u << u;
          s[u] = make_uint2(r + u * 32, r + u * 32);
        }
      }
    }
    if (OUTS && last) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (!((bad >> u) & 1u)) p.s[size_t(r) + u * 32] = s[u];
    }
    if (last && !gather) break;
    uint32_t odd = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      odd |= s[u].x ^ s[u].y;
      at[u] = s[u].x;
    }
    pairs = __any_sync(kFullMask, odd != 0);
    if (pairs) {
      two = 0;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        // one column, two neighbours, or two apart: x and y are the columns
        const bool ok = is_run(s[u]) ? s[u].y - s[u].x <= 1 : s[u].x - s[u].y >= 2 && !is_multi(s[u]);
        bad |= (ok ? 0u : 1u) << u;
        const bool gone = (bad >> u) & 1u;
        two |= (!gone && s[u].x != s[u].y ? 1u : 0u) << u;
        at[u] = gone ? r + u * 32 : s[u].x;
        at2[u] = s[u].y;
      }
    }
    if (gather) {
#pragma unroll
      for (int u = 0; u < U; ++u) s[u] = p.b ? ld_slot(p.b, at[u]) : make_uint2(at[u], at[u]);
      if (pairs) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (!((two >> u) & 1u)) continue;
          if (!unite(s[u], p.b ? ld_slot(p.b, at2[u]) : make_uint2(at2[u], at2[u]))) bad |= 1u << u;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (have) {
          const bool touch = s[u].x <= min(s[u].y, acc[u].y + 1) && acc[u].x <= s[u].y + 1;
          bad |= (touch ? 0u : 1u) << u;
          acc[u].x = min(acc[u].x, s[u].x);
          acc[u].y = max(acc[u].y, s[u].y);
        } else {
          acc[u] = s[u];
        }
      }
      have = true;
    }
  }
  if (OUTC) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if ((bad >> u) & 1u) continue;
      p.c[size_t(r) + u * 32] = acc[u];
      if (COUNT) {
        const uint32_t c = slot_count(acc[u]);
        cnt += c;
        for (uint32_t t = 0; t < c; ++t) {
          const uint2 v = slot_range(p.arena, acc[u], t);
          nnz += v.y - v.x + 1;
        }
      }
    }
  }
  return bad;
}

// ---- rows that need more than that -------------------------------------------

// A warp's shared memory: the rows it walks next, and the lists of its
// walks (entry k of lane t at [k * 32 + t]) or, for rows of more runs than
// those hold, a row's bitmaps (bitmap_row) or a bitmap window (warp_union).
constexpr int kRowWords = 320;  // words of S_j: 10,240 columns
constexpr int kSumWords = 384;  // and of c: 12,288 columns
constexpr uint32_t kRowBack = 64 * 32;  // columns that a bitmap has before the first one it gets
struct WarpSmem {
  union {
    uint2 list[3][kSRuns * 32];
    struct {
      uint32_t bits[kSWin], reach[kSWin];
    } win;
    struct {
      uint32_t s[2][kRowWords], c[kSumWords];
      uint16_t cols[32 * 32];
    } row;
  };
  uint32_t todo[32];
};

// Merges v into the nr runs at L; returns their new number, or kFull.
constexpr uint32_t kFull = 0xffffffffu;
__device__ __noinline__ uint32_t list_merge(uint2* L, uint32_t nr, uint2 v) {
  if (nr == 0 || L[(nr - 1) * 32].y + 1 < v.x) {  // past the last run
    if (nr == uint32_t(kSRuns)) return kFull;
    L[nr * 32] = v;
    return nr + 1;
  }
  uint32_t k = 0;
  while (L[k * 32].y + 1 < v.x) ++k;
  if (v.y + 1 < L[k * 32].x) {
    if (nr == uint32_t(kSRuns)) return kFull;
    for (uint32_t m = nr; m > k; --m) L[m * 32] = L[(m - 1) * 32];
    L[k * 32] = v;
    return nr + 1;
  }
  uint2 w = L[k * 32];
  w.x = min(w.x, v.x);
  w.y = max(w.y, v.y);
  uint32_t m = k + 1;
  while (m < nr && w.y + 1 >= L[m * 32].x) {
    w.y = max(w.y, L[m * 32].y);
    ++m;
  }
  L[k * 32] = w;
  const uint32_t gone = m - k - 1;
  if (gone)
    for (uint32_t q = m; q < nr; ++q) L[(q - gone) * 32] = L[q * 32];
  return nr - gone;
}

// The nd runs at D |= the rows of `mat` that the ns runs at L name (mat null:
// the runs themselves).  Returns their new number, or kFull: too many runs, or one
// too long for a lane.
__device__ __noinline__ uint32_t list_product(const uint2* arena, const uint2* L, uint32_t ns, const uint2* mat,
                                              uint2* D, uint32_t nd) {
  uint2 run = empty_slot();
  for (uint32_t k = 0; k < ns; ++k) {
    const uint2 a = L[k * 32];
    if (a.y - a.x >= kLaneColumns && mat) return kFull;
    for (uint32_t x = a.x; x <= a.y; ++x) {
      const uint2 s = mat ? ld_slot(mat, x) : a;
      const uint32_t c = slot_count(s);
      for (uint32_t t = 0; t < c; ++t) {
        const uint2 v = slot_range(arena, s, t);
        // extends the open run, or merges it into the list and opens another
        if (v.x <= run.y + 1 && run.x <= v.y + 1) {
          run.x = min(run.x, v.x);
          run.y = max(run.y, v.y);
        } else {
          if (run.x <= run.y) {
            nd = list_merge(D, nd, run);
            if (nd == kFull) return kFull;
          }
          run = v;
        }
      }
      if (!mat) break;
    }
  }
  return run.x <= run.y ? list_merge(D, nd, run) : nd;
}

// The quick form of a walk.  The columns that a row's S_j holds lie close
// together -- the ends of paths of one length -- so they are a 64-bit mask from
// a base column, and a product ORs the named rows' ranges into the next mask.
// A product's loads -- the named rows of the factor and, where c takes S_j, of B --
// are requested together, two columns at a time, so a factor is one trip to memory
// for most rows, and one copy of the code handles the columns in turn.  The walk of
// a row is a chain of such trips, and the slowest warp's chain bounds a small pass.
// (Against a separate form for rows of a single column, then two trips a factor:
// 238 -> 220 us for A^10 at 1e6 nodes, 193 -> 178 for the build at 1e5; 3, 4 and 6
// columns at a time cost up to 6 % more.)  c's row is at most two runs in registers.
// Writes the runs of s and c to the lists; false where the row does not fit.
template <bool OUTS, bool OUTC>
__device__ __forceinline__ bool quick_row(const ChainArgs& p, uint32_t row, uint2* Ls, uint32_t& ns, uint2* Lc,
                                          uint32_t& nc) {
  constexpr int kAhead = 2;
  unsigned long long mask = 1ull;
  uint32_t base = row;
  uint2 r0 = empty_slot(), r1 = empty_slot();
  bool ok = true;
  auto add_c = [&](uint2 v) {
    if (!is_run(r0)) {
      r0 = v;
    } else if (unite(r0, v)) {
      if (unite(r0, r1)) r1 = empty_slot();
    } else if (!is_run(r1)) {
      r1 = r0;
      r0 = v;
    } else if (unite(r1, v)) {
      if (unite(r0, r1)) r1 = empty_slot();
    } else {
      ok = false;
    }
  };
#pragma unroll 1
  for (uint32_t j = 0;; ++j) {
    const bool gather = OUTC && ((p.bits >> j) & 1u), go = j < p.k;
    if (!gather && !go) break;
    const uint2* mat = go ? p.m[j] : nullptr;
    unsigned long long to = 0;
    uint32_t from = 0;
    auto add_s = [&](uint2 v) {
      if (!to) from = v.x > 16 ? v.x - 16 : 0;  // later rows may start a little before the first
      const uint32_t lo = v.x - from, hi = v.y - from;
      if (lo > 63 || hi > 63) {
        ok = false;
        return;
      }
      to |= (~0ull << lo) & (~0ull >> (63 - hi));
    };
    for (unsigned long long w = mask; w;) {
      uint32_t x[kAhead];
      uint2 sm[kAhead], sb[kAhead];
      int n = 0;
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        x[q] = base + uint32_t(__ffsll(w) - 1);
        n += w ? 1 : 0;
        w &= w - 1;
      }
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        sm[q] = go && q < n ? ld_slot(mat, x[q]) : empty_slot();
        sb[q] = gather && q < n ? (p.b ? ld_slot(p.b, x[q]) : make_uint2(x[q], x[q])) : empty_slot();
      }
#pragma unroll 1
      for (int q = 0; q < n; ++q) {  // (one copy of the code for the columns in turn)
        const uint2 s = sm[0], b = sb[0];
#pragma unroll
        for (int i = 0; i + 1 < kAhead; ++i) {
          sm[i] = sm[i + 1];
          sb[i] = sb[i + 1];
        }
        if (is_run(s)) {
          add_s(s);
        } else {
          const uint32_t c = slot_count(s);
          for (uint32_t t = 0; t < c; ++t) add_s(slot_range(p.arena, s, t));
        }
        if (is_run(b)) {
          add_c(b);
        } else {
          const uint32_t c = slot_count(b);
          for (uint32_t t = 0; t < c; ++t) add_c(slot_range(p.arena, b, t));
        }
      }
    }
    if (!go || !ok) break;
    mask = to;
    base = from;
  }
  if (!ok) return false;
  if (OUTS) {
    ns = 0;
    for (unsigned long long w = mask; w;) {
      const int lo = __ffsll(w) - 1, n = __ffsll(~(w >> lo)) - 1;  // (n < 0: all 64 columns)
      const int hi = n < 0 ? 63 : lo + n - 1;
      if (ns == uint32_t(kSRuns)) return false;
      Ls[ns++ * 32] = make_uint2(base + lo, base + hi);
      w &= hi < 63 ? ~0ull << (hi + 1) : 0ull;
    }
  }
  if (OUTC) {
    if (is_run(r1) && r1.x < r0.x) {
      const uint2 t = r0;
      r0 = r1;
      r1 = t;
    }
    nc = 0;
    if (is_run(r0)) Lc[nc++ * 32] = r0;
    if (is_run(r1)) Lc[nc++ * 32] = r1;
  }
  return true;
}

__device__ __forceinline__ bool given_up(const ChainArgs& p) { return __ldcg(p.abort) != 0; }

// The union of the rows of `mat` that the slot `left` names (mat null: none)
// and of the slots d and e, by a warp, any number of runs: bitmap windows over
// the columns that its ranges cover, the next window starting at the first
// column past the last one.  Returns the row's slot (uniform); of
// no column where the chain is given up, for the union's own cost or another reason.
// The arena is read past L1: a slot may be one that this warp has just written.
__device__ uint2 warp_union(const ChainArgs& p, uint2 left, const uint2* mat, uint2 d, uint2 e,
                            uint32_t* bits, uint32_t* reach) {
  const int lane = lane_id();
  // every range of the union, spread over the lanes
  auto each = [&](auto&& f) {
    auto range = [&](uint2 s, uint32_t t) { return is_multi(s) ? __ldcg(p.arena + s.y + t) : slot_range(p.arena, s, t); };
    for (uint2 s : {d, e}) {
      const uint32_t c = slot_count(s);
      for (uint32_t t = lane; t < c; t += 32) f(range(s, t));
    }
    if (!mat) return;
    auto rows = [&](uint64_t x, uint32_t end, uint32_t step) {
      for (; x <= end; x += step) {
        const uint2 s = ld_slot(mat, x);
        const uint32_t c = slot_count(s);
        for (uint32_t t = 0; t < c; ++t) f(range(s, t));
      }
    };
    // a lane takes whole short ranges of the left row; the warp shares the long ones
    const uint32_t c = slot_count(left);
    for (uint32_t t0 = 0; t0 < c; t0 += 32) {
      const uint2 r = t0 + lane < c ? range(left, t0 + lane) : empty_slot();
      const bool is_long = is_run(r) && r.y - r.x >= 32;
      if (is_run(r) && !is_long) rows(r.x, r.y, 1);
      for (unsigned m = __ballot_sync(kFullMask, is_long); m; m &= m - 1) {
        const int q = __ffs(m) - 1;
        const uint32_t x = __shfl_sync(kFullMask, r.x, q), y = __shfl_sync(kFullMask, r.y, q);
        rows(uint64_t(x) + lane, y, 32);
      }
    }
  };
  auto give_up = [&](unsigned long long why) {
    if (lane == 0) atomicOr(p.abort, why);
    return empty_slot();
  };
  if (__any_sync(kFullMask, given_up(p))) return empty_slot();
  uint32_t named = 0;  // rows (at most kWideColumns + 1 counted of a range)
  for (uint32_t t = lane, c = mat ? slot_count(left) : 0; t < c; t += 32) {
    const uint2 r = is_multi(left) ? __ldcg(p.arena + left.y + t) : slot_range(p.arena, left, t);
    named = min(named + min(r.y - r.x, kWideColumns) + 1, kWideColumns + 1);
  }
  named = __reduce_add_sync(kFullMask, named);
  if (named > kWideColumns) return give_up(kWideRows);
  uint32_t first = 0xffffffffu, end = 0;
  each([&](uint2 v) {
    first = min(first, v.x);
    end = max(end, v.y);
  });
  __syncwarp();
  first = __reduce_min_sync(kFullMask, first);
  end = __reduce_max_sync(kFullMask, end);
  if (first == 0xffffffffu) return empty_slot();
  const unsigned long long cost = 2ull * (named / 32 + 1) * ((end - first) / (32 * kSWin) + 1);
  unsigned long long spent = 0;
  if (lane == 0) spent = atomicAdd(p.wide, cost);
  if (__shfl_sync(kFullMask, spent, 0) + cost > p.wide_max) return give_up(kWideRows);
  uint64_t off = 0;
  uint32_t total = 0;
  for (int pass = 0; pass < 2; ++pass) {  // count, then write to the arena
    uint32_t count = 0;                   // runs begun
    uint2 open = empty_slot();            // y: the last column, where a run goes on past the words so far
    uint32_t next = first;
    while (next != 0xffffffffu) {
      const uint64_t cb = next & ~31u, ce = cb + 32ull * kSWin - 1;
      // the words that the union can cover, in whole turns of the warp
      const uint32_t words = min(uint32_t(kSWin), uint32_t((end - cb) / 1024 + 1) * 32);
      for (uint32_t w = lane; w < words; w += 32) bits[w] = reach[w] = 0;
      __syncwarp();
      uint32_t after = 0xffffffffu;  // the first covered column past the window
      each([&](uint2 v) {
        if (uint64_t(v.y) > ce) after = min(after, max(v.x, uint32_t(ce + 1)));
        if (uint64_t(v.y) < cb || uint64_t(v.x) > ce) return;
        const uint32_t s = uint32_t(max(uint64_t(v.x), cb) - cb), t = uint32_t(min(uint64_t(v.y), ce) - cb);
        const uint32_t ws = s >> 5, we = t >> 5;
        const uint32_t lo = ~0u << (s & 31), hi = ~0u >> (31 - (t & 31));
        if (ws == we) {
          atomicOr(bits + ws, lo & hi);
        } else {
          atomicOr(bits + ws, lo);
          atomicOr(bits + we, hi);
          if (we > ws + 1) atomicMax(reach + ws + 1, we);
        }
      });
      after = group_min<32>(kFullMask, after);
      __syncwarp();
      uint32_t run_reach = 0;
      for (uint32_t wb = 0; wb < words; wb += 32) {
        const uint32_t w = wb + lane;
        uint32_t x = bits[w];
        const uint32_t rr = max(group_incl_max<32>(kFullMask, reach[w], lane), run_reach);
        if (rr > w) x = ~0u;
        run_reach = __shfl_sync(kFullMask, rr, 31);
        const uint32_t prev = __shfl_up_sync(kFullMask, x, 1), after_word = __shfl_down_sync(kFullMask, x, 1);
        const uint32_t col = uint32_t(cb) + 32 * w;
        const bool carry = lane ? (prev >> 31) : (is_run(open) && open.y + 1 == col);
        const uint32_t starts = x & ~((x << 1) | (carry ? 1u : 0u));
        const uint32_t nb = __popc(starts);
        const uint32_t incl = group_incl_sum<32>(kFullMask, nb, lane);
        if (pass == 1) {
          // starts in order; an end goes to the run that it closes, or to the
          // last one begun before this word where that goes on here
          uint32_t k = count + incl - nb;
          for (uint32_t b = starts; b; b &= b - 1) p.arena[off + k++].x = col + uint32_t(__ffs(b) - 1);
          uint32_t ends = x & ~(x >> 1);
          if (lane < 31 && (after_word & 1u)) ends &= 0x7fffffffu;  // the next word ends it
          uint32_t q = count + incl - nb - (carry && (x & 1u) ? 1u : 0u);
          for (uint32_t b = ends; b; b &= b - 1) p.arena[off + q++].y = col + uint32_t(__ffs(b) - 1);
          __syncwarp();  // the next words may prolong the last run
        }
        const uint32_t last = __shfl_sync(kFullMask, x, 31);
        count += __shfl_sync(kFullMask, incl, 31);
        open = last >> 31 ? make_uint2(0u, uint32_t(cb) + 32 * (wb + 31) + 31) : empty_slot();
      }
      __syncwarp();
      next = after;
    }
    if (pass == 0) {
      total = count;
      if (lane == 0) off = atomicAdd(p.top, (unsigned long long)total);
      off = __shfl_sync(kFullMask, off, 0);
      if (total > kMultiMax) return give_up(kLongRow);
      if (off + total > p.arena_cap) return give_up(kArenaFull);
    }
  }
  __syncwarp();
  return total == 1 ? __ldcg(p.arena + off) : make_uint2(kMulti + total, uint32_t(off));
}

// The slot of the row whose columns from `base` on the words lo .. hi of W hold, the
// first and the last of them not empty (lo > hi: no column), by a warp; its ranges and
// columns to `cnt` and `nnz`.  All uniform but nnz, a lane's share.
__device__ __forceinline__ uint2 bitmap_slot(const ChainArgs& p, const uint32_t* W, uint32_t base, uint32_t lo,
                                             uint32_t hi, uint32_t& cnt, unsigned long long& nnz) {
  const int lane = lane_id();
  cnt = 0;
  if (lo > hi) return empty_slot();
  // a lane's word of 32, and the first and last columns of its runs
  auto word = [&](uint32_t w, uint32_t& starts, uint32_t& ends) {
    const uint32_t x = w <= hi ? W[w] : 0u;
    starts = x & ~(x << 1 | (x && w > lo ? W[w - 1] >> 31 : 0u));
    ends = x & ~(x >> 1 | (x && w < hi ? W[w + 1] << 31 : 0u));
    return x;
  };
  for (uint32_t g = lo; g <= hi; g += 32) {
    uint32_t starts, ends;
    nnz += __popc(word(g + lane, starts, ends));
    cnt += __popc(starts);
  }
  cnt = __reduce_add_sync(kFullMask, cnt);
  if (cnt == 1) return make_uint2(base + 32 * lo + __ffs(W[lo]) - 1, base + 32 * hi + 31 - __clz(W[hi]));
  unsigned long long off = 0;
  if (lane == 0) off = atomicAdd(p.top, (unsigned long long)cnt);
  off = __shfl_sync(kFullMask, off, 0);
  if (off + cnt > p.arena_cap) {
    if (lane == 0) atomicOr(p.abort, kArenaFull);
    cnt = 0;
    return empty_slot();
  }
  uint32_t k = 0, q = 0;
  for (uint32_t g = lo; g <= hi; g += 32) {
    uint32_t starts, ends;
    word(g + lane, starts, ends);
    // (starts and ends up to this lane's word, 16 bits each: a turn has at most 512)
    const uint32_t mine = __popc(starts) | __popc(ends) << 16;
    const uint32_t incl = group_incl_sum<32>(kFullMask, mine, lane), all = __shfl_sync(kFullMask, incl, 31);
    const uint32_t col = base + 32 * (g + lane);
    uint32_t a = k + ((incl - mine) & 0xffffu), b = q + ((incl - mine) >> 16);
    for (; starts; starts &= starts - 1) p.arena[off + a++].x = col + uint32_t(__ffs(starts) - 1);
    for (; ends; ends &= ends - 1) p.arena[off + b++].y = col + uint32_t(__ffs(ends) - 1);
    k += all & 0xffffu;
    q += all >> 16;
  }
  return make_uint2(kMulti + cnt, uint32_t(off));
}

// A row by a warp: S_j and c as bitmaps in shared memory, each from a column a little
// before the first one that it gets.  The columns of S_j are laid out in a list, and a
// lane takes every 32nd of them: its rows of the factor and of B are requested together,
// so that a factor is one trip to memory for 32 columns (two, for rows in the arena).
// False where the columns lie further apart than the bitmaps reach.
//
// Bound: those trips, about 1.5 us a factor.  Unions by windows instead (warp_union)
// read every row three times and scan up to 8,192 columns twice, 8 us each and one for
// every S_j and sum, all of them kept in the arena.
template <bool OUTS, bool OUTC>
__device__ bool bitmap_row(const ChainArgs& p, WarpSmem& M, uint32_t row, uint2& s, uint2& c, uint32_t& nc,
                           unsigned long long& z) {
  const int lane = lane_id();
  uint32_t *S = M.row.s[0], *T = M.row.s[1], *const C = M.row.c;
  for (uint32_t w = lane; w < uint32_t(kSumWords); w += 32) C[w] = 0;
  uint32_t sbase = row & ~31u, s_lo = 0, s_hi = 0;  // S's first column; its words that hold any
  if (lane == 0) S[0] = 1u << (row & 31u);
  uint32_t cbase = 0, c_lo = 0xffffffffu, c_hi = 0;
  bool c_any = false;
  __syncwarp();
#pragma unroll 1
  for (uint32_t j = 0;; ++j) {
    const bool gather = OUTC && ((p.bits >> j) & 1u), go = j < p.k;
    if (!gather && !go) break;
    const uint2* mat = go ? p.m[j] : nullptr;
    for (uint32_t w = lane; go && w < uint32_t(kRowWords); w += 32) T[w] = 0;
    uint32_t tbase = 0, t_lo = 0xffffffffu, t_hi = 0;
    bool t_any = false, ok = true;
    // where a bitmap begins that gets these ranges first
    auto place = [&](bool has, uint2 v, uint32_t& base, bool& any) {
      const uint32_t first = __reduce_min_sync(kFullMask, has ? v.x : 0xffffffffu);
      if (first == 0xffffffffu) return;
      base = (first & ~31u) > kRowBack ? (first & ~31u) - kRowBack : 0u;
      any = true;
    };
    auto put = [&](uint32_t* W, uint32_t words, uint32_t base, uint2 v, uint32_t& lo, uint32_t& hi) {
      if (v.x < base || (v.y - base) / 32 >= words) {
        ok = false;
        return;
      }
      const uint32_t a = v.x - base, b = v.y - base, wa = a / 32, wb = b / 32;
      for (uint32_t w = wa; w <= wb; ++w)
        atomicOr(W + w, (w == wa ? ~0u << (a & 31) : ~0u) & (w == wb ? ~0u >> (31 - (b & 31)) : ~0u));
      lo = min(lo, wa);
      hi = max(hi, wb);
    };
    for (uint32_t g = s_lo; g <= s_hi; g += 32) {
      uint32_t w = g + lane <= s_hi ? S[g + lane] : 0u;
      const uint32_t incl = group_incl_sum<32>(kFullMask, uint32_t(__popc(w)), lane);
      const uint32_t total = __shfl_sync(kFullMask, incl, 31);
      uint32_t at = incl - __popc(w);
      for (; w; w &= w - 1) M.row.cols[at++] = uint16_t(32 * (g + lane) + __ffs(w) - 1);
      __syncwarp();
      for (uint32_t t0 = 0; t0 < total; t0 += 32) {
        const bool have = t0 + lane < total;
        const uint32_t x = have ? sbase + M.row.cols[t0 + lane] : 0u;
        const uint2 sm = have && go ? ld_slot(mat, x) : empty_slot();
        const uint2 sb = have && gather ? (p.b ? ld_slot(p.b, x) : make_uint2(x, x)) : empty_slot();
        const uint32_t nm = slot_count(sm), nb = slot_count(sb);
        const uint2 m0 = nm ? slot_range(p.arena, sm, 0) : empty_slot();
        const uint2 b0 = nb ? slot_range(p.arena, sb, 0) : empty_slot();
        if (go && !t_any) place(nm != 0, m0, tbase, t_any);
        if (gather && !c_any) place(nb != 0, b0, cbase, c_any);
        if (nm) put(T, kRowWords, tbase, m0, t_lo, t_hi);
        for (uint32_t q = 1; q < nm; ++q) put(T, kRowWords, tbase, slot_range(p.arena, sm, q), t_lo, t_hi);
        if (nb) put(C, kSumWords, cbase, b0, c_lo, c_hi);
        for (uint32_t q = 1; q < nb; ++q) put(C, kSumWords, cbase, slot_range(p.arena, sb, q), c_lo, c_hi);
        __syncwarp();
      }
      __syncwarp();
    }
    if (!__all_sync(kFullMask, ok)) return false;
    if (!go) break;
    uint32_t* const last = S;
    S = T;
    T = last;
    sbase = tbase;
    s_lo = __reduce_min_sync(kFullMask, t_lo);  // (no column: past s_hi, nothing is read)
    s_hi = __reduce_max_sync(kFullMask, t_hi);
    __syncwarp();
  }
  uint32_t ns = 0;
  unsigned long long zs = 0;
  if (OUTS) s = bitmap_slot(p, S, sbase, s_lo, s_hi, ns, zs);
  if (OUTC) {
    c_lo = __reduce_min_sync(kFullMask, c_lo);
    c_hi = __reduce_max_sync(kFullMask, c_hi);
    c = bitmap_slot(p, C, cbase, c_lo, c_hi, nc, z);
    z = group_sum<32>(kFullMask, z);
  }
  __syncwarp();
  return true;
}

template <bool OUTS, bool OUTC>
__device__ __forceinline__ void leave_empty(const ChainArgs& p, uint32_t r) {
  if (OUTS) p.s[r] = empty_slot();
  if (OUTC) p.c[r] = empty_slot();
}

// A row by the whole warp, however many runs it has (none, where the chain is given up);
// c's ranges and columns.  (A function of its own, so that its registers are not the
// lanes' walks'.)
struct RowCount {
  uint32_t ranges;
  unsigned long long columns;
};
template <bool OUTS, bool OUTC>
__device__ __noinline__ RowCount warp_row(const ChainArgs& p, WarpSmem& S, uint32_t r) {
  const int lane = lane_id();
  uint2 s = make_uint2(r, r), c = empty_slot();
  uint32_t k = 0;
  unsigned long long z = 0;
  if (__any_sync(kFullMask, given_up(p))) {
    if (lane == 0) leave_empty<OUTS, OUTC>(p, r);
    __syncwarp();
    return {0, 0};
  }
  if (!bitmap_row<OUTS, OUTC>(p, S, r, s, c, k, z)) {
    __syncwarp();
    s = make_uint2(r, r);
    c = empty_slot();
    for (uint32_t j = 0;; ++j) {
      if (OUTC && ((p.bits >> j) & 1u))
        c = p.b ? warp_union(p, s, p.b, c, empty_slot(), S.win.bits, S.win.reach)
                : warp_union(p, s, nullptr, c, s, S.win.bits, S.win.reach);
      if (j == p.k) break;
      s = warp_union(p, s, p.m[j], empty_slot(), empty_slot(), S.win.bits, S.win.reach);
    }
    k = OUTC ? slot_count(c) : 0;
    z = 0;
    for (uint32_t q = lane; q < k; q += 32) {
      const uint2 v = is_multi(c) ? __ldcg(p.arena + c.y + q) : slot_range(p.arena, c, q);
      z += v.y - v.x + 1;
    }
    z = group_sum<32>(kFullMask, z);
  }
  if (OUTS && lane == 0) p.s[r] = s;
  if (OUTC && lane == 0) p.c[r] = c;
  __syncwarp();
  return {k, z};
}

// Rows that a lane cannot walk are put into the pass's queue, and other warps take rows
// from it, one at a time, when their own are done: they come in clumps, all 32 of a batch
// of them, and one after another in their warp would be what the pass lasts.  A^300 of
// 1e6 bases of a variant-dense graph, 4,172 such rows: 9.9 ms by unions of windows in
// the row's own warp, 1.2 by bitmaps through the queue; A^100, 52 such rows: 1.72 ms and
// 0.24; the build for [1000, 1300], 1,910: 4.3 and 0.86.  Where no row needs it, the queue
// and the longer code cost up to 3 % of a small build (2e3 bases 84.0 -> 86.3 us).  Nobody
// waits: a place is settled by one atomic each of the warp that puts a row in and of the
// one that takes it, and where the taker comes first (kGone) the row stays with the warp
// that had it.  What earlier passes left there has another epoch and counts as empty, so
// the queue is cleared when it is made and never again.  A warp looks into the
// queue when it has walked rows: one whose rows were all quick ones is done before others
// put theirs in, and does not.
constexpr uint32_t kGone = 0xffffffffu;
__device__ __forceinline__ unsigned long long in_queue(const ChainArgs& p, uint32_t v) {
  return (unsigned long long)p.epoch << 32 | v;
}
template <bool OUTS, bool OUTC, class Tally>
__device__ void take_rows(const ChainArgs& p, WarpSmem& S, Tally&& tally) {
  for (;;) {
    const uint2 places = __ldcg(reinterpret_cast<const uint2*>(p.taken));
    if (__shfl_sync(kFullMask, places.x >= min(places.y, p.queue_cap), 0)) return;
    uint32_t r = 0;  // row + 1
    if (lane_id() == 0) {
      const uint32_t at = atomicAdd(p.taken, 1u);
      if (at < p.queue_cap) {
        const unsigned long long was = atomicExch(p.queue + at, in_queue(p, kGone));
        if (was >> 32 == p.epoch) r = uint32_t(was);
      }
    }
    r = __shfl_sync(kFullMask, r, 0);
    if (r == 0) continue;
    const RowCount n = warp_row<OUTS, OUTC>(p, S, r - 1);
    if (lane_id() == 0 && n.ranges) tally(r - 1, n.ranges, n.columns);
  }
}

// Walks the `batch` rows of the warp's list, a row a lane; rows of more runs
// than a lane's lists hold go to the queue (take_rows), or to the whole warp at once
// where that is full.  Returns whether rows wait there.
// tally(row, ranges, columns) for each row of c that has any.
template <bool OUTS, bool OUTC, bool QUEUE, class Tally>
__device__ __forceinline__ bool walk_batch(const ChainArgs& p, WarpSmem& S, uint32_t batch, Tally&& tally) {
  const int lane = lane_id();
  uint32_t row = 0, ns = 0, nc = 0, cur = 0;
  bool done = false;
  uint2* const C = S.list[2] + lane;
  if (uint32_t(lane) < batch) {
    row = S.todo[lane];
    done = quick_row<OUTS, OUTC>(p, row, S.list[0] + lane, ns, C, nc);
  }
  const bool slow = __any_sync(kFullMask, uint32_t(lane) < batch && !done);
  if (uint32_t(lane) < batch && !done) {
    S.list[0][lane] = make_uint2(row, row);
    ns = 1;
    nc = 0;
#pragma unroll 1
    for (uint32_t j = 0;; ++j) {
      const uint2* L = S.list[cur] + lane;
      if (OUTC && ((p.bits >> j) & 1u)) nc = list_product(p.arena, L, ns, p.b, C, nc);
      if (j == p.k || nc == kFull) break;
      ns = list_product(p.arena, L, ns, p.m[j], S.list[cur ^ 1u] + lane, 0);
      if (ns == kFull) break;
      cur ^= 1u;
    }
    done = ns != kFull && nc != kFull;
  }
  __syncwarp();
  unsigned left = __ballot_sync(kFullMask, uint32_t(lane) < batch && !done);
  // (the look comes while the rows are written)
  const uint2 places = QUEUE && slow ? __ldcg(reinterpret_cast<const uint2*>(p.taken)) : make_uint2(0u, 0u);
  const bool put_in = left != 0;
  // places in the arena for the rows of several runs, one request a warp
  // (a row of two columns needs none)
  const uint2* const T = S.list[cur] + lane;
  auto place = [&](const uint2* L, uint32_t n) {
    return n == 2 && L[0].x == L[0].y && L[32].x == L[32].y ? 0u : n > 1 ? n : 0u;
  };
  const uint32_t ws = OUTS && done ? place(T, ns) : 0u, wc = OUTC && done ? place(C, nc) : 0u;
  const uint32_t incl = group_incl_sum<32>(kFullMask, ws + wc, lane);
  const uint32_t all = __shfl_sync(kFullMask, incl, 31);
  unsigned long long off = 0;
  bool fits = true;
  if (all) {
    if (lane == 31) off = atomicAdd(p.top, (unsigned long long)all);
    off = __shfl_sync(kFullMask, off, 31);
    fits = off + all <= p.arena_cap;
    if (!fits && lane == 0) atomicOr(p.abort, kArenaFull);
    off += incl - ws - wc;
  }
  auto put = [&](uint2* to, const uint2* L, uint32_t n, uint32_t want) {
    uint2 v = empty_slot();
    if (n == 1) v = L[0];
    else if (n == 2 && !want) v = make_uint2(L[32].x, L[0].x);
    else if (want && fits) v = make_uint2(kMulti + n, uint32_t(off));
    to[row] = v;
    if (fits)
      for (uint32_t k = 0; k < want; ++k) p.arena[off + k] = L[k * 32];
    off += want;
  };
  if (done) {
    if (OUTS) put(p.s, T, ns, ws);
    if (OUTC) {
      put(p.c, C, nc, wc);
      unsigned long long z = 0;
      for (uint32_t k = 0; k < nc; ++k) z += C[k * 32].y - C[k * 32].x + 1;
      if (nc) tally(row, nc, z);
    }
  }
  __syncwarp();
  if (left && lane == 0) atomicAdd(&p.ctl->slow_rows, (unsigned long long)__popc(left));
  if (QUEUE && left) {
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(p.taken + 1, uint32_t(__popc(left)));
    at = __shfl_sync(kFullMask, at, 0) + __popc(left & ((1u << lane) - 1u));
    const bool queued = ((left >> lane) & 1u) && at < p.queue_cap &&
                        atomicExch(p.queue + at, in_queue(p, row + 1)) != in_queue(p, kGone);
    left &= ~__ballot_sync(kFullMask, queued);
  }
  for (; left; left &= left - 1) {
    const uint32_t r = __shfl_sync(kFullMask, row, __ffs(left) - 1);
    const RowCount n = warp_row<OUTS, OUTC>(p, S, r);
    if (lane == 0 && n.ranges) tally(r, n.ranges, n.columns);
  }
  __syncwarp();
  return put_in || places.x < min(places.y, p.queue_cap);
}

// The kernels of a chain follow one another closely: each waits for the kernel before
// to end, with all that it wrote visible, before it touches memory, and then lets the
// next one's blocks be placed as soon as all of its own are.  Every block waits, so a
// kernel's end means the end of all before it.
__device__ __forceinline__ void follow() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ---- the passes ---------------------------------------------------------------
// A pass over a large matrix is two kernels.  k_chain_rows streams it: nearly
// all rows of a sequence graph's powers are a single column, and their part of
// the pass is k + 1 dependent loads, each near the row's own diagonal, for
// kSRows rows a lane at once.  It needs few registers, so that enough loads
// are in flight to keep HBM busy, and leaves the other rows marked in a
// bitmap.  k_chain_walk reads the bitmap and walks those, 32 at a time, a row a
// lane, so that no lane waits for another's longer row and a walk's chain of
// dependent loads is paid once for 32 rows; the rows that need a warp go through a
// queue (take_rows).
//
// Bound: HBM, 8 bytes a row for each matrix read and written (all but the first
// read of a matrix come from L2), and instructions.  k_chain_rows on 1e7 rows: 53 to 66
// us for 180 to 300 MB, 2.8 to 5.5 TB/s with issue slots 43 to 75 % busy -- the first
// pass, whose sum is of the identity's rows, and the counting one are the busy ones;
// six blocks an SM (40 registers) against four: 2.75 and 2.90 ms a 5e7-locus build.
// k_chain_walk: 25 to 45 us, the latency of a walk, whatever few rows there are; 24 to
// 33 % of an SM's warps are active where 44 % fit, so most have ended by then.  Walking
// the rows in the streaming kernel instead, behind a block's barrier or a warp at a
// time, held the loads of its other rows back (8.9 and 4.1 ms a build).
template <bool OUTS, bool OUTC, bool COUNT>
__global__ void __launch_bounds__(kSThreads, 6) k_chain_rows(const __grid_constant__ ChainArgs p) {
  follow();
  const uint64_t r0 = (uint64_t(blockIdx.x) * kSWarps + (threadIdx.x >> 5)) * (32 * kSRows);
  if (r0 >= p.n) return;
  const int lane = lane_id();
  uint32_t bad = 0, cnt = 0;
  unsigned long long nnz = 0;
  if (r0 + 32 * kSRows <= p.n) {
    bad = chain_rows<OUTS, OUTC, COUNT, kSRows>(p, uint32_t(r0), cnt, nnz);
  } else {  // the last, ragged rows are all walked
#pragma unroll
    for (int u = 0; u < kSRows; ++u) bad |= (r0 + u * 32 + lane < p.n ? 1u : 0u) << u;
  }
  uint32_t word = 0;
#pragma unroll
  for (int u = 0; u < kSRows; ++u) {
    const uint32_t w = __ballot_sync(kFullMask, (bad >> u) & 1u);
    if (lane == u) word = w;
  }
  if (lane < kSRows && r0 + lane * 32 < p.n) p.masks[r0 / 32 + lane] = word;
  if (COUNT) {
    cnt = __reduce_add_sync(kFullMask, cnt);
    nnz = group_sum<32>(kFullMask, nnz);
    if (lane == 0) {
      p.group_cnt[r0 / kCountRows] = cnt;
      p.group_nnz[r0 / kCountRows] = nnz;
    }
  }
}

template <bool OUTS, bool OUTC, bool COUNT>
__global__ void __launch_bounds__(kWThreads, kWBlocks) k_chain_walk(const __grid_constant__ ChainArgs p) {
  follow();
  __shared__ WarpSmem smem[kWWarps];
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  WarpSmem& S = smem[warp];
  // rows to walk come in clumps, the length of a left factor before a bubble:
  // a warp's words lie a grid's width apart, so that each gets its share
  const uint64_t words = (uint64_t(p.n) + 31) / 32, stride = gridDim.x * kWWarps;
  uint64_t next = blockIdx.x * kWWarps + warp;
  auto tally = [&](uint32_t row, uint32_t cnt, unsigned long long nnz) {
    if (!COUNT) return;
    atomicAdd(p.group_cnt + row / kCountRows, cnt);
    atomicAdd(p.group_nnz + row / kCountRows, nnz);
  };
  bool look = false;
  uint32_t x = 0, at = 0;  // a lane's word: its rows still to walk, and the first of its 32
  while (true) {
    const unsigned spent = __ballot_sync(kFullMask, x == 0);
    uint32_t have = __reduce_add_sync(kFullMask, uint32_t(__popc(x)));
    if (have < 32 && next < words) {  // lanes whose word is done take the next ones
      const uint64_t w = next + __popc(spent & ((1u << lane) - 1u)) * stride;
      if (x == 0 && w < words) {
        x = p.masks[w];
        at = uint32_t(w) * 32;
      }
      next += __popc(spent) * stride;
      continue;
    }
    if (have == 0) break;
    // the first 32 rows
    uint32_t k = group_incl_sum<32>(kFullMask, uint32_t(__popc(x)), lane) - __popc(x);
    for (; x && k < 32; x &= x - 1) S.todo[k++] = at + uint32_t(__ffs(x) - 1);
    __syncwarp();
    if (walk_batch<OUTS, OUTC, true>(p, S, min(have, 32u), tally)) look = true;
  }
  if (look) take_rows<OUTS, OUTC>(p, S, tally);
}

// A pass over a small matrix, where a launch costs more than the rows: both in
// one kernel, a block kCountRows rows, a warp 32 of them.  A product alone does
// without the queue: a row of it is one factor, and looking and being looked at cost
// 3 of its 43 us at 1e5 rows.
template <bool OUTS, bool OUTC, bool COUNT, bool QUEUE>
__global__ void __launch_bounds__(kWThreads, kWBlocks) k_chain_small(const __grid_constant__ ChainArgs p) {
  follow();
  static_assert(kWThreads == kCountRows, "a block's rows are counted together");
  __shared__ WarpSmem smem[kWWarps];
  __shared__ unsigned long long sum[2];
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  WarpSmem& S = smem[warp];
  if (COUNT) {
    if (threadIdx.x < 2) sum[threadIdx.x] = 0;
    __syncthreads();
  }
  const uint64_t r0 = uint64_t(blockIdx.x) * kWThreads + warp * 32;
  unsigned long long nnz = 0;
  uint32_t cnt = 0;
  bool look = false;
  if (r0 < p.n) {
    uint32_t bad;
    if (r0 + 32 <= p.n) bad = chain_rows<OUTS, OUTC, COUNT, 1>(p, uint32_t(r0), cnt, nnz);
    else bad = r0 + lane < p.n ? 1u : 0u;
    const unsigned who = __ballot_sync(kFullMask, bad != 0);
    if (bad) S.todo[__popc(who & ((1u << lane) - 1u))] = uint32_t(r0) + lane;
    __syncwarp();
    if (who)
      look = walk_batch<OUTS, OUTC, QUEUE>(p, S, __popc(who), [&](uint32_t, uint32_t c, unsigned long long z) {
        cnt += c;
        nnz += z;
      });
  }
  // (any block's rows: the counts start at zero, and every block adds to them)
  if (QUEUE && look)
    take_rows<OUTS, OUTC>(p, S, [&](uint32_t row, uint32_t c, unsigned long long z) {
      if (!COUNT) return;
      atomicAdd(p.group_cnt + row / kCountRows, c);
      atomicAdd(p.group_nnz + row / kCountRows, z);
    });
  if (COUNT) {
    cnt = __reduce_add_sync(kFullMask, cnt);
    nnz = group_sum<32>(kFullMask, nnz);
    if (lane == 0) {
      atomicAdd(&sum[0], (unsigned long long)cnt);
      atomicAdd(&sum[1], nnz);
    }
    __syncthreads();
    if (threadIdx.x == 0 && QUEUE) {
      atomicAdd(p.group_cnt + blockIdx.x, uint32_t(sum[0]));
      atomicAdd(p.group_nnz + blockIdx.x, sum[1]);
    } else if (threadIdx.x == 0) {
      p.group_cnt[blockIdx.x] = uint32_t(sum[0]);
      p.group_nnz[blockIdx.x] = sum[1];
    }
  }
}

// The matrices of a chain laid side by side on the diagonal, each from a
// multiple of kCrsRows rows on, so that every block of the conversions below
// works on one of them: block b's is number part_of[b] (a null table: all
// blocks are `one`'s, the only one).
struct Parts {
  const SlotPart* table;
  const uint32_t* part_of;
  SlotPart one;
};
__device__ __forceinline__ SlotPart my_part(const Parts& q) { return q.table ? q.table[q.part_of[blockIdx.x]] : q.one; }

// Range CRS -> slots.  Canonical input: a row of several ranges is copied to
// the arena as it is.  Rows past a part's last are rows of the identity: one
// column each, whatever the pass.
__global__ void __launch_bounds__(kSThreads) k_crs_to_slots(const __grid_constant__ Parts q,
                                                            const __grid_constant__ ChainArgs p) {
  follow();
  constexpr int kIter = kCrsRows / kSThreads;
  const SlotPart part = my_part(q);
  const int lane = lane_id();
  const uint64_t b0 = uint64_t(blockIdx.x) * kCrsRows + threadIdx.x;
  if (p.add_counts && threadIdx.x < kCrsRows / kCountRows) {
    const uint64_t g = uint64_t(blockIdx.x) * (kCrsRows / kCountRows) + threadIdx.x;
    if (g * kCountRows < p.n) {
      p.group_cnt[g] = 0;
      p.group_nnz[g] = 0;
    }
  }
  uint64_t a0[kIter], cnt[kIter];
#pragma unroll
  for (int u = 0; u < kIter; ++u) {
    const uint64_t i = b0 + u * kSThreads - part.row0;
    a0[u] = cnt[u] = 0;
    if (i < part.n) {
      a0[u] = part.rowmap[i] >> 1;
      cnt[u] = (part.rowmap[i + 1] >> 1) - a0[u];
    }
  }
  auto range = [&](uint64_t k) {
    uint2 v = load_range(part.entries, k);
    v.x += part.row0;
    v.y += part.row0;
    return v;
  };
  uint2 v[kIter];
#pragma unroll
  for (int u = 0; u < kIter; ++u) v[u] = cnt[u] ? range(a0[u]) : empty_slot();
#pragma unroll
  for (int u = 0; u < kIter; ++u) {
    const uint64_t r = b0 + u * kSThreads;
    uint64_t want = cnt[u] > 1 ? cnt[u] : 0;
    if (cnt[u] == 2) {
      const uint2 w = range(a0[u] + 1);
      if (v[u].x == v[u].y && w.x == w.y) {
        v[u] = make_uint2(w.x, v[u].x);
        want = 0;
      }
    }
    if (__any_sync(kFullMask, want != 0)) {
      const uint64_t incl = group_incl_sum<32>(kFullMask, want, lane);
      unsigned long long off = 0;
      if (lane == 31) off = atomicAdd(p.top, (unsigned long long)incl);
      off = __shfl_sync(kFullMask, off, 31) + incl - want;
      if (want) {
        if (want > kMultiMax || off + want > p.arena_cap) {
          atomicOr(p.abort, want > kMultiMax ? kLongRow : kArenaFull);
          v[u] = empty_slot();
        } else {
          for (uint64_t k = 0; k < want; ++k) p.arena[off + k] = range(a0[u] + k);
          v[u] = make_uint2(kMulti + uint32_t(want), uint32_t(off));
        }
      }
    }
    if (r < p.n) p.s[r] = r - part.row0 < part.n ? v[u] : make_uint2(uint32_t(r), uint32_t(r));
  }
}

// Sums of kSuperGroups counts each, a block a sum; the totals of the result.
__global__ void __launch_bounds__(kSThreads) k_slot_sums(const uint32_t* cnt, const unsigned long long* nnz,
                                                         uint64_t groups, unsigned long long* sums,
                                                         DeviceControl* ctl) {
  follow();
  __shared__ unsigned long long part[2][kSWarps];
  unsigned long long s = 0, z = 0;
  for (uint32_t k = threadIdx.x; k < kSuperGroups; k += kSThreads) {
    const uint64_t g = uint64_t(blockIdx.x) * kSuperGroups + k;
    if (g < groups) {
      s += cnt[g];
      z += nnz[g];
    }
  }
  s = group_sum<32>(kFullMask, s);
  z = group_sum<32>(kFullMask, z);
  if (lane_id() == 0) {
    part[0][threadIdx.x >> 5] = s;
    part[1][threadIdx.x >> 5] = z;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kSWarps; ++w) {
      s += part[0][w];
      z += part[1][w];
    }
    sums[blockIdx.x] = s;
    atomicAdd(&ctl->total, 2 * s);
    atomicAdd(&ctl->nnz, z);
  }
}

// Ranges and columns of every part's result, a block a part (its last rows of
// the identity are no part of it).
__global__ void __launch_bounds__(kSThreads) k_part_totals(const Parts q, const uint32_t* cnt,
                                                           const unsigned long long* nnz, uint32_t n,
                                                           unsigned long long* totals) {
  follow();
  __shared__ unsigned long long sum[2][kSWarps];
  const SlotPart part = q.table[blockIdx.x];
  const uint64_t end = min((uint64_t(part.row0) + part.n + kCrsRows - 1) / kCrsRows * kCrsRows, uint64_t(n));
  unsigned long long s = 0, z = 0;
  for (uint64_t g = part.row0 / kCountRows + threadIdx.x; g < (end + kCountRows - 1) / kCountRows; g += kSThreads) {
    s += cnt[g];
    z += nnz[g];
  }
  s = group_sum<32>(kFullMask, s);
  z = group_sum<32>(kFullMask, z);
  if (lane_id() == 0) {
    sum[0][threadIdx.x >> 5] = s;
    sum[1][threadIdx.x >> 5] = z;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kSWarps; ++w) {
      s += sum[0][w];
      z += sum[1][w];
    }
    const uint64_t pad = end - part.row0 - part.n;
    totals[2 * blockIdx.x] = s - pad;
    totals[2 * blockIdx.x + 1] = z - pad;
  }
}

// Slots -> range CRS.  A block takes kCrsRows rows; the ranges before them are
// the sums of the super groups before its own and the counts of the groups
// before it in that one, less those before its part, so no block waits for
// another.  A warp takes 32 consecutive rows at a time.
//
// Bound: HBM, 8 bytes a row read and 8 a row and 8 a range written, and instructions
// (78 % of the issue slots).  They were 71 % busy at 1e7 rows, 78 us: rows nearly all
// have at most two ranges, so
// two ballots give their places in place of a scan, and runs and pairs are written
// without a loop: 53 us, and 186 in place of 189 us for a product of 1e7 rows
// with the slots requested first and seven blocks an SM (a build of 5e7 rows: 2.78
// to 2.65 ms).
__global__ void __launch_bounds__(kSThreads, 7) k_slots_to_crs(const __grid_constant__ Parts q,
                                                               const uint2* slots, const uint2* arena,
                                                               const unsigned long long* sums,
                                                               const uint32_t* group_cnt, DeviceControl* ctl) {
  follow();
  constexpr int kIter = kCrsRows / kSThreads;
  __shared__ unsigned long long pre[kSWarps];
  __shared__ uint32_t wsum[kSWarps];
  const SlotPart part = my_part(q);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t tile = blockIdx.x, g0 = tile * (kCrsRows / kCountRows), sup = g0 / kSuperGroups;
  // the warp's rows: kIter groups of 32
  const uint64_t w0 = uint64_t(tile) * kCrsRows + uint64_t(warp) * (kIter * 32);
  uint2 v[kIter];
  uint32_t c[kIter];
#pragma unroll
  for (int u = 0; u < kIter; ++u) {
    const uint64_t r = w0 + u * 32 + lane;
    v[u] = r - part.row0 < part.n ? ld_slot(slots, r) : empty_slot();
  }
  unsigned long long before = 0;
  for (uint32_t k = tid; k < sup; k += kSThreads) before += sums[k];
  for (uint32_t k = sup * kSuperGroups + tid; k < g0; k += kSThreads) before += group_cnt[k];
  uint32_t sum = 0;
#pragma unroll
  for (int u = 0; u < kIter; ++u) {
    const uint32_t k = slot_count(v[u]), upto = ~0u >> (31 - lane);
    const unsigned one = __ballot_sync(kFullMask, k > 0), two = __ballot_sync(kFullMask, k > 1);
    c[u] = __popc(one & upto) + __popc(two & upto);  // inclusive within the group
    if (two && __any_sync(kFullMask, k > 2)) c[u] = group_incl_sum<32>(kFullMask, k, lane);
    sum += __shfl_sync(kFullMask, c[u], 31);
  }
  before = group_sum<32>(kFullMask, before);
  if (lane == 0) {
    pre[warp] = before;
    wsum[warp] = sum;
  }
  __syncthreads();
  unsigned long long at = 0ull - part.before;
#pragma unroll
  for (int w = 0; w < kSWarps; ++w) {
    at += pre[w];
    if (w < warp) at += wsum[w];
  }
  uint2* out = reinterpret_cast<uint2*>(part.c_entries) + at;
  uint64_t* const rowmap = part.c_rowmap + (w0 - part.row0) + lane + 1;
  const uint64_t left = w0 - part.row0 < part.n ? part.n - (w0 - part.row0) : 0;  // the part's rows from here on
  if (left && w0 == part.row0 && lane == 0) part.c_rowmap[0] = 0;
#pragma unroll
  for (int u = 0; u < kIter; ++u) {
    if (u * 32 + lane < left) rowmap[u * 32] = 2 * (at + c[u]);
    const uint32_t tot = __shfl_sync(kFullMask, c[u], 31), k = slot_count(v[u]);
    if (at + tot > part.c_ranges) {
      if (lane == 0) atomicOr(&ctl->status, 256ull);
    } else {
      uint2* const o = out + (c[u] - k);
      if (is_multi(v[u])) {
        for (uint32_t t = 0; t < k; ++t) {
          const uint2 w = slot_range(arena, v[u], t);
          o[t] = make_uint2(w.x - part.row0, w.y - part.row0);
        }
      } else {
        const uint2 w = make_uint2(v[u].x - part.row0, v[u].y - part.row0);  // a run, or two columns {y, x}
        if (k) o[0] = make_uint2(k > 1 ? w.y : w.x, w.y);
        if (k > 1) o[1] = make_uint2(w.x, w.x);
      }
    }
    at += tot;
    out += tot;
  }
}

// A launch behind another kernel of the chain; `close`: see kCloseRows.
template <class... P, class... A>
void launch_next(dvg_context* ctx, bool close, void (*kernel)(P...), uint64_t blocks, int threads, const A&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(blocks));
  cfg.blockDim = dim3(unsigned(threads));
  cfg.stream = ctx->stream;
  cfg.attrs = &attr;
  cfg.numAttrs = close ? 1 : 0;
  DVG_CUDA(cudaLaunchKernelEx(&cfg, kernel, P(args)...));
  ctx->stats.kernel_launches++;
}

template <bool OUTS, bool OUTC, bool COUNT>
void launch_pass(dvg_context* ctx, bool close, const ChainArgs& p, bool alone) {
  // one kernel while a warp a 32 rows fits the chip at once; the second
  // kernel's launch costs more than it saves there
  if (p.n <= kSmallRows) {
    const uint64_t blocks = (uint64_t(p.n) + kWThreads - 1) / kWThreads;
    if (!OUTS && COUNT && alone) launch_next(ctx, close, k_chain_small<false, true, true, false>, blocks, kWThreads, p);
    else launch_next(ctx, close, k_chain_small<OUTS, OUTC, COUNT, true>, blocks, kWThreads, p);
    return;
  }
  launch_next(ctx, close, k_chain_rows<OUTS, OUTC, COUNT>,
              (uint64_t(p.n) + kSThreads * kSRows - 1) / (kSThreads * kSRows), kSThreads, p);
  const uint64_t want = (uint64_t(p.n) + 32 * kWWarps - 1) / (32 * kWWarps);
  launch_next(ctx, close, k_chain_walk<OUTS, OUTC, COUNT>, std::min<uint64_t>(want, uint64_t(kWBlocks) * ctx->num_sms), kWThreads, p);
}

}  // namespace

// What the left factors of one pass may add up to in steps of A: past it most
// rows would have left the single column on the way, and walking a product of
// several factors a row repeats what one factor at a time shares between rows.
static unsigned chain_reach(double branching) {
  const double r = kChainReach / std::max(branching, 1e-9);
  return r >= 1e9 ? 1000000000u : std::max(1u, unsigned(r));
}

SlotPlan plan_slots(unsigned dlo, unsigned dup, double branching) {
  SlotPlan pl;
  const unsigned K = dup - dlo, reach = chain_reach(branching);
  auto top_bit = [](unsigned v) { return v ? 31 - __builtin_clz(v) : -1; };
  struct Power {
    unsigned e;  // A^e
    int mat;
  };
  std::vector<Power> P{{1u, 0}};
  auto pass = [&](const std::vector<Power>& left, int b, unsigned bits, bool s, bool c) {
    SlotStep st;
    st.k = int(left.size());
    for (int j = 0; j < st.k; ++j) st.m[j] = left[j].mat;
    st.b = b;
    st.bits = bits;
    if (s) st.s = pl.nmats++;
    if (c) st.c = pl.nmats++;
    pl.steps.push_back(st);
  };
  // (A + I)^(2^t) = Q by doubling, with the powers of A on the way: from A^e and
  // (A + I)^e to their f-th powers in one pass, f = 4 while the reach allows
  const int t = top_bit(K);
  const unsigned q_top = K > 0 ? 1u << t : 0u;
  const unsigned rest = K > 0 ? K - q_top : 0;
  // from A^e on the way to A^top (and, first, to (A + I)^q_top): the next power
  auto factor = [&](unsigned e, unsigned top) {
    return 4ull * e <= (e < q_top ? q_top : top) && 4ull * e <= reach ? 4u : 2u;
  };
  auto levels = [&](unsigned top) {
    std::vector<unsigned> v{1u};
    for (unsigned e = 1; e < std::max(top, q_top);) {
      e *= factor(e, top);
      if (e <= top) v.push_back(e);
    }
    return v;
  };
  // passes that multiply by A^v, its factors the largest powers that fit
  // (counted, not listed: A^v has up to v / have[0] of them)
  auto passes = [&](unsigned v, const std::vector<unsigned>& have) {
    uint64_t n = 0, k = 0, sum = 0;  // passes, and the last one's factors and their exponents
    for (size_t j = have.size(); j-- > 0; v %= have[j]) {
      const uint64_t e = have[j], fit = std::clamp<uint64_t>(reach / e, 1, kChainMax);
      uint64_t q = v / e;
      if (n && q) {
        const uint64_t more = sum >= reach ? 0 : std::min<uint64_t>({q, kChainMax - k, (reach - sum) / e});
        q -= more;
        k += more;
        sum += more * e;
      }
      if (q) {
        n += (q + fit - 1) / fit;
        k = (q - 1) % fit + 1;
        sum = k * e;
      }
    }
    return n;
  };
  // powers up to half of Q's, and further where that saves passes over A^dlo
  unsigned p_top = q_top > 1 ? q_top / 2 : 1;
  if (rest) p_top = std::max(p_top, 1u << top_bit(rest));
  uint64_t best = ~uint64_t(0);
  for (unsigned long long top = p_top; top <= std::max<unsigned long long>(p_top, dlo); top *= 2) {
    const std::vector<unsigned> have = levels(unsigned(top));
    uint64_t cost = passes(rest, have) + passes(dlo, have);
    for (unsigned e = 1; e < std::max(unsigned(top), q_top); ++cost) e *= factor(e, unsigned(top));
    if (cost < best) {
      best = cost;
      p_top = unsigned(top);
    }
  }
  int Q = -1;
  unsigned e = 1;  // the last power and the sum stand at e
  while (e < std::max(p_top, q_top)) {
    const unsigned f = factor(e, p_top);
    const bool s = e * f <= p_top, c = K > 0 && e * f <= q_top;
    if (!s && !c) break;
    const Power last = P.back();
    // the factors S_1 .. S_f; c needs S_0 .. S_(f-1) times (A + I)^e, for e = 1
    // that is S_0 .. S_f itself
    const unsigned bits = e == 1 ? (1u << (f + 1)) - 1 : (1u << f) - 1;
    const unsigned k = s || e == 1 ? f : f - 1;
    pass(std::vector<Power>(k, last), e == 1 ? -1 : Q, c ? bits : 0u, s, c);
    if (s) P.push_back({e * f, pl.steps.back().s});
    if (c) Q = pl.steps.back().c;
    e *= f;
  }
  // the fewest factors whose exponents add up to v, the largest first
  auto factors = [&](unsigned v) {
    std::vector<Power> f;
    for (int j = int(P.size()) - 1; j >= 0; --j)
      for (; v >= P[j].e; v -= P[j].e) f.push_back(P[j]);
    return f;
  };
  // takes the next pass's factors off the list
  auto next = [&](std::vector<Power>& f) {
    std::vector<Power> g;
    unsigned long long sum = 0;
    while (!f.empty() && int(g.size()) < kChainMax && (g.empty() || sum + f.back().e <= reach)) {
      sum += f.back().e;
      g.push_back(f.back());
      f.pop_back();
    }
    return g;
  };
  int R = Q;
  if (K == 1) {  // I + A
    pass({P[0]}, -1, 3u, false, true);
    R = pl.steps.back().c;
  }
  // (A + I)^(v + w) = (A + I)^v + A^w (A + I)^v for w <= v + 1
  for (std::vector<Power> f = factors(rest); !f.empty();) {
    const std::vector<Power> g = next(f);
    pass(g, R, 1u | (1u << g.size()), false, true);
    R = pl.steps.back().c;
  }
  // A^dlo from the left: the right operand is a sum of powers, whose rows are
  // one run, not a power, whose rows fall apart
  std::vector<Power> f = factors(dlo);
  if (R < 0) {  // A^dlo alone: its largest factor is the first right operand
    R = f.front().mat;
    f.erase(f.begin());
  }
  while (!f.empty()) {
    const std::vector<Power> g = next(f);
    pass(g, R, 1u << g.size(), false, true);
    R = pl.steps.back().c;
  }
  // the last pass counts the result
  if (pl.steps.empty() || pl.steps.back().s >= 0 || pl.steps.back().c != R) {
    pass({}, R, 1u, false, true);
    R = pl.steps.back().c;
  }
  pl.out = R;
  return pl;
}

// Rows of a sequence graph's adjacency hold about one range of one or two
// columns.  Where A has more than 1.5 ranges a row or ranges of more than two
// columns on average, the powers' rows soon leave the slots for the arena, or
// name so many rows that a thread walks them for long: such input, input whose
// rows are not canonical, and matrices whose columns reach the marker of a
// several-run row stay with the range-CRS row kernel.  (No sharp line: products and
// powers of 1e5 rows take 0.25 to 0.95 of its time at 1.48 ranges a row; at 1.6 to 2 0.25
// to 1.05 where the arena holds, and longer chains run full; at 3, and with three
// columns a range, most of them do.)  So does large input of more
// than a quarter of a column a row beyond its first, which no sequence graph has.  At 1e6
// rows A^2 of a path with skips took 88 us against 110 in range CRS at 0.2 columns, 104
// against 109 at 0.29 and 160 against 116 at 0.48, of random bands 195 against 146 at 0.3
// and 364 against 213 at 0.7; A^4 250 against 365, 380 against 410, and of the bands
// 696 against 581 and 1,856 against 1,074.  Up to 2^18 rows the row kernel's fixed costs
// are more than that: at 1e5 rows all of these take 0.5 to 0.95 of its time.
constexpr double kDenseBranching = 0.25;
constexpr uint32_t kDenseRows = 1u << 18;
bool slots_suit(const dvg_context* ctx, const dvg_matrix* a) {
  const uint64_t ranges = a->nentries / 2;
  return a->canonical && a->nrows == a->ncols && a->nrows > 0 && a->ncols < kSlotMulti &&
         2 * ranges <= 3ull * a->nrows && a->nnz <= 2 * ranges &&
         (a->nrows <= kDenseRows || branching(a->nnz + a->empty_rows, a->nrows) <= kDenseBranching) &&
         ctx->opt_slots != 0;
}

// Chains over such matrices for such a window, as far as whether they fit goes: sizes
// within a factor of two, densities within a fifth.  (Products: dlo 1, dup 0.)
SlotKey slot_key(unsigned dlo, unsigned dup, uint64_t nnz, uint64_t nrows) {
  const double b = branching(nnz, nrows);
  return {dlo, dup, int(64 - __builtin_clzll(nrows | 1)), b > 0 ? int(std::floor(4 * std::log2(b))) : -1000};
}

bool slots_due(dvg_context* ctx, const SlotKey& key) {
  const auto it = ctx->slot_misses.find(key);
  if (it == ctx->slot_misses.end() || it->second.left == 0) return true;
  --it->second.left;
  return false;
}

// A chain that is given up costs what its passes did until then, so the next ones like
// it go the range-CRS way at once: 1 call, then 3, 7 and so on up to 63 between two
// attempts.
static void slots_missed(dvg_context* ctx, const SlotKey& key) {
  constexpr size_t kMost = 256;
  constexpr uint32_t kLongest = 63;
  if (ctx->slot_misses.size() >= kMost && !ctx->slot_misses.count(key)) ctx->slot_misses.clear();
  SlotMiss& m = ctx->slot_misses[key];
  m.wait = std::min(2 * m.wait + 1, kLongest);
  m.left = m.wait;
}

static unsigned conversion_blocks(const SlotBuild& sb) { return unsigned((uint64_t(sb.n) + kCrsRows - 1) / kCrsRows); }

// The buffer of each of a plan's matrices, `count` of them together: a matrix takes that
// of one whose last reader is an earlier pass (the chain's own buffers only: chains that
// run side by side share none).
static std::vector<int> assign_buffers(const SlotPlan& plan, int& count) {
  std::vector<int> last(plan.nmats, -1), buffer(plan.nmats, 0), spare;
  auto reads = [&](const SlotStep& s, auto&& f) {
    for (int j = 0; j < s.k; ++j) f(s.m[j]);
    if (s.b >= 0) f(s.b);
  };
  for (size_t i = 0; i < plan.steps.size(); ++i) reads(plan.steps[i], [&](int k) { last[k] = int(i); });
  auto take = [&](int k) {
    if (spare.empty()) spare.push_back(count++);
    buffer[k] = spare.back();
    spare.pop_back();
  };
  for (int k = 0; k < plan.inputs; ++k) take(k);
  for (size_t i = 0; i < plan.steps.size(); ++i) {
    if (plan.steps[i].s >= 0) take(plan.steps[i].s);
    if (plan.steps[i].c >= 0) take(plan.steps[i].c);
    std::vector<int> done;
    reads(plan.steps[i], [&](int k) {
      if (last[k] == int(i) && k != plan.out && std::find(done.begin(), done.end(), k) == done.end()) done.push_back(k);
    });
    for (int k : done) spare.push_back(buffer[k]);
  }
  return buffer;
}

uint64_t predict_slots_bytes(uint32_t nrows, uint64_t nentries, unsigned dlo, unsigned dup) {
  // (the density decides the passes; the buffers of a few stand for all)
  int buffers = 0;
  size_t steps = 0;
  for (double density : {0.0, 0.001, 0.01, 0.1, 1.0}) {
    int count = 0;
    const SlotPlan plan = plan_slots(dlo, dup, density);
    assign_buffers(plan, count);
    buffers = std::max(buffers, count);
    steps = std::max(steps, plan.steps.size());
  }
  const uint64_t n = (uint64_t(nrows) + kSlotPartRows - 1) / kSlotPartRows * kSlotPartRows;
  const uint64_t ranges = std::min<uint64_t>(uint64_t(kSlotGrowthMax * double(n)) + 4096, kMulti);
  const uint64_t input = 8 * n + 4 * nentries, result = 8 * n + 16 * n, scratch = n + steps * 8 + kQueueBytes;
  // (blocks are up to a quarter larger than what they hold)
  return (input + 8 * n * buffers + 8 * ranges + result + scratch) / 4 * 5;
}

// The context's queue, for chains that run one after another.
static unsigned long long* slot_queue(dvg_context* ctx, uint32_t passes, uint32_t& epoch) {
  if (ctx->slot_epoch > 0xffffffffu - passes) ctx->slot_epoch = 0;  // (and cleared once more)
  if (!ctx->d_slot_queue) ctx->d_slot_queue = static_cast<unsigned long long*>(dalloc(ctx, kQueueBytes));
  if (ctx->slot_epoch == 0) DVG_CUDA(cudaMemsetAsync(ctx->d_slot_queue, 0, kQueueBytes, ctx->stream));
  epoch = ctx->slot_epoch + 1;
  ctx->slot_epoch += passes;
  return ctx->d_slot_queue;
}

SlotBuild prepare_slots(dvg_context* ctx, const SlotPlan& plan, uint32_t n, bool own_queue) {
  SlotBuild sb;
  sb.plan = plan;
  sb.n = n;
  sb.mat.assign(plan.nmats, nullptr);
  const uint64_t groups = (uint64_t(n) + kCountRows - 1) / kCountRows;
  const uint64_t supers = (groups + kSuperGroups - 1) / kSuperGroups;
  auto round = [](size_t x) { return (x + 15) & ~size_t(15); };
  // counters, the passes' places and the chain's own queue, cleared together
  const size_t taken_off = sizeof(SlotCounters);
  const size_t queue_off = std::max<size_t>(512, round(taken_off + plan.steps.size() * 8));
  sb.queue_cap = own_queue ? uint32_t(std::clamp<uint64_t>(n / 8, 256, kQueueRows)) : kQueueRows;
  sb.cleared = queue_off + (own_queue ? sb.queue_cap * sizeof(unsigned long long) : 0);
  const size_t nnz_off = round(sb.cleared), cnt_off = nnz_off + groups * 8, sums_off = round(cnt_off + groups * 4);
  const size_t masks_off = sums_off + supers * 8;
  static_assert(sizeof(SlotCounters) <= 512, "the counters come first");
  // (below kMulti, so that the slot of a row of several runs has y < x)
  sb.arena_cap = std::min<uint64_t>(uint64_t(ctx->slot_growth * double(n)) + 4096, kMulti);
  const double room = 0.5 * double(device_free_bytes(ctx) + ctx->cached_bytes);
  if (double(sb.arena_cap) * 8.0 > room) sb.arena_cap = uint64_t(room / 8.0) + 4096;
  if (n <= kEarlyRows && 16.0 * double(n) < room / 8.0) sb.early = 2ull * n;
  int nbuffers = 0;
  const std::vector<int> buffer = assign_buffers(plan, nbuffers);
  try {
    sb.scratch = dalloc(ctx, masks_off + (uint64_t(n) + 31) / 32 * 4);
    char* base = static_cast<char*>(sb.scratch);
    sb.ctl = reinterpret_cast<DeviceControl*>(base);
    sb.top = reinterpret_cast<unsigned long long*>(base + 256);
    sb.abort = sb.top + 1;
    sb.wide = sb.top + 2;
    sb.taken = reinterpret_cast<uint32_t*>(base + taken_off);
    sb.epoch = 1;
    sb.queue = own_queue ? reinterpret_cast<unsigned long long*>(base + queue_off)
                         : slot_queue(ctx, uint32_t(plan.steps.size()), sb.epoch);
    sb.sums = reinterpret_cast<unsigned long long*>(base + sums_off);
    sb.group_nnz = reinterpret_cast<unsigned long long*>(base + nnz_off);
    sb.group_cnt = reinterpret_cast<uint32_t*>(base + cnt_off);
    sb.masks = reinterpret_cast<uint32_t*>(base + masks_off);
    sb.arena = static_cast<uint2*>(dalloc(ctx, sb.arena_cap * sizeof(uint2)));
    for (int k = 0; k < nbuffers; ++k)
      sb.buffers.push_back(static_cast<uint2*>(dalloc(ctx, size_t(n) * sizeof(uint2))));
    for (int k = 0; k < plan.nmats; ++k) sb.mat[k] = sb.buffers[buffer[k]];
  } catch (...) {
    release_slots(ctx, sb);
    throw;
  }
  return sb;
}

void release_slots(dvg_context* ctx, SlotBuild& sb) {
  for (uint2* b : sb.buffers) dfree(ctx, b);
  sb.buffers.clear();
  if (sb.arena) dfree(ctx, sb.arena);
  sb.arena = nullptr;
  if (sb.scratch) dfree(ctx, sb.scratch);
  sb.scratch = nullptr;
}

void launch_slots(dvg_context* ctx, SlotBuild& sb, const SlotParts& parts, bool timed, const SlotPart* right) {
  const uint64_t t0 = now_ns();
  // (512 bytes with up to 28 passes and the context's queue; more than a few KB take 4 us longer)
  DVG_CUDA(cudaMemsetAsync(sb.scratch, 0, sb.cleared, ctx->stream));
  ctx->stats.kernel_launches++;
  ChainArgs p{};
  p.arena = sb.arena;
  p.top = sb.top;
  p.arena_cap = sb.arena_cap;
  p.ctl = sb.ctl;
  p.abort = sb.abort;
  p.wide = sb.wide;
  p.wide_max = kWideCost + sb.n / 16;
  p.masks = sb.masks;
  const bool alone = sb.plan.steps.size() == 1 && sb.plan.steps[0].k <= 1;  // a product
  p.add_counts = sb.n <= kSmallRows && !alone;
  p.queue = sb.queue;
  p.queue_cap = sb.queue_cap;
  p.group_cnt = sb.group_cnt;
  p.group_nnz = sb.group_nnz;
  p.n = sb.n;
  p.s = sb.mat[0];
  k_crs_to_slots<<<conversion_blocks(sb), kSThreads, 0, ctx->stream>>>(Parts{parts.table, parts.part_of, parts.one}, p);
  DVG_CUDA(cudaGetLastError());
  ctx->stats.kernel_launches++;
  if (right) {
    p.s = sb.mat[1];
    launch_next(ctx, sb.close, k_crs_to_slots, conversion_blocks(sb), kSThreads, Parts{nullptr, nullptr, *right}, p);
  }
  for (size_t i = 0; i < sb.plan.steps.size(); ++i) {
    const SlotStep& st = sb.plan.steps[i];
    p.taken = sb.taken + 2 * i;
    p.epoch = sb.epoch + uint32_t(i);
    p.k = uint32_t(st.k);
    p.bits = st.bits;
    for (int j = 0; j < kChainMax; ++j) p.m[j] = j < st.k ? sb.mat[st.m[j]] : nullptr;
    p.b = st.b >= 0 ? sb.mat[st.b] : nullptr;
    p.s = st.s >= 0 ? sb.mat[st.s] : nullptr;
    p.c = st.c >= 0 ? sb.mat[st.c] : nullptr;
    cudaEvent_t ev = timed ? span_begin(ctx) : nullptr;
    if (i + 1 == sb.plan.steps.size()) launch_pass<false, true, true>(ctx, sb.close, p, alone);
    else if (p.s && p.c) launch_pass<true, true, false>(ctx, sb.close, p, false);
    else if (p.s) launch_pass<true, false, false>(ctx, sb.close, p, false);
    else launch_pass<false, true, false>(ctx, sb.close, p, false);
    span_end(ctx, ev, kProduct);
  }
  const uint64_t groups = (uint64_t(sb.n) + kCountRows - 1) / kCountRows;
  launch_next(ctx, sb.close, k_slot_sums, (groups + kSuperGroups - 1) / kSuperGroups, kSThreads, sb.group_cnt,
              sb.group_nnz, groups, sb.sums, sb.ctl);
  ctx->stats.host_launch_ns += now_ns() - t0;
}

void launch_slots_totals(dvg_context* ctx, const SlotBuild& sb, const SlotParts& parts, uint32_t nparts,
                         unsigned long long* totals) {
  launch_next(ctx, sb.close, k_part_totals, nparts, kSThreads, Parts{parts.table, parts.part_of, parts.one},
              sb.group_cnt, sb.group_nnz, sb.n, totals);
}

void launch_slots_out(dvg_context* ctx, const SlotBuild& sb, const SlotParts& parts, DeviceControl* ctl) {
  launch_next(ctx, sb.close, k_slots_to_crs, conversion_blocks(sb), kSThreads,
              Parts{parts.table, parts.part_of, parts.one}, sb.mat[sb.plan.out], sb.arena, sb.sums, sb.group_cnt,
              ctl ? ctl : ctx->d_ctl);
}

bool check_slots(dvg_context* ctx, const SlotBuild& sb, const SlotCounters& c) {
  if (c.abort) {
    // the caller takes the range-CRS path; where only the arena was too small, later
    // chains get a larger one, and otherwise chains like this wait
    const bool bigger = c.abort == kArenaFull && ctx->slot_growth < kSlotGrowthMax &&
                        double(sb.arena_cap) >= std::min(ctx->slot_growth * double(sb.n), double(kMulti));
    if (bigger) ctx->slot_growth = std::min(2.0 * ctx->slot_growth, kSlotGrowthMax);
    else slots_missed(ctx, sb.key);
    return false;
  }
  ctx->slot_misses.erase(sb.key);
  // statistics: what every pass had to move, 8 bytes a row for each matrix it
  // reads or writes, and the products that it stands for
  uint64_t bytes = 0, products = 0, adds = 0;
  for (const SlotStep& st : sb.plan.steps) {
    std::vector<int> seen;
    auto once = [&](int k) {
      if (k < 0 || std::find(seen.begin(), seen.end(), k) != seen.end()) return;
      seen.push_back(k);
      bytes += 8ull * sb.n;
    };
    for (int j = 0; j < st.k; ++j) once(st.m[j]);
    for (int k : {st.b, st.s, st.c}) once(k);
    const int gathers = __builtin_popcount(st.bits >> 1);
    products += st.s >= 0 ? std::max(st.k - 1, 0) : 0;
    if (st.c >= 0) products += st.b >= 0 ? gathers + (st.s >= 0 ? 0 : st.k - 1) : (st.s >= 0 ? 0 : st.k);
    adds += st.c >= 0 && (st.bits & (st.bits - 1)) ? __builtin_popcount(st.bits) - 1 : 0;
  }
  ctx->stats.alg_bytes += bytes;
  ctx->stats.spgemm_alg_bytes += bytes;
  ctx->stats.spgemm_calls += products;
  ctx->stats.spgemm_light += products;
  ctx->stats.spgemm_fused_adds += adds;
  ctx->stats.spgemm_slow_rows += c.ctl.slow_rows;
  return true;
}

static SlotPart whole(const dvg_matrix* a) {
  SlotPart p{};
  p.rowmap = a->rowmap;
  p.entries = a->entries;
  p.n = a->nrows;
  return p;
}

static dvg_matrix* run_slots(dvg_context* ctx, const SlotPlan& plan, const dvg_matrix* a, const dvg_matrix* b,
                             const SlotKey& key, bool build, bool* settled) {
  SlotBuild sb;
  try {
    sb = prepare_slots(ctx, plan, a->nrows, false);
    sb.key = key;
  } catch (const Error& e) {
    if (e.status != DVG_ERR_OOM) throw;
    return nullptr;
  }
  dvg_matrix* m = nullptr;
  if (build) sb.early = std::min(sb.early, uint64_t(ctx->early_growth * double(a->nrows)) + kEarlySpare);
  sb.close = a->nrows <= (plan.steps.size() == 1 ? kEarlyRows : kCloseRows);
  try {
    SlotParts parts{};
    parts.one = whole(a);
    const SlotPart right = b ? whole(b) : SlotPart{};
    launch_slots(ctx, sb, parts, ctx->opt_timing, b ? &right : nullptr);
    auto out = [&](uint64_t ranges, DeviceControl* ctl) {
      m = new_matrix(ctx, a->nrows, a->ncols, 2 * ranges);
      m->canonical = true;
      parts.one.c_rowmap = m->rowmap;
      parts.one.c_entries = m->entries;
      parts.one.c_ranges = ranges;
      launch_slots_out(ctx, sb, parts, ctl);
    };
    try {
      if (sb.early) out(sb.early, sb.ctl);
    } catch (const Error& e) {
      if (e.status != DVG_ERR_OOM) throw;
    }
    auto* h = static_cast<SlotCounters*>(host_stage(ctx, sizeof(SlotCounters)));
    DVG_CUDA(cudaMemcpyAsync(h, sb.scratch, sizeof(SlotCounters), cudaMemcpyDeviceToHost, ctx->stream));
    const uint64_t t0 = now_ns();
    DVG_CUDA(cudaStreamSynchronize(ctx->stream));
    ctx->stats.host_sync_ns += now_ns() - t0;
    ctx->stats.host_syncs++;
    resolve_spans(ctx);
    const SlotCounters c = *h;
    const bool whole_chain = check_slots(ctx, sb, c);
    if (m && (!whole_chain || c.ctl.total > m->nentries)) {
      free_matrix(ctx, m);
      m = nullptr;
    }
    bool ended = m != nullptr;
    if (m) {
      if (c.ctl.status)
        throw Error(DVG_ERR_DEVICE, "row slots: a result and its counts differ (code " + std::to_string(c.ctl.status) + ")");
    } else if (whole_chain) {
      try {
        out(c.ctl.total / 2, nullptr);
      } catch (const Error& e) {  // beside the chain's buffers; in range CRS it may fit
        if (e.status != DVG_ERR_OOM) throw;
      }
    }
    if (m) {
      const uint64_t room = m->nentries;
      m->nentries = c.ctl.total;
      m->nnz = c.ctl.nnz;
      if (build) {
        ctx->early_growth = std::clamp(kEarlySlack * double(c.ctl.total / 2) / double(a->nrows), kEarlySlack, 2.0);
        if (give_back(ctx, m, room)) ended = false;
      }
      if (settled) *settled = ended;
    }
  } catch (...) {
    free_matrix(ctx, m);
    release_slots(ctx, sb);
    throw;
  }
  release_slots(ctx, sb);
  return m;
}

dvg_matrix* slots_chain(dvg_context* ctx, const dvg_matrix* a, unsigned dlo, unsigned dup, bool build, bool* settled) {
  return run_slots(ctx, plan_slots(dlo, dup, branching(a->nnz, a->nrows)), a, nullptr, slot_key(dlo, dup, a), build,
                   settled);
}

bool slots_product_suits(const dvg_context* ctx, const dvg_matrix* a, const dvg_matrix* b) {
  return a->nrows >= kProductRows && a->nrows == b->nrows && slots_suit(ctx, a) && slots_suit(ctx, b);
}

dvg_matrix* slots_product(dvg_context* ctx, const dvg_matrix* a, const dvg_matrix* b, bool* settled) {
  SlotPlan pl;
  pl.inputs = a == b ? 1 : 2;
  pl.out = pl.inputs;
  pl.nmats = pl.inputs + 1;
  SlotStep st;  // c = S_1 B, S_1 = A
  st.k = 1;
  st.m[0] = 0;
  st.b = pl.inputs - 1;
  st.bits = 2;
  st.c = pl.out;
  pl.steps.push_back(st);
  return run_slots(ctx, pl, a, a == b ? nullptr : b, product_key(a, b), false, settled);
}

}  // namespace dvg
