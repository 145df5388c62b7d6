// dvg_spgemm_wide.cu -- range SpGEMM for products whose rows name many B
// ranges (long A ranges over wide B rows): a warp per C row.
//
// Same result as the reference's symbolic + numeric SpGEMM
// (include/diverg/range_sparse.hpp:1132-1442 in cartoonist/diverg, dispatched
// by range_spgemm :2215-2281): row r of C is the union of the ranges of B
// rows s..f for every range [s, f] of A's row r, emitted as sorted maximal
// runs (merge rule start <= hi + 1).
//
// A warp takes a C row.  Its lanes load the row's A ranges and, for each, the
// bounds of the B slice it names (B rows s..f are contiguous in B's entries),
// all at once; the slices are then read with coalesced loads, a first time for
// the row's column bounds and a second time (from L1) to OR every range into a
// bitmap window of the warp in shared memory (two word masks a range, plus a
// "reach" mark for the words a long range covers whole, as the reference's
// HBitVector sets runs).  The runs come out of the window with the map01 /
// map10 boundary masks of hbitvector.hpp:576-597 (gather_chunk); a row wider
// than the window takes further windows.  The cost is per B range named, not
// per column.  Where B's rows are named often enough, the product reads bitmaps
// of unions of B rows instead (BandTables, band_rows): two steps an A range.
//
// Chunks of kWRows rows are taken from a ticket by persistent CTAs; the warps
// of a CTA walk its rows (runs kept in a per-warp buffer), a chunk-local
// prefix gives offsets, the chunk's aggregate is published and its image --
// the whole chunk's output -- waits in shared memory to be resolved one
// iteration later by a warp look-back (by then its predecessors have long
// published), then written out with coalesced stores.  A chunk whose output
// does not fit the image is resolved and written in its own iteration.  Reads
// A and B once (plus L1 re-reads), writes C once.  Waits are bounded.
#include "dvg_spgemm_common.cuh"

namespace dvg {
namespace {

#ifndef DVG_WIDE_THREADS
#define DVG_WIDE_THREADS 256
#endif
#ifndef DVG_WIDE_ROWS
#define DVG_WIDE_ROWS 128
#endif
#ifndef DVG_WIDE_MINB
#define DVG_WIDE_MINB 4
#endif
constexpr int kWThreads = DVG_WIDE_THREADS;
constexpr int kWWarps = kWThreads / 32;
constexpr int kWRows = DVG_WIDE_ROWS;  // rows of a chunk
// With the tables a chunk is 64 rows: 128 are 3 % faster where a row holds few runs
// (1.06 against 1.09 ms on 2^20 rows of 9 entries), but a chunk of more than 2,048
// entries misses its image and waits for its place (16 entries a row: 4.3 ms
// against 1.3; 22 a row: 1.9 against 1.1).
constexpr uint32_t kWBandRows = 64, kWRowsMin = 64;
constexpr int kWRowsLane = kWRows / 32;  // rows of the chunk prefix a lane sums
static_assert(kWRows % 32 == 0 && kWRowsLane >= 1, "chunk rows are a multiple of 32");
constexpr int kWWin = 128;     // window words of a warp (4,096 columns)
constexpr int kWBuf = 256;     // run entries of a warp's rows kept from the count
constexpr int kWImage = 2048;  // output entries of a chunk held for its deferred write-out

template <bool BAND>
struct WideSmem {
  // a warp's windows: one row's bits and reach, or four rows' bits
  uint32_t win[kWWarps][(BAND ? 4 : 2) * kWWin];
  uint32_t buf[kWWarps][kWBuf];  // runs of the warp's rows of the counted chunk, in row order
  uint32_t img[2][kWImage];      // images of the counted and the pending chunk
  uint32_t incl[2][kWRows];      // their chunk-local inclusive row counts
  uint32_t cnt_row[kWRows];      // entries of each row of the counted chunk
  uint32_t kept[kWRows];         // 1: the row's runs are in its warp's buffer
  unsigned long long prefix[2];  // exclusive prefixes: the pending chunk's, a chunk written in place
  uint32_t pend_t[2], pend_rows[2], pend_cnt[2];
  uint32_t next;
  uint32_t cnt;
};

__device__ __forceinline__ void wide_sync() { asm volatile("barrier.sync 0;" ::: "memory"); }

// Warp 0 walks back from chunk t (its aggregate published) to the nearest
// inclusive prefix, publishes t's inclusive prefix (and, for the last chunk,
// the product's total, with the overflow check) and leaves t's exclusive
// prefix in *out; the caller's barrier makes it visible.  Bounded.
__device__ void wide_lookback(unsigned long long* out, const FusedArgs& p, uint32_t t, unsigned long long cnt) {
  const int lane = lane_id();
  ChunkDesc* d = p.desc;
  unsigned long long pre = 0;
  int64_t j = int64_t(t) - 1;
  uint32_t spins = 0;
  const uint32_t limit = p.spin_limit ? p.spin_limit : kSpinLimit;
  while (j >= 0) {
    const int64_t idx = j - lane;
    int st = 2;  // 2: inclusive prefix (or before chunk 0), 1: aggregate, 0: nothing yet
    unsigned long long v = 0;
    if (idx >= 0) {
      unsigned long long va, vi;
      asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(va), "=l"(vi) : "l"(&d[idx].agg) : "memory");
      if (vi & kFlag) {
        v = vi & ~kFlag;
      } else if (va & kFlag) {
        st = 1;
        v = va & ~kFlag;
      } else {
        st = 0;
      }
    }
    const unsigned im = __ballot_sync(kFullMask, st == 2), wm = __ballot_sync(kFullMask, st == 0);
    const int fi = im ? __ffs(im) - 1 : 32;
    const unsigned before = fi == 32 ? kFullMask : ((1u << fi) - 1u);
    if (wm & before) {
      if (++spins > limit) {
        if (lane == 0) raise_flag(p, &p.ctl->timeout, 1ull);
        break;
      }
      __nanosleep(32);
      continue;
    }
    unsigned long long sv = lane <= fi ? v : 0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sv += __shfl_xor_sync(kFullMask, sv, o);
    pre += sv;
    if (fi < 32) break;
    j -= 32;
  }
  if (lane == 0) {
    st_relaxed(&d[t].incl, kFlag | (pre + cnt));
    *out = pre;
    if (t == p.nchunks - 1) {
      p.ctl->total = pre + cnt;
      if (pre + cnt > p.cap) raise_flag(p, &p.ctl->overflow, pre + cnt);
    }
  }
}

// Four consecutive rows of C = A B, from `row` on (`rows` of them), from the tables
// of unions of B rows, eight lanes a row: an A range [s, f] is the rows' union in
// steps of the largest table that fits (the last step ends at f and may overlap
// the one before).  A step ORs a table's row into the row's window in shared
// memory, 16 bytes a lane: window quad q belongs to lane q % 8, so that no two
// lanes meet on one, and a step is ORed in once the next one's loads are under
// way.  Runs out: keep(place, value) for entry `place` of the four rows' runs
// together; cnt[g] takes row g's entries, or kByRange where the row has more A
// ranges than kBandRanges or is wider than the window and has to be walked range
// by range.
//
// Bound: latency, and instructions: a row's chain of dependent steps (row pointers,
// ranges, block boxes, table rows, the ORs), with 32 warps an SM to hide it (64 registers
// a thread) and issue slots 56 % busy.  An A range takes two steps, a row about 460
// instructions instead of the 1,300 of ORing each of its ~100 B ranges with two shared
// atomics.  On the
// banded product of 4.2e6 rows (half-width 512, four ranges of ~32 columns a row)
// 6.54 -> 4.00 ms, 1.0 of it the tables; 3.2e6 rows whose products hold 16 entries
// a row, 37.1 -> 3.7 ms.  A warp a row, its window in registers,
// took 930 (a word a lane) and 720 instructions a row (16 bytes a lane): a step
// covers ten 16-byte words, so most lanes were idle.
constexpr uint32_t kBandMaxWords = 64;  // of a table's row: two quads for each of a row's eight lanes
constexpr uint32_t kByRange = 0xffffffffu;
// The table that a range of `len` rows steps in, and the rows of a step.
__device__ __forceinline__ uint32_t band_level(uint32_t len) {
  return len >= 4 ? min(30u - uint32_t(__clz(len)), uint32_t(kBandLevels) - 1) : 0u;  // 4: 1, 8: 2, .. 64: 5
}
__device__ __forceinline__ uint32_t band_by(uint32_t level) { return level ? 2u << level : 1u; }
constexpr uint32_t kBandRanges = 64;
template <class Keep>
__device__ __forceinline__ void band_rows(const FusedArgs& p, uint64_t row, uint32_t rows, uint4* window, uint32_t* cnt,
                                          unsigned long long& nnz, Keep&& keep) {
  static_assert(kWWin == 128, "sixteen window words a lane");
  const int lane = lane_id(), g = lane >> 3, l = lane & 7;
  uint4* const win = window + g * (kWWin / 4);
  uint64_t a0 = 0, a1 = 0;
  if (uint32_t(g) < rows) {
    a0 = __ldg(p.a_rowmap + row + g) >> 1;
    a1 = __ldg(p.a_rowmap + row + g + 1) >> 1;
  }
  // a step: where its table's row starts, and its box (the quads that it covers)
  const uint32_t quads = p.band.stride / 4;
  auto place = [&](uint32_t level, uint32_t j, uint2 box) {
    return level * uint32_t(p.band.table) + j / kBandBlock * (kBandBlock * quads) + j % kBandBlock * (box.y / 4);
  };
  // a range's first and last step, and whether it has more between them
  struct Range {
    uint32_t q[2];
    uint2 box[2];
    uint32_t steps;  // 0: no range
    bool more;
  };
  auto range = [&](uint64_t k) {
    Range r{{0, 0}, {make_uint2(0u, 0u), make_uint2(0u, 0u)}, 0, false};
    if (k >= a1) return r;
    const uint2 ar = load_range(p.a_entries, k);
    if (ar.y < ar.x) return r;
    const uint32_t level = band_level(ar.y - ar.x + 1), last = ar.y + 1 - band_by(level);
    r.box[0] = __ldg(p.band.blk + ar.x / kBandBlock);
    r.box[1] = __ldg(p.band.blk + last / kBandBlock);
    r.q[0] = place(level, ar.x, r.box[0]);
    r.q[1] = place(level, last, r.box[1]);
    r.steps = last == ar.x ? 1u : 2u;
    r.more = last - ar.x > band_by(level);
    return r;
  };
  uint32_t lo = 0xffffffffu, hi = 0;
  auto cover = [&](uint2 w) {
    if (w.y) {
      lo = min(lo, w.x);
      hi = max(hi, w.x + w.y);
    }
  };
  const Range mine = range(a0 + l);
  const bool many = a1 - a0 > kBandRanges;
  bool more = false;  // some range of the row has steps between its first and last
  for (uint64_t k = a0 + l; k < a1 && !many; k += 8) {
    const Range w = k == a0 + l ? mine : range(k);
    if (!w.steps) continue;
    cover(w.box[0]);
    cover(w.box[1]);
    more |= w.more;
    if (w.more) {
      const uint2 ar = load_range(p.a_entries, k);
      for (uint32_t b = ar.x / kBandBlock + 1; b < ar.y / kBandBlock; ++b) cover(__ldg(p.band.blk + b));
    }
  }
  __syncwarp();
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(kFullMask, lo, o));
    hi = max(hi, __shfl_xor_sync(kFullMask, hi, o));
  }
  // the window's last word stays empty, which ends the last run
  const bool walk = many || (lo < hi && hi - lo > uint32_t(kWWin) - 4);
#pragma unroll
  for (int i = 0; i < kWWin / 32; ++i) win[i * 8 + l] = make_uint4(0u, 0u, 0u, 0u);
  uint4 v0 = make_uint4(0u, 0u, 0u, 0u), v1 = v0;
  uint32_t to0 = l, to1 = l;  // where they go (quads of the lane's)
  auto flush = [&](uint32_t to, uint4 v) {
    uint4 x = win[to];
    x.x |= v.x;
    x.y |= v.y;
    x.z |= v.z;
    x.w |= v.w;
    win[to] = x;
  };
  // (at, n): the step's first quad in the window, and how many
  auto step = [&](uint32_t q, uint32_t at, uint32_t n) {
    const uint32_t k = (l - at) & 7u;
    const uint4* __restrict__ t = p.band.t + (q + k);
    uint4 n0 = make_uint4(0u, 0u, 0u, 0u), n1 = n0;
    if (k < n) n0 = __ldg(t);
    if (k + 8 < n) n1 = __ldg(t + 8);
    flush(to0, v0);
    flush(to1, v1);
    v0 = n0;
    v1 = n1;
    if (k < n) to0 = at + k;
    if (k + 8 < n) to1 = at + k + 8;
  };
  auto boxed = [&](uint2 b) { return b.y ? (b.x - lo) / 4 << 16 | b.y / 4 : 0u; };
  // every range's first and last step, range k's from lane k % 8 of its row (the
  // trip counts are the warp's, so that its lanes stay together)
  const uint32_t count = walk ? 0u : uint32_t(a1 - a0);
  const uint32_t most = __reduce_max_sync(kFullMask, count);
  Range r = mine;
  uint32_t box0 = boxed(r.box[0]), box1 = boxed(r.box[1]);
  for (uint32_t k = 0; k < most; ++k) {
    const int src = (lane & 24) + (k & 7);
    if (k >= 8 && (k & 7) == 0) {  // (rows of more than eight ranges)
      r = range(a0 + k + l);
      box0 = boxed(r.box[0]);
      box1 = boxed(r.box[1]);
    }
    const uint32_t steps = __shfl_sync(kFullMask, r.steps, src);
    const uint32_t q0 = __shfl_sync(kFullMask, r.q[0], src), q1 = __shfl_sync(kFullMask, r.q[1], src);
    const uint32_t w0 = __shfl_sync(kFullMask, box0, src), w1 = __shfl_sync(kFullMask, box1, src);
    if (k < count) {
      step(q0, w0 >> 16, steps ? w0 & 0xffffu : 0u);
      if (steps > 1) step(q1, w1 >> 16, w1 & 0xffffu);
    }
    __syncwarp();
  }
  // the steps between, of ranges of 128 rows and more
  if (__any_sync(kFullMask, more && !walk)) {
    for (uint32_t k = 0; k < most; ++k) {
      if (k >= count) continue;
      const uint2 ar = load_range(p.a_entries, a0 + k);
      if (ar.y < ar.x) continue;
      const uint32_t level = band_level(ar.y - ar.x + 1), by = band_by(level);
      for (uint32_t j = ar.x + by; j < ar.y + 1 - by; j += by) {
        const uint2 b = __ldg(p.band.blk + j / kBandBlock);
        const uint32_t w = boxed(b);
        step(place(level, j, b), w >> 16, w & 0xffffu);
      }
    }
    __syncwarp();
  }
  flush(to0, v0);
  flush(to1, v1);
  __syncwarp();
  // runs: the lane takes words 16 l .. 16 l + 15; where a column differs from the one
  // before, a run starts or has ended
  uint32_t n = 0, some = 0;
  const uint32_t* const words = reinterpret_cast<const uint32_t*>(win);
  if (!walk && lo < hi && 16 * l <= int(hi - lo)) {
    uint32_t prev = l ? words[16 * l - 1] : 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 x = win[4 * l + i];
      const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t b = w[k] ^ __funnelshift_l(prev, w[k], 1);
        n += __popc(b);
        some |= (b ? 1u : 0u) << (4 * i + k);
        nnz += __popc(w[k]);
        prev = w[k];
      }
    }
  }
  __syncwarp();
  uint32_t incl = group_incl_sum<32>(kFullMask, n, lane);
  const uint32_t before = incl - n;
  const uint32_t ends = __shfl_sync(kFullMask, incl, lane | 7);
  uint32_t start = __shfl_sync(kFullMask, incl, ((lane & 24) - 1) & 31);
  if (g == 0) start = 0;
  if (l == 0 && uint32_t(g) < rows) cnt[g] = walk ? kByRange : ends - start;
  uint32_t k = before;
  for (; some; some &= some - 1) {
    const int i = __ffs(some) - 1;
    const uint32_t w = words[16 * l + i], prev = 16 * l + i ? words[16 * l + i - 1] : 0u;
    const uint32_t col = 32u * (lo + 16u * l + i);
    for (uint32_t d = w ^ __funnelshift_l(prev, w, 1); d; d &= d - 1, ++k)
      keep(k, col + uint32_t(__ffs(d) - 1) - ((k - start) & 1u));
  }
  __syncwarp();
}

template <bool BAND>
__global__ void __launch_bounds__(kWThreads, DVG_WIDE_MINB) k_spgemm_wide(const __grid_constant__ FusedArgs p) {
  extern __shared__ __align__(16) unsigned char wide_smem_raw[];
  auto& S = *reinterpret_cast<WideSmem<BAND>*>(wide_smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t* const bits = S.win[warp];
  uint32_t* const reach = bits + kWWin;
  uint32_t* const buf = S.buf[warp];
  unsigned long long nnz_acc = 0;
  // the warp's rows of a chunk, in the order in which its buffer keeps them
  constexpr uint32_t kRun = BAND ? 4 : 1;  // consecutive ones
  auto each_row = [&](uint32_t crows, auto&& f) {
    if constexpr (!BAND) {
      for (uint32_t r = warp; r < crows; r += kWWarps) f(r);
    } else {
      for (uint32_t r0 = warp * kRun; r0 < crows; r0 += kWWarps * kRun)
        for (uint32_t r = r0; r < min(r0 + kRun, crows); ++r) f(r);
    }
  };
  if (tid == 0) S.next = atomicAdd(p.ticket, 1u);
  wide_sync();
  uint32_t t = S.next, b = 0;
  bool pend = false;  // a counted chunk waits in image buffer b ^ 1
  while (t < p.nchunks || pend) {
    const bool have = t < p.nchunks;
    const uint32_t c0 = have ? t * p.chunk_rows : 0u;
    const uint32_t crows = have ? min(p.chunk_rows, p.nrows - c0) : 0u;
    uint32_t cnt = 0;
    bool imaged = false;
    if (have) {
      // 1. count: warp w walks rows w, w + kWWarps, ...; their runs go to its buffer
      uint32_t bpos = 0;
      if constexpr (BAND) {
        uint4* const window = reinterpret_cast<uint4*>(S.win[warp]);
        for (uint32_t r = warp * kRun; r < crows; r += kWWarps * kRun) {
          const uint32_t start = bpos, rows = min(kRun, crows - r);
          band_rows(p, uint64_t(c0) + r, rows, window, S.cnt_row + r, nnz_acc, [&](uint32_t k, uint32_t v) {
            if (start + k < uint32_t(kWBuf)) buf[start + k] = v;
          });
          __syncwarp();
          const uint32_t c = uint32_t(lane) < rows ? S.cnt_row[r + lane] : 0u;
          const unsigned walk = __ballot_sync(kFullMask, c == kByRange);
          const uint32_t upto = bpos + group_incl_sum<32>(kFullMask, c == kByRange ? 0u : c, lane);
          if (uint32_t(lane) < rows) S.kept[r + lane] = c != kByRange && upto <= uint32_t(kWBuf) ? 1u : 0u;
          // (rows that fit lie where they are even if the buffer has no room for later ones)
          bpos = __shfl_sync(kFullMask, upto, 31);
          for (unsigned m = walk; m; m &= m - 1) {
            const uint32_t j = __ffs(m) - 1;
            const uint64_t n = wide_row<kWWin>(p, uint64_t(c0) + r + j, bits, reach, &nnz_acc, [](uint64_t, uint32_t) {});
            if (n > 0xfffffffeull) raise_flag(p, &p.ctl->status, 16ull);
            if (lane == 0) S.cnt_row[r + j] = uint32_t(n);
          }
        }
      } else
      for (uint32_t r = warp; r < crows; r += kWWarps) {
        const uint32_t start = bpos;
        const uint64_t c = wide_row<kWWin>(p, uint64_t(c0) + r, bits, reach, &nnz_acc, [&](uint64_t k, uint32_t v) {
          if (start + k < uint64_t(kWBuf)) buf[start + k] = v;
        });
        const bool kept = start + c <= uint64_t(kWBuf);
        if (c > 0xffffffffull) raise_flag(p, &p.ctl->status, 16ull);
        if (lane == 0) {
          S.cnt_row[r] = uint32_t(c);
          S.kept[r] = kept ? 1u : 0u;
        }
        if (kept) bpos += uint32_t(c);
      }
      wide_sync();
      // 2. chunk-local prefix (warp 0: kWRowsLane consecutive rows a lane)
      if (warp == 0) {
        uint32_t v[kWRowsLane];
        uint64_t sum = 0;
#pragma unroll
        for (int k = 0; k < kWRowsLane; ++k) {
          const uint32_t r = kWRowsLane * lane + k;
          v[k] = r < crows ? S.cnt_row[r] : 0u;
          sum += v[k];
        }
        uint64_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint64_t u = __shfl_up_sync(kFullMask, incl, o);
          if (lane >= o) incl += u;
        }
        const uint64_t total = __shfl_sync(kFullMask, incl, 31);
        if (total > 0xffffffffull) {
          if (lane == 0) raise_flag(p, &p.ctl->status, 16ull);
        }
        uint64_t run = incl - sum;
#pragma unroll
        for (int k = 0; k < kWRowsLane; ++k) {
          const uint32_t r = kWRowsLane * lane + k;
          run += v[k];
          if (r < crows) S.incl[b][r] = uint32_t(run);
        }
        if (lane == 0) {
          S.cnt = uint32_t(total);
          publish_aggregate(p, t, total);
          S.next = atomicAdd(p.ticket, 1u);  // the next chunk, taken once this one is counted
        }
      }
      wide_sync();
      cnt = S.cnt;
      // 3. the chunk's image in buffer b: kept rows copied, the rest walked again
      imaged = cnt <= uint32_t(kWImage);
      if (imaged) {
        uint32_t* img = S.img[b];
        uint32_t bp = 0;
        auto image_row = [&](uint32_t r) {
          const uint32_t n = S.cnt_row[r], o = r ? S.incl[b][r - 1] : 0u;
          if (S.kept[r]) {
            for (uint32_t k = lane; k < n; k += 32) img[o + k] = buf[bp + k];
            bp += n;
          } else {
            bool bad = false;
            const uint64_t c = wide_row<kWWin>(p, uint64_t(c0) + r, bits, reach, nullptr, [&](uint64_t k, uint32_t v) {
              if (k < n) img[o + k] = v;
              else bad = true;
            });
            if (bad || c != n) raise_flag(p, &p.ctl->status, 8ull);
          }
        };
        if constexpr (BAND) {
          for (uint32_t r0 = warp * kRun; r0 < crows; r0 += kWWarps * kRun) {
            const uint32_t rows = min(kRun, crows - r0);
            if (__all_sync(kFullMask, uint32_t(lane) >= rows || S.kept[r0 + lane])) {
              // consecutive rows in the buffer and in the image
              const uint32_t o = r0 ? S.incl[b][r0 - 1] : 0u, n = S.incl[b][r0 + rows - 1] - o;
              for (uint32_t k = lane; k < n; k += 32) img[o + k] = buf[bp + k];
              bp += n;
            } else {
              for (uint32_t r = r0; r < r0 + rows; ++r) image_row(r);
            }
          }
        } else {
          each_row(crows, image_row);
        }
      }
    }
    // 4. the pending chunk (counted last iteration): look-back, row map, entries
    if (pend) {
      const uint32_t pt = S.pend_t[b ^ 1u], prow = S.pend_rows[b ^ 1u], pcnt = S.pend_cnt[b ^ 1u];
      if (warp == 0) wide_lookback(&S.prefix[0], p, pt, pcnt);
      wide_sync();
      const unsigned long long prefix = S.prefix[0];
      for (uint32_t r = tid; r < prow; r += kWThreads)
        p.c_rowmap[uint64_t(pt) * p.chunk_rows + r + 1] = prefix + S.incl[b ^ 1u][r];
      if (pt == 0 && tid == 0) p.c_rowmap[0] = 0;
      if (prefix + pcnt <= p.cap) {
        uint32_t* dst = p.c_entries + prefix;
        for (uint32_t k = tid; k < pcnt; k += kWThreads) dst[k] = S.img[b ^ 1u][k];
      } else if (tid == 0 && pcnt) {
        raise_flag(p, &p.ctl->overflow, 1ull);
      }
      pend = false;
    }
    // 5. a chunk whose output does not fit its image: resolved now, in place
    if (have && !imaged) {
      if (warp == 0) wide_lookback(&S.prefix[1], p, t, cnt);
      wide_sync();
      const unsigned long long prefix = S.prefix[1];
      for (uint32_t r = tid; r < crows; r += kWThreads) p.c_rowmap[uint64_t(c0) + r + 1] = prefix + S.incl[b][r];
      if (t == 0 && tid == 0) p.c_rowmap[0] = 0;
      uint32_t bp = 0;
      each_row(crows, [&](uint32_t r) {
        const uint32_t n = S.cnt_row[r], o = r ? S.incl[b][r - 1] : 0u;
        const bool kept = S.kept[r] != 0;
        if (n && prefix + o + n > p.cap) {
          if (lane == 0) raise_flag(p, &p.ctl->overflow, 1ull);
        } else if (kept) {
          uint32_t* dst = p.c_entries + prefix + o;
          for (uint32_t k = lane; k < n; k += 32) dst[k] = buf[bp + k];
        } else if (n) {
          uint32_t* dst = p.c_entries + prefix + o;
          bool bad = false;
          const uint64_t c = wide_row<kWWin>(p, uint64_t(c0) + r, bits, reach, nullptr, [&](uint64_t k, uint32_t v) {
            if (k < n) dst[k] = v;
            else bad = true;
          });
          if (bad || c != n) raise_flag(p, &p.ctl->status, 8ull);
        }
        if (kept) bp += n;
      });
    }
    if (have && imaged) {
      if (tid == 0) {
        S.pend_t[b] = t;
        S.pend_rows[b] = crows;
        S.pend_cnt[b] = cnt;
      }
      pend = true;
      b ^= 1u;
    }
    // every thread is done with the buffers and images it needs; S.next and
    // the pending record are visible
    wide_sync();
    t = have ? S.next : 0xffffffffu;
  }
  // the product's nnz: one atomic per warp
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) nnz_acc += __shfl_xor_sync(kFullMask, nnz_acc, o);
  if (lane == 0 && nnz_acc) atomicAdd(&p.ctl->nnz, nnz_acc);
}

// ---- the tables -----------------------------------------------------------------

// blk[b]: the words, in whole fours, that the ranges of the rows cover that a union
// from block b reaches (the block's and the 63 after them), a warp a block; the
// widest into *widest.
constexpr uint32_t kBandReach = kBandBlock + 63;
__global__ void __launch_bounds__(kWThreads) k_band_blocks(const uint64_t* __restrict__ rowmap,
                                                           const uint32_t* __restrict__ entries, uint32_t nrows,
                                                           uint2* __restrict__ blk, unsigned long long* widest) {
  const int lane = lane_id();
  const uint64_t b = (uint64_t(blockIdx.x) * kWThreads + threadIdx.x) >> 5, r0 = b * kBandBlock;
  if (r0 >= nrows) return;
  const uint64_t e0 = __ldg(rowmap + r0) >> 1, e1 = __ldg(rowmap + min(r0 + kBandReach, uint64_t(nrows))) >> 1;
  uint32_t lo = 0xffffffffu, hi = 0;
  for (uint64_t e = e0 + lane; e < e1; e += 32) {
    const uint2 r = load_range(entries, e);
    if (r.y < r.x) continue;
    lo = min(lo, (r.x >> 5) & ~3u);
    hi = max(hi, ((r.y >> 5) & ~3u) + 4u);
  }
  lo = group_min<32>(kFullMask, lo);
  hi = group_max<32>(kFullMask, hi);
  if (lane == 0) {
    blk[b] = lo < hi ? make_uint2(lo, hi - lo) : make_uint2(0u, 0u);
    if (lo < hi) atomicMax(widest, (unsigned long long)(hi - lo));
  }
}

// The unions from a block's rows: the rows that they reach as bitmaps in shared
// memory, then in place 4 rows' unions from those, 8 from 4 and so on to 64, each
// written out on the way.
// Bound: the tables' writes, 24 bytes a word of a row's band.
constexpr uint32_t kBandRows = kBandBlock + 64;  // rows in shared memory (the last of them empty)
__global__ void __launch_bounds__(kWThreads) k_band_tables(const uint64_t* __restrict__ rowmap,
                                                           const uint32_t* __restrict__ entries, uint32_t nrows,
                                                           BandTables t, uint4* __restrict__ out) {
  extern __shared__ __align__(16) uint4 band_smem[];
  static_assert(2 * kBandRows == kWThreads, "two threads a row");
  constexpr int kMine = kBandMaxWords / 4 * kBandRows / kWThreads;  // quads of a thread
  const uint32_t r0 = kBandBlock * blockIdx.x, tid = threadIdx.x;
  const uint2 box = t.blk[blockIdx.x];
  const uint32_t v = box.y / 4;  // 16-byte words of a row
  if (v == 0) return;            // nothing there: no step reads these
  const uint32_t all = kBandRows * v;
  for (uint32_t k = tid; k < all; k += kWThreads) band_smem[k] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  const uint32_t r = tid / 2;
  if (r < kBandReach && uint64_t(r0) + r < nrows) {
    uint32_t* const bits = reinterpret_cast<uint32_t*>(band_smem + r * v);
    const uint64_t e1 = __ldg(rowmap + r0 + r + 1) >> 1;
    for (uint64_t e = (__ldg(rowmap + r0 + r) >> 1) + tid % 2; e < e1; e += 2) {
      const uint2 c = load_range(entries, e);
      if (c.y < c.x) continue;
      const uint32_t ws = (c.x >> 5) - box.x, we = (c.y >> 5) - box.x;
      const uint32_t lo = ~0u << (c.x & 31), hi = ~0u >> (31 - (c.y & 31));
      for (uint32_t k = ws; k <= we; ++k) atomicOr(bits + k, (k == ws ? lo : ~0u) & (k == we ? hi : ~0u));
    }
  }
  __syncthreads();
  // the thread's quads tid, tid + kWThreads, ... of the block's rows, kept in
  // registers while the others' are read
  const uint32_t mine = min(kBandBlock, nrows - r0) * v;  // quads that are written out
  uint4* const to = out + size_t(r0) * (t.stride / 4);  // the block's rows, v quads each
  auto either = [](uint4 a, uint4 b) { return make_uint4(a.x | b.x, a.y | b.y, a.z | b.z, a.w | b.w); };
  uint4 q[kMine];
#pragma unroll
  for (int i = 0; i < kMine; ++i) {
    const uint32_t k = tid + i * kWThreads;
    if (k < all) q[i] = band_smem[k];
    if (k < mine) to[k] = q[i];
  }
#pragma unroll 1
  for (int level = 1; level < kBandLevels; ++level) {
    // rows of the level before that one of this level takes besides its own
    const uint32_t by = level == 1 ? 1u : 1u << level, n = level == 1 ? 3u : 1u;
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      const uint32_t k = tid + i * kWThreads;
      if (k >= all) break;
      for (uint32_t m = 1; m <= n; ++m)
        if (k + m * by * v < all) q[i] = either(q[i], band_smem[k + m * by * v]);
      if (k < mine) to[size_t(level) * t.table + k] = q[i];
    }
    if (level + 1 == kBandLevels) break;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kMine; ++i) {
      const uint32_t k = tid + i * kWThreads;
      if (k < all) band_smem[k] = q[i];
    }
    __syncthreads();
  }
}

}  // namespace

// The tables cost about 0.25 us a 1,000 B rows of 40 words, a row walked range by
// range 1.5 ns for each B row that it names: a product has to name B's rows often
// (at 45 times each it gains 13 %, at 113 times 26 % with 1.3e5 rows and 70 % with
// 4.2e6), and one that names fewer than 2^21 is over before the read-back is.
constexpr uint64_t kBandMinUses = 32, kBandMinRows = 1u << 21;

BandTables build_band_tables(dvg_context* ctx, const dvg_matrix* a, const dvg_matrix* b) {
  BandTables none{};
  if (b->nrows == 0 || b->nentries == 0 || a->nnz < kBandMinRows || a->nnz < kBandMinUses * b->nrows) return none;
  const uint32_t blocks = uint32_t((uint64_t(b->nrows) + kBandBlock - 1) / kBandBlock);
  const size_t blk_bytes = (size_t(blocks) * sizeof(uint2) + 255) & ~size_t(255);
  void *head = nullptr, *mem = nullptr;
  try {
    head = dalloc(ctx, blk_bytes + 256);
    auto* blk = static_cast<uint2*>(head);
    auto* widest = reinterpret_cast<unsigned long long*>(static_cast<char*>(head) + blk_bytes);
    DVG_CUDA(cudaMemsetAsync(widest, 0, 8, ctx->stream));
    k_band_blocks<<<(blocks + kWWarps - 1) / kWWarps, kWThreads, 0, ctx->stream>>>(b->rowmap, b->entries, b->nrows, blk,
                                                                                widest);
    DVG_CUDA(cudaGetLastError());
    auto* h = static_cast<unsigned long long*>(host_stage(ctx, 8));
    DVG_CUDA(cudaMemcpyAsync(h, widest, 8, cudaMemcpyDeviceToHost, ctx->stream));
    DVG_CUDA(cudaStreamSynchronize(ctx->stream));
    ctx->stats.host_syncs++;
    ctx->stats.kernel_launches += 2;
    const uint64_t words = *h;
    const size_t table = size_t(b->nrows) * words * 4;
    if (words == 0 || words > kBandMaxWords || kBandLevels * table / 16 > 0xffffffffull ||
        kBandLevels * table > (device_free_bytes(ctx) + ctx->cached_bytes) / 4) {
      dfree(ctx, head);
      return none;
    }
    mem = dalloc(ctx, blk_bytes + kBandLevels * table);
    auto* out = reinterpret_cast<uint4*>(static_cast<char*>(mem) + blk_bytes);
    BandTables t{};
    t.t = out;
    t.table = table / 16;
    t.blk = static_cast<const uint2*>(mem);
    t.stride = uint32_t(words);
    t.mem = mem;
    DVG_CUDA(cudaMemcpyAsync(mem, head, blk_bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    const int smem = int(kBandRows * words * 4);
    DVG_CUDA(cudaFuncSetAttribute(k_band_tables, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    cudaEvent_t ev = span_begin(ctx);
    k_band_tables<<<blocks, kWThreads, smem, ctx->stream>>>(b->rowmap, b->entries, b->nrows, t, out);
    span_end(ctx, ev, kLevels);
    DVG_CUDA(cudaGetLastError());
    ctx->stats.kernel_launches++;
    dfree(ctx, head);
    return t;
  } catch (const Error& e) {
    if (head) dfree(ctx, head);
    if (mem) dfree(ctx, mem);
    if (e.status == DVG_ERR_OOM) return none;  // range by range instead
    throw;
  }
}

size_t spgemm_wide_desc_bytes(uint32_t nrows) {
  return size_t((uint64_t(nrows) + kWRowsMin - 1) / kWRowsMin) * sizeof(ChunkDesc);
}

void launch_spgemm_wide(dvg_context* ctx, const dvg_matrix* a, const dvg_matrix* b, const dvg_matrix* d,
                        uint64_t* c_rowmap, uint32_t* c_entries, uint64_t cap, void* desc, unsigned* ticket,
                        const BandTables* band) {
  const uint32_t n = a->nrows;
  if (n == 0) return;
  FusedArgs p{};
  p.a_rowmap = a->rowmap;
  p.a_entries = a->entries;
  p.b_rowmap = b->rowmap;
  p.b_entries = b->entries;
  p.d_rowmap = d ? d->rowmap : nullptr;
  p.d_entries = d ? d->entries : nullptr;
  p.c_rowmap = c_rowmap;
  p.c_entries = c_entries;
  p.cap = cap;
  p.desc = static_cast<ChunkDesc*>(desc);
  p.ticket = ticket;
  p.ctl = ctx->d_ctl;
  p.nrows = n;
  p.chunk_rows = band ? kWBandRows : kWRows;
  p.nchunks = uint32_t((uint64_t(n) + p.chunk_rows - 1) / p.chunk_rows);
  if (band) p.band = *band;
  auto kern = band ? k_spgemm_wide<true> : k_spgemm_wide<false>;
  const int smem = int(band ? sizeof(WideSmem<true>) : sizeof(WideSmem<false>));
  DVG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  int per_sm = 0;
  DVG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kWThreads, smem));
  if (per_sm < 1) throw Error(DVG_ERR_DEVICE, "wide spgemm: shared memory layout does not fit");
  const unsigned grid = unsigned(std::min<uint64_t>(p.nchunks, uint64_t(per_sm) * ctx->num_sms));
  kern<<<grid, kWThreads, smem, ctx->stream>>>(p);
  DVG_CUDA(cudaGetLastError());
  ctx->stats.kernel_launches++;
}

}  // namespace dvg

// ---- the on-chip rate of a range operation ------------------------------------
//
// The measured denominator of this kernel's on-chip roofline: warps OR 8-byte
// ranges, read from a small table that stays in L1/L2, into their bitmap
// windows exactly as wide_row does (masks, reach marks, shared atomics), 512
// ranges a "row", and take each row's runs out of the window with the same
// gather -- the work of a range operation with none of the A / B indirection,
// the chunk bookkeeping or the write-out.  Ranges lie within 2,048 columns and
// are up to 63 columns long, as in the banded microbenchmark.
namespace dvg {
namespace {

constexpr uint32_t kCalRanges = 4096;
constexpr uint32_t kCalRowsPerWarp = 256;

__global__ void k_rangeop_table(uint2* t) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kCalRanges) return;
  uint32_t h = i * 2654435761u + 12345u;
  h ^= h >> 15;
  h *= 2246822519u;
  h ^= h >> 13;
  const uint32_t s = h % 1984u;
  t[i] = make_uint2(s, s + ((h >> 16) & 63u));
}

__global__ void __launch_bounds__(kWThreads, 4) k_rangeop_calibrate(const uint2* __restrict__ table,
                                                                    unsigned long long* sink) {
  __shared__ uint32_t cal_bits[kWWarps][kWWin];
  __shared__ uint32_t cal_reach[kWWarps][kWWin];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* bits = cal_bits[warp];
  uint32_t* reach = cal_reach[warp];
  const uint32_t gw = blockIdx.x * kWWarps + warp;
  unsigned long long total = 0, nnz = 0;
  for (uint32_t row = 0; row < kCalRowsPerWarp; ++row) {
    for (uint32_t w = lane; w < uint32_t(kWWin); w += 32) {
      bits[w] = 0;
      reach[w] = 0;
    }
    __syncwarp();
    uint32_t top = 0;
    const uint32_t base = gw * 131u + row * 517u;
    for (uint32_t it = 0; it < 16; it += 2) {
      const uint2 x = __ldg(table + ((base + it * 32 + lane) & (kCalRanges - 1)));
      const uint2 y = __ldg(table + ((base + (it + 1) * 32 + lane) & (kCalRanges - 1)));
      for (const uint2 r : {x, y}) {
        const uint32_t ws = r.x >> 5, we = r.y >> 5;
        const uint32_t lo = ~0u << (r.x & 31);
        const uint32_t hi = ~0u >> (31 - (r.y & 31));
        top = max(top, we + 1);
        atomicOr(bits + ws, ws == we ? lo & hi : lo);
        if (ws != we) atomicMax(reach + ws, r.y + 1u);
      }
    }
    __syncwarp();
    const uint32_t nw = min(uint32_t(kWWin), group_max<32>(kFullMask, top) + 1);
    uint64_t count = 0;
    uint32_t carry = 0, run_reach = 0;
    for (uint32_t wb = 0; wb < nw; wb += 32) {
      const uint32_t w = wb + lane;
      const bool valid = w < nw;
      uint32_t x = 0, rr = 0;
      if (valid) {
        x = bits[w];
        rr = reach[w];
      }
      const uint32_t cov = reach_cover(w, rr, run_reach, lane);
      if (valid) x |= cov;
      nnz += __popc(x);
      count += gather_chunk(x, valid, 32ull * w, 32, lane, kFullMask, carry, count, min(31u, nw - 1 - wb),
                            [](uint64_t, uint32_t) {});
    }
    __syncwarp();
    total += count;
  }
  // keeps the work observable
  if (lane == 0) atomicAdd(sink, total + (nnz & 1ull));
}

}  // namespace

double calibrate_range_ops(dvg_context* ctx) {
  void* mem = dalloc(ctx, kCalRanges * sizeof(uint2) + 256);
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  float best = 0.f;
  try {
    auto* table = static_cast<uint2*>(mem);
    auto* sink = reinterpret_cast<unsigned long long*>(static_cast<char*>(mem) + kCalRanges * sizeof(uint2));
    DVG_CUDA(cudaMemsetAsync(sink, 0, 8, ctx->stream));
    k_rangeop_table<<<(kCalRanges + 255) / 256, 256, 0, ctx->stream>>>(table);
    DVG_CUDA(cudaGetLastError());
    DVG_CUDA(cudaEventCreate(&e0));
    DVG_CUDA(cudaEventCreate(&e1));
    const unsigned grid = unsigned(4 * ctx->num_sms);
    for (int rep = 0; rep < 4; ++rep) {  // the first is a warm-up; the best of the rest
      DVG_CUDA(cudaEventRecord(e0, ctx->stream));
      k_rangeop_calibrate<<<grid, kWThreads, 0, ctx->stream>>>(table, sink);
      DVG_CUDA(cudaGetLastError());
      DVG_CUDA(cudaEventRecord(e1, ctx->stream));
      DVG_CUDA(cudaEventSynchronize(e1));
      float ms = 0.f;
      DVG_CUDA(cudaEventElapsedTime(&ms, e0, e1));
      if (rep > 0 && (best == 0.f || ms < best)) best = ms;
    }
    ctx->stats.kernel_launches += 5;
  } catch (...) {
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    dfree(ctx, mem);
    throw;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  dfree(ctx, mem);
  const double ops = double(4 * ctx->num_sms) * kWWarps * kCalRowsPerWarp * 512.0;
  return best > 0.f ? ops / (double(best) * 1e-3) : 0.0;
}

}  // namespace dvg
