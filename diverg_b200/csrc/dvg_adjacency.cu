// dvg_adjacency.cu -- the adjacency matrix of a sequence graph, built on the
// device in range CRS.
//
// Same result as util::range_adjacency_matrix (include/diverg/adjacency.hpp:
// 249-265 in cartoonist/diverg), which builds the Basic adjacency
// (adjacency_matrix, :170-228) and converts it with crs_matrix::append
// (crs_matrix.hpp:197-242):
//   * one row and one column per base (locus); the loci of node ids
//     lower .. upper-1 are numbered in rank order from 0 (id_to_charorder
//     minus that of `lower`);
//   * every locus but a node's last links to the next locus;
//   * a node's last locus links to the first locus of each successor, the
//     columns sorted; the Basic row becomes ranges by extending the open
//     range only with the column right after its end (col == end + 1), so a
//     repeated successor yields a repeated single-column range, as in append.
// nnz is the number of Basic entries, (loci - nodes) + edges.
//
// Kernels: edges are checked, counted per source node and scattered into
// per-node segments (counting sort, any edge order), each node sorts its segment
// and counts its ranges, a scan gives every node's first entry, then a thread
// per locus writes the row map and its row.  The output is allocated for the
// most entries that so many bases and edges can have (a few more than there
// are, in most graphs), so nothing is waited for until the end; a node range's
// edges are counted first.  Where so much does not fit, the entries are counted
// before the output is allocated, and where much of it stays empty, it is given back.
//
// Bound: the matrix's writes, 16 bytes a locus; below ~1e6 loci the launches and
// the one wait.  1e7 loci of 3.4e4 nodes and 4.6e4 edges: 449 -> 163 us a call, of which
// k_adj_rows 128 -> 45 us (a binary search over all nodes for every locus before)
// and the scans 18 -> 5 each (one block a scan before).
#include <algorithm>
#include <cstring>
#include <vector>

#include "dvg_device.cuh"
#include "dvg_internal.h"

namespace dvg {
namespace {

constexpr int kAdjThreads = 256;
constexpr size_t kAdjStaged = 8u << 20;  // input bytes up to which they go through pinned staging

unsigned adj_grid(dvg_context* ctx, uint64_t n) {
  const uint64_t want = (n + kAdjThreads - 1) / kAdjThreads;
  const uint64_t cap = uint64_t(ctx->num_sms) * 16;
  return unsigned(std::max<uint64_t>(1, std::min(want, cap)));
}

struct AdjArgs {
  uint32_t nnodes;            // nodes of the range
  uint32_t lower, upper;      // node ids [lower, upper), 1-based
  uint64_t nedges;            // edges of the whole graph
  const uint32_t* node_len;   // [nnodes]
  const uint32_t* edges;      // [2 nedges]: (from_id, to_id)
  uint64_t* start;            // [nnodes + 1]: first locus of each node
  uint64_t* eoff;             // [nnodes + 1]: first edge slot of each node
  uint64_t* cursor;           // [nnodes]: scatter cursors
  uint32_t* cols;             // [edges of the range]: successor loci
  uint64_t* base;             // [nnodes + 1]: first entry of each node's rows
  uint64_t* start_n;          // their counts, from [1] on: the same arrays where they
  uint64_t* eoff_n;           // are scanned in place
  uint64_t* base_n;
  uint64_t* c_rowmap;
  uint32_t* c_entries;
  DeviceControl* ctl;
};

// start_n[v + 1] = node_len[v], eoff_n[v + 1] = out-degree of node v within the
// range (scanned afterwards).  Bit 2 of invalid: an endpoint that is no node; bit 1: a
// successor outside the range of a node inside it (its column would not exist).
__global__ void k_adj_counts(AdjArgs p, uint32_t all_nodes) {
  const uint64_t t0 = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x, stride = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t v = t0; v < p.nnodes; v += stride) p.start_n[v + 1] = p.node_len[v];
  for (uint64_t e = t0; e < p.nedges; e += stride) {
    const uint32_t from = p.edges[2 * e], to = p.edges[2 * e + 1];
    if (from < 1 || from > all_nodes || to < 1 || to > all_nodes) {
      atomicOr(&p.ctl->invalid, 2ull);
      continue;
    }
    if (from < p.lower || from >= p.upper) continue;
    if (to < p.lower || to >= p.upper) {
      atomicOr(&p.ctl->invalid, 1ull);
      continue;
    }
    atomicAdd(reinterpret_cast<unsigned long long*>(p.eoff_n + (from - p.lower) + 1), 1ull);
  }
}

// Inclusive scans of a[1 .. n] to to_a and b[1 .. n] to to_b, an element a thread.
// A block adds up the elements before its own by itself, from L2, so that no block
// waits for another: for the node counts of most graphs one such launch beats the
// three that a scan over the whole chip takes (two scans of 3.4e4 nodes:
// 33 us, 18 by one block each, 5 so).
constexpr uint32_t kAdjScanThreads = 1024, kAdjScanMax = 1u << 17;
__global__ void __launch_bounds__(kAdjScanThreads) k_adj_scan(const uint64_t* __restrict__ a, uint64_t* to_a,
                                                              const uint64_t* __restrict__ b, uint64_t* to_b,
                                                              uint32_t n) {
  constexpr uint32_t kAhead = 8;
  static_assert(kAdjScanThreads == 32 * 32, "a lane a warp's sums");
  __shared__ uint64_t sums[32], before[32];
  const uint64_t* const x = (blockIdx.y ? b : a) + 1;
  uint64_t* const y = (blockIdx.y ? to_b : to_a) + 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t i0 = blockIdx.x * kAdjScanThreads, i = i0 + threadIdx.x;
  const uint64_t mine = i < n ? x[i] : 0;
  uint64_t sum = 0;
  for (uint32_t j = threadIdx.x; j < i0; j += kAhead * kAdjScanThreads) {
    uint64_t v[kAhead];
#pragma unroll
    for (uint32_t k = 0; k < kAhead; ++k) v[k] = j + k * kAdjScanThreads < i0 ? x[j + k * kAdjScanThreads] : 0;
#pragma unroll
    for (uint32_t k = 0; k < kAhead; ++k) sum += v[k];
  }
  sum = group_sum<32>(kFullMask, sum);
  const uint64_t incl = group_incl_sum<32>(kFullMask, mine, lane);
  if (lane == 0) before[warp] = sum;
  if (lane == 31) sums[warp] = incl;
  __syncthreads();
  const uint64_t run = group_sum<32>(kFullMask, before[lane] + (lane < warp ? sums[lane] : uint64_t(0)));
  if (i < n) y[i] = run + incl;
}

// (counts of more than kAdjScanMax nodes lie in the scanned arrays)
void scan_nodes(dvg_context* ctx, const uint64_t* a, uint64_t* to_a, const uint64_t* b, uint64_t* to_b, uint32_t n) {
  if (n <= kAdjScanMax) {
    k_adj_scan<<<dim3((n + kAdjScanThreads - 1) / kAdjScanThreads, b ? 2 : 1), kAdjScanThreads, 0, ctx->stream>>>(
        a, to_a, b, to_b, n);
    DVG_CUDA(cudaGetLastError());
    ctx->stats.kernel_launches++;
    return;
  }
  launch_rowmap_scan(ctx, to_a, n);
  if (b) launch_rowmap_scan(ctx, to_b, n);
}

// each edge's successor locus into its source node's segment
__global__ void k_adj_scatter(AdjArgs p) {
  for (uint64_t e = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; e < p.nedges; e += uint64_t(gridDim.x) * blockDim.x) {
    const uint32_t from = p.edges[2 * e], to = p.edges[2 * e + 1];  // (what k_adj_counts counted)
    if (from < p.lower || from >= p.upper || to < p.lower || to >= p.upper) continue;
    const uint32_t v = from - p.lower;
    const uint64_t slot = atomicAdd(reinterpret_cast<unsigned long long*>(p.cursor + v), 1ull);
    p.cols[p.eoff[v] + slot] = uint32_t(p.start[to - p.lower]);
  }
}

// Sorts a[0..n) ascending: insertion sort for short segments, heap sort
// (no scratch, n log n) for long ones.
__device__ void sort_segment(uint32_t* a, uint64_t n) {
  if (n <= 32) {
    for (uint64_t i = 1; i < n; ++i) {
      const uint32_t x = a[i];
      uint64_t j = i;
      while (j > 0 && a[j - 1] > x) {
        a[j] = a[j - 1];
        --j;
      }
      a[j] = x;
    }
    return;
  }
  auto sift = [&](uint64_t root, uint64_t end) {
    for (;;) {
      uint64_t child = 2 * root + 1;
      if (child >= end) return;
      if (child + 1 < end && a[child + 1] > a[child]) ++child;
      if (a[root] >= a[child]) return;
      const uint32_t t = a[root];
      a[root] = a[child];
      a[child] = t;
      root = child;
    }
  };
  for (uint64_t i = n / 2; i-- > 0;) sift(i, n);
  for (uint64_t end = n; end > 1; --end) {
    const uint32_t t = a[0];
    a[0] = a[end - 1];
    a[end - 1] = t;
    sift(0, end - 1);
  }
}

// Ranges of a sorted Basic row under append's rule: a column extends the
// open range only when it is the column right after the range's end.
__device__ __forceinline__ uint64_t row_ranges(const uint32_t* a, uint64_t n, bool& repeated) {
  uint64_t r = 0;
  uint32_t end = 0;
  for (uint64_t i = 0; i < n; ++i) {
    if (r && uint64_t(a[i]) == uint64_t(end) + 1) {
      ++end;
      continue;
    }
    if (r && a[i] <= end) repeated = true;
    ++r;
    end = a[i];
  }
  return r;
}

// per node: sort its successor loci, base[v + 1] = the entries of its rows
__global__ void k_adj_nodes(AdjArgs p) {
  for (uint64_t v = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; v < p.nnodes; v += uint64_t(gridDim.x) * blockDim.x) {
    uint32_t* a = p.cols + p.eoff[v];
    const uint64_t n = p.eoff[v + 1] - p.eoff[v];
    sort_segment(a, n);
    bool repeated = false;
    const uint64_t r = row_ranges(a, n, repeated);
    if (repeated) atomicOr(&p.ctl->invalid, 16ull);
    p.base_n[v + 1] = 2 * (uint64_t(p.node_len[v]) - 1) + 2 * r;
  }
}

// Per locus: the row map and the row's ranges.  A block takes kAdjTile consecutive
// loci; their nodes -- the last one that starts at or before the first locus, and
// every one that starts after it within the tile -- are found once, and a locus
// searches only those.
constexpr uint32_t kAdjTile = 1024;
__global__ void __launch_bounds__(kAdjThreads) k_adj_rows(AdjArgs p, uint64_t nloci) {
  __shared__ uint32_t first[kAdjTile + 1];  // first loci of its nodes, from the tile's first (the first node: 0)
  const uint64_t i0 = uint64_t(blockIdx.x) * kAdjTile;
  const uint32_t rows = uint32_t(min(uint64_t(kAdjTile), nloci - i0));
  // the last of `len` nodes from v on that starts at or before x (v does): every
  // thread tries one, a few rounds for any graph
  auto last_at = [&](uint64_t x, uint32_t v, uint32_t len) {
    while (len > 1) {
      const uint32_t step = (len + kAdjThreads - 1) / kAdjThreads, k = threadIdx.x * step;
      const uint32_t c = uint32_t(__syncthreads_count(k < len && p.start[v + k] <= x)) - 1;
      v += c * step;
      len = min(step, len - c * step);
    }
    return v;
  };
  const uint32_t v0 = last_at(i0, 0, p.nnodes);
  // (every node has a locus: at most `rows` nodes)
  const uint32_t n = last_at(i0 + rows - 1, v0, min(rows, p.nnodes - v0)) - v0 + 1;
  for (uint32_t v = threadIdx.x; v < n; v += kAdjThreads) first[v] = v ? uint32_t(p.start[v0 + v] - i0) : 0u;
  __syncthreads();
  for (uint32_t t = threadIdx.x; t < rows; t += kAdjThreads) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) / 2;
      if (first[mid] <= t) lo = mid;
      else hi = mid;
    }
    const uint32_t v = v0 + lo;
    const uint64_t i = i0 + t, k = i - p.start[v];
    const uint64_t at = p.base[v] + 2 * k;
    if (k + 1 < p.node_len[v]) {
      *reinterpret_cast<uint2*>(p.c_entries + at) = make_uint2(uint32_t(i + 1), uint32_t(i + 1));
      p.c_rowmap[i + 1] = at + 2;
    } else {  // the node's last row: its successors
      const uint32_t* a = p.cols + p.eoff[v];
      const uint64_t ns = p.eoff[v + 1] - p.eoff[v], end_at = p.base[v + 1];
      uint64_t w = at;
      auto put = [&](uint32_t lo_col, uint32_t hi_col) {
        if (w + 2 <= end_at) *reinterpret_cast<uint2*>(p.c_entries + w) = make_uint2(lo_col, hi_col);
        w += 2;
      };
      bool open = false;
      uint32_t begin = 0, end = 0;
      for (uint64_t q = 0; q < ns; ++q) {
        if (open && uint64_t(a[q]) == uint64_t(end) + 1) {
          ++end;
          continue;
        }
        if (open) put(begin, end);
        begin = end = a[q];
        open = true;
      }
      if (open) put(begin, end);
      if (w != end_at) atomicOr(&p.ctl->status, 32ull);
      p.c_rowmap[i + 1] = end_at;
    }
    if (i == 0) p.c_rowmap[0] = 0;
  }
}

}  // namespace

dvg_matrix* adjacency_from_graph(dvg_context* ctx, uint32_t nnodes, const uint32_t* node_len, uint64_t nedges,
                                 const uint32_t* edges, uint32_t lower, uint32_t upper) {
  if (upper == 0) upper = nnodes + 1;
  if (nnodes == 0 || lower < 1 || lower > nnodes || upper <= lower || upper > nnodes + 1)
    throw Error(DVG_ERR_INVALID_ARG, "adjacency: node range must satisfy 1 <= lower < upper <= nnodes + 1");
  if (!node_len || (nedges && !edges)) throw Error(DVG_ERR_INVALID_ARG, "adjacency: null argument");
  const uint32_t m = upper - lower;
  const uint32_t* lens = node_len + (lower - 1);
  uint64_t nloci = 0;
  uint32_t shortest = 0xffffffffu;
  for (uint32_t v = 0; v < m; ++v) {
    nloci += lens[v];
    shortest = std::min(shortest, lens[v]);
  }
  if (shortest == 0) throw Error(DVG_ERR_INVALID_ARG, "adjacency: a node has length 0");
  if (nloci > 0xFFFFFFFEull) throw Error(DVG_ERR_OVERFLOW, "adjacency: more loci than 32-bit columns hold");

  AdjArgs p{};
  p.nnodes = m;
  p.lower = lower;
  p.upper = upper;
  p.nedges = nedges;
  p.ctl = ctx->d_ctl;
  std::vector<void*> scratch;
  auto grab = [&](size_t bytes) {
    void* q = dalloc(ctx, bytes);
    scratch.push_back(q);
    return q;
  };
  dvg_matrix* out = nullptr;
  try {
    // the edges, then the lengths
    const size_t edge_bytes = nedges * 8, len_bytes = size_t(m) * 4;
    char* d_in = static_cast<char*>(grab(edge_bytes + len_bytes));
    if (edge_bytes + len_bytes <= kAdjStaged) {
      // one copy from pinned memory, under way while the rest is prepared (two
      // copies of pageable memory are waited for in turn)
      char* h = static_cast<char*>(host_stage(ctx, edge_bytes + len_bytes));
      if (nedges) std::memcpy(h, edges, edge_bytes);
      std::memcpy(h + edge_bytes, lens, len_bytes);
      DVG_CUDA(cudaMemcpyAsync(d_in, h, edge_bytes + len_bytes, cudaMemcpyHostToDevice, ctx->stream));
    } else {
      if (nedges) DVG_CUDA(cudaMemcpyAsync(d_in, edges, edge_bytes, cudaMemcpyHostToDevice, ctx->stream));
      DVG_CUDA(cudaMemcpyAsync(d_in + edge_bytes, lens, len_bytes, cudaMemcpyHostToDevice, ctx->stream));
    }
    ctx->stats.h2d_bytes += edge_bytes + len_bytes;
    p.edges = reinterpret_cast<const uint32_t*>(d_in);
    p.node_len = reinterpret_cast<const uint32_t*>(d_in + edge_bytes);
    // start | eoff | cursor | base, and the counts that the first, second and last
    // are scanned from, all zero at first
    const size_t words = size_t(m) + 1, arrays = m <= kAdjScanMax ? 7 : 4;
    p.start = static_cast<uint64_t*>(grab(arrays * words * 8));
    p.eoff = p.start + words;
    p.cursor = p.eoff + words;
    p.base = p.cursor + words;
    p.start_n = arrays > 4 ? p.base + words : p.start;
    p.eoff_n = arrays > 4 ? p.start_n + words : p.eoff;
    p.base_n = arrays > 4 ? p.eoff_n + words : p.base;
    uint64_t* h_sizes = reinterpret_cast<uint64_t*>(ctx->h_ctl + 1);
    uint64_t most_edges = nedges;  // of the range
    uint64_t cap = 0;              // entries that the result has room for
    auto make_result = [&](uint64_t entries) {
      out = new_matrix(ctx, uint32_t(nloci), uint32_t(nloci), entries);
      cap = entries;
      p.c_rowmap = out->rowmap;
      p.c_entries = out->entries;
    };
    auto allocate = [&]() {
      p.cols = static_cast<uint32_t*>(grab(std::max<uint64_t>(most_edges, 1) * 4));
      try {
        // at most a range a base but the last of a node, and one an edge
        make_result(2 * (nloci - m) + 2 * most_edges);
      } catch (const Error& e) {
        if (e.status != DVG_ERR_OOM) throw;  // (counted first, below)
      }
    };
    const bool whole = m == nnodes;
    if (whole) allocate();
    reset_control(ctx);
    DVG_CUDA(cudaMemsetAsync(p.start, 0, arrays * words * 8, ctx->stream));
    k_adj_counts<<<adj_grid(ctx, std::max<uint64_t>(m, nedges)), kAdjThreads, 0, ctx->stream>>>(p, nnodes);
    DVG_CUDA(cudaGetLastError());
    scan_nodes(ctx, p.start_n, p.start, p.eoff_n, p.eoff, m);
    if (!whole) {  // a component may hold few of the graph's edges: its own number sizes the result
      DVG_CUDA(cudaMemcpyAsync(h_sizes, p.eoff + m, 8, cudaMemcpyDeviceToHost, ctx->stream));
      read_control(ctx);
      most_edges = h_sizes[0];
      allocate();
    }
    if (nedges) {
      k_adj_scatter<<<adj_grid(ctx, nedges), kAdjThreads, 0, ctx->stream>>>(p);
      DVG_CUDA(cudaGetLastError());
    }
    k_adj_nodes<<<adj_grid(ctx, m), kAdjThreads, 0, ctx->stream>>>(p);
    DVG_CUDA(cudaGetLastError());
    scan_nodes(ctx, p.base_n, p.base, nullptr, nullptr, m);
    if (!out) {
      DVG_CUDA(cudaMemcpyAsync(h_sizes, p.base + m, 8, cudaMemcpyDeviceToHost, ctx->stream));
      read_control(ctx);
      make_result(h_sizes[0]);
    }
    k_adj_rows<<<unsigned((nloci + kAdjTile - 1) / kAdjTile), kAdjThreads, 0, ctx->stream>>>(p, nloci);
    DVG_CUDA(cudaGetLastError());
    ctx->stats.kernel_launches += 4 + (nedges ? 1 : 0);
    DVG_CUDA(cudaMemcpyAsync(h_sizes, p.base + m, 8, cudaMemcpyDeviceToHost, ctx->stream));
    DVG_CUDA(cudaMemcpyAsync(h_sizes + 1, p.eoff + m, 8, cudaMemcpyDeviceToHost, ctx->stream));
    DVG_CUDA(cudaMemcpyAsync(ctx->h_ctl, ctx->d_ctl, sizeof(DeviceControl), cudaMemcpyDeviceToHost, ctx->stream));
    const uint64_t t0 = now_ns();
    DVG_CUDA(cudaStreamSynchronize(ctx->stream));
    ctx->stats.host_sync_ns += now_ns() - t0;
    ctx->stats.host_syncs++;
    resolve_spans(ctx);
    const DeviceControl c = *ctx->h_ctl;
    if (c.invalid & 2) throw Error(DVG_ERR_INVALID_ARG, "edge endpoint is not a node id in 1..nnodes");
    if (c.invalid & 1) throw Error(DVG_ERR_INVALID_ARG, "adjacency: an edge leaves the node range [lower, upper)");
    if (c.status) throw Error(DVG_ERR_DEVICE, "adjacency: internal consistency check failed on the device");
    out->nentries = h_sizes[0];
    out->canonical = !(c.invalid & 16);
    out->nnz = (nloci - m) + h_sizes[1];
    if (give_back(ctx, out, cap)) DVG_CUDA(cudaStreamSynchronize(ctx->stream));  // the caller waits no more
  } catch (...) {
    for (void* q : scratch) dfree(ctx, q);
    if (out) free_matrix(ctx, out);
    throw;
  }
  for (void* q : scratch) dfree(ctx, q);
  return out;
}

}  // namespace dvg
