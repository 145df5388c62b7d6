// dvg_slots.h -- chains of products in the row-slot format (dvg_slots.cu).
#pragma once

#include <algorithm>

#include "dvg_internal.h"

namespace dvg {

// First start column that marks a row of several runs; columns lie below.
constexpr uint32_t kSlotMulti = 0xFFFF0000u;

constexpr int kChainMax = 6;  // left factors of one pass

// One pass over the rows: with S_0 = I and S_(j+1) = S_j m[j], s = S_k and
// c = union of S_j b over the set bits j (b = -1: the identity).  Matrices are
// numbered, the inputs first; -1: no such output.
struct SlotStep {
  int k = 0;
  int m[kChainMax] = {-1, -1, -1, -1, -1, -1};
  int b = -1;
  unsigned bits = 0;
  int s = -1, c = -1;
};
struct SlotPlan {
  std::vector<SlotStep> steps;
  int inputs = 1;
  int nmats = 1;
  int out = 0;
};
// A^dlo (A + I)^(dup - dlo) as passes over powers of A, for an A whose rows have
// `branching` columns beyond their first on average.
SlotPlan plan_slots(unsigned dlo, unsigned dup, double branching);

// Whether a chain over `a` runs in the row-slot format.
bool slots_suit(const dvg_context* ctx, const dvg_matrix* a);

// A chain may run over several matrices at once, side by side on the diagonal
// (a power of a block-diagonal matrix has the blocks' powers as blocks): each
// from a multiple of kSlotPartRows rows on, the rows between filled with the
// identity's.
constexpr uint32_t kSlotPartRows = 1024;
struct SlotPart {
  const uint64_t* rowmap;      // the part, range CRS
  const uint32_t* entries;
  uint64_t* c_rowmap;          // its result
  uint32_t* c_entries;
  unsigned long long c_ranges; // ranges that c_entries holds
  unsigned long long before;   // ranges of the chain's result before the part's
  uint32_t row0, n;            // its first row in the chain, and its rows
};
struct SlotParts {
  const SlotPart* table;       // device; null: one part, `one`
  const uint32_t* part_of;     // device: part of every kSlotPartRows rows
  SlotPart one;
};

struct SlotCounters {          // the head of a chain's scratch
  DeviceControl ctl;
  char pad[256 - sizeof(DeviceControl)];
  unsigned long long top, abort, wide;
};
struct SlotBuild {
  SlotPlan plan;
  SlotKey key{};
  uint32_t n = 0;
  std::vector<uint2*> mat;     // per matrix, as the launches use them
  std::vector<uint2*> buffers; // theirs
  uint2* arena = nullptr;
  uint64_t arena_cap = 0;      // ranges
  bool close = false;          // the kernels' blocks are placed while the kernel before ends
  uint64_t early = 0;          // room for the result's ranges before their number is known; 0: none
  // counters | places of each pass | the queue, where it is the chain's own | counts of the
  // result | sums of the counts | bitmap
  void* scratch = nullptr;
  size_t cleared = 0;          // its first bytes, up to the counts, which a chain starts by clearing
  uint32_t queue_cap = 0;
  uint32_t* taken = nullptr;
  unsigned long long* queue = nullptr;
  uint32_t epoch = 0;          // its first pass's
  DeviceControl* ctl = nullptr;
  unsigned long long* top = nullptr;
  unsigned long long* abort = nullptr;
  unsigned long long* wide = nullptr;
  unsigned long long* sums = nullptr;
  unsigned long long* group_nnz = nullptr;
  uint32_t* group_cnt = nullptr;
  uint32_t* masks = nullptr;
};

// Allocates what the chain needs (no device work beyond stream-ordered
// allocation); issues it (no host round trip: it may be captured).
// A plan of two inputs takes `right` as its second.
// Chains that run side by side have queues of their own.
SlotBuild prepare_slots(dvg_context* ctx, const SlotPlan& plan, uint32_t n, bool own_queue);
// Device memory that an index build as a chain may take, its input and result included.
uint64_t predict_slots_bytes(uint32_t nrows, uint64_t nentries, unsigned dlo, unsigned dup);
void launch_slots(dvg_context* ctx, SlotBuild& sb, const SlotParts& parts, bool timed, const SlotPart* right = nullptr);
// Ranges and columns of each part's result (device, two words a part), once
// the chain has run.
void launch_slots_totals(dvg_context* ctx, const SlotBuild& sb, const SlotParts& parts, uint32_t nparts,
                         unsigned long long* totals);
// The parts' results, into the arrays that the table now names; `ctl` (null: the
// context's) takes a status where an array is too small.
void launch_slots_out(dvg_context* ctx, const SlotBuild& sb, const SlotParts& parts, DeviceControl* ctl = nullptr);
// Books a finished chain's counters; false when it was given up and there is no result.
bool check_slots(dvg_context* ctx, const SlotBuild& sb, const SlotCounters& c);
void release_slots(dvg_context* ctx, SlotBuild& sb);

// The chain over `a`, waited for once; null when it or its result did not fit.  Sets
// *settled where that wait has seen all of the result's kernels end, and checked them.
// `build`: an index, which holds no more memory than it needs; a power or a product
// keeps the room that was made for it.
dvg_matrix* slots_chain(dvg_context* ctx, const dvg_matrix* a, unsigned dlo, unsigned dup, bool build, bool* settled);

// A B alone, where that is faster than the range-CRS row kernel; null and
// *settled likewise.
bool slots_product_suits(const dvg_context* ctx, const dvg_matrix* a, const dvg_matrix* b);
dvg_matrix* slots_product(dvg_context* ctx, const dvg_matrix* a, const dvg_matrix* b, bool* settled);

// Columns of a row beyond its first, on average: how fast rows leave the single column.
inline double branching(uint64_t nnz, uint64_t nrows) {
  return nnz > nrows ? double(nnz - nrows) / double(nrows) : 0.0;
}

SlotKey slot_key(unsigned dlo, unsigned dup, uint64_t nnz, uint64_t nrows);
inline SlotKey slot_key(unsigned dlo, unsigned dup, const dvg_matrix* a) { return slot_key(dlo, dup, a->nnz, a->nrows); }
inline SlotKey product_key(const dvg_matrix* a, const dvg_matrix* b) {
  return slot_key(1, 0, std::max(a->nnz, b->nnz), a->nrows);
}
// Whether a chain is to be tried: chains like it were not just given up.  Counts the call.
bool slots_due(dvg_context* ctx, const SlotKey& key);

}  // namespace dvg
