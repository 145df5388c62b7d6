// dvg_slots.h -- chains of products in the row-slot format (dvg_slots.cu).
#pragma once

#include "dvg_internal.h"

namespace dvg {

// First start column that marks a row of several runs; columns lie below.
constexpr uint32_t kSlotMulti = 0xFFFF0000u;

constexpr int kChainMax = 6;  // left factors of one pass

// One pass over the rows: with S_0 = I and S_(j+1) = S_j m[j], s = S_k and
// c = union of S_j b over the set bits j (b = -1: the identity).  Matrices are
// numbered, 0 is the input; -1: no such output.
struct SlotStep {
  int k = 0;
  int m[kChainMax] = {-1, -1, -1, -1, -1, -1};
  int b = -1;
  unsigned bits = 0;
  int s = -1, c = -1;
};
struct SlotPlan {
  std::vector<SlotStep> steps;
  int nmats = 1;
  int out = 0;
};
// A^dlo (A + I)^(dup - dlo) as passes over powers of A.
SlotPlan plan_slots(unsigned dlo, unsigned dup);

// Whether a chain over `a` runs in the row-slot format.
bool slots_suit(const dvg_context* ctx, const dvg_matrix* a);

struct SlotBuild {
  SlotPlan plan;
  uint32_t n = 0;
  std::vector<uint2*> mat;   // per matrix, as the launches use them
  std::vector<char> live;
  uint2* arena = nullptr;
  uint64_t arena_cap = 0;    // ranges
  void* scratch = nullptr;   // counters | sums of the counts | counts of the result's ranges
  DeviceControl* ctl = nullptr;
  unsigned long long* top = nullptr;
  unsigned long long* abort = nullptr;
  unsigned long long* sums = nullptr;
  unsigned long long* group_nnz = nullptr;
  uint32_t* group_cnt = nullptr;
  uint32_t* masks = nullptr;
};

// Allocates what the chain needs (no device work beyond stream-ordered
// allocation), issues it (no host round trip: it may be captured), and after
// the stream has been waited for turns the result into range CRS.
SlotBuild prepare_slots(dvg_context* ctx, const SlotPlan& plan, uint32_t n);
void launch_slots(dvg_context* ctx, SlotBuild& sb, const uint64_t* rowmap, const uint32_t* entries);
// Reads the counters back (one synchronisation), allocates the result and
// issues its conversion; null when the arena ran full (all buffers released,
// the context's estimate raised).
dvg_matrix* finish_slots(dvg_context* ctx, SlotBuild& sb);
void release_slots(dvg_context* ctx, SlotBuild& sb);

// prepare, launch and finish; null when the chain did not fit its arena.
dvg_matrix* slots_chain(dvg_context* ctx, const dvg_matrix* a, unsigned dlo, unsigned dup);

}  // namespace dvg
