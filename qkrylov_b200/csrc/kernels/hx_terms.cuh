// The compiled operator as the kernels walk it: sector tables and term groups.
#pragma once

#include "common.cuh"

namespace qkd {

struct DevPlan {
  int L;
  uint64_t lmask;
  const double* __restrict__ diag_re;
  const uint64_t* __restrict__ A;
  const uint32_t* __restrict__ B;
  const uint32_t* __restrict__ llist;
  const qk_term_t* __restrict__ terms;
  const qk_group_t* __restrict__ groups;
  const qk_tile_t* __restrict__ tiles;
  uint32_t nterms, ngroups, ntiles;
  int has_diag;
  uint64_t row_lo, row_hi;  // rows computed by k_hx: [row_lo, row_hi) (tiles never straddle a block)
};

// Sum of the valid terms of one group on state s: returns false when none is valid.
template <bool CC, class R>
__device__ __forceinline__ bool group_coef(const qk_term_t* t, uint32_t first, uint32_t count,
                                           uint64_t s, R& cr, R& ci) {
  bool any = false;
  cr = R(0); ci = R(0);
  for (uint32_t q = first; q < first + count; ++q) {
    const qk_term_t term = t[q];
    if ((s & term.cmask) != term.cval) continue;
    any = true;
    const bool neg = __popcll(s & term.smask) & 1;
    const R wr = R(term.wre);
    cr += neg ? -wr : wr;
    if (CC) { const R wi = R(term.wim); ci += neg ? -wi : wi; }
  }
  return any;
}

}  // namespace qkd
