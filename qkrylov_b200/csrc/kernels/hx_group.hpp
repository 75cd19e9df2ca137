// Host interface of the grouped row kernel (hx_group.cu).
#pragma once

#include <vector>

#include "common.cuh"

namespace qkd {

constexpr uint32_t kGroupMax = 4;

// Up to kGroupMax sector blocks with the same low class, combo and crossing flags.
struct alignas(16) GroupRec {
  uint32_t size, lst, tile0;  // rows per block, llist position and first warp tile of the class
  uint16_t combo, count;      // sign pattern of the crossing diagonal terms; blocks
  uint32_t base[kGroupMax], ebeg[kGroupMax];  // block offsets, first entries in bent
  uint32_t nh[kGroupMax];                     // high entries
  double dh[kGroupMax];                       // diagonal terms inside the high part
};

struct GroupPlan {
  const GroupRec* rec;
  uint32_t nitems, qsplit;
  const uint2* bent;   // per block: high entries (base, coef) then crossing (base, flags)
  // warp tiles (32 consecutive positions of a low class): first 4-slot group
  // and groups per coefficient class (8 bits each); four slots of a row per
  // uint2 ([group][lane], in-class ranks; zero_slot .. zero_slot + 7: no target)
  const uint2* wrec;
  const uint2* wgrp;
  const uint16_t* crk;
  const double* dtab;
  const uint32_t* crk32;
  const uint32_t* crm;
  const double* diag_full;
  const uint8_t* sm_die;
  uint32_t nsmid, nllist, zero_slot, prefetch;
  int ncross, ncls, cpad;
  uint64_t dim;
  double coef[32], lcls[4];
  int uniform_high;   // every high entry has the coefficient high_coef
  double high_coef;
};

struct GroupBlock { uint32_t base, size, lst, tile0, ebeg, nh, combo; double dh; };

struct GroupHandle;
GroupHandle* group_plan_create(const GroupPlan& tables, const std::vector<GroupBlock>& blocks,
                               const std::vector<uint2>& bent, int n0, int n1, size_t* dev_bytes);
void group_plan_destroy(GroupHandle* h);
int group_apply(const GroupHandle* h, bool gen, qk_dtype t, const void* x, void* y, cudaStream_t s, qk_workspace* w,
                double* dot_out, uint32_t* wq, const double* diag_full, uint32_t row_lo, uint32_t row_hi);

}  // namespace qkd
