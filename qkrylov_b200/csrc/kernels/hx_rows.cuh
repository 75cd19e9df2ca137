// Tables and device helpers shared by the row kernels: one CTA per sector
// block (hx_spin.cu) and one per group of blocks (hx_group.cu).
#pragma once

#include "reduce.cuh"
#include "../engine/sector.hpp"

namespace qkd {

constexpr int kSpinThreads = 512;
constexpr int kMaxBonds = 64;
constexpr int kMaxDiag = 128;

struct SpinBond {
  uint32_t lo_mask, hi_mask;  // flip split into the low / high part
  double c[4];                // coefficient for (bit_i, bit_j) = 00, 10, 01, 11
  uint8_t bi, bj;             // bit positions
  uint8_t kind;               // 0 low, 1 high, 2 crossing
  uint8_t valid_mask;         // which combos have a valid term
};

struct RowBlock {
  uint32_t base, size, lst, ebeg;  // block offset, rows, llist position, first entry in bent
  uint32_t nh, combo;              // high entries; sign pattern of the crossing Sz Sz terms
  double dh;                       // diagonal terms inside the high part
};

struct SpinPlan {
  int L, H;
  uint64_t dim;
  int nbonds, ndiag;
  // bond classes (host-side, for building the row tables)
  int nlow, nhigh, ncross, ndcross;
  uint32_t low_mask[kMaxBonds], high_mask[kMaxBonds], cross_lo[kMaxBonds], cross_hi[kMaxBonds];
  uint8_t low_i[kMaxBonds], high_i[kMaxBonds], cross_li[kMaxBonds];
  double low_c01[kMaxBonds], low_c10[kMaxBonds], high_c01[kMaxBonds], high_c10[kMaxBonds];
  double cross_c01[kMaxBonds], cross_c10[kMaxBonds];   // c01: low bit 0 / high bit 1
  uint32_t max_block;      // largest block size
  double coef[2 * kMaxBonds];
  int ncoef;
  uint32_t dcross_mask[kMaxDiag];
  double dcross_w[kMaxDiag];
  SpinBond bonds[kMaxBonds];
  uint32_t diag_smask[kMaxDiag];
  double diag_w[kMaxDiag];
  const uint32_t* A32;   // 2^H block offsets (global copy, staged to smem)
  const uint16_t* B16;   // 2^L in-class ranks (global copy, staged to smem)
  const uint16_t* lrow;  // llist as u16
  const qk_tile_t* tiles;
  uint32_t ntiles;
  size_t smem;
  // class and block tables of the row kernel
  const uint2* rrec;     // per llist position: first 4-entry group; groups per low class, 4 bits each
  const uint2* lgrp;     // 4 in-class ranks (u16) per group; padding entries name the zero slot
  const uint16_t* crk;   // [pos][cpad]: (low-side bit << 15) | partner in-class rank
  const double* dtab;    // [combo][pos]: low-part diagonal plus the crossing Sz Sz terms
  const RowBlock* brec;  // per sector block
  const uint2* bent;     // per block: high entries (base, coef) then crossing (base, coef | bit_h << 16)
  double lcls[4];        // coefficient of each low class
  int ncls, cpad, ncombo;
  uint32_t zero_slot, nllist;
  bool rows_ok;
  // two-part operators (any factorisable group, e.g. Hubbard and t-J hops)
  bool gen;
  uint32_t nblocks;       // block records (all 2^H, or only the non-empty ones)
  const uint32_t* crk32;  // [ncross][pos] (coalesced over rows): rank | lv0 << 24 | ls0 << 25 | lv1 << 26 | ls1 << 27
  const uint32_t* crm;    // [pos]: bit q set when a term of crossing group q has its low condition
  const double* diag_full;  // two-part operators: the diagonal per row, summed in term order
  const uint4* btiles;      // block apply: (block record, first row, rows) runs of <= 256 rows
  uint32_t nbtiles;
  const uint32_t* border;   // order in which the row kernel visits the block records (null: record order)
  // per-die work queues of the row kernel: the SMs of die 0 take the visiting
  // positions [0, qsplit), those of die 1 [qsplit, nblocks); a CTA whose
  // queue is empty takes from the other one
  const uint8_t* sm_die;    // die of each SM id (null: one die)
  uint32_t nsmid, qsplit;
};

// table limits of the row kernels
constexpr int kRowCoef = 32, kRowEnt = 48, kRowCross = 16, kRowCls = 4;

__device__ __forceinline__ void sld(const double2* s, uint32_t k, double& re, double& im) {
  const double2 v = s[k]; re = v.x; im = v.y;
}
__device__ __forceinline__ void sld(const float2* s, uint32_t k, float& re, float& im) {
  const float2 v = s[k]; re = v.x; im = v.y;
}
__device__ __forceinline__ void sld(const double* s, uint32_t k, double& re, double& im) { re = s[k]; im = 0; }
__device__ __forceinline__ void sld(const float* s, uint32_t k, float& re, float& im) { re = s[k]; im = 0; }
__device__ __forceinline__ void szero(double2& v) { v = make_double2(0.0, 0.0); }
__device__ __forceinline__ void szero(float2& v) { v = make_float2(0.f, 0.f); }
__device__ __forceinline__ void szero(double& v) { v = 0.0; }
__device__ __forceinline__ void szero(float& v) { v = 0.f; }

// L2 prefetch of elements [first, first + count) of a vector of `es`-byte
// elements, rounded inward to 16-byte boundaries (bulk prefetch operands
// must be 16-byte aligned and sized).
__device__ __forceinline__ void l2_prefetch(const void* base, uint32_t es, uint32_t first, uint32_t count) {
  const uintptr_t b = reinterpret_cast<uintptr_t>(base);
  const uintptr_t lo = (b + uintptr_t(first) * es + 15) & ~uintptr_t(15);
  const uintptr_t hi = (b + uintptr_t(first + count) * es) & ~uintptr_t(15);
  if (hi > lo)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(lo), "r"(uint32_t(hi - lo)) : "memory");
}

// Coefficient of a two-part crossing group in a row: up to two terms, each
// valid when its low condition (row table word `ent`) and its high
// condition (block entry flags `bf`) hold, signed by the parities of both
// parts.  Terms are added in order (first, then second).
template <class R>
__device__ __forceinline__ R cross_coef(uint32_t ent, uint32_t bf, const R* s_coef) {
  R c = R(0);
  if ((ent >> 24) & (bf >> 16) & 1u) {
    const R w = s_coef[bf & 0xFFu];
    c += (((ent >> 25) ^ (bf >> 17)) & 1u) ? -w : w;
  }
  if ((ent >> 26) & (bf >> 18) & 1u) {
    const R w = s_coef[(bf >> 8) & 0xFFu];
    c += (((ent >> 27) ^ (bf >> 19)) & 1u) ? -w : w;
  }
  return c;
}

__device__ __forceinline__ RowBlock load_block(const RowBlock* p) {
  const uint4* q = reinterpret_cast<const uint4*>(p);
  const uint4 a = __ldg(q), b = __ldg(q + 1);
  RowBlock r;
  r.base = a.x; r.size = a.y; r.lst = a.z; r.ebeg = a.w;
  r.nh = b.x; r.combo = b.y;
  r.dh = __hiloint2double(int(b.w), int(b.z));
  return r;
}

// Next visiting position for this CTA from the per-die queues (wq[0], wq[1];
// wq[2] counts CTAs that are done, the last one resets all three for the
// next launch).  Returns nblocks when both queues are empty.
__device__ __forceinline__ uint32_t wq_fetch(const SpinPlan& p, uint32_t* wq, int die) {
  for (int k = 0; k < 2; ++k) {
    const int q = die ^ k;
    const uint32_t beg = q ? p.qsplit : 0u, n = q ? p.nblocks - p.qsplit : p.qsplit;
    const uint32_t i = atomicAdd(wq + q, 1u);
    if (i < n) return beg + i;
  }
  return p.nblocks;
}

__device__ __forceinline__ int sm_die_of(const SpinPlan& p) {
  uint32_t s;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(s));
  return (p.sm_die && s < p.nsmid) ? int(__ldg(p.sm_die + s)) : 0;
}

__device__ __forceinline__ void wq_done(uint32_t* wq) {
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(wq + 2, 1u) == gridDim.x - 1) {
      atomicExch(wq, 0u);
      atomicExch(wq + 1, 0u);
      atomicExch(wq + 2, 0u);
    }
  }
}

}  // namespace qkd
