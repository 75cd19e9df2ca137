// H.x of small sectors from precomputed row lists.
//
// The row and pair kernels rebuild a row's targets from sector tables: a
// chain of dependent loads (plan, queue, block record, entries, class tables,
// targets) that a large sector hides behind its other rows and a small one
// cannot.  A sector whose target lists fit in the L2 caches reads them
// instead: slices of 32 consecutive rows, per slice one word per row for
// every term group that is valid in at least one of its rows (24 bits of
// target rank, 8 bits of coefficient class; class 0: no term, target = the
// row itself).  Slots are groups, not packed per row, so the rows of a warp
// follow the same bond and their targets are neighbouring addresses.  One
// launch.  k_hx_list: three dependent loads (slice start, words, targets);
// k_hx_list_small, for the smallest sectors: two (their slices have one width).
//
// Bound: latency up to ~2^17 rows, above that the L1/L2 traffic of words and
// targets (4 + sizeof(element) bytes per slot and row).  Four slots of a row
// share a 16-byte load (against one 4-byte word per slot: Heisenberg N=21
// c128 14.4 -> 12.9 us, t-J N=16 f64 16.4 -> 13.7 us) and a batch of eight
// loads the next batch's words before its own targets.  Against the row and
// pair kernels (us per apply, launches back to back on a caller's stream):
// Heisenberg N=16 c128 10.3 -> 4.1, N=20 18.6 -> 10.3, Hubbard chain 8 float64
// 14.4 -> 3.7, t-J N=17 float64 38 -> 25.  A call without a stream costs
// another 0.3 us (it waits for the default stream).
#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "hx_terms.cuh"
#include "reduce.cuh"
#include "../engine/sector.hpp"

namespace qkd {

constexpr int kListClasses = 64;   // coefficient values (class 0 is zero); 8 bits of the word
constexpr int kListThreads = 128;  // four slices per CTA: a 2^14-row sector still spreads over every SM
constexpr uint64_t kListMaxDim = 1ull << 24;  // 24-bit ranks
constexpr uint32_t kListSmall = 148 * 16;     // slices whose CTAs are all resident at once (k_hx_list_small);
// 148 * 60 instead: Heisenberg N=20 float64 8.2 -> 10.3 us
// Largest table.  The words have to stay in the L2 caches (126 MB, lines read
// by both dies held twice) from apply to apply.  Where the line lies depends on
// what runs instead, us per apply with lists / without: exchange tables
// Heisenberg N=22 c128 (41 MB) 25.6 / 24.0, float64 16.4 / 19.7, N=23 (85 MB)
// float64 31.5 / 25.9: 64 MB; spin-product 4x3 Hubbard float32 (93 MB) 34.7 /
// 23.3: 64 MB; two-part tables, whose rows decode slowest, t-J N=17 (72 MB)
// float64 24.6 / 35.4, c128 47.1 / 44.9: 96 MB.
constexpr size_t kListMaxBytes = size_t(96) << 20;

struct ListPlan {
  uint32_t dim, nslice;
  uint32_t row_lo, row_hi, slice0;  // rows written; first slice that holds one of them
  uint32_t width;         // groups of every slice where they are padded to one width, else 0
  const uint32_t* start;  // per slice: first 4-slot group (nslice + 1)
  const uint4* words;     // four slots of a row per 16 bytes: [slot / 4][lane]
  const double* diag;     // or null
  int ncoef;
  double coef[kListClasses];
};

struct ListHandle {
  ListPlan plan{};
  void* bufs[3] = {};
};

struct BlockListPlan {
  uint32_t dim;
  uint32_t tile;          // rows per tile
  const uint32_t* start;  // per row: first 4-word group (dim + 1)
  const uint4* words;
  const double* diag;     // or null
  uint32_t* wq;           // per-die tile queues (null: grid-stride)
  const uint8_t* sm_die;
  uint32_t nsmid;
  int n0, n1;             // SMs per die
  double coef[kListClasses];
};

struct BlockListHandle {
  BlockListPlan plan{};
  void* bufs[3] = {};
  mutable std::mutex mu;
  mutable double* part = nullptr;  // per-tile column dots, sized on first use
  mutable size_t part_cap = 0;
};

bool die_map(const uint8_t** dev_map, int* nsmid, int* n0, int* n1);

namespace {

constexpr unsigned long long kNoCoef = 0x7FF8DEADBEEF0001ull;  // empty slot of the coefficient table (a NaN)

__global__ void k_list_states(DevPlan p, uint64_t* __restrict__ st) {
  for (uint32_t ti = blockIdx.x; ti < p.ntiles; ti += gridDim.x) {
    const qk_tile_t t = p.tiles[ti];
    if (threadIdx.x < t.count)
      st[t.row0 + threadIdx.x] = (uint64_t(t.h) << p.L) | __ldg(p.llist + t.lstart + threadIdx.x);
  }
}

// Class of a coefficient value in an open-addressed table (at most
// kListClasses probes); 0 for zero, kListClasses when the table is full.
__device__ __forceinline__ uint32_t coef_class(double c, unsigned long long* table) {
  if (c == 0.0) return 0u;
  const unsigned long long bits = __double_as_longlong(c);
  uint32_t h = uint32_t((bits * 0x9E3779B97F4A7C15ull) >> 58);
  for (int k = 0; k < kListClasses; ++k, ++h) {
    h &= kListClasses - 1u;
    if (h == 0) continue;  // class 0 is the zero coefficient
    // a slot is written once: read first, or every target of every row queues
    // at the same few atomics (Heisenberg N=24: 25 of 30 ms of the plan)
    unsigned long long old = *reinterpret_cast<volatile unsigned long long*>(table + h);
    if (old == kNoCoef) old = atomicCAS(table + h, kNoCoef, bits);
    if (old == kNoCoef || old == bits) return h;
  }
  return uint32_t(kListClasses);
}

// FILL false: width of every slice (groups valid in at least one row) and
// the coefficient table; FILL true: the words.  One warp per slice.
template <bool FILL>
__global__ void __launch_bounds__(256) k_list_build(DevPlan p, uint32_t dim, const uint64_t* __restrict__ st,
                                                    uint32_t* __restrict__ start, uint32_t* __restrict__ words,
                                                    unsigned long long* table, int* overflow) {
  const uint32_t lane = threadIdx.x & 31, nslice = (dim + 31) / 32;
  for (uint32_t sl = blockIdx.x * 8 + (threadIdx.x >> 5); sl < nslice; sl += gridDim.x * 8) {
    const uint32_t row = sl * 32 + lane;
    const uint64_t s = st[min(row, dim - 1)];
    uint32_t n = 0;
    for (uint32_t g = p.has_diag ? 1u : 0u; g < p.ngroups; ++g) {
      const qk_group_t grp = p.groups[g];
      double c = 0.0, ci;
      uint32_t col = min(row, dim - 1), cls = 0;
      if (row < dim && group_coef<false, double>(p.terms, grp.first, grp.count, s, c, ci)) {
        const uint64_t t = s ^ grp.flip;
        const uint64_t a = __ldg(p.A + (t >> p.L));
        const uint32_t b = __ldg(p.B + (t & p.lmask));
        if (uint32_t(a >> 56) == (b >> 24)) {
          cls = coef_class(c, table);
          if (cls == uint32_t(kListClasses)) { *overflow = 1; cls = 0; }
          if (cls) col = uint32_t((a & qkb::kOffsetMask) + (b & qkb::kRankMask));
        }
      }
      if (!__ballot_sync(0xffffffffu, cls != 0)) continue;
      if (FILL) words[(size_t(start[sl]) + n / 4) * 128 + lane * 4 + n % 4] = col | (cls << 24);
      ++n;
    }
    if (!FILL && lane == 0) start[sl] = (n + 3) / 4;
    if (FILL)
      for (; n % 4; ++n) words[(size_t(start[sl]) + n / 4) * 128 + lane * 4 + n % 4] = 0u;
  }
}

// Packed lists for blocks of vectors: FILL false: targets of every row (and
// the coefficient table); FILL true: the words, at 4 * start[row], padded to
// whole groups of four with words of class 0.  One thread per row.
template <bool FILL>
__global__ void __launch_bounds__(256) k_packed_build(DevPlan p, uint32_t dim, const uint64_t* __restrict__ st,
                                                      uint32_t* __restrict__ start, uint32_t* __restrict__ words,
                                                      unsigned long long* table, int* overflow) {
  for (uint32_t row = blockIdx.x * 256 + threadIdx.x; row < dim; row += gridDim.x * 256) {
    const uint64_t s = st[row];
    uint32_t n = 0;
    uint32_t* out = FILL ? words + size_t(start[row]) * 4 : nullptr;
    for (uint32_t g = p.has_diag ? 1u : 0u; g < p.ngroups; ++g) {
      const qk_group_t grp = p.groups[g];
      double c, ci;
      if (!group_coef<false, double>(p.terms, grp.first, grp.count, s, c, ci)) continue;
      const uint64_t t = s ^ grp.flip;
      const uint64_t a = __ldg(p.A + (t >> p.L));
      const uint32_t b = __ldg(p.B + (t & p.lmask));
      if (uint32_t(a >> 56) != (b >> 24)) continue;
      const uint32_t cls = coef_class(c, table);
      if (cls == uint32_t(kListClasses)) { *overflow = 1; continue; }
      if (cls == 0) continue;
      if (FILL) out[n] = uint32_t((a & qkb::kOffsetMask) + (b & qkb::kRankMask)) | (cls << 24);
      ++n;
    }
    if (FILL) for (; n % 4; ++n) out[n] = 0u;
    else start[row] = (n + 3) / 4;
  }
}

// Y = H X (gacc: Y += diag(gacc) H X) for R = LPR * VPL row-interleaved
// vectors from the packed lists: LPR lanes share a row, the words of a row are
// one broadcast load per four targets, and the four target rows are in flight
// together with nothing to decode between them.  The block kernels on the
// sector tables chain about eleven dependent loads per row (record, groups,
// masks, crossing words, then targets a few at a time) at 16 to 32 warps per
// SM and are bound by that latency; the words are 4 bytes per target against
// 128 to 1024 bytes of its row.  Registers for five CTAs per SM at up to 16
// bytes per lane, three at 32: eight targets in flight at fewer CTAs were
// 10-20% slower (t-J N=18, 64 float32 vectors: 757 us with 3 CTAs, 721 with 4,
// four targets and 5 CTAs 624; J1-J2 N=24, 32 float64 vectors: 1774 us with 2
// CTAs, four targets and 3 CTAs 1514; kernel alone, fastest of several runs).
// Whole applies against k_hx_rows_block: those two 1120 -> 680-705 and 2180 ->
// 1570-1655 us; t-J N=20, 64 vectors float32 4.97 -> 3.41, float64 9.24 -> 6.60
// ms; t-J N=13, 64 float32 56 -> 18 us.  Tiles of
// kBlockTile rows from a queue per die; column dots per tile (sum_items).
// Sectors with fewer than kBlockTiles tiles (two per resident CTA) take tiles
// of 64 or 32 rows, so that a warp's rows, one after the other, are not the
// length of the kernel: J1-J2 N=16, 64 float32 vectors 20.5 -> 12.5 us, t-J
// N=14, 64 float64 101 -> 82 us; a limit of 148 * 20 or 148 * 40 costs J1-J2
// N=22, 32 float64 0 and 4%.
constexpr uint32_t kBlockTile = 128;
constexpr uint32_t kBlockTileMin = 32, kBlockTiles = 148 * 10;
template <class E, int VPL> struct alignas(sizeof(E) * VPL >= 16 ? 16 : sizeof(E) * VPL) ListPack { E v[VPL]; };
template <int DT> __device__ __forceinline__ void unpk(const typename VT<DT>::E& e, typename VT<DT>::R& re, typename VT<DT>::R& im) {
  if constexpr (VT<DT>::cplx) { re = e.x; im = e.y; } else { re = e; im = typename VT<DT>::R(0); }
}

template <int DT, int LPR, int VPL, int MINC>
__global__ void __launch_bounds__(256, MINC)
k_hx_block_list(const __grid_constant__ BlockListPlan p, const void* __restrict__ X, void* __restrict__ Y,
                const double* __restrict__ gacc, uint32_t ntiles, uint32_t qsplit, double* part) {
  using T = VT<DT>;
  using R = typename T::R;
  using E = typename T::E;
  using Pack = ListPack<E, VPL>;
  constexpr int RV = LPR * VPL, RPW = 32 / LPR;
  __shared__ R s_coef[kListClasses];
  __shared__ double red[(256 / 32) * RV * 2];
  __shared__ uint32_t s_tile[2];
  if (threadIdx.x < kListClasses) s_coef[threadIdx.x] = R(p.coef[threadIdx.x]);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane / LPR, l = lane % LPR;
  const E* __restrict__ Xe = reinterpret_cast<const E*>(X) + l * VPL;
  E* __restrict__ Ye = reinterpret_cast<E*>(Y) + l * VPL;
  int die = 0;
  if (p.wq) {
    uint32_t sid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(sid));
    die = (p.sm_die && sid < p.nsmid) ? int(__ldg(p.sm_die + sid)) : 0;
  }
  auto fetch = [&](uint32_t prev) -> uint32_t {
    if (!p.wq) return prev + gridDim.x;
    for (int k = 0; k < 2; ++k) {
      const int q = die ^ k;
      const uint32_t beg = q ? qsplit : 0u, n = q ? ntiles - qsplit : qsplit;
      const uint32_t i = atomicAdd(p.wq + q, 1u);
      if (i < n) return beg + i;
    }
    return ntiles;
  };
  if (threadIdx.x == 0) s_tile[0] = p.wq ? fetch(0) : blockIdx.x;
  __syncthreads();
  uint32_t tile = s_tile[0];
  R gcol[VPL];
  #pragma unroll
  for (int v = 0; v < VPL; ++v) gcol[v] = gacc ? R(gacc[l * VPL + v]) : R(1);
  for (uint32_t it = 1; tile < ntiles; ++it) {
    if (threadIdx.x == 0) s_tile[it & 1] = fetch(tile);
    const uint32_t r1 = min(p.dim, (tile + 1) * p.tile);
    double dr[VPL], di[VPL];
    #pragma unroll
    for (int v = 0; v < VPL; ++v) { dr[v] = 0.0; di[v] = 0.0; }
    uint32_t r = tile * p.tile + warp * RPW + sub;
    uint32_t b0 = 0, b1 = 0;
    if (r < r1) { b0 = __ldg(p.start + r); b1 = __ldg(p.start + r + 1); }
    for (; r < r1; r += (256 / 32) * RPW) {
      const uint4* __restrict__ w = p.words + b0;
      const uint32_t n = b1 - b0;
      uint4 q = n ? __ldg(w) : make_uint4(0u, 0u, 0u, 0u);
      const Pack own = *reinterpret_cast<const Pack*>(Xe + size_t(r) * RV);
      const R d = p.diag ? R(__ldg(p.diag + r)) : R(0);
      const uint32_t rn = r + (256 / 32) * RPW;
      if (rn < r1) { b0 = __ldg(p.start + rn); b1 = __ldg(p.start + rn + 1); }
      R ar[VPL], ai[VPL];
      #pragma unroll
      for (int v = 0; v < VPL; ++v) { ar[v] = R(0); ai[v] = R(0); }
      for (uint32_t j = 0; j < n; ++j) {
        const uint32_t e[4] = {q.x, q.y, q.z, q.w};
        Pack t[4];
        #pragma unroll
        for (int u = 0; u < 4; ++u)  // padding (class 0) reads row 0, always there, and is not added
          t[u] = *reinterpret_cast<const Pack*>(Xe + size_t(e[u] & 0xFFFFFFu) * RV);
        if (j + 1 < n) q = __ldg(w + j + 1);
        #pragma unroll
        for (int u = 0; u < 4; ++u)
          if (e[u] >> 24) {
            const R c = s_coef[e[u] >> 24];
            #pragma unroll
            for (int v = 0; v < VPL; ++v) {
              R vr, vi;
              unpk<DT>(t[u].v[v], vr, vi);
              ar[v] += c * vr;
              if (T::cplx) ai[v] += c * vi;
            }
          }
      }
      // the diagonal last: the hops are rounded against their own sum; none is
      // not a zero one, which would turn an infinite x into a NaN
      if (p.diag) {
        #pragma unroll
        for (int v = 0; v < VPL; ++v) {
          R xr, xi;
          unpk<DT>(own.v[v], xr, xi);
          ar[v] += d * xr;
          if (T::cplx) ai[v] += d * xi;
        }
      }
      Pack* yp = reinterpret_cast<Pack*>(Ye + size_t(r) * RV);
      if (gacc) {
        const Pack y0 = *yp;
        #pragma unroll
        for (int v = 0; v < VPL; ++v) {
          R y0r, y0i;
          unpk<DT>(y0.v[v], y0r, y0i);
          ar[v] = y0r + gcol[v] * ar[v];
          if (T::cplx) ai[v] = y0i + gcol[v] * ai[v];
        }
      }
      Pack yv;
      #pragma unroll
      for (int v = 0; v < VPL; ++v) {
        if constexpr (T::cplx) { yv.v[v].x = ar[v]; yv.v[v].y = ai[v]; } else yv.v[v] = ar[v];
        R xr, xi;
        unpk<DT>(own.v[v], xr, xi);
        if (T::cplx) {
          dr[v] += double(xr) * double(ar[v]) + double(xi) * double(ai[v]);
          di[v] += double(xr) * double(ai[v]) - double(xi) * double(ar[v]);
        } else {
          dr[v] += double(xr) * double(ar[v]);
        }
      }
      *yp = yv;
    }
    if (part) {
      #pragma unroll
      for (int v = 0; v < VPL; ++v)
        #pragma unroll
        for (int o = LPR; o < 32; o <<= 1) {
          dr[v] += __shfl_xor_sync(0xffffffffu, dr[v], o);
          if (T::cplx) di[v] += __shfl_xor_sync(0xffffffffu, di[v], o);
        }
      if (lane < LPR) {
        #pragma unroll
        for (int v = 0; v < VPL; ++v) {
          red[(warp * RV + l * VPL + v) * 2] = dr[v];
          red[(warp * RV + l * VPL + v) * 2 + 1] = T::cplx ? di[v] : 0.0;
        }
      }
    }
    __syncthreads();
    if (part) {
      for (int c = threadIdx.x; c < RV; c += 256) {
        double sr = 0.0, si = 0.0;
        for (int k = 0; k < 256 / 32; ++k) { sr += red[(k * RV + c) * 2]; si += red[(k * RV + c) * 2 + 1]; }
        double* o = part + (size_t(c) * ntiles + tile) * 2;
        o[0] = sr;
        o[1] = si;
      }
      __syncthreads();
    }
    tile = s_tile[it & 1];
  }
  if (p.wq && threadIdx.x == 0) {  // the last CTA resets the queues for the next launch
    __threadfence();
    if (atomicAdd(p.wq + 2, 1u) == gridDim.x - 1) {
      atomicExch(p.wq, 0u);
      atomicExch(p.wq + 1, 0u);
      atomicExch(p.wq + 2, 0u);
    }
  }
}

// out[2c..2c+1] = sum over the n items of column c, in a fixed order, one CTA
// per column (the last CTA of the block kernels summed all columns by itself:
// about 100 us of the 2175 us of J1-J2 N=24, 32 columns).
__global__ void __launch_bounds__(256) k_sum_items(const double* __restrict__ part, uint32_t n, double* __restrict__ out) {
  const double2* __restrict__ p = reinterpret_cast<const double2*>(part) + size_t(blockIdx.x) * n;
  double re = 0.0, im = 0.0;
  for (uint32_t i = threadIdx.x; i < n; i += 256) {
    const double2 v = __ldg(p + i);
    re += v.x;
    im += v.y;
  }
  __shared__ double sbuf[2 * (256 / 32)];
  block_sum2(re, im, sbuf);
  if (threadIdx.x == 0) { out[2 * blockIdx.x] = re; out[2 * blockIdx.x + 1] = im; }
}

// The smallest sectors: a CTA of four warps per slice, each warp every fourth
// group of slots, partial sums added in pairs through shared memory.  The
// slices have one width, so the words are the first loads of the kernel and
// their targets the second: nothing else is on the path (Heisenberg N=16
// complex128, launches back to back: 5.4 us with k_hx_list, 4.3 us here).
template <int DT, bool DOT>
__global__ void __launch_bounds__(kListThreads) k_hx_list_small(const __grid_constant__ ListPlan p,
                                                                const void* __restrict__ x, void* __restrict__ y,
                                                                double* partials, unsigned* ticket, double* dot_out) {
  using T = VT<DT>;
  using R = typename T::R;
  constexpr int NW = kListThreads / 32;
  __shared__ R s_coef[kListClasses];
  __shared__ R s_sum[2][NW][32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double dr = 0.0, di = 0.0;
  bool first = true;
  for (uint32_t sl = p.slice0 + blockIdx.x; sl < p.nslice; sl += gridDim.x) {
    const uint4* __restrict__ w = p.words + size_t(sl) * p.width * 32 + lane;
    uint4 q = warp < p.width ? __ldg(w + warp * 32) : make_uint4(0u, 0u, 0u, 0u);
    const uint32_t row = sl * 32 + lane;
    const bool in = row >= p.row_lo && row < p.row_hi;
    R xr = R(0), xi = R(0), d = R(0);
    if (warp == 0 && in) {
      T::ld(x, row, xr, xi);
      if (p.diag) d = R(__ldg(p.diag + row));
    }
    if (first && threadIdx.x < kListClasses) s_coef[threadIdx.x] = R(p.coef[threadIdx.x]);
    __syncthreads();  // the coefficients; the previous slice's sums have been read
    first = false;
    R ar = R(0), ai = R(0);
    for (uint32_t j = warp; j < p.width; j += NW) {
      const uint32_t e[4] = {q.x, q.y, q.z, q.w};
      if (j + NW < p.width) q = __ldg(w + (j + NW) * 32);
      R vr[4], vi[4];
      #pragma unroll
      for (int u = 0; u < 4; ++u) {
        vr[u] = R(0);
        vi[u] = R(0);
        if (e[u] >> 24) T::ld(x, e[u] & 0xFFFFFFu, vr[u], vi[u]);
      }
      #pragma unroll
      for (int u = 0; u < 4; ++u)
        if (e[u] >> 24) {
          const R c = s_coef[e[u] >> 24];
          ar += c * vr[u];
          if (T::cplx) ai += c * vi[u];
        }
    }
    s_sum[0][warp][lane] = ar;
    if (T::cplx) s_sum[1][warp][lane] = ai;
    __syncthreads();
    if (warp == 0) {
      static_assert(NW == 4, "four partial sums");
      ar = (s_sum[0][0][lane] + s_sum[0][1][lane]) + (s_sum[0][2][lane] + s_sum[0][3][lane]);
      if (T::cplx) ai = (s_sum[1][0][lane] + s_sum[1][1][lane]) + (s_sum[1][2][lane] + s_sum[1][3][lane]);
      if (p.diag) {
        ar += d * xr;
        if (T::cplx) ai += d * xi;
      }
      if (in) {
        T::st(y, row, ar, ai);
        if (DOT) {
          dr += double(xr) * double(ar) + double(xi) * double(ai);
          di += double(xr) * double(ai) - double(xi) * double(ar);
        }
      }
    }
  }
  if (DOT) {
    __shared__ double sbuf[2 * NW];
    block_sum2(dr, di, sbuf);
    if (threadIdx.x == 0) { partials[2 * blockIdx.x] = dr; partials[2 * blockIdx.x + 1] = di; }
    grid_finish(partials, ticket, 1, dot_out);
  }
}

template <int DT, bool DOT>
__global__ void __launch_bounds__(kListThreads) k_hx_list(const __grid_constant__ ListPlan p,
                                                          const void* __restrict__ x, void* __restrict__ y,
                                                          double* partials, unsigned* ticket, double* dot_out) {
  using T = VT<DT>;
  using R = typename T::R;
  __shared__ R s_coef[kListClasses];
  const uint32_t lane = threadIdx.x & 31, nw = gridDim.x * (kListThreads / 32);
  uint32_t sl = p.slice0 + blockIdx.x * (kListThreads / 32) + (threadIdx.x >> 5);
  uint32_t b0 = 0, b1 = 0;
  if (sl < p.nslice) { b0 = __ldg(p.start + sl); b1 = __ldg(p.start + sl + 1); }
  if (threadIdx.x < kListClasses) s_coef[threadIdx.x] = R(p.coef[threadIdx.x]);
  __syncthreads();
  double dr = 0.0, di = 0.0;
  while (sl < p.nslice) {
    const uint32_t row = sl * 32 + lane;
    const bool in = row >= p.row_lo && row < p.row_hi;
    R xr = R(0), xi = R(0), d = R(0);
    if (in) {
      T::ld(x, row, xr, xi);
      if (p.diag) d = R(__ldg(p.diag + row));
    }
    R ar = R(0), ai = R(0);
    const uint4* __restrict__ w = p.words + size_t(b0) * 32 + lane;
    const uint32_t n = b1 - b0;
    uint4 q[2];
    #pragma unroll
    for (uint32_t u = 0; u < 2; ++u) q[u] = u < n ? __ldg(w + u * 32) : make_uint4(0u, 0u, 0u, 0u);
    for (uint32_t j = 0; j < n; j += 2) {
      const uint32_t e[8] = {q[0].x, q[0].y, q[0].z, q[0].w, q[1].x, q[1].y, q[1].z, q[1].w};
      #pragma unroll
      for (uint32_t u = 0; u < 2; ++u)  // the next words while this batch's targets arrive
        q[u] = j + 2 + u < n ? __ldg(w + (j + 2 + u) * 32) : make_uint4(0u, 0u, 0u, 0u);
      R vr[8], vi[8];
      #pragma unroll
      for (int u = 0; u < 8; ++u) {
        vr[u] = R(0);
        vi[u] = R(0);
        if (e[u] >> 24) T::ld(x, e[u] & 0xFFFFFFu, vr[u], vi[u]);
      }
      #pragma unroll
      for (int u = 0; u < 8; ++u)
        if (e[u] >> 24) {
          const R c = s_coef[e[u] >> 24];
          ar += c * vr[u];
          if (T::cplx) ai += c * vi[u];
        }
    }
    if (p.diag) {
      ar += d * xr;
      if (T::cplx) ai += d * xi;
    }
    if (in) T::st(y, row, ar, ai);
    if (DOT) {
      dr += double(xr) * double(ar) + double(xi) * double(ai);
      di += double(xr) * double(ai) - double(xi) * double(ar);
    }
    sl += nw;
    if (sl < p.nslice) { b0 = __ldg(p.start + sl); b1 = __ldg(p.start + sl + 1); }
  }
  if (DOT) {
    __shared__ double sbuf[2 * (kListThreads / 32)];
    block_sum2(dr, di, sbuf);
    if (threadIdx.x == 0) { partials[2 * blockIdx.x] = dr; partials[2 * blockIdx.x + 1] = di; }
    grid_finish(partials, ticket, 1, dot_out);
  }
}

}  // namespace

void list_plan_destroy(ListHandle* h) {
  if (!h) return;
  for (void* b : h->bufs) cudaFree(b);
  delete h;
}

// Row lists of a real operator with its real diagonal (diag: dim device
// doubles, or null for none); two_part: the operator would run on the two-part
// tables or the generic kernel.  Null when they do not fit the limit, the
// ranks 24 bits or the coefficients the class table.
ListHandle* list_plan_create(const DevPlan& p, uint64_t dim, const double* diag, bool two_part, size_t* dev_bytes) {
  const size_t max_bytes = two_part ? kListMaxBytes : kListMaxBytes * 2 / 3;
  const uint32_t nslice = uint32_t((dim + 31) / 32);
  // at least one slot per slice: cheap refusal of sectors that cannot fit
  if (dim == 0 || dim > kListMaxDim || p.ngroups == 0 || size_t(nslice) * 512 > max_bytes) return nullptr;
  uint64_t* st = nullptr;
  unsigned long long* table = nullptr;  // kListClasses values, then the overflow flag
  uint32_t *start = nullptr, *words = nullptr;
  std::vector<uint32_t> hs(size_t(nslice) + 1);
  std::vector<unsigned long long> ht(kListClasses + 1, kNoCoef);
  ht[kListClasses] = 0;
  const unsigned g = std::max(1u, std::min((nslice + 7) / 8, 148u * 8u));
  bool ok = cudaMalloc(&st, dim * 8) == cudaSuccess && cudaMalloc(&table, ht.size() * 8) == cudaSuccess &&
            cudaMalloc(&start, hs.size() * 4) == cudaSuccess &&
            cudaMemcpy(table, ht.data(), ht.size() * 8, cudaMemcpyHostToDevice) == cudaSuccess;
  if (ok) {
    k_list_states<<<std::max(1u, std::min(p.ntiles, 148u * 8u)), 256>>>(p, st);
    k_list_build<false><<<g, 256>>>(p, uint32_t(dim), st, start, nullptr, table,
                                    reinterpret_cast<int*>(table + kListClasses));
    ok = cudaGetLastError() == cudaSuccess &&
         cudaMemcpy(hs.data(), start, size_t(nslice) * 4, cudaMemcpyDeviceToHost) == cudaSuccess &&
         cudaMemcpy(ht.data(), table, ht.size() * 8, cudaMemcpyDeviceToHost) == cudaSuccess && ht[kListClasses] == 0;
  }
  size_t total = 0;
  for (uint32_t i = 0; ok && i < nslice; ++i) {
    const uint32_t n = hs[i];
    hs[i] = uint32_t(total);
    total += n;
    ok = total * 512 <= max_bytes;
  }
  hs[nslice] = uint32_t(total);
  // small sectors: every slice padded to the widest one
  uint32_t width = 0;
  for (uint32_t i = 0; ok && i < nslice; ++i) width = std::max(width, hs[i + 1] - hs[i]);
  if (nslice > kListSmall || width == 0) width = 0;
  if (width) {
    for (uint32_t i = 0; i <= nslice; ++i) hs[i] = i * width;
    total = size_t(nslice) * width;
  }
  ok = ok && cudaMalloc(&words, std::max<size_t>(total, 1) * 512) == cudaSuccess &&
       cudaMemcpy(start, hs.data(), hs.size() * 4, cudaMemcpyHostToDevice) == cudaSuccess;
  if (ok && width) ok = cudaMemset(words, 0, total * 512) == cudaSuccess;
  if (ok) {
    k_list_build<true><<<g, 256>>>(p, uint32_t(dim), st, start, words, table,
                                   reinterpret_cast<int*>(table + kListClasses));
    ok = cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess;
  }
  cudaFree(st);
  cudaFree(table);
  if (!ok) {
    (void)cudaGetLastError();
    cudaFree(start);
    cudaFree(words);
    return nullptr;
  }
  auto* h = new ListHandle;
  h->bufs[0] = start;
  h->bufs[1] = words;
  *dev_bytes += hs.size() * 4 + std::max<size_t>(total, 1) * 512;
  ListPlan& l = h->plan;
  l.dim = uint32_t(dim);
  l.nslice = nslice;
  l.start = start;
  l.width = width;
  l.words = reinterpret_cast<const uint4*>(words);
  l.diag = diag;
  l.ncoef = kListClasses;
  for (int k = 0; k < kListClasses; ++k) {
    l.coef[k] = 0.0;
    if (k && ht[k] != kNoCoef) std::memcpy(&l.coef[k], &ht[k], 8);
  }
  return h;
}

// Rows [row_lo, row_hi) of y = H x, row_lo < row_hi <= dim; with dot_out
// (whole vectors only) also <x, y>.
int list_apply(const ListHandle* h, qk_dtype t, const void* x, void* y, cudaStream_t s, qk_workspace* w,
               double* dot_out, uint64_t row_lo, uint64_t row_hi) {
  ListPlan p = h->plan;
  p.row_lo = uint32_t(row_lo);
  p.row_hi = uint32_t(row_hi);
  p.slice0 = p.row_lo / 32;
  p.nslice = (p.row_hi + 31) / 32;
  const unsigned n = p.nslice - p.slice0, g = p.width ? n : (n + kListThreads / 32 - 1) / (kListThreads / 32);
  QKD_DISPATCH(t, {
    auto kd = p.width ? k_hx_list_small<DT, true> : k_hx_list<DT, true>;
    auto kn = p.width ? k_hx_list_small<DT, false> : k_hx_list<DT, false>;
    if (dot_out) kd<<<std::min<unsigned>(g, kMaxG), kListThreads, 0, s>>>(p, x, y, w->partials, w->ticket, dot_out);
    else kn<<<g, kListThreads, 0, s>>>(p, x, y, nullptr, nullptr, nullptr);
  });
  QKD_LAUNCH_CHECK();
  return QKD_OK;
}


int sum_items(const double* part, uint32_t n, int columns, double* out, cudaStream_t s) {
  k_sum_items<<<columns, 256, 0, s>>>(part, n, out);
  QKD_LAUNCH_CHECK();
  return QKD_OK;
}

void block_list_destroy(BlockListHandle* h) {
  if (!h) return;
  for (void* b : h->bufs) cudaFree(b);
  cudaFree(h->part);
  delete h;
}

bool block_list_possible(const DevPlan& p, uint64_t dim) { return dim > 0 && dim <= kListMaxDim && p.ngroups > 0; }

// Packed lists of a real operator (diag as in list_plan_create) for which
// block_list_possible; null when they exceed max_bytes, the coefficients the
// class table, or the memory is not there.  *list_bytes: the size of the words
// once they are counted, ~0 when the class table is too small for them.
BlockListHandle* block_list_create(const DevPlan& p, uint64_t dim, const double* diag, size_t max_bytes,
                                   size_t* list_bytes, size_t* dev_bytes) {
  uint64_t* st = nullptr;
  unsigned long long* table = nullptr;
  uint32_t *start = nullptr, *words = nullptr, *wq = nullptr;
  std::vector<uint32_t> hs(dim + 1);
  std::vector<unsigned long long> ht(kListClasses + 1, kNoCoef);
  ht[kListClasses] = 0;
  const unsigned g = unsigned(std::max<uint64_t>(1, std::min<uint64_t>((dim + 255) / 256, 148u * 8u)));
  bool ok = cudaMalloc(&st, dim * 8) == cudaSuccess && cudaMalloc(&table, ht.size() * 8) == cudaSuccess &&
            cudaMalloc(&start, hs.size() * 4) == cudaSuccess &&
            cudaMemcpy(table, ht.data(), ht.size() * 8, cudaMemcpyHostToDevice) == cudaSuccess;
  if (ok) {
    k_list_states<<<std::max(1u, std::min(p.ntiles, 148u * 8u)), 256>>>(p, st);
    k_packed_build<false><<<g, 256>>>(p, uint32_t(dim), st, start, nullptr, table,
                                      reinterpret_cast<int*>(table + kListClasses));
    ok = cudaGetLastError() == cudaSuccess &&
         cudaMemcpy(hs.data(), start, dim * 4, cudaMemcpyDeviceToHost) == cudaSuccess &&
         cudaMemcpy(ht.data(), table, ht.size() * 8, cudaMemcpyDeviceToHost) == cudaSuccess;
    if (ok && ht[kListClasses] != 0) {
      *list_bytes = ~size_t(0);
      ok = false;
    }
  }
  uint64_t total = 0;
  for (uint64_t i = 0; ok && i < dim; ++i) {
    const uint32_t n = hs[i];
    hs[i] = uint32_t(total);
    total += n;
  }
  hs[dim] = uint32_t(total);
  if (ok) *list_bytes = size_t(total) * 16;
  ok = ok && total < (1ull << 32) && total * 16 <= max_bytes &&
       cudaMalloc(&words, std::max<uint64_t>(total, 1) * 16) == cudaSuccess &&
       cudaMemcpy(start, hs.data(), hs.size() * 4, cudaMemcpyHostToDevice) == cudaSuccess;
  if (ok) {
    k_packed_build<true><<<g, 256>>>(p, uint32_t(dim), st, start, words, table,
                                     reinterpret_cast<int*>(table + kListClasses));
    ok = cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess;
  }
  cudaFree(st);
  cudaFree(table);
  auto* h = ok ? new BlockListHandle : nullptr;
  if (!h) {
    (void)cudaGetLastError();
    cudaFree(start);
    cudaFree(words);
    return nullptr;
  }
  const uint8_t* map = nullptr;
  int nsmid = 0, n0 = 0, n1 = 0;
  // the first apply may run on a stream that does not wait for the memset
  if (die_map(&map, &nsmid, &n0, &n1) && cudaMalloc(&wq, 16) == cudaSuccess && cudaMemset(wq, 0, 16) == cudaSuccess &&
      cudaStreamSynchronize(nullptr) == cudaSuccess) {
    h->plan.wq = wq;
    h->plan.sm_die = map;
    h->plan.nsmid = uint32_t(nsmid);
    h->plan.n0 = n0;
    h->plan.n1 = n1;
  } else {
    (void)cudaGetLastError();
  }
  h->bufs[0] = start;
  h->bufs[1] = words;
  h->bufs[2] = wq;
  *dev_bytes += hs.size() * 4 + std::max<uint64_t>(total, 1) * 16;
  h->plan.dim = uint32_t(dim);
  h->plan.tile = kBlockTile;
  while (h->plan.tile > kBlockTileMin && dim / h->plan.tile < kBlockTiles) h->plan.tile /= 2;
  h->plan.start = start;
  h->plan.words = reinterpret_cast<const uint4*>(words);
  h->plan.diag = diag;
  for (int k = 0; k < kListClasses; ++k) {
    h->plan.coef[k] = 0.0;
    if (k && ht[k] != kNoCoef) std::memcpy(&h->plan.coef[k], &ht[k], 8);
  }
  return h;
}

// lanes per row 32, 16 or 8 (R / lanes <= 8, 4 to 64 bytes per lane);
// QKD_EINVAL for other shapes, or when the dots' partials have no memory
// (during a capture, before a first use outside it).
int block_list_apply(const BlockListHandle* h, qk_dtype t, int R, int lpr, bool queues, const void* X, void* Y,
                     double* dots, cudaStream_t s, const double* gacc) {
  BlockListPlan p = h->plan;
  if (!queues) p.wq = nullptr;
  const uint32_t ntiles = (p.dim + p.tile - 1) / p.tile;
  const uint32_t qsplit = uint32_t(uint64_t(ntiles) * p.n0 / std::max(1, p.n0 + p.n1));
  double* part = nullptr;
  if (dots) {
    std::lock_guard<std::mutex> lk(h->mu);
    const size_t need = size_t(ntiles) * R * 2;
    if (h->part_cap < need) {
      cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
      if (cudaStreamIsCapturing(s, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) return QKD_EINVAL;
      cudaFree(h->part);
      h->part = nullptr;
      h->part_cap = 0;
      if (cudaMalloc(&h->part, need * 8) != cudaSuccess) {
        (void)cudaGetLastError();
        return QKD_EINVAL;
      }
      h->part_cap = need;
    }
    part = h->part;
  }
#define QKD_BL(RR, L, V)                                                                                     \
  if (R == RR && lpr == L) {                                                                                 \
    QKD_DISPATCH(t, {                                                                                        \
      constexpr int B = V * int(sizeof(VT<DT>::E));                                                          \
      if constexpr (B <= 32) {                                                                               \
        auto k = k_hx_block_list<DT, L, V, B <= 16 ? 5 : 3>;                                                 \
        k<<<resident_grid(k, 256, 0, ntiles), 256, 0, s>>>(p, X, Y, gacc, ntiles, qsplit, part);             \
      } else {                                                                                               \
        return QKD_EINVAL;                                                                                   \
      }                                                                                                      \
    });                                                                                                      \
    QKD_LAUNCH_CHECK();                                                                                      \
    return dots ? sum_items(part, ntiles, R, dots, s) : QKD_OK;                                              \
  }
  QKD_BL(32, 32, 1) QKD_BL(32, 16, 2) QKD_BL(32, 8, 4)
  QKD_BL(64, 32, 2) QKD_BL(64, 16, 4) QKD_BL(64, 8, 8)
  QKD_BL(128, 32, 4) QKD_BL(128, 16, 8)
#undef QKD_BL
  return QKD_EINVAL;
}

}  // namespace qkd
