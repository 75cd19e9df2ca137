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
// launch, three dependent loads: slice start, words, targets.
//
// Bound: latency up to ~2^17 rows, above that the L1/L2 traffic of words and
// targets (4 + sizeof(element) bytes per slot and row).  Four slots of a row
// share a 16-byte load (against one 4-byte word per slot: Heisenberg N=21
// c128 14.4 -> 12.9 us, t-J N=16 f64 16.4 -> 13.7 us) and a batch of eight
// loads the next batch's words before its own targets.  Against the row and
// pair kernels (us per apply, launches back to back): Heisenberg N=16 c128
// 10.3 -> 6.2, N=20 18.6 -> 10.3, t-J N=14 f64 16.3 -> 6.2, Hubbard chain 10
// c128 18.5 -> 6.2, transverse Ising N=18 f64 16.4 -> 10.3.
#include <algorithm>
#include <cstring>
#include <vector>

#include "hx_terms.cuh"
#include "reduce.cuh"
#include "../engine/sector.hpp"

namespace qkd {

constexpr int kListClasses = 64;   // coefficient values (class 0 is zero); 8 bits of the word
constexpr int kListThreads = 128;  // four slices per CTA: a 2^14-row sector still spreads over every SM
constexpr uint64_t kListMaxDim = 1ull << 24;  // 24-bit ranks
// Largest table: about one die's L2 (63 MB), so that with the vectors it stays
// in the caches from apply to apply; beyond it the words stream from DRAM.
// Measured against the row / pair kernels (us per apply): Heisenberg N=22 c128
// 34.5 -> 23.3 (41 MB), N=24 87 -> 100 (165 MB); transverse Ising N=20 c64
// 31.6 -> 34.8 (80 MB); 4x3 Hubbard f32 30.7 -> 34.7 (93 MB).
constexpr size_t kListMaxBytes = size_t(64) << 20;

struct ListPlan {
  uint32_t dim, nslice;
  uint32_t row_lo, row_hi, slice0;  // rows written; first slice that holds one of them
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
    const unsigned long long old = atomicCAS(table + h, kNoCoef, bits);
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
    ar += d * xr;
    if (T::cplx) ai += d * xi;
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
// doubles, or null for none); null when they do not fit kListMaxBytes, the
// ranks 24 bits or the coefficients the class table.
ListHandle* list_plan_create(const DevPlan& p, uint64_t dim, const double* diag, size_t* dev_bytes) {
  const uint32_t nslice = uint32_t((dim + 31) / 32);
  // at least one slot per slice: cheap refusal of sectors that cannot fit
  if (dim == 0 || dim > kListMaxDim || p.ngroups == 0 || size_t(nslice) * 512 > kListMaxBytes) return nullptr;
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
    ok = total * 512 <= kListMaxBytes;
  }
  hs[nslice] = uint32_t(total);
  ok = ok && cudaMalloc(&words, std::max<size_t>(total, 1) * 512) == cudaSuccess &&
       cudaMemcpy(start, hs.data(), hs.size() * 4, cudaMemcpyHostToDevice) == cudaSuccess;
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
  const unsigned g = (p.nslice - p.slice0 + kListThreads / 32 - 1) / (kListThreads / 32);
  if (dot_out) {
    QKD_DISPATCH(t, (k_hx_list<DT, true><<<std::min<unsigned>(g, kMaxG), kListThreads, 0, s>>>(
                        p, x, y, w->partials, w->ticket, dot_out)));
  } else {
    QKD_DISPATCH(t, (k_hx_list<DT, false><<<g, kListThreads, 0, s>>>(p, x, y, nullptr, nullptr, nullptr)));
  }
  QKD_LAUNCH_CHECK();
  return QKD_OK;
}

}  // namespace qkd
