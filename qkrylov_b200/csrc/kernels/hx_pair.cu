// H.x for operators with the spin-product structure of the Hubbard model:
// two bits per site (up at bit 2i, down at 2i+1), N_up and N_dn conserved,
// every off-diagonal term a hop of one spin species.  In the basis ordered by
// (up configuration, down configuration), with the sign
//   S(u, d) = (-1)^(number of pairs (down at site i, up at site j > i)),
// the reference's matrix is exactly
//   S H S = T_up (x) 1 + 1 (x) T_dn + D
// (the Jordan-Wigner strings of one species no longer see the other): a
// sparse matrix over the up configurations acting on whole rows of the
// product-ordered vector, one over the down configurations acting inside each
// row, and the diagonal.  The plan builder derives T_up and T_dn from the
// compiled terms and checks the structure before it is used (any failure:
// no plan, the two-part row kernel stays in charge).
//
// One apply is three passes over the vector:
//   k_pair_in   x_p[u][d] = S(u, d) x[rank(u, d)]       (reference -> product order)
//   k_pair_up   y_p[u][:] = sum_u' T_up[u][u'] x_p[u'][:]  (rows of the product
//               order; CTAs sweep column slabs so the partner rows of a slab
//               stay in L2)
//   k_pair_dn   y[rank(u, d)] = S(u, d) (y_p[u][d] + D[u][d] x_p[u][d]
//               + sum_d' T_dn[d][d'] x_p[u][d'])  (row u staged in shared memory;
//               fused column dot <x, y> when asked)
// rank(u, d) is the reference's index of the interleaved state, from the
// sector's two-level tables (offset of the high part + rank of the low part).
#include <algorithm>
#include <mutex>
#include <vector>

#include "hx_slots.hpp"
#include "reduce.cuh"
#include "../engine/sector.hpp"

namespace qkd {

struct PairPlan {
  uint32_t Du, Dd;         // up and down configurations
  // elements per row of every product-ordered array (x_p, y_p, D, ranks): Dd
  // rounded up to 32, so that rows start on 128-byte lines in every type and
  // can be read as 16-byte packs (what a row holds beyond Dd is never used)
  uint32_t ld;
  int L;                   // low bits of the sector tables
  uint32_t lmask;
  const uint64_t* A;       // sector tables (device copies owned by the qk_plan)
  const uint32_t* B;
  const uint32_t* ulist;   // up configurations (compressed site bits), ascending
  const uint32_t* dlist;
  // T_up: per row its first quad and its hops; a quad is four hops (target
  // indices, elements), the last one of a row filled with zeros
  const uint2* up_rec;
  const uint4* up_col;
  const double2* up_val;
  const uint32_t* dn_ptr;  // CSR of T_dn (Dd + 1)
  const uint32_t* dn_col;
  const double* dn_val;
  // T_dn in slots, when its elements have at most kMags magnitudes: per tile
  // of 32 rows the first group and the groups of each magnitude (8 bits each);
  // four slots of a row per uint2 ([group][lane]), each the target index with
  // the sign in bit 15 (indices Dd .. Dd + 7: no target, a zero pack)
  const uint2 *dn_rec, *dn_slot;
  double dn_mag[4];
  const double* diag;      // D in product order (Du * ld)
  const uint32_t* perm;    // rank(u, d) in product order (Du * ld), or null: computed from A, B
};

namespace {

constexpr int kMags = 4;  // magnitudes of the slot tables
constexpr int kPT = 256;  // threads per CTA of the gather
constexpr int kDT = 1024; // k_pair_dn: one staged row shared by 32 warps (two CTAs per SM)

__device__ __forceinline__ uint32_t spread16(uint32_t x) {  // bit i -> bit 2i (16 -> 32 bits)
  x &= 0xFFFFu;
  x = (x | (x << 8)) & 0x00FF00FFu;
  x = (x | (x << 4)) & 0x0F0F0F0Fu;
  x = (x | (x << 2)) & 0x33333333u;
  x = (x | (x << 1)) & 0x55555555u;
  return x;
}

// S(u, d): parity of the pairs (down at i, up at j > i) = parity(u & P) with
// P_j = XOR of d's bits below j
__device__ __forceinline__ double pair_sign(uint32_t u, uint32_t d) {
  uint32_t p = d << 1;
  p ^= p << 1; p ^= p << 2; p ^= p << 4; p ^= p << 8; p ^= p << 16;
  return (__popc(u & p) & 1) ? -1.0 : 1.0;
}

__device__ __forceinline__ uint32_t pair_rank(const PairPlan& p, uint32_t u, uint32_t d) {
  const uint32_t s = spread16(u) | (spread16(d) << 1);
  return uint32_t(__ldg(p.A + (s >> p.L)) & qkb::kOffsetMask) + (__ldg(p.B + (s & p.lmask)) & qkb::kRankMask);
}

// Work items of the gather: (u, kInCols * kPT columns), kInCols columns per
// thread so that as many ranks, then as many gathers, are in flight.
constexpr int kInCols = 4;
__host__ __device__ inline uint64_t in_items(uint32_t Du, uint32_t Dd) {
  return uint64_t(Du) * ((Dd + kInCols * kPT - 1) / (kInCols * kPT));
}

// SIGN false: the plain gather (the diagonal, on which S acts twice)
template <int DT, bool SIGN>
__global__ void __launch_bounds__(kPT) k_pair_in(const PairPlan* __restrict__ pp, const void* __restrict__ x,
                                                 void* __restrict__ xp) {
  using T = VT<DT>;
  using R = typename T::R;
  const PairPlan& p = *pp;
  const uint32_t Dd = p.Dd, nc = (Dd + kInCols * kPT - 1) / (kInCols * kPT);
  const uint64_t items = in_items(p.Du, Dd);
  for (uint64_t it = blockIdx.x; it < items; it += gridDim.x) {
    const uint32_t iu = uint32_t(it / nc), c0 = uint32_t(it - uint64_t(iu) * nc) * (kInCols * kPT) + threadIdx.x;
    const uint64_t row = uint64_t(iu) * p.ld;
    const uint32_t u = __ldg(p.ulist + iu);
    uint32_t d[kInCols], rk[kInCols];
    #pragma unroll
    for (int k = 0; k < kInCols; ++k) {  // spare columns of the last item repeat column Dd - 1
      const uint32_t c = min(c0 + k * kPT, Dd - 1);
      d[k] = __ldg(p.dlist + c);
      rk[k] = p.perm ? __ldg(p.perm + row + c) : pair_rank(p, u, d[k]);
    }
    R re[kInCols], im[kInCols];
    #pragma unroll
    for (int k = 0; k < kInCols; ++k) T::ld(x, rk[k], re[k], im[k]);
    #pragma unroll
    for (int k = 0; k < kInCols; ++k) {
      const R sg = SIGN ? R(pair_sign(u, d[k])) : R(1);
      if (c0 + k * kPT < Dd) T::st(xp, row + c0 + k * kPT, sg * re[k], sg * im[k]);
    }
  }
}

// perm[u][d] = rank(u, d)
__global__ void __launch_bounds__(kPT) k_pair_perm(const PairPlan* __restrict__ pp, uint32_t* __restrict__ perm) {
  const PairPlan& p = *pp;
  for (uint32_t iu = blockIdx.x; iu < p.Du; iu += gridDim.x) {
    const uint32_t u = __ldg(p.ulist + iu);
    for (uint32_t c = threadIdx.x; c < p.Dd; c += kPT) perm[uint64_t(iu) * p.ld + c] = pair_rank(p, u, __ldg(p.dlist + c));
  }
}

// A 16-byte pack of NE elements that a hop reads with one load.
template <class E, int NE>
struct alignas(sizeof(E) * NE) RowPack { E v[NE]; };

template <class P>
__device__ __forceinline__ P ldg_pack(const P* p) {
  static_assert(sizeof(P) == 16, "one 16-byte load");
  const uint4 q = __ldg(reinterpret_cast<const uint4*>(p));
  return *reinterpret_cast<const P*>(&q);
}

// y_p[u][...] = sum_u' T_up[u][u'] x_p[u'][...]: work item (slab of columns,
// u) in slab-major order, so that a slab of x_p (4 KB per row, 53 MB at 12,870
// rows) stays in L2 while its rows are combined.  The hops re-read x_p from
// L2, and the loads bound the kernel: L1 wavefronts (88% of its rate with
// 8-byte loads of unaligned rows and four one-word loads of index and element
// per hop and warp) and the bytes in flight.  So: 16-byte loads of aligned
// rows, four hops of two packs in flight per thread, three 16-byte loads for
// the indices and elements of four hops.  Whole apply, before -> after:
// Hubbard 4x4 float64 5.59 -> 4.86 ms, float32 3.81 -> 2.82 ms, 13 sites
// complex64 74.1 -> 70 us.  One pack per thread with 256 threads costs
// complex128 7% (7x2: 515 us against 480); eight hops in flight at fewer
// CTAs, 64 x 2 and 64 x 4 threads x packs are equal or slower.
constexpr int kUT = 128;  // threads
constexpr int kUP = 2;    // packs per thread
template <int DT>
__global__ void __launch_bounds__(kUT, 8) k_pair_up(const PairPlan* __restrict__ pp, const void* __restrict__ xp,
                                                 void* __restrict__ yp) {
  using T = VT<DT>;
  using R = typename T::R;
  constexpr int NR = 16 / int(sizeof(R));  // reals per pack
  using Pack = RowPack<R, NR>;
  const PairPlan& p = *pp;
  const uint32_t npk = p.ld / (16 / uint32_t(sizeof(typename T::E)));  // packs per row
  const uint32_t nslab = (npk + kUP * kUT - 1) / (kUP * kUT);
  const uint32_t items = nslab * p.Du;
  for (uint32_t it = blockIdx.x; it < items; it += gridDim.x) {
    const uint32_t slab = it / p.Du, iu = it - slab * p.Du;
    const uint32_t c = slab * kUP * kUT + threadIdx.x;
    const uint2 rec = __ldg(p.up_rec + iu);
    const uint4* __restrict__ col = p.up_col + rec.x;
    const double2* __restrict__ val = p.up_val + size_t(rec.x) * 2;
    const Pack* x[kUP];
    #pragma unroll
    for (int k = 0; k < kUP; ++k) x[k] = static_cast<const Pack*>(xp) + min(c + k * kUT, npk - 1);
    R a[kUP][NR];
    #pragma unroll
    for (int k = 0; k < kUP; ++k)
      #pragma unroll
      for (int r = 0; r < NR; ++r) a[k][r] = R(0);
    auto add = [&](const Pack (&v)[kUP], double w) {
      #pragma unroll
      for (int k = 0; k < kUP; ++k)
        #pragma unroll
        for (int r = 0; r < NR; ++r) a[k][r] += R(w) * v[k].v[r];
    };
    auto ld = [&](Pack (&v)[kUP], uint32_t row) {
      #pragma unroll
      for (int k = 0; k < kUP; ++k) v[k] = ldg_pack(x[k] + uint64_t(row) * npk);
    };
    uint32_t left = rec.y;
    Pack v[4][kUP];
    for (; left >= 4; left -= 4, ++col, val += 2) {
      const uint4 t = __ldg(col);
      ld(v[0], t.x); ld(v[1], t.y); ld(v[2], t.z); ld(v[3], t.w);
      const double2 w0 = __ldg(val), w1 = __ldg(val + 1);
      add(v[0], w0.x); add(v[1], w0.y); add(v[2], w1.x); add(v[3], w1.y);
    }
    if (left) {
      const uint4 t = __ldg(col);
      ld(v[0], t.x);
      if (left > 1) ld(v[1], t.y);
      if (left > 2) ld(v[2], t.z);
      const double2 w0 = __ldg(val), w1 = __ldg(val + 1);
      add(v[0], w0.x);
      if (left > 1) add(v[1], w0.y);
      if (left > 2) add(v[2], w1.x);
    }
    #pragma unroll
    for (int k = 0; k < kUP; ++k) {
      Pack o;
      #pragma unroll
      for (int r = 0; r < NR; ++r) o.v[r] = a[k][r];
      if (c + k * kUT < npk) static_cast<Pack*>(yp)[uint64_t(iu) * npk + c + k * kUT] = o;
    }
  }
}

__device__ __forceinline__ double flip_sign(double v, uint32_t e) {  // -v when bit 15 of e is set
  return __hiloint2double(__double2hiint(v) ^ int((e & 0x8000u) << 16), __double2loint(v));
}
__device__ __forceinline__ float flip_sign(float v, uint32_t e) {
  return __int_as_float(__float_as_int(v) ^ int((e & 0x8000u) << 16));
}

// The hops of row c (tile c / 32) on the staged packs: sum over magnitudes of
// magnitude * (sum of +-pack).  kAhead slot groups are loaded together, the
// next ones while these are summed (whole apply, Hubbard 4x4 complex64: two
// 4.40 ms, three 4.48, four 4.60; 7x2 float64: 262, 263, 269, six 281 us).
constexpr int kAhead = 2;
template <class T, class Pack, int NE>
__device__ __forceinline__ void hop_sum(const uint2* __restrict__ rec, const uint2* __restrict__ slot,
                                        const double* mag, uint32_t c, const Pack* xs, typename T::R (&sr)[NE],
                                        typename T::R (&si)[NE]) {
  using R = typename T::R;
  #pragma unroll
  for (int r = 0; r < NE; ++r) { sr[r] = R(0); si[r] = R(0); }
  const uint2 t = __ldg(rec + c / 32);
  const uint2* __restrict__ g = slot + size_t(t.x) * 32 + (c & 31u);
  for (int m = 0; m < kMags; ++m) {
    const uint32_t ng = (t.y >> (8 * m)) & 0xFFu;
    if (ng == 0) break;
    R ar[NE], ai[NE];
    #pragma unroll
    for (int r = 0; r < NE; ++r) { ar[r] = R(0); ai[r] = R(0); }
    auto hop = [&](uint32_t e) {
      const Pack pk = xs[e & 0x7FFFu];
      #pragma unroll
      for (int r = 0; r < NE; ++r) {
        if constexpr (T::cplx) {
          ar[r] += flip_sign(pk.v[r].x, e);
          ai[r] += flip_sign(pk.v[r].y, e);
        } else {
          ar[r] += flip_sign(pk.v[r], e);
        }
      }
    };
    uint2 q[kAhead];
    #pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (uint32_t(u) < ng) q[u] = __ldg(g + u * 32);
    for (uint32_t j = 0; j < ng; j += kAhead) {
      uint2 w[kAhead];
      #pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        w[u] = q[u];
        if (j + kAhead + u < ng) q[u] = __ldg(g + (j + kAhead + u) * 32);
      }
      #pragma unroll
      for (int u = 0; u < kAhead; ++u)
        if (j + u < ng) {
          hop(w[u].x & 0xFFFFu);
          hop(w[u].x >> 16);
          hop(w[u].y & 0xFFFFu);
          hop(w[u].y >> 16);
        }
    }
    g += ng * 32;
    const R f = R(mag[m]);
    #pragma unroll
    for (int r = 0; r < NE; ++r) { sr[r] += f * ar[r]; si[r] += f * ai[r]; }
  }
}

// NE * PL rows u of the product order staged in shared memory as PL planes
// of NE interleaved rows (16 bytes per column), so that one load fetches a
// column of NE rows; per column d the down hops are decoded once for all rows
// (SLOTS: from the slot tables, one plane; otherwise a CSR walk); per element the
// hops and the diagonal are added to y_p and the result goes to its
// reference-order place with the sign S.  DOT: <x, y> summed per
// CTA in a fixed order, then over CTAs (deterministic for a given grid).
template <int DT, bool DOT, int NE, int PL, int NT, bool SLOTS>
__global__ void __launch_bounds__(NT) k_pair_dn(const PairPlan* __restrict__ pp, const void* __restrict__ xp,
                                                const void* __restrict__ yp, void* __restrict__ y,
                                                double* partials, unsigned* ticket, double* dot_out) {
  using T = VT<DT>;
  using R = typename T::R;
  using E = typename T::E;
  constexpr int NR = NE * PL;
  using Pack = RowPack<E, NE>;
  extern __shared__ __align__(16) unsigned char smraw[];
  Pack* xs = reinterpret_cast<Pack*>(smraw);
  __shared__ double s_red[2 * (NT / 32)];
  const PairPlan& p = *pp;
  const uint32_t Dd = p.Dd, stride = Dd + 8;
  double dr = 0.0, di = 0.0;
  auto split = [](const E& v, R& re, R& im) {
    if constexpr (T::cplx) { re = v.x; im = v.y; } else { re = v; im = R(0); }
  };
  if (threadIdx.x < 8 * PL) {  // slots without a target
    Pack z;
    #pragma unroll
    for (int r = 0; r < NE; ++r) z.v[r] = E{};
    xs[(threadIdx.x / 8) * stride + Dd + threadIdx.x % 8] = z;
  }
  for (uint32_t iu0 = blockIdx.x * NR; iu0 < p.Du; iu0 += gridDim.x * NR) {
    const uint32_t nr = min(uint32_t(NR), p.Du - iu0);
    __syncthreads();  // the previous rows are finished with the staging
    for (uint32_t c = threadIdx.x; c < Dd; c += NT) {
      #pragma unroll
      for (int pl = 0; pl < PL; ++pl) {
        Pack v;
        #pragma unroll
        for (int r = 0; r < NE; ++r) {
          const uint32_t k = pl * NE + r;
          v.v[r] = k < nr ? __ldg(reinterpret_cast<const E*>(xp) + uint64_t(iu0 + k) * p.ld + c) : E{};
        }
        xs[pl * stride + c] = v;
      }
    }
    __syncthreads();
    for (uint32_t c = threadIdx.x; c < Dd; c += NT) {
      const uint32_t d = __ldg(p.dlist + c);
      // what the end of the row needs, in flight during the hops
      R ar[NR], ai[NR];
      double dg[NR];
      uint32_t rk[NR];
      #pragma unroll
      for (int r = 0; r < NR; ++r) {
        const uint32_t u = iu0 + (uint32_t(r) < nr ? r : 0);
        const uint64_t i = uint64_t(u) * p.ld + c;
        T::ld(yp, i, ar[r], ai[r]);
        dg[r] = __ldg(p.diag + i);
        rk[r] = p.perm ? __ldg(p.perm + i) : pair_rank(p, __ldg(p.ulist + u), d);
      }
      R sr[NR], si[NR];
      if constexpr (SLOTS) {
        static_assert(PL == 1, "the slot tables serve one plane");
        hop_sum<T, Pack, NE>(p.dn_rec, p.dn_slot, p.dn_mag, c, xs, sr, si);
      } else {
        const uint32_t k0 = __ldg(p.dn_ptr + c), k1 = __ldg(p.dn_ptr + c + 1);
        #pragma unroll
        for (int r = 0; r < NR; ++r) { sr[r] = R(0); si[r] = R(0); }
        for (uint32_t k = k0; k < k1; ++k) {
          const uint32_t t = __ldg(p.dn_col + k);
          const R w = R(__ldg(p.dn_val + k));
          #pragma unroll
          for (int pl = 0; pl < PL; ++pl) {
            const Pack pk = xs[pl * stride + t];
            #pragma unroll
            for (int r = 0; r < NE; ++r) {
              R vr, vi;
              split(pk.v[r], vr, vi);
              sr[pl * NE + r] += w * vr;
              if (T::cplx) si[pl * NE + r] += w * vi;
            }
          }
        }
      }
      #pragma unroll
      for (int pl = 0; pl < PL; ++pl) {
        const Pack own = xs[pl * stride + c];
        #pragma unroll
        for (int q = 0; q < NE; ++q) {
          const int r = pl * NE + q;
          if (uint32_t(r) < nr) {
            R xr, xi;
            split(own.v[q], xr, xi);
            ar[r] += R(dg[r]) * xr + sr[r];
            if (T::cplx) ai[r] += R(dg[r]) * xi + si[r];
            const R sg = R(pair_sign(__ldg(p.ulist + iu0 + r), d));
            T::st(y, rk[r], sg * ar[r], sg * ai[r]);
            if (DOT) {  // <x, y> = <x_p, y_p> (S^2 = 1)
              dr += double(xr) * double(ar[r]) + double(xi) * double(ai[r]);
              di += double(xr) * double(ai[r]) - double(xi) * double(ar[r]);
            }
          }
        }
      }
    }
  }
  if (DOT) {
    block_sum2(dr, di, s_red);
    if (threadIdx.x == 0) { partials[2 * blockIdx.x] = dr; partials[2 * blockIdx.x + 1] = di; }
    grid_finish(partials, ticket, 1, dot_out);
  }
}

}  // namespace

struct PairHandle {
  PairPlan host{};
  PairPlan* dev = nullptr;
  std::vector<void*> bufs;
  mutable std::mutex mu;
  mutable void* scr = nullptr;  // x_p and y_p, sized on first use
  mutable size_t scr_bytes = 0;
};

void pair_plan_destroy(PairHandle* h) {
  if (!h) return;
  for (void* b : h->bufs) cudaFree(b);
  cudaFree(h->scr);
  cudaFree(h->dev);
  delete h;
}

namespace {
uint32_t compress(uint64_t s, int shift, int nsites) {  // the bits of one species
  uint32_t v = 0;
  for (int i = 0; i < nsites; ++i) v |= uint32_t((s >> (2 * i + shift)) & 1u) << i;
  return v;
}
uint64_t interleave(uint32_t u, uint32_t d, int nsites) {
  uint64_t s = 0;
  for (int i = 0; i < nsites; ++i) s |= (uint64_t((u >> i) & 1u) << (2 * i)) | (uint64_t((d >> i) & 1u) << (2 * i + 1));
  return s;
}
int host_pair_sign(uint32_t u, uint32_t d, int nsites) {
  int c = 0;
  for (int i = 0; i < nsites; ++i)
    if ((d >> i) & 1u) c += __builtin_popcount(u >> (i + 1));
  return (c & 1) ? -1 : 1;
}
}  // namespace

// Slot tables (SlotTile) of a sparse matrix in CSR form, per tile of 32 rows
// and magnitude.  4x4 torus, 8 particles, 17.1 entries per row: 24 slots and 96
// wavefronts per warp (one slot per hop of the lattice: 28.9 slots and 134
// wavefronts, the whole kernel 2.69 -> 2.35 ms; by position in the row: 155
// wavefronts).  False when the elements have more than kMags magnitudes.
static bool hop_slots(const std::vector<uint32_t>& ptr, const std::vector<uint32_t>& col,
                      const std::vector<double>& val, double* mag, std::vector<uint2>& rec, std::vector<uint2>& slot) {
  const uint32_t n = uint32_t(ptr.size() - 1);
  if (n + 8 > 0x8000u) return false;
  int nmag = 0;
  std::vector<uint8_t> cls(val.size());
  for (size_t k = 0; k < val.size(); ++k) {
    int m = 0;
    while (m < nmag && mag[m] != std::abs(val[k])) ++m;
    if (m == kMags) return false;
    if (m == nmag) mag[nmag++] = std::abs(val[k]);
    cls[k] = uint8_t(m);
  }
  for (uint32_t r0 = 0; r0 < n; r0 += 32) {
    uint2 rc = make_uint2(uint32_t(slot.size() / 32), 0u);
    int out = 0;
    // magnitudes without an entry in this tile would end the kernel's walk
    // early, so every tile lists all of them: an absent one gets a group of
    // zero packs unless no later one is present
    int last = -1;
    for (uint32_t k = ptr[r0]; k < ptr[std::min(n, r0 + 32)]; ++k) last = std::max(last, int(cls[k]));
    for (int m = 0; m <= last; ++m, ++out) {
      SlotTile t(0x7FFFu);
      for (uint32_t i = 0; i < 32 && r0 + i < n; ++i)
        for (uint32_t k = ptr[r0 + i]; k < ptr[r0 + i + 1]; ++k)
          if (cls[k] == m) t.add(i, col[k] | (val[k] < 0 ? 0x8000u : 0u));
      const uint32_t ng = std::max(1u, t.groups());
      if (ng > 255) return false;
      rc.y |= ng << (8 * out);
      t.write(ng, n, slot);
    }
    rec.push_back(rc);
  }
  if (slot.empty()) slot.push_back(make_uint2(0, 0));
  return true;
}

// Host side: eligibility, T_up / T_dn from the compiled terms (the matrix
// element of row s is the term's coefficient with its parity sign, target
// s ^ flip; products with S on both sides), a check that they do not depend
// on the other species' configuration, and the device tables.  Returns
// nullptr when the operator does not have the structure.  A, B: the plan's
// device copies of the sector tables.  diag_ref: the operator's diagonal
// (device, reference order, dim doubles).
PairHandle* pair_plan_create(const qk_plan_desc* d, const uint64_t* A_dev, const uint32_t* B_dev,
                             const double* diag_ref, size_t* dev_bytes) {
  if (!d->pair_sites || !d->all_real || d->nbits > 32 || (d->nbits & 1) || d->dim == 0 || d->dim >= (1ull << 32))
    return nullptr;
  const int ns = d->nbits / 2;
  if (ns > 16 || d->L <= 0 || d->L > 16) return nullptr;
  // the first state fixes N_up and N_dn; the sector must hold every
  // combination of those (its size is the product)
  uint64_t s0 = ~0ull;
  for (uint64_t h = 0; h < d->nA && s0 == ~0ull; ++h) {
    const uint32_t need = uint32_t(d->A[h] >> 56);
    if (need == qkb::kEmptyBlockKey) continue;
    if (d->key_off[need + 1] == d->key_off[need]) continue;
    s0 = (h << d->L) | d->llist[d->key_off[need]];
  }
  if (s0 == ~0ull) return nullptr;
  const int nu = __builtin_popcount(compress(s0, 0, ns)), nd = __builtin_popcount(compress(s0, 1, ns));
  std::vector<uint32_t> ul, dl;
  for (uint32_t v = 0; v < (1u << ns); ++v) {
    if (__builtin_popcount(v) == nu) ul.push_back(v);
    if (__builtin_popcount(v) == nd) dl.push_back(v);
  }
  if (uint64_t(ul.size()) * dl.size() != d->dim || dl.size() >= 32768) return nullptr;
  auto in_sector = [&](uint64_t s) {
    const uint64_t a = d->A[s >> d->L];
    const uint32_t b = d->B[s & ((1ull << d->L) - 1)];
    return uint32_t(a >> 56) == (b >> 24);
  };
  if (!in_sector(interleave(ul.back(), dl.back(), ns)) || !in_sector(interleave(ul[0], dl.back(), ns))) return nullptr;
  // off-diagonal groups: hops of one species (flip within the even or the odd bits)
  const uint64_t even = 0x5555555555555555ull & ((ns >= 32) ? ~0ull : ((1ull << (2 * ns)) - 1));
  std::vector<uint32_t> gup, gdn;
  for (uint32_t gi = d->has_diag ? 1u : 0u; gi < d->ngroups; ++gi) {
    const qk_group_t& g = d->groups[gi];
    if (g.flip == 0) return nullptr;
    if ((g.flip & ~even) == 0) gup.push_back(gi);
    else if ((g.flip & even) == 0) gdn.push_back(gi);
    else return nullptr;
    for (uint32_t q = g.first; q < g.first + g.count; ++q)
      if (d->terms[q].wim != 0.0) return nullptr;
  }
  std::vector<uint32_t> uidx(size_t(1) << ns, ~0u), didx(size_t(1) << ns, ~0u);
  for (uint32_t i = 0; i < ul.size(); ++i) uidx[ul[i]] = i;
  for (uint32_t i = 0; i < dl.size(); ++i) didx[dl[i]] = i;
  // row `a` of T_species at a fixed configuration `o` of the other species:
  // (column index, value) pairs in term order
  auto row = [&](bool up, uint32_t a, uint32_t o, std::vector<std::pair<uint32_t, double>>& out) -> bool {
    out.clear();
    const uint64_t s = up ? interleave(a, o, ns) : interleave(o, a, ns);
    const int ss = up ? host_pair_sign(a, o, ns) : host_pair_sign(o, a, ns);
    const std::vector<uint32_t>& groups = up ? gup : gdn;
    for (uint32_t gi : groups) {
      const qk_group_t& g = d->groups[gi];
      const uint64_t t = s ^ g.flip;
      double c = 0.0;
      for (uint32_t q = g.first; q < g.first + g.count; ++q) {
        const qk_term_t& tm = d->terms[q];
        if ((s & tm.cmask) != tm.cval) continue;
        c += (__builtin_popcountll(s & tm.smask) & 1) ? -tm.wre : tm.wre;
      }
      if (c == 0.0) continue;
      const uint32_t a2 = up ? compress(t, 0, ns) : compress(t, 1, ns);
      const uint32_t o2 = up ? compress(t, 1, ns) : compress(t, 0, ns);
      if (o2 != o) return false;
      const uint32_t idx = up ? uidx[a2] : didx[a2];
      if (idx == ~0u) return false;
      const int ts = up ? host_pair_sign(a2, o, ns) : host_pair_sign(o, a2, ns);
      out.push_back({idx, double(ss * ts) * c});
    }
    return true;
  };
  std::vector<uint2> urec;
  std::vector<uint32_t> ucol, dptr(1, 0), dcol;
  std::vector<double> uval, dval;
  std::vector<std::pair<uint32_t, double>> r, r2;
  const uint32_t o_chk[2][2] = {{dl[dl.size() / 2], dl.back()}, {ul[ul.size() / 2], ul.back()}};
  for (int sp = 0; sp < 2; ++sp) {
    const bool up = sp == 0;
    const std::vector<uint32_t>& own = up ? ul : dl;
    const uint32_t o0 = up ? dl[0] : ul[0];
    for (uint32_t a : own) {
      if (!row(up, a, o0, r)) return nullptr;
      for (int k = 0; k < 2; ++k) {  // the row must not depend on the other species
        if (!row(up, a, o_chk[sp][k], r2) || r2 != r) return nullptr;
      }
      if (up) urec.push_back(make_uint2(uint32_t(ucol.size() / 4), uint32_t(r.size())));
      for (auto& e : r) {
        (up ? ucol : dcol).push_back(e.first);
        (up ? uval : dval).push_back(e.second);
      }
      for (; up && ucol.size() % 4; uval.push_back(0.0)) ucol.push_back(0);
      if (!up) dptr.push_back(uint32_t(dcol.size()));
    }
  }
  std::vector<uint2> drec, dslot;
  double dmag[kMags] = {0.0, 0.0, 0.0, 0.0};
  const bool dslots = hop_slots(dptr, dcol, dval, dmag, drec, dslot);
  auto* out = new PairHandle;
  bool ok = true;
  auto up_ = [&](const void* src, size_t bytes) -> void* {
    void* p = nullptr;
    if (!ok) return nullptr;
    bytes = std::max<size_t>(bytes, 8);
    if (cudaMalloc(&p, bytes) != cudaSuccess) { ok = false; return nullptr; }
    out->bufs.push_back(p);
    *dev_bytes += bytes;
    if (src && cudaMemcpy(p, src, bytes, cudaMemcpyHostToDevice) != cudaSuccess) ok = false;
    return p;
  };
  PairPlan& h = out->host;
  h.Du = uint32_t(ul.size()); h.Dd = uint32_t(dl.size());
  h.ld = (h.Dd + 31u) & ~31u;
  const size_t np = size_t(h.Du) * h.ld;
  h.L = d->L; h.lmask = uint32_t((1ull << d->L) - 1);
  h.A = A_dev; h.B = B_dev;
  h.ulist = static_cast<const uint32_t*>(up_(ul.data(), ul.size() * 4));
  h.dlist = static_cast<const uint32_t*>(up_(dl.data(), dl.size() * 4));
  h.up_rec = static_cast<const uint2*>(up_(urec.data(), urec.size() * sizeof(uint2)));
  h.up_col = static_cast<const uint4*>(up_(ucol.data(), ucol.size() * 4));
  h.up_val = static_cast<const double2*>(up_(uval.data(), uval.size() * 8));
  h.dn_ptr = static_cast<const uint32_t*>(up_(dptr.data(), dptr.size() * 4));
  if (dslots) {
    h.dn_rec = static_cast<const uint2*>(up_(drec.data(), drec.size() * sizeof(uint2)));
    h.dn_slot = static_cast<const uint2*>(up_(dslot.data(), dslot.size() * sizeof(uint2)));
  } else {
    h.dn_col = static_cast<const uint32_t*>(up_(dcol.data(), dcol.size() * 4));
    h.dn_val = static_cast<const double*>(up_(dval.data(), dval.size() * 8));
  }
  for (int m = 0; m < kMags; ++m) h.dn_mag[m] = dmag[m];
  double* dp = static_cast<double*>(up_(nullptr, np * 8));
  h.diag = dp;
  if (ok) {
    out->dev = nullptr;
    ok = cudaMalloc(reinterpret_cast<void**>(&out->dev), sizeof(PairPlan)) == cudaSuccess &&
         cudaMemcpy(out->dev, &h, sizeof(PairPlan), cudaMemcpyHostToDevice) == cudaSuccess;
    if (ok) *dev_bytes += sizeof(PairPlan);
  }
  if (ok) {  // the diagonal in product order (no sign: S D S = D)
    const unsigned g = resident_grid(k_pair_in<QK_F64, false>, kPT, 0, unsigned(std::min<uint64_t>(4096, in_items(h.Du, h.Dd))));
    k_pair_in<QK_F64, false><<<g, kPT>>>(out->dev, diag_ref, dp);
    ok = cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess;
  }
  if (ok) {
    // the reference rank of every product index, read coalesced by the
    // gather and the scatter instead of two scattered table lookups per
    // element (4 bytes per state; without the memory the kernels compute it)
    uint32_t* pm = nullptr;
    if (cudaMalloc(&pm, np * 4) == cudaSuccess) {
      out->bufs.push_back(pm);
      *dev_bytes += np * 4;
      k_pair_perm<<<resident_grid(k_pair_perm, kPT, 0, 4096), kPT>>>(out->dev, pm);
      ok = cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess;
      h.perm = pm;
      ok = ok && cudaMemcpy(out->dev, &h, sizeof(PairPlan), cudaMemcpyHostToDevice) == cudaSuccess;
    } else {
      (void)cudaGetLastError();
    }
  }
  if (!ok) {
    (void)cudaGetLastError();
    pair_plan_destroy(out);
    return nullptr;
  }
  return out;
}

// y = H x (and <x, y> into dot_out when given) through the product order.
// QKD_EINVAL when the scratch is missing and cannot be allocated now (during
// a stream capture): the caller then takes the row kernel.
int pair_apply(const PairHandle* h, qk_dtype t, const void* x, void* y, cudaStream_t s, qk_workspace* w,
               double* dot_out) {
  if (!h || !x || !y || x == y) return QKD_EINVAL;
  const size_t es = qk_dtype_size(t);
  const size_t half = (size_t(h->host.Du) * h->host.ld * es + 255) & ~size_t(255);  // x_p and y_p on 256-byte boundaries
  void* scr = nullptr;
  {
    std::lock_guard<std::mutex> lk(h->mu);
    if (h->scr_bytes < 2 * half) {
      cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
      if (cudaStreamIsCapturing(s, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) return QKD_EINVAL;
      cudaFree(h->scr);
      h->scr = nullptr;
      h->scr_bytes = 0;
      if (cudaMalloc(&h->scr, 2 * half) != cudaSuccess) {
        (void)cudaGetLastError();
        return QKD_EINVAL;
      }
      h->scr_bytes = 2 * half;
    }
    scr = h->scr;
  }
  void* xp = scr;
  void* yp = static_cast<char*>(scr) + half;
  // rows staged per pass of the down-hop kernel: as many as fill 16 bytes per
  // column (fewer where the stage cannot hold them); the CSR walk, which the
  // decoding bounds, takes up to four
  constexpr size_t kStage = 220 * 1024;
  const size_t cols = size_t(h->host.Dd) + 8;
  if (es * size_t(h->host.Dd) > kStage) return QKD_EINVAL;
  int ne = int(std::max<size_t>(1, std::min<size_t>(16 / es, kStage / (es * cols))));
  ne = ne >= 4 ? 4 : ne >= 2 ? 2 : 1;
  int pl = 1;
  if (!h->host.dn_rec && size_t(ne) * es == 16)
    while (ne * pl < 4 && es * cols * ne * pl * 2 <= kStage) pl *= 2;
  const size_t smem = es * cols * ne * pl;
#define QKD_PAIR_DN1(DT, DOT, NE, PL, NT, SL)                                                               \
  {                                                                                                        \
    auto k = k_pair_dn<DT, DOT, NE, PL, NT, SL>;                                                           \
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess)     \
      return QKD_EINVAL;                                                                                   \
    const unsigned rows = (h->host.Du + NE * PL - 1) / (NE * PL);                                          \
    const unsigned g = resident_grid(k, NT, smem, DOT ? std::min<unsigned>(rows, kMaxG) : rows);           \
    k<<<g, NT, smem, s>>>(h->dev, xp, yp, y, DOT ? w->partials : nullptr, DOT ? w->ticket : nullptr, dot_out); \
  }
#define QKD_PAIR_DN(DT, DOT, NE)                                                                           \
  {                                                                                                        \
    constexpr bool full = NE * sizeof(VT<DT>::E) == 16;                                                    \
    if (h->host.dn_rec) {                                                                                  \
      if (smem <= kStage / 2) QKD_PAIR_DN1(DT, DOT, NE, 1, 512, true)                                      \
      else QKD_PAIR_DN1(DT, DOT, NE, 1, kDT, true)                                                         \
    } else if (full && pl == 4) QKD_PAIR_DN1(DT, DOT, NE, (full && NE == 1 ? 4 : 1), kDT, false)           \
    else if (full && pl == 2) QKD_PAIR_DN1(DT, DOT, NE, (full && NE <= 2 ? 2 : 1), kDT, false)             \
    else QKD_PAIR_DN1(DT, DOT, NE, 1, kDT, false)                                                          \
  }
#define QKD_PAIR_DNS(DT, DOT)                                                                              \
  {                                                                                                        \
    constexpr int MAXR = 16 / int(sizeof(VT<DT>::E));                                                      \
    if constexpr (MAXR >= 4) { if (ne == 4) QKD_PAIR_DN(DT, DOT, 4) }                                      \
    if constexpr (MAXR >= 2) { if (ne == 2) QKD_PAIR_DN(DT, DOT, 2) }                                      \
    if (ne == 1) QKD_PAIR_DN(DT, DOT, 1)                                                                   \
  }
#define QKD_PAIR(DT)                                                                                       \
  {                                                                                                        \
    const unsigned gi = unsigned(std::min<uint64_t>(1u << 20, in_items(h->host.Du, h->host.Dd)));          \
    k_pair_in<DT, true><<<resident_grid(k_pair_in<DT, true>, kPT, 0, gi), kPT, 0, s>>>(h->dev, x, xp);     \
    k_pair_up<DT><<<resident_grid(k_pair_up<DT>, kUT, 0, 1u << 20), kUT, 0, s>>>(h->dev, xp, yp);          \
    if (dot_out) QKD_PAIR_DNS(DT, true) else QKD_PAIR_DNS(DT, false)                                       \
  }
  switch (t) {
    case QK_C128: QKD_PAIR(QK_C128); break;
    case QK_C64: QKD_PAIR(QK_C64); break;
    case QK_F64: QKD_PAIR(QK_F64); break;
    case QK_F32: QKD_PAIR(QK_F32); break;
    default: return QKD_EINVAL;
  }
#undef QKD_PAIR
#undef QKD_PAIR_DNS
#undef QKD_PAIR_DN
#undef QKD_PAIR_DN1
  QKD_LAUNCH_CHECK();
  return QKD_OK;
}

}  // namespace qkd
