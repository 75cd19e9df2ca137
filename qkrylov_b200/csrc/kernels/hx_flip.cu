// H.x of unconditional bit flips on a complete basis (transverse-field Ising,
// XYZ chains written in Sx and Sy, ...): every off-diagonal group is valid in
// every state, so with all 2^n states present the row of x a group reads is
// row ^ flip and nothing has to be looked up.
//
// A CTA owns a tile of 2^10 or 2^11 rows staged in shared memory.  Groups whose
// flip stays inside the tile read it there (row ^ flip permutes a warp's
// addresses, so without bank conflicts), the others read the partner tile,
// whole aligned lines.  K rows per thread keep K partner loads in flight per
// group.  Bound: L2 -> SM traffic of the groups above the tile (n - 10 loads
// per row).  Transverse Ising, us per apply, two-part row kernel -> this
// kernel: N=20 complex64 31.2 -> 14.3, float64 38.0 -> 14.3, float32 28.7 ->
// 10.2; N=22 complex128 133 -> 82; N=14 complex64 10.2 -> 5.1 (row lists 5.1).
#include <algorithm>
#include <vector>

#include "reduce.cuh"

namespace qkd {

// Rows per tile (log2) and per thread: float32 2^11 and 8, wider types 2^10 and
// 4 (twice the tiles, so a smaller last wave).  Transverse Ising N=22, us per
// apply with 2^11 x 8 / 2^10 x 4: float32 26.6 / 30.8, float64 47.6 / 45.1,
// complex128 (2^11 x 4) 101 / 82; N=12 complex64 5.1 / 4.5.
constexpr int kFlipMinBits = 11;
template <int DT> constexpr int kFlipBits = DT == QK_F32 ? 11 : 10;
template <int DT> constexpr int kFlipK = DT == QK_F32 ? 8 : 4;
constexpr int kFlipMaxGroups = 128;

// coefficient w0 + (-1)^popcount(row & smask) w1
struct FlipGroup { uint32_t flip, smask; double w0, w1; };

struct FlipPlan {
  uint32_t ngroups, nlow10, nlow11;  // groups [0, nlow) stay inside a tile of 2^10 / 2^11 rows
  uint32_t row_lo, row_hi;
  const FlipGroup* groups;
  const double* diag;           // or null
};

struct FlipHandle {
  FlipPlan plan{};
  void* buf = nullptr;
};

namespace {

template <int DT, bool DOT>
__global__ void __launch_bounds__((1 << kFlipBits<DT>) / kFlipK<DT>)
k_hx_flip(const FlipPlan p, const void* __restrict__ x, void* __restrict__ y, double* partials, unsigned* ticket,
          double* dot_out) {
  using T = VT<DT>;
  using R = typename T::R;
  using E = typename T::E;
  constexpr int BITS = kFlipBits<DT>, K = kFlipK<DT>, NT = (1 << BITS) / K;
  const uint32_t nlow = BITS == 10 ? p.nlow10 : p.nlow11;
  __shared__ __align__(16) E sx[1 << BITS];
  __shared__ uint2 s_m[kFlipMaxGroups];
  __shared__ R s_w0[kFlipMaxGroups], s_w1[kFlipMaxGroups];
  for (uint32_t g = threadIdx.x; g < p.ngroups; g += NT) {
    const FlipGroup f = p.groups[g];
    s_m[g] = make_uint2(f.flip, f.smask);
    s_w0[g] = R(f.w0);
    s_w1[g] = R(f.w1);
  }
  double dr = 0.0, di = 0.0;
  const uint32_t t_hi = (p.row_hi + (1u << BITS) - 1) >> BITS;
  for (uint32_t tile = (p.row_lo >> BITS) + blockIdx.x; tile < t_hi; tile += gridDim.x) {
    const uint32_t r0 = (tile << BITS) + threadIdx.x;  // rows r0 + k * NT, all below 2^nbits
    R xr[K], xi[K], ar[K], ai[K];
    double d[K];
    #pragma unroll
    for (int k = 0; k < K; ++k) {
      T::ld(x, r0 + k * NT, xr[k], xi[k]);
      d[k] = p.diag ? __ldg(p.diag + r0 + k * NT) : 0.0;
    }
    if (tile != (p.row_lo >> BITS) + blockIdx.x) __syncthreads();  // the previous tile has been read
    #pragma unroll
    for (int k = 0; k < K; ++k) {
      T::st(sx, threadIdx.x + k * NT, xr[k], xi[k]);
      ar[k] = R(0);
      ai[k] = R(0);
    }
    __syncthreads();
    // adds group g's contribution from its partner values; groups without a
    // sign mask (uniform over the grid) have a nonzero constant coefficient
    auto add = [&](uint32_t g, const R (&vr)[K], const R (&vi)[K]) {
      const uint32_t m = s_m[g].y;
      const R w0 = s_w0[g];
      if (m == 0) {
        #pragma unroll
        for (int k = 0; k < K; ++k) {
          ar[k] += w0 * vr[k];
          if (T::cplx) ai[k] += w0 * vi[k];
        }
        return;
      }
      const R w1 = s_w1[g];
      #pragma unroll
      for (int k = 0; k < K; ++k) {
        const R c = (__popc((r0 + k * NT) & m) & 1) ? w0 - w1 : w0 + w1;
        if (c != R(0)) {  // no matrix element: an infinite x there must not reach y
          ar[k] += c * vr[k];
          if (T::cplx) ai[k] += c * vi[k];
        }
      }
    };
    for (uint32_t g = nlow; g < p.ngroups; ++g) {
      const uint32_t flip = s_m[g].x;
      R vr[K], vi[K];
      #pragma unroll
      for (int k = 0; k < K; ++k) T::ld(x, (r0 + k * NT) ^ flip, vr[k], vi[k]);
      add(g, vr, vi);
    }
    // the low flips in a sum of their own: half the terms, half the rounding
    R hr[K], hi[K];
    #pragma unroll
    for (int k = 0; k < K; ++k) { hr[k] = ar[k]; hi[k] = ai[k]; ar[k] = R(0); ai[k] = R(0); }
    for (uint32_t g = 0; g < nlow; ++g) {
      const uint32_t flip = s_m[g].x;
      R vr[K], vi[K];
      #pragma unroll
      for (int k = 0; k < K; ++k) T::ld_plain(sx, (threadIdx.x + k * NT) ^ flip, vr[k], vi[k]);
      add(g, vr, vi);
    }
    #pragma unroll
    for (int k = 0; k < K; ++k) {
      const uint32_t row = r0 + k * NT;
      ar[k] += hr[k];
      if (T::cplx) ai[k] += hi[k];
      if (p.diag) {  // none is not a zero one: an infinite x must not become a NaN
        ar[k] += R(d[k]) * xr[k];
        if (T::cplx) ai[k] += R(d[k]) * xi[k];
      }
      if (row >= p.row_lo && row < p.row_hi) {
        T::st(y, row, ar[k], ai[k]);
        if (DOT) {
          dr += double(xr[k]) * double(ar[k]) + double(xi[k]) * double(ai[k]);
          di += double(xr[k]) * double(ai[k]) - double(xi[k]) * double(ar[k]);
        }
      }
    }
  }
  if (DOT) {
    __shared__ double sbuf[2 * (NT / 32)];
    block_sum2(dr, di, sbuf);
    if (threadIdx.x == 0) { partials[2 * blockIdx.x] = dr; partials[2 * blockIdx.x + 1] = di; }
    grid_finish(partials, ticket, 1, dot_out);
  }
}

}  // namespace

void flip_plan_destroy(FlipHandle* h) {
  if (!h) return;
  cudaFree(h->buf);
  delete h;
}

// Whether the compiled operator consists of unconditional flips on all
// 2^nbits states (at least one tile of them): fills the groups.
static bool flip_groups(const qk_plan_desc* d, std::vector<FlipGroup>& out) {
  if (!d->all_real || d->nbits < kFlipMinBits || d->nbits > 31 || d->dim != (1ull << d->nbits)) return false;
  const uint32_t g0 = d->has_diag ? 1u : 0u;
  if (d->ngroups <= g0 || d->ngroups - g0 > uint32_t(kFlipMaxGroups)) return false;
  for (uint32_t gi = g0; gi < d->ngroups; ++gi) {
    const qk_group_t& g = d->groups[gi];
    FlipGroup f{uint32_t(g.flip), 0u, 0.0, 0.0};
    for (uint32_t q = g.first; q < g.first + g.count; ++q) {
      const qk_term_t& t = d->terms[q];
      if (t.cmask != 0) return false;
      if (t.smask == 0) f.w0 += t.wre;
      else if (f.smask == 0 || f.smask == uint32_t(t.smask)) { f.smask = uint32_t(t.smask); f.w1 += t.wre; }
      else return false;
    }
    if (f.smask != 0 || f.w0 != 0.0) out.push_back(f);
  }
  return !out.empty();
}

FlipHandle* flip_plan_create(const qk_plan_desc* d, const double* diag, size_t* dev_bytes) {
  std::vector<FlipGroup> g;
  if ((d->has_diag && !diag) || !flip_groups(d, g)) return nullptr;
  auto inside = [](int bits) { return [bits](const FlipGroup& f) { return (f.flip >> bits) == 0; }; };
  const auto mid11 = std::stable_partition(g.begin(), g.end(), inside(11));
  const auto mid10 = std::stable_partition(g.begin(), mid11, inside(10));
  auto* h = new FlipHandle;
  if (cudaMalloc(&h->buf, g.size() * sizeof(FlipGroup)) != cudaSuccess ||
      cudaMemcpy(h->buf, g.data(), g.size() * sizeof(FlipGroup), cudaMemcpyHostToDevice) != cudaSuccess) {
    (void)cudaGetLastError();
    flip_plan_destroy(h);
    return nullptr;
  }
  *dev_bytes += g.size() * sizeof(FlipGroup);
  h->plan.ngroups = uint32_t(g.size());
  h->plan.nlow10 = uint32_t(mid10 - g.begin());
  h->plan.nlow11 = uint32_t(mid11 - g.begin());
  h->plan.groups = static_cast<const FlipGroup*>(h->buf);
  h->plan.diag = d->has_diag ? diag : nullptr;
  return h;
}

bool flip_eligible(const qk_plan_desc* d) {
  std::vector<FlipGroup> g;
  return flip_groups(d, g);
}

// Rows [row_lo, row_hi) of y = H x; with dot_out (whole vectors) also <x, y>.
int flip_apply(const FlipHandle* h, qk_dtype t, const void* x, void* y, cudaStream_t s, qk_workspace* w,
               double* dot_out, uint64_t row_lo, uint64_t row_hi) {
  FlipPlan p = h->plan;
  p.row_lo = uint32_t(row_lo);
  p.row_hi = uint32_t(row_hi);
  QKD_DISPATCH(t, {
    constexpr int BITS = kFlipBits<DT>, NT = (1 << BITS) / kFlipK<DT>;
    const unsigned tiles = unsigned(((row_hi + (1u << BITS) - 1) >> BITS) - (row_lo >> BITS));
    if (dot_out)
      k_hx_flip<DT, true><<<std::min<unsigned>(tiles, kMaxG), NT, 0, s>>>(p, x, y, w->partials, w->ticket, dot_out);
    else
      k_hx_flip<DT, false><<<tiles, NT, 0, s>>>(p, x, y, nullptr, nullptr, nullptr);
  });
  QKD_LAUNCH_CHECK();
  return QKD_OK;
}

}  // namespace qkd
