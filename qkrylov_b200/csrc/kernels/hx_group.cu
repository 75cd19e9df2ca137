// Row kernel over groups of sector blocks.
//
// k_hx_spin_rows (hx_spin.cu) decodes a row's tables for one block at a time:
// 390 (complex128, Heisenberg N=28) to 680 (t-J N=20) instructions per 32 rows,
// most of them for indices that do not depend on the block.  Here a CTA takes
// G blocks with the same low-part class, the same sign pattern of the crossing
// diagonal terms and the same crossing flags, and a thread computes the same
// class position of all G blocks: the low targets, the crossing ranks, their
// validity and coefficients are read and decoded once for G rows, and G rows'
// loads are in flight together.
//   staging  x of the G blocks interleaved in 16-byte packs ([plane][position],
//            16 / sizeof(element) blocks per pack), so that a low target is one
//            16-byte load per plane
//   low      the targets of 32 consecutive positions (a warp) in slots without
//            bank conflicts (hx_slots.hpp), four slots per 8-byte table load,
//            grouped by coefficient class; one slot per bond instead, half of its
//            rows without the bond: t-J N=20 complex128 424 -> 451 us, J1-J2
//            N=24 float64 71.7 -> 76.0, Heisenberg N=28 complex128 893 -> 918
//   high     per block, its entries (partner block, coefficient) from shared
//            memory; U entries of every block in flight, without branches
//   crossing per row table words shared by the G blocks
// Groups shorter than G repeat their first block and do not store it.
//
// Bound: latency of the partner rows and the tables (issue 35-55%, L1 data
// pipe 45-70% busy), so resident warps count: 64 registers and 32 warps for
// float32 and complex128, 48 registers and 40 warps for the 8-byte types; more
// entries in flight, tables or slots loaded a row ahead and unconditional
// crossing loads were each slower.  us per apply, one-block kernel -> this one:
// Heisenberg N=24 float32 46.6 -> 35, N=25 float64 102 -> 69, N=24 complex128
// 86 -> 64, N=28 float32 437 -> 325, float64 590 -> 513; J1-J2 N=24 float32 81 ->
// 57; t-J N=19 float64 177 -> 96, N=20 float64 333 -> 222, complex128 529 -> 425.
// Heisenberg N=28 complex128 depends on where the vectors lie: 980 -> 896 in two
// buffers of cudaMalloc, 990-1033 -> 951-999 in two of torch's allocator (the
// cause of the difference is not known).
#include <algorithm>
#include <cstring>
#include <map>
#include <vector>

#include "hx_group.hpp"
#include "hx_rows.cuh"

namespace qkd {

namespace {

constexpr int kRecWords = sizeof(GroupRec) / 4;

template <class R> struct alignas(sizeof(R) == 4 ? 8 : 16) GroupEnt { uint32_t base; R c; };

template <class E> struct alignas(16) Pack16 { E v[16 / sizeof(E)]; };

__device__ __forceinline__ uint32_t group_fetch(const GroupPlan& p, uint32_t* wq, int die) {
  for (int k = 0; k < 2; ++k) {
    const int q = die ^ k;
    const uint32_t beg = q ? p.qsplit : 0u, n = q ? p.nitems - p.qsplit : p.qsplit;
    const uint32_t i = atomicAdd(wq + q, 1u);
    if (i < n) return beg + i;
  }
  return p.nitems;
}

template <int DT, bool DOT, bool GEN, int G, int U, int NT, int MINC>
__global__ void __launch_bounds__(NT, MINC)
k_hx_group(const __grid_constant__ GroupPlan p, const void* __restrict__ x, void* __restrict__ y, double* partials,
           unsigned* ticket, double* dot_out, uint32_t* wq, uint32_t row_lo, uint32_t row_hi) {
  using T = VT<DT>;
  using R = typename T::R;
  using E = typename T::E;
  using Ent = GroupEnt<R>;
  using Pack = Pack16<E>;
  constexpr int EPP = 16 / int(sizeof(E)), PL = (G + EPP - 1) / EPP;  // blocks per pack, planes
  extern __shared__ __align__(16) unsigned char sm[];
  Pack* sx = reinterpret_cast<Pack*>(sm);
  const E* __restrict__ xg = reinterpret_cast<const E*>(x);
  __shared__ __align__(16) uint32_t s_rec[2][kRecWords];
  __shared__ Ent s_ent[G][kRowEnt];
  __shared__ uint32_t s_cb[G][kRowCross], s_cf[kRowCross], s_pos[2];
  __shared__ R s_cc[kRowCross], s_coef[kRowCoef], s_lc[kRowCls];
  __shared__ double s_dot[2 * (NT / 32)];
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  const uint32_t stride = p.zero_slot + 8, nll = p.nllist;
  const int ncross = p.ncross, ncls = p.ncls;
  for (int i = tid; i < kRowCoef; i += NT) s_coef[i] = R(p.coef[i]);
  if (tid < kRowCls) s_lc[tid] = R(p.lcls[tid]);
  if (tid < 8 * PL) {
    Pack z;
    #pragma unroll
    for (int u = 0; u < EPP; ++u) szero(z.v[u]);
    sx[(tid / 8) * stride + p.zero_slot + tid % 8] = z;
  }
  // one coefficient for every high entry (uniform chains): summed, then scaled;
  // complex128 alone gains (Heisenberg N=28, before the coloured slots, 959 -> 924 us), the others need the
  // registers (float64 531 -> 580)
  const bool uni = DT == QK_C128 && !GEN && p.uniform_high;
  const R high = R(p.high_coef);
  int die = 0;
  if (wq) {
    uint32_t sid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(sid));
    die = (p.sm_die && sid < p.nsmid) ? int(__ldg(p.sm_die + sid)) : 0;
  }
  // items: this one's record in s_rec[b], the next one's number in s_pos[b]
  if (tid == 0) {
    s_pos[0] = wq ? group_fetch(p, wq, die) : blockIdx.x;
    s_pos[1] = wq ? group_fetch(p, wq, die) : blockIdx.x + gridDim.x;
  }
  __syncthreads();
  uint32_t item = s_pos[0], next = s_pos[1];
  if (item < p.nitems && tid < kRecWords) s_rec[0][tid] = __ldg(reinterpret_cast<const uint32_t*>(p.rec + item) + tid);
  uint32_t prev = p.nitems;
  double dr = 0.0, di = 0.0;
  __syncthreads();
  for (uint32_t it = 0; item < p.nitems; ++it) {
    const uint32_t b = it & 1;
    if (DOT && prev < p.nitems && tid == 0) {
      double sr = 0.0, si = 0.0;
      for (int w = 0; w < NT / 32; ++w) { sr += s_dot[2 * w]; si += s_dot[2 * w + 1]; }
      partials[2 * size_t(prev)] = sr;
      partials[2 * size_t(prev) + 1] = si;
    }
    const GroupRec& rec = *reinterpret_cast<const GroupRec*>(s_rec[b]);
    // the next record and the number after it arrive while this item runs
    uint32_t nword = 0, npos = 0;
    if (next < p.nitems && tid < kRecWords) nword = __ldg(reinterpret_cast<const uint32_t*>(p.rec + next) + tid);
    if (tid == 0) npos = wq ? group_fetch(p, wq, die) : next + gridDim.x;
    const uint32_t size = rec.size, lst = rec.lst, tile0 = rec.tile0;
    uint32_t base[G];
    bool act[G];
    bool any = false;
    #pragma unroll
    for (int g = 0; g < G; ++g) {
      base[g] = rec.base[g];
      act[g] = g < int(rec.count) && base[g] >= row_lo && base[g] < row_hi;
      any = any || act[g];
    }
    if (any) {
      for (uint32_t i = tid; i < G * (kRowEnt + kRowCross); i += NT) {
        const uint32_t g = i / (kRowEnt + kRowCross), e = i - g * (kRowEnt + kRowCross), nh = rec.nh[g];
        if (e < kRowEnt) {
          if (e < nh) {
            const uint2 q = __ldg(p.bent + rec.ebeg[g] + e);
            s_ent[g][e].base = q.x;
            s_ent[g][e].c = R(p.coef[q.y & 0xFFFFu]);
            if (p.prefetch) l2_prefetch(x, sizeof(E), q.x, min(size, uint32_t(2 * NT)));
          } else {  // loaded beyond the last entry, not added
            s_ent[g][e].base = rec.base[g];
          }
        } else if (e - kRowEnt < uint32_t(ncross)) {
          const uint32_t q = e - kRowEnt;
          const uint2 w = __ldg(p.bent + rec.ebeg[g] + nh + q);
          s_cb[g][q] = w.x;
          if (g == 0) {  // the same in every block of the group
            s_cf[q] = GEN ? w.y : w.y >> 16;
            s_cc[q] = GEN ? R(0) : R(p.coef[w.y & 0xFFFFu]);
          }
        }
      }
      for (uint32_t l = tid; l < size; l += NT) {
        #pragma unroll
        for (int pl = 0; pl < PL; ++pl) {
          Pack v;
          #pragma unroll
          for (int u = 0; u < EPP; ++u) {
            szero(v.v[u]);
            if (pl * EPP + u < G) v.v[u] = __ldg(xg + base[pl * EPP + u] + l);
          }
          sx[pl * stride + l] = v;
        }
      }
    }
    __syncthreads();
    uint32_t chm = 0u;  // two-part: crossing groups with a term whose high condition holds in these blocks
    if constexpr (GEN)
      for (int q = 0; q < ncross; ++q) chm |= (((s_cf[q] >> 16) | (s_cf[q] >> 18)) & 1u) << q;
    const double* __restrict__ dtab = p.dtab + size_t(rec.combo) * nll + lst;
    const uint32_t* __restrict__ ckw = reinterpret_cast<const uint32_t*>(p.crk);
    const uint32_t cw = uint32_t(p.cpad) >> 1;
    // entries per block: in registers for exchange tables (Heisenberg N=26
    // float64 151.5 -> 147.4 us), re-read from shared memory for two-part ones,
    // whose crossing loop needs the registers (t-J N=20 float32 202 -> 183 us)
    uint32_t nhr[G], nmax = 0;
    #pragma unroll
    for (int g = 0; g < G; ++g) { nhr[g] = rec.nh[g]; nmax = max(nmax, nhr[g]); }
    const uint32_t* const nhs = rec.nh;
    auto nh = [&](int g) { return GEN ? nhs[g] : nhr[g]; };
    for (uint32_t l = tid; any && l < size; l += NT) {
      if (p.prefetch) {  // the partner rows two chunks ahead go to L2
        const uint32_t ahead = l - tid + 2u * NT;
        if (ahead < size)
          for (uint32_t i = tid; i < G * kRowEnt; i += NT) {
            const uint32_t g = i / kRowEnt, e = i - g * kRowEnt;
            if (e < rec.nh[g]) l2_prefetch(x, sizeof(E), s_ent[g][e].base + ahead, min(size - ahead, uint32_t(NT)));
          }
      }
      const uint32_t pos = lst + l;
      const uint2 wr = __ldg(p.wrec + tile0 + l / 32);
      const double dt = GEN ? 0.0 : __ldg(dtab + l);
      const uint32_t tw0 = GEN ? __ldg(p.crm + pos) : ncross ? __ldg(ckw + size_t(pos) * cw) : 0u;
      const uint2* __restrict__ wg = p.wgrp + size_t(wr.x) * 32 + lane;
      const uint32_t nt = (wr.y & 0xFFu) + ((wr.y >> 8) & 0xFFu) + ((wr.y >> 16) & 0xFFu) + (wr.y >> 24);
      R ar[G], ai[G];
      #pragma unroll
      for (int g = 0; g < G; ++g) { ar[g] = R(0); ai[g] = R(0); }
      // high bonds: the same position of a partner block, U entries of every
      // block in flight together.  The loads are unconditional (entries past a
      // block's last one name the block itself and are not added): with
      // branches around them Heisenberg N=24 float32 took 50 us instead of 37
      for (uint32_t e0 = 0; e0 < nmax; e0 += U) {
        R vr[G][U], vi[G][U];
        #pragma unroll
        for (int g = 0; g < G; ++g)
          #pragma unroll
          for (int u = 0; u < U; ++u) {
            T::ld(x, uint64_t(s_ent[g][e0 + u].base) + l, vr[g][u], vi[g][u]);
          }
        #pragma unroll
        for (int g = 0; g < G; ++g)
          #pragma unroll
          for (int u = 0; u < U; ++u)
            if (e0 + u < nh(g)) {
              const R c = uni ? R(1) : s_ent[g][e0 + u].c;
              ar[g] += c * vr[g][u];
              if (T::cplx) ai[g] += c * vi[g][u];
            }
      }
      if (uni) {
        #pragma unroll
        for (int g = 0; g < G; ++g) { ar[g] *= high; if (T::cplx) ai[g] *= high; }
      }
      if constexpr (GEN) {
        // two-part crossing groups whose low and high masks both allow a term,
        // two at a time: coefficient and rank are the same for all G blocks
        for (uint32_t m = tw0 & chm; m;) {
          int qq[2];
          uint32_t ent[2];
          #pragma unroll
          for (int u = 0; u < 2; ++u) {
            qq[u] = m ? __ffs(m) - 1 : -1;
            m &= m - 1u;
            ent[u] = qq[u] >= 0 ? __ldg(p.crk32 + size_t(qq[u]) * nll + pos) : 0u;
          }
          R c[2], vr[2][G], vi[2][G];
          #pragma unroll
          for (int u = 0; u < 2; ++u) {
            c[u] = qq[u] >= 0 ? cross_coef<R>(ent[u], s_cf[qq[u]], s_coef) : R(0);
            #pragma unroll
            for (int g = 0; g < G; ++g)  // no term: the block's own row, not added
              T::ld(x, c[u] != R(0) ? uint64_t(s_cb[g][qq[u]]) + (ent[u] & 0xFFFFFFu) : uint64_t(base[g]) + l, vr[u][g],
                    vi[u][g]);
          }
          #pragma unroll
          for (int u = 0; u < 2; ++u)
            if (c[u] != R(0)) {
              #pragma unroll
              for (int g = 0; g < G; ++g) { ar[g] += c[u] * vr[u][g]; if (T::cplx) ai[g] += c[u] * vi[u][g]; }
            }
        }
      } else {
        uint32_t tw = tw0;
        for (int q = 0; q < ncross; q += 2) {
          uint32_t twn = 0u;
          if (q + 2 < ncross) twn = __ldg(ckw + size_t(pos) * cw + ((q + 2) >> 1));
          #pragma unroll
          for (int u = 0; u < 2; ++u) {
            const uint32_t ent = u ? (tw >> 16) : (tw & 0xFFFFu);
            if (q + u < ncross && (ent >> 15) != s_cf[q + u]) {
              const R c = s_cc[q + u];
              R vr[G], vi[G];
              #pragma unroll
              for (int g = 0; g < G; ++g) T::ld(x, uint64_t(s_cb[g][q + u]) + (ent & 0x7FFFu), vr[g], vi[g]);
              #pragma unroll
              for (int g = 0; g < G; ++g) { ar[g] += c * vr[g]; if (T::cplx) ai[g] += c * vi[g]; }
            }
          }
          tw = twn;
        }
      }
      // low bonds: summed per coefficient class
      uint32_t left = wr.y & 0xFFu;
      int cls = 0;
      R sr[G], si[G];
      #pragma unroll
      for (int g = 0; g < G; ++g) { sr[g] = R(0); si[g] = R(0); }
      for (uint32_t j = 0; j < nt; ++j) {
        while (left == 0) {  // uniform over the warp: the next class
          const R lc = s_lc[cls];
          #pragma unroll
          for (int g = 0; g < G; ++g) {
            ar[g] += lc * sr[g];
            if (T::cplx) ai[g] += lc * si[g];
            sr[g] = R(0);
            si[g] = R(0);
          }
          ++cls;
          left = (wr.y >> (8 * cls)) & 0xFFu;
        }
        --left;
        const uint2 q = __ldg(wg + j * 32);
        const uint32_t t4[4] = {q.x & 0xFFFFu, q.x >> 16, q.y & 0xFFFFu, q.y >> 16};
        #pragma unroll
        for (int u = 0; u < 4; ++u)
          #pragma unroll
          for (int pl = 0; pl < PL; ++pl) {
            const Pack v = sx[pl * stride + t4[u]];
            #pragma unroll
            for (int w = 0; w < EPP; ++w)
              if (pl * EPP + w < G) {
                R vr, vi;
                sld(v.v, w, vr, vi);
                sr[pl * EPP + w] += vr;
                if (T::cplx) si[pl * EPP + w] += vi;
              }
          }
      }
      if (nt) {
        const R lc = s_lc[cls];
        #pragma unroll
        for (int g = 0; g < G; ++g) { ar[g] += lc * sr[g]; if (T::cplx) ai[g] += lc * si[g]; }
      }
      #pragma unroll
      for (int pl = 0; pl < PL; ++pl) {
        const Pack v = sx[pl * stride + l];
        #pragma unroll
        for (int w = 0; w < EPP; ++w) {
          const int g = pl * EPP + w;
          if (g < G) {
            R x0r, x0i;
            sld(v.v, w, x0r, x0i);
            const R d = GEN ? R(__ldg(p.diag_full + base[g] + l)) : R(rec.dh[g]) + R(dt);
            ar[g] += d * x0r;
            if (T::cplx) ai[g] += d * x0i;
            if (act[g]) {
              T::st_cs(y, uint64_t(base[g]) + l, ar[g], ai[g]);
              if (DOT) {
                dr += double(x0r) * double(ar[g]) + double(x0i) * double(ai[g]);
                di += double(x0r) * double(ai[g]) - double(x0i) * double(ar[g]);
              }
            }
          }
        }
      }
    }
    if (DOT) {
      dr = warp_sum(dr);
      di = warp_sum(di);
      if (lane == 0) { s_dot[2 * (tid >> 5)] = dr; s_dot[2 * (tid >> 5) + 1] = di; }
      dr = 0.0;
      di = 0.0;
    }
    if (tid < kRecWords) s_rec[b ^ 1][tid] = nword;
    if (tid == 0) s_pos[b] = npos;
    prev = item;
    item = next;
    __syncthreads();  // this item is finished; the next record and number are in place
    next = s_pos[b];
  }
  if (DOT && prev < p.nitems && tid == 0) {
    double sr = 0.0, si = 0.0;
    for (int w = 0; w < NT / 32; ++w) { sr += s_dot[2 * w]; si += s_dot[2 * w + 1]; }
    partials[2 * size_t(prev)] = sr;
    partials[2 * size_t(prev) + 1] = si;
  }
  if (wq) wq_done(wq);
  if (DOT) grid_finish_items(partials, ticket, p.nitems, dot_out);
}

template <int DT, bool GEN, int G, int U, int NT, int MINC>
int launch(const GroupPlan& p, const void* x, void* y, cudaStream_t s, qk_workspace* w, double* dot_out, uint32_t* wq,
           uint32_t rlo, uint32_t rhi) {
  using E = typename VT<DT>::E;
  constexpr int EPP = 16 / int(sizeof(E)), PL = (G + EPP - 1) / EPP;
  const size_t smem = size_t(PL) * 16 * (p.zero_slot + 8);
  auto go = [&](auto k, unsigned cap, double* part, unsigned* tick) -> int {
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) {
      (void)cudaGetLastError();
      return QKD_EINVAL;
    }
    k<<<resident_grid(k, NT, smem, cap), NT, smem, s>>>(p, x, y, part, tick, dot_out, wq, rlo, rhi);
    QKD_LAUNCH_CHECK();
    return QKD_OK;
  };
  if (dot_out) return go(k_hx_group<DT, true, GEN, G, U, NT, MINC>, std::min(p.nitems, unsigned(kMaxG)), w->partials, w->ticket);
  return go(k_hx_group<DT, false, GEN, G, U, NT, MINC>, p.nitems, nullptr, nullptr);
}

}  // namespace

struct GroupHandle {
  GroupPlan plan[4];  // groups of 4, of 2 and single blocks; of 2 in the visiting order
  std::vector<void*> bufs;
};

void group_plan_destroy(GroupHandle* h) {
  if (!h) return;
  for (void* b : h->bufs) cudaFree(b);
  delete h;
}

// Number of every block's kind: blocks that share class, combo and crossing
// flags have the same one.
static std::vector<uint32_t> block_kinds(const std::vector<GroupBlock>& blocks, const std::vector<uint2>& bent,
                                         int ncross) {
  std::map<std::vector<uint32_t>, uint32_t> known;
  std::vector<uint32_t> kind, key;
  for (const GroupBlock& k : blocks) {
    key.clear();
    if (k.size) {
      key.assign({k.lst, k.combo});
      for (int q = 0; q < ncross; ++q) key.push_back(bent[k.ebeg + k.nh + q].y);
    }
    kind.push_back(known.emplace(key, uint32_t(known.size())).first->second);
  }
  return kind;
}

// Groups of at most G blocks of `blocks` (visiting order) of one kind.
static std::vector<GroupRec> make_groups(const std::vector<GroupBlock>& blocks, const std::vector<uint32_t>& kind,
                                         uint32_t G) {
  std::vector<GroupRec> out;
  constexpr uint32_t kNone = ~0u;
  std::vector<uint32_t> open(blocks.size(), kNone);  // per kind: its group being filled
  for (size_t i = 0; i < blocks.size(); ++i) {
    const GroupBlock& k = blocks[i];
    if (k.size == 0) continue;
    uint32_t& at = open[kind[i]];
    if (at == kNone || out[at].count == G) {
      GroupRec r{};
      r.size = k.size; r.lst = k.lst; r.tile0 = k.tile0; r.combo = k.combo;
      for (uint32_t g = 0; g < kGroupMax; ++g) { r.base[g] = k.base; r.ebeg[g] = k.ebeg + k.nh; r.nh[g] = 0; r.dh[g] = k.dh; }
      at = uint32_t(out.size());
      out.push_back(r);
    }
    GroupRec& r = out[at];
    const uint32_t g = r.count++;
    r.base[g] = k.base; r.ebeg[g] = k.ebeg; r.nh[g] = uint16_t(k.nh); r.dh[g] = k.dh;
  }
  return out;
}

// Largest groups first, dealt in turn to the two dies' halves, so that no large
// group is left for the end of the queue and SMs idle.  For vectors of up to the
// L2 caches' size (kL2Bytes), which do not need the visiting order's locality.
// us per apply, visiting order -> this: t-J N=20 (9.2 M rows) float32 173 -> 132,
// float64 266 -> 220, complex128 425 -> 425; Heisenberg N=25 float32 54.0 ->
// 49.7, float64 73.4 -> 68.7, N=26 float64 (83 MB) 145 -> 138, N=27 float32
// (80 MB) 179 -> 171, float64 (160 MB) 259.7 -> 260.6.  complex128 on exchange
// tables loses (N=25 126 -> 134) and keeps the visiting order.
constexpr uint64_t kL2Bytes = 126000000;
static void largest_first(std::vector<GroupRec>& rec) {
  std::stable_sort(rec.begin(), rec.end(), [](const GroupRec& a, const GroupRec& b) {
    return uint64_t(a.size) * a.count > uint64_t(b.size) * b.count;
  });
  std::vector<GroupRec> out;
  for (size_t k = 0; k < 2; ++k)
    for (size_t i = k; i < rec.size(); i += 2) out.push_back(rec[i]);
  rec.swap(out);
}

GroupHandle* group_plan_create(const GroupPlan& tables, const std::vector<GroupBlock>& blocks,
                               const std::vector<uint2>& bent, int n0, int n1, size_t* dev_bytes) {
  auto* h = new GroupHandle;
  const std::vector<uint32_t> kind = block_kinds(blocks, bent, tables.ncross);
  for (int i = 0; i < 4; ++i) {
    std::vector<GroupRec> rec = make_groups(blocks, kind, i == 3 ? 2u : 4u >> i);
    if (i < 2 && tables.dim * (i == 0 ? 4 : 8) <= kL2Bytes) largest_first(rec);  // float32; the 8-byte types
    GroupPlan& p = h->plan[i];
    p = tables;
    void* d = nullptr;
    if (rec.empty() || cudaMalloc(&d, rec.size() * sizeof(GroupRec)) != cudaSuccess ||
        cudaMemcpy(d, rec.data(), rec.size() * sizeof(GroupRec), cudaMemcpyHostToDevice) != cudaSuccess) {
      (void)cudaGetLastError();
      cudaFree(d);
      group_plan_destroy(h);
      return nullptr;
    }
    h->bufs.push_back(d);
    *dev_bytes += rec.size() * sizeof(GroupRec);
    p.rec = static_cast<const GroupRec*>(d);
    p.nitems = uint32_t(rec.size());
    uint64_t total = 0, acc = 0;
    for (const GroupRec& r : rec) total += uint64_t(r.size) * r.count;
    p.qsplit = 0;
    while (p.qsplit < p.nitems && acc * uint64_t(n0 + n1) < total * uint64_t(n0)) {
      acc += uint64_t(rec[p.qsplit].size) * rec[p.qsplit].count;
      ++p.qsplit;
    }
  }
  return h;
}

// QKD_EINVAL when the staged blocks do not fit shared memory or the dot
// partials the workspace: the one-block kernel then runs.
int group_apply(const GroupHandle* h, bool gen, qk_dtype t, const void* x, void* y, cudaStream_t s, qk_workspace* w,
                double* dot_out, uint32_t* wq, const double* diag_full, uint32_t row_lo, uint32_t row_hi) {
  if (!h || t < QK_C128 || t > QK_F32) return QKD_EINVAL;
  const size_t es = qk_dtype_size(t);
  const size_t rows = size_t(h->plan[0].zero_slot) + 8;
  // blocks per group: 16 bytes per position for float32 (4), two planes of
  // 16 bytes or one for the others (2); complex128 alone (1) where two staged
  // blocks would leave room for fewer than three CTAs (Heisenberg N=28: 1071
  // us with two, 922 with one)
  int gi = t == QK_F32 ? 0 : 1;
  if (t == QK_C128) gi = rows * 32 > 60 * 1024 ? 2 : gen ? 1 : 3;
  GroupPlan p = h->plan[gi];
  p.diag_full = diag_full;
  const size_t smem = std::max<size_t>(16, (gi == 3 ? 2u : 4u >> gi) * es) * rows;
  if (smem > 200 * 1024 || (dot_out && size_t(p.nitems) > size_t(kMaxK) * kMaxG)) return QKD_EINVAL;
  p.prefetch = p.dim * es > (size_t(48) << 20) ? 1u : 0u;
  const bool big = smem > 48 * 1024;
  // threads per CTA and CTAs per SM (registers): 256 x 4 or 5 for blocks whose
  // stage leaves room for them; above 48 KB 384 or 512 threads x 3 (t-J N=20
  // float64 512 x 2 302 us, 640 x 2 293, 512 x 3 278, 384 x 3 285, and
  // Heisenberg N=28 552, 568, 544, 531), float32 exchange tables 512 x 2
  // (Heisenberg N=28 345 us; 384 x 3 365)
#define QKD_GRP1(DT, GG, UU, MS, MSG, NTB, MB, NTBG, MBG)                                                     \
  {                                                                                                           \
    if (gen) return big ? launch<DT, true, GG, UU, NTBG, MBG>(p, x, y, s, w, dot_out, wq, row_lo, row_hi)     \
                        : launch<DT, true, GG, 2, 256, MSG>(p, x, y, s, w, dot_out, wq, row_lo, row_hi);      \
    return big ? launch<DT, false, GG, UU, NTB, MB>(p, x, y, s, w, dot_out, wq, row_lo, row_hi)               \
               : launch<DT, false, GG, 2, 256, MS>(p, x, y, s, w, dot_out, wq, row_lo, row_hi);               \
  }
  switch (t) {
    case QK_C128:
      if (gi != 2) QKD_GRP1(QK_C128, 2, 2, 4, 4, 512, 2, 512, 2)
      QKD_GRP1(QK_C128, 1, 1, 4, 4, 512, 3, 512, 3)
    case QK_C64: QKD_GRP1(QK_C64, 2, 2, 5, 5, 384, 3, 384, 3)
    case QK_F64: QKD_GRP1(QK_F64, 2, 2, 5, 5, 384, 3, 384, 3)
    case QK_F32: QKD_GRP1(QK_F32, 4, 2, 4, 5, 512, 2, 384, 3)
  }
#undef QKD_GRP1
  return QKD_EINVAL;
}

}  // namespace qkd
