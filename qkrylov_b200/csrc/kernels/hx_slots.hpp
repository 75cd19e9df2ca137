// Slot tables for gathers of 16-byte packs staged in shared memory.
//
// A warp loads a pack per row and slot; the hardware serves eight lanes (a
// quarter warp) per wavefront when their packs lie in eight different 16-byte
// bank groups.  The order of a row's entries is free, so the entries of the
// eight rows are spread over slots that repeat neither a row nor a bank group:
// an edge colouring of the bipartite multigraph of rows and bank groups, which
// needs no more slots than the fullest row or bank group has entries.  Rows
// without an entry in a slot read that one of eight zero packs whose bank group
// is still free, so every slot takes four wavefronts, the least it can.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#include <vector_types.h>

namespace qkd {

// Entries of 32 rows, each a 16-bit word whose low 15 bits (MASK) are the
// pack's index.
class SlotTile {
 public:
  explicit SlotTile(uint32_t mask) : mask_(mask) {}

  void add(uint32_t lane, uint32_t word) {
    Quarter& q = q_[lane / 8];
    const int r = int(lane & 7u), b = int(word & mask_ & 7u);
    q.row.push_back(uint8_t(r));
    q.word.push_back(word);
    need_ = std::max({need_, ++q.in_row[r], ++q.in_bank[b]});
  }

  // groups of four slots
  uint32_t groups() const { return uint32_t(need_ + 3) / 4; }

  // Appends ng >= groups() groups to `out`, [group][lane], two words per
  // component; zero: index of the first of the eight zero packs.
  void write(uint32_t ng, uint32_t zero, std::vector<uint2>& out) const {
    std::vector<uint32_t> t(size_t(ng) * 4 * 32, kNone);  // [slot][lane]
    for (uint32_t ph = 0; ph < 4; ++ph) {
      const Quarter& q = q_[ph];
      const std::vector<int> s = colours(q, int(ng) * 4);
      for (size_t k = 0; k < s.size(); ++k) t[size_t(s[k]) * 32 + 8 * ph + q.row[k]] = q.word[k];
      for (uint32_t c = 0; c < ng * 4; ++c) {
        uint32_t* l = &t[size_t(c) * 32 + 8 * ph];
        uint32_t banks = 0, z = 0;
        for (int i = 0; i < 8; ++i)
          if (l[i] != kNone) banks |= 1u << (l[i] & mask_ & 7u);
        for (int i = 0; i < 8; ++i)
          if (l[i] == kNone) {
            while (banks >> ((zero + z) & 7u) & 1u) ++z;
            l[i] = zero + z++;
          }
      }
    }
    for (uint32_t g = 0; g < ng; ++g)
      for (uint32_t i = 0; i < 32; ++i) {
        const uint32_t* u = &t[size_t(g) * 128 + i];
        uint2 w;
        w.x = u[0] | (u[32] << 16);
        w.y = u[64] | (u[96] << 16);
        out.push_back(w);
      }
  }

 private:
  static constexpr uint32_t kNone = ~0u;
  struct Quarter {
    std::vector<uint8_t> row;
    std::vector<uint32_t> word;
    int in_row[8] = {}, in_bank[8] = {};
  };

  // An entry without a colour free at both its row and its bank swaps the two
  // free ones along the alternating path from the bank; in a bipartite graph
  // that path does not reach the row.
  std::vector<int> colours(const Quarter& q, int ncol) const {
    const size_t n = q.row.size(), nw = (size_t(ncol) + 63) / 64;
    std::vector<int> slot(n, -1), at(size_t(16) * ncol, -1);
    std::vector<uint64_t> open(16 * nw, ~0ull);  // colours free at each row, then at each bank group
    if (ncol % 64)
      for (size_t v = 0; v < 16; ++v) open[v * nw + nw - 1] = (1ull << (ncol % 64)) - 1;
    auto row = [&](size_t e) { return size_t(q.row[e]); };
    auto bank = [&](size_t e) { return size_t(8 + (q.word[e] & mask_ & 7u)); };
    auto put = [&](size_t v, int c, int e) {
      at[v * ncol + c] = e;
      const uint64_t bit = 1ull << (c & 63);
      uint64_t& w = open[v * nw + size_t(c) / 64];
      w = e < 0 ? w | bit : w & ~bit;
    };
    auto first = [&](size_t u, size_t v) {  // lowest colour free at both, -1: none
      for (size_t w = 0; w < nw; ++w)
        if (const uint64_t m = open[u * nw + w] & open[v * nw + w]) return int(w * 64) + __builtin_ctzll(m);
      return -1;
    };
    for (size_t k = 0; k < n; ++k) {
      const size_t r = row(k), b = bank(k);
      int c = first(r, b);
      if (c < 0) {
        const int fr = first(r, r), fb = first(b, b);
        std::vector<int> path;
        int a = fr;
        for (int e = at[b * ncol + a]; e >= 0;) {
          path.push_back(e);
          a = a == fr ? fb : fr;
          e = at[((path.size() & 1) ? row(e) : bank(e)) * ncol + a];
        }
        for (int e : path) { put(row(e), slot[e], -1); put(bank(e), slot[e], -1); }
        for (int e : path) {
          slot[e] = slot[e] == fr ? fb : fr;
          put(row(e), slot[e], e);
          put(bank(e), slot[e], e);
        }
        c = fr;
      }
      slot[k] = c;
      put(r, c, int(k));
      put(b, c, int(k));
    }
    return slot;
  }

  uint32_t mask_;
  Quarter q_[4];
  int need_ = 0;
};

}  // namespace qkd
