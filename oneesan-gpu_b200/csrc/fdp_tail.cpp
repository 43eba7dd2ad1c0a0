// Host half of the fused row tail: the per-class item tables (fdp_tail.h).
#include "fdp_tail.h"

#include <algorithm>

namespace fdp {

namespace {

inline uint32_t sym(uint32_t w, int q) { return (w >> (2 * q)) & 3u; }
inline uint32_t put_sym(uint32_t w, int q, uint32_t v) { return (w & ~(3u << (2 * q))) | (v << (2 * q)); }
inline uint32_t put_pair(uint32_t w, int p, uint32_t a, uint32_t b) { return put_sym(put_sym(w, p, a), p - 1, b); }

// Height above position p of a bottom word that starts at height g, and
// whether the path down to there stays at or above it.
int height_above(uint32_t w, int s, int p, int g, bool *is_min) {
  int h = g, low = g;
  for (int q = s - 1; q > p; --q) {
    h += sym(w, q) == SYM_L ? 1 : (sym(w, q) == SYM_R ? -1 : 0);
    low = std::min(low, h);
  }
  *is_min = low == h;
  return h;
}

uint32_t at(const std::vector<uint32_t> &words, uint32_t w) {
  return uint32_t(std::lower_bound(words.begin(), words.end(), w) - words.begin());
}

// An item's words: NN and LR, or own and other, then the blocked word and (N
// items: RL, at most (s - 2) / 2 + 1 closures and the escape sum) its sources.
struct Item {
  uint32_t own, other, blk;
  std::vector<uint16_t> src;
};

// Shared memory serves 16-byte accesses eight threads at a time, and two threads
// share an item's 32-byte words: the four items of an aligned group conflict
// unless their like operands lie in different quarters of the banks (word
// number mod 4).  Within items [i, e), which may run in any order, choose the
// order so that they do as far as a look ahead allows.
void spread_banks(std::vector<Item> &items, size_t i, size_t e) {
  const size_t kLook = 512;
  std::vector<uint32_t> used(3 + 8);
  for (; i < e; ++i) {
    if (i % 4 == 0) std::fill(used.begin(), used.end(), 0u);
    size_t best = i;
    int least = 1 << 30;
    auto bit = [](uint32_t w) { return 1u << (w % 4); };
    for (size_t k = i; k < e && k < i + kLook && least > 0; ++k) {
      const Item &it = items[k];
      // own and blk are read and written, other is read (and written at N items).
      int cost = 2 * !!(used[0] & bit(it.own)) + 2 * !!(used[1] & bit(it.other)) + 2 * !!(used[2] & bit(it.blk));
      for (size_t q = 0; q < it.src.size() && q < 8; ++q) cost += !!(used[3 + q] & bit(it.src[q]));
      if (cost < least) {
        least = cost;
        best = k;
      }
    }
    std::rotate(items.begin() + long(i), items.begin() + long(best), items.begin() + long(best) + 1);
    const Item &it = items[i];
    used[0] |= bit(it.own);
    used[1] |= bit(it.other);
    used[2] |= bit(it.blk);
    for (size_t q = 0; q < it.src.size() && q < 8; ++q) used[3 + q] |= bit(it.src[q]);
  }
}

}  // namespace

std::vector<uint32_t> tail_words(int s, int g) {
  std::vector<uint32_t> w{0};
  std::vector<int> h{g};
  for (int left = s - 1; left >= 0; --left) {
    std::vector<uint32_t> nw;
    std::vector<int> nh;
    for (size_t i = 0; i < w.size(); ++i)
      for (uint32_t c = 0; c < 3; ++c) {
        const int x = h[i] + (c == SYM_L ? 1 : (c == SYM_R ? -1 : 0));
        if (x < 0 || x > left) continue;
        nw.push_back(w[i] << 2 | c);
        nh.push_back(x);
      }
    w.swap(nw);
    h.swap(nh);
  }
  if (s == 0 && g != 0) w.clear();
  return w;  // built in lexicographic, so numeric, order
}

static TailTables build_tables(int s, bool whole) {
  TailTables t;
  t.s = s;
  t.cls.resize(size_t(s) + 1);
  std::vector<std::vector<uint32_t>> mw, bw;
  for (int g = 0; g <= s; ++g) {
    mw.push_back(tail_words(s, g));
    bw.push_back(tail_words(s - 1, g));
  }
  // Escape words each class writes: by cell, bottoms with pair RR whose path
  // stays at or above the height h' >= 2 above the pair.
  std::vector<std::vector<std::vector<uint32_t>>> esc(size_t(s) + 1, std::vector<std::vector<uint32_t>>(size_t(s)));
  for (int g = 0; g <= s; ++g) {
    if (whole && g != 1) continue;
    TailClass &c = t.cls[size_t(g)];
    c = TailClass{};
    c.nmain = uint32_t(mw[size_t(g)].size());
    c.nblk = uint32_t(bw[size_t(g)].size());
    for (int p = s - 1; p >= 1 && !whole; --p) {
      auto &e = esc[size_t(g)][size_t(p)];
      TailCell &cell = c.cell[p];
      cell.o0 = uint32_t(t.out.size());
      for (size_t i = 0; i < mw[size_t(g)].size(); ++i) {
        const uint32_t w = mw[size_t(g)][i];
        bool low;
        if (sym(w, p) != SYM_R || sym(w, p - 1) != SYM_R) continue;
        const int h = height_above(w, s, p, g, &low);
        if (!low || h < 2) continue;
        e.push_back(w);
        t.out.push_back(uint16_t(i));
      }
      cell.no = uint32_t(e.size());
      c.nout += cell.no;
    }
  }
  for (int g = 0; g <= s; ++g) {
    if (whole && g != 1) continue;
    TailClass &c = t.cls[size_t(g)];
    const auto &W = mw[size_t(g)], &B = bw[size_t(g)];
    const uint32_t zero = c.nmain;
    c.nin = g + 2 <= s ? t.cls[size_t(g) + 2].nout : 0;
    c.words = c.nmain + 1 + c.nblk + c.nin;
    c.h0 = uint32_t(t.slot_h.size());
    uint32_t slot0 = 0;  // first slot of the cell
    for (int p = s - 1; p >= 1; --p) {
      static const std::vector<uint32_t> none;
      const auto &in = g + 2 <= s ? esc[size_t(g) + 2][size_t(p)] : none;
      std::vector<uint32_t> slot_height(in.size(), 0);
      TailCell &cell = c.cell[p];
      cell.i0 = uint32_t(t.item.size() / 4);
      std::vector<Item> items, xs;
      for (size_t j = 0; j < B.size(); ++j) {
        // The main word of blocked word j with N at p.
        const uint32_t lowmask = (1u << (2 * p)) - 1u;
        const uint32_t u = (B[j] & lowmask) | ((B[j] & ~lowmask) << 2);
        const uint32_t centre = sym(u, p - 1);
        const uint32_t blk = c.nmain + 1 + uint32_t(j);
        if (centre != SYM_N) {
          const uint32_t own = at(W, u), other = at(W, put_pair(u, p, centre, SYM_N));
          xs.push_back(Item{own, other, blk, {}});
          continue;
        }
        Item it;
        it.own = at(W, u);
        it.other = at(W, put_pair(u, p, SYM_L, SYM_R));
        it.blk = blk;
        bool low;
        const int h = height_above(u, s, p, g, &low);
        if (p >= 2 && h > 0) it.src.push_back(uint16_t(at(W, put_pair(u, p, SYM_R, SYM_L))));
        int depth = 1;
        if (p >= 2)
          for (int q = p - 2; q >= 0 && depth > 0; --q) {  // LL: a depth-1 L below, as R
            if (sym(u, q) == SYM_L) {
              if (depth == 1) it.src.push_back(uint16_t(at(W, put_sym(put_pair(u, p, SYM_L, SYM_L), q, SYM_R))));
              ++depth;
            } else if (sym(u, q) == SYM_R) {
              --depth;
            }
          }
        depth = 1;
        for (int q = p + 1; q < s && depth > 0; ++q) {  // RR: a depth-1 R above, as L
          if (sym(u, q) == SYM_R) {
            if (depth == 1) it.src.push_back(uint16_t(at(W, put_sym(put_pair(u, p, SYM_R, SYM_R), q, SYM_L))));
            ++depth;
          } else if (sym(u, q) == SYM_L) {
            --depth;
          }
        }
        if (low && !in.empty()) {
          const uint32_t src = put_pair(u, p, SYM_R, SYM_R);
          const uint32_t e = at(in, src);
          if (e < in.size() && in[e] == src) {
            it.src.push_back(uint16_t(c.nmain + 1 + c.nblk + slot0 + e));
            slot_height[e] = uint32_t(h);
          }
        }
        items.push_back(it);
      }
      // Items with like numbers of sources together, so that a warp's lanes agree.
      std::stable_sort(items.begin(), items.end(), [](const Item &a, const Item &b) { return a.src.size() < b.src.size(); });
      cell.nn = uint32_t(items.size());
      cell.nx = uint32_t(xs.size());
      items.insert(items.end(), xs.begin(), xs.end());
      for (size_t i = 0, e; i < items.size() && !whole; i = e) {
        for (e = i + 1; e < items.size() && items[e].src.size() == items[i].src.size() && (e < cell.nn) == (i < cell.nn);) ++e;
        spread_banks(items, i, e);
      }
      for (size_t i = 0; i < items.size(); ++i) {
        Item &it = items[i];
        if (i >= cell.nn) {
          t.item.insert(t.item.end(), {it.own | it.other << 16, it.blk, 0u, 0u});
          t.more.insert(t.more.end(), {0u, 0u});
          continue;
        }
        const uint32_t count = uint32_t(it.src.size());
        it.src.resize(8, uint16_t(zero));
        auto two = [&](int k) { return uint32_t(it.src[size_t(k)]) | uint32_t(it.src[size_t(k) + 1]) << 16; };
        t.item.insert(t.item.end(), {it.own | it.other << 16, it.blk | count << 16, two(0), two(2)});
        t.more.insert(t.more.end(), {two(4), two(6)});
      }
      for (uint32_t h : slot_height) t.slot_h.push_back(uint8_t(h));
      slot0 += uint32_t(in.size());
    }
  }
  return t;
}

TailTables build_tail_tables(int s) { return build_tables(s, false); }
TailTables build_whole_tables(int W) { return build_tables(W, true); }

const TopCounts &top_counts(int g) {
  static const std::vector<TopCounts> all = [] {
    std::vector<TopCounts> v;
    for (int k = 0; k < FDP_TAIL_MAX_G + 2; ++k) {
      TopCounts c{};
      c.P[0][k] = 1;
      for (int l = 1; l <= FDP_TAIL_MAX_T; ++l)
        for (int h = 0; h < FDP_TAIL_HT; ++h)
          c.P[l][h] = c.P[l - 1][h] + (h > 0 ? c.P[l - 1][h - 1] : 0u) + (h + 1 < FDP_TAIL_HT ? c.P[l - 1][h + 1] : 0u);
      v.push_back(c);
    }
    return v;
  }();
  return all[size_t(g)];
}

}  // namespace fdp
