// Fused tail of a row sweep: cells p = s-1 .. 1 in one pass over the state.
//
// Split a main word into its top part T (positions W-1..s, ending at height g)
// and its bottom (positions s-1..0).  In canonical order the H[s][g] words of
// one T are contiguous, and so are the H[s-1][g] blocked words that start with
// the same symbols.  A cell p < s changes symbols at p, p-1 and, in a closure,
// one more symbol at depth 1 below p-1 (LL) or above p (RR).  So a T's block
// is closed under cells s-1..1 except for the RR closures whose flipped R lies
// in T: those read a word of another block T', T with one R turned into L.
// T' ends at height g + 2, so blocks are processed from the highest g down,
// and a block leaves the values its lower neighbours will read (its words with
// pair RR at (p, p-1), taken when cell p runs) in an escape array.
//
// Everything inside a block depends on (s, g) alone: the tables below list, for
// each cell, which local words an item reads and writes.  They are small enough
// to stay in cache, so the kernel decodes no ranks.
//
// Escape slots.  The RR word of T' is read by T exactly when the symbols
// between the flipped R and p keep the height at or above the height h just
// above p, which splits into a condition on T (fdp_tail_cand) and one on the
// bottom: the path from g down to p stays at or above its end h.  Target and
// source bottoms carry the same symbols apart from the pair (NN and RR), so
// slot e of the words that class g reads is slot e of those class g + 2 writes.
#pragma once
#include <stdint.h>

#include <vector>

#include "fdp_core.cuh"

#define FDP_TAIL_MAX_S 12   // widest bottom part
#define FDP_TAIL_MAX_G 13   // end heights 0..12
#define FDP_TAIL_MAX_T 20   // longest top part
#define FDP_TAIL_HT 24      // heights of the top part's count tables

namespace fdp {

// One cell of one class: item[i0 ..], the nn N items before the nx X items.
// N items (centre N), {NN | LR << 16, blocked | sources << 16, s0 | s1 << 16,
// s2 | s3 << 16} and sources 4.. in more[i] = {s4 | s5 << 16, s6 | s7 << 16}:
// LR' = LR + NN, NN' = NN + blocked, blocked' = sum of the sources (at p = 1 the
// sum goes to NN'): the RL word, the closures and the escape sum.  Unused
// sources are the zero word (local index nmain).  X items (centre R or L), {own |
// other << 16, blocked, 0, 0}: own' = own + other + blocked, blocked' = own (at
// p = 1 other' = other + own instead).
struct TailCell {
  uint32_t i0, nn, nx;
  uint32_t o0, no;  // local words written to the escape array, in slot order
};

// The block of one end height g.  Local words: nmain main words, a word that
// stays zero, nblk blocked words, nin escape sums.
struct TailClass {
  uint32_t nmain, nblk, nin, nout;
  uint32_t h0;      // slot_h[h0 + e]: height h of escape slot e it reads
  uint32_t words;   // nmain + 1 + nblk + nin
  TailCell cell[FDP_TAIL_MAX_S];  // by p, 1..s-1
};

struct TailTables {
  int s = 0;  // (build_whole_tables fills cls[1] alone)
  std::vector<TailClass> cls;  // by g, 0..s
  std::vector<uint32_t> item;  // four words each
  std::vector<uint32_t> more;  // two words for each item
  std::vector<uint16_t> out;   // escape words
  std::vector<uint8_t> slot_h;
};

// Tables for bottom parts of s symbols, every end height 0..s (2 <= s <= 12).
TailTables build_tail_tables(int s);

// The whole space of a width W <= 12 as one block (end height 1, no top part and
// so no escapes), items in canonical order within like numbers of sources.
TailTables build_whole_tables(int W);

// Local code of bottom word `i` of class g: two bits a symbol, canonical order.
std::vector<uint32_t> tail_words(int s, int g);

// P[len][h]: words of len symbols from height h to height g.
struct TopCounts {
  uint32_t P[FDP_TAIL_MAX_T + 1][FDP_TAIL_HT];
};
const TopCounts &top_counts(int g);  // 0 <= g < FDP_TAIL_MAX_G + 2

// Top word number r of the tl-symbol words from height 1 to the height P leads
// to: its symbols, the first one in the highest bits.
template <typename PT>
FDP_HD uint64_t fdp_tail_unrank(uint32_t r, int tl, const PT &P) {
  uint64_t sym = 0;
  int h = 1;
  for (int i = 0; i < tl; ++i) {
    const int rem = tl - 1 - i;
    const uint32_t zN = P[rem][h], below = P[rem][h > 0 ? h - 1 : 0], zR = zN + (h > 0 ? below : 0u);
    const bool ge1 = r >= zN, ge2 = r >= zR;
    r -= ge2 ? zR : (ge1 ? zN : 0u);
    sym = (sym << 2) | (ge2 ? SYM_L : (ge1 ? SYM_R : SYM_N));
    h += ge2 ? 1 : (ge1 ? -1 : 0);
  }
  return sym;
}

FDP_HD int fdp_popc64(uint64_t v) {
#if defined(__CUDA_ARCH__)
  return __popcll(v);
#else
  return __builtin_popcountll(v);
#endif
}

// What symbol i of top word `sym` adds to the main and blocked ranks of the
// word's block (H: the full space's counts; symbol i is at main position
// W-1-i, blocked position W-2-i).
template <typename Idx, typename HT>
FDP_HD void fdp_tail_base(uint64_t sym, int tl, int W, int i, const HT &H, Idx &bm, Idx &bb) {
  bm = bb = 0;
  if (i >= tl) return;
  const uint64_t above = i ? sym >> (2 * (tl - i)) : 0;  // symbols before i
  const int h = 1 + fdp_popc64((above >> 1) & 0x5555555555555555ull) - fdp_popc64(above & 0x5555555555555555ull);
  const uint32_t s = uint32_t(sym >> (2 * (tl - 1 - i))) & 3u;
  if (s == SYM_N) return;
  const int q = W - 1 - i;
  bm = H[q][h];
  bb = H[q - 1][h];
  if (s == SYM_L && h > 0) {
    bm += H[q][h - 1];
    bb += H[q - 1][h - 1];
  }
}

// Whether the symbol i of top word `sym` is an R whose flip to L gives a block
// that the word's block reads from; if so the height h of the escape slots it
// serves and the number of the flipped word among those that end two higher
// (P2: their counts).
template <typename PT>
FDP_HD bool fdp_tail_cand(uint64_t sym, int tl, int i, const PT &P2, int &hc, uint32_t &rank) {
  int h = 1;
  uint32_t r = 0;
  bool ok = i < tl;
  hc = 0;
  for (int j = 0; j < tl; ++j) {
    const int rem = tl - 1 - j;
    uint32_t s = uint32_t(sym >> (2 * rem)) & 3u;
    const int hs = j > i ? h + 2 : h;  // the flipped word's height
    if (j == i) {
      if (s != SYM_R) ok = false;
      hc = h - 1;
    }
    const uint32_t s2 = j == i ? uint32_t(SYM_L) : s;
    if (s2 != SYM_N) {
      r += P2[rem][hs];
      if (s2 == SYM_L && hs > 0) r += P2[rem][hs - 1];
    }
    h += s == SYM_L ? 1 : (s == SYM_R ? -1 : 0);
    if (j > i && h < hc) ok = false;
  }
  rank = r;
  return ok;
}

}  // namespace fdp
