// Host check of the fused row tail (fdp_tail.h): the block tables, the top-word
// walk and the escape slots, run block by block from the highest end height
// down as the kernel does, against the oracle's cells s-1 .. 1.
// Test infrastructure: built and run by tests/test_host_kernel_logic.py.
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "fdp_host.h"
#include "fdp_tail.h"

extern "C" int oracle_forward_cell(int, int, uint32_t, const uint32_t *, const uint32_t *, uint32_t *, uint32_t *);

using namespace fdp;

static int run(int W, int s, uint32_t mod, uint64_t seed) {
  const TailTables t = build_tail_tables(s);
  const int tl = W - s;
  const uint64_t M = main_states(W), D = blocked_states(W);
  std::mt19937_64 rng(seed);
  std::vector<uint32_t> main(M), blk(D);
  for (auto &v : main) v = uint32_t(rng() % mod);
  for (auto &v : blk) v = uint32_t(rng() % mod);
  std::vector<uint32_t> wm = main, wb = blk;
  for (int p = s - 1; p >= 1; --p) {
    std::vector<uint32_t> a(M), b(D);
    oracle_forward_cell(W, p, mod, wm.data(), wb.data(), a.data(), b.data());
    wm.swap(a);
    wb.swap(b);
  }
  const CountTable &H = counts();
  int bad = 0;
  std::vector<std::vector<uint32_t>> esc(size_t(s) + 3);
  std::vector<uint8_t> seen(M, 0);
  for (int g = s; g >= 0; --g) {
    const TailClass &c = t.cls[size_t(g)];
    const TopCounts &P = top_counts(g), &P2 = top_counts(g + 2);
    const uint32_t nT = P.P[tl][1];
    esc[size_t(g)].assign(size_t(nT) * c.nout, 0);
    for (uint32_t r = 0; r < nT; ++r) {
      uint64_t bm = 0, bb = 0;
      const uint64_t sym = fdp_tail_unrank(r, tl, P.P);
      for (int i = 0; i < tl; ++i) {
        uint64_t m, b;
        fdp_tail_base<uint64_t>(sym, tl, W, i, H.H, m, b);
        bm += m;
        bb += b;
      }
      if (bm + c.nmain > M || bb + c.nblk > D) { ++bad; continue; }
      std::vector<uint32_t> x(c.words, 0);
      for (uint32_t i = 0; i < c.nmain; ++i) { x[i] = main[bm + i]; seen[bm + i]++; }
      for (uint32_t i = 0; i < c.nblk; ++i) x[c.nmain + 1 + i] = blk[bb + i];
      for (int i = 0; i < tl; ++i) {
        int h;
        uint32_t r2;
        if (!fdp_tail_cand(sym, tl, i, P2.P, h, r2)) continue;
        for (uint32_t e = 0; e < c.nin; ++e)
          if (t.slot_h[c.h0 + e] == h) {
            uint32_t &v = x[c.nmain + 1 + c.nblk + e];
            v = add_mod(v, esc[size_t(g) + 2].at(size_t(r2) * c.nin + e), mod);
          }
      }
      uint32_t o = 0;
      for (int p = s - 1; p >= 1; --p) {
        const TailCell &q = c.cell[p];
        for (uint32_t e = 0; e < q.no; ++e) esc[size_t(g)][size_t(r) * c.nout + o++] = x[t.out[q.o0 + e]];
        for (uint32_t i = q.i0 + q.nn; i < q.i0 + q.nn + q.nx; ++i) {
          const uint32_t own = t.item[4 * i] & 0xffff, oth = t.item[4 * i] >> 16, b = t.item[4 * i + 1];
          const uint32_t vo = x[own], vx = x[oth];
          x[own] = add_mod(add_mod(vo, vx, mod), x[b], mod);
          if (p >= 2) x[b] = vo;
          else { x[oth] = add_mod(vx, vo, mod); x[b] = 0; }
        }
        for (uint32_t i = q.i0; i < q.i0 + q.nn; ++i) {
          const uint32_t *n = &t.item[4 * size_t(i)];
          const uint32_t nn = n[0] & 0xffff, lr = n[0] >> 16, b = n[1] & 0xffff, count = n[1] >> 16;
          const uint32_t src[8] = {n[2] & 0xffff, n[2] >> 16, n[3] & 0xffff, n[3] >> 16, t.more[2 * i] & 0xffff,
                                   t.more[2 * i] >> 16, t.more[2 * i + 1] & 0xffff, t.more[2 * i + 1] >> 16};
          uint32_t acc = 0;
          if (count > 8) ++bad;
          for (uint32_t k = 0; k < 8; ++k) {
            if (k >= count && src[k] != c.nmain) ++bad;
            acc = add_mod(acc, x[src[k]], mod);
          }
          const uint32_t v = x[nn];
          x[lr] = add_mod(x[lr], v, mod);
          x[nn] = add_mod(v, x[b], mod);
          if (p >= 2) x[b] = acc;
          else { x[nn] = add_mod(x[nn], acc, mod); x[b] = 0; }
        }
        if (x[c.nmain]) ++bad;  // the zero word
      }
      for (uint32_t i = 0; i < c.nmain; ++i) main[bm + i] = x[i];
      for (uint32_t i = 0; i < c.nblk; ++i) blk[bb + i] = x[c.nmain + 1 + i];
    }
  }
  for (uint64_t i = 0; i < M; ++i) bad += main[i] != wm[i] || seen[i] != 1;
  for (uint64_t i = 0; i < D; ++i) bad += blk[i] != wb[i];
  if (bad) printf("tail W=%d s=%d mod=%u bad=%d\n", W, s, mod, bad);
  return bad;
}

int main(int argc, char **argv) {
  const int wmax = argc > 1 ? atoi(argv[1]) : 12;
  int bad = 0;
  for (int W = 2; W <= wmax; ++W)
    for (int s = 2; s <= W && s <= FDP_TAIL_MAX_S; ++s) {
      bad += run(W, s, 4294967291u, uint64_t(100 * W + s));
      bad += run(W, s, 2u, uint64_t(7 * W + s));
    }
  printf("bad=%d\n", bad);
  return bad != 0;
}
