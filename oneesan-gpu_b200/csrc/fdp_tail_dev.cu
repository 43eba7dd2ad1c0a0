// Fused row tail on the GPU: cells s-1..1 of a row in one pass over the state.
//
// A CTA holds one or more blocks of the same end height g (fdp_tail.h) in
// shared memory, eight columns at a time: the K lanes of a state's panel times
// 8 / PW blocks, so one table entry serves eight columns whatever the lane
// count.  A local word is 32 bytes (its eight columns) and two threads share an
// item, each on four columns.  The CTA loads the main and blocked words and the
// sums of the escape words its blocks read, runs the cells with one barrier
// each, and writes the main words back; the escape words of the blocks it is
// the source of go out as each cell reaches them.
//
// Launches run from the highest end height down, two heights at a time: a block
// of height g reads only escapes of height g + 2.
//
// Bound: instruction issue and latency at two CTAs per SM (46 % of issue slots,
// shared memory 37 %, DRAM 1.5 TB/s at n = 18, 8 lanes).  A block moves main
// twice, blocked once and 1.2 escape words a main word, 3.6 words for eight
// cells, where single cells move 2.2 words each and their low cells run at half
// the DRAM rate.  Eight low cells of a row, n = 20, before and after: one lane
// 14.3 -> 2.5 ms, 8 lanes 31 -> 20 ms.  Tried beside it: bottoms of 8 symbols
// (more CTAs per SM, one cell less: 8 lanes 768 -> 870 ms a pass), eight columns
// a thread (fewer instructions, 1.4 x the bank conflicts, equal time), 256 to 384
// threads (384 fastest by 2 %).
#include <algorithm>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <vector>

#include "fdp_host.h"
#include "fdp_tail.h"
#include "fdp_tail_dev.h"

namespace fdp {

namespace {

constexpr int kThreads = 384;
constexpr int kSegs = 10;                   // two heights x at most five panels
constexpr int kMaxBlocks = 16;              // blocks of a CTA
constexpr size_t kSmemBudget = 113 * 1024;  // two CTAs per SM
constexpr int kAhead = 3;                   // items a thread reads one cell ahead

// One (panel, end height) of a launch: CTAs [cta0, next segment's cta0).
struct TailSeg {
  uint32_t cta0, nT;
  int g, lane0, pw, groups;  // column groups per CTA
};

struct TailArgs {
  const uint4 *item;
  const uint2 *more;
  const uint16_t *out;
  const uint8_t *slot_h;
  const TopCounts *top;  // by end height
  const void *tables;    // WidthTables<Idx>
  uint32_t *main;
  const uint32_t *blk;
  uint32_t *esc;
  uint64_t M, D, E;      // words of one lane
  uint64_t ebase[FDP_TAIL_MAX_G + 3];  // first escape word of end height g
  uint32_t mod[16];
  int W, s, nsegs, top_g;
  TailSeg seg[kSegs];
  TailClass cls[2];      // end heights top_g, top_g - 1
};

// Shared-memory layout: the local words, then the per-block records.
template <typename Idx>
struct TailBlocks {
  Idx bm[kMaxBlocks], bb[kMaxBlocks];        // main and blocked rank of the block
  uint64_t sym[kMaxBlocks];
  uint32_t mask[kMaxBlocks][FDP_TAIL_MAX_G];  // flips that serve height h
  uint32_t num[kMaxBlocks][FDP_TAIL_MAX_T];  // flipped word's number, by flipped symbol
  TopCounts P, P2;
  Idx H[FDP_TAIL_MAX_T + 1][FDP_TAIL_HT];    // counts of main positions s-1 ..
};

// A thread works on one half of a local word, four of its eight columns.
struct V4 {
  uint32_t v[4];
};
__device__ __forceinline__ V4 lds4(const unsigned char *m, uint32_t i) {
  const uint4 a = *reinterpret_cast<const uint4 *>(m + i * 32u);
  return V4{{a.x, a.y, a.z, a.w}};
}
__device__ __forceinline__ void sts4(unsigned char *m, uint32_t i, const V4 &x) {
  *reinterpret_cast<uint4 *>(m + i * 32u) = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
}

// Sums modulo p with q = 2^32 - p.  A residue a < p plus any 32-bit
// representative b is a 32-bit representative again: on a carry out of a + b
// the sum is at most p - 2 and 2^32 = q (mod p) is added back without another
// carry.  With p above 2^31 (WIDE: every lane's modulus) a representative is
// below 2 p, so one conditional subtraction, min(x + q, x) in 32 bits, makes it
// a residue at the end of a chain of sums; smaller moduli do it at each sum.
template <bool WIDE>
__device__ __forceinline__ uint32_t add_rep(uint32_t a, uint32_t b, uint32_t q) {
  uint32_t s;
  asm("{\n\t.reg .u32 c;\n\t"
      "add.cc.u32 %0, %1, %2;\n\t"
      "addc.u32 c, 0, 0;\n\t"
      "mad.lo.u32 %0, c, %3, %0;\n\t}"
      : "=&r"(s)
      : "r"(a), "r"(b), "r"(q));
  return WIDE ? s : __viaddmin_u32(s, q, s);
}
__device__ __forceinline__ uint32_t residue(uint32_t x, uint32_t q) { return __viaddmin_u32(x, q, x); }

template <bool WIDE>
__device__ __forceinline__ V4 add_rep4(const V4 &a, const V4 &b, const uint32_t *q) {
  V4 r;
#pragma unroll
  for (int c = 0; c < 4; ++c) r.v[c] = add_rep<WIDE>(a.v[c], b.v[c], q[c]);
  return r;
}
__device__ __forceinline__ V4 residue4(const V4 &a, const uint32_t *q) {
  V4 r;
#pragma unroll
  for (int c = 0; c < 4; ++c) r.v[c] = residue(a.v[c], q[c]);
  return r;
}

// The four columns of a half in global memory: half a panel word (PW = 8), one
// word, or the words of two or four blocks.  at(b): word of the half's block b;
// the first `valid` blocks exist.
template <int PW, typename At>
__device__ __forceinline__ V4 gather4(const uint32_t *src, uint32_t valid, At at) {
  V4 r{};
  constexpr uint32_t N = PW >= 4 ? 1 : 4 / PW, L = 4 / N;
#pragma unroll
  for (uint32_t b = 0; b < N; ++b)
    if (b < valid) ld_panel<L>(src + at(b), r.v + b * L);
  return r;
}
template <int PW, typename At>
__device__ __forceinline__ void scatter4(uint32_t *dst, uint32_t valid, At at, const V4 &x) {
  constexpr uint32_t N = PW >= 4 ? 1 : 4 / PW, L = 4 / N;
#pragma unroll
  for (uint32_t b = 0; b < N; ++b)
    if (b < valid) st_panel<L>(dst + at(b), x.v + b * L);
}

__device__ __forceinline__ void async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(uint32_t(__cvta_generic_to_shared(dst))), "l"(src)
               : "memory");
}
__device__ __forceinline__ void async8(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(uint32_t(__cvta_generic_to_shared(dst))), "l"(src)
               : "memory");
}

// One N item on four columns (q: 2^32 - modulus).
template <bool WIDE>
__device__ __forceinline__ void tail_n(const TailArgs &a, unsigned char *m, const uint4 &it, uint32_t i, bool last,
                                       const uint32_t *q) {
  const uint32_t nn = it.x & 0xffffu, lr = it.x >> 16, bl = it.y & 0xffffu, count = it.y >> 16;
  V4 acc{};
  if (count > 0) acc = lds4(m, it.z & 0xffffu);
  if (count > 1) acc = add_rep4<WIDE>(lds4(m, it.z >> 16), acc, q);
  if (count > 2) {
    acc = add_rep4<WIDE>(lds4(m, it.w & 0xffffu), acc, q);
    if (count > 3) acc = add_rep4<WIDE>(lds4(m, it.w >> 16), acc, q);
    if (count > 4) {
      const uint2 e = a.more[i];
      acc = add_rep4<WIDE>(lds4(m, e.x & 0xffffu), acc, q);
      acc = add_rep4<WIDE>(lds4(m, e.x >> 16), acc, q);
      if (count > 6) {
        acc = add_rep4<WIDE>(lds4(m, e.y & 0xffffu), acc, q);
        acc = add_rep4<WIDE>(lds4(m, e.y >> 16), acc, q);
      }
    }
  }
  const V4 v = lds4(m, nn), vb = lds4(m, bl);
  sts4(m, lr, residue4(add_rep4<WIDE>(lds4(m, lr), v, q), q));
  if (!last) {
    sts4(m, nn, residue4(add_rep4<WIDE>(v, vb, q), q));
    sts4(m, bl, residue4(acc, q));
  } else {
    sts4(m, nn, residue4(add_rep4<WIDE>(v, add_rep4<WIDE>(vb, acc, q), q), q));
  }
}

template <bool WIDE>
__device__ __forceinline__ void tail_x(unsigned char *m, const uint4 &it, bool last, const uint32_t *q) {
  const uint32_t own = it.x & 0xffffu, oth = it.x >> 16, bl = it.y;
  const V4 vo = lds4(m, own), vx = lds4(m, oth), vb = lds4(m, bl);
  const V4 sum = add_rep4<WIDE>(vo, vx, q);
  sts4(m, own, residue4(add_rep4<WIDE>(vb, sum, q), q));
  if (!last) sts4(m, bl, vo);
  else sts4(m, oth, residue4(sum, q));
}

template <typename Idx, bool WIDE, int PW>
__device__ __forceinline__ void tail_body(const TailArgs &a, const TailSeg &sg, unsigned char *smem) {
  constexpr uint32_t BPG = 8 / PW;                // blocks of a column group
  constexpr uint32_t BPH = PW == 8 ? 1 : 4 / PW;  // blocks of a half (PW = 8: half of one)
  const TailClass &c = a.cls[a.top_g - sg.g];
  const uint32_t nmain = c.nmain, nblk = c.nblk, nin = c.nin, nout = c.nout;
  const uint32_t tid = threadIdx.x, nthr = blockDim.x;
  const uint32_t half = tid & 1, t2 = tid >> 1, n2 = nthr >> 1;  // this thread's half, its number among them
  const int tl = a.W - a.s;
  TailBlocks<Idx> &tb = *reinterpret_cast<TailBlocks<Idx> *>(smem);
  unsigned char *const cols = smem + ((sizeof(TailBlocks<Idx>) + 31) & ~size_t(31)) + half * 16;
  const uint32_t gstride = c.words * 32u;
  const uint32_t t0 = (blockIdx.x - sg.cta0) * uint32_t(sg.groups) * BPG;
  const uint32_t nb = min(uint32_t(sg.groups) * BPG, sg.nT - t0);
  const uint32_t groups = (nb + BPG - 1) / BPG;
  uint32_t q4[4];  // 2^32 - modulus of the four columns
#pragma unroll
  for (int l = 0; l < 4; ++l) q4[l] = 0u - a.mod[sg.lane0 + (PW == 8 ? int(half) * 4 + l : (l & (PW - 1)))];
  // The half's blocks in group grp: the first one, and how many exist.
  auto first_block = [&](uint32_t grp) { return PW == 8 ? grp : (grp * 2 + half) * BPH; };
  auto blocks_left = [&](uint32_t grp) {
    const uint32_t b0 = first_block(grp);
    return b0 < nb ? nb - b0 : 0u;
  };
  constexpr uint32_t SH = PW == 8 ? 4 : 0;  // lanes before the half within a panel word
  // Counts, then one warp per block: its symbols and its ranks.
  const WidthTables<Idx> *wt = reinterpret_cast<const WidthTables<Idx> *>(a.tables);
  for (uint32_t i = tid; i < uint32_t(tl + 1) * FDP_TAIL_HT; i += nthr) {
    const uint32_t l = i / FDP_TAIL_HT, h = i % FDP_TAIL_HT;
    tb.H[l][h] = wt->H[a.s - 1 + l][h];
    if (l < uint32_t(tl)) {
      tb.P.P[l][h] = a.top[sg.g].P[l][h];
      tb.P2.P[l][h] = a.top[sg.g + 2].P[l][h];
    }
  }
  for (uint32_t grp = t2; grp < groups; grp += n2) sts4(cols + grp * gstride, nmain, V4{});
  uint4 ahead[kAhead];
  uint32_t out_ahead = 0;
  auto read_ahead = [&](const TailCell &q) {
    const uint32_t n = q.nn + q.nx;
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const uint32_t u = t2 + uint32_t(k) * n2;
      if (u < n) ahead[k] = a.item[q.i0 + u];
    }
    if (t2 < q.no) out_ahead = a.out[q.o0 + t2];
  };
  __syncthreads();
  const uint32_t lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
  for (uint32_t b = warp; b < nb; b += nwarps) {
    const uint64_t sym = fdp_tail_unrank(t0 + b, tl, tb.P.P);
    Idx bm, bb;
    fdp_tail_base<Idx>(sym, tl, a.W, int(lane), tb.H - (a.s - 1), bm, bb);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      bm += __shfl_xor_sync(0xffffffffu, bm, o);
      bb += __shfl_xor_sync(0xffffffffu, bb, o);
    }
    if (lane == 0) {
      tb.bm[b] = bm;
      tb.bb[b] = bb;
      tb.sym[b] = sym;
    }
  }
  __syncthreads();
  uint32_t *const gmain = a.main + size_t(sg.lane0) * a.M + half * SH;
  const uint32_t *const gblk = a.blk + size_t(sg.lane0) * a.D + half * SH;
  uint32_t *const gesc = a.esc + size_t(sg.lane0) * a.E + half * SH;
  // Main and blocked words: local word i < nmain + nblk of every block, by
  // asynchronous copies where a panel word has at least 8 bytes.
  const uint32_t load = nmain + nblk;
  for (uint32_t grp = 0; grp < groups; ++grp) {
    unsigned char *const m = cols + grp * gstride;
    const uint32_t b0 = first_block(grp), valid = blocks_left(grp);
    if constexpr (PW >= 2) {
#pragma unroll
      for (uint32_t r = 0; r < BPH; ++r) {
        if (r >= valid) break;
        const uint32_t *const pm = gmain + size_t(tb.bm[b0 + r]) * PW, *const pb = gblk + size_t(tb.bb[b0 + r]) * PW;
        for (uint32_t i = t2; i < load; i += n2) {
          const bool blocked = i >= nmain;
          const uint32_t *src = blocked ? pb + size_t(i - nmain) * PW : pm + size_t(i) * PW;
          unsigned char *dst = m + (blocked ? i + 1 : i) * 32u + r * 8;
          if constexpr (PW >= 4) async16(dst, src);
          else async8(dst, src);
        }
      }
    } else {
      constexpr int B = 4;  // words in flight
      for (uint32_t i0 = t2; i0 < load; i0 += B * n2) {
        V4 x[B];
#pragma unroll
        for (int k = 0; k < B; ++k) {
          const uint32_t i = i0 + uint32_t(k) * n2;
          if (i < nmain)
            x[k] = gather4<PW>(gmain, valid, [&](uint32_t r) { return size_t(tb.bm[b0 + r]) + i; });
          else if (i < load)
            x[k] = gather4<PW>(gblk, valid, [&](uint32_t r) { return size_t(tb.bb[b0 + r]) + (i - nmain); });
        }
#pragma unroll
        for (int k = 0; k < B; ++k) {
          const uint32_t i = i0 + uint32_t(k) * n2;
          if (i < load) sts4(m, i < nmain ? i : i + 1, x[k]);
        }
      }
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  // Escape sums, while the copies run.
  if (nin) {
    for (uint32_t b = warp; b < nb; b += nwarps) {
      int h = 0;
      uint32_t num = 0;
      const bool ok = fdp_tail_cand(tb.sym[b], tl, int(lane), tb.P2.P, h, num);
      for (int q = 0; q <= sg.g; ++q) {
        const uint32_t m = __ballot_sync(0xffffffffu, ok && h == q);
        if (lane == 0) tb.mask[b][q] = m;
      }
      if (ok) tb.num[b][lane] = num;
    }
    __syncthreads();
    const uint32_t *const src = gesc + a.ebase[sg.g + 2] * PW;
    for (uint32_t grp = 0; grp < groups; ++grp) {
      const uint32_t b0 = first_block(grp), valid = blocks_left(grp);
      for (uint32_t e = t2; e < nin; e += n2) {
        const uint32_t h = a.slot_h[c.h0 + e];
        uint32_t mask[BPH], any = 0;
#pragma unroll
        for (uint32_t r = 0; r < BPH; ++r) {
          mask[r] = r < valid ? tb.mask[b0 + r][h] : 0u;
          any |= mask[r];
        }
        V4 x{};
        while (any) {  // two words of each block in flight
          V4 y{}, z{};
          any = 0;
          constexpr int L = 4 / BPH;
#pragma unroll
          for (uint32_t r = 0; r < BPH; ++r)
            if (mask[r]) {
              const uint32_t k = __ffs(int(mask[r])) - 1;
              mask[r] &= mask[r] - 1;
              ld_panel<L>(src + (uint64_t(tb.num[b0 + r][k]) * nin + e) * PW, y.v + r * L);
              if (mask[r]) {
                const uint32_t k2 = __ffs(int(mask[r])) - 1;
                mask[r] &= mask[r] - 1;
                any |= mask[r];
                ld_panel<L>(src + (uint64_t(tb.num[b0 + r][k2]) * nin + e) * PW, z.v + r * L);
              }
            }
          x = add_rep4<WIDE>(z, add_rep4<WIDE>(y, x, q4), q4);
        }
        sts4(cols + grp * gstride, nmain + 1 + nblk + e, residue4(x, q4));
      }
    }
  }
  read_ahead(c.cell[a.s - 1]);
  asm volatile("cp.async.wait_all;" ::: "memory");
  // The cells.  An item's table entry was read one cell earlier; escape words
  // are not changed by the cell that reads them out.
  uint32_t slot0 = 0;
  uint32_t *const dst = gesc + a.ebase[sg.g] * PW;
  for (int p = a.s - 1; p >= 1; --p) {
    const TailCell &q = c.cell[p];
    const uint32_t i0 = q.i0, nn = q.nn, n = q.nn + q.nx, o0 = q.o0, no = q.no;
    const bool last = p == 1;
    uint4 now[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) now[k] = ahead[k];
    const uint32_t out_now = out_ahead;
    if (!last) read_ahead(c.cell[p - 1]);
    __syncthreads();
    for (uint32_t grp = 0; grp < groups; ++grp) {
      unsigned char *const m = cols + grp * gstride;
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        const uint32_t u = t2 + uint32_t(k) * n2;
        if (u < nn) tail_n<WIDE>(a, m, now[k], i0 + u, last, q4);
        else if (u < n) tail_x<WIDE>(m, now[k], last, q4);
      }
      for (uint32_t u = t2 + kAhead * n2; u < n; u += n2) {
        const uint4 it = a.item[i0 + u];
        if (u < nn) tail_n<WIDE>(a, m, it, i0 + u, last, q4);
        else tail_x<WIDE>(m, it, last, q4);
      }
      const uint32_t b0 = first_block(grp), valid = blocks_left(grp);
      for (uint32_t e = t2; e < no; e += n2) {
        const uint32_t w = e == t2 ? out_now : uint32_t(a.out[o0 + e]);
        scatter4<PW>(dst, valid, [&](uint32_t r) { return (uint64_t(t0 + b0 + r) * nout + slot0 + e) * PW; }, lds4(m, w));
      }
    }
    slot0 += no;
  }
  __syncthreads();
  for (uint32_t grp = 0; grp < groups; ++grp) {
    const unsigned char *const m = cols + grp * gstride;
    const uint32_t b0 = first_block(grp), valid = blocks_left(grp);
    for (uint32_t i = t2; i < nmain; i += n2)
      scatter4<PW>(gmain, valid, [&](uint32_t r) { return (size_t(tb.bm[b0 + r]) + i) * PW; }, lds4(m, i));
  }
}

template <typename Idx, bool WIDE>
__global__ void __launch_bounds__(kThreads, 2) tail_kernel(const __grid_constant__ TailArgs a) {
  extern __shared__ __align__(32) unsigned char smem[];
  int k = 0;
  while (k + 1 < a.nsegs && blockIdx.x >= a.seg[k + 1].cta0) ++k;
  const TailSeg &sg = a.seg[k];
  switch (sg.pw) {
    case 8: tail_body<Idx, WIDE, 8>(a, sg, smem); break;
    case 4: tail_body<Idx, WIDE, 4>(a, sg, smem); break;
    case 2: tail_body<Idx, WIDE, 2>(a, sg, smem); break;
    default: tail_body<Idx, WIDE, 1>(a, sg, smem); break;
  }
}

// One lane of a whole solve, its state in shared memory: the first-row state,
// W - 2 rows of cells, the dot product with the first-row state.  One barrier a
// cell, no launch between cells.
// Bound: the latency of a cell (barrier, shared-memory round trips) up to n = 9,
// the item tables' L2 reads (16 bytes an item and cell) at n = 11.  Launching
// each cell costs 8 to 11 us: device time of a pass, n = 9, two lanes 688 -> 89 us,
// n = 10 849 -> 174 us.
struct WholeArgs {
  const uint4 *item;
  const uint2 *more;
  const uint16_t *first;  // local words of the 2^(W-1) first-row states
  uint32_t *residues;
  uint32_t mod[16];
  int W;
  TailClass cls;
};

constexpr int kWholeAhead = 4;

__global__ void __launch_bounds__(1024, 1) whole_kernel(const __grid_constant__ WholeArgs a) {
  extern __shared__ __align__(16) uint32_t w[];
  __shared__ unsigned long long part[32];
  const uint32_t tid = threadIdx.x, nthr = blockDim.x;
  const uint32_t p_ = a.mod[blockIdx.x], nfirst = 1u << (a.W - 1);
  const TailClass &c = a.cls;
  for (uint32_t i = tid; i < c.words; i += nthr) w[i] = 0;
  __syncthreads();
  for (uint32_t i = tid; i < nfirst; i += nthr) w[a.first[i]] = 1u;
  uint4 ahead[kWholeAhead];
  auto read_ahead = [&](const TailCell &q) {
    const uint32_t n = q.nn + q.nx;
#pragma unroll
    for (int k = 0; k < kWholeAhead; ++k) {
      const uint32_t u = tid + uint32_t(k) * nthr;
      if (u < n) ahead[k] = a.item[q.i0 + u];
    }
  };
  auto item_n = [&](const uint4 &it, uint32_t i, bool last) {
    const uint32_t nn = it.x & 0xffffu, lr = it.x >> 16, bl = it.y & 0xffffu, count = it.y >> 16;
    uint32_t acc = count > 0 ? w[it.z & 0xffffu] : 0u;
    if (count > 1) acc = add_mod(acc, w[it.z >> 16], p_);
    if (count > 2) {
      acc = add_mod(acc, w[it.w & 0xffffu], p_);
      acc = add_mod(acc, w[it.w >> 16], p_);  // the zero word past the last source
      if (count > 4) {
        const uint2 e = a.more[i];
        acc = add_mod(add_mod(acc, w[e.x & 0xffffu], p_), w[e.x >> 16], p_);
        acc = add_mod(add_mod(acc, w[e.y & 0xffffu], p_), w[e.y >> 16], p_);
      }
    }
    const uint32_t v = w[nn], vb = w[bl], vl = w[lr];
    w[lr] = add_mod(vl, v, p_);
    const uint32_t vn = add_mod(v, vb, p_);
    w[nn] = last ? add_mod(vn, acc, p_) : vn;
    w[bl] = last ? 0u : acc;
  };
  auto item_x = [&](const uint4 &it, bool last) {
    const uint32_t own = it.x & 0xffffu, oth = it.x >> 16, bl = it.y;
    const uint32_t vo = w[own], vx = w[oth], sum = add_mod(vo, vx, p_);
    w[own] = add_mod(sum, w[bl], p_);
    if (last) w[oth] = sum;
    w[bl] = last ? 0u : vo;  // the next row starts without blocked words
  };
  const int rows = a.W >= 3 ? a.W - 2 : 0;
  if (rows) read_ahead(c.cell[a.W - 1]);
  for (int row = 0; row < rows; ++row)
    for (int p = a.W - 1; p >= 1; --p) {
      const TailCell &q = c.cell[p];
      const uint32_t n = q.nn + q.nx;
      uint4 now[kWholeAhead];
#pragma unroll
      for (int k = 0; k < kWholeAhead; ++k) now[k] = ahead[k];
      read_ahead(c.cell[p > 1 ? p - 1 : a.W - 1]);
      __syncthreads();
#pragma unroll
      for (int k = 0; k < kWholeAhead; ++k) {
        const uint32_t u = tid + uint32_t(k) * nthr;
        if (u < q.nn) item_n(now[k], q.i0 + u, p == 1);
        else if (u < n) item_x(now[k], p == 1);
      }
#pragma unroll 4
      for (uint32_t u = tid + kWholeAhead * nthr; u < n; u += nthr) {
        const uint4 it = a.item[q.i0 + u];
        if (u < q.nn) item_n(it, q.i0 + u, p == 1);
        else item_x(it, p == 1);
      }
    }
  __syncthreads();
  unsigned long long acc = 0;
  for (uint32_t i = tid; i < nfirst; i += nthr) acc += w[a.first[i]];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((tid & 31) == 0) part[tid >> 5] = acc;
  __syncthreads();
  if (tid == 0) {
    for (uint32_t k = 1; k < nthr / 32; ++k) acc += part[k];
    a.residues[blockIdx.x] = uint32_t(acc % p_);
  }
}

template <typename Idx>
constexpr size_t blocks_bytes() { return (sizeof(TailBlocks<Idx>) + 31) & ~size_t(31); }

struct TailDevice {
  TailTables host;
  uint4 *item = nullptr;
  uint2 *more = nullptr;
  uint16_t *out = nullptr;
  uint8_t *slot_h = nullptr;
  TopCounts *top = nullptr;
  std::vector<void *> allocs;
  ~TailDevice() {
    for (void *p : allocs) cudaFree(p);
  }
};

std::mutex g_mu;
std::map<std::pair<int, int>, std::unique_ptr<TailDevice>> g_tail;  // (device, s)

template <typename T, typename D>
cudaError_t upload(TailDevice &d, const std::vector<T> &h, D **out) {
  cudaError_t e = cudaMalloc(reinterpret_cast<void **>(out), std::max<size_t>(16, h.size() * sizeof(T)));
  if (e != cudaSuccess) return e;
  d.allocs.push_back(*out);
  return h.empty() ? cudaSuccess : cudaMemcpy(*out, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
}

const TailTables &host_tables(int s) {
  static std::mutex mu;
  static std::map<int, std::unique_ptr<TailTables>> tabs;
  std::lock_guard<std::mutex> lk(mu);
  auto &t = tabs[s];
  if (!t) t = std::make_unique<TailTables>(build_tail_tables(s));
  return *t;
}

cudaError_t tail_device(int s, TailDevice **out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(g_mu);
  auto &slot = g_tail[{dev, s}];
  if (!slot) {
    auto d = std::make_unique<TailDevice>();
    d->host = host_tables(s);
    std::vector<TopCounts> top;
    for (int g = 0; g <= s + 2; ++g) top.push_back(top_counts(g));
    if ((e = upload(*d, d->host.item, &d->item)) != cudaSuccess) return e;
    if ((e = upload(*d, d->host.more, &d->more)) != cudaSuccess) return e;
    if ((e = upload(*d, d->host.out, &d->out)) != cudaSuccess) return e;
    if ((e = upload(*d, d->host.slot_h, &d->slot_h)) != cudaSuccess) return e;
    if ((e = upload(*d, top, &d->top)) != cudaSuccess) return e;
    for (auto f : {tail_kernel<uint32_t, true>, tail_kernel<uint32_t, false>, tail_kernel<uint64_t, true>,
                   tail_kernel<uint64_t, false>})
      if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemBudget))) != cudaSuccess)
        return e;
    slot = std::move(d);
  }
  *out = slot.get();
  return cudaSuccess;
}

}  // namespace

struct WholeDevice {
  TailClass cls;
  uint4 *item = nullptr;
  uint2 *more = nullptr;
  uint16_t *first = nullptr;
};

static std::map<std::pair<int, int>, WholeDevice> g_whole;  // (device, W), guarded by g_mu

bool solves_whole(int W) { return W <= 12; }

cudaError_t prepare_whole(int W) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(g_mu);
  if (g_whole.count({dev, W})) return cudaSuccess;
  static std::map<std::pair<int, int>, std::unique_ptr<TailDevice>> owners;  // free the arrays at exit
  const TailTables t = build_whole_tables(W);
  auto d = std::make_unique<TailDevice>();
  WholeDevice wd;
  wd.cls = t.cls[1];
  std::vector<uint16_t> first;
  for (uint64_t m = 0; m < (1ull << (W - 1)); ++m) first.push_back(uint16_t(rank_word(first_row_state(m, W), W)));
  if ((e = upload(*d, t.item, &wd.item)) != cudaSuccess) return e;
  if ((e = upload(*d, t.more, &wd.more)) != cudaSuccess) return e;
  if ((e = upload(*d, first, &wd.first)) != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(whole_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024)) != cudaSuccess)
    return e;
  owners[{dev, W}] = std::move(d);
  g_whole[{dev, W}] = wd;
  return cudaSuccess;
}

cudaError_t launch_whole(int W, int K, const uint32_t *mods, uint32_t *residues, cudaStream_t st) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  WholeArgs a{};
  {
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_whole.find({dev, W});
    if (it == g_whole.end()) return cudaErrorNotReady;  // prepare_whole first (outside capture)
    a.item = it->second.item;
    a.more = it->second.more;
    a.first = it->second.first;
    a.cls = it->second.cls;
  }
  a.residues = residues;
  a.W = W;
  for (int l = 0; l < K; ++l) a.mod[l] = mods[l];
  const unsigned threads = std::min(1024u, std::max(64u, (a.cls.nblk + 31) / 32 * 32));
  whole_kernel<<<unsigned(K), threads, size_t(a.cls.words) * 4, st>>>(a);
  return cudaGetLastError();
}

int tail_symbols(int W) { return W >= 14 ? 9 : 0; }

uint64_t tail_escape_words(int W) {
  const int s = tail_symbols(W);
  if (!s) return 0;
  const TailTables &t = host_tables(s);
  uint64_t n = 0;
  for (int g = 0; g <= s; ++g) n += uint64_t(top_counts(g).P[W - s][1]) * t.cls[size_t(g)].nout;
  return n;
}

cudaError_t prepare_tail(int W) {
  TailDevice *d = nullptr;
  return tail_symbols(W) ? tail_device(tail_symbols(W), &d) : cudaSuccess;
}

cudaError_t launch_tail(const DevTables &t, int K, const uint32_t *mods, uint32_t *main, const uint32_t *blk,
                        uint32_t *esc, cudaStream_t st, uint64_t *launches) {
  const int s = tail_symbols(t.W);
  if (!s || !t.ptr || K < 1 || K > kMaxLanes || t.cap < FDP_FULL_CAP || !esc) return cudaErrorInvalidValue;
  TailDevice *d = nullptr;
  cudaError_t e = tail_device(s, &d);
  if (e != cudaSuccess) return e;
  const int tl = t.W - s;
  TailArgs a{};
  a.item = d->item;
  a.more = d->more;
  a.out = d->out;
  a.slot_h = d->slot_h;
  a.top = d->top;
  a.tables = t.ptr;
  a.main = main;
  a.blk = blk;
  a.esc = esc;
  a.M = main_states(t.W);
  a.D = blocked_states(t.W);
  uint32_t nT[FDP_TAIL_MAX_G + 1] = {};
  for (int g = 0; g <= s; ++g) {
    nT[g] = top_counts(g).P[tl][1];
    a.ebase[g] = a.E;
    a.E += uint64_t(nT[g]) * d->host.cls[size_t(g)].nout;
  }
  bool wide = true;
  for (int l = 0; l < K; ++l) {
    a.mod[l] = mods[l];
    wide = wide && mods[l] > 0x80000000u;
  }
  a.W = t.W;
  a.s = s;
  const size_t rec = (t.u64 ? blocks_bytes<uint64_t>() : blocks_bytes<uint32_t>());
  for (int top = s; top >= 0; top -= 2) {
    uint32_t ctas = 0;
    a.nsegs = 0;
    a.top_g = top;
    a.cls[0] = d->host.cls[size_t(top)];
    if (top) a.cls[1] = d->host.cls[size_t(top) - 1];
    for (int l0 = 0; l0 < K;) {
      const int pw = (K - l0 >= 8) ? 8 : (K - l0 >= 4) ? 4 : (K - l0 >= 2) ? 2 : 1;
      for (int g = top; g >= top - 1 && g >= 0; --g) {
        if (!nT[g]) continue;
        const size_t col = size_t(d->host.cls[size_t(g)].words) * 32;
        int groups = int((kSmemBudget - rec) / col);
        groups = std::max(1, std::min(groups, kMaxBlocks * pw / 8));
        // Small widths: as many CTAs as the blocks allow before CTAs take several groups.
        const uint64_t all = (uint64_t(nT[g]) * pw + 7) / 8;
        groups = int(std::max<uint64_t>(1, std::min<uint64_t>(groups, all / (uint64_t(device_sm_count()) * 2))));
        TailSeg &sg = a.seg[a.nsegs++];
        sg = TailSeg{ctas, nT[g], g, l0, pw, groups};
        const uint32_t per = uint32_t(groups) * uint32_t(8 / pw);
        ctas += (nT[g] + per - 1) / per;
      }
      l0 += pw;
    }
    if (!ctas) continue;
    const auto kernel = t.u64 ? (wide ? tail_kernel<uint64_t, true> : tail_kernel<uint64_t, false>)
                              : (wide ? tail_kernel<uint32_t, true> : tail_kernel<uint32_t, false>);
    kernel<<<ctas, kThreads, kSmemBudget, st>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (launches) ++*launches;
  }
  return cudaSuccess;
}

}  // namespace fdp
