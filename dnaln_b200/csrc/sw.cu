// sw.cu — banded affine-gap Smith–Waterman (score-only and with traceback) for sm_100a.
//
// The recurrence is the reference's diagonal-coordinate band (src/align.hpp:3-15,
// src/align.cpp:31-84): row i, band column d in [0, W), target column i+d,
//   hd = H(i-1,d) + s(q_i, t_{i+d})
//   E(i,d) = max(H(i-1,d+1) - (O+E), E(i-1,d+1) - E)
//   F(i,d) = max(H(i,d-1) - (O+E),   F(i,d-1) - E)
//   H(i,d) = max(hd, E(i,d), F(i,d), 0)
// with H = E = 0 for row -1 and for the fixed out-of-band cell d = W, F = H(left) = 0 at
// each row start, and the target N-padded to qlen + W - 1.
//
// Kernels:
//  * k_sw_u2<W> (a thread owns whole alignments, no intra-row shuffles): two alignments per
//    thread, one in each 16-bit half of 32-bit registers, the band row (H, E of W+1 cells, W
//    target selectors) in registers.
//    Values are kept biased by +16384, so every half stays positive and every add or
//    subtract of the recurrence is one 32-bit integer add on both halves (no borrow can
//    cross halves); E and F are DPX add-maxima (viaddmax), the other maxima unsigned 16x2
//    max (vmaxu2 / DPX vimax3_u16x2). The substitution scores of both alignments are one
//    prmt.b32 from an 8-byte per-row profile {s(qA, A..T) + 64, s(qB, A..T) + 64}.
//    Direction flags are the signs of non-negative differences (cell2).
//    With traceback it stores the direction codes and only the best cell; the walk is a
//    separate kernel (k_sw_walk, few registers, full occupancy) so the DP kernel's
//    register footprint does not carry the walk.
//  * k_sw_wide<W, LANES, CH>: the same cells, several lanes per pair of alignments.
//  * A task whose target window may contain an N (the 4-entry profile cannot score it),
//    or whose scores or lengths do not fit the biased 16-bit range, is appended by
//    them to a device-side list; k_sw_fb and k_sw_fb_lanes run the same cell update in
//    int32 for the listed tasks, same outputs and codes. Genome windows that the task
//    builder marked N-free (kTaskNoN) skip the per-task N scan.
//  * k_sw_any: any band width and any scores (int32, band rows in per-warp scratch).
//
// Direction code of a cell (4 bits):
//   kNotDiag: H > hd                           kNotE: H > E
//   kExtE: E extends E(i-1,d+1) (ee > eo)      kExtF: F extends F(i,d-1) (fe > fo)
// The codes of four neighbouring cells share 16 bits, cell c's at bits c (kNotDiag), 4 + c
// (kExtE), 8 + c (kNotE) and 12 + c (kExtF): the order in which cell2 gets them. (k_sw_any's: see
// WordCodes.)
// On every cell the walk reads, H is the positive value being traced; there it came from the
// diagonal if h == hd (src/align.cpp:67), else from E if h == e, and otherwise from F — so
// the walk (src/align.cpp:87-143) takes the reference's steps. The best cell is the first strict
// maximum in row-major order (per-row maximum with its first column, then strict across rows).
#include <algorithm>
#include <climits>
#include <type_traits>

#include "common.cuh"
#include "sw.cuh"

namespace dnb {

namespace {

constexpr int kSwThreads = 128;
// k_sw_u2 and k_sw_wide: blocks of one warp, as many as are resident, which take 32 / LANES
// pairs at a time: first those of their block index, then the next by an atomic add until
// none is left. The list is ordered longest first and often counted on the device only.
// Against a grid over the longest possible list, with blocks of four warps: blocks go to the
// GPCs in turn, so the SMs of a small GPC held 16 warps where the others held 8 to 12 and set
// the kernel's time, and an empty list of 262,144 cost 15 us. (Claiming the first pairs too
// lets the SMs that start first take whole lists: 219 -> 303 us for 58,000 tasks.)
constexpr int kDpThreads = 32;
constexpr uint32_t kNotDiag = 1u, kExtE = 0x10u, kNotE = 0x100u, kExtF = 0x1000u, kCode = 0x1111u;
constexpr uint32_t kBias = 16384u, kBias2 = 0x40004000u;
constexpr int kScoreBias = 64;  // profile bytes are score + 64, in [0, 127]
constexpr int kAhead = 8;       // cells of a diagonal run the walk fetches at once

// prmt.b32 in its default mode (the sign-replicate bit of each selector nibble is
// honoured; the __byte_perm intrinsic uses only the low 3 bits of each nibble).
__device__ __forceinline__ uint32_t prmt(uint32_t lo, uint32_t hi, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(lo), "r"(hi), "r"(sel));
  return r;
}

// Selector of the sign-extended profile byte c (0..7) as one 32-bit value.
__device__ __forceinline__ uint32_t sel1(uint32_t c) {
  const uint32_t s = c | 8u;
  return c | (s << 4) | (s << 8) | (s << 12);
}

// Selector of two zero-extended 16-bit values: byte a (0..3) of the low profile word into
// the low half, byte b of the high word into the high half (the profile bytes are
// below 128, so the sign-replicating nibbles give zero high bytes).
__device__ __forceinline__ uint32_t sel2(uint32_t a, uint32_t b) {
  const uint32_t x = 4u + b;
  return a | ((a | 8u) << 4) | (x << 8) | ((x | 8u) << 12);
}

__device__ __forceinline__ uint32_t tcode(const uint8_t* __restrict__ tbase, const SwTask& tk, int64_t j) {
  const int64_t x = tk.t_start + j;
  if (x < tk.t_lo || x >= tk.t_hi) return 4;
  const uint32_t c = __ldg(tbase + x);
  return c > 3 ? 4u : c;
}

// Profile word of query code qc for the int32 path: byte t = match if t == qc else
// -mismatch; an N query row scores -ambig everywhere.
__device__ __forceinline__ uint32_t prof_lo(const SwParams& p, uint32_t qc) {
  if (qc > 3) return p.prof_n;
  const uint32_t mm = (static_cast<uint32_t>(static_cast<uint8_t>(-p.mismatch))) * 0x01010101u;
  const uint32_t sh = 8u * qc;
  return (mm & ~(0xFFu << sh)) | (static_cast<uint32_t>(static_cast<uint8_t>(p.match)) << sh);
}

// The same profile biased by +64 (every byte in [0, 127]) for the 16-bit path.
__device__ __forceinline__ uint32_t prof_biased(const SwParams& p, uint32_t qc) {
  if (qc > 3) return static_cast<uint32_t>(kScoreBias - p.ambig) * 0x01010101u;
  const uint32_t mm = static_cast<uint32_t>(kScoreBias - p.mismatch) * 0x01010101u;
  const uint32_t sh = 8u * qc;
  return (mm & ~(0xFFu << sh)) | (static_cast<uint32_t>(kScoreBias + p.match) << sh);
}

__device__ __forceinline__ uint32_t pack2(uint32_t v) { return (v & 0xFFFFu) * 0x10001u; }

// A cell's code, its flags STEP bits apart. diag: hd >= E and max(hd, E) >= F; from_e: the latter,
// which is H = E on every cell the walk asks it for (H > 0 and not from the diagonal). Neither
// waits for H: compared with H itself, k_sw_fb<43> spilled and took 181 us for 64 tasks of 150
// rows, like this 154.
template <int STEP = 4>
__device__ __forceinline__ uint32_t dir_code32(bool diag, bool from_e, bool e_not_ext, bool f_not_ext) {
  return (diag ? 0u : 1u) | (e_not_ext ? 0u : 1u << STEP) | (from_e ? 0u : 1u << 2 * STEP) |
         (f_not_ext ? 0u : 1u << 3 * STEP);
}

// Global store with an L2 evict-first policy: streaming data (the direction codes, read
// once by the walk) should not push the resident index out of L2.
__device__ __forceinline__ uint64_t l2_evict_first_policy() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
__device__ __forceinline__ void st_evict_first(uint32_t* p, uint32_t v, uint64_t pol) {
  asm volatile("st.global.L2::cache_hint.b32 [%0], %1, %2;" ::"l"(p), "r"(v), "l"(pol) : "memory");
}

// One cell of two alignments in biased 16-bit halves. H is kept as H - (O+E), which is what
// both neighbours open a gap from: E and F are one DPX add-max each (max(a + b, c), signed
// 16x2: the biased values lie in [0, 32767], where signed and unsigned order agree).
//
// Adds, maxima, prmt and logic run on the ALU pipe at one instruction every two cycles, and
// integer multiply-adds beside it at the same rate, so some of the cell's additions are
// written as multiply-adds by 1 or -1 that the compiler cannot fold. Measured, 88,000
// tracebacks at W = 129 and 262,144 of 150 rows at W = 33: as below 1,154 and 631 us; every
// addition a multiply-add 1,200 and 708; none 1,439 and, in the flags' former form, 677.
struct CellParams {
  uint32_t oe, nge, khd;  // O+E; -E in each signed half; O+E - profile bias
  uint32_t one, mone;     // 1 and -1, as values known at run time only
};
__device__ __forceinline__ CellParams cell_params(const SwParams& p) {
  return {pack2(p.oe), pack2(static_cast<uint32_t>(-p.ge)), pack2(p.oe) - pack2(kScoreBias), p.one, p.mone};
}
__device__ __forceinline__ uint32_t mad(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}
// hdiag, hup, hleft, the result: H - (O+E); s: profile value; f: F of the left cell, then of
// this one. TB: code holds the direction code in the bits of every cell of the word, for
// insert_code. A flag is x > y for some x >= y, both below 2^14 + 16000, so x - y + 0x7FFF
// carries it in the sign bit of its half, with no borrow or carry between the halves; two
// prmt spread the four sign bits over bytes and a select merges them.
template <bool TB>
__device__ __forceinline__ uint32_t cell2(const CellParams& c, uint32_t hdiag, uint32_t s, uint32_t hup, uint32_t eup,
                                          uint32_t hleft, uint32_t& f, uint32_t& e, uint32_t& code) {
  const uint32_t hd = hdiag + c.khd + s;
  e = __viaddmax_s16x2(eup, c.nge, hup);
  f = __viaddmax_s16x2(f, c.nge, hleft);
  const uint32_t h = __vimax3_u16x2(__vmaxu2(hd, e), f, kBias2);
  if constexpr (TB) {
    constexpr uint32_t k = 0x7FFF7FFFu;
    const uint32_t hk = mad(h, c.one, k);
    const uint32_t de = prmt(mad(hd, c.mone, hk), mad(e, c.mone, hk), 0xFBD9u);  // bytes: A kNotDiag, A kNotE, B, B
    const uint32_t ex = prmt(e - hup + k, mad(hleft, c.mone, f) + k, 0xFBD9u);
    code = (de & 0x0F0F0F0Fu) | (ex & 0xF0F0F0F0u);
  }
  return mad(c.oe, c.mone, h);
}
// Cell c (0..3) of its word; c = 0 starts the word.
__device__ __forceinline__ uint32_t insert_code(uint32_t dw, uint32_t code, int c) {
  const uint32_t m = 0x11111111u << c;
  return c == 0 ? code : (dw & ~m) | (code & m);
}

struct CigarWriter {
  uint32_t* out;
  int cap, n;
  uint32_t op;
  int len;
  __device__ void push(uint32_t o, int l) {
    if (o == op) {
      len += l;
      return;
    }
    flush();
    op = o;
    len = l;
  }
  __device__ void flush() {
    if (len) {
      if (n < cap) out[n] = static_cast<uint32_t>(len) << 4 | op;
      ++n;
    }
    len = 0;
  }
};

// Direction codes of the pair layout: word (i, g), g < WQ = ceil(W/4), holds cells 4g..4g+3
// of both alignments of a thread (A in the low 16 bits, B in the high 16); the 32 pairs of a warp
// are interleaved word by word.
struct PairCodes {
  static constexpr uint32_t kFromNotE = kNotE, kEExt = kExtE, kFExt = kExtF, kAll = kCode;
  const uint32_t* D;  // this pair's first word
  int WQ, half;
  __device__ uint32_t word(int i, int d) const { return D[(static_cast<size_t>(i) * WQ + (d >> 2)) * 32]; }
  __device__ int shift(int d) const { return 16 * half + (d & 3); }
  __device__ uint32_t operator()(int i, int d) const { return (word(i, d) >> shift(d)) & kCode; }
};

// Direction codes of the generic kernel: word (i, w), w < WW = ceil(W/8), holds cells
// 8w..8w+7, the flags of cell 8w + c at bits c, 8 + c, 16 + c and 24 + c; 32 alignments of a warp
// interleaved word by word. One shift places a cell's flags: two groups of four cells side by side
// took 2,923 us for 64 tasks of 150 rows at W = 201, this 2,810.
struct WordCodes {
  static constexpr int kStep = 8;
  static constexpr uint32_t kEExt = 1u << kStep, kFromNotE = 1u << 2 * kStep, kFExt = 1u << 3 * kStep,
                            kAll = 1u | kEExt | kFromNotE | kFExt;
  const uint32_t* D;
  int WW;
  __device__ uint32_t word(int i, int d) const { return D[(static_cast<size_t>(i) * WW + (d >> 3)) * 32]; }
  __device__ int shift(int d) const { return d & 7; }
  __device__ uint32_t operator()(int i, int d) const { return (word(i, d) >> shift(d)) & kAll; }
};

// High bit of each byte of x set where that byte is zero, every other bit clear.
__device__ __forceinline__ uint64_t zero_bytes(uint64_t x) {
  constexpr uint64_t kLow7 = 0x7F7F7F7F7F7F7F7Full;
  return ~(((x & kLow7) + kLow7) | x | kLow7);
}

// The bytes p[0..7] as one little-endian word, from the aligned 8-byte word holding p[0]
// and, unless p is aligned, the next one. Each of the two holds at least one of the eight
// bytes asked for, so neither lies outside the pages those bytes are in.
__device__ __forceinline__ uint64_t load8u(const uint8_t* p) {
  static_assert(kAhead == 8, "one 8-byte word per block of the diagonal run");
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  const uint64_t* w = reinterpret_cast<const uint64_t*>(a & ~static_cast<uintptr_t>(7));
  const unsigned sh = static_cast<unsigned>(a & 7) * 8u;
  const uint64_t lo = __ldg(w);
  if (sh == 0) return lo;
  return (lo >> sh) | (__ldg(w + 1) << (64u - sh));
}

// Walks the direction codes back from (bi, bd) (src/align.cpp:87-143). CIGAR ops are
// written in walk order (last op first), adjacent equal ops merged as the reference's
// push() does. Guards flag, and never read, a cell outside the band.
template <class Codes>
__device__ void traceback(const Codes& code, int W, int bi, int bd, int best, const uint8_t* __restrict__ q,
                          const uint8_t* __restrict__ tbase, const SwTask& tk, const SwParams& p, SwResult& r,
                          uint32_t* __restrict__ cig, int cap, uint32_t* __restrict__ err) {
  CigarWriter cw{cig, cap, 0, 0xFu, 0};
  int i = bi, d = bd, v = best, nm = 0;
  const int smax = max(p.match, max(-p.mismatch, -p.ambig));  // the most one step can lower v
  if (d < 0 || d >= W) {
    atomicOr(err, kErrTracebackBounds);
    i = -1;
    v = 0;
  }
  for (;;) {
    int run = 0;
    uint32_t x = 0;
    if (i >= 0 && v > 0 && (d < 0 || d >= W)) {
      atomicOr(err, kErrTracebackBounds);
      break;
    }
    // Diagonal run. The next kAhead cells (i-k, d) are fetched together (codes, query and
    // target bases: independent loads, one memory latency per kAhead steps) and then
    // consumed in order exactly as the one-cell-at-a-time walk would.
    bool stop = false;
    while (!stop && i >= 0 && v > 0) {
      uint32_t cx[kAhead];
      int qa[kAhead], ta[kAhead];
      const int64_t x0 = tk.t_start + (i - (kAhead - 1)) + d;  // target of row i - 7
      if (i >= kAhead - 1 && x0 >= tk.t_lo && x0 + kAhead <= tk.t_hi) {
        // the block's 8 query and 8 target bytes are contiguous: two 8-byte words each
        // instead of 16 byte loads (the walk is bound by its L1 requests)
        const uint64_t qw = load8u(q + i - (kAhead - 1)), tw = load8u(tbase + x0);
        uint32_t wk[kAhead], any = 0;
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
          wk[k] = code.word(i - k, d);
          any |= wk[k];
        }
        const int sh = code.shift(d);
        // A block that is diagonal throughout, with v > 0 before each of its steps (each
        // step lowers v by at most smax), is taken whole: its score and mismatches from the
        // two byte words (bytes equal and both below 4: match; either above 3: ambiguous;
        // else mismatch), exactly the sums of the steps below.
        if (((any >> sh) & kNotDiag) == 0 && v > (kAhead - 1) * smax) {
          const uint64_t amb = (qw | tw) & 0xFCFCFCFCFCFCFCFCull;
          const uint64_t ok_amb = zero_bytes(amb);
          const int n_match = __popcll(zero_bytes(qw ^ tw) & ok_amb);
          const int n_amb = kAhead - __popcll(ok_amb);
          v -= n_match * p.match - (kAhead - n_match - n_amb) * p.mismatch - n_amb * p.ambig;
          nm += kAhead - n_match;
          run += kAhead;
          i -= kAhead;
          continue;
        }
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
          cx[k] = (wk[k] >> sh) & Codes::kAll;
          qa[k] = static_cast<int>((qw >> (8 * (kAhead - 1 - k))) & 0xFFu);
          const int t8 = static_cast<int>((tw >> (8 * (kAhead - 1 - k))) & 0xFFu);
          ta[k] = t8 > 3 ? 4 : t8;
        }
      } else {
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
          cx[k] = 0;
          qa[k] = ta[k] = 0;
          if (i - k >= 0) {
            cx[k] = code(i - k, d);
            qa[k] = q[i - k];
            ta[k] = static_cast<int>(tcode(tbase, tk, static_cast<int64_t>(i - k) + d));
          }
        }
      }
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        if (i < 0 || v <= 0) {
          stop = true;
          break;
        }
        x = cx[k];
        if (x & kNotDiag) {  // not from the diagonal
          stop = true;
          break;
        }
        v -= sub_score(p, qa[k], ta[k]);
        nm += (qa[k] != ta[k] || qa[k] > 3) ? 1 : 0;
        ++run;
        --i;
      }
    }
    if (run) cw.push(0u /* M */, run);
    if (i < 0 || v <= 0) break;
    run = 0;
    bool ext;
    if (!(x & Codes::kFromNotE)) {  // from E, an insertion: E(i,d) <- (i-1, d+1)
      do {
        if (i < 0 || d >= W) {
          atomicOr(err, kErrTracebackBounds);
          goto done;
        }
        ext = (code(i, d) & Codes::kEExt) != 0;
        v += ext ? p.ge : p.oe;
        ++run;
        --i;
        ++d;
      } while (ext);
      cw.push(1u /* I */, run);
    } else {  // from F, a deletion: F(i,d) <- (i, d-1)
      do {
        if (d < 0 || d >= W) {
          atomicOr(err, kErrTracebackBounds);
          goto done;
        }
        ext = (code(i, d) & Codes::kFExt) != 0;
        v += ext ? p.ge : p.oe;
        ++run;
        --d;
      } while (ext);
      cw.push(2u /* D */, run);
    }
    nm += run;
  }
done:
  cw.flush();
  if (cw.n > cap) atomicOr(err, kErrCigarOverflow);
  r.qb = i + 1;
  r.tb = i + 1 + d;
  r.qe = bi + 1;
  r.te = bi + bd + 1;
  r.nm = nm;
  r.n_ops = cw.n < cap ? cw.n : cap;
}


// Best-row checkpoints of the two halves of a pair share two row buffers: a row that
// improves both halves is stored once (the packed row serves both), and a half that
// improves alone writes the buffer the other half is not using. Returns the buffer to
// write; buf_a / buf_b say where each half's best row is.
__device__ __forceinline__ int row_buffer(bool up_a, bool up_b, int buf_a, int buf_b) {
  if (up_a && up_b) return buf_a;
  if (up_a) return buf_a == buf_b ? 1 - buf_b : buf_a;
  return buf_a == buf_b ? 1 - buf_a : buf_b;
}

// The fallback list of a launch: fb[0] its length, fb[1] and fb[2] the warps' claims of the short
// lists' form and of the main one, then local task indices.
constexpr int kFbList = kSwFbHead;

// The warp's next claim after its first, blockIdx.x, in every lane.
__device__ __forceinline__ int next_claim(int* claim) {
  int w = 0;
  if ((threadIdx.x & 31) == 0) w = static_cast<int>(gridDim.x) + atomicAdd(claim, 1);
  return __shfl_sync(0xffffffffu, w, 0);
}

// The DP kernels leave, for the walk, the best cell in the result: qb = its row, qe = its
// column (the walk kernel then writes the final coordinates).
__device__ __forceinline__ SwResult stash(int score, int bi, int bd) { return SwResult{score, bi, bd, 0, 0, 0, 0, 0}; }

// Direction-code base of local task lt (pairs 2p, 2p+1 share words; 32 pairs per warp).
__device__ __forceinline__ uint32_t* pair_base(uint32_t* dir, int lt, int rows_max, int WQ) {
  const int pair = lt >> 1;
  return dir + static_cast<size_t>(pair >> 5) * rows_max * WQ * 32 + (pair & 31);
}

// One alignment, int32 scores, band row of compile-time width W in registers; direction
// codes into its half of the pair layout (DP = the pair's first word).
template <int W, bool TB>
__device__ SwResult sw_one_reg(const SwTask& tk, const uint8_t* __restrict__ qbase, const uint8_t* __restrict__ tbase,
                               const SwParams& p, uint32_t* __restrict__ DP, int half) {
  constexpr int WQ = (W + 3) / 4;
  const uint8_t* __restrict__ q = qbase + tk.q_off;
  const int ql = tk.qlen;
  int H[W + 1], E[W + 1];
  uint32_t T[W];
#pragma unroll
  for (int d = 0; d <= W; ++d) {
    H[d] = 0;
    E[d] = 0;
  }
#pragma unroll
  for (int d = 0; d < W; ++d) T[d] = sel1(tcode(tbase, tk, d));
  int best = 0, bi = -1, bd = -1;
  for (int i = 0; i < ql; ++i) {
    const uint32_t qc = min(static_cast<uint32_t>(q[i]), 4u);
    const uint32_t plo = prof_lo(p, qc), phi = p.prof_n;
    const uint32_t t_next = sel1(tcode(tbase, tk, static_cast<int64_t>(i) + W));
    int f = 0, hleft = 0, hdiag = H[0], rmax = 0, rd = -1;
    uint32_t dw = 0;
#pragma unroll
    for (int d = 0; d < W; ++d) {
      const int hup = H[d + 1], eup = E[d + 1];
      const int hd = hdiag + static_cast<int>(prmt(plo, phi, T[d]));
      const int eo = hup - p.oe, ee = eup - p.ge, fo = hleft - p.oe, fe = f - p.ge;
      const int e = max(eo, ee);
      f = max(fo, fe);
      const int m1 = max(hd, e);
      const int h = max(max(m1, f), 0);
      H[d] = h;
      E[d] = e;
      if constexpr (TB) {
        dw |= dir_code32(hd >= e && m1 >= f, m1 >= f, eo >= ee, fo >= fe) << (d & 3);
        if ((d & 3) == 3 || d == W - 1) {
          reinterpret_cast<uint16_t*>(DP + (static_cast<size_t>(i) * WQ + (d >> 2)) * 32)[half] =
              static_cast<uint16_t>(dw);
          dw = 0;
        }
        if (d == 0 || h > rmax) {  // first strict maximum of the row (every H >= 0)
          rmax = h;
          rd = d;
        }
      } else {
        best = max(best, h);
      }
      hleft = h;
      hdiag = hup;
    }
    if (TB && rmax > best) {
      best = rmax;
      bi = i;
      bd = rd;
    }
#pragma unroll
    for (int d = 0; d + 1 < W; ++d) T[d] = T[d + 1];
    T[W - 1] = t_next;
  }
  return TB ? stash(best, bi, bd) : stash(best, 0, 0);
}

// True if the target window [0, qlen + W - 1) of the task reads any N, including the
// padding outside the candidate's contig or past a short target.
__device__ bool window_has_n(const SwTask& tk, int W, const uint8_t* __restrict__ tbase) {
  if (tk.flags & kTaskNoN) return false;
  const int64_t tmax = static_cast<int64_t>(tk.qlen) + W - 1;
  if (tk.t_lo > tk.t_start || tk.t_hi < tk.t_start + tmax) return true;
  const uint8_t* t = tbase + tk.t_start;
  bool any = false;
  for (int64_t j = 0; j < tmax; ++j) any |= __ldg(t + j) > 3;
  return any;
}

// Two alignments per thread in biased 16-bit halves (A low, B high), a cell at a time by
// cell2. Pairs it cannot take (an N in a target window, or scores/lengths outside the 16-bit
// range) are listed in fb for k_sw_fb. With traceback at W <= 33 the launch bound asks for
// twelve resident warps (<= 170 registers, no spills).
//  * the substitution scores of both alignments are one prmt.b32 on the row's profile
//    words, taken from a 5-entry table in shared memory one row ahead;
//  * target codes are read without range or N checks: the pair reaches the DP only when
//    both windows [0, qlen + W - 1) are N-free and inside their contigs, and reads past a
//    window are clamped to its last base (a row past a query's end is an N row for it,
//    whose scores do not depend on the target), so a code is always 0..3 and the prmt
//    selector of two codes is two multiply-adds.
template <int W, bool TB>
__global__ void __launch_bounds__(kDpThreads, (TB && W <= 33) ? 12 : 1)
    k_sw_u2(const SwTask* __restrict__ tasks, int base, int n, const int* __restrict__ n_dev, int few,
             const uint8_t* __restrict__ qbase, const uint8_t* __restrict__ tbase, SwParams p,
             SwResult* __restrict__ res, uint32_t* __restrict__ dir, int rows_max, int* __restrict__ fb,
             int* __restrict__ claim) {
  static_assert(W >= 3, "a window of at least two columns past an empty query");
  constexpr int WQ = (W + 3) / 4;
  __shared__ uint32_t s_prof[8];
  if (threadIdx.x < 5) s_prof[threadIdx.x] = prof_biased(p, threadIdx.x);
  __syncthreads();
  if (n_dev && *n_dev <= few) return;  // a short list is the narrowest form's
  const int nn = n_dev ? min(n, *n_dev) : n, pairs = (nn - base + 1) / 2;
  const auto align = [&](const int lt) {  // lt: pair index within this launch
  const int ia = base + 2 * lt, ib = ia + 1;
  const bool has_b = ib < nn;
  uint32_t* DP = TB ? pair_base(dir, 2 * lt, rows_max, WQ) : nullptr;
  const SwTask ta = tasks[ia];
  SwTask tb = ta;
  if (has_b) tb = tasks[ib];
  else tb.qlen = 0;
  const int qmax = max(ta.qlen, tb.qlen);
  const bool fits = qmax * p.match + 2 * (p.oe + p.ge + p.mismatch + p.ambig) < 16000 &&
                    p.match + kScoreBias <= 127 && p.mismatch <= kScoreBias && p.ambig <= kScoreBias;
  if (!fits || window_has_n(ta, W, tbase) || (has_b && window_has_n(tb, W, tbase))) {
    const int k = atomicAdd(fb, has_b ? 2 : 1);
    fb[kFbList + k] = 2 * lt;
    if (has_b) fb[kFbList + 1 + k] = 2 * lt + 1;
    return;
  }
  const uint8_t* __restrict__ qa = qbase + ta.q_off;
  const uint8_t* __restrict__ qb = qbase + tb.q_off;
  const int qla = ta.qlen, qlb = tb.qlen;
  // both windows are N-free over [0, qlen + W - 1): column j of each reads its window at
  // min(j, qlen + W - 2), a code in 0..3
  const uint8_t* __restrict__ wa = tbase + ta.t_start;
  const uint8_t* __restrict__ wb = tbase + tb.t_start;
  const int ja = qla + W - 2, jb = qlb + W - 2;
  auto tc2 = [&](int j) {
    const uint32_t a = __ldg(wa + min(j, ja)), b = __ldg(wb + min(j, jb));
    return a * 17u + b * 4352u + 50304u;  // sel2(a, b)
  };
  auto qcode = [&](const uint8_t* __restrict__ q, int ql, int i) {
    return i < ql ? min(static_cast<uint32_t>(q[i]), 4u) : 4u;
  };
  const CellParams cp = cell_params(p);
  const uint32_t h_zero = kBias2 - cp.oe;  // H = 0
  uint32_t H[W + 1], E[W + 1], T[W];
#pragma unroll
  for (int d = 0; d <= W; ++d) {
    H[d] = h_zero;
    E[d] = kBias2;
  }
#pragma unroll
  for (int d = 0; d < W; ++d) T[d] = tc2(d);
  const uint32_t zero = kBias - static_cast<uint32_t>(p.oe);
  uint32_t best2 = h_zero, best_a = zero, best_b = zero;
  int bi_a = -1, bi_b = -1;
  extern __shared__ __align__(16) uint32_t sw_rows[];  // k_sw_wide stores 16 bytes at a time
  uint32_t* const row_a = sw_rows + threadIdx.x;
  uint32_t* const row_b = sw_rows + W * kDpThreads + threadIdx.x;
  int buf_a = 0, buf_b = 1;
  uint32_t plo = s_prof[qcode(qa, qla, 0)], phi = s_prof[qcode(qb, qlb, 0)];
  uint32_t ca = qcode(qa, qla, 1), cb = qcode(qb, qlb, 1);  // codes of the next row
  uint32_t* rowp = DP;
  const uint64_t pol = l2_evict_first_policy();
  for (int i = 0; i < qmax; ++i) {
    // the next row's codes and profile words and the target column entering the band are
    // loaded up front, so their latency hides behind this row
    const uint32_t t_next = tc2(i + W);
    const uint32_t plo_next = s_prof[ca], phi_next = s_prof[cb];
    const uint32_t ca_next = qcode(qa, qla, i + 2), cb_next = qcode(qb, qlb, i + 2);
    uint32_t f = kBias2, hleft = h_zero, hdiag = H[0], rmax = 0, dw = 0;
#pragma unroll
    for (int d = 0; d < W; ++d) {
      const uint32_t hup = H[d + 1];
      uint32_t e, code = 0;
      const uint32_t h = cell2<TB>(cp, hdiag, prmt(plo, phi, T[d]), hup, E[d + 1], hleft, f, e, code);
      if constexpr (TB) {
        dw = insert_code(dw, code, d & 3);
        if ((d & 3) == 3 || d == W - 1) st_evict_first(rowp + (d >> 2) * 32, dw, pol);
      }
      // the row's maximum (score only: the maximum so far), two cells at a time
      uint32_t& top = TB ? rmax : best2;
      if (d & 1) top = __vimax3_u16x2(top, hleft, h);
      else if (d == W - 1) top = __vmaxu2(top, h);
      H[d] = h;
      E[d] = e;
      hleft = h;
      hdiag = hup;
    }
    if constexpr (TB) {  // a strictly better row (rows in order: the first strict maximum)
      const bool up_a = (rmax & 0xFFFFu) > best_a, up_b = (rmax >> 16) > best_b;
      if (up_a || up_b) {
        const int dst = row_buffer(up_a, up_b, buf_a, buf_b);
        uint32_t* const row = dst ? row_b : row_a;
#pragma unroll
        for (int d = 0; d < W; ++d) row[d * kDpThreads] = H[d];
        if (up_a) {
          best_a = rmax & 0xFFFFu;
          bi_a = i;
          buf_a = dst;
        }
        if (up_b) {
          best_b = rmax >> 16;
          bi_b = i;
          buf_b = dst;
        }
      }
      rowp += WQ * 32;
    }
#pragma unroll
    for (int d = 0; d + 1 < W; ++d) T[d] = T[d + 1];
    T[W - 1] = t_next;
    plo = plo_next;
    phi = phi_next;
    ca = ca_next;
    cb = cb_next;
  }
  int bd_a = 0, bd_b = 0;
  if constexpr (!TB) {
    best_a = best2 & 0xFFFFu;
    best_b = best2 >> 16;
  } else {  // first column of the best row holding the best value, per half
    bd_a = bi_a >= 0 ? W : -1;
    bd_b = bi_b >= 0 ? W : -1;
    const uint32_t* const ra = buf_a ? row_b : row_a;
    const uint32_t* const rb = buf_b ? row_b : row_a;
#pragma unroll 1
    for (int d = W - 1; d >= 0; --d) {
      if (bi_a >= 0 && (ra[d * kDpThreads] & 0xFFFFu) == best_a) bd_a = d;
      if (bi_b >= 0 && (rb[d * kDpThreads] >> 16) == best_b) bd_b = d;
    }
  }
  res[ta.slot] = stash(static_cast<int>(best_a - zero), TB ? bi_a : 0, bd_a);
  if (has_b) res[tb.slot] = stash(static_cast<int>(best_b - zero), TB ? bi_b : 0, bd_b);
  };
  for (int w = blockIdx.x; w * 32 < pairs; w = next_claim(claim)) {
    if (w * 32 + static_cast<int>(threadIdx.x) < pairs) align(w * 32 + threadIdx.x);
    __syncwarp();
  }
}

// W <= CH * LANES + 1: LANES consecutive lanes of a warp share one pair of
// alignments (A and B in the 16-bit halves, as in k_sw_u2), lane c holding band cells
// [CH c, CH c + CH) of the row in registers (the last lane also cell W - 1). Fewer cells a
// lane: more warps and a shorter row, but its fixed work (shuffles, codes, the best row) is
// paid for fewer cells, and the skew grows. Lane c works on
// row t - c at step t, so its left neighbour finished the same row one step earlier: the
// row's running F and H(left) arrive by one shuffle at the start of the step. The one value
// a lane needs from its right neighbour — H and E of the previous row at the neighbour's
// first cell (the E input of the lane's last cell) — is exactly what the neighbour
// computes first in the same step, so a second shuffle after each lane's first cell
// delivers it; every lane is busy on every step. Each lane tracks the first strict
// maximum of its own cells (best-row checkpoint in shared memory, as k_sw_u2), and the
// lanes of a pair combine (value, then earliest row, then smallest column) at the end:
// the first strict maximum of the whole band in row-major order. Pairs k_sw_u2 would
// hand to the int32 kernel are listed in fb the same way.
// With a row's codes taken by shuffles, additions spread over two pipes (cell2), the best rows
// saved by 16-byte stores and warps that claim their pairs, against loads by every lane in
// every row and a grid over the list, tracebacks: 58,000 tasks of 150 rows at W = 33 214 ->
// 179 us (now 8 cells a lane, before 32), 150,000 of 50 to 1,000 rows 924 -> 643 (8, before
// 16); 88,000 at W = 129 1,484 -> 1,154 (32); 4,001 of 1,000 to 5,000 rows at W = 65 1,732 ->
// 1,186 (4). At 8 cells a lane ALU and multiply-add pipe are each busy about 60 % of the time.
// Resident warps per SM (sw_wide_warps), same lists: 8 cells 16 / 20 / 24 warps 185 / 176 /
// 190 us; 32 cells 12 / 10 / 8 warps 1,333 / 1,311 / 1,200; 4 cells 20 / 24 1,262 / 1,218.
constexpr int sw_wide_warps(int cells) { return cells == 4 ? 24 : (cells == 8 ? 20 : (cells == 16 ? 12 : 8)); }
template <int W, int LANES, int CH, bool TB>
__global__ void __launch_bounds__(kDpThreads, TB ? sw_wide_warps(CH) : 1)
    k_sw_wide(const SwTask* __restrict__ tasks, int base, int n, const int* __restrict__ n_dev, int above, int upto,
              const uint8_t* __restrict__ qbase, const uint8_t* __restrict__ tbase, SwParams p,
              SwResult* __restrict__ res, uint32_t* __restrict__ dir, int rows_max, int* __restrict__ fb,
              int* __restrict__ claim) {
  static_assert(CH % 4 == 0, "a lane's cells fill whole direction words");
  static_assert(W <= CH * LANES + 1, "a band's cells have lanes");
  constexpr int WQ = (W + 3) / 4;
  // band column W - 1: an extra cell of the last lane, or cell kLastCell of lane kLastLane, past
  // which cells and lanes hold nothing
  constexpr bool kExtra = W == CH * LANES + 1;
  constexpr int kLastLane = kExtra ? LANES - 1 : (W - 1) / CH, kLastCell = kExtra ? CH : (W - 1) % CH;
  constexpr unsigned FULL = 0xffffffffu;
  if (n_dev && (*n_dev <= above || *n_dev > upto)) return;  // a list of another form's length
  __shared__ uint32_t s_prof[8];  // profile words of the five query codes
  if (threadIdx.x < 5) s_prof[threadIdx.x] = prof_biased(p, threadIdx.x);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int c = lane % LANES;  // chunk of this lane
  const int nn = n_dev ? min(n, *n_dev) : n, pairs = (nn - base + 1) / 2;
  const auto align = [&](const int lt) {  // lt: pair index within this launch
  const int ia = base + 2 * lt, ib = ia + 1;
  const bool live = lt < pairs, has_b = live && ib < nn;
  SwTask ta{}, tb{};
  if (live) ta = tasks[ia];
  if (has_b) tb = tasks[ib];
  else tb = ta, tb.qlen = 0;
  const int qmax = live ? max(ta.qlen, tb.qlen) : 0;
  const bool fits = qmax * p.match + 2 * (p.oe + p.ge + p.mismatch + p.ambig) < 16000 &&
                    p.match + kScoreBias <= 127 && p.mismatch <= kScoreBias && p.ambig <= kScoreBias;
  bool skip = !live;
  if (live && (!fits || window_has_n(ta, W, tbase) || (has_b && window_has_n(tb, W, tbase)))) {
    skip = true;
    if (c == 0) {
      const int k = atomicAdd(fb, has_b ? 2 : 1);
      fb[kFbList + k] = 2 * lt;
      if (has_b) fb[kFbList + 1 + k] = 2 * lt + 1;
    }
  }
  const int steps = __reduce_max_sync(FULL, skip ? 0 : qmax + LANES - 1);
  uint32_t* DP = TB ? pair_base(dir, 2 * lt, rows_max, WQ) : nullptr;
  const uint8_t* __restrict__ qa = qbase + ta.q_off;
  const uint8_t* __restrict__ qb = qbase + tb.q_off;
  const int qla = ta.qlen, qlb = tb.qlen;
  // called for pairs that run here only: both windows [0, qlen + W - 1) N-free and inside
  // their contigs, so column j reads its window at min(j, qlen + W - 2), a code in 0..3
  // (past a window's end it feeds N rows only), and the prmt selector of two codes is two
  // multiply-adds (as k_sw_u2)
  const uint8_t* __restrict__ wa = tbase + ta.t_start;
  const uint8_t* __restrict__ wb = tbase + tb.t_start;
  const int ja = ta.qlen + W - 2, jb = tb.qlen + W - 2;
  auto tc2 = [&](int j) {
    const uint32_t a = __ldg(wa + min(j, ja)), b = __ldg(wb + min(j, jb));
    return a * 17u + b * 4352u + 50304u;  // sel2(a, b)
  };
  auto qcode = [&](const uint8_t* __restrict__ q, int ql, int i) {
    return i >= 0 && i < ql ? min(static_cast<uint32_t>(q[i]), 4u) : 4u;
  };
  const int d0 = CH * c;  // band column of local cell 0
  const CellParams cp = cell_params(p);
  const uint32_t h_zero = kBias2 - cp.oe;  // H = 0
  uint32_t H[CH + 1], E[CH + 1], T[CH + 1];
#pragma unroll
  for (int k = 0; k <= CH; ++k) {
    H[k] = h_zero;
    E[k] = kBias2;
  }
#pragma unroll
  for (int k = 0; k <= CH; ++k) T[k] = skip ? 0u : tc2(d0 + k);  // row 0
  uint32_t best2 = h_zero;
  int bi_a = -1, bi_b = -1;
  extern __shared__ __align__(16) uint32_t sw_rows[];  // k_sw_wide stores 16 bytes at a time
  uint4* const row_a = reinterpret_cast<uint4*>(sw_rows) + threadIdx.x;  // cells 4g .. 4g + 3 at [g * kDpThreads]
  uint4* const row_b = row_a + CH / 4 * kDpThreads;
  uint32_t* const last_a = sw_rows + 2 * CH * kDpThreads + threadIdx.x;  // cell CH
  uint32_t* const last_b = last_a + kDpThreads;
  uint32_t hout = h_zero, fout = kBias2;  // this lane's last cell of its previous row
  // Codes. Narrow chunks (kStream) load them LANES steps at a time: at a block's first step
  // lane c holds the profile words of row t + c and the target column the last lane shifts in
  // at step t + c, loaded a block earlier; a step takes row i's words by a shuffle from lane
  // i mod LANES (rows before 0 are N rows), and the column entering a lane's window is the
  // right neighbour's T[2] (its row is one behind). Otherwise each lane loads its own row's
  // codes two steps and its profile words and column one step ahead.
  constexpr bool kStream = LANES >= 4;
  uint32_t plo, phi, x_qa, x_qb, x_ta = 0, x_tb = 0, old_lo = 0, old_hi = 0, cur_t = 0;
  const auto fetch = [&](int t) {
    x_qa = qcode(qa, qla, t + c);
    x_qb = qcode(qb, qlb, t + c);
    if (!skip) {
      const int j = t + c + 2 - LANES + LANES * CH;
      x_ta = __ldg(wa + min(j, ja));
      x_tb = __ldg(wb + min(j, jb));
    }
  };
  if constexpr (kStream) {
    plo = phi = s_prof[4];
    fetch(0);
  } else {
    // row -c of a lane that has not reached row 0 is N
    plo = s_prof[qcode(qa, qla, -c)];
    phi = s_prof[qcode(qb, qlb, -c)];
    x_qa = qcode(qa, qla, 1 - c);
    x_qb = qcode(qb, qlb, 1 - c);
  }
  const int end = skip || c > kLastLane ? 0 : qmax;
  uint32_t* dp = TB ? DP + (d0 >> 2) * 32 - c * (WQ * 32) : nullptr;  // row i's first word of this lane
  const auto step = [&](const int t, auto steady) {
    constexpr bool kSteady = decltype(steady)::value;
    const int i = t - c;
    [[maybe_unused]] const bool act = static_cast<unsigned>(i) < static_cast<unsigned>(end);
    // H, E and the target window advance once the lane has reached row 0 (rows past the
    // pair's end are N rows: they change no result and no code is stored for them); from
    // step LANES - 1 on every lane has, so the steady steps carry no per-cell guard
    const bool he_ok = kSteady || i >= 0;
    // row i's F and H(left) at column d0 - 1, from the left lane (its step t - 1)
    uint32_t hleft = __shfl_up_sync(FULL, hout, 1), f = __shfl_up_sync(FULL, fout, 1);
    if (c == 0) {
      hleft = h_zero;
      f = kBias2;
    }
    uint32_t lo, hi, t_next;
    if constexpr (kStream) {
      const int s = t & (LANES - 1);
      if (s == 0) {  // plo, phi: this block's words; old_lo, old_hi: the last one's
        old_lo = plo;
        old_hi = phi;
        plo = s_prof[x_qa];
        phi = s_prof[x_qb];
        cur_t = x_ta * 17u + x_tb * 4352u + 50304u;  // sel2
        fetch(t + LANES);
      }
      const bool now = c <= s;
      lo = __shfl_sync(FULL, now ? plo : old_lo, i, LANES);
      hi = __shfl_sync(FULL, now ? phi : old_hi, i, LANES);
      t_next = __shfl_down_sync(FULL, he_ok ? T[2] : T[1], 1);
      const uint32_t entering = __shfl_sync(FULL, cur_t, s, LANES);
      if (c == LANES - 1) t_next = entering;
    } else {
      lo = plo;
      hi = phi;
      plo = s_prof[x_qa];
      phi = s_prof[x_qb];
      x_qa = qcode(qa, qla, i + 2);
      x_qb = qcode(qb, qlb, i + 2);
      // past the pair's end the window shifts in a valid selector (code A for both): the
      // profile of an N row scores every target alike
      t_next = act ? tc2(i + 1 + d0 + CH) : sel2(0u, 0u);
    }
    // local cell 0, then hand (H, E) of it to the left lane: the E input of its last cell
    uint32_t rmax = 0, dw = 0, e0;
    const bool edge = !kExtra && c == kLastLane;
    const bool cut0 = kLastCell == 0 && edge;
    const uint32_t h0 = cell2<TB>(cp, H[0], prmt(lo, hi, T[0]), cut0 ? h_zero : H[1], cut0 ? kBias2 : E[1], hleft, f,
                                  e0, dw);
    uint32_t hdiag = H[1];  // past the band's edge a cell's diagonal is never used
    hleft = h0;
    // a lane that has not reached row 0 passes row -1's values (zero)
    uint32_t nh = __shfl_down_sync(FULL, he_ok ? h0 : h_zero, 1);
    uint32_t ne = __shfl_down_sync(FULL, he_ok ? e0 : kBias2, 1);
    if (kExtra && c == LANES - 1) {
      nh = H[CH];
      ne = E[CH];
    }
    if (he_ok) {
      H[0] = h0;
      E[0] = e0;
    }
    uint32_t& top = TB ? rmax : best2;  // the row's maximum (score only: the maximum so far)
    if (!kExtra) top = __vmaxu2(top, h0);
#pragma unroll
    for (int k = 1; k < CH + kExtra; ++k) {
      if (k == CH && c != LANES - 1) break;  // the extra cell W - 1 belongs to the last lane
      uint32_t hup = k == CH - 1 ? nh : (k == CH ? h_zero : H[k + 1]);
      uint32_t eup = k == CH - 1 ? ne : (k == CH ? kBias2 : E[k + 1]);
      if (k == kLastCell && edge) {
        hup = h_zero;
        eup = kBias2;
      }
      uint32_t e, code = 0;
      const uint32_t h = cell2<TB>(cp, hdiag, prmt(lo, hi, T[k]), hup, eup, hleft, f, e, code);
      if (he_ok) {
        H[k] = h;
        E[k] = e;
      }
      if constexpr (TB) {
        dw = insert_code(dw, code, k & 3);
        const bool inside = (kLastLane * CH + k) / 4 < WQ || c < kLastLane;
        if (((k & 3) == 3 || k == CH) && act && inside) dp[(k >> 2) * 32] = dw;
      }
      if (!kExtra) top = __vmaxu2(top, k > kLastCell && edge ? h_zero : h);
      else if (k & 1) top = __vimax3_u16x2(top, hleft, h);
      else if (k == CH) top = __vmaxu2(top, h);
      hleft = h;
      hdiag = hup;
    }
    hout = hleft;
    fout = f;
    if constexpr (TB) {
      if (act) {  // a strictly better row of this lane's cells
        const uint32_t b2 = __vmaxu2(best2, rmax), up = b2 ^ best2;
        best2 = b2;
        if (up & 0xFFFFu) {
          bi_a = i;
#pragma unroll
          for (int g = 0; g < CH / 4; ++g)
            row_a[g * kDpThreads] = make_uint4(H[4 * g], H[4 * g + 1], H[4 * g + 2], H[4 * g + 3]);
          *last_a = H[CH];
        }
        if (up >> 16) {
          bi_b = i;
#pragma unroll
          for (int g = 0; g < CH / 4; ++g)
            row_b[g * kDpThreads] = make_uint4(H[4 * g], H[4 * g + 1], H[4 * g + 2], H[4 * g + 3]);
          *last_b = H[CH];
        }
      }
      dp += WQ * 32;
    }
    if (he_ok) {
#pragma unroll
      for (int k = 0; k < CH; ++k) T[k] = T[k + 1];
      T[CH] = t_next;
    }
  };
  const int ramp = steps < LANES - 1 ? steps : LANES - 1;
  for (int t = 0; t < ramp; ++t) step(t, std::false_type{});
  for (int t = ramp; t < steps; ++t) step(t, std::true_type{});
  // combine the lanes of the pair: larger value, then earlier row, then smaller column
  uint64_t key_a, key_b;
  const int ncell = c == kLastLane ? kLastCell + 1 : CH;
  if constexpr (TB) {
    int bd_a = 0xFFF, bd_b = 0xFFF;
    const uint32_t best_a = best2 & 0xFFFFu, best_b = best2 >> 16;
#pragma unroll 1
    for (int k = ncell - 1; k >= 0; --k) {
      const uint32_t a = k == CH ? *last_a : reinterpret_cast<const uint32_t*>(row_a + (k >> 2) * kDpThreads)[k & 3];
      const uint32_t b = k == CH ? *last_b : reinterpret_cast<const uint32_t*>(row_b + (k >> 2) * kDpThreads)[k & 3];
      if (bi_a >= 0 && (a & 0xFFFFu) == best_a) bd_a = d0 + k;
      if (bi_b >= 0 && (b >> 16) == best_b) bd_b = d0 + k;
    }
    key_a = static_cast<uint64_t>(best_a) << 40 | static_cast<uint64_t>(0xFFFFFu - static_cast<uint32_t>(bi_a + 1)) << 12 |
            (0xFFFu - static_cast<uint32_t>(bd_a));
    key_b = static_cast<uint64_t>(best_b) << 40 | static_cast<uint64_t>(0xFFFFFu - static_cast<uint32_t>(bi_b + 1)) << 12 |
            (0xFFFu - static_cast<uint32_t>(bd_b));
  } else {
    key_a = c > kLastLane ? 0 : static_cast<uint64_t>(best2 & 0xFFFFu) << 40;
    key_b = c > kLastLane ? 0 : static_cast<uint64_t>(best2 >> 16) << 40;
  }
#pragma unroll
  for (int o = 1; o < LANES; o <<= 1) {
    const uint64_t xa = __shfl_xor_sync(FULL, key_a, o), xb = __shfl_xor_sync(FULL, key_b, o);
    key_a = xa > key_a ? xa : key_a;
    key_b = xb > key_b ? xb : key_b;
  }
  if (c != 0 || skip) return;
  const int zero = static_cast<int>(kBias) - p.oe;
  const auto unpack = [zero](uint64_t key) {
    const int best = static_cast<int>(key >> 40) - zero;
    const int bi = static_cast<int>(0xFFFFFu - static_cast<uint32_t>((key >> 12) & 0xFFFFFu)) - 1;
    const int bd = static_cast<int>(0xFFFu - static_cast<uint32_t>(key & 0xFFFu));
    return TB ? stash(best, bi, bd) : stash(best, 0, 0);
  };
  res[ta.slot] = unpack(key_a);
  if (has_b) res[tb.slot] = unpack(key_b);
  };
  constexpr int kPairs = 32 / LANES;
  for (int w = blockIdx.x; w * kPairs < pairs; w = next_claim(claim)) {
    align(w * kPairs + lane / LANES);
    __syncwarp();
  }
}

// The pairs k_sw_u2 listed, one alignment per thread, int32.
template <int W, bool TB>
__global__ void __launch_bounds__(kSwThreads) k_sw_fb(const SwTask* __restrict__ tasks, int base,
                                                      const uint8_t* __restrict__ qbase,
                                                      const uint8_t* __restrict__ tbase, SwParams p,
                                                      SwResult* __restrict__ res, uint32_t* __restrict__ dir,
                                                      int rows_max, const int* __restrict__ fb, int above) {
  constexpr int WQ = (W + 3) / 4;
  const int nfb = fb[0];
  if (nfb <= above) return;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < nfb; j += gridDim.x * blockDim.x) {
    const int lt = fb[kFbList + j];
    const SwTask tk = tasks[base + lt];
    res[tk.slot] = sw_one_reg<W, TB>(tk, qbase, tbase, p, TB ? pair_base(dir, lt, rows_max, WQ) : nullptr, lt & 1);
  }
}

// The tasks k_sw_u2 / k_sw_wide listed (an N in the target window, or outside the biased
// 16-bit range) for bands of W = CH * LANES + 1 columns, one alignment per LANES lanes in
// int32: lane c holds band columns [CH c, CH c + CH) (the last lane also column W - 1) and
// computes row t - c at step t — k_sw_wide's skewed wavefront, exchanging the left lane's
// last (H, F) and the right lane's first (H, E) by shuffles. Scores come from the 5-entry
// profile (N scored as the reference scores it), direction codes go to the task's half of
// the pair words, the best cell is the first strict maximum in row-major order: the same
// results and codes as sw_one_reg, which runs one alignment per thread and, at W = 129,
// spills its band to local memory. The list is short (windows that cross a contig end or
// an N run), so the kernel's time is one task's serial latency: narrow chunks (8 or 16
// cells per lane) spread a task over more lanes and shorten it.
template <int LANES, int CH, bool TB>
__global__ void __launch_bounds__(kSwThreads)
    k_sw_fb_lanes(const SwTask* __restrict__ tasks, int base, const uint8_t* __restrict__ qbase,
                  const uint8_t* __restrict__ tbase, SwParams p, SwResult* __restrict__ res,
                  uint32_t* __restrict__ dir, int rows_max, const int* __restrict__ fb, int above, int upto) {
  static_assert(CH % 4 == 0, "a lane's cells fill whole direction words");
  constexpr int W = CH * LANES + 1, WQ = (W + 3) / 4;
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int c = lane % LANES;
  const int nfb = fb[0];
  if (nfb <= above || nfb > upto) return;  // a list of another form's length
  const int stride = static_cast<int>(gridDim.x * blockDim.x / LANES);
  // a warp takes 32 / LANES consecutive entries of the fallback list per round (jw, the
  // first, is warp-uniform, so every lane takes the same rounds)
  for (int jw = static_cast<int>((blockIdx.x * blockDim.x + (threadIdx.x & ~31)) / LANES); jw < nfb; jw += stride) {
  const int j = jw + lane / LANES;  // entry of the fallback list
  const bool live = j < nfb;
  const int lt = live ? fb[kFbList + j] : 0;
  SwTask tk{};
  if (live) tk = tasks[base + lt];
  const int ql = live ? tk.qlen : 0;
  const int steps = __reduce_max_sync(FULL, live ? ql + LANES - 1 : 0);
  const uint8_t* __restrict__ q = qbase + tk.q_off;
  uint32_t* DP = TB ? pair_base(dir, lt, rows_max, WQ) : nullptr;
  const int half = lt & 1;
  const int d0 = CH * c;
  int H[CH + 2], E[CH + 2];
  uint32_t T[CH + 1];
#pragma unroll
  for (int k = 0; k < CH + 2; ++k) {
    H[k] = 0;
    E[k] = 0;
  }
#pragma unroll
  for (int k = 0; k <= CH; ++k) T[k] = live ? sel1(tcode(tbase, tk, d0 + k)) : sel1(4u);
  int best = 0, bi = -1, bd = -1;
  int hout = 0, fout = 0;  // this lane's last cell of its previous row
  for (int t = 0; t < steps; ++t) {
    const int i = t - c;
    const bool act = live && i >= 0 && i < ql;
    int hleft = __shfl_up_sync(FULL, hout, 1), f = __shfl_up_sync(FULL, fout, 1);
    if (c == 0) hleft = f = 0;
    const uint32_t qc = act ? min(static_cast<uint32_t>(q[i]), 4u) : 4u;
    const uint32_t plo = prof_lo(p, qc), phi = p.prof_n;
    const uint32_t t_next = act ? sel1(tcode(tbase, tk, static_cast<int64_t>(i) + 1 + d0 + CH)) : sel1(4u);
    int hdiag = H[0], rmax = 0, rk = 0;
    uint32_t dw = 0;
    int h0, e0;
    {
      const int hup = H[1], eup = E[1];
      const int hd = hdiag + static_cast<int>(prmt(plo, phi, T[0]));
      const int eo = hup - p.oe, ee = eup - p.ge, fo = hleft - p.oe, fe = f - p.ge;
      e0 = max(eo, ee);
      f = max(fo, fe);
      const int m1 = max(hd, e0);
      h0 = max(max(m1, f), 0);
      if constexpr (TB) dw = dir_code32(hd >= e0 && m1 >= f, m1 >= f, eo >= ee, fo >= fe);
      rmax = h0;
      hleft = h0;
      hdiag = hup;
    }
    // a lane that has not reached row 0 passes row -1's values (zero)
    int nh = __shfl_down_sync(FULL, i >= 0 ? h0 : 0, 1);
    int ne = __shfl_down_sync(FULL, i >= 0 ? e0 : 0, 1);
    if (c == LANES - 1) {
      nh = H[CH];
      ne = E[CH];
    }
    if (act) {
      H[0] = h0;
      E[0] = e0;
    }
#pragma unroll
    for (int k = 1; k <= CH; ++k) {
      if (k == CH && c != LANES - 1) break;  // the extra cell W - 1 belongs to the last lane
      const int hup = k == CH - 1 ? nh : (k == CH ? 0 : H[k + 1]);
      const int eup = k == CH - 1 ? ne : (k == CH ? 0 : E[k + 1]);
      const int hd = hdiag + static_cast<int>(prmt(plo, phi, T[k]));
      const int eo = hup - p.oe, ee = eup - p.ge, fo = hleft - p.oe, fe = f - p.ge;
      const int e = max(eo, ee);
      f = max(fo, fe);
      const int m1 = max(hd, e);
      const int h = max(max(m1, f), 0);
      if (act) {
        H[k] = h;
        E[k] = e;
      }
      if constexpr (TB) {
        dw |= dir_code32(hd >= e && m1 >= f, m1 >= f, eo >= ee, fo >= fe) << (k & 3);
        if ((k & 3) == 3) {
          if (act) reinterpret_cast<uint16_t*>(DP + (static_cast<size_t>(i) * WQ + ((d0 + k) >> 2)) * 32)[half] =
              static_cast<uint16_t>(dw);
          dw = 0;
        } else if (k == CH) {  // cell W - 1 opens the last, partial word
          if (act) reinterpret_cast<uint16_t*>(DP + (static_cast<size_t>(i) * WQ + ((d0 + k) >> 2)) * 32)[half] =
              static_cast<uint16_t>(dw);
        }
        if (h > rmax) {  // first strict maximum of the lane's part of the row
          rmax = h;
          rk = k;
        }
      } else {
        rmax = max(rmax, h);
      }
      hleft = h;
      hdiag = hup;
    }
    hout = hleft;
    fout = f;
    if (act) {
      if (rmax > best) {
        best = rmax;
        bi = i;
        bd = d0 + rk;
      }
#pragma unroll
      for (int k = 0; k < CH; ++k) T[k] = T[k + 1];
      T[CH] = t_next;
    }
  }
  // the lanes of the alignment: larger value, then earlier row, then smaller column (rows and
  // scores here pass 2^20 and 2^24, so a key holds 32 bits of each and the column goes beside it)
  uint64_t key = static_cast<uint64_t>(best) << 32 | ~static_cast<uint32_t>(bi + 1);
#pragma unroll
  for (int o = 1; o < LANES; o <<= 1) {
    const uint64_t xk = __shfl_xor_sync(FULL, key, o);
    const int xd = __shfl_xor_sync(FULL, bd, o);
    if (xk > key || (xk == key && xd < bd)) {
      key = xk;
      bd = xd;
    }
  }
  if (c == 0 && live) {
    const int kb = static_cast<int>(key >> 32), kbi = static_cast<int>(~static_cast<uint32_t>(key)) - 1;
    res[tk.slot] = TB ? stash(kb, kbi, bd) : stash(kb, 0, 0);
  }
  }
}

// Traceback of every task of the launch from the stashed best cell (the DP kernels are done
// with the scratch), src/align.cpp:87-143. A walk is a chain of dependent memory latencies,
// so kWalkLanes lanes share a task: on a diagonal run lane l fetches the codes and bases of
// rows i - 8l .. i - 8l - 7, a prefix sum over the lanes gives each the score its block
// starts from, and all leading blocks that are diagonal throughout, with the score above
// what their steps can use up, are taken at once, 64 rows per memory latency instead of 8.
// The first block that is not is stepped through by its lane as the one-cell walk would.
// Against one thread per task: 4,001 reads of 1-5 kbp 1,789 -> 236 us, 200,003 of 50-1000 bp
// 398 -> 258, 64 of 100-300 bp 43 -> 17. Where short walks fill the SMs by themselves
// (262,144 of 150 bp) the lanes' extra instructions cost more than the latencies they hide
// (122 -> 181 us), so those run one thread per task. Short lists take a warp per task, 256 rows
// per latency: 4,001 of 1-5 kbp 222 -> 82 us, 64 of 100-300 bp 17 -> 11; 8 lanes against 32, of
// 150 rows 19 and 17 us at 4,096, 21 and 23 at 8,192, of 1,000 rows 62 and 53 at 8,192, 84 and 95
// at 16,384.
constexpr int kWalkLanes = 8;
constexpr int kWalkMany = 98304, kWalkShort = 256;  // more tasks of at most this many rows: one thread each
constexpr int kWalkFew = 6144;                      // up to this many tasks: a warp each

// The walks of tasks [base, base + nn), G lanes each.
template <int W, int G>
__device__ __forceinline__ void walk_lanes(const SwTask* __restrict__ tasks, int base, int nn,
                                           const uint8_t* __restrict__ qbase, const uint8_t* __restrict__ tbase,
                                           const SwParams& p, SwResult* __restrict__ res,
                                           const uint32_t* __restrict__ dir, int rows_max, uint32_t* __restrict__ cig,
                                           const int64_t* __restrict__ cig_off, uint32_t* __restrict__ err) {
  constexpr int WQ = (W + 3) / 4;
  const int lane = threadIdx.x & 31, gl = lane & (G - 1);
  const unsigned gm = (G == 32 ? 0xffffffffu : (1u << (G & 31)) - 1u) << (lane & ~(G - 1));
  const int smax = max(p.match, max(-p.mismatch, -p.ambig));  // the most one step can lower v
  const int stride = static_cast<int>(gridDim.x * blockDim.x) / G;
  for (int lt = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x) / G; lt < nn; lt += stride) {
    const SwTask tk = tasks[base + lt];
    const SwResult s = res[tk.slot];
    __syncwarp(gm);  // every lane has the best cell before the group's first lane overwrites it
    SwResult r{s.score, 0, 0, 0, 0, 0, 0, 0};
    if (s.score > 0) {
      const PairCodes code{pair_base(const_cast<uint32_t*>(dir), lt, rows_max, WQ), WQ, lt & 1};
      const uint8_t* __restrict__ q = qbase + tk.q_off;
      const int cap = 2 * tk.qlen + 1;
      CigarWriter cw{cig + cig_off[tk.slot], gl == 0 ? cap : 0, 0, 0xFu, 0};  // the first lane writes
      int i = s.qb, d = s.qe, v = s.score, nm = 0;
      bool broken = d < 0 || d >= W || i >= tk.qlen;
      while (!broken) {
        int run = 0;
        uint32_t x = 0;
        bool stop = false;
        while (!stop && i >= 0 && v > 0) {
          const int top = i - kAhead * gl;  // this lane's block: rows top, top - 1, .. top - 7
          const int sh = code.shift(d);
          uint32_t cx = 0;  // row top - k of the block: kNotDiag in bit k, kNotE in bit 8 + k
          uint64_t qw = 0, tw = 0;  // its bases, row top - k in byte 7 - k; N past any end
          int lost = 0;             // what the block takes from v, times 1,024, and its mismatches
          bool clean = false;
          if (top >= 0) {
            const int64_t x0 = tk.t_start + (top - (kAhead - 1)) + d;  // target of row top - 7
            if (top >= kAhead - 1 && x0 >= tk.t_lo && x0 + kAhead <= tk.t_hi) {
              qw = load8u(q + top - (kAhead - 1));
              tw = load8u(tbase + x0);
#pragma unroll
              for (int k = 0; k < kAhead; ++k) cx |= ((code.word(top - k, d) >> sh) & (kNotDiag | kNotE)) << k;
              clean = (cx & 0xFFu) == 0;
              // bytes equal and both below 4: match; either above 3: ambiguous; else mismatch
              const uint64_t ok_amb = zero_bytes((qw | tw) & 0xFCFCFCFCFCFCFCFCull);
              const int n_match = __popcll(zero_bytes(qw ^ tw) & ok_amb);
              const int n_amb = kAhead - __popcll(ok_amb);
              lost = (n_match * p.match - (kAhead - n_match - n_amb) * p.mismatch - n_amb * p.ambig) * 1024 +
                     (kAhead - n_match);
            } else {
#pragma unroll
              for (int k = 0; k < kAhead; ++k) {
                if (top - k >= 0) {
                  cx |= (code(top - k, d) & (kNotDiag | kNotE)) << k;
                  qw |= static_cast<uint64_t>(q[top - k]) << (8 * (kAhead - 1 - k));
                  tw |= static_cast<uint64_t>(tcode(tbase, tk, static_cast<int64_t>(top - k) + d))
                        << (8 * (kAhead - 1 - k));
                }
              }
            }
          }
          int sum = lost;  // inclusive prefix over the lanes (mismatches stay below 1,024)
#pragma unroll
          for (int o = 1; o < G; o <<= 1) {
            const int y = __shfl_up_sync(gm, sum, o, G);
            if (gl >= o) sum += y;
          }
          const int before = (sum - lost) >> 10;  // the arithmetic shift drops the mismatches
          const bool take = clean && v - before > (kAhead - 1) * smax;
          const unsigned not_ok = (__ballot_sync(gm, !take) & gm) >> (lane & ~(G - 1));
          const int c = not_ok ? __ffs(not_ok) - 1 : G;
          if (c > 0) {
            const int t = __shfl_sync(gm, sum, c - 1, G);
            v -= t >> 10;
            nm += t & 1023;
            run += kAhead * c;
            i -= kAhead * c;
          }
          if (c == G) continue;
          if (gl == c) {  // top == i
#pragma unroll 1
            for (int k = 0; k < kAhead; ++k) {
              if (i < 0 || v <= 0) {
                stop = true;
                break;
              }
              x = cx >> k;
              if (x & kNotDiag) {  // not from the diagonal
                stop = true;
                break;
              }
              const int qa = static_cast<int>((qw >> (8 * (kAhead - 1 - k))) & 0xFFu);
              const int t8 = static_cast<int>((tw >> (8 * (kAhead - 1 - k))) & 0xFFu);
              const int tt = t8 > 3 ? 4 : t8;
              v -= sub_score(p, qa, tt);
              nm += (qa != tt || qa > 3) ? 1 : 0;
              ++run;
              --i;
            }
          }
          i = __shfl_sync(gm, i, c, G);
          v = __shfl_sync(gm, v, c, G);
          nm = __shfl_sync(gm, nm, c, G);
          run = __shfl_sync(gm, run, c, G);
          x = __shfl_sync(gm, x, c, G);
          stop = __shfl_sync(gm, static_cast<int>(stop), c, G) != 0;
        }
        if (run && gl == 0) cw.push(0u /* M */, run);
        if (i < 0 || v <= 0) break;
        run = 0;
        bool ext = true;
        if (!(x & kNotE)) {  // from E, an insertion: E(i,d) <- (i-1, d+1)
          while (ext) {
            if (i < 0 || d >= W) {
              broken = true;
              break;
            }
            ext = (code(i, d) & kExtE) != 0;
            v += ext ? p.ge : p.oe;
            ++run;
            --i;
            ++d;
          }
          if (!broken && gl == 0) cw.push(1u /* I */, run);
        } else {  // from F, a deletion: F(i,d) <- (i, d-1)
          while (ext) {
            if (d < 0 || d >= W) {
              broken = true;
              break;
            }
            ext = (code(i, d) & kExtF) != 0;
            v += ext ? p.ge : p.oe;
            ++run;
            --d;
          }
          if (!broken && gl == 0) cw.push(2u /* D */, run);
        }
        nm += run;
        broken = broken || (i >= 0 && v > 0 && (d < 0 || d >= W));
      }
      if (gl == 0) {
        if (broken) atomicOr(err, kErrTracebackBounds);
        cw.flush();
        if (cw.n > cap) atomicOr(err, kErrCigarOverflow);
        r.qb = i + 1;
        r.tb = i + 1 + d;
        r.qe = s.qb + 1;
        r.te = s.qb + s.qe + 1;
        r.nm = nm;
        r.n_ops = cw.n < cap ? cw.n : cap;
      }
    }
    if (gl == 0) res[tk.slot] = r;
  }
}

template <int W>
__global__ void __launch_bounds__(kSwThreads, 7) k_sw_walk(const SwTask* __restrict__ tasks, int base, int count, int n,
                                                        const int* __restrict__ n_dev,
                                                        const uint8_t* __restrict__ qbase,
                                                        const uint8_t* __restrict__ tbase, SwParams p,
                                                        SwResult* __restrict__ res, const uint32_t* __restrict__ dir,
                                                        int rows_max, uint32_t* __restrict__ cig,
                                                        const int64_t* __restrict__ cig_off,
                                                        uint32_t* __restrict__ err) {
  constexpr int WQ = (W + 3) / 4;
  const int nn = min(base + count, n_dev ? min(n, *n_dev) : n) - base;  // tasks of this launch
  if (rows_max <= kWalkShort && nn > kWalkMany) {  // the launch has a thread per task then
    const int lt = blockIdx.x * blockDim.x + threadIdx.x;
    if (lt >= nn) return;
    const SwTask tk = tasks[base + lt];
    const SwResult s = res[tk.slot];
    SwResult r{s.score, 0, 0, 0, 0, 0, 0, 0};
    if (s.score > 0) {
      const PairCodes codes{pair_base(const_cast<uint32_t*>(dir), lt, rows_max, WQ), WQ, lt & 1};
      traceback(codes, W, s.qb, s.qe, s.score, qbase + tk.q_off, tbase, tk, p, r, cig + cig_off[tk.slot],
                2 * tk.qlen + 1, err);
    }
    res[tk.slot] = r;
    return;
  }
  if (nn <= kWalkFew) walk_lanes<W, 32>(tasks, base, nn, qbase, tbase, p, res, dir, rows_max, cig, cig_off, err);
  else walk_lanes<W, kWalkLanes>(tasks, base, nn, qbase, tbase, p, res, dir, rows_max, cig, cig_off, err);
}

// Any band width and any scores: one alignment per thread, int32, band rows H, E in
// per-warp scratch, lane-interleaved ([d][lane]); walks its own traceback.
template <bool TB>
__global__ void __launch_bounds__(kSwThreads) k_sw_any(const SwTask* __restrict__ tasks, int base, int n,
                                                       const int* __restrict__ n_dev,
                                                       const uint8_t* __restrict__ qbase,
                                                       const uint8_t* __restrict__ tbase, SwParams p,
                                                       SwResult* __restrict__ res, uint32_t* __restrict__ dir,
                                                       int rows_max, uint32_t* __restrict__ cig,
                                                       const int64_t* __restrict__ cig_off, int* __restrict__ band,
                                                       uint32_t* __restrict__ err) {
  const int W = p.W, WW = (W + 7) / 8;
  const int lt = blockIdx.x * blockDim.x + threadIdx.x;  // index within this launch
  const int gt = base + lt;
  if (gt >= (n_dev ? min(n, *n_dev) : n)) return;
  const int lane = threadIdx.x & 31;
  const SwTask tk = tasks[gt];
  const uint8_t* __restrict__ q = qbase + tk.q_off;
  const int ql = tk.qlen;
  uint32_t* D = TB ? dir + (static_cast<size_t>(lt >> 5) * rows_max * WW) * 32 + lane : nullptr;
  int* Hs = band + static_cast<size_t>(lt >> 5) * 2 * (W + 1) * 32 + lane;
  int* Es = Hs + static_cast<size_t>(W + 1) * 32;
  for (int d = 0; d <= W; ++d) {
    Hs[d * 32] = 0;
    Es[d * 32] = 0;
  }
  int best = 0, bi = -1, bd = -1;
  for (int i = 0; i < ql; ++i) {
    const int qc = min(static_cast<int>(q[i]), 4);
    int f = 0, hleft = 0, hdiag = Hs[0], rmax = 0, rd = -1;
    uint32_t dw = 0;
    for (int d = 0; d < W; ++d) {
      const int hup = Hs[(d + 1) * 32], eup = Es[(d + 1) * 32];
      const int tc = static_cast<int>(tcode(tbase, tk, static_cast<int64_t>(i) + d));
      const int hd = hdiag + sub_score(p, qc, tc);
      const int eo = hup - p.oe, ee = eup - p.ge, fo = hleft - p.oe, fe = f - p.ge;
      const int e = max(eo, ee);
      f = max(fo, fe);
      const int m1 = max(hd, e);
      const int h = max(max(m1, f), 0);
      Hs[d * 32] = h;
      Es[d * 32] = e;
      if (TB) {
        dw |= dir_code32<WordCodes::kStep>(hd >= e && m1 >= f, m1 >= f, eo >= ee, fo >= fe) << (d & 7);
        if ((d & 7) == 7 || d == W - 1) {
          D[(static_cast<size_t>(i) * WW + (d >> 3)) * 32] = dw;
          dw = 0;
        }
        if (d == 0 || h > rmax) {
          rmax = h;
          rd = d;
        }
      } else {
        best = max(best, h);
      }
      hleft = h;
      hdiag = hup;
    }
    if (TB && rmax > best) {
      best = rmax;
      bi = i;
      bd = rd;
    }
  }
  SwResult r{best, 0, 0, 0, 0, 0, 0, 0};
  if (TB && best > 0)
    traceback(WordCodes{D, WW}, W, bi, bd, best, q, tbase, tk, p, r, cig + cig_off[tk.slot], 2 * ql + 1, err);
  res[tk.slot] = r;
}

// What a launch hands to its kernels.
struct SwLaunch {
  cudaStream_t st;
  bool tb;
  const SwTask* tasks;
  int base, count, n;
  const int* n_dev;
  const uint8_t* qbase;
  const uint8_t* tbase;
  const SwParams& p;
  SwResult* res;
  uint32_t* dir;
  int rows_max;
  uint32_t* cig;
  const int64_t* cig_off;
  int* fb;
  uint32_t* err;
  const KernelTrace& kt;
};

// Cells per lane of kSwIntraNarrow: 8 against 16, 58,000 tracebacks of 150 rows at W = 33 188
// and 212 us; 88,000 of 50 to 1,000 rows at W = 129 1,871 and 1,307.
constexpr int sw_narrow_cells(int W) { return W == 129 ? 16 : 8; }

// Bands of registers with the forms of 32 and of fewer cells per lane.
constexpr bool sw_has_intra(int W) { return W == 33 || W == 65 || W == 129; }
constexpr bool sw_has_narrow(int W) { return W == 43 || sw_has_intra(W); }

// Lanes per pair at `cells` a lane: a power of two, the last one with a cell more if need be.
constexpr int sw_lanes(int W, int cells) {
  int l = 1;
  while (cells * l + 1 < W) l *= 2;
  return l;
}

// Blocks of one warp for `warps` claims: all of them, up to what is resident.
template <class Kernel>
int dp_blocks(int64_t warps, Kernel* kernel, int smem, std::atomic<int>* resident) {
  int dev = 0, v = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices) {
    v = resident[dev].load(std::memory_order_relaxed);
    if (v <= 0 && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, kernel, kDpThreads, smem) == cudaSuccess && v > 0)
      resident[dev].store(v, std::memory_order_relaxed);
  }
  cudaGetLastError();
  return static_cast<int>(std::min<int64_t>(warps, int64_t{v > 0 ? v : 8} * device_sm_count()));
}

template <int W, int CH>
void run_wide(const SwLaunch& a, int count, int above, int upto) {
  constexpr int LANES = sw_lanes(W, CH);
  const int64_t pairs = (static_cast<int64_t>(count) + 1) / 2;
  int* const claim = a.fb + (upto == INT_MAX ? 2 : 1);
  const auto run = [&](auto* kernel, int smem, std::atomic<int>* resident) {
    kernel<<<dp_blocks((pairs * LANES + 31) / 32, kernel, smem, resident), kDpThreads, smem, a.st>>>(
        a.tasks, a.base, a.n, a.n_dev, above, upto, a.qbase, a.tbase, a.p, a.res, a.dir, a.rows_max, a.fb,
        claim);
  };
  constexpr int kRowBytes = 2 * (CH + 1) * kDpThreads * 4;  // the two saved best rows of each lane
  static std::atomic<int> resident[2][kMaxDevices];
  a.kt.begin(a.st, a.tb ? "k_sw_wide<tb>" : "k_sw_wide<score>");
  if (a.tb) run(k_sw_wide<W, LANES, CH, true>, kRowBytes, resident[1]);
  else run(k_sw_wide<W, LANES, CH, false>, 0, resident[0]);
  a.kt.end(a.st);
}

template <int W>
void run_u2(const SwLaunch& a, int above) {
  const auto run = [&](auto* kernel, int smem, std::atomic<int>* resident) {
    const int64_t warps = ((static_cast<int64_t>(a.count) + 1) / 2 + 31) / 32;
    kernel<<<dp_blocks(warps, kernel, smem, resident), kDpThreads, smem, a.st>>>(
        a.tasks, a.base, a.n, a.n_dev, above, a.qbase, a.tbase, a.p, a.res, a.dir, a.rows_max, a.fb, a.fb + 2);
  };
  constexpr int kRowBytes = 2 * W * kDpThreads * 4;  // the two saved best rows of each thread
  static_assert(kRowBytes <= 48 * 1024);
  static std::atomic<int> resident[2][kMaxDevices];
  a.kt.begin(a.st, a.tb ? "k_sw_u2<tb>" : "k_sw_u2<score>");
  if (a.tb) run(k_sw_u2<W, true>, kRowBytes, resident[1]);
  else run(k_sw_u2<W, false>, 0, resident[0]);
  a.kt.end(a.st);
}

// The int32 kernel over the listed tasks. The list's length is known on the device only
// (usually short or empty), so the kernels stride over it with a few resident waves. A short
// list's time is one task's serial latency, so four cells a lane, whose row is the shortest; a
// longer one's is its instructions: 8 or 16 cells, or a thread per task. Tracebacks of 150
// rows, us, short form against the other: W = 17 54 and 89 for 500 tasks, 91 and 93 for 12,000,
// 111 and 95 for 16,000; W = 33 54 and 74 for 500, 89 and 103 for 6,000, 111 and 105 for 8,000;
// W = 65 54 and 105, 91 and 107 for 3,000, 115 and 107 for 4,000; W = 129 60 and 105, 105 and 105
// for 1,500, 132 and 107 for 2,000 (rows of 1,000 and scores alone cross at the same lengths).
// (One kernel with both forms ran the longer lists 5 to 45 % slower.)
template <int W>
int run_fb(const SwLaunch& a) {  // the kernels launched
  constexpr bool kShort = (W - 1) % 4 == 0, kLanes = W == 33 || W == 65 || W == 129;
  constexpr int CH = W == 33 ? 8 : 16;
  const int few = kShort ? 196608 / (W - 1) : 0;
  const auto grid = [&](int lanes) {
    return std::min(8 * device_sm_count(),
                    static_cast<int>((static_cast<int64_t>(a.count) * lanes + kSwThreads - 1) / kSwThreads));
  };
  const auto lanes = [&](auto kernel, int l, int above, int upto) {
    kernel<<<grid(l), kSwThreads, 0, a.st>>>(a.tasks, a.base, a.qbase, a.tbase, a.p, a.res, a.dir, a.rows_max, a.fb,
                                             above, upto);
  };
  a.kt.begin(a.st, a.tb ? "k_sw_fb<tb>" : "k_sw_fb<score>");
  if constexpr (kShort) {
    constexpr int L = (W - 1) / 4;
    a.tb ? lanes(k_sw_fb_lanes<L, 4, true>, L, 0, few) : lanes(k_sw_fb_lanes<L, 4, false>, L, 0, few);
  }
  if (a.count > few) {
    if constexpr (kLanes) {
      constexpr int L = (W - 1) / CH;
      a.tb ? lanes(k_sw_fb_lanes<L, CH, true>, L, few, INT_MAX) : lanes(k_sw_fb_lanes<L, CH, false>, L, few, INT_MAX);
    } else {
      const auto run = [&](auto kernel) {
        kernel<<<grid(1), kSwThreads, 0, a.st>>>(a.tasks, a.base, a.qbase, a.tbase, a.p, a.res, a.dir, a.rows_max,
                                                 a.fb, few);
      };
      a.tb ? run(k_sw_fb<W, true>) : run(k_sw_fb<W, false>);
    }
  }
  a.kt.end(a.st);
  return (kShort ? 1 : 0) + (a.count > few ? 1 : 0);
}

// One band width: the form for short lists (few > 0: it takes a device count of at most
// `few`, the main form any other), the main form, the int32 kernel, the walk. Returns the kernels
// launched.
template <int W>
int launch_band(const SwLaunch& a, SwForm form, int few) {
  cudaMemsetAsync(a.fb, 0, kFbList * sizeof(int), a.st);
  int launched = 1;  // the main form
  if (form == kSwIntraFew) {
    run_wide<W, 4>(a, a.count, 0, INT_MAX);
  } else if (few > 0) {
    run_wide<W, 4>(a, std::min(a.count, few), 0, few);
    ++launched;
  }
  if constexpr (sw_has_intra(W)) {
    if (form == kSwIntra) run_wide<W, 32>(a, a.count, few, INT_MAX);
  }
  if constexpr (sw_has_narrow(W)) {
    if (form == kSwIntraNarrow) run_wide<W, sw_narrow_cells(W)>(a, a.count, few, INT_MAX);
  }
  if constexpr (W != 129) {
    if (form == kSwInter) run_u2<W>(a, few);
  }
  launched += run_fb<W>(a);
  if (a.tb) {
    const int lane_blocks = std::min(
        16 * device_sm_count(),
        static_cast<int>((static_cast<int64_t>(a.count) * 32 + kSwThreads - 1) / kSwThreads));
    const int blocks = a.rows_max <= kWalkShort && a.count > kWalkMany
                           ? std::max(lane_blocks, (a.count + kSwThreads - 1) / kSwThreads)
                           : lane_blocks;
    a.kt.begin(a.st, "k_sw_walk");
    k_sw_walk<W><<<blocks, kSwThreads, 0, a.st>>>(a.tasks, a.base, a.count, a.n, a.n_dev, a.qbase, a.tbase, a.p,
                                                  a.res, a.dir, a.rows_max, a.cig, a.cig_off, a.err);
    a.kt.end(a.st);
    ++launched;
  }
  return launched;
}

}  // namespace

bool sw_bytes_ok(const dnaln_score_params& s) {
  return s.match <= 127 && s.mismatch <= 128 && s.ambig <= 128 && s.match >= -128;
}

bool sw_band_in_registers(int W) { return W == 11 || W == 17 || W == 33 || W == 43 || W == 65 || W == 129; }

bool sw_uses_generic(int W, bool bytes_ok) { return !(bytes_ok && sw_band_in_registers(W)); }

SwParams make_sw_params(const dnaln_score_params& s) {
  SwParams p;
  p.match = s.match;
  p.mismatch = s.mismatch;
  p.oe = s.gap_open + s.gap_ext;
  p.ge = s.gap_ext;
  p.ambig = s.ambig;
  p.bw = s.bw;
  p.W = 2 * s.bw + 1;
  p.prof_n = static_cast<uint32_t>(static_cast<uint8_t>(-s.ambig)) * 0x01010101u;
  p.one = 1u;
  p.mone = 0u - 1u;
  return p;
}

size_t sw_dir_bytes_per_task(int W, int rows_max) {
  const size_t pair = static_cast<size_t>((W + 3) / 4) * 2, nib = static_cast<size_t>((W + 7) / 8) * 4;
  return static_cast<size_t>(rows_max > 0 ? rows_max : 1) * (pair > nib ? pair : nib);
}

size_t sw_band_bytes_per_task(int W, bool bytes_ok) {
  return sw_uses_generic(W, bytes_ok) ? static_cast<size_t>(2) * (W + 1) * sizeof(int) : 0;
}

// Up to this many tasks the form of four cells per lane is the fastest: its row step is the
// shortest serial chain, and a short list leaves lanes idle anyway. Measured against the
// best other form, us for 150-row tracebacks: W = 33 51 against 67 at 1,024 tasks, 94
// against 91 at 16,384; W = 65 51 against 64 and, at 8,192, 97 against 85; W = 129 57
// against 90 and, at 4,096, 117 against 95; W = 17 55 against 92 and, at 32,768, 99
// against 97; W = 43 44 against 58 and, at 8,192, 86 against 77; W = 11 50 against 69 and, at
// 32,768, 91 against 74.
int sw_few_tasks(int W) {
  switch (W) {
    case 11: return 20480;
    case 17: return 28672;
    case 33: return 14336;
    case 43: return 5120;
    case 65: return 4608;
    default: return 3072;  // 129
  }
}

bool sw_has_form(int W, bool bytes_ok, SwForm form) {
  if (sw_uses_generic(W, bytes_ok)) return form == kSwInter;
  switch (form) {
    case kSwInter: return W != 129;
    case kSwIntra: return sw_has_intra(W);
    case kSwIntraNarrow: return sw_has_narrow(W);
    case kSwIntraFew: return true;
    default: return false;
  }
}

int sw_lanes_per_pair(int W, SwForm form) {
  if (form == kSwIntra) return sw_lanes(W, 32);
  if (form == kSwIntraNarrow) return sw_lanes(W, sw_narrow_cells(W));
  if (form == kSwIntraFew) return sw_lanes(W, 4);
  return 1;
}

int launch_sw(cudaStream_t st, bool tb, bool bytes_ok, const SwTask* tasks, int base, int count, int n,
              const int* n_dev, const uint8_t* qbase, const uint8_t* tbase, const SwParams& p, SwResult* res,
              uint32_t* dir, int rows_max, uint32_t* cig, const int64_t* cig_off, int* band, int* fb, uint32_t* err,
              const KernelTrace* kt, SwForm form, int few) {
  if (count <= 0) return 0;
  const bool generic = sw_uses_generic(p.W, bytes_ok);
  if ((tb && !dir) || (generic && !band) || (!generic && !fb) || (base % kSwTaskGroup) != 0) return -1;
  // the kernels bound their tasks by n (and the device count): a launch covers tasks
  // [base, base + count) only, so that no thread of a grid rounded up past `count` takes a
  // task of the next chunk, whose scratch this launch does not hold
  if (n > base + count) n = base + count;
  if (!generic) {
    const KernelTrace none;
    const SwLaunch a{st, tb,  tasks,    base, count,   n,  n_dev, qbase, tbase,
                     p,  res, dir,      rows_max, cig, cig_off, fb, err, kt ? *kt : none};
    if (!sw_has_form(p.W, bytes_ok, form)) form = p.W == 129 ? kSwIntra : kSwInter;
    if (!sw_has_form(p.W, bytes_ok, kSwIntraFew)) few = 0;
    switch (p.W) {
      case 11: return launch_band<11>(a, form, few);
      case 17: return launch_band<17>(a, form, few);
      case 33: return launch_band<33>(a, form, few);
      case 43: return launch_band<43>(a, form, few);
      case 65: return launch_band<65>(a, form, few);
      case 129: return launch_band<129>(a, form, few);
      default: break;
    }
  }
  const int blocks = (count + kSwThreads - 1) / kSwThreads;
  if (kt) kt->begin(st, tb ? "k_sw_any<tb>" : "k_sw_any<score>");
  if (tb)
    k_sw_any<true><<<blocks, kSwThreads, 0, st>>>(tasks, base, n, n_dev, qbase, tbase, p, res, dir, rows_max, cig,
                                                 cig_off, band, err);
  else
    k_sw_any<false><<<blocks, kSwThreads, 0, st>>>(tasks, base, n, n_dev, qbase, tbase, p, res, dir, rows_max, cig,
                                                  cig_off, band, err);
  if (kt) kt->end(st);
  return 1;
}

}  // namespace dnb
