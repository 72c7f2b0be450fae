// seed_colinear.cu — seeding and chaining of the reads whose anchors form one colinear
// chain (sm_100a): sketch, probe and, instead of storing, sorting and chaining the anchors,
// a check as they arrive that the reference's chaining (src/chain.cpp:12-69) can only give
// that one chain. Every other read is listed for the kernels that run the DP in full
// (seed_thread.cu, seed_long.cu, seed.cu).
//
// The check. A read's anchors split into the main ones and at most kMaxStray strays. The
// main ones share a strand and are strictly monotone in both coordinates; each consecutive
// pair is a valid predecessor (dr in (0, max_gap], |dr - dq| <= band) with a gain g =
// min(dq, dr, k) - cost(|dr - dq|) >= 1. No stray makes a valid pair with a main anchor:
// another strand, more than max_gap away, or more than band diagonals off (|dr - dq| is the
// difference of the two anchors' diagonals rpos - qpos). A stray that sorts between main
// anchors only takes a place of their lookback, so there are fewer strays than the lookback
// is long. Let
// G(j, i) be the gains summed from anchor j to anchor i. The DP's choice for i is i - 1 (it
// scans from the nearest and replaces only for a strictly better score) if for every
// earlier j in reach G(j, i) >= min(dq, dr, k) - cost of the pair (j, i):
//  * G(j, i) >= k is enough, since no pair gains more than k;
//  * if the diagonal (rpos - qpos) changes at most once between j and i it always holds:
//    the pair's gap, hence its cost, is that one change's, and min(k, x + y) <= min(k, x) +
//    min(k, y);
//  * so only pairs across two changes matter, and it suffices that G from the anchor before
//    one change to the anchor after the next is at least k.
// All of this is symmetric in the direction, so it can be checked in the order the
// minimizers come, although a reverse-strand read's anchors sort the other way round. Then
// f rises along the main anchors and they are a chain with score k + the gains. The strays
// chain among themselves at most: alone with score k, which the filters drop (the host checks
// min_anchors >= 2 or min_score > k), or, where two k-mers in a row hit the same wrong place,
// with k + at most the sum of every stray's best gain from a predecessor, which is checked to
// stay below min_score. One chain gives one candidate
// (src/mapper.cpp:40-62).
//
// Two kernels:
//  * k_sketch_reads: the minimizers (src/minimizer.cpp:5-68) of N-free reads (a read with an
//    N is listed), G lanes per read, each sketching one stretch of its windows (a stretch
//    starts w k-mers early, so it knows the window before its first). 16 code bytes a load,
//    packed to 2 bits a base; a block of w k-mers is cut from 32 packed bases at fixed shifts,
//    the reverse complements from the complemented words, the forward ones from the reversed
//    words, so no k-mer waits for the one before it; window minima by van Herk / Gil-Werman,
//    ties to the earlier position. G = 1 where the batch has reads enough to fill the SMs,
//    more where a few reads would leave the launch to one read's serial latency.
//  * k_probe_reads: one warp per read, a lane per minimizer: probe (src/index.hpp:24-38), two
//    buckets a round, then the check across the lanes by ballots and shuffles, 32 minimizers
//    at a time, the chunks' summaries merged by the same rules. The probe is a gather with a
//    short dependent chain, so it wants many warps with little state; one thread per read
//    held a sketch's registers through it and kept 20 warps per SM waiting for memory.
#include <algorithm>
#include <climits>

#include "common.cuh"
#include "seed.cuh"

namespace dnb {

namespace {

constexpr int kCW = 10;         // window length of the compiled sketch
constexpr int kCThreads = 128;
constexpr int kMaxStray = 32;  // a lane each
// A read with a key of more occurrences goes to the full kernels. 262,144 reads of 150 bases of the
// 120 Mbp repeat genome, all kernels, at 4, 8 and 16: 2,054, 2,048 and 2,010 us; 60,000 of 50 to
// 1,000 bases: 6,314, 6,326 and 6,464.
constexpr int kMaxHits = 8;
constexpr int kMaxBandC = 256;  // chaining band the shared gap-cost table holds
constexpr int kMaxLenC = 1 << 30;  // a minimizer's word is pos << 1 | strand

// The main anchors of a stretch of a read, in minimizer order.
struct Run {
  int m = 0;
  uint32_t strand = 0;
  int first_pos = 0, last_pos = 0;
  uint32_t first_r = 0, last_r = 0;
  int gain = 0;            // from the first anchor to the last
  int head = 0, tail = 0;  // first anchor .. past the first diagonal change; before the last .. last anchor
  bool changed = false;
  int dmin = INT_MAX, dmax = INT_MIN;
};

// The gain of the pair (p, q), consecutive in minimizer order, or 0 if it is not a valid one.
__device__ __forceinline__ int pair_gain(const ChainParamsDev& cp, const int32_t* lut, uint32_t strand, int pos_p,
                                         uint32_t r_p, int pos_q, uint32_t r_q, bool& change) {
  const int dq = pos_q - pos_p;
  const int dr = static_cast<int>(strand ? r_p - r_q : r_q - r_p);  // both below 2^31
  const int dd = dr > dq ? dr - dq : dq - dr;
  change = dd != 0;
  if (dr <= 0 || dr > cp.max_gap || dq <= 0 || dd > cp.band) return 0;
  int g = dq < dr ? dq : dr;
  if (g > cp.k) g = cp.k;
  g -= lut[dd];
  return g > 0 ? g : 0;
}

// b's anchors after a's (both in minimizer order) into a. Returns false if the two do not
// make one chain; an anchor left alone goes to *stray (strand << 31 | rpos, diagonal).
__device__ __forceinline__ bool append(Run& a, const Run& b, const ChainParamsDev& cp, const int32_t* lut,
                                       uint2* stray, int* strays) {
  if (b.m == 0) return true;
  bool change = false, ok = true;
  const int g = a.m > 0 && a.strand == b.strand
                    ? pair_gain(cp, lut, a.strand, a.last_pos, a.last_r, b.first_pos, b.first_r, change)
                    : 0;
  if (g > 0) {
    if (change) {
      if (a.changed && a.tail + g < cp.k) ok = false;
      if (b.changed && g + b.head < cp.k) ok = false;
    } else if (a.changed && b.changed && a.tail + g + b.head < cp.k) {
      ok = false;
    }
    if (!a.changed) a.head = a.gain + g + (change ? 0 : b.head);
    a.tail = b.changed ? b.tail : (change ? g + b.gain : a.tail + g + b.gain);
    a.changed = a.changed || change || b.changed;
    a.gain += g + b.gain;
    a.m += b.m;
    a.last_pos = b.last_pos;
    a.last_r = b.last_r;
    a.dmin = min(a.dmin, b.dmin);
    a.dmax = max(a.dmax, b.dmax);
    return ok;
  }
  if (a.m > 1 && b.m > 1) return false;
  if (a.m > 1) {
    *stray = make_uint2(b.strand << 31 | b.first_r, static_cast<uint32_t>(b.dmin));
    *strays += 1;
    return true;
  }
  if (a.m == 1) {  // a's only anchor becomes a stray and b's take over
    *stray = make_uint2(a.strand << 31 | a.first_r, static_cast<uint32_t>(a.dmin));
    *strays += 1;
  }
  a = b;
  return true;
}

// The last step of hash64 (key + (key << 31)) leaves a key below 2^31 alone, and the others
// are multiplications by constants: hash32 (seed.cuh) for 2k <= 30.
__device__ __forceinline__ uint32_t hash30(uint32_t key, uint32_t mask) {
  key = (key * 0x1FFFFFu - 1u) & mask;  // ~key + (key << 21)
  key ^= key >> 24;
  key = (key * 265u) & mask;  // key + (key << 3) + (key << 8)
  key ^= key >> 14;
  key = (key * 21u) & mask;  // key + (key << 2) + (key << 4)
  return key ^ key >> 28;
}

// 16 code bytes (0..3 each) as 2-bit fields, the first in bits 0-1.
__device__ __forceinline__ uint32_t pack16(uint4 v) {
  const auto four = [](uint32_t x) {
    x &= 0x03030303u;
    x |= x >> 6;
    return (x | x >> 12) & 0xFFu;
  };
  return four(v.x) | four(v.y) << 8 | four(v.z) << 16 | four(v.w) << 24;
}

// The 2-bit fields of x in reverse order.
__device__ __forceinline__ uint32_t reverse16(uint32_t x) {
  x = __brev(x);
  return (x >> 1 & 0x55555555u) | (x & 0x55555555u) << 1;
}

// Minimizers of read r, stretch g (windows [g * seg, (g + 1) * seg), seg = stretch_windows):
// hash | (pos << 1 | strand) << 32 at mins[pofs[r] + g * seg + j], j < counts[r * G + g]
// (-1: a read for the full kernels).
template <int W, int G>
__device__ __forceinline__ int stretch_windows(int len, int k) {
  const int nw = len - k + 1 - W + 1;
  return nw > 0 ? (nw + G - 1) / G : 0;
}

template <int W, int G>
__global__ void __launch_bounds__(kCThreads, 6)
    k_sketch_reads(const uint8_t* __restrict__ codes, const int64_t* __restrict__ pofs,
                   const int32_t* __restrict__ seq_len, const int32_t* __restrict__ order, int64_t n, int k,
                   uint64_t* __restrict__ mins, int32_t* __restrict__ counts) {
  const int64_t t = static_cast<int64_t>(blockIdx.x) * kCThreads + threadIdx.x;
  if (t / G >= n) return;
  const int g = static_cast<int>(t % G);
  const int64_t r = order ? order[t / G] : t / G;
  const int len = seq_len[r];
  // this lane's windows: those that end at k-mers [s_begin, s_end); k-mers from p0 on
  const int seg = stretch_windows<W, G>(len, k);
  const int w0 = g * seg, w1 = min(len - k + 1 - W + 1, w0 + seg);
  if (w0 >= w1 || len > kMaxLenC) {
    counts[r * G + g] = len > kMaxLenC ? -1 : 0;
    return;
  }
  const int s_begin = w0 + W - 1, s_end = w1 + W - 1;
  const int p0 = g == 0 ? 0 : s_begin - W;
  const uint32_t mask2k = (1u << (2 * k)) - 1u;
  uint64_t* const out0 = mins + pofs[r] + w0;
  uint64_t* out = out0;
  // stream word j: bases p0 + 16j .. p0 + 16j + 15, from the aligned 16-byte chunks around
  // them (chunks past the read hold its reverse strand's codes, or the buffer's padding)
  const int bases = s_end - p0 + k - 1;  // of this lane's stretch
  const uint8_t* fw = codes + 2 * pofs[r] + p0;
  const int o = static_cast<int>(reinterpret_cast<uintptr_t>(fw) & 15u);
  const uint4* chunk = reinterpret_cast<const uint4*>(reinterpret_cast<uintptr_t>(fw) - static_cast<uintptr_t>(o));
  int got = -o;  // bases of the stretch before the next chunk
  uint32_t ns = 0, packed = 0;
  uint4 raw = __ldg(chunk);
  // packs the loaded chunk, loads the next
  const auto step_chunk = [&]() {
    const uint32_t prev = packed;
    if (got + 16 <= bases && got >= 0) {
      ns |= (raw.x | raw.y | raw.z | raw.w) & 0x04040404u;
    } else {  // a chunk only partly of the stretch: bytes [-got, bases - got) of it
      const auto part = [&](uint32_t x, int at) {
        const int lo = max(0, -at), hi = min(4, bases - at);
        if (lo < hi) ns |= x & 0x04040404u & (0xFFFFFFFFu >> (8 * (4 - hi))) & (0xFFFFFFFFu << (8 * lo));
      };
      part(raw.x, got);
      part(raw.y, got + 4);
      part(raw.z, got + 8);
      part(raw.w, got + 12);
    }
    packed = pack16(raw);
    got += 16;
    ++chunk;
    if (got < bases) raw = __ldg(chunk);
    return __funnelshift_r(prev, packed, 2 * o);
  };
  step_chunk();
  uint32_t a0 = step_chunk(), a1 = step_chunk(), a2 = step_chunk();
  uint32_t sh = 0;  // bits of a0 already used
  uint32_t suf_h[W], suf_p[W];
#pragma unroll
  for (int u = 0; u < W; ++u) suf_h[u] = suf_p[u] = 0;
  uint32_t prev_p = 0xFFFFFFFFu;
  const uint32_t back = 64u - 2u * k - 2u * (W - 1);  // >= 64 - 30 - 18
  for (int s0 = p0; s0 < s_end; s0 += W) {
    // 32 bases from k-mer s0's first on, and the same in reverse order
    const uint32_t f0 = __funnelshift_r(a0, a1, sh), f1 = __funnelshift_r(a1, a2, sh);
    const uint64_t rv = (static_cast<uint64_t>(reverse16(f0)) << 32 | reverse16(f1)) >> back;
    const uint32_t r0 = static_cast<uint32_t>(rv), r1 = static_cast<uint32_t>(rv >> 32);
    sh += 2 * W;
    if (sh >= 32) {
      sh -= 32;
      a0 = a1;
      a1 = a2;
      a2 = step_chunk();
    }
    uint32_t cur_h[W], cur_p[W];
#pragma unroll
    for (int u = 0; u < W; ++u) {
      const uint32_t rev = ~__funnelshift_r(f0, f1, 2 * u) & mask2k;
      const uint32_t fwd = __funnelshift_r(r0, r1, 2 * (W - 1 - u)) & mask2k;
      cur_h[u] = fwd != rev ? hash30(min(fwd, rev), mask2k) : 0xFFFFFFFFu;
      cur_p[u] = static_cast<uint32_t>(s0 + u) << 1 | (rev < fwd ? 1u : 0u);
    }
    uint32_t pre_h = 0xFFFFFFFFu, pre_p = 0;
#pragma unroll
    for (int u = 0; u < W; ++u) {
      if (u == 0 || cur_h[u] < pre_h) {  // prefix of this block: ties keep the earlier
        pre_h = cur_h[u];
        pre_p = cur_p[u];
      }
      // window [s - W + 1, s]: suffix of the previous block from u + 1 (to the left, so it
      // wins ties), prefix of this one; the first whole window ends at the first block's last k-mer
      uint32_t m_h = pre_h, m_p = pre_p;
      if (u + 1 < W && !(pre_h < suf_h[u + 1 < W ? u + 1 : 0])) {
        m_h = suf_h[u + 1 < W ? u + 1 : 0];
        m_p = suf_p[u + 1 < W ? u + 1 : 0];
      }
      const int s = s0 + u;
      if (m_h == 0xFFFFFFFFu || s < p0 + W - 1) m_p = 0xFFFFFFFFu;  // all palindromes; no whole window
      if (m_p != prev_p && m_p != 0xFFFFFFFFu && s >= s_begin && s < s_end)
        *out++ = static_cast<uint64_t>(m_p) << 32 | m_h;
      prev_p = m_p;
    }
    // suffix minima of this block for the next one (ties keep the earlier)
    suf_h[W - 1] = cur_h[W - 1];
    suf_p[W - 1] = cur_p[W - 1];
#pragma unroll
    for (int u = W - 2; u >= 0; --u) {
      const bool left = cur_h[u] <= suf_h[u + 1];
      suf_h[u] = left ? cur_h[u] : suf_h[u + 1];
      suf_p[u] = left ? cur_p[u] : suf_p[u + 1];
    }
  }
  counts[r * G + g] = ns ? -1 : static_cast<int32_t>(out - out0);
}

template <int W, int G>
__global__ void __launch_bounds__(kCThreads)
    k_probe_reads(const int64_t* __restrict__ pofs, const int32_t* __restrict__ seq_len, int64_t n,
                  const uint64_t* __restrict__ mins, const int32_t* __restrict__ counts, DevIndex ix, SeedParams sp,
                  ChainParamsDev cp, CandParams cand, CandBuf cb, int32_t* __restrict__ n_min,
                  int64_t* __restrict__ n_anchor, int32_t* __restrict__ n_anc_t, MinBuf mb, int32_t* __restrict__ list,
                  int* __restrict__ list_n, int long_len,
                  unsigned long long* __restrict__ long_done, uint32_t* __restrict__ err) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int kWarps = kCThreads / 32;
  __shared__ int32_t lut[kMaxBandC + 1];
  __shared__ uint2 s_stray[kWarps][kMaxStray];  // strand << 31 | rpos, diagonal
  __shared__ int32_t s_list[kWarps][32];  // reads for the full kernels, appended 32 at a time
  for (int d = threadIdx.x; d <= cp.band; d += kCThreads) lut[d] = cp.cost[d];
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t mask = static_cast<uint32_t>(ix.mask);
  const int k = sp.k;
  uint2* const stray = s_stray[wid];
  int32_t* const mine = s_list[wid];
  int listed = 0, long_reads = 0;
  const auto flush = [&]() {
    __syncwarp();
    int at = 0;
    if (lane == 0) at = atomicAdd(list_n, listed);
    at = __shfl_sync(FULL, at, 0);
    if (lane < listed) list[at + lane] = mine[lane];
    listed = 0;
    __syncwarp();
  };
  // the bucket of minimizer m (src/index.hpp:24-38), two buckets a round
  const auto probe = [&](uint64_t m, uint32_t& pw, uint32_t& off, uint32_t& c) {
    const uint32_t h = static_cast<uint32_t>(m);
    pw = static_cast<uint32_t>(m >> 32);
    uint32_t slot = h & mask;
    for (uint64_t round = 0;; ++round) {
      const ulonglong2 b0 = __ldg(ix.table + slot), b1 = __ldg(ix.table + ((slot + 1) & mask));
      // keys are below 2^30, an empty bucket's is ~0
      const bool in0 = b0.x == h, end0 = static_cast<uint32_t>(b0.x >> 32) != 0;
      const bool in1 = b1.x == h, end1 = static_cast<uint32_t>(b1.x >> 32) != 0;
      if (in0 || end0 || in1 || end1) {
        const uint64_t y = in0 ? b0.y : b1.y;
        off = static_cast<uint32_t>(y);
        c = in0 || (in1 && !end0) ? static_cast<uint32_t>(y >> 32) : 0u;
        break;
      }
      slot = (slot + 2) & mask;
      if (round > ix.mask) {  // the table is at most half full: an empty bucket ends every walk
        atomicOr(err, kErrProbeLoop);
        break;
      }
    }
    if (c > sp.max_occ) c = 0;
  };
  const int64_t warps = static_cast<int64_t>(gridDim.x) * kWarps;
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * kWarps + wid; r < n; r += warps) {
    const int len = seq_len[r];
    const int64_t base = pofs[r];
    // the stretches' counts: total, and where each starts
    int total, start = 0;
    bool bad;
    if constexpr (G == 1) {
      total = counts[r];
      bad = total < 0;
    } else {
      const int c = lane < G ? counts[r * G + lane] : 0;
      bad = __any_sync(FULL, c < 0);
      start = warp_exclusive_scan(c, &total);
      if (bad) total = -1;
    }
    const int seg = G > 1 ? stretch_windows<W, G>(len, k) : 0;
    const auto place = [&](int j) {  // of the read's minimizer j
      if constexpr (G == 1) return base + j;
      int s = 0;  // the last stretch that starts at or before j
#pragma unroll
      for (int step = G / 2; step > 0; step >>= 1)
        if (__shfl_sync(FULL, start, s + step) <= j) s += step;
      return base + static_cast<int64_t>(s) * seg + (j - __shfl_sync(FULL, start, s));
    };
    Run run;
    int na = 0, ns = 0;
    for (int j0 = 0; j0 < total && !bad; j0 += 32) {
      const int j = j0 + lane;
      const int64_t at = place(j);
      uint32_t pw = 0, off = 0, c = 0;
      if (j < total) probe(__ldg(mins + at), pw, off, c);
      if (__any_sync(FULL, c > kMaxHits)) {
        bad = true;
        break;
      }
      const uint32_t v = c ? __ldg(ix.positions + off) : 0u;
      const int pos = static_cast<int>(pw >> 1);
      uint32_t rpos = v >> 1, strand = (v ^ pw) & 1u;
      na += __reduce_add_sync(FULL, c);
      unsigned in = __ballot_sync(FULL, c == 1);  // lanes with a main anchor
      // ---- keys with several occurrences: the one that pairs with the nearest lane of a
      // single occurrence on either side is the main one, the others are strays
      if (__any_sync(FULL, c > 1)) {
        const unsigned left = in & lt, right = in & ~lt;
        const int lref = left ? 31 - __clz(left) : lane, rref = right ? __ffs(right) - 1 : lane;
        const int l_pos = __shfl_sync(FULL, pos, lref), r_pos = __shfl_sync(FULL, pos, rref);
        const uint32_t l_r = __shfl_sync(FULL, rpos, lref), l_s = __shfl_sync(FULL, strand, lref);
        const uint32_t r_r = __shfl_sync(FULL, rpos, rref), r_s = __shfl_sync(FULL, strand, rref);
        const int most = static_cast<int>(__reduce_max_sync(FULL, c));
        bool found = false;
        uint32_t got_r = 0, got_s = 0;
        for (int t = 0; t < most; ++t) {
          const bool act = c > 1 && t < static_cast<int>(c);
          const uint32_t vt = act ? (t ? __ldg(ix.positions + off + t) : v) : 0u;
          const uint32_t st = (vt ^ pw) & 1u, rt = vt >> 1;
          bool change, pairs = false;
          if (act && !found && left && st == l_s) pairs = pair_gain(cp, lut, st, l_pos, l_r, pos, rt, change) > 0;
          if (act && !found && !pairs && right && st == r_s)
            pairs = pair_gain(cp, lut, st, pos, rt, r_pos, r_r, change) > 0;
          if (pairs) {
            found = true;
            got_r = rt;
            got_s = st;
          }
          const unsigned alone = __ballot_sync(FULL, act && !pairs);
          const int x = ns + __popc(alone & lt);
          if (act && !pairs && x < kMaxStray)
            stray[x] = make_uint2(vt >> 1 | st << 31, rt - static_cast<uint32_t>(st ? len - pos - k : pos));
          ns += __popc(alone);
        }
        if (found) {
          rpos = got_r;
          strand = got_s;
        }
        in = __ballot_sync(FULL, c == 1 || found);
        if (ns > kMaxStray) {
          bad = true;
          break;
        }
      }
      // ---- each main anchor with the one before it
      int gain = 0;
      bool change = false;
      unsigned linked = 0;
      const auto link = [&]() {
        const unsigned before = in & lt;
        const int p = before ? 31 - __clz(before) : lane;
        const int p_pos = __shfl_sync(FULL, pos, p);
        const uint32_t p_r = __shfl_sync(FULL, rpos, p), p_s = __shfl_sync(FULL, strand, p);
        gain = 0;
        change = false;
        if (((in >> lane) & 1u) && before && p_s == strand)
          gain = pair_gain(cp, lut, strand, p_pos, p_r, pos, rpos, change);
        linked = __ballot_sync(FULL, gain > 0);
      };
      link();
      if (__popc(linked) + 1 < __popc(in)) {
        // runs of one or two anchors (but the longest run) are strays, unless without the
        // others they pair with a neighbour after all (a stray stood between); the rest must
        // make one chain
        const unsigned starts = in & ~linked;
        const unsigned upto = starts & (lt | 1u << lane), later = starts & ~lt & ~(1u << lane);
        const int s0 = upto ? 31 - __clz(upto) : 0;  // start of the run this lane's anchor is in
        const unsigned span = (later ? (later & (0u - later)) - 1u : FULL) & ~((1u << s0) - 1u);
        const bool member = (in >> lane) & 1u;
        const int size = member ? __popc(in & span) : 0;
        const int longest = __reduce_max_sync(FULL, size ? size << 5 | (31 - s0) : 0);
        unsigned alone = __ballot_sync(FULL, member && size <= 2 && (size << 5 | (31 - s0)) != longest);
        in &= ~alone;
        const unsigned left = in & lt, right = in & ~lt;
        const int ref = left ? 31 - __clz(left) : (right ? __ffs(right) - 1 : lane);
        const int ref_pos = __shfl_sync(FULL, pos, ref);
        const uint32_t ref_r = __shfl_sync(FULL, rpos, ref), ref_s = __shfl_sync(FULL, strand, ref);
        bool pairs = false;
        if (((alone >> lane) & 1u) && ref != lane && ref_s == strand)
          pairs = (left ? pair_gain(cp, lut, strand, ref_pos, ref_r, pos, rpos, change)
                        : pair_gain(cp, lut, strand, pos, rpos, ref_pos, ref_r, change)) > 0;
        const unsigned back = __ballot_sync(FULL, pairs);
        alone &= ~back;
        in |= back;
        const int x = ns + __popc(alone & lt);
        if (((alone >> lane) & 1u) && x < kMaxStray)
          stray[x] = make_uint2(strand << 31 | rpos, rpos - static_cast<uint32_t>(strand ? len - pos - k : pos));
        ns += __popc(alone);
        link();
        if (ns > kMaxStray || __popc(linked) + 1 < __popc(in)) {
          bad = true;
          break;
        }
      }
      if (!in) continue;
      // ---- the chunk's summary
      const int diag = static_cast<int>(rpos) - (strand ? len - pos - k : pos);
      const bool member = (in >> lane) & 1u;
      const int f = __ffs(in) - 1, l = 31 - __clz(in);
      Run b;
      b.m = __popc(in);
      b.strand = __shfl_sync(FULL, strand, f);
      b.first_pos = __shfl_sync(FULL, pos, f);
      b.first_r = __shfl_sync(FULL, rpos, f);
      b.last_pos = __shfl_sync(FULL, pos, l);
      b.last_r = __shfl_sync(FULL, rpos, l);
      b.gain = __reduce_add_sync(FULL, gain);
      const unsigned changes = __ballot_sync(FULL, gain > 0 && change);
      if (changes) {
        int before = gain;  // gains up to and with this lane's
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int y = __shfl_up_sync(FULL, before, d);
          if (lane >= d) before += y;
        }
        b.dmin = __reduce_min_sync(FULL, member ? diag : INT_MAX);
        b.dmax = __reduce_max_sync(FULL, member ? diag : INT_MIN);
        b.changed = true;
        const int c0 = __ffs(changes) - 1, c1 = 31 - __clz(changes);
        b.head = __shfl_sync(FULL, before, c0);
        b.tail = b.gain - __shfl_sync(FULL, before - gain, c1);
        // two changes in a row: the gains from before the first to after the second
        const unsigned earlier = changes & lt;
        const int e = earlier ? 31 - __clz(earlier) : lane;
        const int from = __shfl_sync(FULL, before - gain, e);
        if (__any_sync(FULL, ((changes >> lane) & 1u) && earlier && before - from < k)) bad = true;
      } else {
        b.dmin = b.dmax = __shfl_sync(FULL, diag, f);
      }
      uint2 one = make_uint2(0, 0);
      int ones = 0;
      if (!append(run, b, cp, lut, &one, &ones)) bad = true;
      if (ones) {
        if (ns < kMaxStray) {
          if (lane == 0) stray[ns] = one;
        } else {
          bad = true;
        }
        ++ns;
      }
    }
    __syncwarp();
    // strays: no valid pair with a main anchor, no chain of their own that the filters keep
    const uint32_t r_lo = run.strand ? run.last_r : run.first_r, r_hi = run.strand ? run.first_r : run.last_r;
    if (!bad && ns) {
      const uint32_t gap = static_cast<uint32_t>(cp.max_gap);
      bool pairs = ns >= cp.lookback;
      int best = 0;
      if (lane < ns) {
        const uint32_t rx = stray[lane].x & 0x7FFFFFFFu, sx = stray[lane].x >> 31;
        const int dx = static_cast<int>(stray[lane].y);
        if (run.m > 0 && sx == run.strand && rx + gap >= r_lo && rx <= r_hi + gap && dx >= run.dmin - cp.band &&
            dx <= run.dmax + cp.band)
          pairs = true;
        for (int y = 0; y < ns; ++y) {
          const int dr = static_cast<int>(rx) - static_cast<int>(stray[y].x & 0x7FFFFFFFu);
          const int shift = dx - static_cast<int>(stray[y].y), dq = dr - shift;
          const int dd = shift < 0 ? -shift : shift;
          if (sx == stray[y].x >> 31 && dr > 0 && dq > 0 && dr <= cp.max_gap && dd <= cp.band)
            best = max(best, min(min(dr, dq), k) - lut[dd]);
        }
      }
      const int own = __reduce_add_sync(FULL, best);
      bad = __any_sync(FULL, pairs) || (own > 0 && k + own >= cp.min_score);
      __syncwarp();
    }
    if (bad) {
      // its minimizers and their buckets for the warp kernels (an N read's are still to be made: -1)
      int64_t anchors = 0;
      const bool sketched = total >= 0;
      for (int j0 = 0; j0 < total && sketched; j0 += 32) {
        const int j = j0 + lane;
        const int64_t at = place(j);
        uint32_t pw = 0, off = 0, c = 0;
        if (j < total) {
          probe(__ldg(mins + at), pw, off, c);
          mb.pos[base + j] = pw >> 1 | pw << 31;
          mb.hit_off[base + j] = off;
          mb.hit_cnt[base + j] = c;
        }
        anchors += __reduce_add_sync(FULL, c);
      }
      if (lane == 0) {
        mine[listed] = static_cast<int32_t>(r);
        n_min[r] = sketched ? total : 0;
        n_anchor[r] = sketched ? anchors : -1;
        n_anc_t[r] = 0;
      }
      if (++listed == 32) flush();
      continue;
    }
    const int score = k + run.gain;
    const bool keep = run.m > 0 && score >= cp.min_score && run.m >= cp.min_anchors &&
                      !(static_cast<double>(score) < static_cast<double>(score) * cand.pri_ratio);
    if (lane == 0) {
      if (keep) {
        const int64_t ci = r * cand.max_cand;
        const int64_t diag = static_cast<int32_t>(run.dmin + (static_cast<int64_t>(run.dmax) - run.dmin) / 2);
        cb.rev[ci] = static_cast<uint8_t>(run.strand);
        cb.contig[ci] = contig_of(ix, r_hi);  // the last anchor in sorted order
        cb.diag[ci] = diag;
        cb.wstart[ci] = diag - cand.bw;
      }
      n_anchor[r] = 0;  // no anchor scratch
      n_min[r] = total;
      n_anc_t[r] = na;
      cb.n_cand[r] = keep ? 1 : 0;
    }
    long_reads += len > long_len ? 1 : 0;
  }
  if (listed) flush();
  if (lane == 0 && long_reads) atomicAdd(long_done, static_cast<unsigned long long>(long_reads));
}

// Reads (of a list, or all) per length bin, and the read ids by bin.
__global__ void k_read_bins(const int32_t* __restrict__ seq_len, const int32_t* __restrict__ list,
                            const int* __restrict__ list_n, int n, int* __restrict__ hist, int bin_shift) {
  __shared__ int s[kLengthBins];
  const int m = list_n ? *list_n : n;
  if (static_cast<int>(blockIdx.x * blockDim.x) >= m) return;
  for (int b = threadIdx.x; b < kLengthBins; b += blockDim.x) s[b] = 0;
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x)
    atomicAdd(s + length_bin(seq_len[list ? list[i] : i], bin_shift), 1);
  __syncthreads();
  for (int b = threadIdx.x; b < kLengthBins; b += blockDim.x)
    if (s[b]) atomicAdd(hist + b, s[b]);
}

__global__ void __launch_bounds__(256)
    k_read_order(const int32_t* __restrict__ seq_len, const int32_t* __restrict__ list,
                 const int* __restrict__ list_n, int n, const int* __restrict__ hist, int* __restrict__ taken,
                 int bin_shift, int32_t* __restrict__ order) {
  __shared__ int first[kLengthBins];
  const int m = list_n ? *list_n : n;
  if (static_cast<int>(blockIdx.x * blockDim.x) >= m) return;
  scan_length_bins(hist, first);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    const int r = list ? list[i] : i;
    const int b = length_bin(seq_len[r], bin_shift);
    order[first[b] + atomicAdd(taken + b, 1)] = r;
  }
}

}  // namespace

bool seed_colinear_supported(const SeedParams& sp, const ChainParamsDev& cp, const DevIndex& ix) {
  return sp.w == kCW && sp.k >= 4 && sp.k <= 15 && cp.max_gap >= 0 && cp.max_gap < (1 << 29) && cp.band >= 0 &&
         cp.band <= kMaxBandC && cp.lookback >= 1 && (cp.min_anchors >= 2 || cp.min_score > sp.k) &&
         ix.mask <= 0xFFFFFFFFull;
}

// As many lanes a read as keep all reads resident at once, each with 32 bases and more. k_sketch_reads,
// us, with the next smaller number and with this: 20,000 reads of 150 bases (2) 20.8 and 20.7,
// 4,557 of 100 to 300 (4) 14.5 and 13.7, 800 of 300 to 1,000 (16) 18.9 and 14.6, 4,001 of 1,000 to
// 5,000 (16) 77.8 and 59.8.
int seed_colinear_lanes(int64_t n, int64_t max_len) {
  const int64_t want = static_cast<int64_t>(device_sm_count()) * 6 * kCThreads;  // resident lanes
  int g = 1;
  while (g < 32 && n * g * 2 <= want && max_len / (2 * g) >= 32) g *= 2;
  return g;
}

void launch_sketch_reads(cudaStream_t st, const uint8_t* codes, const int64_t* pofs, const int32_t* seq_len,
                         const int32_t* order, int64_t n, int lanes, const SeedParams& sp, uint64_t* mins,
                         int32_t* counts) {
  const unsigned blocks = static_cast<unsigned>((n * lanes + kCThreads - 1) / kCThreads);
  const auto run = [&](auto kernel) {
    kernel<<<blocks, kCThreads, 0, st>>>(codes, pofs, seq_len, order, n, sp.k, mins, counts);
  };
  switch (lanes) {
    case 2: return run(k_sketch_reads<kCW, 2>);
    case 4: return run(k_sketch_reads<kCW, 4>);
    case 8: return run(k_sketch_reads<kCW, 8>);
    case 16: return run(k_sketch_reads<kCW, 16>);
    case 32: return run(k_sketch_reads<kCW, 32>);
    default: return run(k_sketch_reads<kCW, 1>);
  }
}

void launch_probe_reads(cudaStream_t st, const int64_t* pofs, const int32_t* seq_len, int64_t n, int lanes,
                        const uint64_t* mins, const int32_t* counts, const DevIndex& ix, const SeedParams& sp,
                        const ChainParamsDev& cp, const CandParams& cand, CandBuf cb, int32_t* n_min,
                        int64_t* n_anchor, int32_t* n_anc_t, MinBuf mb, int32_t* list, int* list_n,
                        int long_len, unsigned long long* long_done, uint32_t* err) {
  const unsigned blocks = static_cast<unsigned>(
      std::min<int64_t>((n + kCThreads / 32 - 1) / (kCThreads / 32), int64_t{32} * device_sm_count()));
  const auto run = [&](auto kernel) {
    kernel<<<blocks, kCThreads, 0, st>>>(pofs, seq_len, n, mins, counts, ix, sp, cp, cand, cb, n_min, n_anchor, n_anc_t,
                                         mb, list, list_n, long_len, long_done, err);
  };
  switch (lanes) {
    case 2: return run(k_probe_reads<kCW, 2>);
    case 4: return run(k_probe_reads<kCW, 4>);
    case 8: return run(k_probe_reads<kCW, 8>);
    case 16: return run(k_probe_reads<kCW, 16>);
    case 32: return run(k_probe_reads<kCW, 32>);
    default: return run(k_probe_reads<kCW, 1>);
  }
}

void launch_read_order(cudaStream_t st, const int32_t* seq_len, const int32_t* list, const int* list_n, int n,
                       int64_t max_len, int* bins, int32_t* order) {
  if (n <= 0) return;
  const int bin_shift = length_bin_shift(max_len);
  const int blocks = std::min((n + 255) / 256, 2 * device_sm_count());
  k_read_bins<<<blocks, 256, 0, st>>>(seq_len, list, list_n, n, bins, bin_shift);
  k_read_order<<<blocks, 256, 0, st>>>(seq_len, list, list_n, n, bins, bins + kLengthBins, bin_shift, order);
}

}  // namespace dnb
