// sw_ungapped.cu — the banded Smith–Waterman tasks whose answer is one run of diagonal
// steps, proved from bit vectors instead of computed cell by cell (sm_100a).
//
// A mapped read without an indel aligns along the band's middle diagonal d0 = bw. Its DP
// (src/align.cpp:31-84) then does 2bw+1 cells per base to find what the diagonal alone
// shows. k_sw_ungapped reads a task's query and window once, as two bit planes of 32 bases
// a word, walks the mismatches of d0 (the local score u(i) = max(0, u(i-1) + s(i, d0)), its
// first maximum B at row i*, the row where that run starts) and then tests every other
// diagonal of the band with word operations. When the tests hold, the DP's result is known
// exactly: score B, best cell (i*, d0), and a traceback of diagonal steps only. Every other
// task is listed for the DP kernels (sw.cu), in full.
//
// Why the tests suffice. Scores A (match), -B' (mismatch), gap of length g costs O + gE;
// kernel preconditions: no N in the query or the window, A, B' >= 1, G := A + B' <= O + E,
// B' <= A + E. Call a row that mismatches on d0 an X row, and value a path's rows relative
// to d0's: a step on another diagonal d is worth at most +G on an X row, 0 on a row where d
// matches too and -G where d mismatches; an insertion row, its run's first E moved to the
// gap, at most +B' on an X row and -A or -(A + E) elsewhere. Test 1: strictly between two
// consecutive X rows, every diagonal d != d0 mismatches at least once. Then a stretch of a
// path off d0 on one diagonal, with the insertion rows at its ends, is worth at most G (each
// further X row it credits is paid for by the mismatch or insertion rows before it), and
// every change of diagonal costs at least O + E >= G. So a path that has a row on d0 before
// or after its stretches off it never exceeds d0's own sum over its rows:
//  * on d0 itself H(i, d0) = u(i), and along the run E, F <= hd: the walk, which prefers the
//    diagonal, takes only diagonal steps (src/align.cpp:87-143);
//  * elsewhere H <= u(i), so below B before row i* and never above it after. On row i* the
//    columns left of d0 are reached by an insertion; test 1 applied to (last X row, i*] too
//    keeps the stretch that ends there below G, hence H(i*, d) < B for d < d0: the first
//    strict maximum in row-major order is (i*, d0).
// A path that never touches d0 is a chain of matching runs of at most R rows, each two
// separated by a mismatch or a gap, so it scores at most L (A - c/R) + c, c = min(B', O + E).
// Test 2: that bound is below B with R = 14, because no other diagonal matches a whole
// aligned block of 8 rows (a run of 15 covers such a block). Test 2 also settles test 1 for
// every interval of 15 rows or more, so test 1 runs only where two X rows are closer.
//
// Layout: G lanes per task (four at bw <= 16, else eight). A word step takes 32 rows: each
// lane packs eight bytes of the query, of the window or of both, loaded a step ahead,
// shuffles give every lane the word of all planes, and lane l tests diagonals l, l + G, ...
// (skipping d0) with six instructions each. The kernel is bound by instruction issue.
// Measured, SW with traceback: 262,144 x 150 bp at W = 33 (82% of the tasks proved) 678 us
// of DP and 122 of walks -> 136 of this kernel, 215 and 62; 100,003 reads of 50-1000 bp at
// W = 129 2,315 and 161 -> 327, 1,500 and 99. Eight lanes per task at W = 33 took 203 us.
#include <algorithm>

#include "common.cuh"
#include "sw.cuh"

namespace dnb {

namespace {

constexpr int kThreads = 128;
// Grid-stride: a few resident waves, whatever the capacity of the list. At 6, 12 and 24, us: 262,144
// tasks of 150 rows 142, 136 and 130, 100,003 of 50 to 1,000 rows at W = 129 381, 330 and 316, an
// empty list (the scores of a batch without ties) 6.1, 7.0 and 8.1; the first batch's kernels
// together 985, 955 and 973.
constexpr int kBlocksPerSm = 12;
constexpr int kRun = 14;          // longest match run test 2 allows off d0
constexpr int kNear = 15;         // intervals of fewer rows may hold no aligned block of 8

// The bytes base[off .. off + 8) as two little-endian words, bytes at or past len zero. Only
// aligned 32-bit words that hold at least one byte below len are read.
__device__ __forceinline__ uint2 load8(const uint8_t* __restrict__ base, int off, int len) {
  const int valid = len - off;
  if (valid <= 0) return make_uint2(0u, 0u);
  const uintptr_t a = reinterpret_cast<uintptr_t>(base) + static_cast<uintptr_t>(off);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3));
  const int s = static_cast<int>(a & 3u);
  const uint32_t w0 = __ldg(w);
  const uint32_t w1 = valid > 4 - s ? __ldg(w + 1) : 0u;
  const uint32_t w2 = s != 0 && valid > 8 - s ? __ldg(w + 2) : 0u;
  uint32_t lo = __funnelshift_r(w0, w1, 8 * s), hi = __funnelshift_r(w1, w2, 8 * s);
  if (valid < 8) {
    const uint64_t m = (uint64_t(1) << (8 * valid)) - 1u;
    lo &= static_cast<uint32_t>(m);
    hi &= static_cast<uint32_t>(m >> 32);
  }
  return make_uint2(lo, hi);
}

// Bit 0 of each byte of v into bits 0..3 (the product's bits 24..27 are the four bits, and
// no two of its partial products meet).
__device__ __forceinline__ uint32_t low_bits(uint32_t v) { return ((v & 0x01010101u) * 0x01020408u) >> 24; }

// NT: plane words a word step sees, 32 rows and the band: 2bw + 32 <= 32 NT. G: lanes per
// task.
template <int NT, int G, bool TB>
__global__ void __launch_bounds__(kThreads)
    k_sw_ungapped(const SwTask* __restrict__ tasks, int n, const int* __restrict__ n_dev,
                  const uint8_t* __restrict__ qbase, const uint8_t* __restrict__ tbase, SwParams p,
                  SwResult* __restrict__ res, uint32_t* __restrict__ cig, const int64_t* __restrict__ cig_off,
                  SwTask* __restrict__ todo, int* __restrict__ todo_n, int* __restrict__ hist, int bin_shift) {
  static_assert(G == 4 || G == 8, "a word's planes are packed by four lanes per string");
  constexpr int K = 32 * (NT - 1) / G;  // diagonals per lane, at most
  constexpr int kPerWarp = 32 / G;
  constexpr unsigned FULL = 0xffffffffu;
  const int nn = n_dev ? min(n, *n_dev) : n;
  const int lane = threadIdx.x & 31, gl = lane & (G - 1);
  const unsigned gm = ((1u << G) - 1u) << (lane & ~(G - 1));
  const int warps = gridDim.x * (kThreads / 32), warp = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  const int bw = p.bw, nd = 2 * bw;  // diagonals other than d0
  const int A = p.match, Bm = p.mismatch, cst = min(p.mismatch, p.oe);
  const bool upper = gl >= 4;
  const uint32_t sel_pair = (gl & 1) ? 0x1054u : 0x5410u;
  const uint32_t sel_p0 = (gl & 2) ? 0x2064u : 0x6420u, sel_p1 = (gl & 2) ? 0x3175u : 0x7531u;
  for (int t0 = warp * kPerWarp; t0 < nn; t0 += warps * kPerWarp) {
    const int ti = t0 + lane / G;
    const bool live = ti < nn;
    SwTask tk{};
    if (live) tk = tasks[ti];
    const int L = tk.qlen, wlen = L + nd;
    // the whole window lies in the target (columns past it count as N)
    bool ok = live && L > 0 && static_cast<int64_t>(L) * A < (1 << 30) && tk.t_lo <= tk.t_start &&
              tk.t_hi >= tk.t_start + wlen;
    int B = 0, best_i = -1, best_start = 0, best_nm = 0;
    if (ok) {
      const uint8_t* __restrict__ q = qbase + tk.q_off;
      const uint8_t* __restrict__ t = tbase + tk.t_start;
      uint32_t ta[NT], tb[NT];  // planes of window columns 32w .. 32w + 32 NT
      uint32_t qa = 0, qb = 0, bad = 0, runs = 0, open = 0;
      struct Raw {
        uint2 q, t;  // G = 8: t only, a query piece in the lower four lanes
      };
      const auto load = [&](int wq, int wt) {  // query word wq (none if negative) and window word wt
        Raw r{};
        if constexpr (G == 8) {
          if (upper) r.t = load8(t, 32 * wt + 8 * (gl - 4), wlen);
          else if (wq >= 0) r.t = load8(q, 32 * wq + 8 * gl, L);
        } else {
          if (wq >= 0) r.q = load8(q, 32 * wq + 8 * gl, L);
          r.t = load8(t, 32 * wt + 8 * gl, wlen);
        }
        return r;
      };
      // the word of both planes from the four lanes' eight bytes each
      const auto pack = [&](uint2 v, uint32_t& pa, uint32_t& pb) {
        bad |= (v.x | v.y) & 0xFCFCFCFCu;  // an N
        const uint32_t c = low_bits(v.x) | low_bits(v.y) << 4 | low_bits(v.x >> 1) << 8 | low_bits(v.y >> 1) << 12;
        const uint32_t c2 = __byte_perm(c, __shfl_xor_sync(gm, c, 1), sel_pair);
        const uint32_t o2 = __shfl_xor_sync(gm, c2, 2);
        pa = __byte_perm(c2, o2, sel_p0);
        pb = __byte_perm(c2, o2, sel_p1);
      };
      const auto take = [&](const Raw& r) {
        uint32_t na, nb;
        pack(r.t, na, nb);
        if constexpr (G == 8) {
          const uint32_t xa = __shfl_xor_sync(gm, na, 4), xb = __shfl_xor_sync(gm, nb, 4);
          qa = upper ? xa : na;
          qb = upper ? xb : nb;
          na = upper ? na : xa;
          nb = upper ? nb : xb;
        } else {
          pack(r.q, qa, qb);
        }
#pragma unroll
        for (int j = 0; j + 1 < NT; ++j) {
          ta[j] = ta[j + 1];
          tb[j] = tb[j + 1];
        }
        ta[NT - 1] = na;
        tb[NT - 1] = nb;
      };
#pragma unroll
      for (int j = 0; j < NT; ++j) ta[j] = tb[j] = 0;
      Raw next = load(-1, 0);
#pragma unroll
      for (int j = 0; j + 1 < NT; ++j) {
        const Raw r = next;
        next = load(j + 2 < NT ? -1 : 0, j + 1);
        take(r);
      }
      // a B at or below this fails test 2
      const int64_t need = (static_cast<int64_t>(L) * (A * kRun - cst) + cst * kRun) / kRun;
      const int floor_b = static_cast<int>(need);
      int u = 0, start = 0, nm = 0, last_x = -2 * kNear;
      for (int w = 0; 32 * w < L; ++w) {
        const Raw r = next;
        next = load(w + 1, w + NT);
        take(r);
        const int rem = L - 32 * w, rows = min(rem, 32);
        const uint32_t V = rem >= 32 ? FULL : (1u << rem) - 1u;
        const int j0 = NT > 3 && bw > 32 ? 1 : 0;  // window word that holds d0 + 32w's first bit
        const uint32_t a0 = __funnelshift_rc(j0 ? ta[NT > 3 ? 1 : 0] : ta[0], j0 ? ta[NT > 3 ? 2 : 1] : ta[1], bw - 32 * j0);
        const uint32_t b0 = __funnelshift_rc(j0 ? tb[NT > 3 ? 1 : 0] : tb[0], j0 ? tb[NT > 3 ? 2 : 1] : tb[1], bw - 32 * j0);
        uint32_t X = ((a0 ^ qa) | (b0 ^ qb)) & V;
        int at = 0;         // rows of this word the score has taken
        bool near = false;  // two X rows closer than kNear, the later in this word
        for (uint32_t rest = X; rest; rest &= rest - 1) {
          const int k = __ffs(rest) - 1;
          u += A * (k - at);
          if (u > B) {
            B = u;
            best_i = 32 * w + k - 1;
            best_start = start;
            best_nm = nm;
          }
          near |= 32 * w + k - last_x <= kNear;
          last_x = 32 * w + k;
          u -= Bm;
          ++nm;
          at = k + 1;
          if (u <= 0) {
            u = 0;
            start = 32 * w + at;
            nm = 0;
          }
        }
        u += A * (rows - at);
        if (u > B) {
          B = u;
          best_i = 32 * w + rows - 1;
          best_start = start;
          best_nm = nm;
        }
        if (max(B, u + A * (rem - rows)) <= floor_b) {  // out of test 2's reach
          bad = 1u;
          break;
        }
        // test 1's interval that ends the run at the read's last row: one more X row past it
        if (rem < 32 && best_i == L - 1) {
          X |= 1u << rem;
          near |= L - last_x <= kNear;
        }
        // mismatch rows of this lane's diagonals: e below d0, e + 1 past it
        uint32_t mm[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const int e = gl + G * k, j = G * k >> 5;
          const int sh = (G * k & 31) + gl + (e >= bw ? 1 : 0);
          const uint32_t a = __funnelshift_rc(ta[j], ta[j + 1], sh);
          const uint32_t b = __funnelshift_rc(tb[j], tb[j + 1], sh);
          mm[k] = (a ^ qa) | (b ^ qb);
          if (rem < 32) mm[k] |= ~V;
          if (e >= nd) mm[k] = FULL;
          runs |= (mm[k] - 0x01010101u) & ~mm[k];
        }
        if (near) {
          // a carry from just past each X row runs through the rows where both diagonals
          // match; one that arrives at the next X row met no mismatch on its way
#pragma unroll
          for (int k = 0; k < K; ++k) bad |= (~(mm[k] | X) + (X << 1 | ((open >> k) & 1u))) & X;
        }
        open = 0;
        if (32 * w + 32 - last_x <= kNear) {  // diagonals without a mismatch since the last X row
          const uint32_t after = ~0u << (last_x & 31) << 1;
#pragma unroll
          for (int k = 0; k < K; ++k) open |= (mm[k] & after) == 0 ? 1u << k : 0u;
        }
        if (__any_sync(gm, (bad | (runs & 0x80808080u)) != 0)) {
          bad = 1u;
          break;
        }
      }
      if ((L & 31) == 0 && best_i == L - 1) bad |= open;  // that interval ends with a word
      ok = !__any_sync(gm, bad != 0) && B > floor_b;
    }
    __syncwarp();
    const bool lead = gl == 0 && live;
    if (lead && ok) {
      SwResult r{B, 0, 0, 0, 0, 0, 0, 0};
      if constexpr (TB) {
        r = SwResult{B, best_start, best_i + 1, best_start + bw, best_i + bw + 1, best_nm, 1, 0};
        cig[cig_off[tk.slot]] = static_cast<uint32_t>(best_i + 1 - best_start) << 4;
      }
      res[tk.slot] = r;
    }
    const unsigned left = __ballot_sync(FULL, lead && !ok);
    if (left) {
      int at = 0;
      if (lane == 0) at = atomicAdd(todo_n, __popc(left));
      at = __shfl_sync(FULL, at, 0);
      if (lead && !ok) {
        todo[at + __popc(left & ((1u << lane) - 1u))] = tk;
        if (hist) atomicAdd(hist + length_bin(L, bin_shift), 1);
      }
    }
  }
}

// Lengths of the tasks per bin (see launch_order_tasks).
__global__ void k_length_bins(const SwTask* __restrict__ tasks, int n, const int* __restrict__ n_dev,
                              int* __restrict__ hist, int bin_shift) {
  const int nn = n_dev ? min(n, *n_dev) : n;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x)
    atomicAdd(hist + length_bin(tasks[i].qlen, bin_shift), 1);
}

// out = the tasks by length bin (bin 0, the longest, first), in any order within a bin: every
// block scans the bins, every task takes the next place of its bin.
__global__ void __launch_bounds__(256)
    k_order_tasks(const SwTask* __restrict__ tasks, int n, const int* __restrict__ n_dev,
                  const int* __restrict__ hist, int* __restrict__ taken, int bin_shift, SwTask* __restrict__ out) {
  __shared__ int first[kLengthBins];
  const int nn = n_dev ? min(n, *n_dev) : n;
  if (static_cast<int>(blockIdx.x * blockDim.x) >= nn) return;
  scan_length_bins(hist, first);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x) {
    const SwTask t = tasks[i];
    const int b = length_bin(t.qlen, bin_shift);
    out[first[b] + atomicAdd(taken + b, 1)] = t;
  }
}

}  // namespace

bool sw_ungapped_supported(const SwParams& p, bool bytes_ok) {
  const int g = p.match + p.mismatch;
  return bytes_ok && p.W <= 129 && p.bw >= 1 && p.match >= 1 && p.mismatch >= 1 && g <= p.oe &&
         p.mismatch <= p.match + p.ge && p.match * kRun >= std::min(p.mismatch, p.oe);
}

// The DP of a short list takes one task's latency, whether a fifth or all of the list is left to it,
// so the pass in front of it is lost time unless it proves every task, as it may of a handful.
// Tracebacks of 150 rows, a fifth of them with a gap, us without and with the pass:
//   W = 11   8,192 67 and 80, 20,000 96 and 86       W = 43   2,048 63 and 74, 4,096 75 and 74
//   W = 17   8,192 80 and 92, 20,000 111 and 102     W = 65   2,048 69 and 82, 4,096 83 and 83
//   W = 33   4,096 73 and 84, 8,192 83 and 86,       W = 129  512 71 and 86, 2,048 90 and 88
//            20,000 176 and 111
// and 64 tasks of 1,000 rows at W = 33 275 and 334. One task that is proved 59 and 31 (1,000 rows
// 245 and 54), one that is not 63 and 72. The widths without a form for short lists run a thread
// per task (k_sw_any), which any task spared is worth.
bool sw_ungapped_pays(int W, bool bytes_ok, int64_t n) {
  return n <= 4 || n > sw_few_tasks(W) / 2 || !sw_has_form(W, bytes_ok, kSwIntraFew);
}

void launch_sw_ungapped(cudaStream_t st, bool tb, const SwTask* tasks, int n, const int* n_dev, const uint8_t* qbase,
                        const uint8_t* tbase, const SwParams& p, SwResult* res, uint32_t* cig, const int64_t* cig_off,
                        SwTask* todo, int* todo_n, int* hist, int bin_shift) {
  if (n <= 0) return;
  const int per_block = kThreads / (p.bw <= 16 ? 4 : 8);
  const int blocks = std::min((n + per_block - 1) / per_block, kBlocksPerSm * device_sm_count());
  const auto run = [&](auto kernel) {
    kernel<<<blocks, kThreads, 0, st>>>(tasks, n, n_dev, qbase, tbase, p, res, cig, cig_off, todo, todo_n, hist,
                                        bin_shift);
  };
  if (p.bw <= 16) tb ? run(k_sw_ungapped<2, 4, true>) : run(k_sw_ungapped<2, 4, false>);
  else if (p.bw <= 32) tb ? run(k_sw_ungapped<3, 8, true>) : run(k_sw_ungapped<3, 8, false>);
  else tb ? run(k_sw_ungapped<5, 8, true>) : run(k_sw_ungapped<5, 8, false>);
}

void launch_length_bins(cudaStream_t st, const SwTask* tasks, int n, const int* n_dev, int* hist, int bin_shift) {
  if (n <= 0) return;
  const int blocks = std::min((n + 255) / 256, 4 * device_sm_count());
  k_length_bins<<<blocks, 256, 0, st>>>(tasks, n, n_dev, hist, bin_shift);
}

void launch_order_tasks(cudaStream_t st, const SwTask* tasks, int n, const int* n_dev, const int* hist, int* taken,
                        int bin_shift, SwTask* out) {
  if (n <= 0) return;
  const int blocks = std::min((n + 255) / 256, 4 * device_sm_count());
  k_order_tasks<<<blocks, 256, 0, st>>>(tasks, n, n_dev, hist, taken, bin_shift, out);
}

}  // namespace dnb
