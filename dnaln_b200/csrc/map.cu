// map.cu — per-read bookkeeping between the pipeline's compute stages: building SW
// tasks from candidate loci, choosing among equally scored candidates, MAPQ and the
// final records with their soft-clipped CIGARs. One thread per read; all integer except
// MAPQ, which is evaluated in FP64 with explicitly rounded operations in the
// reference's operation order (src/mapper.cpp:217-218).
#include "map.cuh"

namespace dnb {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

// The block's sum of each of N values is added to ctr[k] by one atomic each; *last (may be
// null) = the block's sum of the last value. 262,144 reads made 24,600 atomics on three words
// warp by warp; now k_choose also sums the seeds and fills the CIGAR slots and k_records sums
// the operations, which took nine launches more: k_choose 23 -> 21 us, and a batch of 64 reads
// 269 -> 253 us, of 262,144 972 -> 876 us, with the other launches saved.
template <int N>
__device__ __forceinline__ void block_add(const unsigned long long (&v)[N], unsigned long long* const (&ctr)[N],
                                          long long* last = nullptr) {
  __shared__ unsigned long long part[N][kWarps];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const unsigned long long x = warp_sum(v[k]);
    if ((threadIdx.x & 31) == 0) part[k][threadIdx.x >> 5] = x;
  }
  __syncthreads();
  if (threadIdx.x < N) {
    unsigned long long x = 0;
    for (int w = 0; w < kWarps; ++w) x += part[threadIdx.x][w];
    if (x) atomicAdd(ctr[threadIdx.x], x);
    if (last && threadIdx.x == N - 1) *last = static_cast<long long>(x);
  }
}

// First of the `want` entries this thread gets after *counter, one atomic per block.
__device__ __forceinline__ int block_reserve(int want, int* counter) {
  __shared__ int part[kWarps + 1];
  int total;
  const int ex = warp_exclusive_scan(want, &total);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = total;
  __syncthreads();
  if (threadIdx.x == 0) {
    int all = 0;
    for (int w = 0; w < kWarps; ++w) {
      const int x = part[w];
      part[w] = all;
      all += x;
    }
    part[kWarps] = all ? atomicAdd(counter, all) : 0;
  }
  __syncthreads();
  return part[kWarps] + part[threadIdx.x >> 5] + ex;
}

// ---- packed offsets of the reads: exclusive sums of their lengths --------------------------
// Blocks of per_block reads (a multiple of kLenTile): k_len_sums leaves each block's sum,
// k_len_scan adds up those before its own and scans its reads. One block needs no sums.
constexpr int kLenTile = 4 * kThreads;
constexpr int64_t kLenBlocks = 2048;   // at most
constexpr int64_t kLenSingle = 4 * kLenTile;  // reads one block takes

int64_t len_per_block(int64_t n) {
  if (n <= kLenSingle) return kLenSingle;
  const int64_t tiles = (n + kLenTile - 1) / kLenTile;
  return (tiles + kLenBlocks - 1) / kLenBlocks * kLenTile;
}

__global__ void __launch_bounds__(kThreads)
    k_len_sums(const int32_t* __restrict__ len, int64_t n, int64_t per_block, long long* __restrict__ sums,
               unsigned long long* __restrict__ max_len, unsigned long long* __restrict__ total) {
  const int64_t lo = blockIdx.x * per_block, hi = lo + per_block < n ? lo + per_block : n;
  unsigned long long sum = 0;
  int most = 0;
  for (int64_t i = lo + threadIdx.x; i < hi; i += kThreads) {
    const int l = len[i] < 0 ? 0 : len[i];
    sum += static_cast<unsigned>(l);
    most = max(most, l);
  }
  __shared__ unsigned long long part[kWarps];
  __shared__ int part_max[kWarps];
  sum = warp_sum(sum);
  most = __reduce_max_sync(0xffffffffu, most);
  if ((threadIdx.x & 31) == 0) {
    part[threadIdx.x >> 5] = sum;
    part_max[threadIdx.x >> 5] = most;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kWarps; ++w) {
      sum += part[w];
      most = max(most, part_max[w]);
    }
    if (sums) sums[blockIdx.x] = static_cast<long long>(sum);
    if (most > 0) atomicMax(max_len, static_cast<unsigned long long>(most));
    if (total && sum) atomicAdd(total, sum);
  }
}

__global__ void __launch_bounds__(kThreads)
    k_len_scan(const int32_t* __restrict__ len, int64_t n, int64_t per_block, const long long* __restrict__ sums,
               int64_t* __restrict__ pofs, unsigned long long* __restrict__ max_len) {
  __shared__ long long part[2][32];
  long long base = 0;
  if (blockIdx.x > 0) {
    long long acc = 0;
    for (int x = threadIdx.x; x < static_cast<int>(blockIdx.x); x += kThreads) acc += sums[x];
    block_exclusive_scan_ll(acc, &base, part[0]);
    __syncthreads();
  }
  const int64_t lo = blockIdx.x * per_block, hi = lo + per_block < n ? lo + per_block : n;
  int most = 0, flip = 0;
  for (int64_t t = lo; t < hi; t += kLenTile, flip ^= 1) {
    const int64_t i = t + 4 * threadIdx.x;
    int l[4];
    long long sum = 0, total;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      l[k] = i + k < hi ? max(len[i + k], 0) : 0;
      sum += l[k];
      most = max(most, l[k]);
    }
    long long at = base + block_exclusive_scan_ll(sum, &total, part[flip]);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i + k < hi) pofs[i + k] = at;
      at += l[k];
    }
    base += total;
  }
  if (hi == n && threadIdx.x == 0) pofs[n] = base;
  if (!sums) {  // the only block
    most = __reduce_max_sync(0xffffffffu, most);
    if ((threadIdx.x & 31) == 0 && most > 0) atomicMax(max_len, static_cast<unsigned long long>(most));
  }
}

// CIGAR operations before a read's: k_records leaves the sum of each block of kThreads reads
// and of each kOpGroup blocks, k_cigar_gather adds up those before its own.
constexpr int kOpGroup = 64;
__host__ __device__ __forceinline__ int64_t op_blocks_for(int64_t n) { return (n + kThreads - 1) / kThreads; }
__host__ __device__ __forceinline__ int64_t op_groups_for(int64_t n) {
  return (op_blocks_for(n) + kOpGroup - 1) / kOpGroup;
}

// SW task of candidate c of read r: query = forward or reverse-complement codes, target
// window = genome[wstart, wstart + len + 2bw) with N outside the candidate's contig
// (src/mapper.cpp:100-121, src/reference.cpp:34-47).
__device__ __forceinline__ SwTask cand_task(int64_t r, int c, const int64_t* pofs, const int32_t* seq_len,
                                            const CandBuf& cb, const DevIndex& ix, const MapConsts& mc) {
  const int64_t ci = r * mc.max_cand + c;
  const int len = seq_len[r];
  const int ctg = cb.contig[ci];
  const int64_t ws = cb.wstart[ci];
  const int64_t cb0 = static_cast<int64_t>(ix.contig_off[ctg]), ce = cb0 + ix.contig_len[ctg];
  const int64_t we = ws + len + 2 * static_cast<int64_t>(mc.bw);
  SwTask t;
  t.q_off = 2 * pofs[r] + (cb.rev[ci] ? len : 0);
  t.qlen = len;
  t.t_start = ws;
  t.t_lo = ws > cb0 ? ws : cb0;
  t.t_hi = we < ce ? we : ce;
  t.slot = 0;
  // the whole window inside the contig and clear of the genome's N runs: no N to score
  t.flags = (t.t_lo == ws && t.t_hi == we && !genome_has_n(ix, ws, we)) ? kTaskNoN : 0;
  t.pad_ = 0;
  return t;
}

__global__ void k_score_tasks(int64_t n, const int64_t* __restrict__ pofs, const int32_t* __restrict__ seq_len,
                              CandBuf cb, DevIndex ix, MapConsts mc, SwTask* __restrict__ tasks,
                              int* __restrict__ counter, unsigned long long* __restrict__ ctr) {
  const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int nc = r < n ? cb.n_cand[r] : 0;
  const int want = nc >= 2 ? nc : 0;
  const int first = block_reserve(want, counter);
  for (int c = 0; c < want; ++c) {
    SwTask t = cand_task(r, c, pofs, seq_len, cb, ix, mc);
    t.slot = static_cast<int32_t>(r * mc.max_cand + c);
    tasks[first + c] = t;
  }
  // cells of the ranking pass, counted as the reference's MapStats::cells (src/mapper.cpp:139)
  const unsigned long long cells[1] = {want ? static_cast<unsigned long long>(want) * seq_len[r] * mc.W : 0ull};
  unsigned long long* const to[1] = {ctr};
  block_add(cells, to);
}

__global__ void k_choose(int64_t n, const int64_t* __restrict__ pofs, const int32_t* __restrict__ seq_len, CandBuf cb,
                         const SwResult* __restrict__ res_score, const uint32_t* __restrict__ name_hash, DevIndex ix,
                         MapConsts mc, int32_t* __restrict__ chosen, int32_t* __restrict__ s2o,
                         SwTask* __restrict__ tb_tasks, int* __restrict__ tb_counter,
                         int64_t* __restrict__ cig_slot, long long* __restrict__ op_groups,
                         const int32_t* __restrict__ n_min, const int32_t* __restrict__ n_anc,
                         unsigned long long* __restrict__ seeds, unsigned long long* __restrict__ ctr) {
  const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  int pick_c = -1, s2 = 0, nc = 0;
  if (r < n) {
    nc = cb.n_cand[r];
    if (nc == 1) {
      pick_c = 0;
    } else if (nc >= 2) {
      const SwResult* rs = res_score + r * mc.max_cand;
      int s1 = -1, ties = 0;
      for (int c = 0; c < nc; ++c) {
        const int sw = rs[c].score;
        if (sw > s1) {
          s1 = sw;
          ties = 1;
        } else if (sw == s1) {
          ++ties;
        }
      }
      if (ties > 1) {
        s2 = s1;
      } else {
        for (int c = 0; c < nc; ++c)
          if (rs[c].score != s1 && rs[c].score > s2) s2 = rs[c].score;
      }
      uint32_t pick = name_hash[r] % static_cast<uint32_t>(ties);
      for (int c = 0; c < nc; ++c)
        if (rs[c].score == s1 && pick-- == 0) {
          pick_c = c;
          break;
        }
    }
    chosen[r] = pick_c;
    s2o[r] = s2;
    cig_slot[r] = 2 * pofs[r] + r;
    if (r < op_groups_for(n)) op_groups[r] = 0;
  }
  const int at = block_reserve(pick_c >= 0 ? 1 : 0, tb_counter);
  if (pick_c >= 0) {
    SwTask t = cand_task(r, pick_c, pofs, seq_len, cb, ix, mc);
    t.slot = static_cast<int32_t>(r);
    tb_tasks[at] = t;
  }
  // traceback cells (src/mapper.cpp:186), candidates, and the seeding's totals
  const unsigned long long sums[4] = {
      pick_c >= 0 ? static_cast<unsigned long long>(seq_len[r]) * mc.W : 0ull, static_cast<unsigned long long>(nc),
      r < n ? static_cast<unsigned long long>(n_min[r]) : 0ull,
      r < n && n_anc ? static_cast<unsigned long long>(n_anc[r]) : 0ull};
  unsigned long long* const to[4] = {ctr, ctr + 2, seeds, seeds + 1};
  block_add(sums, to);
}

__global__ void k_records(int64_t n, const int32_t* __restrict__ seq_len, CandBuf cb,
                          const int32_t* __restrict__ chosen, const int32_t* __restrict__ s2o,
                          const SwResult* __restrict__ res_tb, DevIndex ix, MapConsts mc,
                          dnaln_map_record* __restrict__ out, int32_t* __restrict__ op_count,
                          long long* __restrict__ op_sums, long long* __restrict__ op_groups,
                          unsigned long long* __restrict__ ctr) {
  const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  int32_t ops = 0;
  bool mapped = false;
  if (r < n) {
  dnaln_map_record m;
  m.pos = 0;
  m.cigar_off = 0;
  m.contig = -1;
  m.score = 0;
  m.nm = 0;
  m.n_cand = cb.n_cand[r];
  m.cigar_len = 0;
  m.rev = 0;
  m.mapq = 0;
  m.pad_[0] = m.pad_[1] = 0;
  const int c = chosen[r];
  if (c >= 0) {
    const SwResult a = res_tb[r];
    if (a.score >= mc.min_aln_score) {
      const int64_t ci = r * mc.max_cand + c;
      const int ctg = cb.contig[ci];
      m.contig = ctg;
      m.rev = cb.rev[ci];
      m.pos = cb.wstart[ci] + a.tb - static_cast<int64_t>(ix.contig_off[ctg]);
      m.score = a.score;
      m.nm = a.nm;
      if (m.n_cand <= 1) {
        m.mapq = 60;
      } else {
        const int s2 = s2o[r];
        double q = 0.0;
        if (s2 < a.score)
          q = __dadd_rn(__ddiv_rn(__dmul_rn(6.02, static_cast<double>(a.score - s2)), static_cast<double>(mc.match)),
                        0.499);
        m.mapq = static_cast<uint8_t>(static_cast<int>(q < 60.0 ? q : 60.0));
      }
      ops = (a.qb > 0 ? 1 : 0) + a.n_ops + (seq_len[r] > a.qe ? 1 : 0);
      mapped = true;
    }
  }
  out[r] = m;
  op_count[r] = ops;
  }
  const unsigned long long sums[2] = {mapped ? 1ull : 0ull, static_cast<unsigned long long>(ops)};
  long long* const group = op_groups + blockIdx.x / kOpGroup;
  unsigned long long* const to[2] = {ctr + 1, reinterpret_cast<unsigned long long*>(group)};
  block_add(sums, to, op_sums + blockIdx.x);
}

__global__ void k_cigar_gather(int64_t n, const int64_t* __restrict__ pofs, const int32_t* __restrict__ seq_len,
                               const SwResult* __restrict__ res_tb, const uint32_t* __restrict__ cig_src,
                               const int32_t* __restrict__ op_count, const long long* __restrict__ op_sums,
                               const long long* __restrict__ op_groups, const int64_t* __restrict__ rec_base,
                               dnaln_map_record* __restrict__ out, uint32_t* __restrict__ dst, int64_t cap,
                               long long* __restrict__ total_ops, uint32_t* __restrict__ err) {
  __shared__ long long part[2][32];
  const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int b = blockIdx.x, g = b / kOpGroup;
  long long before = 0, base, block_ops;
  for (int x = threadIdx.x; x < g; x += kThreads) before += op_groups[x];
  if (static_cast<int>(threadIdx.x) < b % kOpGroup) before += op_sums[g * kOpGroup + threadIdx.x];
  block_exclusive_scan_ll(before, &base, part[0]);
  const int64_t cnt = r < n ? op_count[r] : 0;
  const int64_t o = base + block_exclusive_scan_ll(cnt, &block_ops, part[1]);
  if (threadIdx.x == 0 && blockIdx.x + 1 == gridDim.x) *total_ops = base + block_ops;
  if (r >= n) return;
  out[r].cigar_off = *rec_base + o;
  out[r].cigar_len = static_cast<int32_t>(cnt);
  if (cnt == 0) return;
  if (o + cnt > cap) {  // the caller's buffer is too small: the call reports the size it needs
    atomicOr(err, kErrOutputCapacity);
    return;
  }
  const SwResult a = res_tb[r];
  const uint32_t* src = cig_src + 2 * pofs[r] + r;
  int64_t x = o;
  if (a.qb > 0) dst[x++] = static_cast<uint32_t>(a.qb) << 4 | 4u;  // S
  for (int i = a.n_ops - 1; i >= 0; --i) dst[x++] = src[i];
  if (seq_len[r] > a.qe) dst[x++] = static_cast<uint32_t>(seq_len[r] - a.qe) << 4 | 4u;
}

// Tasks of dnaln_gpu_align from its offset and length columns (query at i, target at n + i),
// the target cut to the band's reach; ops[i] (may be null) = room for the task's CIGAR.
__global__ void k_align_tasks(int64_t n, const int64_t* __restrict__ off, const int32_t* __restrict__ len, int W,
                              SwTask* __restrict__ tasks, int64_t* __restrict__ ops) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) {
    const int64_t ql = len[i], tl = len[n + i], tmax = ql + W - 1;
    SwTask t;
    t.q_off = off[i];
    t.t_start = t.t_lo = off[n + i];
    t.t_hi = t.t_start + (tl < tmax ? tl : tmax);
    t.qlen = static_cast<int32_t>(ql);
    t.slot = static_cast<int32_t>(i);
    t.flags = 0;
    t.pad_ = 0;
    tasks[i] = t;
    if (ops) ops[i] = 2 * ql + 1;
  }
  if (i == n && ops) ops[n] = 0;
}

__global__ void k_align_scores(int64_t n, const SwResult* __restrict__ res, dnaln_align_result* __restrict__ out) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  dnaln_align_result o{};
  o.score = res[i].score;
  out[i] = o;
}

__global__ void k_align_counts(int64_t n, const SwResult* __restrict__ res, int64_t* __restrict__ counts) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) counts[i] = res[i].n_ops;
  if (i == n) counts[n] = 0;
}

__global__ void k_align_gather(int64_t n, const SwResult* __restrict__ res, const uint32_t* __restrict__ cig_src,
                               const int64_t* __restrict__ src_off, const int64_t* __restrict__ dst_off,
                               dnaln_align_result* __restrict__ out, uint32_t* __restrict__ dst) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const SwResult a = res[i];
  dnaln_align_result o;
  o.score = a.score;
  o.qb = a.qb;
  o.qe = a.qe;
  o.tb = a.tb;
  o.te = a.te;
  o.nm = a.nm;
  o.cigar_off = dst_off[i];
  o.cigar_len = a.n_ops;
  o.pad_ = 0;
  out[i] = o;
  const uint32_t* src = cig_src + src_off[i];
  for (int k = 0; k < a.n_ops; ++k) dst[o.cigar_off + k] = src[a.n_ops - 1 - k];
}

inline unsigned blocks_for(int64_t n) { return static_cast<unsigned>((n + kThreads - 1) / kThreads); }

}  // namespace

void launch_score_tasks(cudaStream_t st, int64_t n, const int64_t* pofs, const int32_t* seq_len, CandBuf cb,
                        const DevIndex& ix, const MapConsts& mc, SwTask* tasks, int* counter,
                        unsigned long long* ctr) {
  if (n > 0) k_score_tasks<<<blocks_for(n), kThreads, 0, st>>>(n, pofs, seq_len, cb, ix, mc, tasks, counter, ctr);
}

void launch_choose(cudaStream_t st, int64_t n, const int64_t* pofs, const int32_t* seq_len, CandBuf cb,
                   const SwResult* res_score, const uint32_t* name_hash, const DevIndex& ix, const MapConsts& mc,
                   int32_t* chosen, int32_t* s2, SwTask* tb_tasks, int* tb_counter, int64_t* cig_slot, OpSums ops,
                   const int32_t* n_min, const int32_t* n_anc, unsigned long long* seeds, unsigned long long* ctr) {
  if (n > 0)
    k_choose<<<blocks_for(n), kThreads, 0, st>>>(n, pofs, seq_len, cb, res_score, name_hash, ix, mc, chosen, s2,
                                                 tb_tasks, tb_counter, cig_slot, ops.groups, n_min, n_anc, seeds, ctr);
}

void launch_records(cudaStream_t st, int64_t n, const int32_t* seq_len, CandBuf cb, const int32_t* chosen,
                    const int32_t* s2, const SwResult* res_tb, const DevIndex& ix, const MapConsts& mc,
                    dnaln_map_record* out, OpSums ops, unsigned long long* ctr) {
  k_records<<<blocks_for(n), kThreads, 0, st>>>(n, seq_len, cb, chosen, s2, res_tb, ix, mc, out, ops.count, ops.sums,
                                                ops.groups, ctr);
}

void launch_cigar_gather(cudaStream_t st, int64_t n, const int64_t* pofs, const int32_t* seq_len,
                         const SwResult* res_tb, const uint32_t* cig_src, OpSums ops, const int64_t* rec_base,
                         dnaln_map_record* out, uint32_t* dst, int64_t cap, long long* total_ops, uint32_t* err) {
  if (n <= 0) return;
  k_cigar_gather<<<blocks_for(n), kThreads, 0, st>>>(n, pofs, seq_len, res_tb, cig_src, ops.count, ops.sums,
                                                     ops.groups, rec_base, out, dst, cap, total_ops, err);
}

int64_t op_sum_words(int64_t n) { return op_blocks_for(n) + op_groups_for(n); }

OpSums make_op_sums(int64_t n, int32_t* count, long long* words) { return {count, words, words + op_blocks_for(n)}; }

int64_t len_sum_words(int64_t n) { return (n + len_per_block(n) - 1) / len_per_block(n); }

int launch_read_offsets(cudaStream_t st, const int32_t* len, int64_t n, long long* sums, int64_t* pofs,
                        unsigned long long* max_len) {
  const int64_t per = len_per_block(n);
  const unsigned blocks = static_cast<unsigned>((n + per - 1) / per);
  if (blocks > 1) k_len_sums<<<blocks, kThreads, 0, st>>>(len, n, per, sums, max_len, nullptr);
  k_len_scan<<<blocks, kThreads, 0, st>>>(len, n, per, blocks > 1 ? sums : nullptr, pofs, max_len);
  return blocks > 1 ? 2 : 1;
}

void launch_read_totals(cudaStream_t st, const int32_t* len, int64_t n, unsigned long long* max_len,
                        unsigned long long* total) {
  const int64_t per = (len_per_block(n) + 3) / 4;
  k_len_sums<<<static_cast<unsigned>((n + per - 1) / per), kThreads, 0, st>>>(len, n, per, nullptr, max_len, total);
}

void launch_align_tasks(cudaStream_t st, int64_t n, const int64_t* off, const int32_t* len, int W, SwTask* tasks,
                        int64_t* ops) {
  k_align_tasks<<<blocks_for(n + 1), kThreads, 0, st>>>(n, off, len, W, tasks, ops);
}

void launch_align_scores(cudaStream_t st, int64_t n, const SwResult* res, dnaln_align_result* out) {
  if (n > 0) k_align_scores<<<blocks_for(n), kThreads, 0, st>>>(n, res, out);
}

void launch_align_counts(cudaStream_t st, int64_t n, const SwResult* res, int64_t* counts) {
  k_align_counts<<<blocks_for(n + 1), kThreads, 0, st>>>(n, res, counts);
}

void launch_align_gather(cudaStream_t st, int64_t n, const SwResult* res, const uint32_t* cig_src,
                         const int64_t* src_off, const int64_t* dst_off, dnaln_align_result* out, uint32_t* dst) {
  if (n > 0) k_align_gather<<<blocks_for(n), kThreads, 0, st>>>(n, res, cig_src, src_off, dst_off, out, dst);
}

}  // namespace dnb
