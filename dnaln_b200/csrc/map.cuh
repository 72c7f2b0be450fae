// map.cuh — batch bookkeeping kernels of the mapping pipeline (map.cu).
#pragma once

#include "common.cuh"
#include "seed.cuh"

namespace dnb {

struct MapConsts {
  int32_t max_cand, bw, W, min_aln_score, match;
};

// Counters shared by the bookkeeping kernels: ctr[0] SW cells (qlen * (2bw+1) per task,
// as MapStats::cells), ctr[1] mapped reads, ctr[2] candidate loci.

// Packed offsets pofs[0, n] of reads of the given lengths (below 0 counts as 0) and *max_len
// (0 before) = the longest; sums: len_sum_words(n) words. Returns its launches.
int64_t len_sum_words(int64_t n);
int launch_read_offsets(cudaStream_t st, const int32_t* len, int64_t n, long long* sums, int64_t* pofs,
                        unsigned long long* max_len);
// The longest read and the sum of the lengths only (both 0 before).
void launch_read_totals(cudaStream_t st, const int32_t* len, int64_t n, unsigned long long* max_len,
                        unsigned long long* total);

// CIGAR operations of each read, and their sums per block and per group of blocks of reads
// (words: op_sum_words(n) entries).
struct OpSums {
  int32_t* count;
  long long *sums, *groups;
};
int64_t op_sum_words(int64_t n);
OpSums make_op_sums(int64_t n, int32_t* count, long long* words);

// Score-only tasks for every candidate of reads with >= 2 candidates
// (src/mapper.cpp:125-133); task slot = r * max_cand + c. *counter += tasks.
void launch_score_tasks(cudaStream_t st, int64_t n, const int64_t* pofs, const int32_t* seq_len, CandBuf cb,
                        const DevIndex& ix, const MapConsts& mc, SwTask* tasks, int* counter,
                        unsigned long long* ctr);

// Choice among a read's candidates (src/mapper.cpp:142-174) and its traceback task
// (slot = r). chosen[r] = candidate index or -1; s2[r] = second-best score; cig_slot[r] = its
// place in the walk's CIGAR buffer. Clears ops.groups. seeds[0], seeds[1] += the reads' n_min
// and n_anc (may be null).
void launch_choose(cudaStream_t st, int64_t n, const int64_t* pofs, const int32_t* seq_len, CandBuf cb,
                   const SwResult* res_score, const uint32_t* name_hash, const DevIndex& ix, const MapConsts& mc,
                   int32_t* chosen, int32_t* s2, SwTask* tb_tasks, int* tb_counter, int64_t* cig_slot, OpSums ops,
                   const int32_t* n_min, const int32_t* n_anc, unsigned long long* seeds, unsigned long long* ctr);

// Records + MAPQ (src/mapper.cpp:189-222); ops: CIGAR operations including soft clips.
void launch_records(cudaStream_t st, int64_t n, const int32_t* seq_len, CandBuf cb, const int32_t* chosen,
                    const int32_t* s2, const SwResult* res_tb, const DevIndex& ix, const MapConsts& mc,
                    dnaln_map_record* out, OpSums ops, unsigned long long* ctr);

// Writes each mapped read's CIGAR (leading S, the walk's ops reversed, trailing S) at
// dst + the operations of the reads before it, and sets out[r].cigar_off (plus *rec_base) and
// cigar_len; a CIGAR that would end past cap ops is not written and sets kErrOutputCapacity.
// *total_ops = all operations.
// cig_src slot of read r is 2 * pofs[r] + r.
void launch_cigar_gather(cudaStream_t st, int64_t n, const int64_t* pofs, const int32_t* seq_len,
                         const SwResult* res_tb, const uint32_t* cig_src, OpSums ops, const int64_t* rec_base,
                         dnaln_map_record* out, uint32_t* dst, int64_t cap, long long* total_ops, uint32_t* err);

// GpuAligner: the tasks of n (offset, length) pairs, queries at [0, n) and targets at [n, 2n)
// of off and len; ops (n + 1 entries, may be null) = 2 * qlen + 1 each, then 0.
void launch_align_tasks(cudaStream_t st, int64_t n, const int64_t* off, const int32_t* len, int W, SwTask* tasks,
                        int64_t* ops);
// GpuAligner: score-only results.
void launch_align_scores(cudaStream_t st, int64_t n, const SwResult* res, dnaln_align_result* out);

// GpuAligner: reversed walk ops of task i (slot i, source cig_src + src_off[i]) to
// dst + dst_off[i]; fills out[i].
void launch_align_gather(cudaStream_t st, int64_t n, const SwResult* res, const uint32_t* cig_src,
                         const int64_t* src_off, const int64_t* dst_off, dnaln_align_result* out, uint32_t* dst);

// ops count per align result -> counts[i] (for the scan of dst offsets)
void launch_align_counts(cudaStream_t st, int64_t n, const SwResult* res, int64_t* counts);

}  // namespace dnb
