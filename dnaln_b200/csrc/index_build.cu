// index_build.cu — MinimizerIndex::build (src/index.cpp:10-45) on the device.
//
// The genome is already resident (one code per byte). Steps:
//   1. minimizers of every contig (src/minimizer.cpp:5-68), in tiles of kTile window ends:
//      a block stages its bases, forms the canonical k-mer hashes of the tile plus the w
//      k-mers before it, and each thread decides, for 8 consecutive window ends, whether
//      the window is whole (w consecutive N-free k-mers of one contig) and whether its
//      leftmost minimum is emitted (valid, and not the same position as the previous
//      window's minimum — the reference's `last` can only repeat from the window just
//      before, because minimum positions never decrease inside an N-free run and an
//      all-palindrome window keeps no valid minimum). A tile emits a position at most once
//      and after all the tile before it emits, so it only sets bits in a mask of its
//      region; the masks' words, counted and scanned, then place the (hash, position) pairs
//      in genome order, so the stable radix sort by hash below leaves positions ascending
//      within a key: the reference's (hash, pos) order. The runs of non-ACGT codes (used by
//      SW task builders) are counted and placed the same way, by words of the genome;
//   2. stable radix sort of (hash, pos << 1 | strand) by hash;
//   3. distinct keys: the sorted hashes' heads, ranked by a scan, with their offsets;
//   4. the bucket table: cap = smallest power of two >= max(16, 2 * n_keys), keys placed
//      by linear probing from hash & mask as if inserted one by one in ascending hash
//      order (the reference's loop). In parallel: every key walks from its home bucket and
//      claims buckets with atomicMin on its rank (its place in ascending hash order); a key
//      that takes a bucket from a higher rank sends that key on from the next bucket. A
//      bucket's rank only decreases, so at the end every key sits in the first bucket from
//      its home not held by a lower rank — by induction on the rank, the bucket sequential
//      insertion gives it.
// Device memory is what a build used to spend its time on (4.6 Mbp: 0.5 ms of kernels, 10 ms
// and more with some forty allocations and frees, each of which also waits for the device):
// all temporary arrays are cut from one workspace the caller keeps, and the built arrays
// from one allocation, made when their sizes are known.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cstdio>
#include <vector>

#include "common.cuh"
#include "index_build.cuh"

namespace dnb {
namespace {

constexpr int kThreads = 256;
constexpr int kPerThread = 8;
constexpr int kTile = kThreads * kPerThread;  // window ends per block
constexpr int kMaxW = 255;
constexpr int kMaxK = 28;
constexpr uint32_t kEmptyRank = 0xFFFFFFFFu;
constexpr int kTileWords = (kTile + kMaxW) / 32 + 2;  // words of 32 positions a tile's minimizers lie in

struct TileSmem {
  uint8_t base[kTile + kMaxW + kMaxK];
  uint64_t hash[kTile + kMaxW];  // kInvalidHash for palindromes
  uint8_t ok[kTile + kMaxW];     // k-mer inside the contig and N-free
};

// Window ending at k-mer e (region index x = e - r0): whole, and its leftmost minimum.
__device__ __forceinline__ void window_at(const TileSmem& sm, int x, int w, bool& whole, int& arg) {
  whole = x >= w - 1;
  uint64_t best = kInvalidHash;
  arg = -1;
  for (int y = x - w + 1; y <= x && whole; ++y) {
    if (!sm.ok[y]) whole = false;
    if (sm.hash[y] < best) {  // strict: ties keep the leftmost
      best = sm.hash[y];
      arg = y;
    }
  }
  if (!whole || best == kInvalidHash) arg = -1;
}

// The minimizers of tile b as bits of its kTileWords words, bit i of word x being position
// 32 (tile_word[b] + x) + i, and their number per word. Tile b of contig c is its window
// ends [contig_off[c] + (b - first_tile[c]) * kTile, + kTile).
__global__ void __launch_bounds__(kThreads)
    k_genome_minimizers(const uint8_t* __restrict__ genome, const uint64_t* __restrict__ contig_off,
                        const uint32_t* __restrict__ contig_len, const int64_t* __restrict__ first_tile,
                        int n_contigs, int k, int w, uint32_t* __restrict__ bits, uint32_t* __restrict__ counts,
                        uint32_t* __restrict__ tile_word) {
  __shared__ TileSmem sm;
  __shared__ uint32_t s_bits[kTileWords];
  int lo = 0, hi = n_contigs;  // the last contig whose first tile is at or before this block
  while (hi - lo > 1) {
    const int mid = (lo + hi) / 2;
    if (first_tile[mid] <= static_cast<int64_t>(blockIdx.x)) lo = mid;
    else hi = mid;
  }
  const int64_t cs = static_cast<int64_t>(contig_off[lo]), ce = cs + contig_len[lo];
  const int64_t t0 = cs + (blockIdx.x - first_tile[lo]) * kTile, t1 = t0 + kTile < ce ? t0 + kTile : ce;
  // region of k-mer starts [r0, t1): the tile and the w k-mers before it
  const int64_t r0 = t0 - w;
  const int nk = static_cast<int>(t1 - r0);
  const int nb = nk + k - 1;
  for (int i = threadIdx.x; i < nb; i += kThreads) {
    const int64_t p = r0 + i;
    sm.base[i] = (p >= cs && p < ce) ? genome[p] : 4;
  }
  for (int i = threadIdx.x; i < kTileWords; i += kThreads) s_bits[i] = 0;
  __syncthreads();
  const uint64_t mask = (1ULL << (2 * k)) - 1;
  for (int i = threadIdx.x; i < nk; i += kThreads) {
    const int64_t s = r0 + i;
    bool ok = s >= cs && s + k <= ce;
    uint64_t fwd = 0, rev = 0;
    for (int m = 0; m < k; ++m) {
      const uint32_t c = sm.base[i + m];
      ok = ok && c <= 3;
      fwd = fwd << 2 | (c & 3u);
      rev |= static_cast<uint64_t>(3u - (c & 3u)) << (2 * m);
    }
    sm.ok[i] = ok;
    sm.hash[i] = (ok && fwd != rev) ? hash64(rev < fwd ? rev : fwd, mask) : kInvalidHash;
  }
  __syncthreads();
  // this thread's window ends: region indices x in [w + 8t, w + 8t + 8) within the tile
  const int x0 = w + threadIdx.x * kPerThread;
  const int64_t word0 = (r0 < 0 ? 0 : r0) >> 5;
  if (x0 < nk) {
    bool whole_prev;
    int arg_prev;
    window_at(sm, x0 - 1, w, whole_prev, arg_prev);
    for (int d = 0; d < kPerThread && x0 + d < nk; ++d) {
      bool whole;
      int arg;
      window_at(sm, x0 + d, w, whole, arg);
      if (arg >= 0 && !(whole_prev && arg_prev == arg)) {
        const int64_t p = r0 + arg;
        atomicOr(s_bits + ((p >> 5) - word0), 1u << (p & 31));
      }
      whole_prev = whole;
      arg_prev = arg;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kTileWords; i += kThreads) {
    const int64_t x = static_cast<int64_t>(blockIdx.x) * kTileWords + i;
    bits[x] = s_bits[i];
    counts[x] = __popc(s_bits[i]);
  }
  if (threadIdx.x == 0) tile_word[blockIdx.x] = static_cast<uint32_t>(word0);
}

// Runs of non-ACGT codes that start in each word of 32 bases.
__global__ void k_word_counts(const uint8_t* __restrict__ g, int64_t n, int64_t words, uint32_t* __restrict__ n_run) {
  const int64_t w = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (w > words) return;
  uint32_t r = 0;
  if (w < words) {
    bool before = w > 0 && g[32 * w - 1] > 3;
    const int64_t end = 32 * w + 32 < n ? 32 * w + 32 : n;
    for (int64_t p = 32 * w; p < end; ++p) {
      const bool here = g[p] > 3;
      r += here && !before;
      before = here;
    }
  }
  n_run[w] = r;  // the entry past the last word ends the scan
}

// (hash, position << 1 | strand) of every minimizer, tile by tile in genome order.
__global__ void k_word_minimizers(const uint8_t* __restrict__ g, const uint32_t* __restrict__ bits,
                                  const uint32_t* __restrict__ tile_word, int64_t words, int k,
                                  const uint32_t* __restrict__ first, uint64_t* __restrict__ out_hash,
                                  uint32_t* __restrict__ out_val) {
  const int64_t w = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (w >= words) return;
  const uint64_t mask = (1ULL << (2 * k)) - 1;
  const int64_t base = 32 * (static_cast<int64_t>(tile_word[w / kTileWords]) + w % kTileWords);
  uint32_t o = first[w];
  for (uint32_t b = bits[w]; b; b &= b - 1) {
    const int64_t p = base + __ffs(b) - 1;
    uint64_t fwd = 0, rev = 0;
    for (int m = 0; m < k; ++m) {
      const uint64_t c = g[p + m];
      fwd = fwd << 2 | c;
      rev |= (3 - c) << (2 * m);
    }
    const uint32_t st = rev < fwd;
    out_hash[o] = hash64(st ? rev : fwd, mask);
    out_val[o] = static_cast<uint32_t>(p) << 1 | st;
    ++o;
  }
}

// The runs [x, y) of non-ACGT codes: run j starts in the word whose scanned count reaches j,
// and as many runs end before a word as start before it, less the one open at its start.
__global__ void k_word_runs(const uint8_t* __restrict__ g, int64_t n, int64_t words, const uint32_t* __restrict__ first,
                            uint2* __restrict__ runs) {
  const int64_t w = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (w >= words) return;
  const int64_t b = 32 * w, end = b + 32 < n ? b + 32 : n;
  bool before = w > 0 && g[b - 1] > 3;
  uint32_t starts = first[w], ends = starts - (before && g[b] > 3 ? 1u : 0u);
  for (int64_t p = b; p < end; ++p) {
    const bool here = g[p] > 3;
    if (here && !before) runs[starts++].x = static_cast<uint32_t>(p);
    if (here && (p == n - 1 || g[p + 1] <= 3)) runs[ends++].y = static_cast<uint32_t>(p + 1);
    before = here;
  }
}

// Heads of the sorted hashes' runs, and, ranked, the keys and where each key's run starts.
__global__ void k_key_heads(const uint64_t* __restrict__ hash, int64_t n, uint32_t* __restrict__ head) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i <= n) head[i] = i < n && (i == 0 || hash[i] != hash[i - 1]);
}
__global__ void k_key_list(const uint64_t* __restrict__ hash, int64_t n, const uint32_t* __restrict__ rank,
                           uint64_t* __restrict__ keys, uint32_t* __restrict__ start) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i > n) return;
  if (i == n) {
    start[rank[n]] = static_cast<uint32_t>(n);
  } else if (rank[i + 1] != rank[i]) {
    keys[rank[i]] = hash[i];
    start[rank[i]] = static_cast<uint32_t>(i);
  }
}

// Bucket placement by rank (see the file comment); err set if a walk passes every bucket.
__global__ void k_place_keys(const uint64_t* __restrict__ keys, int64_t n_keys, uint64_t mask,
                             uint32_t* __restrict__ slot_rank, uint32_t* __restrict__ err) {
  const int64_t r0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (r0 >= n_keys) return;
  uint32_t r = static_cast<uint32_t>(r0);
  uint64_t s = keys[r] & mask;
  for (uint64_t steps = 0; steps <= 4 * (mask + 1) + 64; ++steps) {
    const uint32_t old = atomicMin(slot_rank + s, r);
    if (old == kEmptyRank) return;  // placed in an empty bucket
    // old > r: r took the bucket and the displaced key walks on from the next bucket (every
    // bucket from its home up to here holds a lower rank: it walked past them, and a
    // bucket's rank only decreases); old < r: a lower rank holds the bucket, r walks on
    if (old > r) r = old;
    s = (s + 1) & mask;
  }
  atomicOr(err, kErrProbeLoop);
}

__global__ void k_fill_table(const uint32_t* __restrict__ slot_rank, uint64_t n_buckets,
                             const uint64_t* __restrict__ keys, const uint32_t* __restrict__ start,
                             ulonglong2* __restrict__ table, uint32_t* __restrict__ max_count) {
  const uint64_t s = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  uint32_t count = 0;
  if (s < n_buckets) {
    const uint32_t r = slot_rank[s];
    ulonglong2 b = make_ulonglong2(kInvalidHash, 0);
    if (r != kEmptyRank) {
      const uint32_t o = start[r];
      count = start[r + 1] - o;
      b = make_ulonglong2(keys[r], static_cast<uint64_t>(o) | static_cast<uint64_t>(count) << 32);
    }
    table[s] = b;
  }
  count = __reduce_max_sync(0xffffffffu, count);
  if ((threadIdx.x & 31) == 0 && count > *max_count) atomicMax(max_count, count);
}

inline unsigned blocks_for(int64_t n, int t = 256) { return static_cast<unsigned>((n + t - 1) / t); }

}  // namespace

// Arrays cut one after another from the workspace; without one (base null), only counted.
struct Cutter {
  uint8_t* base;
  size_t used = 0;
  template <class T>
  T* get(size_t count) {
    T* p = reinterpret_cast<T*>(base + used);
    used += ((count ? count : 1) * sizeof(T) + 255) & ~size_t(255);
    return p;
  }
};

namespace {

struct RunScan {  // N runs
  int64_t words;
  uint32_t *count, *first;
  void* tmp;
  size_t tmp_bytes = 0;
  RunScan(Cutter& cut, uint64_t n_bases) {
    words = static_cast<int64_t>((n_bases + 31) / 32);
    count = cut.get<uint32_t>(words + 1);
    first = cut.get<uint32_t>(words + 1);
    cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, count, first, words + 1);
    tmp = cut.get<uint8_t>(tmp_bytes);
  }
};

struct TileScan {  // minimizers
  int64_t words;
  uint32_t *bits, *count, *first, *tile_word, *flags;
  int64_t* first_tile;
  void* tmp;
  size_t tmp_bytes = 0;
  TileScan(Cutter& cut, int64_t n_tiles, int32_t n_contigs) {
    words = n_tiles * kTileWords;
    bits = cut.get<uint32_t>(words);
    count = cut.get<uint32_t>(words + 1);
    first = cut.get<uint32_t>(words + 1);
    tile_word = cut.get<uint32_t>(n_tiles);
    flags = cut.get<uint32_t>(2);  // [0] error bits, [1] largest count
    first_tile = cut.get<int64_t>(static_cast<size_t>(n_contigs) + 1);
    cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, count, first, words + 1);
    tmp = cut.get<uint8_t>(tmp_bytes);
  }
};

struct KeySort {  // the second half, once the minimizers are counted
  uint64_t *h_in, *h_out, *keys;
  uint32_t *v_in, *v_out, *head, *rank, *start, *slot_rank;
  void* tmp;
  size_t tmp_bytes;
  static uint64_t buckets(uint64_t n_keys) {
    uint64_t cap = 16;
    while (cap < n_keys * 2) cap <<= 1;
    return cap;
  }
  KeySort(Cutter& cut, int64_t n_min, int k) {
    h_in = cut.get<uint64_t>(n_min);
    h_out = cut.get<uint64_t>(n_min);
    keys = cut.get<uint64_t>(n_min);
    v_in = cut.get<uint32_t>(n_min);
    v_out = cut.get<uint32_t>(n_min);
    head = cut.get<uint32_t>(n_min + 1);
    rank = cut.get<uint32_t>(n_min + 1);
    start = cut.get<uint32_t>(n_min + 1);
    slot_rank = cut.get<uint32_t>(buckets(static_cast<uint64_t>(n_min)));
    size_t a = 0, b = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, a, h_in, h_out, v_in, v_out, n_min, 0, 2 * k);
    cub::DeviceScan::ExclusiveSum(nullptr, b, head, rank, n_min + 1);
    tmp_bytes = a > b ? a : b;
    tmp = cut.get<uint8_t>(tmp_bytes);
  }
};

int report(char* err, size_t err_len, const char* what, cudaError_t e) {
  snprintf(err, err_len, "index build (%s): %s", what, cudaGetErrorString(e));
  cudaGetLastError();
  return e == cudaErrorMemoryAllocation ? DNALN_ERR_OOM : DNALN_ERR_CUDA;
}

}  // namespace

int find_n_runs_on_device(cudaStream_t st, const uint8_t* d_genome, uint64_t n_bases, uint2** runs_out,
                          int32_t* n_runs_out, char* err, size_t err_len) {
  *runs_out = nullptr;
  *n_runs_out = 0;
  Cutter size{nullptr};
  RunScan(size, n_bases);
  struct Slab {
    void* p = nullptr;
    ~Slab() { cudaFree(p); }
  } slab;
  cudaError_t e = cudaMalloc(&slab.p, size.used);
  if (e != cudaSuccess) return report(err, err_len, "N runs", e);
  Cutter cut{static_cast<uint8_t*>(slab.p)};
  RunScan rs(cut, n_bases);
  const int64_t n = static_cast<int64_t>(n_bases);
  uint32_t n_runs = 0;
  k_word_counts<<<blocks_for(rs.words + 1), 256, 0, st>>>(d_genome, n, rs.words, rs.count);
  e = cub::DeviceScan::ExclusiveSum(rs.tmp, rs.tmp_bytes, rs.count, rs.first, rs.words + 1, st);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(&n_runs, rs.first + rs.words, sizeof n_runs, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  uint2* runs = nullptr;
  if (e == cudaSuccess) e = cudaMalloc(&runs, (n_runs ? n_runs : 1) * sizeof(uint2));
  if (e != cudaSuccess) return report(err, err_len, "N runs", e);
  *runs_out = runs;
  *n_runs_out = static_cast<int32_t>(n_runs);
  if (n_runs) k_word_runs<<<blocks_for(rs.words), 256, 0, st>>>(d_genome, n, rs.words, rs.first, runs);
  // the scratch is freed on return: the kernel must be done with it first
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess || (e = cudaGetLastError()) != cudaSuccess)
    return report(err, err_len, "N runs", e);
  return DNALN_OK;
}

int build_index_on_device(cudaStream_t st, const uint8_t* d_genome, uint64_t n_bases, const uint64_t* d_contig_off,
                          const uint32_t* d_contig_len, const uint32_t* contig_len, int32_t n_contigs, int k, int w,
                          const DeviceAlloc& workspace, const DeviceAlloc& keep, int64_t* pinned,
                          DeviceIndexBuild* out, char* err, size_t err_len) {
  *out = DeviceIndexBuild{};
  if (k < 4 || k > kMaxK || w < 1 || w > kMaxW) {
    snprintf(err, err_len, "index build: k or w out of range");
    return DNALN_ERR_INVALID_ARG;
  }
  const int64_t n = static_cast<int64_t>(n_bases);
  // tiles of window ends, never across a contig
  std::vector<int64_t> first_tile(static_cast<size_t>(n_contigs) + 1, 0);
  for (int32_t c = 0; c < n_contigs; ++c) first_tile[c + 1] = first_tile[c] + (contig_len[c] + kTile - 1) / kTile;
  const int64_t n_tiles = first_tile[n_contigs];
  // the workspace, at once for the usual density of 2 / (w + 1) minimizers per base and more
  Cutter size{nullptr};
  RunScan(size, n_bases);
  TileScan(size, n_tiles, n_contigs);
  KeySort(size, std::min<int64_t>(n, static_cast<int64_t>(2.6 * static_cast<double>(n) / (w + 1)) + 1024), k);
  void* slab = workspace(size.used);
  if (!slab) return report(err, err_len, "workspace", cudaErrorMemoryAllocation);
  const size_t have = size.used;
  Cutter cut{static_cast<uint8_t*>(slab)};
  RunScan rs(cut, n_bases);
  TileScan ts(cut, n_tiles, n_contigs);
  cudaError_t e = cudaMemcpyAsync(ts.first_tile, first_tile.data(), first_tile.size() * sizeof(int64_t),
                                  cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(ts.count + ts.words, 0, sizeof(uint32_t), st);
  if (e == cudaSuccess) e = cudaMemsetAsync(ts.flags, 0, 2 * sizeof(uint32_t), st);
  if (e != cudaSuccess) return report(err, err_len, "upload", e);
  // 1. minimizers in genome order, N runs
  if (n_tiles)
    k_genome_minimizers<<<static_cast<unsigned>(n_tiles), kThreads, 0, st>>>(
        d_genome, d_contig_off, d_contig_len, ts.first_tile, n_contigs, k, w, ts.bits, ts.count, ts.tile_word);
  k_word_counts<<<blocks_for(rs.words + 1), 256, 0, st>>>(d_genome, n, rs.words, rs.count);
  e = cub::DeviceScan::ExclusiveSum(ts.tmp, ts.tmp_bytes, ts.count, ts.first, ts.words + 1, st);
  if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(rs.tmp, rs.tmp_bytes, rs.count, rs.first, rs.words + 1, st);
  uint32_t* const got = reinterpret_cast<uint32_t*>(pinned);
  if (e == cudaSuccess) e = cudaMemcpyAsync(got, ts.first + ts.words, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(got + 1, rs.first + rs.words, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return report(err, err_len, "minimizer count", e);
  const int64_t n_min = got[0], n_runs = got[1];
  Cutter second{nullptr, cut.used};
  KeySort(second, n_min, k);
  // a genome denser than expected: the rest in an allocation of its own
  struct Slab {
    void* p = nullptr;
    ~Slab() {
      if (p) cudaFree(p);
    }
  } extra;
  if (second.used > have) {
    const size_t need = second.used - cut.used;
    if ((e = cudaMalloc(&extra.p, need)) != cudaSuccess) return report(err, err_len, "minimizer buffers", e);
    cut = Cutter{static_cast<uint8_t*>(extra.p)};
  }
  KeySort ks(cut, n_min, k);
  int64_t n_keys = 0;
  if (n_min) {
    k_word_minimizers<<<blocks_for(ts.words), 256, 0, st>>>(d_genome, ts.bits, ts.tile_word, ts.words, k, ts.first,
                                                            ks.h_in, ks.v_in);
    // 2. stable sort by hash: positions stay ascending within a key
    e = cub::DeviceRadixSort::SortPairs(ks.tmp, ks.tmp_bytes, ks.h_in, ks.h_out, ks.v_in, ks.v_out, n_min, 0, 2 * k,
                                        st);
    if (e != cudaSuccess) return report(err, err_len, "sort", e);
    // 3. distinct keys and their offsets
    k_key_heads<<<blocks_for(n_min + 1), 256, 0, st>>>(ks.h_out, n_min, ks.head);
    e = cub::DeviceScan::ExclusiveSum(ks.tmp, ks.tmp_bytes, ks.head, ks.rank, n_min + 1, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(got, ks.rank + n_min, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) {
      k_key_list<<<blocks_for(n_min + 1), 256, 0, st>>>(ks.h_out, n_min, ks.rank, ks.keys, ks.start);
      e = cudaStreamSynchronize(st);
    }
    if (e != cudaSuccess) return report(err, err_len, "distinct keys", e);
    n_keys = got[0];
  }
  // 4. the bucket table, with the positions and the N runs in one allocation
  const uint64_t cap = KeySort::buckets(static_cast<uint64_t>(n_keys));
  Cutter built{nullptr};
  built.get<ulonglong2>(cap);
  built.get<uint32_t>(static_cast<size_t>(n_min));
  built.get<uint2>(static_cast<size_t>(n_runs));
  void* mem = keep(built.used);
  if (!mem) return report(err, err_len, "table", cudaErrorMemoryAllocation);
  built = Cutter{static_cast<uint8_t*>(mem)};
  out->table = built.get<ulonglong2>(cap);
  out->positions = built.get<uint32_t>(static_cast<size_t>(n_min));
  out->n_runs = built.get<uint2>(static_cast<size_t>(n_runs));
  out->n_buckets = cap;
  out->n_pos = static_cast<uint64_t>(n_min);
  out->n_n_runs = static_cast<int32_t>(n_runs);
  e = cudaMemsetAsync(ks.slot_rank, 0xFF, cap * sizeof(uint32_t), st);
  if (e == cudaSuccess && n_min)
    e = cudaMemcpyAsync(out->positions, ks.v_out, n_min * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st);
  if (e != cudaSuccess) return report(err, err_len, "table", e);
  if (n_keys) k_place_keys<<<blocks_for(n_keys), 256, 0, st>>>(ks.keys, n_keys, cap - 1, ks.slot_rank, ts.flags);
  k_fill_table<<<blocks_for(static_cast<int64_t>(cap)), 256, 0, st>>>(ks.slot_rank, cap, ks.keys, ks.start, out->table,
                                                                       ts.flags + 1);
  if (n_runs) k_word_runs<<<blocks_for(rs.words), 256, 0, st>>>(d_genome, n, rs.words, rs.first, out->n_runs);
  if ((e = cudaMemcpyAsync(got, ts.flags, 2 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
      (e = cudaStreamSynchronize(st)) != cudaSuccess || (e = cudaGetLastError()) != cudaSuccess)
    return report(err, err_len, "kernels", e);
  if (got[0]) {
    snprintf(err, err_len, "index build: a key walked past every bucket (flags 0x%x)", got[0]);
    return DNALN_ERR_DEVICE;
  }
  out->n_keys = static_cast<uint64_t>(n_keys);
  out->max_count = got[1];
  out->mask = cap - 1;
  return DNALN_OK;
}

}  // namespace dnb
