// Prefix scan, stable LSD radix sort and tile binning.
//
// The reference bins with count → scan → expand (item-major) → stable 32-bit
// sort by depth → gather tile keys → stable 32-bit sort by tile → ranges
// (crates/gs-kernels/src/binning.rs:171-238, tile_binning.wgsl:30-103,
// crates/gs-wgpu/src/shaders/radix_sort.wgsl): sixteen 4-bit passes over the
// entries, equivalent to one sort by (tile, depth, entry index).
//
// Here the depth order is established on the ITEMS (one per surfel and view,
// 4 passes of 8 bits over N·V keys), items are expanded in that order, and
// the entries are stably sorted by tile id alone (⌈log2 tiles / 8⌉ passes,
// usually 2). Within one tile each item owns at most one entry and entry
// indices grow with item index, so the result is exactly the reference's
// (tile, depth, entry) order.
//
// All passes read element counts from device memory, so a step needs no host
// synchronisation and can be captured in a CUDA graph. A sort pass and the
// entry scan read their input once: a block takes a tile by ticket, publishes
// its counts and sums the tiles before it by looking back at their published
// counts (the single-pass scan of Merrill and Garland 2016; applied to radix
// passes by Adinets and Merrill, "Onesweep", 2022). A block only ever waits
// for tiles with lower tickets, which are running or done. The waits are
// bounded and end in the same result: a block that has waited long enough for
// a tile counts that tile itself, from the pass's input, which nothing writes
// meanwhile.
#include <algorithm>

#include <cub/block/block_reduce.cuh>
#include <cub/block/block_scan.cuh>

#include "gs_common.cuh"
#include "gs_kernels.h"

namespace gs {
namespace {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ uint64_t read_n(uint64_t n_host, const uint32_t* n_dev) {
  if (n_dev == nullptr) return n_host;
  uint64_t d = *n_dev;
  return d < n_host ? d : n_host;
}

// ------------------------------------------------------------------ scan
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_reduce(const uint32_t* in, uint64_t n_host,
                                                              const uint32_t* n_dev, unsigned long long* bsum) {
  const uint64_t n = read_n(n_host, n_dev);
  const uint64_t chunk = (n + gridDim.x - 1) / gridDim.x;
  const uint64_t beg = blockIdx.x * chunk, end = min(n, beg + chunk);
  unsigned long long s = 0;
  for (uint64_t i = beg + threadIdx.x; i < end; i += SCAN_THREADS) s += in[i];
  using BR = cub::BlockReduce<unsigned long long, SCAN_THREADS>;
  __shared__ typename BR::TempStorage tmp;
  s = BR(tmp).Sum(s);
  if (threadIdx.x == 0) bsum[blockIdx.x] = s;
}

__global__ void __launch_bounds__(SCAN_GRID) k_scan_blocks(unsigned long long* bsum, uint32_t* total_u32) {
  using BS = cub::BlockScan<unsigned long long, SCAN_GRID>;
  __shared__ typename BS::TempStorage tmp;
  unsigned long long v = bsum[threadIdx.x], excl, agg;
  BS(tmp).ExclusiveSum(v, excl, agg);
  bsum[threadIdx.x] = excl;
  if (threadIdx.x == 0 && total_u32) *total_u32 = agg > 0xffffffffull ? 0xffffffffu : (uint32_t)agg;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_down(const uint32_t* in, uint32_t* out, uint64_t n_host,
                                                            const uint32_t* n_dev, const unsigned long long* boff) {
  const uint64_t n = read_n(n_host, n_dev);
  const uint64_t chunk = (n + gridDim.x - 1) / gridDim.x;
  const uint64_t beg = blockIdx.x * chunk, end = min(n, beg + chunk);
  using BS = cub::BlockScan<uint32_t, SCAN_THREADS>;
  __shared__ typename BS::TempStorage tmp;
  uint32_t running = (uint32_t)boff[blockIdx.x];
  for (uint64_t t0 = beg; t0 < end; t0 += SCAN_TILE) {
    uint32_t v[SCAN_ITEMS];
    uint32_t loc = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
      const uint64_t i = t0 + (uint64_t)threadIdx.x * SCAN_ITEMS + k;
      v[k] = i < end ? in[i] : 0u;
      loc += v[k];
    }
    uint32_t excl, agg;
    BS(tmp).ExclusiveSum(loc, excl, agg);
    uint32_t r = running + excl;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
      const uint64_t i = t0 + (uint64_t)threadIdx.x * SCAN_ITEMS + k;
      if (i < end) out[i] = r;
      r += v[k];
    }
    running += agg;
    __syncthreads();
  }
}

// ------------------------------------------------------- bounded look-back
// Words of a sort's or scan's header (zeroed by launch_sort_reset).
constexpr int SH_HIST = 0;        // [4][256] digit counts of all passes
constexpr int SH_TICKET = 1024;   // [4] tile tickets, one per pass
static_assert(SH_TICKET + 4 <= SORT_HDR_WORDS, "header words");

// A published count: the state in the top two bits, the value below. Flag and
// value travel in one word, so relaxed accesses suffice.
template <typename W>
struct Published {
  static constexpr int SHIFT = (int)sizeof(W) * 8 - 2;
  static constexpr W VALUE = ((W)1 << SHIFT) - 1;
  static constexpr W AGGREGATE = (W)1 << SHIFT;  // the tile's own count
  static constexpr W PREFIX = (W)2 << SHIFT;     // the count of all tiles up to and including this one
};
__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Sum of everything before tile t in the column of published words at
// `col` (stride `stride` words per tile), t > 0. LB predecessors are read at
// once, so a chain of tiles that published only their own counts costs one
// memory latency per LB tiles. After `wait` cycles without the next tile's
// word, `recount` (tile -> its own count) takes its place: the sum is the
// same, and the loop ends whatever the other blocks do.
template <int LB, typename W, class F>
__device__ __forceinline__ W look_back(const W* col, uint32_t stride, uint32_t t, long long wait, F&& recount) {
  using P = Published<W>;
  W sum = 0;
  uint32_t left = t;  // tiles [0, left) still to be summed
  long long t0 = 0;
  for (;;) {
    W v[LB];
#pragma unroll
    for (int k = 0; k < LB; ++k)
      v[k] = (uint32_t)k < left ? ld_relaxed(col + (size_t)(left - 1 - k) * stride) : P::PREFIX;
    bool stop = false;
    uint32_t used = 0;
#pragma unroll
    for (int k = 0; k < LB; ++k) {
      if (!stop) {
        if ((v[k] & ~P::VALUE) == 0) {
          stop = true;
        } else {
          sum += v[k] & P::VALUE;
          ++used;
          if (v[k] & P::PREFIX) return sum;
        }
      }
    }
    left -= used;
    if (stop && used == 0) {
      const long long now = clock64();
      if (t0 == 0) t0 = now;
      if (now - t0 >= wait) {
        sum += recount(left - 1);
        --left;
        t0 = 0;
      }
    } else {
      t0 = 0;
    }
  }
}

// ------------------------------------------------------------ radix sort
// LSD passes of up to 8-bit digits (the key bits spread evenly over the
// passes). One kernel counts the digits of every pass; then one kernel per
// pass takes tiles of RS_TILE elements by ticket: warp w holds elements
// [256w, 256w+256) of the tile in 8 rounds of 32, ranks them stably by
// ballot multi-split, the block combines the warps' digit counts in warp
// order, publishes them, reorders the tile through shared memory while the
// tiles before it publish theirs, looks back for its digits' positions and
// writes the tile out in digit runs. Elements are (key, value) pairs, either
// in two arrays or interleaved as uint2.
//
// Against counting, scanning and scattering in five kernels per pass, each
// pass reads its input once instead of twice, and a 32-bit sort takes 6
// launches instead of 20. Whole 32-bit sorts of random keys in two arrays,
// kernel time before and after: 16 thousand pairs 69 -> 33 us, 300 thousand
// 76 -> 43, 1 million 97 -> 62, 4 million 182 -> 161, 12 million 585 -> 436; 32
// million pairs of 16 bits 772 -> 566 us. Tile sorts of interleaved entries in
// depth order, the larger ones by chunks (below): 2.9 million 85 -> 62 us, 8.6
// million 164 -> 161, the 33 million of a 1080p frame 532 -> 516. A tile takes 6
// us by itself (chains of ballots, barriers and L2 round trips), and the
// look-back grows with the tiles in flight: 2 blocks of 512 threads per SM ran
// the 4-million pass in 39 us (37.5 since match_digit has no branches), 3 blocks
// in 52, 6 of 256 threads in 71, 8192-element tiles in 46 to 53; reading 16 or
// 32 tiles back at once instead of 8, 40 and 43 us.
constexpr int RS_THREADS = 512;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_ROUNDS = RS_TILE / RS_THREADS;     // elements per thread per tile
constexpr int RS_BINS = 256;
constexpr int RS_CTAS = 2;                          // resident blocks per SM
static_assert(RS_TILE == RS_THREADS * RS_ROUNDS && RS_ROUNDS % 2 == 0, "whole rounds");
static_assert(RS_THREADS >= RS_BINS, "one thread per digit");

// Lanes of the warp whose digit (of nbits bits, nothing above them) equals this
// lane's: multi-split by ballots, one per bit. Without a test for each bit:
// with `if (b < nbits)` around it, every bit of every round was a branch
// (156 million instructions a pass at 29 million pairs, 105 now; whole sorts of
// 32 million pairs of 16 bits 627 -> 563 us, tile sorts of 2.9 million entries 71
// -> 62). SHORT (tile ids, whose digits are often of 6 bits): the last two only
// where they are used (29 million 252 -> 230 us for a pass of 6 bits; random keys
// of 8 bits lose 2 % by it).
template <bool SHORT>
__device__ __forceinline__ uint32_t match_digit(uint32_t d, int nbits, uint32_t active) {
  uint32_t peers = active;
  auto step = [&](int b) {
    const uint32_t bal = __ballot_sync(FULL, (d >> b) & 1u);
    peers &= bal ^ (((d >> b) & 1u) - 1u);
  };
#pragma unroll
  for (int b = 0; b < 6; ++b) step(b);
  if (!SHORT || nbits > 6) {
    step(6);
    step(7);
  }
  return peers;
}

// Many interleaved pairs go by chunks of whole tiles, one per half of a
// resident block (chunk_pass). Against tiles by look-back, a tile's ranking
// and writing then overlap the next tile's loads, and there is one look-back
// per chunk; but every pass after the first reads its keys once more to count
// them. Tile sorts (two passes) of entries in depth order, counting included:
// 2.9 million 62 us by look-back and 74 by chunks, 5.8 million 113 and 115, 8.6
// million 157 and 161, two frames of 9.5 million 349 and 318, 11.5 million 216
// and 204, 18 million 341 and 317, 29 million 510 and 464, the 33 million of a
// 1080p frame 580 and 516. With one pass (up to 256 tiles) look-back stays
// ahead (5.8 million 96 and 131), and so it does for two arrays (32 million
// pairs of 16 bits: 294 us a pass by look-back when chunks, counted and scanned
// by kernels of their own, took 341).
constexpr int RC_THREADS = RS_THREADS / 2, RC_WARPS = RC_THREADS / 32;
constexpr int RC_TILE = RS_TILE / 2, RC_ROUNDS = RC_TILE / RC_THREADS;
constexpr uint32_t RC_CHUNKS = 148 * RS_CTAS * 2;
constexpr int RC_GROUP = 25;  // chunks whose counts are summed first
constexpr int RC_GROUPS = (RC_CHUNKS + RC_GROUP - 1) / RC_GROUP;
constexpr uint64_t RC_MIN = 9000000;
static_assert(RC_THREADS == RS_BINS, "one thread per digit");
static_assert(RC_CHUNKS + RC_GROUPS <= RC_MIN / RS_TILE, "look-back words of the chunks and their groups");
static_assert(RC_GROUPS <= RC_GROUP, "a look-back reads all groups at once");
__device__ __forceinline__ uint64_t chunk_len(uint64_t n) {
  return ((n + RC_CHUNKS - 1) / RC_CHUNKS + RC_TILE - 1) / RC_TILE * RC_TILE;
}

// Element access: two arrays, or one interleaved uint2 array.
// SplitIO's optional gather (final pass only): gdst[position] = gsrc[value],
// e.g. each item's tile count in sorted order for the entry scan, which then
// reads it sequentially instead of through the permutation. PairIO's optional
// value array (final pass only) receives the values alone.
struct SplitIO {
  static constexpr bool CHUNKS = false, SHORT = false;
  const uint32_t* kin; const uint32_t* vin; uint32_t* kout; uint32_t* vout;
  const uint32_t* gsrc = nullptr; uint32_t* gdst = nullptr;
  SplitIO plain() const { SplitIO y = *this; y.gdst = nullptr; return y; }
  __device__ __forceinline__ void skip(uint64_t b) { kin += b; vin += b; kout += b; vout += b; }
  __device__ __forceinline__ uint32_t key(uint64_t i) const { return __ldg(kin + i); }
  __device__ __forceinline__ uint2 load(uint64_t i) const { return make_uint2(kin[i], vin[i]); }
  __device__ __forceinline__ void store(size_t g, uint2 e) const {
    kout[g] = e.x;
    vout[g] = e.y;
    if (gdst != nullptr) gdst[g] = __ldg(gsrc + e.y);
  }
};
template <bool BY_CHUNKS>  // RC_MIN elements and more go by chunks
struct PairIO {
  static constexpr bool CHUNKS = BY_CHUNKS, SHORT = true;
  const uint2* in; uint2* out;
  uint32_t* values = nullptr;
  PairIO plain() const { PairIO y = *this; y.values = nullptr; return y; }
  __device__ __forceinline__ void skip(uint64_t b) { in += b; out += b; }
  __device__ __forceinline__ uint32_t key(uint64_t i) const {
    return __ldg(reinterpret_cast<const uint32_t*>(in + i));
  }
  __device__ __forceinline__ uint2 load(uint64_t i) const { return __ldg(in + i); }
  __device__ __forceinline__ void store(size_t g, uint2 e) const {
    if (values != nullptr) values[g] = e.y;
    else out[g] = e;
  }
};

// Digit counts of every pass in one read of the keys; also zeroes the first
// pass's look-back words (each pass zeroes the next one's) and, for the tile
// sort, the ranges its final pass fills. Blocks take contiguous chunks of at
// least 8 tiles' worth of threads, so that few elements flush few counters.
constexpr int RH_THREADS = 512;
static_assert(RC_MIN >= (uint64_t)RC_CHUNKS * 8 * RH_THREADS, "k_rs_hist has a block per chunk");
template <class IO, typename W>
__global__ void __launch_bounds__(RH_THREADS) k_rs_hist(IO io, uint64_t n_host, const uint32_t* n_dev, int passes,
                                                        int dbits, int key_bits, uint32_t* hdr, W* state,
                                                        uint2* ranges, uint32_t num_ranges,
                                                        const unsigned long long* base) {
  __shared__ uint32_t s_h[4][RS_BINS];
  const int tid = threadIdx.x;
  for (int k = tid; k < 4 * RS_BINS; k += RH_THREADS) (&s_h[0][0])[k] = 0;
  const uint64_t gtid = (uint64_t)blockIdx.x * RH_THREADS + tid, gsize = (uint64_t)gridDim.x * RH_THREADS;
  for (uint64_t k = gtid; k < num_ranges; k += gsize) ranges[k] = make_uint2(0u, 0u);
  const uint64_t n = read_n(n_host, n_dev);
  const bool by_chunks = IO::CHUNKS && n >= RC_MIN;
  if (by_chunks) {  // (a chunk's own words are written below)
    if (blockIdx.x < RC_GROUPS && tid < RS_BINS) state[(size_t)(RC_CHUNKS + blockIdx.x) * RS_BINS + tid] = 0;
  } else {
    const uint64_t words = (n + RS_TILE - 1) / RS_TILE * RS_BINS;
    for (uint64_t k = gtid; k < words; k += gsize) state[k] = 0;
  }
  const uint64_t chunk =
      by_chunks ? chunk_len(n) : max((n + gridDim.x - 1) / gridDim.x, (uint64_t)(8 * RH_THREADS));
  const uint64_t beg = blockIdx.x * chunk, end = min(n, beg + chunk);
  if (beg >= end) return;
  if (base != nullptr) io.skip(*base);
  __syncthreads();
  const uint32_t mask = (1u << dbits) - 1u;
  const uint32_t top = key_bits < 32 ? (1u << key_bits) - 1u : 0xffffffffu;
  auto count = [&](uint32_t key) {
    key &= top;
#pragma unroll
    for (int p = 0; p < 4; ++p)
      if (p < passes) atomicAdd(&s_h[p][(key >> (p * dbits)) & mask], 1u);
  };
  uint64_t i = beg + tid;
  for (; i + 3 * RH_THREADS < end; i += 4 * RH_THREADS) {
    const uint32_t k0 = io.key(i), k1 = io.key(i + RH_THREADS), k2 = io.key(i + 2 * RH_THREADS),
                   k3 = io.key(i + 3 * RH_THREADS);
    count(k0); count(k1); count(k2); count(k3);
  }
  for (; i < end; i += RH_THREADS) count(io.key(i));
  __syncthreads();
  for (int k = tid; k < passes * RS_BINS; k += RH_THREADS) {
    const uint32_t c = (&s_h[0][0])[k];
    if (c) atomicAdd(hdr + SH_HIST + k, c);
    if (by_chunks && k < RS_BINS)  // the first pass's counts of this chunk
      state[(size_t)blockIdx.x * RS_BINS + k] = Published<W>::AGGREGATE | (W)c;
  }
}

// How many of a whole tile's, or a range of tiles', keys have this digit
// (look_back's recount). Not inlined: it is hardly ever called, and the passes
// are short of registers (sort of 4 million pairs 223 us without it, 220 with).
template <class IO>
__device__ __noinline__ uint32_t count_digit(IO io, uint64_t tile, int shift, uint32_t mask, uint32_t digit) {
  uint32_t c = 0;
#pragma unroll 8
  for (int i = 0; i < RS_TILE; ++i) c += ((io.key(tile * RS_TILE + i) >> shift) & mask) == digit;
  return c;
}
template <class IO>
__device__ __noinline__ uint32_t count_range(IO io, uint64_t beg, uint64_t end, int shift, uint32_t mask,
                                             uint32_t digit) {
  uint32_t c = 0;
#pragma unroll 4
  for (uint64_t i = beg; i < end; ++i) c += ((io.key(i) >> shift) & mask) == digit;
  return c;
}

// A pass over many pairs (RC_MIN and more): half h of block b moves chunk
// 2b + h of the input tile by tile, the next tile's elements in flight during
// the write-out. It counts the chunk's digits first (the first pass finds them
// in its look-back words, from k_rs_hist), adds the counts of the chunks before
// it, its group's one by one and then the earlier groups', and needs no other
// chunk after that. Only lower blocks and the own first half are waited for,
// with look_back's bound. (Chunks by block number, not by ticket: 265 instead
// of 282 us a pass at 33 million pairs.)
template <class IO, typename W>
__device__ __forceinline__ void chunk_pass(const IO& io, uint64_t n, int pass, int shift, int nbits, W* state,
                                           W* next_state, uint2* ranges, uint32_t num_ranges, uint32_t b0,
                                           long long wait, uint2* s_e, uint16_t (*s_wh)[RS_BINS], uint32_t* s_start,
                                           uint32_t* s_gofs, uint32_t* s_warp, uint32_t digit_base) {
  using P = Published<W>;
  const int half = threadIdx.x / RC_THREADS, tid = threadIdx.x % RC_THREADS, lane = tid & 31, warp = tid >> 5;
  auto sync_half = [&] {
    if (half) asm volatile("bar.sync 2, %0;" ::"n"(RC_THREADS) : "memory");
    else asm volatile("bar.sync 1, %0;" ::"n"(RC_THREADS) : "memory");
  };
  const uint32_t mask = (1u << nbits) - 1u;
  const uint64_t len = chunk_len(n);
  const uint32_t c = 2 * blockIdx.x + half, group = c / RC_GROUP, at = c % RC_GROUP;
  const uint64_t beg = c * len, end = min(n, beg + len);
  if (beg >= n) return;
  W* mine = state + (size_t)c * RS_BINS + tid;
  W* groups = state + (size_t)RC_CHUNKS * RS_BINS + tid;
  if (next_state != nullptr) {
    next_state[(size_t)c * RS_BINS + tid] = 0;
    if (at == 0) next_state[(size_t)(RC_CHUNKS + group) * RS_BINS + tid] = 0;
  }
  W cnt;
  if (pass == 0) {
    cnt = *mine & P::VALUE;
  } else {
    uint32_t* h = reinterpret_cast<uint32_t*>(s_e);  // [RC_WARPS][RS_BINS]
    for (int k = tid; k < RC_WARPS * RS_BINS; k += RC_THREADS) h[k] = 0;
    sync_half();
    uint32_t* hw = h + warp * RS_BINS;
    uint64_t i = beg + tid;
    for (; i + 3 * RC_THREADS < end; i += 4 * RC_THREADS) {
      uint32_t k[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) k[u] = io.key(i + u * RC_THREADS);
#pragma unroll
      for (int u = 0; u < 4; ++u) atomicAdd(hw + ((k[u] >> shift) & mask), 1u);
    }
    for (; i < end; i += RC_THREADS) atomicAdd(hw + ((io.key(i) >> shift) & mask), 1u);
    sync_half();
    uint32_t s = 0;
#pragma unroll
    for (int w = 0; w < RC_WARPS; ++w) s += h[w * RS_BINS + tid];
    cnt = s;
    st_relaxed(mine, P::AGGREGATE | cnt);
    sync_half();  // h is the staged tile's memory
  }
  auto recount = [&](uint64_t from, uint32_t chunks) {
    return (W)count_range(io, from * len, (from + chunks) * len, shift, mask, (uint32_t)tid);
  };
  W before = 0;
  if (at > 0)
    before = look_back<RC_GROUP>(state + (size_t)(c - at) * RS_BINS + tid, RS_BINS, at, wait,
                                 [&](uint32_t k) { return recount(c - at + k, 1); });
  if (at == RC_GROUP - 1) st_relaxed(groups + (size_t)group * RS_BINS, P::AGGREGATE | (before + cnt));
  if (group > 0)
    before += look_back<RC_GROUP>(groups, RS_BINS, group, wait,
                                  [&](uint32_t k) { return recount((uint64_t)k * RC_GROUP, RC_GROUP); });
  uint32_t run = digit_base + (uint32_t)before;  // where this digit's next element goes
  uint2 e[RC_ROUNDS];
  auto load_tile = [&](uint64_t t0) {
    const int tn = (int)min((uint64_t)RC_TILE, end - t0);
#pragma unroll
    for (int r = 0; r < RC_ROUNDS; ++r) {
      const int idx = warp * (RC_ROUNDS * 32) + r * 32 + lane;
      e[r] = idx < tn ? io.load(t0 + idx) : make_uint2(0u, 0u);
    }
  };
  load_tile(beg);
  for (uint64_t t0 = beg; t0 < end; t0 += RC_TILE) {
    const int tn = (int)min((uint64_t)RC_TILE, end - t0);
    for (int k = tid; k < RC_WARPS * RS_BINS / 2; k += RC_THREADS) reinterpret_cast<uint32_t*>(&s_wh[0][0])[k] = 0;
    sync_half();
    uint32_t pre[RC_ROUNDS];  // ranks within (warp, digit)
#pragma unroll
    for (int r = 0; r < RC_ROUNDS; ++r) {
      const int idx = warp * (RC_ROUNDS * 32) + r * 32 + lane;
      const bool valid = idx < tn;
      const uint32_t d = (e[r].x >> shift) & mask;
      const uint32_t act = __ballot_sync(FULL, valid);
      const uint32_t peers = match_digit<true>(d, nbits, act);
      uint32_t basev = 0;
      if (valid) basev = s_wh[warp][d];
      __syncwarp();
      if (valid && (peers & lanemask_lt()) == 0) s_wh[warp][d] = (uint16_t)(basev + __popc(peers));
      __syncwarp();
      pre[r] = basev + __popc(peers & lanemask_lt());
    }
    sync_half();
    uint32_t s = 0;
#pragma unroll
    for (int w = 0; w < RC_WARPS; ++w) {
      const uint32_t x = s_wh[w][tid];
      s_wh[w][tid] = (uint16_t)s;
      s += x;
    }
    uint32_t excl = s;  // inclusive over the warp, then exclusive over the half
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(FULL, excl, o);
      if (lane >= o) excl += x;
    }
    if (lane == 31) s_warp[warp] = excl;
    sync_half();
    excl -= s;
#pragma unroll
    for (int w = 0; w < RC_WARPS; ++w)
      if (w < warp) excl += s_warp[w];
    s_start[tid] = excl;
    s_gofs[tid] = run - excl;  // output position = s_gofs[d] + position in the tile
    run += s;
    sync_half();
#pragma unroll
    for (int r = 0; r < RC_ROUNDS; ++r) {
      const int idx = warp * (RC_ROUNDS * 32) + r * 32 + lane;
      if (idx < tn) {
        const uint32_t d = (e[r].x >> shift) & mask;
        s_e[s_start[d] + s_wh[warp][d] + pre[r]] = e[r];
      }
    }
    if (t0 + RC_TILE < end) load_tile(t0 + RC_TILE);
    sync_half();
#pragma unroll 4
    for (int i = tid; i < tn; i += RC_THREADS) {
      const uint2 v = s_e[i];
      const uint32_t pos = s_gofs[(v.x >> shift) & mask] + (uint32_t)i;
      io.store((size_t)pos, v);
      if (ranges != nullptr && v.x < num_ranges) {
        if (i == 0 || s_e[i - 1].x != v.x) atomicMax(&ranges[v.x].x, ~(b0 + pos));
        if (i == tn - 1 || s_e[i + 1].x != v.x) atomicMax(&ranges[v.x].y, b0 + pos + 1u);
      }
    }
    sync_half();
  }
}

// ranges (final pass of a key sort only, else null): every run of one key
// inside a staged tile is folded into that key's output range, stored as
// (~first position, one past the last position) with atomicMax on both, so
// the zero-filled buffer needs no other initialisation (launch_ranges_fix
// turns it into [start, end) afterwards). Staged tiles are ordered by the
// full key in the final pass: by this pass's digit, and within a digit by
// the lower digits the earlier passes sorted.
template <class IO, typename W>
__global__ void __launch_bounds__(RS_THREADS, RS_CTAS) k_rs_pass(IO io, uint64_t n_host, const uint32_t* n_dev,
                                                                 int pass, int shift, int nbits,
                                                                 uint32_t* hdr, W* state, W* next_state, uint2* ranges,
                                                                 uint32_t num_ranges, const unsigned long long* base,
                                                                 long long wait) {
  using P = Published<W>;
  __shared__ uint2 s_e[RS_TILE];
  __shared__ uint16_t s_wh[RS_WARPS][RS_BINS];
  constexpr int HALVES = IO::CHUNKS ? 2 : 1;  // chunk_pass: each half has its own
  __shared__ uint32_t s_start[HALVES * RS_BINS], s_gofs[HALVES * RS_BINS];
  __shared__ uint32_t s_tile;
  using BS = cub::BlockScan<uint32_t, RS_THREADS>;
  __shared__ typename BS::TempStorage tmp;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint64_t n = read_n(n_host, n_dev);
  const uint32_t tiles = (uint32_t)((n + RS_TILE - 1) / RS_TILE);
  if (blockIdx.x >= tiles) return;
  const uint32_t b0 = base != nullptr ? (uint32_t)*base : 0u;  // range positions are whole-buffer positions
  if (b0) io.skip(b0);
  const uint32_t mask = (1u << nbits) - 1u;
  uint32_t digit_base;
  BS(tmp).ExclusiveSum(tid < RS_BINS ? hdr[SH_HIST + pass * RS_BINS + tid] : 0u, digit_base);
  if constexpr (IO::CHUNKS) {
    if (n >= RC_MIN) {
      __shared__ uint32_t s_warp[2][RC_WARPS];
      if (tid < RS_BINS) s_start[tid] = s_start[RS_BINS + tid] = digit_base;
      __syncthreads();
      digit_base = s_start[tid];
      const int half = tid / RC_THREADS;
      chunk_pass<IO, W>(io, n, pass, shift, nbits, state, next_state, ranges, num_ranges, b0, wait,
                        s_e + half * RC_TILE, s_wh + half * RC_WARPS, s_start + half * RS_BINS,
                        s_gofs + half * RS_BINS, s_warp[half], digit_base);
      return;
    }
  }
  for (;;) {
    if (tid == 0) s_tile = atomicAdd(hdr + SH_TICKET + pass, 1u);
    for (int k = tid; k < RS_WARPS * RS_BINS / 2; k += RS_THREADS) reinterpret_cast<uint32_t*>(&s_wh[0][0])[k] = 0;
    __syncthreads();
    const uint32_t t = s_tile;
    if (t >= tiles) return;
    const uint64_t t0 = (uint64_t)t * RS_TILE;
    const int tn = (int)min((uint64_t)RS_TILE, n - t0);
    uint2 e[RS_ROUNDS];
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; ++r) {
      const int idx = warp * (RS_ROUNDS * 32) + r * 32 + lane;
      e[r] = idx < tn ? io.load(t0 + idx) : make_uint2(0u, 0u);
    }
    if (next_state != nullptr && tid < RS_BINS) next_state[(size_t)t * RS_BINS + tid] = 0;
    uint32_t pre[RS_ROUNDS / 2];  // 16-bit ranks within (warp, digit)
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; ++r) {
      const int idx = warp * (RS_ROUNDS * 32) + r * 32 + lane;
      const bool valid = idx < tn;
      const uint32_t d = (e[r].x >> shift) & mask;
      const uint32_t act = __ballot_sync(FULL, valid);
      const uint32_t peers = match_digit<IO::SHORT>(d, nbits, act);
      uint32_t basev = 0;
      if (valid) basev = s_wh[warp][d];
      __syncwarp();
      if (valid && (peers & lanemask_lt()) == 0) s_wh[warp][d] = (uint16_t)(basev + __popc(peers));
      __syncwarp();
      const uint32_t rank = basev + __popc(peers & lanemask_lt());
      if (r & 1) pre[r >> 1] |= rank << 16;
      else pre[r >> 1] = rank;
    }
    __syncthreads();
    uint32_t cnt = 0;
    W* mine = state + (size_t)t * RS_BINS + tid;
    if (tid < RS_BINS) {
#pragma unroll
      for (int w = 0; w < RS_WARPS; ++w) {
        const uint32_t c = s_wh[w][tid];
        s_wh[w][tid] = (uint16_t)cnt;
        cnt += c;
      }
      st_relaxed(mine, (t == 0 ? P::PREFIX : P::AGGREGATE) | (W)cnt);
    }
    uint32_t excl;
    BS(tmp).ExclusiveSum(cnt, excl);
    if (tid < RS_BINS) s_start[tid] = excl;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; ++r) {
      const int idx = warp * (RS_ROUNDS * 32) + r * 32 + lane;
      if (idx < tn) {
        const uint32_t d = (e[r].x >> shift) & mask;
        s_e[s_start[d] + s_wh[warp][d] + ((pre[r >> 1] >> (16 * (r & 1))) & 0xffffu)] = e[r];
      }
    }
    W before = 0;
    if (t > 0 && tid <= (int)mask) {
      before = look_back<8>(state + tid, RS_BINS, t, wait, [&](uint32_t tile) {
        return (W)count_digit(io, tile, shift, mask, (uint32_t)tid);
      });
      st_relaxed(mine, P::PREFIX | (before + (W)cnt));
    }
    if (tid < RS_BINS) s_gofs[tid] = digit_base + (uint32_t)before - excl;  // output position = s_gofs[d] + position in the tile
    __syncthreads();
#pragma unroll 4
    for (int i = tid; i < tn; i += RS_THREADS) {
      const uint2 v = s_e[i];
      const uint32_t pos = s_gofs[(v.x >> shift) & mask] + (uint32_t)i;
      io.store((size_t)pos, v);
      if (ranges != nullptr && v.x < num_ranges) {
        if (i == 0 || s_e[i - 1].x != v.x) atomicMax(&ranges[v.x].x, ~(b0 + pos));
        if (i == tn - 1 || s_e[i + 1].x != v.x) atomicMax(&ranges[v.x].y, b0 + pos + 1u);
      }
    }
    __syncthreads();
  }
}

// Few elements: one block sorts them through all passes in shared memory (no
// other launch, no counters to clear). Whole 32-bit sort of 3000 pairs:
// 69 us in 20 launches, 26 us here.
constexpr int SM_ROUNDS = 8;
static_assert(RS_SMALL == 1024 * SM_ROUNDS, "largest single-block sort");
template <int NT>
constexpr size_t small_smem() {
  return sizeof(uint2) * NT * SM_ROUNDS + sizeof(uint16_t) * (NT / 32) * RS_BINS;
}
template <int NT>
__global__ void __launch_bounds__(NT) k_rs_small(SplitIO io, int n, int passes, int dbits, int key_bits) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint2* s_e = reinterpret_cast<uint2*>(smem);
  uint16_t(*s_wh)[RS_BINS] = reinterpret_cast<uint16_t(*)[RS_BINS]>(smem + sizeof(uint2) * NT * SM_ROUNDS);
  __shared__ uint32_t s_start[RS_BINS];
  using BS = cub::BlockScan<uint32_t, NT>;
  __shared__ typename BS::TempStorage tmp;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint2 e[SM_ROUNDS];
#pragma unroll
  for (int r = 0; r < SM_ROUNDS; ++r) {
    const int idx = warp * (SM_ROUNDS * 32) + r * 32 + lane;
    e[r] = idx < n ? io.load(idx) : make_uint2(0u, 0u);
  }
  for (int p = 0; p < passes; ++p) {
    const int shift = p * dbits, nbits = min(dbits, key_bits - shift);
    const uint32_t mask = (1u << nbits) - 1u;
    for (int k = tid; k < (NT / 32) * RS_BINS / 2; k += NT) reinterpret_cast<uint32_t*>(&s_wh[0][0])[k] = 0;
    __syncthreads();
    uint32_t pre[SM_ROUNDS];
#pragma unroll
    for (int r = 0; r < SM_ROUNDS; ++r) {
      const int idx = warp * (SM_ROUNDS * 32) + r * 32 + lane;
      const bool valid = idx < n;
      const uint32_t d = (e[r].x >> shift) & mask;
      const uint32_t act = __ballot_sync(FULL, valid);
      const uint32_t peers = match_digit<false>(d, nbits, act);
      uint32_t basev = 0;
      if (valid) basev = s_wh[warp][d];
      __syncwarp();
      if (valid && (peers & lanemask_lt()) == 0) s_wh[warp][d] = (uint16_t)(basev + __popc(peers));
      __syncwarp();
      pre[r] = basev + __popc(peers & lanemask_lt());
    }
    __syncthreads();
    uint32_t cnt = 0;
    if (tid < RS_BINS) {
#pragma unroll
      for (int w = 0; w < NT / 32; ++w) {
        const uint32_t c = s_wh[w][tid];
        s_wh[w][tid] = (uint16_t)cnt;
        cnt += c;
      }
    }
    uint32_t excl;
    BS(tmp).ExclusiveSum(cnt, excl);
    if (tid < RS_BINS) s_start[tid] = excl;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < SM_ROUNDS; ++r) {
      const int idx = warp * (SM_ROUNDS * 32) + r * 32 + lane;
      if (idx < n) {
        const uint32_t d = (e[r].x >> shift) & mask;
        s_e[s_start[d] + s_wh[warp][d] + pre[r]] = e[r];
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < SM_ROUNDS; ++r) {
      const int idx = warp * (SM_ROUNDS * 32) + r * 32 + lane;
      if (idx < n) e[r] = s_e[idx];
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < SM_ROUNDS; ++r) {
    const int idx = warp * (SM_ROUNDS * 32) + r * 32 + lane;
    if (idx < n) io.store(idx, e[r]);
  }
}

// -------------------------------------------------------------- entry scan
__device__ __forceinline__ uint32_t scan_in(const uint32_t* in, const uint32_t* perm, uint64_t i) {
  return perm ? in[perm[i]] : in[i];
}

// Exclusive scan of the items' tile counts in one pass over tiles of
// ES_TILE, and the entry-capacity guard: when the scene needs more entries
// than were allocated (base + total > capacity), the totals are set to zero
// so that no later pass reads an entry that was never written.
constexpr int ES_THREADS = 256, ES_ITEMS = ES_TILE / ES_THREADS;
__global__ void __launch_bounds__(ES_THREADS) k_entry_scan(EntryScanArgs a, uint32_t* hdr, unsigned long long* state,
                                                           long long wait) {
  using P = Published<unsigned long long>;
  using BS = cub::BlockScan<unsigned long long, ES_THREADS>;
  __shared__ typename BS::TempStorage tmp;
  __shared__ unsigned long long s_before;
  __shared__ uint32_t s_tile;
  const int tid = threadIdx.x, lane = tid & 31;
  const uint64_t n = read_n(a.n_host, a.n_dev);
  const uint32_t tiles = n ? (uint32_t)((n + ES_TILE - 1) / ES_TILE) : 1u;
  auto finish = [&](unsigned long long total) {
    if (a.capacity && (a.base != nullptr ? *a.base : 0ull) + total > a.capacity) {
      if (a.error_word != nullptr) atomicOr(a.error_word, ERR_ENTRY_CAPACITY);
      total = 0;
    }
    if (a.total_u32 != nullptr) *a.total_u32 = total > 0xffffffffull ? 0xffffffffu : (uint32_t)total;
    if (a.total_u64 != nullptr) *a.total_u64 = total;
  };
  for (;;) {
    if (tid == 0) s_tile = atomicAdd(hdr + SH_TICKET, 1u);
    __syncthreads();
    const uint32_t t = s_tile;
    if (t >= tiles) return;
    const uint64_t i0 = (uint64_t)t * ES_TILE + (uint64_t)tid * ES_ITEMS;
    uint32_t c[ES_ITEMS];
    if (a.perm == nullptr && i0 + ES_ITEMS <= n) {
#pragma unroll
      for (int k = 0; k < ES_ITEMS; k += 4) {
        const uint4 q = *reinterpret_cast<const uint4*>(a.in + i0 + k);
        c[k] = q.x; c[k + 1] = q.y; c[k + 2] = q.z; c[k + 3] = q.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < ES_ITEMS; ++k) c[k] = i0 + k < n ? scan_in(a.in, a.perm, i0 + k) : 0u;
    }
    unsigned long long loc = 0, excl, agg;
#pragma unroll
    for (int k = 0; k < ES_ITEMS; ++k) loc += c[k];
    BS(tmp).ExclusiveSum(loc, excl, agg);
    if (tid < 32) {  // the first warp looks back, 32 tiles at a time
      unsigned long long before = 0;
      if (lane == 0) st_relaxed(state + t, (t == 0 ? P::PREFIX : P::AGGREGATE) | agg);
      uint32_t left = t;
      long long t0 = 0;
      while (left > 0) {
        const unsigned long long v = (uint32_t)lane < left ? ld_relaxed(state + (left - 1 - lane)) : P::PREFIX;
        const uint32_t ready = __ballot_sync(FULL, (v & ~P::VALUE) != 0);
        const uint32_t pref = __ballot_sync(FULL, (v & P::PREFIX) != 0);
        const int run = ready == FULL ? 32 : __ffs(~ready) - 1;           // lanes 0..run-1 are published
        const int first = pref ? __ffs(pref) - 1 : 32;                    // the nearest prefix
        const int take = first < run ? first + 1 : run;
        before += warp_sum(lane < take ? (v & P::VALUE) : 0ull);
        if (first < run) break;
        left -= (uint32_t)take;
        if (take == 0) {
          const long long now = clock64();
          if (t0 == 0) t0 = now;
          if (__any_sync(FULL, now - t0 >= wait)) {  // sum the next tile (a whole one) here
            const uint64_t j0 = (uint64_t)(left - 1) * ES_TILE;
            unsigned long long s = 0;
            for (int k = lane; k < ES_TILE; k += 32) s += scan_in(a.in, a.perm, j0 + k);
            before += warp_sum(s);
            --left;
            t0 = 0;
          }
        } else {
          t0 = 0;
        }
      }
      if (lane == 0) {
        if (t > 0) st_relaxed(state + t, P::PREFIX | (before + agg));
        s_before = before;
        if (t + 1 == tiles) finish(before + agg);
      }
    }
    __syncthreads();
    uint32_t r = (uint32_t)(s_before + excl);
    if (i0 + ES_ITEMS <= n) {
#pragma unroll
      for (int k = 0; k < ES_ITEMS; k += 4) {
        uint4 q;
        q.x = r; r += c[k]; q.y = r; r += c[k + 1]; q.z = r; r += c[k + 2]; q.w = r; r += c[k + 3];
        *reinterpret_cast<uint4*>(a.out + i0 + k) = q;
      }
    } else {
#pragma unroll
      for (int k = 0; k < ES_ITEMS; ++k) {
        if (i0 + k < n) a.out[i0 + k] = r;
        r += c[k];
      }
    }
    __syncthreads();
  }
}

// --------------------------------------------------------------- binning
__global__ void __launch_bounds__(256) k_expand(ExpandArgs a) {
  const uint64_t n = read_n(a.n_items_host, a.n_items_dev);
  const uint64_t tot = *a.total;  // zeroed by the entry guard on overflow
  if (tot == 0 || tot > a.capacity) return;
  const int lane = threadIdx.x & 31;
  const uint64_t warps_total = (uint64_t)gridDim.x * (blockDim.x / 32);
  for (uint64_t w = (uint64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); w * 32 < n; w += warps_total) {
    const uint64_t k0 = w * 32, k = k0 + lane;
    const bool valid = k < n;
    uint32_t item = 0, cnt = 0, x0 = 0, y0 = 0, wd = 1, tb = 0, tx = a.tiles_x;
    if (valid) {
      item = a.perm[k];
      cnt = a.sorted_counts != nullptr ? a.sorted_counts[k] : a.counts[item];
      if (cnt) {
        const uint4 r = a.rects[item];
        x0 = r.x; y0 = r.y; wd = r.z - r.x + 1u;
      }
      if (a.views) {
        const ViewInfo* V = a.views + item / a.items_per_view;
        tb = (uint32_t)__ldg(&V->tile_base);
        tx = (uint32_t)__ldg(&V->tiles_x);
      }
    }
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += t;
    }
    const uint32_t excl = incl - cnt;
    const uint32_t total = __shfl_sync(FULL, incl, 31);
    const uint32_t off0 = a.offsets[k0];
    if ((uint64_t)off0 + total > a.capacity) {
      if (lane == 0 && total) atomicOr(a.error_word, ERR_ENTRY_CAPACITY);
      continue;
    }
    if (valid && a.entry_offset) a.entry_offset[item] = off0 + excl;
    for (uint32_t base = 0; base < total; base += 32) {
      const uint32_t j = base + lane;
      int owner = 0;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        const int c = owner + s;
        const uint32_t ec = __shfl_sync(FULL, excl, c < 32 ? c : 31);
        if (c < 32 && ec <= j) owner = c;
      }
      const uint32_t o_excl = __shfl_sync(FULL, excl, owner);
      const uint32_t o_wd = __shfl_sync(FULL, wd, owner);
      const uint32_t o_x0 = __shfl_sync(FULL, x0, owner);
      const uint32_t o_y0 = __shfl_sync(FULL, y0, owner);
      const uint32_t o_item = __shfl_sync(FULL, item, owner);
      const uint32_t o_tb = __shfl_sync(FULL, tb, owner);
      const uint32_t o_tx = __shfl_sync(FULL, tx, owner);
      if (j < total) {
        const uint32_t local = j - o_excl;
        const uint32_t ly = local / o_wd, lx = local - ly * o_wd;
        const uint32_t pos = off0 + j;
        const uint32_t key = o_tb + (o_y0 + ly) * o_tx + (o_x0 + lx);
        uint32_t val = o_item;
        if (a.val_mode == 1) {
          val = pos;
          a.exp_item[pos] = o_item;
        } else if (a.val_mode == 2) {
          val = a.ref_offsets[o_item] + local;
          if (val < tot) a.entry_items[val] = o_item;
        }
        a.pairs[pos] = make_uint2(key, val);
      }
    }
  }
}

// Filtered expansion (occlusion cut and its completion pass): the warp walks
// the candidate tiles of its 32 items' rects in launch_expand's order and
// keeps those the filter accepts, compacted by ballot, so each item's kept
// tiles land at its restricted offset in rect order.
__global__ void __launch_bounds__(256) k_expand_filtered(ExpandFilterArgs a) {
  const uint64_t n = read_n(a.n_items_host, a.n_items_dev);
  const uint64_t tot = *a.total;
  const uint64_t b = a.base != nullptr ? *a.base : 0ull;
  if (tot == 0 || b + tot > a.capacity) return;
  const int lane = threadIdx.x & 31;
  const uint64_t warps_total = (uint64_t)gridDim.x * (blockDim.x / 32);
  for (uint64_t w = (uint64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); w * 32 < n; w += warps_total) {
    const uint64_t k0 = w * 32, k = k0 + lane;
    uint32_t item = 0, cnt = 0, full = 0, x0 = 0, y0 = 0, wd = 1, tb = 0, tx = 0, key = 0;
    if (k < n) {
      item = a.perm[k];
      cnt = a.sorted_counts != nullptr ? a.sorted_counts[k] : a.counts[item];
      if (cnt) {
        const uint4 r = a.rects[item];
        x0 = r.x; y0 = r.y; wd = r.z - r.x + 1u;
        full = wd * (r.w - r.y + 1u);
        const ViewInfo* V = a.views + item / a.items_per_view;
        tb = (uint32_t)__ldg(&V->tile_base);
        tx = (uint32_t)__ldg(&V->tiles_x);
        if (a.cut != nullptr) key = a.key_by_item[item];
      }
    }
    uint32_t incl = full, incl_c = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(FULL, incl, o), tc = __shfl_up_sync(FULL, incl_c, o);
      if (lane >= o) { incl += t; incl_c += tc; }
    }
    const uint32_t excl = incl - full;
    const uint32_t total_full = __shfl_sync(FULL, incl, 31), total_cnt = __shfl_sync(FULL, incl_c, 31);
    if (total_cnt == 0) continue;
    const uint32_t off0 = a.offsets[k0];
    if ((uint64_t)off0 + total_cnt > tot) {
      if (lane == 0) atomicOr(a.error_word, ERR_ENTRY_CAPACITY);
      continue;
    }
    uint32_t run = 0;
    for (uint32_t basej = 0; basej < total_full; basej += 32) {
      const uint32_t j = basej + lane;
      int owner = 0;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        const int c = owner + s;
        const uint32_t ec = __shfl_sync(FULL, excl, c < 32 ? c : 31);
        if (c < 32 && ec <= j) owner = c;
      }
      const uint32_t o_excl = __shfl_sync(FULL, excl, owner);
      const uint32_t o_wd = __shfl_sync(FULL, wd, owner);
      const uint32_t o_x0 = __shfl_sync(FULL, x0, owner);
      const uint32_t o_y0 = __shfl_sync(FULL, y0, owner);
      const uint32_t o_item = __shfl_sync(FULL, item, owner);
      const uint32_t o_tb = __shfl_sync(FULL, tb, owner);
      const uint32_t o_tx = __shfl_sync(FULL, tx, owner);
      const uint32_t o_key = __shfl_sync(FULL, key, owner);
      bool take = false;
      uint32_t tile = 0;
      if (j < total_full) {
        const uint32_t local = j - o_excl;
        const uint32_t ly = local / o_wd, lx = local - ly * o_wd;
        tile = o_tb + (o_y0 + ly) * o_tx + (o_x0 + lx);
        take = a.cut != nullptr ? o_key <= __ldg(a.cut + tile) : __ldg(a.flag + tile) != 0;
      }
      const uint32_t bal = __ballot_sync(FULL, take);
      if (take) {
        const uint32_t slot = run + __popc(bal & lanemask_lt());
        if (slot < total_cnt) a.pairs[b + off0 + slot] = make_uint2(tile, o_item);
        else atomicOr(a.error_word, ERR_ENTRY_CAPACITY);  // counts disagree with the filter: never written past them
      }
      run += __popc(bal);
    }
  }
}

__global__ void k_cut_gate(const uint32_t* inc_count, uint32_t n_items, uint32_t* gate_n) {
  *gate_n = *inc_count ? n_items : 0u;
}

// Listed tiles are held in shared memory as (view, x, y) when there are few
// of them; each item then checks its rect against the list instead of
// reading the flags of every tile in the rect.
constexpr int FLAG_LIST_SMEM = 512;
__global__ void __launch_bounds__(256) k_count_flagged(const uint4* rects, const ViewInfo* views, uint32_t nv,
                                                       uint32_t ipv, uint32_t n, const uint32_t* inc_count,
                                                       const uint32_t* inc_list, const uint8_t* flag,
                                                       uint32_t* counts) {
  const uint32_t m = *inc_count;
  if (m == 0) return;
  __shared__ uint32_t s_v[FLAG_LIST_SMEM], s_x[FLAG_LIST_SMEM], s_y[FLAG_LIST_SMEM];
  const bool listed = m <= (uint32_t)FLAG_LIST_SMEM;
  if (listed) {
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
      const uint32_t t = inc_list[i];
      uint32_t v = 0;
      while (v + 1 < nv && t >= (uint32_t)__ldg(&views[v + 1].tile_base)) ++v;
      const uint32_t lt = t - (uint32_t)__ldg(&views[v].tile_base), tx = (uint32_t)__ldg(&views[v].tiles_x);
      s_v[i] = v; s_y[i] = lt / tx; s_x[i] = lt - (lt / tx) * tx;
    }
    __syncthreads();
  }
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint4 r = rects[i];
    uint32_t c = 0;
    if (r.z >= r.x && r.w >= r.y) {
      const uint32_t v = i / ipv;
      if (listed) {
        for (uint32_t k = 0; k < m; ++k)
          c += (s_v[k] == v && s_x[k] >= r.x && s_x[k] <= r.z && s_y[k] >= r.y && s_y[k] <= r.w) ? 1u : 0u;
      } else {
        const ViewInfo* V = views + v;
        const uint32_t tb = (uint32_t)__ldg(&V->tile_base), tx = (uint32_t)__ldg(&V->tiles_x);
        for (uint32_t y = r.y; y <= r.w; ++y)
          for (uint32_t x = r.x; x <= r.z; ++x) c += __ldg(flag + tb + y * tx + x) != 0 ? 1u : 0u;
      }
    }
    counts[i] = c;
  }
}

__global__ void __launch_bounds__(256) k_ranges_reset_list(const uint32_t* list, const uint32_t* count, uint2* ranges,
                                                           uint32_t max_list) {
  const uint32_t m = min(*count, max_list);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x)
    ranges[list[i]] = make_uint2(0u, 0u);
}

// One block per listed tile: the range recorded by the completion sort
// becomes [start, end), and the row-group summary of the first skip[i]
// entries (those pass 1 composited) moves from src[i] to the new start.
__global__ void __launch_bounds__(256) k_ranges_fix_list(const uint32_t* list, const uint32_t* count, uint2* ranges,
                                                         uint32_t max_list, unsigned long long* entry_total,
                                                         const unsigned long long* total2, uint8_t* gmask,
                                                         const uint32_t* skip, const uint32_t* src) {
  const uint32_t m = min(*count, max_list);
  for (uint32_t i = blockIdx.x; i < m; i += gridDim.x) {
    const uint32_t t = list[i];
    const uint2 r = ranges[t];
    __syncthreads();  // every thread holds the recorded range before it is replaced
    const uint2 f = r.y ? make_uint2(~r.x, r.y) : make_uint2(0u, 0u);
    if (threadIdx.x == 0) ranges[t] = f;
    if (gmask != nullptr) {
      const uint32_t sk = skip[i], from = src[i];
      if (f.y - f.x >= sk)
        for (uint32_t j = threadIdx.x; j < sk; j += blockDim.x) gmask[f.x + j] = gmask[from + j];
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *entry_total += *total2;
}

// Standalone binner: tiles per rect (tile_binning.wgsl:30-43), depth keys and
// the identity permutation for the item sort.
__global__ void __launch_bounds__(256) k_rect_counts(const uint4* rects, const uint32_t* depths, uint32_t n,
                                                     uint32_t* counts, uint32_t* keys, uint32_t* vals) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint4 r = rects[i];
    counts[i] = (r.z >= r.x && r.w >= r.y) ? (r.z - r.x + 1u) * (r.w - r.y + 1u) : 0u;
    keys[i] = depths[i];
    vals[i] = i;
  }
}

int grid_for(uint64_t n_max, int per_block, int cap_blocks) {
  uint64_t g = (n_max + per_block - 1) / per_block;
  if (g < 1) g = 1;
  if (g > (uint64_t)cap_blocks) g = cap_blocks;
  return (int)g;
}

}  // namespace

size_t scan_scratch_bytes() { return sizeof(unsigned long long) * SCAN_GRID; }

int launch_scan(const uint32_t* in, uint32_t* out, uint64_t n_host, const uint32_t* n_dev, uint32_t* total_u32,
                void* scratch, cudaStream_t st) {
  auto* bsum = reinterpret_cast<unsigned long long*>(scratch);
  k_scan_reduce<<<SCAN_GRID, SCAN_THREADS, 0, st>>>(in, n_host, n_dev, bsum);
  k_scan_blocks<<<1, SCAN_GRID, 0, st>>>(bsum, total_u32);
  k_scan_down<<<SCAN_GRID, SCAN_THREADS, 0, st>>>(in, out, n_host, n_dev, bsum);
  return (int)cudaGetLastError();
}

int launch_sort_reset(const SortScratch& sc, cudaStream_t st) {
  return (int)cudaMemsetAsync(sc.hdr[0], 0, sc.reset_bytes, st);
}

int launch_entry_scan(const EntryScanArgs& a, const SortScratch& sc, int which, cudaStream_t st) {
  const int grid = grid_for(a.n_host, ES_TILE, 148 * 4);
  k_entry_scan<<<grid, ES_THREADS, 0, st>>>(a, sc.scan_hdr[which], sc.scan_state[which], sc.wait_cycles);
  return (int)cudaGetLastError();
}

namespace {

template <class IO, typename W, class SWAP>
int radix_passes(IO io, uint64_t n_host, const uint32_t* n_dev, int key_bits, const SortScratch& sc, int hdr,
                 int* result_in_1, cudaStream_t st, SWAP swap, uint2* ranges = nullptr,
                 uint32_t num_ranges = 0, const unsigned long long* base = nullptr, bool zero_ranges = false) {
  const int passes = (key_bits + 7) / 8, dbits = (key_bits + passes - 1) / passes;
  uint32_t* h = sc.hdr[hdr];
  W* state[2] = {reinterpret_cast<W*>(sc.state), reinterpret_cast<W*>(sc.state) + sc.state_words};
  k_rs_hist<IO, W><<<grid_for(n_host, 8 * RH_THREADS, 148 * 4), RH_THREADS, 0, st>>>(
      io, n_host, n_dev, passes, dbits, key_bits, h, state[0], ranges, zero_ranges ? num_ranges : 0u, base);
  const int grid = grid_for(n_host, RS_TILE, 148 * RS_CTAS);
  for (int p = 0; p < passes; ++p) {
    const int shift = p * dbits, nbits = std::min(dbits, key_bits - shift);
    const bool last = p + 1 == passes;
    k_rs_pass<IO, W><<<grid, RS_THREADS, 0, st>>>(last ? io : io.plain(), n_host, n_dev, p, shift, nbits, h,
                                                  state[p & 1], last ? nullptr : state[(p + 1) & 1],
                                                  last ? ranges : nullptr, num_ranges, base, sc.wait_cycles);
    swap(io);
  }
  *result_in_1 = passes & 1;
  return (int)cudaGetLastError();
}

template <int NT>
int launch_small(const SplitIO& io, int n, int passes, int dbits, int key_bits, cudaStream_t st) {
  if constexpr (small_smem<NT>() > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(k_rs_small<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)small_smem<NT>());
    if (e != cudaSuccess) return (int)e;
  }
  k_rs_small<NT><<<1, NT, small_smem<NT>(), st>>>(io, n, passes, dbits, key_bits);
  return (int)cudaGetLastError();
}

}  // namespace

int launch_radix_sort(uint32_t* k0, uint32_t* v0, uint32_t* k1, uint32_t* v1, uint64_t n_host, const uint32_t* n_dev,
                      int key_bits, const SortScratch& sc, int hdr, int* result_in_1, cudaStream_t st,
                      const uint32_t* gather_src, uint32_t* gather_dst) {
  SplitIO io{k0, v0, k1, v1, gather_src, gather_dst};
  if (n_host <= (uint64_t)RS_SMALL && n_dev == nullptr) {  // one launch, 26 us at 3000 pairs; 6 launches take 37 us at 16 thousand
    if (n_host == 0) { *result_in_1 = ((key_bits + 7) / 8) & 1; return 0; }
    const int passes = (key_bits + 7) / 8, dbits = (key_bits + passes - 1) / passes;
    if (!(passes & 1)) { io.kout = k0; io.vout = v0; }  // where the passes in memory would have left the result
    *result_in_1 = passes & 1;
    const int n = (int)n_host;
    if (n <= 256 * SM_ROUNDS) return launch_small<256>(io, n, passes, dbits, key_bits, st);
    return launch_small<1024>(io, n, passes, dbits, key_bits, st);
  }
  auto swap = [](SplitIO& x) {
    SplitIO y{x.kout, x.vout, const_cast<uint32_t*>(x.kin), const_cast<uint32_t*>(x.vin), x.gsrc, x.gdst};
    x = y;
  };
  if (sc.wide)
    return radix_passes<SplitIO, unsigned long long>(io, n_host, n_dev, key_bits, sc, hdr, result_in_1, st, swap);
  return radix_passes<SplitIO, uint32_t>(io, n_host, n_dev, key_bits, sc, hdr, result_in_1, st, swap);
}

int launch_radix_sort_pairs(uint2* p0, uint2* p1, uint64_t n_host, const uint32_t* n_dev, int key_bits,
                            const SortScratch& sc, int hdr, int* result_in_1, cudaStream_t st, uint2* ranges,
                            uint32_t num_ranges, bool zero_ranges, const unsigned long long* base, uint32_t* values) {
  auto sort = [&](auto io) {
    using IO = decltype(io);
    auto swap = [](IO& x) {
      IO y{x.out, const_cast<uint2*>(x.in), x.values};
      x = y;
    };
    if (sc.wide)
      return radix_passes<IO, unsigned long long>(io, n_host, n_dev, key_bits, sc, hdr, result_in_1, st, swap, ranges,
                                                  num_ranges, base, zero_ranges);
    return radix_passes<IO, uint32_t>(io, n_host, n_dev, key_bits, sc, hdr, result_in_1, st, swap, ranges, num_ranges,
                                      base, zero_ranges);
  };
  // Chunks where they can be met and gain; the kernels without them keep
  // look-back's registers (65 against 63 us at 2.8 million).
  if (key_bits > 8 && n_host >= RC_MIN) return sort(PairIO<true>{p0, p1, values});
  return sort(PairIO<false>{p0, p1, values});
}

int launch_expand(const ExpandArgs& a, cudaStream_t st) {
  const int grid = grid_for((uint64_t)a.n_items_host, 256, 148 * 16);
  k_expand<<<grid, 256, 0, st>>>(a);
  return (int)cudaGetLastError();
}

int launch_expand_filtered(const ExpandFilterArgs& a, cudaStream_t st) {
  const int grid = grid_for((uint64_t)a.n_items_host, 256, 148 * 16);
  k_expand_filtered<<<grid, 256, 0, st>>>(a);
  return (int)cudaGetLastError();
}

int launch_cut_gate(const uint32_t* inc_count, uint32_t n_items, uint32_t* gate_n, cudaStream_t st) {
  k_cut_gate<<<1, 1, 0, st>>>(inc_count, n_items, gate_n);
  return (int)cudaGetLastError();
}

int launch_count_flagged(const uint4* rects, const ViewInfo* views, uint32_t n_views, uint32_t items_per_view,
                         uint32_t n_items, const uint32_t* inc_count, const uint32_t* inc_list, const uint8_t* flag,
                         uint32_t* counts, cudaStream_t st) {
  if (n_items == 0) return 0;
  k_count_flagged<<<grid_for(n_items, 256, 148 * 4), 256, 0, st>>>(rects, views, n_views, items_per_view, n_items,
                                                                    inc_count, inc_list, flag, counts);
  return (int)cudaGetLastError();
}

int launch_ranges_reset_list(const uint32_t* list, const uint32_t* count, uint2* ranges, uint32_t max_list,
                             cudaStream_t st) {
  if (max_list == 0) return 0;
  k_ranges_reset_list<<<grid_for(max_list, 256, 148), 256, 0, st>>>(list, count, ranges, max_list);
  return (int)cudaGetLastError();
}

int launch_ranges_fix_list(const uint32_t* list, const uint32_t* count, uint2* ranges, uint32_t max_list,
                           unsigned long long* entry_total, const unsigned long long* total2, uint8_t* gmask,
                           const uint32_t* skip, const uint32_t* src, cudaStream_t st) {
  k_ranges_fix_list<<<148, 256, 0, st>>>(list, count, ranges, max_list, entry_total, total2, gmask, skip, src);
  return (int)cudaGetLastError();
}

namespace {
// (~first, end) from the final sort pass → [first, end); (0, 0) for a key no
// element carried.
__global__ void __launch_bounds__(256) k_ranges_fix(uint2* ranges, uint32_t num_tiles) {
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < num_tiles; t += gridDim.x * blockDim.x) {
    const uint2 r = ranges[t];
    ranges[t] = r.y ? make_uint2(~r.x, r.y) : make_uint2(0u, 0u);
  }
}

__global__ void __launch_bounds__(256) k_tile_words(const uint2* ranges, uint32_t num_tiles, uint32_t* words) {
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < num_tiles; t += gridDim.x * blockDim.x) {
    const uint2 r = ranges[t];
    words[t] = r.y > r.x ? (r.y - r.x + 31u) / 32u : 0u;
  }
}
}  // namespace

int launch_ranges_fix(uint2* ranges, uint32_t num_tiles, cudaStream_t st) {
  if (num_tiles == 0) return 0;
  k_ranges_fix<<<grid_for(num_tiles, 256, 148 * 8), 256, 0, st>>>(ranges, num_tiles);
  return (int)cudaGetLastError();
}

namespace {
// Bucket of a work amount w: 4·⌊log2(w + 1)⌋ plus the two bits below the
// leading one, so four buckets per octave (0..127).
__device__ __forceinline__ uint32_t work_bucket(uint32_t w) {
  const uint32_t x = w + 1u > w ? w + 1u : w;
  const int e = 31 - __clz(x);
  const uint32_t frac = e >= 2 ? (x >> (e - 2)) & 3u : (x << (2 - e)) & 3u;
  return 4u * (uint32_t)e + frac;
}

// One block; a thread's loads of a round are in flight together (35 thousand
// tiles 28 -> 21 us, 3600 tiles 5.2 -> 4.5: one load at a time, and a
// serial sum over the buckets, took most of it).
__global__ void __launch_bounds__(1024) k_tile_order(const uint2* ranges, const uint32_t* lengths, uint32_t num_tiles,
                                                     uint32_t* order) {
  constexpr int NB = 128, NT = 1024, PER = 8;
  __shared__ uint32_t s_cnt[NB], s_warp[NB / 32];
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  if (tid < NB) s_cnt[tid] = 0u;
  __syncthreads();
  auto each = [&](auto use) {
    for (uint32_t t0 = 0; t0 < num_tiles; t0 += NT * PER) {
      uint32_t w[PER];
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const uint32_t t = t0 + k * NT + tid;
        w[k] = 0u;
        if (t < num_tiles) {
          if (lengths) {
            w[k] = lengths[t];
          } else {
            const uint2 r = ranges[t];
            w[k] = r.y - r.x;
          }
        }
      }
#pragma unroll
      for (int k = 0; k < PER; ++k)
        if (t0 + k * NT + tid < num_tiles) use(t0 + k * NT + tid, work_bucket(w[k]));
    }
  };
  each([&](uint32_t, uint32_t b) { atomicAdd(&s_cnt[b], 1u); });
  __syncthreads();
  // exclusive offsets, heaviest bucket first: thread i holds bucket NB-1-i
  uint32_t c = 0, incl = 0;
  if (tid < NB) {
    c = incl = s_cnt[NB - 1 - tid];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(FULL, incl, o);
      if (lane >= (uint32_t)o) incl += v;
    }
    if (lane == 31) s_warp[tid >> 5] = incl;
  }
  __syncthreads();
  if (tid < NB) {
    uint32_t before = 0;
    for (uint32_t k = 0; k < (tid >> 5); ++k) before += s_warp[k];
    s_cnt[NB - 1 - tid] = before + incl - c;
  }
  __syncthreads();
  each([&](uint32_t t, uint32_t b) { order[atomicAdd(&s_cnt[b], 1u)] = t; });
}
}  // namespace

int launch_tile_order(const uint2* ranges, const uint32_t* lengths, uint32_t num_tiles, uint32_t* order,
                      cudaStream_t st) {
  if (num_tiles == 0) return 0;
  k_tile_order<<<1, 1024, 0, st>>>(ranges, lengths, num_tiles, order);
  return (int)cudaGetLastError();
}

int launch_mask_offsets(const uint2* ranges, uint32_t num_tiles, uint32_t* words, uint32_t* mask_off, void* scratch,
                        cudaStream_t st) {
  if (num_tiles == 0) return 0;
  k_tile_words<<<grid_for(num_tiles, 256, 148 * 8), 256, 0, st>>>(ranges, num_tiles, words);
  return launch_scan(words, mask_off, num_tiles, nullptr, nullptr, scratch, st);
}

int launch_rect_counts(const uint4* rects, const uint32_t* depths, uint32_t n, uint32_t* counts, uint32_t* keys,
                       uint32_t* vals, cudaStream_t st) {
  if (n == 0) return 0;
  k_rect_counts<<<grid_for(n, 256, 148 * 16), 256, 0, st>>>(rects, depths, n, counts, keys, vals);
  return (int)cudaGetLastError();
}

int tile_key_bits(uint32_t num_tiles) {
  int b = 1;
  while (b < 32 && (1ull << b) < (unsigned long long)num_tiles) ++b;
  return b;
}

}  // namespace gs
