// scan.cuh -- exclusive prefix sums of int32 on the device, in one launch up to
// a million elements and in two or three beyond, shared by the cell sorts of the
// particle step and of the surrogate's graph.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

namespace scan {

constexpr int kScanThreads = 256, kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;   // elements per scan block
constexpr int kTimeoutCode = 7;                        // status of a wait that ran out (SDEM_E_TIMEOUT)

// ---------------------------------------------------------------------------
// Ordered prefix sums in one launch (decoupled look-back: Merrill and Garland,
// "Single-pass Parallel Prefix Scan with Decoupled Look-back", 2016).  Blocks
// take tiles in order from a ticket, so every earlier tile is running or done;
// each publishes its tile's sum, then adds up its predecessors' words until it
// meets a complete prefix.  A tile's word holds epoch (30 bits), state (1: the
// tile's sum, 2: the prefix through the tile) and value (32 bits) together, so
// a reader needs no fence; the epoch, one per launch, makes the words of
// earlier launches stale without clearing them.
struct ScanCtl {
  int ticket, done;
  unsigned epoch;
  int total;   // ghost passes: images made by the pass
};
constexpr int kSpinLimit = 1 << 20;   // polls of one word before a wait gives up

__device__ __forceinline__ unsigned long long scan_word(unsigned epoch, unsigned state, int v) {
  return (unsigned long long)((epoch << 2) | state) << 32 | (unsigned)v;
}

// Exclusive prefix of `tile` whose sum is `sum` (thread 0's); the whole block
// calls, so that one round looks back over 256 tiles: with one warp's 32 a
// scan of 2,200 tiles took 81 us, the chain of waits alone.  A wait that runs
// out is reported and counts as zero: the prefixes then come out too small,
// never too large, so what is indexed with them stays in range.
__device__ __forceinline__ int scan_lookback(volatile unsigned long long* words, unsigned epoch, int tile, int sum, int* status) {
  __shared__ int part[kScanThreads / 32], first_full[kScanThreads / 32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const unsigned key = epoch & 0x3FFFFFFFu;
  if (t == 0) words[tile] = scan_word(key, tile == 0 ? 2u : 1u, sum);
  int excl = 0;
  for (int j = tile - 1; j >= 0; j -= kScanThreads) {
    const int i = j - t;
    unsigned state = 2u;
    int v = 0;
    if (i >= 0) {
      int polls = 0;
      unsigned long long x;
      do {
        x = words[i];
      } while (((unsigned)(x >> 34) != key || ((unsigned)(x >> 32) & 3u) == 0u) && ++polls < kSpinLimit);
      if (polls < kSpinLimit) {
        state = (unsigned)(x >> 32) & 3u;
        v = (int)(unsigned)x;
      } else if (atomicCAS(status, 0, kTimeoutCode) == 0) {
        status[1] = i;
      }
    }
    // the nearest complete prefix ends the walk
    const unsigned full = __ballot_sync(0xffffffffu, state == 2u);
    const int stop = full ? __ffs(full) - 1 : 31;
    int add = lane <= stop ? v : 0;
    for (int o = 16; o > 0; o >>= 1) add += __shfl_xor_sync(0xffffffffu, add, o);
    if (lane == 0) {
      part[w] = add;
      first_full[w] = full != 0u;
    }
    __syncthreads();
    bool done = false;
    for (int k = 0; k < kScanThreads / 32 && !done; k++) {
      excl += part[k];
      done = first_full[k] != 0;
    }
    __syncthreads();
    if (done) break;
  }
  if (t == 0 && tile > 0) words[tile] = scan_word(key, 2u, excl + sum);
  return excl;
}

// The sum of sums[0, tile); the whole block calls.
__device__ __forceinline__ int sum_before(const int* __restrict__ sums, int tile) {
  __shared__ int part[kScanThreads / 32];
  int v = 0;
  for (int i = threadIdx.x; i < tile; i += kScanThreads) v += sums[i];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  v = 0;
  for (int k = 0; k < kScanThreads / 32; k++) v += part[k];
  return v;
}

// out[i] = sum of in[0..i), out[n] = the total; in[] is left zero for the next
// step's counting.  A tile is 256 threads x 16 elements through shared memory
// (padded: element e at e + e/16, so that the striped int4 copies and the
// per-thread runs of 16 are both free of bank conflicts).
// One launch where the three of a reduce-then-scan took 14.5 us of dependent
// latency: 6 us at 7,000 cells, 9 us at 60,000.
// What a tile adds to its own sums: kOnePass, the look-back's prefix; kTileSums,
// the sums of the tiles before it, added up by each block; kTileOffsets, its entry
// of a scan of those sums.  kScanOfSums is that scan: kOnePass, in[] left as it is.
enum ScanForm { kOnePass, kTileSums, kTileOffsets, kScanOfSums };
inline __host__ __device__ int offsets_at(int tiles) { return (tiles + 3) / 4 * 4; }   // behind the sums
template <ScanForm kForm>
static __global__ void __launch_bounds__(kScanThreads) k_scan(int* __restrict__ in, long long n, int* __restrict__ out,
                                                       ScanCtl* ctl, unsigned long long* words, int* status) {
  __shared__ int sh[kScanTile + kScanTile / kScanItems];
  __shared__ int wsum[kScanThreads / 32];
  __shared__ int s_tile, s_total;
  __shared__ unsigned s_epoch;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  constexpr bool kLookBack = kForm == kOnePass || kForm == kScanOfSums;
  if (kLookBack) {
    if (t == 0) {
      s_epoch = ctl->epoch + 1u;
      s_tile = atomicAdd(&ctl->ticket, 1);
    }
    __syncthreads();
    if (s_tile >= (int)gridDim.x) return;   // (only a caller that shares ctl between overlapping launches gets here)
  }
  const int tile = kLookBack ? s_tile : (int)blockIdx.x;
  const long long base = (long long)tile * kScanTile;
  const bool whole = base + kScanTile <= n;
  auto pad = [](int e) { return e + e / kScanItems; };
  const int* sums = reinterpret_cast<const int*>(words);   // kTileSums, kTileOffsets (see scan_cells)
  if (!kLookBack) {
    // the tiles' sums are known: a tile without counts is neither read nor cleared
    if (sums[tile] == 0) {
      const int excl = kForm == kTileSums ? sum_before(sums, tile) : sums[offsets_at(gridDim.x) + tile];
      if (whole) {
        int4* v = reinterpret_cast<int4*>(out + base);
#pragma unroll
        for (int j = 0; j < kScanItems / 4; j++) v[j * kScanThreads + t] = make_int4(excl, excl, excl, excl);
      } else {
        for (int e = t; e < kScanTile; e += kScanThreads)
          if (base + e < n) out[base + e] = excl;
      }
      if (t == 0 && tile == (int)gridDim.x - 1) out[n] = excl;
      return;
    }
  }
  if (whole) {
    int4* v = reinterpret_cast<int4*>(in + base);
#pragma unroll
    for (int j = 0; j < kScanItems / 4; j++) {
      const int4 q = v[j * kScanThreads + t];
      if (kForm != kScanOfSums && (q.x | q.y | q.z | q.w)) v[j * kScanThreads + t] = make_int4(0, 0, 0, 0);
      const int e = pad((j * kScanThreads + t) * 4);
      sh[e] = q.x;
      sh[e + 1] = q.y;
      sh[e + 2] = q.z;
      sh[e + 3] = q.w;
    }
  } else {
    for (int e = t; e < kScanTile; e += kScanThreads) {
      sh[pad(e)] = base + e < n ? in[base + e] : 0;
      if (kForm != kScanOfSums && base + e < n) in[base + e] = 0;
    }
  }
  __syncthreads();
  int loc[kScanItems];
  int sum = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; i++) {
    const int v = sh[t * (kScanItems + 1) + i];
    loc[i] = sum;
    sum += v;
  }
  int x = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[w] = x;
  __syncthreads();
  if (w == 0) {
    const int v = lane < kScanThreads / 32 ? wsum[lane] : 0;
    int z = v;
    for (int o = 1; o < kScanThreads / 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, z, o);
      if (lane >= o) z += y;
    }
    if (lane < kScanThreads / 32) wsum[lane] = z - v;
    if (lane == kScanThreads / 32 - 1) s_total = z;
  }
  __syncthreads();
  int excl = 0;
  if (kLookBack) excl = scan_lookback(words, s_epoch, tile, s_total, status);
  else if (kForm == kTileSums) excl = sum_before(sums, tile);
  else excl = sums[offsets_at(gridDim.x) + tile];
  const int first = excl + wsum[w] + x - sum;
#pragma unroll
  for (int i = 0; i < kScanItems; i++) sh[t * (kScanItems + 1) + i] = first + loc[i];
  __syncthreads();
  if (whole) {
    int4* v = reinterpret_cast<int4*>(out + base);
#pragma unroll
    for (int j = 0; j < kScanItems / 4; j++) {
      const int e = pad((j * kScanThreads + t) * 4);
      v[j * kScanThreads + t] = make_int4(sh[e], sh[e + 1], sh[e + 2], sh[e + 3]);
    }
  } else {
    for (int e = t; e < kScanTile; e += kScanThreads)
      if (base + e < n) out[base + e] = sh[pad(e)];
  }
  if (t == 0) {
    if (tile == (int)gridDim.x - 1) out[n] = excl + s_total;
    if (kLookBack && atomicAdd(&ctl->done, 1) == (int)gridDim.x - 1) {   // every block has its ticket and epoch
      ctl->ticket = 0;
      ctl->done = 0;
      ctl->epoch = s_epoch;
    }
  }
}

// The tiles' sums, for the forms with more than one launch.
static __global__ void __launch_bounds__(kScanThreads) k_scan_sums(const int* __restrict__ in, long long n, int* __restrict__ sums) {
  __shared__ int part[kScanThreads / 32];
  const long long base = (long long)blockIdx.x * kScanTile;
  int v = 0;
  if (base + kScanTile <= n) {
    const int4* q = reinterpret_cast<const int4*>(in + base);
#pragma unroll
    for (int j = 0; j < kScanItems / 4; j++) {
      const int4 a = q[j * kScanThreads + threadIdx.x];
      v += (a.x + a.y) + (a.z + a.w);
    }
  } else {
    for (int e = threadIdx.x; e < kScanTile; e += kScanThreads)
      if (base + e < n) v += in[base + e];
  }
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    v = 0;
    for (int k = 0; k < kScanThreads / 32; k++) v += part[k];
    sums[blockIdx.x] = v;
  }
}

// Scans n counts into out[0..n] and leaves them zero; launches issued.
// Up to 256 tiles (1M cells) in one launch; beyond, the look-back's chain of
// waits costs more than a second launch: 317 tiles 14.7 against 11.8 us, 2,470
// tiles 77 against 43 us; 128 tiles 10.5 against 11.3 us, 7 tiles 6 against 9.6.
// A large grid is mostly empty (a 400k hopper: 10M cells, 400k of them taken at
// most): tiles without counts are not read a second time, and only words that
// hold a count are cleared.  With that the hopper's step takes 184 us instead of
// 203.  Sums or flags per tile set by the binning instead of k_scan_sums were
// slower (215 and 190 us: all spheres of a tile meet at one address).
// Beyond 12,288 tiles (50M cells) the sums are scanned once, by a third launch:
// each block adding up all sums before its own is quadratic in the tiles.  400k
// counts spread over the grid, two launches against three: 4,096 tiles 53 / 57
// us, 8,192 92 / 92, 16,384 175 / 160, 98,304 1,486 / 757.
constexpr int kOnePassTiles = 256;
constexpr int kSumsTiles = 12288;
inline int scan_tiles(long long n) { return (int)std::max<long long>(1, (n + kScanTile - 1) / kScanTile); }
// 8-byte words of scratch, zero before the first scan: one a tile; with three
// launches the sums, their scan (each from a 16-byte boundary) and its own words.
// A grid has fewer than 2^31 cells, so the scan of the sums takes one launch.
inline size_t scan_words(long long n) {
  const size_t tiles = (size_t)scan_tiles(n);
  return tiles <= (size_t)kSumsTiles ? tiles : (size_t)offsets_at((int)tiles) + 2 + (size_t)scan_tiles((long long)tiles);
}

inline int scan_cells(int* cnt, long long n, int* out, ScanCtl* ctl, unsigned long long* words, int* status, cudaStream_t st) {
  const int tiles = scan_tiles(n);
  if (tiles <= kOnePassTiles) {
    k_scan<kOnePass><<<tiles, kScanThreads, 0, st>>>(cnt, n, out, ctl, words, status);
    return 1;
  }
  int* sums = reinterpret_cast<int*>(words);
  k_scan_sums<<<tiles, kScanThreads, 0, st>>>(cnt, n, sums);
  if (tiles <= kSumsTiles) {
    k_scan<kTileSums><<<tiles, kScanThreads, 0, st>>>(cnt, n, out, ctl, words, status);
    return 2;
  }
  const int at = offsets_at(tiles);   // tiles + 1 offsets, then the look-back's words
  k_scan<kScanOfSums><<<scan_tiles(tiles), kScanThreads, 0, st>>>(sums, tiles, sums + at, ctl, words + at + 2, status);
  k_scan<kTileOffsets><<<tiles, kScanThreads, 0, st>>>(cnt, n, out, ctl, words, status);
  return 3;
}

}  // namespace scan
