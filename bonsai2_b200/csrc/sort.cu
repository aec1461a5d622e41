// sort.cu -- stable LSD radix sort of (u64 key, int value) pairs and a
// multi-block exclusive scan.
//
// The reference sorts with Thrust (sort_by_key / stable_sort_by_key,
// makeGroups.cu:270-277, buildTree.cu:940-944): a stable radix sort, ties in
// input order.  This is a hand-written replacement with the same semantics:
// 8 passes of 8 bits, one-sweep (below): keys are ranked stably inside each
// tile (the lanes of equal digit from bit ballots) with per-warp
// digit counters in shared memory, tile offsets come from a decoupled look-back, and tiles are written
// out through shared memory in contiguous digit runs.  A thread keeps only the
// ranks and packed digits of its keys across the look-back (the keys are
// re-read from L2 for staging): 4 blocks per SM (keeping the keys, 127
// registers and 2 blocks per SM, was 16 % slower per sort than 3 blocks).
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"

namespace bonsai {

constexpr int kSortThreads = 256;
constexpr int kScanChunk = 4096;
// Keys per thread of a one-sweep tile: 4 (1024-key tiles) where a pass is one
// tile's latency, 16 where the digit runs that a tile writes out have to be long,
// 8 between.  Build of a whole step with 4 / 8 / 16 (us): 30,011 particles 126 /
// 139, 131,072 169 / 171 / 200, 250,007 220 / 212 / 229, 500,000 300 / 297 / 308,
// 2^20 - / 411 / 438, 1.15M - / 452 / 475, 1.5M - / 536 / 544, 1.7M - / 602 / 580:
// the upper line is short of where the sides meet.  Same order with any.
constexpr int kSmallItems = 4, kMidItems = 8, kLargeItems = 16;
constexpr int kSortSmallMax = 1 << 17, kSortMidMax = 1 << 20;
static int sort_items(int n) { return n <= kSortSmallMax ? kSmallItems : (n <= kSortMidMax ? kMidItems : kLargeItems); }

int sort_tiles(int n) {
  const int tile = kSortThreads * sort_items(n);
  return (n + tile - 1) / tile;
}

// ---------------------------------------------------------------------------
// exclusive scan of unsigned ints (length m known on the host)
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned block_excl_scan(unsigned v, unsigned* sh, unsigned* total) {
  // 256 threads
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned t = __shfl_up_sync(kFull, x, o);
    if (lane >= o) x += t;
  }
  if (lane == 31) sh[w] = x;
  __syncthreads();
  if (w == 0) {
    unsigned y = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned t = __shfl_up_sync(kFull, y, o);
      if (lane >= o) y += t;
    }
    sh[lane] = y;  // inclusive per-warp totals
  }
  __syncthreads();
  const unsigned wprefix = w ? sh[w - 1] : 0u;
  if (total) *total = sh[(blockDim.x >> 5) - 1];
  __syncthreads();
  return wprefix + x - v;
}

__global__ void __launch_bounds__(256) k_scan_reduce(const unsigned* __restrict__ in, int m,
                                                     unsigned* __restrict__ bsum) {
  __shared__ unsigned sh[32];
  const int b0 = blockIdx.x * kScanChunk;
  unsigned s = 0;
  for (int i = b0 + threadIdx.x; i < min(b0 + kScanChunk, m); i += 256) s += in[i];
  unsigned tot;
  block_excl_scan(s, sh, &tot);
  if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(256) k_scan_top(unsigned* __restrict__ bsum, int nb, unsigned* __restrict__ total) {
  __shared__ unsigned sh[32];
  unsigned carry = 0;
  for (int b0 = 0; b0 < nb; b0 += 256) {
    const int i = b0 + threadIdx.x;
    const unsigned v = i < nb ? bsum[i] : 0u;
    unsigned tot;
    const unsigned e = block_excl_scan(v, sh, &tot);
    if (i < nb) bsum[i] = carry + e;
    carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0 && total) *total = carry;
}

__global__ void __launch_bounds__(256) k_scan_down(const unsigned* __restrict__ in, int m,
                                                   const unsigned* __restrict__ bsum, unsigned* __restrict__ out) {
  __shared__ unsigned sh[32];
  const int b0 = blockIdx.x * kScanChunk;
  // each thread owns 16 consecutive elements of the chunk
  const int i0 = b0 + threadIdx.x * 16;
  unsigned v[16];
  unsigned s = 0;
#pragma unroll
  for (int k = 0; k < 16; k++) {
    v[k] = (i0 + k < m) ? in[i0 + k] : 0u;
    s += v[k];
  }
  unsigned run = block_excl_scan(s, sh, nullptr) + bsum[blockIdx.x];
#pragma unroll
  for (int k = 0; k < 16; k++) {
    if (i0 + k < m) out[i0 + k] = run;
    run += v[k];
  }
}

int scan_blocks(int m) { return (m + kScanChunk - 1) / kScanChunk; }

// out may alias in.  bsum needs scan_blocks(m) entries.
void exclusive_scan(const unsigned* in, unsigned* out, int m, unsigned* bsum, unsigned* total, cudaStream_t s) {
  const int nb = scan_blocks(m);
  if (nb == 0) return;
  k_scan_reduce<<<nb, 256, 0, s>>>(in, m, bsum);
  k_scan_top<<<1, 256, 0, s>>>(bsum, nb, total);
  k_scan_down<<<nb, 256, 0, s>>>(in, m, bsum, out);
}

// ---------------------------------------------------------------------------
// One-sweep passes.  One kernel reads the keys once and builds the digit
// histograms of all eight passes; one kernel per pass then ranks each
// tile (the same stable warp ranking for every tile size), obtains the tile's
// global offset per digit by decoupled look-back over the preceding tiles
// (tiles take ids in launch order from an atomic counter, so a tile only waits
// for tiles that already run; every wait is bounded and sets an error flag
// when the bound is hit), stages the tile in shared memory in digit order and
// writes it out in contiguous runs.  One read and one write of the pairs per
// pass.
// ---------------------------------------------------------------------------
// blocks per SM of the one-sweep pass: the pass is latency-bound, and 4 blocks
// (64 registers, a 40-byte spill) beat 3 (80 registers): build phase at
// N = 2^24 4.49 against 4.71 ms
#ifndef BONSAI_SORT_MINB
#define BONSAI_SORT_MINB 4
#endif
constexpr unsigned kFlagAgg = 1u << 30, kFlagInc = 2u << 30, kValMask = (1u << 30) - 1u;

// The lanes of `live` that hold the same digit (0..255): the intersection of
// eight bit ballots (__match_any_sync was slower on the B200: PH sort + group
// formation at N = 2^24 1.93 against 1.82 ms).
__device__ __forceinline__ unsigned digit_peers(unsigned d, unsigned live) {
  unsigned m = live;
#pragma unroll
  for (int b = 0; b < 8; b++) {
    const unsigned bal = __ballot_sync(kFull, (d >> b) & 1u);
    m &= ((d >> b) & 1u) ? bal : ~bal;
  }
  return m;
}
constexpr int kLookbackSpin = 1 << 22;

__global__ void __launch_bounds__(kSortThreads) k_sort_hist8(const unsigned long long* __restrict__ keys, int n,
                                                             int passes, unsigned* __restrict__ ghist) {
  __shared__ unsigned h[8][256];
  for (int t = threadIdx.x; t < 8 * 256; t += kSortThreads) (&h[0][0])[t] = 0;
  __syncthreads();
  for (int i = blockIdx.x * kSortThreads + threadIdx.x; i < n; i += gridDim.x * kSortThreads) {
    const unsigned long long k = keys[i];
#pragma unroll
    for (int p = 0; p < 8; p++)
      if (p < passes) atomicAdd(&h[p][(unsigned)(k >> (8 * p)) & 255u], 1u);
  }
  __syncthreads();
  for (int t = threadIdx.x; t < passes * 256; t += kSortThreads) {
    const unsigned v = (&h[0][0])[t];
    if (v) atomicAdd(ghist + t, v);
  }
}

// exclusive scan of each 256-entry row in place (one block of 256 threads per row)
__global__ void __launch_bounds__(256) k_sort_hist_scan(unsigned* __restrict__ ghist) {
  __shared__ unsigned sh[32];
  unsigned* row = ghist + blockIdx.x * 256;
  const unsigned e = block_excl_scan(row[threadIdx.x], sh, nullptr);
  row[threadIdx.x] = e;
}

// SYSD: the digit is a byte of the element's system index (sys_of of its
// value, the element's position in the sort's input order), not of its key:
// the passes that make an ensemble sort stable-partition by system last.
// The digits of all items are read before any is ranked: the ranking's warp
// barriers would otherwise hold each load back behind the item before it, one
// memory round trip per item (a pass over 30,011 keys 11.5 -> 6.1 us with the
// smaller tiles).  The look-back reads four tiles' words at once (8 or 16 were no
// faster below a million keys and slower above).
constexpr int kLookback = 4;
template <int ITEMS, bool SYSD>
__global__ void __launch_bounds__(kSortThreads, BONSAI_SORT_MINB) k_sort_onesweep(
    const unsigned long long* __restrict__ keys_in, const int* __restrict__ vals_in, int n, int shift,
    const unsigned* __restrict__ gbase, unsigned* __restrict__ status, unsigned* __restrict__ tile_counter,
    unsigned long long* __restrict__ keys_out, int* __restrict__ vals_out, int* __restrict__ err,
    const int* __restrict__ sys_off, int nsys) {
  constexpr int kTile = kSortThreads * ITEMS;
  __shared__ unsigned wcnt[kSortThreads / 32][256];
  __shared__ unsigned tile_off[256];
  __shared__ unsigned dstart[256];
  __shared__ unsigned long long stage[kTile];  // keys, then values (as 32-bit) in digit order
  __shared__ unsigned char sdig[kTile];
  __shared__ unsigned sh[32];
  __shared__ int tile_sh;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) tile_sh = (int)atomicAdd(tile_counter, 1u);
  for (int t = threadIdx.x; t < (kSortThreads / 32) * 256; t += kSortThreads) (&wcnt[0][0])[t] = 0;
  __syncthreads();
  const int tile = tile_sh;
  const int base = tile * kTile + w * (32 * ITEMS);
  unsigned rank[ITEMS];
  unsigned dpack[ITEMS / 4];
#pragma unroll
  for (int k = 0; k < ITEMS; k++) {
    const int i = base + k * 32 + lane;
    unsigned d = 0u;
    if (i < n) {
      if constexpr (SYSD) d = ((unsigned)sys_of(sys_off, nsys, vals_in ? vals_in[i] : i) >> shift) & 255u;
      else d = (unsigned)(keys_in[i] >> shift) & 255u;
    }
    if ((k & 3) == 0) dpack[k >> 2] = 0u;
    dpack[k >> 2] |= d << (8 * (k & 3));
  }
#pragma unroll
  for (int k = 0; k < ITEMS; k++) {
    const bool ok = base + k * 32 + lane < n;
    const unsigned live = __ballot_sync(kFull, ok);
    const unsigned d = (dpack[k >> 2] >> (8 * (k & 3))) & 255u;
    const unsigned peers = digit_peers(d, live);
    const unsigned before = (unsigned)__popc(peers & lanemask_lt());
    const unsigned cur = ok ? wcnt[w][d] : 0u;
    rank[k] = cur + before;
    __syncwarp();
    if (ok && before == 0) wcnt[w][d] = cur + (unsigned)__popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // per digit: prefix over warps, tile total, tile-local digit offsets
  const unsigned d = threadIdx.x;
  unsigned tot = 0;
#pragma unroll
  for (int ww = 0; ww < kSortThreads / 32; ww++) {
    const unsigned c = wcnt[ww][d];
    wcnt[ww][d] = tot;
    tot += c;
  }
  volatile unsigned* st = status;
  // published before the block's own scan: the tiles behind wait for it
  st[(size_t)tile * 256 + d] = (tile == 0 ? kFlagInc : kFlagAgg) | tot;
  tile_off[d] = block_excl_scan(tot, sh, nullptr);
  // decoupled look-back for the digit's global offset
  unsigned excl = 0;
  bool done = tile == 0;
  for (int t = tile - 1; !done; t -= kLookback) {
    unsigned v[kLookback];
#pragma unroll
    for (int q = 0; q < kLookback; q++) v[q] = t - q >= 0 ? (unsigned)st[(size_t)(t - q) * 256 + d] : (unsigned)kFlagInc;
#pragma unroll
    for (int q = 0; q < kLookback; q++) {
      if (done) break;
      int spin = 0;
      while ((v[q] & ~kValMask) == 0u && spin < kLookbackSpin) {
        __nanosleep(32);
        v[q] = st[(size_t)(t - q) * 256 + d];
        spin++;
      }
      if ((v[q] & ~kValMask) == 0u) {  // bound hit: report and give up (results invalid)
        atomicOr(err, kStatusSortTimeout);
        done = true;
        break;
      }
      excl += v[q] & kValMask;
      done = (v[q] & ~kValMask) == kFlagInc;
    }
  }
  if (tile != 0) st[(size_t)tile * 256 + d] = kFlagInc | (excl + tot);
  dstart[d] = gbase[d] + excl;
  __syncthreads();
  // stage keys in digit order (re-read from L2), write contiguous runs
  const int tile_n = min(kTile, n - tile * kTile);
  unsigned lpos[ITEMS];
#pragma unroll
  for (int k = 0; k < ITEMS; k++) {
    const int i = base + k * 32 + lane;
    if (i < n) {
      const unsigned dd = (dpack[k >> 2] >> (8 * (k & 3))) & 255u;
      lpos[k] = tile_off[dd] + wcnt[w][dd] + rank[k];
      stage[lpos[k]] = keys_in[i];
      sdig[lpos[k]] = (unsigned char)dd;
    }
  }
  __syncthreads();
  for (int j = threadIdx.x; j < tile_n; j += kSortThreads) {
    const unsigned long long kk = stage[j];
    const unsigned dd = sdig[j];
    const unsigned dst = dstart[dd] + (unsigned)j - tile_off[dd];
    if (BONSAI_IN_RANGE(dst, n, 0x601)) keys_out[dst] = kk;
  }
  __syncthreads();
  unsigned* stage32 = reinterpret_cast<unsigned*>(stage);
#pragma unroll
  for (int k = 0; k < ITEMS; k++) {
    const int i = base + k * 32 + lane;
    if (i < n) stage32[lpos[k]] = (unsigned)(vals_in ? vals_in[i] : i);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < tile_n; j += kSortThreads) {
    const unsigned dd = sdig[j];
    const unsigned dst = dstart[dd] + (unsigned)j - tile_off[dd];
    if (BONSAI_IN_RANGE(dst, n, 0x602)) vals_out[dst] = (int)stage32[j];
  }
}

// All eight passes of at most 4096 keys in one block, the pairs in shared
// memory throughout: a launch per pass is latency alone at this size (1024 keys:
// 11.3 us for the whole sort, 8 launches of 7.2 us and two more before it).  Every
// pass ranks as above: warp w's items are the 128 positions from 128 w.
constexpr int kOneThreads = 1024, kOneItems = 4, kOneMax = kOneThreads * kOneItems;
constexpr int kOneWarps = kOneThreads / 32;
constexpr int kOneSmem = kOneMax * (8 + 4) + kOneWarps * 256 * 2 + 256 * 4;
__global__ void __launch_bounds__(kOneThreads) k_sort_block(unsigned long long* __restrict__ keys,
                                                            const int* __restrict__ vals_in,
                                                            int* __restrict__ vals, int n, int passes) {
  extern __shared__ unsigned long long one_sm[];
  unsigned long long* sk = one_sm;
  int* sv = reinterpret_cast<int*>(sk + kOneMax);
  unsigned short* wc = reinterpret_cast<unsigned short*>(sv + kOneMax);  // [warp][digit]
  unsigned* off = reinterpret_cast<unsigned*>(wc + kOneWarps * 256);     // digit offsets
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int base = w * 32 * kOneItems;
  const int nw = (n + 32 * kOneItems - 1) / (32 * kOneItems);  // warps that hold keys
  unsigned long long key[kOneItems];
  int val[kOneItems];
#pragma unroll
  for (int k = 0; k < kOneItems; k++) {
    const int i = base + 32 * k + lane;
    key[k] = i < n ? keys[i] : 0ull;
    val[k] = i < n ? (vals_in ? vals_in[i] : i) : 0;
  }
  for (int p = 0; p < passes; p++) {
    for (int t = threadIdx.x; t < nw * 128; t += (int)blockDim.x) reinterpret_cast<unsigned*>(wc)[t] = 0u;
    __syncthreads();
    unsigned rank[kOneItems];
#pragma unroll
    for (int k = 0; k < kOneItems; k++) {
      const bool ok = base + 32 * k + lane < n;
      const unsigned live = __ballot_sync(kFull, ok);
      const unsigned d = (unsigned)(key[k] >> (8 * p)) & 255u;
      const unsigned peers = digit_peers(d, live);
      const unsigned before = (unsigned)__popc(peers & lanemask_lt());
      const unsigned cur = ok ? wc[w * 256 + d] : 0u;
      rank[k] = cur + before;
      __syncwarp();
      if (ok && before == 0) wc[w * 256 + d] = (unsigned short)(cur + __popc(peers));
      __syncwarp();
    }
    __syncthreads();
    // a thread per digit: its counters become the prefix over the warps that
    // hold keys
    if (threadIdx.x < 256) {
      const int d = threadIdx.x;
      unsigned run = 0;
#pragma unroll 8
      for (int q = 0; q < nw; q++) {
        const unsigned c = wc[q * 256 + d];
        wc[q * 256 + d] = (unsigned short)run;
        run += c;
      }
      off[d] = run;
    }
    __syncthreads();
    if (w == 0) {
      unsigned v[8], s = 0;
#pragma unroll
      for (int q = 0; q < 8; q++) { v[q] = off[lane * 8 + q]; s += v[q]; }
      unsigned run = (unsigned)warp_incl_scan((int)s) - s;
#pragma unroll
      for (int q = 0; q < 8; q++) { off[lane * 8 + q] = run; run += v[q]; }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kOneItems; k++) {
      if (base + 32 * k + lane < n) {
        const unsigned d = (unsigned)(key[k] >> (8 * p)) & 255u;
        const unsigned at = off[d] + wc[w * 256 + d] + rank[k];
        sk[at] = key[k];
        sv[at] = val[k];
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kOneItems; k++) {
      const int i = base + 32 * k + lane;
      if (i < n) {
        key[k] = sk[i];
        val[k] = sv[i];
      }
    }
    // (the next pass writes sk and sv only after three more barriers)
  }
#pragma unroll
  for (int k = 0; k < kOneItems; k++) {
    const int i = base + 32 * k + lane;
    if (i < n) {
      keys[i] = key[k];
      vals[i] = val[k];
    }
  }
}

// digit histograms of the two system-index passes, from the system sizes
__global__ void __launch_bounds__(256) k_sort_hist_sys(const int* __restrict__ sys_off, int nsys,
                                                       unsigned* __restrict__ ghist) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nsys; s += gridDim.x * blockDim.x) {
    const unsigned c = (unsigned)(sys_off[s + 1] - sys_off[s]);
    atomicAdd(ghist + (s & 255), c);
    atomicAdd(ghist + 256 + ((s >> 8) & 255), c);
  }
}

constexpr int kMaxPasses = 10;  // 8 key bytes + 2 system-index bytes

size_t sort_status_words(int n) { return (size_t)sort_tiles(n) * 256 * kMaxPasses + kMaxPasses + kMaxPasses * 256; }

// Stable sort of n (key, value) pairs; values_in == nullptr means 0..n-1.
// Result ends in (keys_a, vals_a) after an even number of passes.  work holds
// sort_status_words(n) unsigned ints: look-back status of every pass, the
// tile counters and the digit histograms; kStatusSortTimeout is or-ed into
// *err if a look-back wait hit its bound.  With nsys > 1 (an ensemble laid
// out as sys_off), two more passes order by system index, so each system's
// pairs are sorted by key within the system's own index range, ties in input
// order: the order each system gets when sorted alone.
template <int ITEMS>
static void radix_sort_passes(unsigned long long* keys_a, unsigned long long* keys_b, int* vals_a, int* vals_b,
                              const int* vals_in, int n, unsigned* work, int* err, int passes, const int* sys_off,
                              int nsys, cudaStream_t s) {
  const int nt = sort_tiles(n);
  const int sys_passes = nsys > 1 ? 2 : 0;
  // counters, histograms, then the look-back words of the passes that run
  unsigned* counters = work;
  unsigned* ghist = counters + kMaxPasses;
  unsigned* status = ghist + kMaxPasses * 256;
  cudaMemsetAsync(work, 0, (kMaxPasses * 257 + (size_t)(passes + sys_passes) * nt * 256) * sizeof(unsigned), s);
  // a block's histograms cost up to 2048 global atomics
  const int per = n <= (1 << 17) ? 1024 : 4096;
  k_sort_hist8<<<std::min((n + per - 1) / per, 1184), kSortThreads, 0, s>>>(keys_a, n, passes, ghist);
  if (sys_passes) k_sort_hist_sys<<<(nsys + 255) / 256, 256, 0, s>>>(sys_off, nsys, ghist + 256 * passes);
  k_sort_hist_scan<<<passes + sys_passes, 256, 0, s>>>(ghist);
  unsigned long long* kin = keys_a;
  unsigned long long* kout = keys_b;
  int* vin = vals_a;
  int* vout = vals_b;
  for (int p = 0; p < passes + sys_passes; p++) {
    const int* vi = p == 0 ? vals_in : vin;
    unsigned* stp = status + (size_t)p * nt * 256;
    if (p < passes)
      k_sort_onesweep<ITEMS, false><<<nt, kSortThreads, 0, s>>>(kin, vi, n, 8 * p, ghist + 256 * p, stp,
                                                                counters + p, kout, vout, err, nullptr, 0);
    else
      k_sort_onesweep<ITEMS, true><<<nt, kSortThreads, 0, s>>>(kin, vi, n, 8 * (p - passes), ghist + 256 * p, stp,
                                                               counters + p, kout, vout, err, sys_off, nsys);
    unsigned long long* tk = kin; kin = kout; kout = tk;
    int* tv = vin; vin = vout; vout = tv;
  }
}

void radix_sort_pairs(unsigned long long* keys_a, unsigned long long* keys_b, int* vals_a, int* vals_b,
                      const int* vals_in, int n, unsigned* work, int* err, int passes, const int* sys_off, int nsys,
                      cudaStream_t s) {
  if (n <= 0) return;
  if (n <= kOneMax && nsys <= 1) {
    cudaFuncSetAttribute(k_sort_block, cudaFuncAttributeMaxDynamicSharedMemorySize, kOneSmem);
    // the warps that hold keys, and a thread per digit
    const int threads = std::max(256, (n + 32 * kOneItems - 1) / (32 * kOneItems) * 32);
    k_sort_block<<<1, threads, kOneSmem, s>>>(keys_a, vals_in, vals_a, n, passes);
  } else if (sort_items(n) == kSmallItems) {
    radix_sort_passes<kSmallItems>(keys_a, keys_b, vals_a, vals_b, vals_in, n, work, err, passes, sys_off, nsys, s);
  } else if (sort_items(n) == kMidItems) {
    radix_sort_passes<kMidItems>(keys_a, keys_b, vals_a, vals_b, vals_in, n, work, err, passes, sys_off, nsys, s);
  } else {
    radix_sort_passes<kLargeItems>(keys_a, keys_b, vals_a, vals_b, vals_in, n, work, err, passes, sys_off, nsys, s);
  }
}

// Self-test of the look-back bound: one pass over three tiles launched as two
// blocks with the tile counter starting at 1, so tile 0 never runs and tile 1
// waits on a flag that nothing sets.  The wait must end at its bound with
// kStatusSortTimeout in *err, and tile 2 must then finish behind tile 1.
// Returns the status bits (or a CUDA error as -1000 - code).
int sort_timeout_selftest(cudaStream_t s) {
  const int n = 3 * kSortThreads * kLargeItems, nt = 3;
  unsigned long long *ka = nullptr, *kb = nullptr;
  int *va = nullptr, *err = nullptr;
  unsigned *status = nullptr, *counter = nullptr, *gbase = nullptr;
  cudaError_t e = cudaSuccess;
  if (e == cudaSuccess) e = cudaMalloc(&ka, n * sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaMalloc(&kb, n * sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaMalloc(&va, 2 * n * sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&err, sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&status, (size_t)nt * 256 * sizeof(unsigned));
  if (e == cudaSuccess) e = cudaMalloc(&counter, sizeof(unsigned));
  if (e == cudaSuccess) e = cudaMalloc(&gbase, 256 * sizeof(unsigned));
  int result = 0;
  if (e == cudaSuccess) {
    cudaMemsetAsync(ka, 0, n * sizeof(unsigned long long), s);
    cudaMemsetAsync(status, 0, (size_t)nt * 256 * sizeof(unsigned), s);
    cudaMemsetAsync(gbase, 0, 256 * sizeof(unsigned), s);
    cudaMemsetAsync(err, 0, sizeof(int), s);
    const unsigned one = 1u;
    cudaMemcpyAsync(counter, &one, sizeof(unsigned), cudaMemcpyHostToDevice, s);
    k_sort_onesweep<kLargeItems, false><<<nt - 1, kSortThreads, 0, s>>>(ka, nullptr, n, 0, gbase, status, counter, kb, va + n, err,
                                                           nullptr, 0);
    cudaMemcpyAsync(&result, err, sizeof(int), cudaMemcpyDeviceToHost, s);
    e = cudaStreamSynchronize(s);
  }
  cudaFree(ka); cudaFree(kb); cudaFree(va); cudaFree(err); cudaFree(status); cudaFree(counter); cudaFree(gbase);
  return e == cudaSuccess ? result : -(int)e - 1000;
}

BONSAI_BOUNDS_ACCESSOR(bounds_word_sort)

}  // namespace bonsai
