// tree.cu -- octree from the sorted octant-path keys, in four launches and no
// host round trip.
//
// The reference builds the tree by a recursive CUDA-dynamic-parallelism
// partition (buildOctant, buildTree.cu:170-722) and then stable-sorts the
// cells by level (buildTree.cu:725-841,932-958).  Its cell set is defined by
// two rules: the root is always split, and a cell with more than nLeaf
// particles is split (buildTree.cu:394-395,444,541).  With particles sorted
// by the octant path, every cell at level L is a maximal run of equal
// 3L-bit key prefix, so the cell set follows from d(i), the level at which
// keys i-1 and i first differ:
//   * with m(i) = min d(i+1..i+nLeaf) (d = 0 past the end), the level-L run
//     starting at i holds more than nLeaf particles iff d(i) <= L < m(i);
//     all of those runs are nodes, and the chain of cells that start at i
//     runs from max(d(i),1) down to the first level whose run is small
//     (a leaf), or to level 21 (a fat leaf, flagged);
//   * a small run starting at i at level d(i) >= 2 is a leaf iff its parent
//     run (level d(i)-1) holds more than nLeaf particles, which is decided
//     from d inside the window i-nLeaf .. i+nLeaf.
// Both rules together: with M(i) = max m(i-nLeaf..i), the level-L run that
// holds position i has more than nLeaf particles iff L < M(i) (some window of
// nLeaf + 1 positions around i lies inside it), so the leaf that holds i is at
// level l(i) = max(M(i), 1), a leaf starts at i iff d(i) <= l(i), and the
// chain of cells that start there is [max(d(i),1), l(i)]: a sliding minimum
// and a sliding maximum over bytes, four positions per instruction.
// Launch 1 computes the chains of a tile of positions (halo 64 >= nLeaf) and a
// per-level histogram; launch 2 scans the histogram rows (one block per row);
// launch 3 writes the cells level-major, key order inside a level (the
// canonical form of the reference's cell order), with children contiguous, the
// leaf list, parent links and the level ranges.  A cell's slot is the number of
// cells of its level that start before it, counted by warp ballots, and every
// other index of the tree is such a count too: a node's first child is the
// number of level L+1 cells that start before it, a cell's parent is the last
// level L-1 cell that starts at or before it, and where a chain [a, b] starts
// at position j, the cells of levels a .. l(j-1) that hold position j-1 end:
// the last cells of those levels that start before j, whose run end is j and
// whose last child is the last level L+1 cell before j.  Launch 4 puts the
// child counts into the node words.  Nothing searches the keys and no level
// waits for another.
#include "common.cuh"
#include "kernels.cuh"

namespace bonsai {

constexpr int kTreeThreads = 256;
constexpr int kTreeWarps = kTreeThreads / 32;
constexpr int kHalo = 64;           // max nLeaf
constexpr int kNL = kMaxLevel + 1;  // rows 0..21 (row 0 unused)

// Positions per tile: a warp of k_tree_cells goes through its 128 positions in
// four chunks of 32.  (4096-position tiles make that a chain of 16 chunks: cells
// of 1.7M particles 93 us against 50, the histogram scan of 16M 240 against 44.)
constexpr int kTreeTile = 1024;
int tree_tiles(int n) { return (n + kTreeTile - 1) / kTreeTile; }

// hist: 2 * kNL rows of tree_tiles(n), then the rows' totals, their bases and
// the scan's ticket (zero before the first build)
size_t tree_hist_words(int n) { return (size_t)2 * kNL * tree_tiles(n) + 4 * kNL + 1; }

// A chain word: first level a (0: no cell starts here) in bits 0..4, bit 7
// where a system starts (d = 0), last level b (the leaf's) in bits 8..12.
__device__ __forceinline__ int chain_a(unsigned c) { return (int)(c & 31u); }
__device__ __forceinline__ int chain_b(unsigned c) { return (int)((c >> 8) & 31u); }

// the word of four bytes that starts `off` bytes after word x (off >= 0)
__device__ __forceinline__ unsigned bytes_at(const unsigned* w, int x, int off) {
  const int q = x + (off >> 2);
  return (off & 3) ? __funnelshift_r(w[q], w[q + 1], 8 * (off & 3)) : w[q];
}

// Bound by instruction issue (the key differences and about ten byte-wise
// steps, four positions each) above a million keys, by one tile's latency below:
// 2^24 keys 456 -> 117 us beside the group branch, 1024 keys 28 -> 4.4 us,
// against the form that looked for the parent run of every position by binary
// lifting, 16 positions in a row per thread.
__global__ void __launch_bounds__(kTreeThreads) k_tree_chains(const unsigned long long* __restrict__ keys, int n,
                                                              int nleaf, uint16_t* __restrict__ chain,
                                                              unsigned* __restrict__ hist, int nb,
                                                              int* __restrict__ status,
                                                              const int* __restrict__ sys_off, int nsys) {
  constexpr int kLen = kTreeTile + 2 * kHalo;  // positions of the tile with its halo, from t0 - kHalo
  constexpr int kWords = kLen / 4;
  __shared__ __align__(16) unsigned char sd[kLen];  // d (0 at and before position 0, and from n on)
  // window minima and maxima; the words past kWords are only read into bytes
  // that no later step takes
  __shared__ unsigned wa[kWords + 20], wb[kWords + 20];
  __shared__ unsigned ha[kNL], hl[kNL];
  const int t0 = blockIdx.x * kTreeTile;
  if (threadIdx.x < kNL) { ha[threadIdx.x] = 0; hl[threadIdx.x] = 0; }
  if (threadIdx.x < 20) { wa[kWords + threadIdx.x] = 0; wb[kWords + threadIdx.x] = 0; }
  for (int j = threadIdx.x; j < kLen; j += kTreeThreads) {
    const int p = t0 - kHalo + j;
    unsigned char v = 0;
    if (p > 0 && p < n) v = (unsigned char)diff_level(__ldg(keys + p - 1), __ldg(keys + p));
    sd[j] = v;
  }
  __syncthreads();
  if (nsys > 1) {
    // In an ensemble d = 0 at every system start: a system's first particle
    // starts a level-1 cell, and no run crosses into the next system (the
    // values d takes at 0 and past n when the system is alone).
    const int lo = max(t0 - kHalo, 0), hi = t0 + kTreeTile + kHalo;
    for (int s = sys_of(sys_off, nsys, min(lo, n - 1)) + threadIdx.x; s < nsys; s += kTreeThreads) {
      const int p = sys_off[s];
      if (p >= hi) break;
      if (p >= lo) sd[p - (t0 - kHalo)] = 0;
    }
    __syncthreads();
  }
  const unsigned* d4 = reinterpret_cast<const unsigned*>(sd);
  for (int x = threadIdx.x; x < kWords; x += kTreeThreads) wa[x] = d4[x];
  __syncthreads();
  unsigned *in = wa, *out = wb;
  // m(s) = min d(s+1 .. s+nleaf): minima of power-of-two windows, then two of
  // them that overlap
  int wp = 1;
  for (; 2 * wp <= nleaf; wp *= 2) {
    for (int x = threadIdx.x; x < kWords; x += kTreeThreads) out[x] = __vminu4(in[x], bytes_at(in, x, wp));
    __syncthreads();
    unsigned* tmp = in; in = out; out = tmp;
  }
  for (int x = threadIdx.x; x < kWords; x += kTreeThreads)
    out[x] = __vminu4(bytes_at(in, x, 1), bytes_at(in, x, 1 + nleaf - wp));
  __syncthreads();
  { unsigned* tmp = in; in = out; out = tmp; }
  // M(i) = max m(i-nleaf .. i), a window of nleaf + 1
  int wq = 1;
  for (; 2 * wq <= nleaf + 1; wq *= 2) {
    for (int x = threadIdx.x; x < kWords; x += kTreeThreads) out[x] = __vmaxu4(in[x], bytes_at(in, x, wq));
    __syncthreads();
    unsigned* tmp = in; in = out; out = tmp;
  }
  bool anyfat = false;
  for (int x = threadIdx.x; x < kTreeTile / 4; x += kTreeThreads) {
    const int p = t0 + 4 * x;
    if (p >= n) break;
    const int off = kHalo - nleaf;  // the window's first byte, from this word's place in the tile
    const unsigned M = __vmaxu4(bytes_at(in, x, off), bytes_at(in, x, kHalo + 1 - wq));
    const unsigned D = d4[x + kHalo / 4];
    unsigned short c[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int d = (int)((D >> (8 * k)) & 255u), m = (int)((M >> (8 * k)) & 255u);
      const int b = max(m, 1);
      c[k] = 0;
      if (p + k < n && d <= kMaxLevel && d <= b) {
        const int a = max(d, 1), be = min(b, kMaxLevel);
        anyfat |= b > kMaxLevel;
        c[k] = (unsigned short)(a | (d == 0 ? 128 : 0) | (be << 8));
        atomicAdd(&ha[a], 1u);
        atomicAdd(&hl[be], 1u);
      }
    }
    if (p + 4 <= n) {
      *reinterpret_cast<ushort4*>(chain + p) = make_ushort4(c[0], c[1], c[2], c[3]);
    } else {
      for (int k = 0; k < 4 && p + k < n; k++) chain[p + k] = c[k];
    }
  }
  if (__any_sync(kFull, anyfat) && lane_id() == 0) set_status(status, kStatusDepth);
  __syncthreads();
  if (threadIdx.x < kNL) {
    // cells of level L: the chains that start at or above it, less those that ended above it
    unsigned c = 0;
    for (int L = 1; L <= (int)threadIdx.x; L++) c += ha[L] - (L > 1 ? hl[L - 1] : 0u);
    hist[threadIdx.x * nb + blockIdx.x] = c;
    hist[(kNL + threadIdx.x) * nb + blockIdx.x] = hl[threadIdx.x];
  }
}

// Exclusive scan of each histogram row across the tiles, one block per row; the
// last block to finish chains the row totals into row bases (cells
// level-major, leaves ordered likewise) and fills the tree info.
__global__ void __launch_bounds__(kTreeThreads) k_tree_scan(unsigned* __restrict__ hist, int nb, int cell_cap,
                                                            int leaf_cap, int n, TreeInfo* __restrict__ info) {
  __shared__ unsigned sh[kTreeWarps];
  __shared__ bool last;
  const int row = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned* h = hist + (size_t)row * nb;
  unsigned* tot = hist + (size_t)2 * kNL * nb;
  unsigned* base = tot + 2 * kNL;
  unsigned* ticket = base + 2 * kNL;
  unsigned carry = 0;
  if (row % kNL > 0) {
    for (int b0 = 0; b0 < nb; b0 += 4 * kTreeThreads) {
      const int b = b0 + 4 * threadIdx.x;
      unsigned v[4], s = 0;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        v[q] = b + q < nb ? h[b + q] : 0u;
        s += v[q];
      }
      const unsigned incl = (unsigned)warp_incl_scan((int)s);
      if (lane == 31) sh[w] = incl;
      __syncthreads();
      unsigned run = carry + incl - s;
#pragma unroll
      for (int q = 0; q < kTreeWarps; q++) {
        if (q < w) run += sh[q];
        carry += sh[q];
      }
#pragma unroll
      for (int q = 0; q < 4; q++) {
        if (b + q < nb) h[b + q] = run;
        run += v[q];
      }
      __syncthreads();
    }
  }
  if (threadIdx.x == 0) {
    tot[row] = carry;
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last || w) return;
  __threadfence();
  // lane L: level L's cells (c) and leaves (l)
  const unsigned c = lane < kNL ? __ldcg(tot + lane) : 0u, l = lane < kNL ? __ldcg(tot + kNL + lane) : 0u;
  const unsigned ce = (unsigned)warp_incl_scan((int)c), le = (unsigned)warp_incl_scan((int)l);
  if (lane < kNL) {
    base[lane] = ce - c;
    base[kNL + lane] = le - l;
  }
  info->level_beg[lane] = (int)(ce - c);
  info->level_end[lane] = (int)ce;
  const unsigned present = __ballot_sync(kFull, c > 0);
  if (lane == 31) {
    info->ncells = (int)ce;
    info->nleaves = (int)le;
    info->nnodes = (int)(ce - le);
    info->nlevels = present ? 31 - __clz(present) : 0;
    info->npart = n;
    if ((int)ce > cell_cap || (int)le > leaf_cap) set_status(&info->status, kStatusCellCapacity);
    *ticket = 0u;
  }
}

__global__ void __launch_bounds__(kTreeThreads, 5) k_tree_cells(
    const uint16_t* __restrict__ chain, const unsigned* __restrict__ hist, int n, int nb, int cell_cap,
    TreeInfo* __restrict__ info, uint4* __restrict__ cell_data, int* __restrict__ cell_parent,
    int* __restrict__ leaf_list, int* __restrict__ cell_last, const int* __restrict__ sys_off, int nsys,
    int* __restrict__ root_beg) {
  constexpr int kSpan = kTreeTile / kTreeWarps;  // positions of a warp
  static_assert(kSpan == 128, "four chain words per lane");
  __shared__ unsigned wc[kTreeWarps][32], wl[kTreeWarps][32];
  if (info->ncells > cell_cap || info->nleaves > cell_cap) return;
  [[maybe_unused]] const int ncells = info->ncells, nleaves = info->nleaves;
  if (nsys > 1 && blockIdx.x == 0 && threadIdx.x == 0) root_beg[nsys] = info->level_end[1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = lanemask_lt();
  const int i0 = blockIdx.x * kTreeTile + w * kSpan, i1 = min(i0 + kSpan, n);
  unsigned cw[kSpan / 32];  // the warp's chain words
#pragma unroll
  for (int k = 0; k < kSpan / 32; k++) {
    const int i = i0 + 32 * k + lane;
    cw[k] = i < i1 ? (unsigned)__ldg(chain + i) : 0u;
  }
  // lane L counts the warp's cells and leaves of level L
  unsigned runc = 0, runl = 0;
#pragma unroll
  for (int k = 0; k < kSpan / 32; k++) {
    const unsigned c = cw[k];
    const int a = chain_a(c), b = chain_b(c);
    const unsigned starts = __ballot_sync(kFull, a != 0);
    if (!starts) continue;
    const int lmin = __reduce_min_sync(kFull, a ? a : 31), lmax = __reduce_max_sync(kFull, b);
    for (int L = lmin; L <= lmax; L++) {
      const unsigned mc = __ballot_sync(kFull, a && a <= L && L <= b);
      const unsigned ml = __ballot_sync(kFull, a && b == L);
      if (lane == L) {
        runc += __popc(mc);
        runl += __popc(ml);
      }
    }
  }
  wc[w][lane] = runc;
  wl[w][lane] = runl;
  __syncthreads();
  // the slots of the warp's first cell and leaf of level L
  const unsigned* base = hist + (size_t)2 * kNL * nb + 2 * kNL;
  runc = runl = 0;
  if (lane < kNL) {
    runc = base[lane] + (lane ? hist[(size_t)lane * nb + blockIdx.x] : 0u);
    runl = base[kNL + lane] + (lane ? hist[(size_t)(kNL + lane) * nb + blockIdx.x] : 0u);
  }
  for (int q = 0; q < w; q++) {
    runc += wc[q][lane];
    runl += wl[q][lane];
  }
  if (i0 >= i1) return;
  // the level of the leaf that holds the position before the warp's first: a
  // leaf holds at most 64 particles, unless it is a fat one of the last level
  int pcarry = 0;
  if (i0 > 0) {
    const unsigned c0 = i0 - 1 - lane >= 0 ? (unsigned)__ldg(chain + i0 - 1 - lane) : 0u;
    const unsigned c1 = i0 - 33 - lane >= 0 ? (unsigned)__ldg(chain + i0 - 33 - lane) : 0u;
    const unsigned s0 = __ballot_sync(kFull, chain_a(c0) != 0), s1 = __ballot_sync(kFull, chain_a(c1) != 0);
    const int b0 = __shfl_sync(kFull, chain_b(c0), s0 ? __ffs(s0) - 1 : 0);
    const int b1 = __shfl_sync(kFull, chain_b(c1), s1 ? __ffs(s1) - 1 : 0);
    pcarry = s0 ? b0 : (s1 ? b1 : kMaxLevel);
  }
#pragma unroll 1
  for (int k = 0; k < kSpan / 32; k++) {
    const int i = i0 + 32 * k + lane;
    const unsigned c = k == 0 ? cw[0] : k == 1 ? cw[1] : k == 2 ? cw[2] : cw[3];
    const int a = chain_a(c), b = chain_b(c);
    const unsigned starts = __ballot_sync(kFull, a != 0);
    if (!starts) continue;
    // pb: level of the leaf that ends at i (0 at position 0: none does)
    const unsigned before = starts & lt;
    const int pl = __shfl_sync(kFull, b, before ? 31 - __clz(before) : 0);
    const int pb = before ? pl : pcarry;
    pcarry = __shfl_sync(kFull, b, 31 - __clz(starts));
    const int lmin = __reduce_min_sync(kFull, a ? a : 31), lmax = __reduce_max_sync(kFull, a ? max(b, pb) : 0);
    // slot, nslot, pslot: cells of level L, L + 1, L - 1 that start before i
    int pslot = __shfl_sync(kFull, (int)runc, lmin - 1);
    unsigned mask = __ballot_sync(kFull, a && a <= lmin && lmin <= b);
    int slot = __shfl_sync(kFull, (int)runc, lmin) + __popc(mask & lt);
    for (int L = lmin; L <= lmax; L++) {
      const unsigned nmask = __ballot_sync(kFull, a && a <= L + 1 && L + 1 <= b);
      const int nslot = __shfl_sync(kFull, (int)runc, L + 1) + __popc(nmask & lt);
      const unsigned lmask = __ballot_sync(kFull, a && b == L);
      const int lslot = __shfl_sync(kFull, (int)runl, L) + __popc(lmask & lt);
      if (a && a <= L) {
        // the cell of level L that holds position i - 1 ends here
        if (L <= pb && BONSAI_IN_RANGE(slot - 1, ncells, 0x104)) {
          cell_data[slot - 1].w = (unsigned)i;
          if (L < pb) cell_last[slot - 1] = nslot;
        }
        if (L <= b && BONSAI_IN_RANGE(slot, ncells, 0x102)) {
          const bool leaf = L == b;
          // the level L - 1 cell that starts here when the chain covers that
          // level, else the last one before
          const int parent = L == 1 ? -1 : pslot - (a <= L - 1 ? 0 : 1);
          if (leaf && BONSAI_IN_RANGE(lslot, nleaves, 0x101)) leaf_list[lslot] = slot;
          // a system's first level-1 cell starts at the system's first particle
          if (nsys > 1 && L == 1 && (c & 128u)) root_beg[sys_of(sys_off, nsys, i)] = slot;
          uint2 xy;
          // level-1 cells: parent 0, as the reference stores them
          xy.x = L == 1 ? (unsigned)(1 << 27) : ((unsigned)parent | ((unsigned)L << 27));
          xy.y = leaf ? 0xFFFFFFFFu : (unsigned)nslot;  // nodes: the first child (the count follows)
          *reinterpret_cast<uint2*>(cell_data + slot) = xy;
          cell_data[slot].z = (unsigned)i;
          cell_parent[slot] = parent;
        }
      }
      if (lane == L) {
        runc += __popc(mask);
        runl += __popc(lmask);
      }
      pslot = slot;
      slot = nslot;
      mask = nmask;
    }
  }
  // the cells still open at the last position end at n
  if (i1 == n) {
    const int nlast = __shfl_down_sync(kFull, (int)runc, 1);
    if (lane >= 1 && lane <= pcarry && BONSAI_IN_RANGE((int)runc - 1, ncells, 0x105)) {
      cell_data[runc - 1].w = (unsigned)n;
      if (lane < pcarry) cell_last[runc - 1] = nlast;
    }
  }
}

// child counts into the nodes' words
__global__ void __launch_bounds__(kTreeThreads) k_tree_counts(const TreeInfo* __restrict__ info,
                                                              uint4* __restrict__ cell_data,
                                                              const int* __restrict__ cell_last, int cell_cap) {
  const int nc = info->ncells;
  if (nc > cell_cap || info->nleaves > cell_cap) return;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += gridDim.x * blockDim.x) {
    const unsigned y = cell_data[c].y;
    if (y != 0xFFFFFFFFu) cell_data[c].y = y | ((unsigned)(cell_last[c] - (int)y - 1) << 29);
  }
}

// Four launches.  (Run ends and child counts used to take one launch per level,
// 21 of 1.6 us each with few cells; cells of 1024 particles 15 -> 7 us.)
void build_tree(const unsigned long long* sorted_keys, int n, int nleaf, int cell_cap, int leaf_cap,
                uint16_t* chain, unsigned* hist, TreeInfo* info, uint4* cell_data, int* cell_parent, int* leaf_list,
                int* cell_last, const int* sys_off, int nsys, int* root_beg, cudaStream_t s) {
  const int nb = tree_tiles(n);
  k_tree_chains<<<nb, kTreeThreads, 0, s>>>(sorted_keys, n, nleaf, chain, hist, nb, &info->status, sys_off, nsys);
  k_tree_scan<<<2 * kNL, kTreeThreads, 0, s>>>(hist, nb, cell_cap, leaf_cap, n, info);
  k_tree_cells<<<nb, kTreeThreads, 0, s>>>(chain, hist, n, nb, cell_cap, info, cell_data, cell_parent, leaf_list,
                                           cell_last, sys_off, nsys, root_beg);
  const int cb = (n + kTreeThreads - 1) / kTreeThreads;
  k_tree_counts<<<cb < 1184 ? cb : 1184, kTreeThreads, 0, s>>>(info, cell_data, cell_last, cell_cap);
}

BONSAI_BOUNDS_ACCESSOR(bounds_word_tree)

}  // namespace bonsai
