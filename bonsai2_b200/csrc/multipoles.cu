// multipoles.cu -- monopole, quadrupole and opening size of every cell, bottom
// up.
//
// The reference (computeCellMultipoles, computeMultipoles.cu:81-190) gives a
// warp to every cell and rescans all of that cell's particles, O(N * depth)
// particle reads, with float products summed in double.  Here each leaf is
// reduced from its own particles (one thread per leaf, FP64, one pass: sums
// about the leaf's first particle, shifted to the centre of mass), and every
// node is combined from its
// children with the parallel-axis theorem, level by level from the deepest.
// Each particle is read once.  The quantities match the reference's definitions:
//   M, COM; Q = second moment about the COM per unit mass (:148-158);
//   particle bounding box -> l = max(2 max h, 1e-6), s = |cvec - COM|,
//   cellOp = l/theta + s, stored squared (:168-177).
// cell_ls = (l, s, M l^3, 1.5 tr I) lets a walk with per-group opening angles
// form (l/theta_g + s)^2.  Stored for the walk as three float4 per cell, in
// the form the force kernel stages them (mass-weighted, pre-scaled and
// negated so that it needs fewer operations; I = M Q):
//   cell_stage[3c]     = (COM, -0.5 tr I)
//   cell_stage[3c + 1] = (M, -3Ixx, -3Iyy, -3Izz)
//   cell_stage[3c + 2] = (-3Ixy, -3Ixz, -3Iyz, -1.5 tr I)
// The FP64 record (MpRec) holds M, COM and the moments; the particle bounding
// box is a separate array, float for float positions and double (DS) for
// double-single positions, where particles enter the FP64 sums as hi + lo,
// extents are exact, and the COM is stored as hi (cell_open) plus lo (cell_lo).
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"

namespace bonsai {

// leaf moments in one pass over the particles (1) or two (0: centre of mass,
// then central moments)
#ifndef BONSAI_MP_ONE_PASS
#define BONSAI_MP_ONE_PASS 1
#endif

template <bool DS>
struct BoxOf {
  typedef float T;
};
template <>
struct BoxOf<true> {
  typedef double T;
};

#ifndef BONSAI_MP_BATCH
#define BONSAI_MP_BATCH 4
#endif
constexpr int kMpBatch = BONSAI_MP_BATCH;  // leaf particles loaded ahead of their sums

// the walk's records of a cell
struct CellOut {
  float4 open, ls, stage[3], lo;
};
template <bool DS>
__device__ __forceinline__ CellOut cell_out(const MpRec& r, const typename BoxOf<DS>::T* bmin,
                                            const typename BoxOf<DS>::T* bmax, float inv_theta) {
  CellOut q;
  const float cx = (float)r.cx, cy = (float)r.cy, cz = (float)r.cz;
  const double tr = r.ixx + r.iyy + r.izz;
  const float t15 = (float)(1.5 * tr);
  float s, l;
  if (DS) {
    // w: the staged record's -0.5 tr I (cell_stage[3c].w), so that the
    // double-single walk, which loads cell_lo for every visited cell, stages
    // an accepted cell without another load
    q.lo = make_float4((float)(r.cx - (double)cx), (float)(r.cy - (double)cy), (float)(r.cz - (double)cz),
                       __fmul_rn(t15, -1.0f / 3.0f));
    // extents and centre offsets from the exact box and COM
    double hm = 0.0, d2 = 0.0;
    const double com[3] = {r.cx, r.cy, r.cz};
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const double v = 0.5 * ((double)bmax[k] + (double)bmin[k]) - com[k];
      hm = fmax(hm, 0.5 * ((double)bmax[k] - (double)bmin[k]));
      d2 += v * v;
    }
    s = (float)sqrt(d2);
    l = fmaxf((float)(2.0 * hm), 1.0e-6f);
  } else {
    const float vx = __fmul_rn(__fadd_rn((float)bmax[0], (float)bmin[0]), 0.5f);
    const float vy = __fmul_rn(__fadd_rn((float)bmax[1], (float)bmin[1]), 0.5f);
    const float vz = __fmul_rn(__fadd_rn((float)bmax[2], (float)bmin[2]), 0.5f);
    const float hx = __fmul_rn(__fsub_rn((float)bmax[0], (float)bmin[0]), 0.5f);
    const float hy = __fmul_rn(__fsub_rn((float)bmax[1], (float)bmin[1]), 0.5f);
    const float hz = __fmul_rn(__fsub_rn((float)bmax[2], (float)bmin[2]), 0.5f);
    const float dx = __fsub_rn(vx, cx), dy = __fsub_rn(vy, cy), dz = __fsub_rn(vz, cz);
    s = __fsqrt_rn(__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx))));
    l = fmaxf(__fmul_rn(2.0f, fmaxf(hx, fmaxf(hy, hz))), 1.0e-6f);
  }
  const float op = __fmaf_rn(l, inv_theta, s);
  q.open = make_float4(cx, cy, cz, __fmul_rn(op, op));
  // per-group opening angles recompute (l/theta_g + s)^2; the relative test
  // compares M l^3 (formed once here, in float) with tau ds^5
  const float mf = (float)r.m;
  // (the relative test's size is the box's l: the mass-weighted rms radius
  // sqrt(tr I / M) in its place ran 3-4 % slower at equal median error)
  const float mk = __fmul_rn(mf, __fmul_rn(l, __fmul_rn(l, l)));
  q.ls = make_float4(l, s, mk, t15);
  // the walk's staged record, copied to shared memory as it is (moments
  // negated so that every difference in the interaction is one add)
  q.stage[0] = make_float4(cx, cy, cz, __fmul_rn(t15, -1.0f / 3.0f));
  q.stage[1] = make_float4(mf, -(float)(3.0 * r.ixx), -(float)(3.0 * r.iyy), -(float)(3.0 * r.izz));
  q.stage[2] = make_float4(-(float)(3.0 * r.ixy), -(float)(3.0 * r.ixz), -(float)(3.0 * r.iyz), -t15);
  return q;
}

// box of cell c as two-element vectors (24 or 48 bytes per cell)
__device__ __forceinline__ void store_box(float* box, int c, const float* lo, const float* hi) {
  float2* b = reinterpret_cast<float2*>(box + 6 * (size_t)c);
  b[0] = make_float2(lo[0], lo[1]); b[1] = make_float2(lo[2], hi[0]); b[2] = make_float2(hi[1], hi[2]);
}
__device__ __forceinline__ void store_box(double* box, int c, const double* lo, const double* hi) {
  double2* b = reinterpret_cast<double2*>(box + 6 * (size_t)c);
  b[0] = make_double2(lo[0], lo[1]); b[1] = make_double2(lo[2], hi[0]); b[2] = make_double2(hi[1], hi[2]);
}
__device__ __forceinline__ void load_box(const float* box, int c, float* lo, float* hi) {
  const float2* q = reinterpret_cast<const float2*>(box + 6 * (size_t)c);
  const float2 a = __ldcg(q), b = __ldcg(q + 1), d = __ldcg(q + 2);
  lo[0] = a.x; lo[1] = a.y; lo[2] = b.x; hi[0] = b.y; hi[1] = d.x; hi[2] = d.y;
}
__device__ __forceinline__ void load_box(const double* box, int c, double* lo, double* hi) {
  const double2* q = reinterpret_cast<const double2*>(box + 6 * (size_t)c);
  const double2 a = __ldcg(q), b = __ldcg(q + 1), d = __ldcg(q + 2);
  lo[0] = a.x; lo[1] = a.y; lo[2] = b.x; hi[0] = b.y; hi[1] = d.x; hi[2] = d.y;
}

// ---------------------------------------------------------------------------
// Nodes, all levels in one cooperative launch: a grid-wide barrier between
// levels, eight lanes per node, one per child.  The records of a node's
// contiguous children are copied to shared memory by consecutive 16-byte
// loads; lanes then hold either a child (its parallel-axis terms) or a
// quantity (its sum over the children in child order), so a node costs about
// three memory round trips and the sums keep their order.  Bound by the
// levels' latency (about 2.5 us a level) below a million particles and by
// record traffic above.  Against one launch per level and one thread per node,
// 20 launches: 1024 particles 57 -> 17 us, 30,011 73 -> 33, 250,007 (leaves of 8)
// 111 -> 75, 2^20 117 -> 99; 2^24 363 -> 416 beside the group branch's gather
// (the whole step is the same there).
// ---------------------------------------------------------------------------
constexpr int kLvThreads = 512;
constexpr int kLvWarps = kLvThreads / 32;
constexpr int kLvMaxBlocksPerSm = 2;
// a node's eight child records in shared memory (doubles): 81, so that the two
// nodes of a half-warp fall on other banks
constexpr int kNodeDoubles = 81;
constexpr int kNarrow = 256;  // cells of a level that one block takes (64 teams)
constexpr int kBarrierSpin = 1 << 22;  // a few seconds

// All blocks have arrived `round` times.  The wait is bounded: past the bound
// it reports, and the caller returns (results invalid).
__device__ __forceinline__ bool grid_barrier(unsigned* count, unsigned round, int* status,
                                             int limit = kBarrierSpin) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(count, 1u);
    const unsigned target = round * gridDim.x;
    volatile unsigned* c = count;
    int spin = 0;
    while (*c < target && spin < limit) {
      __nanosleep(20);
      spin++;
    }
    ok = *c >= target;
    if (!ok) set_status(status, kStatusSortTimeout);
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

// Barrier of the level launch: the one block, the one cluster, or the grid.
enum LevelGroup { kOneBlock, kOneCluster, kWholeGrid };
constexpr int kLvCluster = 8;
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

template <bool DS, LevelGroup G>
__global__ void __launch_bounds__(kLvThreads, kLvMaxBlocksPerSm)
    k_mp_levels(TreeInfo* __restrict__ info, const uint4* __restrict__ cell_data, float inv_theta, MpRec* rec,
                typename BoxOf<DS>::T* box, float4* __restrict__ cell_open, float4* __restrict__ cell_stage,
                float4* __restrict__ cell_ls, int cell_cap, float4* __restrict__ cell_lo, unsigned* barrier) {
  typedef typename BoxOf<DS>::T B;
  extern __shared__ double node_sm[];
  const int ncells = info->ncells;
  if (ncells > cell_cap) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, team = lane >> 3, t = lane & 7;
  double* sm = node_sm + (size_t)(w * 4 + team) * kNodeDoubles;
  const int nwarps = gridDim.x * kLvWarps, gw = blockIdx.x * kLvWarps + w;
  unsigned round = 0;
  const int top = info->nlevels - 1;
  for (int L = top; L >= 1; L--) {
    const int b = info->level_beg[L], e = info->level_end[L];
    // A narrow level of a grid is the first block's alone, and between two
    // narrow levels the block's own barrier will do: a grid-wide one, about as
    // long as the level itself, is taken only before a wide level and after it.
    const bool narrow = G == kWholeGrid && e - b <= kNarrow;
    // cells a warp looks at together: fewer where the level would leave warps idle
    const int nw = narrow ? kLvWarps : nwarps;
    int span = 4;
    while (span < 32 && (long long)span * nw < e - b) span *= 2;
    const int cfirst = b + gw * span;
    // the first cells' words do not wait for the level below
    unsigned yl = (lane < span && cfirst + lane < e) ? __ldg(&cell_data[cfirst + lane].y) : 0xFFFFFFFFu;
    if (L < top) {
      if (G == kOneBlock) {
        __syncthreads();
      } else if (G == kOneCluster) {
        cluster_barrier();
      } else {
        const bool below = info->level_end[L + 1] - info->level_beg[L + 1] <= kNarrow;
        if (narrow && below) __syncthreads();
        else if (!grid_barrier(barrier, ++round, &info->status)) return;
      }
    }
    if (narrow && blockIdx.x != 0) continue;
    for (int c0 = cfirst; c0 < e; c0 += nw * span) {
      if (c0 != cfirst) yl = (lane < span && c0 + lane < e) ? __ldg(&cell_data[c0 + lane].y) : 0xFFFFFFFFu;
      unsigned nodes = __ballot_sync(kFull, yl != 0xFFFFFFFFu);
      while (nodes) {
        // this team's node: the team-th of the remaining ones
        unsigned rest = nodes;
        for (int k = 0; k < team; k++) rest &= rest - 1;
        const int src = rest ? __ffs(rest) - 1 : 0;
        const unsigned y = __shfl_sync(kFull, yl, src);
        const int p = c0 + src;
        const int first = (int)(y & 0x1FFFFFFFu);
        int nch = rest ? (int)(y >> 29) + 1 : 0;
        if (nch && !BONSAI_IN_RANGE(first + nch - 1, ncells, 0x307)) nch = 0;
        for (int k = 0; k < 4 && nodes; k++) nodes &= nodes - 1;
        // the children's records, 5 x 16 bytes each, and this lane's child's box
        const double2* src2 = reinterpret_cast<const double2*>(rec + first);
        double2 v[5];
#pragma unroll
        for (int k = 0; k < 5; k++)
          if (t + 8 * k < 5 * nch) v[k] = __ldcg(src2 + t + 8 * k);
        B lo[3], hi[3];
        if (t < nch) {
          load_box(box, first + t, lo, hi);
        } else {
#pragma unroll
          for (int a = 0; a < 3; a++) { lo[a] = (B)3.0e38; hi[a] = (B)-3.0e38; }
        }
#pragma unroll
        for (int k = 0; k < 5; k++)
          if (t + 8 * k < 5 * nch) {
            sm[2 * (t + 8 * k)] = v[k].x;
            sm[2 * (t + 8 * k) + 1] = v[k].y;
          }
#pragma unroll
        for (int o = 4; o; o >>= 1)
#pragma unroll
          for (int a = 0; a < 3; a++) {
            const B x = __shfl_xor_sync(kFull, lo[a], o), z = __shfl_xor_sync(kFull, hi[a], o);
            lo[a] = DS ? (B)fmin((double)lo[a], (double)x) : (B)fminf((float)lo[a], (float)x);
            hi[a] = DS ? (B)fmax((double)hi[a], (double)z) : (B)fmaxf((float)hi[a], (float)z);
          }
        __syncwarp();
        // lanes 0..3: M and the mass-weighted coordinates, in child order
        double sum = 0.0;
#pragma unroll 4
        for (int k = 0; k < nch; k++) sum = fma(sm[10 * k], (t & 3) ? sm[10 * k + (t & 3)] : 1.0, sum);
        MpRec P;
        P.m = __shfl_sync(kFull, sum, team * 8);
        double com = P.m > 0.0 ? sum / P.m : 0.0;
        if (!(P.m > 0.0) && (t & 3)) {
          const int a = (t & 3) - 1;
          com = 0.5 * ((double)(a == 0 ? lo[0] : a == 1 ? lo[1] : lo[2]) + (a == 0 ? hi[0] : a == 1 ? hi[1] : hi[2]));
        }
        P.cx = __shfl_sync(kFull, com, team * 8 + 1);
        P.cy = __shfl_sync(kFull, com, team * 8 + 2);
        P.cz = __shfl_sync(kFull, com, team * 8 + 3);
        // each lane its child's terms about the new centre, into the child's slots
        if (t < nch) {
          double* q = sm + 10 * t;
          const double mk = q[0];
          const double dx = q[1] - P.cx, dy = q[2] - P.cy, dz = q[3] - P.cz;
          q[4] = q[4] + mk * dx * dx;
          q[5] = q[5] + mk * dy * dy;
          q[6] = q[6] + mk * dz * dz;
          q[7] = q[7] + mk * dx * dy;
          q[8] = q[8] + mk * dx * dz;
          q[9] = q[9] + mk * dy * dz;
        }
        __syncwarp();
        // lanes 0..5: one moment each, in child order
        double in = 0.0;
        if (t < 6) {
#pragma unroll 4
          for (int k = 0; k < nch; k++) in += sm[10 * k + 4 + t];
        }
        P.ixx = __shfl_sync(kFull, in, team * 8);
        P.iyy = __shfl_sync(kFull, in, team * 8 + 1);
        P.izz = __shfl_sync(kFull, in, team * 8 + 2);
        P.ixy = __shfl_sync(kFull, in, team * 8 + 3);
        P.ixz = __shfl_sync(kFull, in, team * 8 + 4);
        P.iyz = __shfl_sync(kFull, in, team * 8 + 5);
        if (nch) {
          // the lanes share the stores
          const CellOut q = cell_out<DS>(P, lo, hi, inv_theta);
          double2* rp = reinterpret_cast<double2*>(rec + p);
          if (t == 0) { rp[0] = make_double2(P.m, P.cx); cell_open[p] = q.open; }
          if (t == 1) { rp[1] = make_double2(P.cy, P.cz); cell_ls[p] = q.ls; }
          if (t == 2) { rp[2] = make_double2(P.ixx, P.iyy); cell_stage[3 * (size_t)p] = q.stage[0]; }
          if (t == 3) { rp[3] = make_double2(P.izz, P.ixy); cell_stage[3 * (size_t)p + 1] = q.stage[1]; }
          if (t == 4) { rp[4] = make_double2(P.ixz, P.iyz); cell_stage[3 * (size_t)p + 2] = q.stage[2]; }
          if (t == 5) store_box(box, p, lo, hi);
          if (DS && t == 6) cell_lo[p] = q.lo;
        }
        __syncwarp();  // the shared records are free for the next nodes
      }
    }
  }
}

// One thread per leaf: the leaf's moments (one pass by default).
template <bool DS>
__global__ void __launch_bounds__(256) k_multipoles(const int* __restrict__ leaf_list, const TreeInfo* __restrict__ info,
                                                    const uint4* __restrict__ cell_data,
                                                    const float4* __restrict__ jpos, float inv_theta,
                                                    MpRec* __restrict__ rec, typename BoxOf<DS>::T* __restrict__ box,
                                                    float4* __restrict__ cell_open, float4* __restrict__ cell_stage, float4* __restrict__ cell_ls,
                                                    int cell_cap,
                                                    const float4* __restrict__ jlo, float4* __restrict__ cell_lo,
                                                    unsigned* __restrict__ barrier) {
  typedef typename BoxOf<DS>::T B;
  if (blockIdx.x == 0 && threadIdx.x == 0) *barrier = 0u;  // of the level launch that follows
  const int nleaves = info->nleaves;
  if (info->ncells > cell_cap) return;
  [[maybe_unused]] const int ncells = info->ncells, npart = info->npart;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nleaves; t += gridDim.x * blockDim.x) {
    const int c = leaf_list[t];
    if (!BONSAI_IN_RANGE(c, ncells, 0x301)) continue;
    const uint4 cd = cell_data[c];
    const int b = (int)cd.z, e = (int)cd.w;
    if (!BONSAI_IN_RANGE(e - 1, npart, 0x302) || !BONSAI_IN_RANGE(b, e, 0x306)) continue;
    MpRec r;
    B mn[3] = {(B)3.0e38, (B)3.0e38, (B)3.0e38}, mx[3] = {(B)-3.0e38, (B)-3.0e38, (B)-3.0e38};
#if BONSAI_MP_ONE_PASS
    // one pass: sums about the leaf's first particle x0 (d = x - x0), then the
    // shift to the centre of mass: COM = x0 + S1/M, I = S2 - S1 S1^T / M; the
    // cancellation is relative to the leaf's extent, not to |x0|
    double x0 = 0, y0 = 0, z0 = 0;
    double m = 0, s1x = 0, s1y = 0, s1z = 0, q[6] = {0, 0, 0, 0, 0, 0};
    // four particles' loads in flight before they are summed (in order)
    for (int i0 = b; i0 < e; i0 += kMpBatch) {
      float4 pb[kMpBatch], lb[kMpBatch];
#pragma unroll
      for (int u = 0; u < kMpBatch; u++) {
        const int i = min(i0 + u, e - 1);
        pb[u] = __ldg(jpos + i);
        if (DS) lb[u] = __ldg(jlo + i);
      }
      if (i0 == b) {
        x0 = pb[0].x; y0 = pb[0].y; z0 = pb[0].z;
        if (DS) { x0 += lb[0].x; y0 += lb[0].y; z0 += lb[0].z; }
      }
#pragma unroll
      for (int u = 0; u < kMpBatch; u++) {
        if (i0 + u >= e) break;
        const float4 p = pb[u];
        double px = p.x, py = p.y, pz = p.z;
        if (DS) {
          const float4 l = lb[u];
          px += l.x; py += l.y; pz += l.z;
          mn[0] = (B)fmin((double)mn[0], px); mn[1] = (B)fmin((double)mn[1], py); mn[2] = (B)fmin((double)mn[2], pz);
          mx[0] = (B)fmax((double)mx[0], px); mx[1] = (B)fmax((double)mx[1], py); mx[2] = (B)fmax((double)mx[2], pz);
        } else {
          mn[0] = (B)fminf((float)mn[0], p.x); mn[1] = (B)fminf((float)mn[1], p.y); mn[2] = (B)fminf((float)mn[2], p.z);
          mx[0] = (B)fmaxf((float)mx[0], p.x); mx[1] = (B)fmaxf((float)mx[1], p.y); mx[2] = (B)fmaxf((float)mx[2], p.z);
        }
        const double w = p.w, dx = px - x0, dy = py - y0, dz = pz - z0;
        m += w;
        s1x += w * dx; s1y += w * dy; s1z += w * dz;
        q[0] += w * dx * dx; q[1] += w * dy * dy; q[2] += w * dz * dz;
        q[3] += w * dx * dy; q[4] += w * dx * dz; q[5] += w * dy * dz;
      }
    }
    if (m > 0.0) {
      const double ux = s1x / m, uy = s1y / m, uz = s1z / m;
      r.cx = x0 + ux; r.cy = y0 + uy; r.cz = z0 + uz;
      q[0] -= s1x * ux; q[1] -= s1y * uy; q[2] -= s1z * uz;
      q[3] -= s1x * uy; q[4] -= s1x * uz; q[5] -= s1y * uz;
    } else {
      r.cx = 0.5 * ((double)mn[0] + mx[0]); r.cy = 0.5 * ((double)mn[1] + mx[1]); r.cz = 0.5 * ((double)mn[2] + mx[2]);
    }
#else
    double m = 0, sx = 0, sy = 0, sz = 0;
    for (int i = b; i < e; i++) {
      const float4 p = __ldg(jpos + i);
      double px = p.x, py = p.y, pz = p.z;
      if (DS) {
        const float4 l = __ldg(jlo + i);
        px += l.x; py += l.y; pz += l.z;
        mn[0] = (B)fmin((double)mn[0], px); mn[1] = (B)fmin((double)mn[1], py); mn[2] = (B)fmin((double)mn[2], pz);
        mx[0] = (B)fmax((double)mx[0], px); mx[1] = (B)fmax((double)mx[1], py); mx[2] = (B)fmax((double)mx[2], pz);
      } else {
        mn[0] = (B)fminf((float)mn[0], p.x); mn[1] = (B)fminf((float)mn[1], p.y); mn[2] = (B)fminf((float)mn[2], p.z);
        mx[0] = (B)fmaxf((float)mx[0], p.x); mx[1] = (B)fmaxf((float)mx[1], p.y); mx[2] = (B)fmaxf((float)mx[2], p.z);
      }
      m += p.w;
      sx += (double)p.w * px; sy += (double)p.w * py; sz += (double)p.w * pz;
    }
    if (m > 0.0) { r.cx = sx / m; r.cy = sy / m; r.cz = sz / m; }
    else {
      r.cx = 0.5 * ((double)mn[0] + mx[0]); r.cy = 0.5 * ((double)mn[1] + mx[1]); r.cz = 0.5 * ((double)mn[2] + mx[2]);
    }
    double q[6] = {0, 0, 0, 0, 0, 0};
    for (int i = b; i < e; i++) {
      const float4 p = __ldg(jpos + i);
      double px = p.x, py = p.y, pz = p.z;
      if (DS) {
        const float4 l = __ldg(jlo + i);
        px += l.x; py += l.y; pz += l.z;
      }
      const double dx = px - r.cx, dy = py - r.cy, dz = pz - r.cz, w = p.w;
      q[0] += w * dx * dx; q[1] += w * dy * dy; q[2] += w * dz * dz;
      q[3] += w * dx * dy; q[4] += w * dx * dz; q[5] += w * dy * dz;
    }
#endif
    r.m = m;
    r.ixx = q[0]; r.iyy = q[1]; r.izz = q[2]; r.ixy = q[3]; r.ixz = q[4]; r.iyz = q[5];
    const CellOut o = cell_out<DS>(r, mn, mx, inv_theta);
    double2* rp = reinterpret_cast<double2*>(rec + c);
    rp[0] = make_double2(r.m, r.cx);
    rp[1] = make_double2(r.cy, r.cz);
    rp[2] = make_double2(r.ixx, r.iyy);
    rp[3] = make_double2(r.izz, r.ixy);
    rp[4] = make_double2(r.ixz, r.iyz);
    store_box(box, c, mn, mx);
    cell_open[c] = o.open;
    cell_ls[c] = o.ls;
    for (int k = 0; k < 3; k++) cell_stage[3 * (size_t)c + k] = o.stage[k];
    if (DS) cell_lo[c] = o.lo;
  }
}

// One block up to 2048 particles, a cluster of eight (its hardware barrier) up to
// 16,384, above that the grid: build of 4096 particles 100 -> 94 us against the
// grid, 16,384 126.5 -> 124.4, 30,011 129 -> 141 (eight blocks are too few).
constexpr int kClusterMin = 2048, kClusterMax = 16384;
constexpr int kLvSmem = kLvWarps * 4 * kNodeDoubles * (int)sizeof(double);

// blocks of the level launch that are resident at once
int multipole_level_blocks(int nsm) {
  int a = 0, b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_mp_levels<false, kWholeGrid>, kLvThreads, kLvSmem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_mp_levels<true, kWholeGrid>, kLvThreads, kLvSmem) != cudaSuccess)
    return 1;
  return std::max(1, nsm * std::min(std::min(a, b), kLvMaxBlocksPerSm));
}

template <bool DS>
static void launch_multipoles_of(const int* leaf_list, TreeInfo* info, const uint4* cell_data, const float4* jpos,
                                 int n, float inv_theta, MpRec* rec, typename BoxOf<DS>::T* box, float4* cell_open,
                                 float4* cell_stage, float4* cell_ls, int cell_cap, const float4* jlo,
                                 float4* cell_lo, int nblocks, unsigned* barrier, int level_blocks, cudaStream_t s) {
  k_multipoles<DS><<<nblocks, 256, 0, s>>>(leaf_list, info, cell_data, jpos, inv_theta, rec, box, cell_open,
                                           cell_stage, cell_ls, cell_cap, jlo, cell_lo, barrier);
  if (n <= kClusterMin) {
    k_mp_levels<DS, kOneBlock><<<1, kLvThreads, kLvSmem, s>>>(info, cell_data, inv_theta, rec, box, cell_open,
                                                              cell_stage, cell_ls, cell_cap, cell_lo, barrier);
    return;
  }
  cudaLaunchAttribute at[1];
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kLvThreads);
  cfg.dynamicSmemBytes = kLvSmem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (n <= kClusterMax) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kLvCluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(kLvCluster);
    cudaLaunchKernelEx(&cfg, k_mp_levels<DS, kOneCluster>, info, cell_data, inv_theta, rec, box, cell_open, cell_stage,
                       cell_ls, cell_cap, cell_lo, barrier);
  } else {
    // about 1024 particles per block: more give the widest level its teams, fewer
    // make the barrier cheaper
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.gridDim = dim3(std::min(level_blocks, n / 1024));
    cudaLaunchKernelEx(&cfg, k_mp_levels<DS, kWholeGrid>, info, cell_data, inv_theta, rec, box, cell_open, cell_stage,
                       cell_ls, cell_cap, cell_lo, barrier);
  }
}

void launch_multipoles(const int* leaf_list, TreeInfo* info, const uint4* cell_data, const float4* jpos, int n,
                       float inv_theta, MpRec* rec, void* box, float4* cell_open, float4* cell_stage,
                       float4* cell_ls, int cell_cap, const float4* jlo, float4* cell_lo, int nblocks,
                       unsigned* barrier, int level_blocks, cudaStream_t s) {
  if (jlo)
    launch_multipoles_of<true>(leaf_list, info, cell_data, jpos, n, inv_theta, rec, static_cast<double*>(box),
                               cell_open, cell_stage, cell_ls, cell_cap, jlo, cell_lo, nblocks, barrier,
                               level_blocks, s);
  else
    launch_multipoles_of<false>(leaf_list, info, cell_data, jpos, n, inv_theta, rec, static_cast<float*>(box),
                                cell_open, cell_stage, cell_ls, cell_cap, nullptr, nullptr, nblocks, barrier,
                                level_blocks, s);
}

// Self-test of the level barrier's bound.  Two blocks meet at round 1, and then
// at round 3 with nobody at round 2: the wait runs out, and both must report and leave.
__global__ void k_barrier_selftest(unsigned* count, int* status, unsigned* left) {
  if (!grid_barrier(count, 1, status)) return;
  const bool late = !grid_barrier(count, 3, status, 1 << 12);
  if (threadIdx.x == 0 && late) atomicAdd(left, 1u);
}

// Returns the status bits, 0 when a block did not report (or a CUDA error as -1000 - code).
int barrier_timeout_selftest(cudaStream_t s) {
  constexpr unsigned kBlocks = 2;
  unsigned* word = nullptr;  // arrivals, status, blocks that gave up
  unsigned host[3] = {0, 0, 0};
  cudaError_t e = cudaMalloc(&word, sizeof(host));
  if (e == cudaSuccess) e = cudaMemsetAsync(word, 0, sizeof(host), s);
  if (e == cudaSuccess) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kBlocks);
    cfg.blockDim = dim3(64);
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, k_barrier_selftest, word, reinterpret_cast<int*>(word + 1), word + 2);
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(host, word, sizeof(host), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cudaFree(word);
  if (e != cudaSuccess) return -(int)e - 1000;
  return host[2] == kBlocks ? (int)host[1] : 0;
}

// Reference-layout view of the multipoles (debug/parity getter):
// size = (COM, cellOp^2), mono = (COM, M), quad0 = (xx,yy,zz,xy), quad1 = (xz,yz)
// with Q per unit mass (computeMultipoles.cu:180-188).
__global__ void k_multipoles_ref_layout(const TreeInfo* __restrict__ info, const float4* __restrict__ cell_open,
                                        const MpRec* __restrict__ rec, float4* __restrict__ size,
                                        float4* __restrict__ mono, float4* __restrict__ quad0,
                                        float2* __restrict__ quad1) {
  const int nc = info->ncells;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += gridDim.x * blockDim.x) {
    const MpRec r = rec[c];
    const float4 o = cell_open[c];
    const double im = r.m > 0 ? 1.0 / r.m : 0.0;
    size[c] = o;
    mono[c] = make_float4(o.x, o.y, o.z, (float)r.m);
    quad0[c] = make_float4((float)(r.ixx * im), (float)(r.iyy * im), (float)(r.izz * im), (float)(r.ixy * im));
    quad1[c] = make_float2((float)(r.ixz * im), (float)(r.iyz * im));
  }
}

BONSAI_BOUNDS_ACCESSOR(bounds_word_multipoles)

}  // namespace bonsai
