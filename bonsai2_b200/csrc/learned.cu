// learned.cu -- per-group opening bounds from a small MLP.
//
// The walk opens a cell when the group is inside its geometric opening
// sphere (computeForces.cu:30-54) at the group's angle theta_g, or -- in the
// relative accuracy mode -- when the cell's octupole truncation error, of
// order M l^3 / ds^5, exceeds the group's bound tau_g.  A single angle must
// suit the worst group; per-group angles alone gain little (their best
// allocation is a few tens of percent and cannot be predicted from group
// features), while a bound on each cell's truncation error relative to the
// group's own acceleration puts the error budget where it matters.  Here a
// 16 -> 64 -> 64 -> 1 network maps group features to y_g = log10(tau_g / A_g),
// A_g being the group's mean |a| of the previous force evaluation; it is
// trained on pairs (features, y label) that the walk and the FP64 direct sum
// generate (bonsai2_b200/learned.py: each group's error and cost over a grid
// of y; the label is the cost-optimal y for the error budget, or the y at
// which the group's error meets the target), with this file's own forward
// and backward kernels.  theta_g is then a fixed safety bound.  Without previous
// accelerations (the first evaluation after particles are loaded) every
// group walks at the fixed angle (theta mode 0's walk, bit for bit).
//
// Features (per group, normalised logs clamped to [-10, 10]): size, radius,
// tree depth (common PH-key prefix), distance from and mass share of its
// system, density, shape, system size, softening over radius, the previous
// acceleration scale A_g and its spread over the group, and -- recorded by
// the previous walk of the group holding the group's middle particle -- the
// number of cells near the opening boundary, the mass share of the accepted
// cells near it, and the force-weighted quadrupole norm of the accepted
// cells.
//
// Weight vector layout (kMlpWeights floats): W1[64][16], b1[64], W2[64][64],
// b2[64], w3[64], b3.  Hidden activations tanh; output
// y = lo + (hi - lo) * sigmoid(z).
#include "common.cuh"
#include "kernels.cuh"

#include <cuda_fp16.h>

namespace bonsai {

constexpr int kF = kMlpFeatures, kH = kMlpHidden;
constexpr int oW1 = 0, oB1 = oW1 + kH * kF, oW2 = oB1 + kH, oB2 = oW2 + kH * kH, oW3 = oB2 + kH, oB3 = oW3 + kH;
static_assert(oB3 + 1 == kMlpWeights, "weight layout");

__device__ __forceinline__ float safe_log10(float x) { return log10f(fmaxf(x, 1e-30f)); }

// ---------------------------------------------------------------------------
// Group features (one warp per group; groups are contiguous in PH order).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_group_features(const int2* __restrict__ groups,
                                                        const TreeInfo* __restrict__ info,
                                                        const float4* __restrict__ ipos,
                                                        const unsigned long long* __restrict__ ph_sorted,
                                                        const MpRec* __restrict__ rec, const Box* __restrict__ box,
                                                        int n, int ncrit, float eps, float* __restrict__ feat,
                                                        const int* __restrict__ sys_off, int nsys,
                                                        const int* __restrict__ root_beg, const PrevEval prev,
                                                        float* __restrict__ amag) {
  const int lane = threadIdx.x & 31;
  const int ng = info->ngroups;
  const bool have_prev = prev.acc_valid && *prev.acc_valid;
  // the group's system: its centre of mass and mass from its level-1 cells,
  // its box and its size (an ensemble's systems each have their own)
  int sys = -1;
  float mtot = 0.f, cx = 0.f, cy = 0.f, cz = 0.f, hs = 0.f;
  int ns = n;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  for (int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < ng; g += nw) {
    const int2 gd = groups[g];
    const int pb = gd.x, np = gd.y;
    const int s = nsys > 1 ? sys_of(sys_off, nsys, pb) : 0;
    if (s != sys) {
      sys = s;
      const int c0 = nsys > 1 ? root_beg[s] : info->level_beg[1];
      const int c1 = nsys > 1 ? root_beg[s + 1] : info->level_end[1];
      double M = 0, X = 0, Y = 0, Z = 0;
      for (int c = c0; c < c1; c++) {
        const double m = rec[c].m;
        M += m; X += m * rec[c].cx; Y += m * rec[c].cy; Z += m * rec[c].cz;
      }
      mtot = (float)M;
      cx = M > 0 ? (float)(X / M) : 0.f; cy = M > 0 ? (float)(Y / M) : 0.f; cz = M > 0 ? (float)(Z / M) : 0.f;
      hs = box[s].hsize;
      ns = nsys > 1 ? sys_off[s + 1] - sys_off[s] : n;
    }
    float mn[3] = {3e38f, 3e38f, 3e38f}, mx[3] = {-3e38f, -3e38f, -3e38f};
    float mg = 0.f, am = 0.f, al = 0.f, al2 = 0.f;
    for (int i = lane; i < np; i += 32) {
      const float4 p = ipos[pb + i];
      mn[0] = fminf(mn[0], p.x); mn[1] = fminf(mn[1], p.y); mn[2] = fminf(mn[2], p.z);
      mx[0] = fmaxf(mx[0], p.x); mx[1] = fmaxf(mx[1], p.y); mx[2] = fmaxf(mx[2], p.z);
      mg += p.w;
      if (have_prev) {
        const int k = pb + i;
        const int j = prev.perm ? __ldg(prev.perm + k) : k;
        const float4 a = BONSAI_IN_RANGE(j, n, 0x501) ? __ldg(prev.acc + j) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float m = sqrtf(a.x * a.x + a.y * a.y + a.z * a.z);
        const float lm = safe_log10(m);
        am += m; al += lm; al2 += lm * lm;
      }
    }
    for (int k = 0; k < 3; k++) { mn[k] = warp_min_f32(mn[k]); mx[k] = warp_max_f32(mx[k]); }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      mg += __shfl_xor_sync(kFull, mg, o);
      am += __shfl_xor_sync(kFull, am, o);
      al += __shfl_xor_sync(kFull, al, o);
      al2 += __shfl_xor_sync(kFull, al2, o);
    }
    const float gx = 0.5f * (mx[0] + mn[0]), gy = 0.5f * (mx[1] + mn[1]), gz = 0.5f * (mx[2] + mn[2]);
    const float sx = 0.5f * (mx[0] - mn[0]), sy = 0.5f * (mx[1] - mn[1]), sz = 0.5f * (mx[2] - mn[2]);
    const float rg = fmaxf(sqrtf(sx * sx + sy * sy + sz * sz), 1e-12f * hs);
    if (lane == 0) {
      const float dg = sqrtf((gx - cx) * (gx - cx) + (gy - cy) * (gy - cy) + (gz - cz) * (gz - cz));
      const int lvl = diff_level(ph_sorted[pb], ph_sorted[pb + np - 1]) - 1;  // common PH prefix (levels)
      const float vol = rg * rg * rg;
      // the previous evaluation: acceleration scale (floored at 1e-4 of the
      // system's M / hsize^2, so that a group at an exact balance point does not
      // open everything) and the statistics of the group that held the
      // group's middle particle
      const float afloor = 1e-4f * mtot / fmaxf(hs * hs, 1e-30f);
      float A = 0.f, spread = 0.f;
      float4 st = make_float4(0.f, 0.f, 0.f, 0.f);
      if (have_prev) {
        A = fmaxf(am / (float)np, afloor);
        const float mu = al / (float)np;
        spread = sqrtf(fmaxf(al2 / (float)np - mu * mu, 0.f));
        const int k = pb + np / 2;
        const int j = prev.perm ? __ldg(prev.perm + k) : k;
        if (prev.acc_valid[1] && BONSAI_IN_RANGE(j, n, 0x502)) {
          const int og = __ldg(prev.part_gid + j);
          if (og >= 0 && og < prev.stats_cap) st = __ldg(prev.stats + og);
        }
      }
      amag[g] = A;
      float f[kF];
      f[0] = (float)np / (float)ncrit;                               // group size
      f[1] = safe_log10(rg / hs) / 6.f;                              // radius
      f[2] = (float)min(lvl, kMaxLevel) / (float)kMaxLevel;          // tree depth
      f[3] = safe_log10(dg / hs + 1e-7f) / 6.f;                      // distance from the system's centre
      f[4] = safe_log10(mg / fmaxf(mtot, 1e-30f)) / 8.f;             // mass share
      f[5] = safe_log10((float)np / vol * hs * hs * hs / (float)ns) / 8.f;  // density
      f[6] = sx / rg; f[7] = sy / rg; f[8] = sz / rg;                // shape
      f[9] = log10f((float)ns) / 8.f;                                // system size
      f[10] = safe_log10(fmaxf(eps, 1e-12f) / rg) / 3.f;             // softening / radius
      f[11] = have_prev ? safe_log10(A * hs * hs / fmaxf(mtot, 1e-30f)) / 3.f : 0.f;  // acceleration scale
      f[12] = spread;                                                // its spread (dex)
      f[13] = log10f(1.0f + st.x) / 4.f;                             // cells near the opening boundary
      f[14] = st.y;                                                  // accepted mass near it
      f[15] = have_prev ? safe_log10(st.z + 1e-12f) / 3.f : 0.f;     // quadrupole norm of accepted cells
      // degenerate groups (a one-particle system's box and radius are floored
      // near 1e-12, so the density's float products under- and overflow) give
      // inf or NaN; the features are normalised logs well inside [-10, 10], and
      // fmaxf returns its other operand for a NaN
      float* o = feat + (size_t)g * kF;
#pragma unroll
      for (int k = 0; k < kF; k++) o[k] = fminf(fmaxf(f[k], -10.0f), 10.0f);
    }
  }
}

// ---------------------------------------------------------------------------
// Inference: FP16 weights in shared memory, FP32 accumulation; one warp per
// group (lane holds hidden units lane and lane+32) writes 1/theta_g.  W1 and
// W2 are staged transposed (input-major), so that the 32 lanes of a step read
// 32 consecutive weights: row-major, lane j's row starts j * 128 bytes apart
// and every lane of the warp hits the same bank.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_mlp_infer(const float* __restrict__ feat, const __half* __restrict__ wh,
                                                   const TreeInfo* __restrict__ info, float lo, float hi,
                                                   const float* __restrict__ amag, const int* __restrict__ acc_valid,
                                                   float inv_bound, float inv_fixed, float start_alpha,
                                                   float* __restrict__ group_inv_theta, float* __restrict__ group_tau) {
  __shared__ __half sw[kMlpWeights + 1];
  __shared__ float sh[8][kH];
  for (int t = threadIdx.x; t < kMlpWeights; t += blockDim.x) {
    int d = t;
    if (t < oB1) d = oW1 + (t % kF) * kH + t / kF;                          // W1[j][k] -> [k][j]
    else if (t >= oW2 && t < oB2) d = oW2 + ((t - oW2) % kH) * kH + (t - oW2) / kH;  // W2[j][i] -> [i][j]
    sw[d] = wh[t];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  const int ng = info->ngroups;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  for (int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < ng; g += nw) {
    const float xk = lane < kF ? feat[(size_t)g * kF + lane] : 0.f;
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int j = lane + 32 * u;
      float a = __half2float(sw[oB1 + j]);
#pragma unroll
      for (int k = 0; k < kF; k++) a = fmaf(__half2float(sw[oW1 + k * kH + j]), __shfl_sync(kFull, xk, k), a);
      sh[wi][j] = tanhf(a);
    }
    __syncwarp();
    float z = 0.f;
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const int j = lane + 32 * u;
      float a = __half2float(sw[oB2 + j]);
#pragma unroll 8
      for (int i = 0; i < kH; i++) a = fmaf(__half2float(sw[oW2 + i * kH + j]), sh[wi][i], a);
      z = fmaf(__half2float(sw[oW3 + j]), tanhf(a), z);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) z += __shfl_xor_sync(kFull, z, o);
    z += __half2float(sw[oB3]);
    if (lane == 0) {
      if (acc_valid[0] && acc_valid[1] != 2) {
        // the previous walk was not a relative walk with statistics (the
        // fixed-angle fallback, or another theta mode): the network never
        // saw such statistics in training, so one evaluation takes the
        // single-parameter bound, the relative walk the training tables were
        // recorded after (after the fallback, the network's own bounds
        // overshot the error target by ~2x in this evaluation)
        group_tau[g] = start_alpha * amag[g];
        group_inv_theta[g] = inv_bound;
      } else if (acc_valid[0]) {
        const float y = lo + (hi - lo) / (1.0f + expf(-z));
        group_tau[g] = amag[g] * exp10f(y);
        group_inv_theta[g] = inv_bound;
      } else {  // no previous accelerations: the fixed angle
        group_tau[g] = 0.0f;
        group_inv_theta[g] = inv_fixed;
      }
    }
    __syncwarp();
  }
}

__global__ void k_relative_tau(const TreeInfo* __restrict__ info, const float* __restrict__ amag,
                               const int* __restrict__ acc_valid, float alpha, float inv_bound, float inv_fixed,
                               float* __restrict__ inv, float* __restrict__ tau) {
  const int ng = info->ngroups;
  const bool v = *acc_valid != 0;
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < ng; g += gridDim.x * blockDim.x) {
    tau[g] = v ? alpha * amag[g] : 0.0f;
    inv[g] = v ? inv_bound : inv_fixed;
  }
}

__global__ void k_weights_to_half(const float* __restrict__ w, __half* __restrict__ wh) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < kMlpWeights; t += gridDim.x * blockDim.x)
    wh[t] = __float2half_rn(w[t]);
}

__global__ void k_fill_inv_theta(const TreeInfo* __restrict__ info, const float* __restrict__ theta, float c,
                                 float* __restrict__ inv) {
  const int ng = info->ngroups;
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < ng; g += gridDim.x * blockDim.x)
    inv[g] = 1.0f / (theta ? theta[g] : c);
}

// ---------------------------------------------------------------------------
// Training.  Loss per sample: 0.5 (theta - y)^2 (1 + over [theta > y]), mean
// over the S samples (over-prediction costs accuracy, so it is weighted).
//
// k_mlp_epoch: one launch takes every sample forward and back and leaves one
// partial gradient per block.  A block of 512 threads works on 64 samples at
// a time: the three layer products and the two weight-gradient products are
// register-tiled (2 samples x 4 units per thread; the 64 x 64 gradient as
// 4 x 4 weights per thread, each half of the block taking 32 of the samples),
// their operands in shared memory, two products per FFMA2.  The gradient
// tiles stay in registers over all of the block's tiles.  k_mlp_fold then
// adds the blocks' partials in block order and takes the Adam step in the
// same launch, so an epoch is two launches and every sum has a fixed order.
// All of it is FP32.  64 samples per block give 128 blocks at S = 8192 (one
// wave on 148 SMs); more per block would leave SMs idle.  Bound by the one
// tile's own chain (weights staged, three products, tanh, gradients) at that
// size: 16.2 us, and 3.0 us for the fold (one B200).  The form it replaced kept
// activations in global memory, one warp per sample, and summed each weight's
// gradient by one thread's serial loop over its samples: 27 + 67 + 2.3 + 1.9
// us an epoch.  100 epochs through the entry point: 13.0 -> 3.2 ms.
// ---------------------------------------------------------------------------
constexpr int kTS = 64;             // samples per tile
constexpr int kEpochThreads = 512;
constexpr int kRow = kH + 4;        // padded row of a 64-wide tile (16-byte aligned, rows on other banks)
constexpr int kXRow = kF + 4;
// shared memory, in floats: W1 and W2 input-major for the forward products,
// W2 as it is for the backward one, biases and w3; then the tile's x, h1, d2,
// d1 (after the last tile the same space folds the gradients)
// (transposed rows padded, so that the strided writes fall on 8 banks, not one)
constexpr int sW1t = 0, sW2t = sW1t + kF * kRow, sW2 = sW2t + kH * kRow, sB1 = sW2 + kH * kH, sB2 = sB1 + kH,
              sW3 = sB2 + kH, sX = sW3 + kH, sH1 = sX + kTS * kXRow, sD2 = sH1 + kTS * kRow,
              sD1 = sD2 + kTS * kRow, kEpochFloats = sD1 + kTS * kRow;

__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4& v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float comp(const float4& v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }

// acc[u] (u = sample, 4 units as two pairs) += sum_k a[s + u][k] * w[k][4 units]
template <int K, int WROW>
__device__ __forceinline__ void tile_product(const float* a, int arow, const float* w, float2 (&acc)[2][2]) {
#pragma unroll 4
  for (int k0 = 0; k0 < K; k0 += 4) {
    const float4 a0 = *reinterpret_cast<const float4*>(a + k0);
    const float4 a1 = *reinterpret_cast<const float4*>(a + arow + k0);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float4 v = *reinterpret_cast<const float4*>(w + (k0 + k) * WROW);
      acc[0][0] = __ffma2_rn(dup2(comp(a0, k)), lo2(v), acc[0][0]);
      acc[0][1] = __ffma2_rn(dup2(comp(a0, k)), hi2(v), acc[0][1]);
      acc[1][0] = __ffma2_rn(dup2(comp(a1, k)), lo2(v), acc[1][0]);
      acc[1][1] = __ffma2_rn(dup2(comp(a1, k)), hi2(v), acc[1][1]);
    }
  }
}

// BACK: with gradients (y and part given); otherwise the prediction alone
template <bool BACK>
__global__ void __launch_bounds__(kEpochThreads, 1)
    k_mlp_epoch(const float* __restrict__ X, const float* __restrict__ y, int S, const float* __restrict__ w,
                float lo, float hi, float over, float* __restrict__ part, float* __restrict__ loss,
                float* __restrict__ pred) {
  extern __shared__ float4 smem4[];
  float* sm = reinterpret_cast<float*>(smem4);
  const int t = threadIdx.x;
  for (int i = t; i < kH * kF; i += kEpochThreads) sm[sW1t + (i % kF) * kRow + i / kF] = w[oW1 + i];
  for (int i = t; i < kH * kH; i += kEpochThreads) {
    const float v = w[oW2 + i];
    sm[sW2 + i] = v;
    sm[sW2t + (i % kH) * kRow + i / kH] = v;
  }
  if (t < kH) { sm[sB1 + t] = w[oB1 + t]; sm[sB2 + t] = w[oB2 + t]; sm[sW3 + t] = w[oW3 + t]; }
  const float b3 = w[oB3];
  const int u0 = (t & 15) * 4;   // this thread's 4 hidden units in the layer products
  const int r0 = (t >> 4) * 2;   // and its 2 samples of the tile
  // gradient tiles: W2[j0 .. j0+3][i0 .. i0+3] and W1[t1 / 4][4 * (t1 & 3) ..] over the samples of this half
  const int half = t >> 8, t1 = t & 255;
  const int j0 = (t1 >> 4) * 4, i0 = (t1 & 15) * 4;
  float2 g2[4][2], g1[2];
  float gb1[4], gb2[4], gw3[4], gb3 = 0.f;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    g2[q][0] = g2[q][1] = dup2(0.f);
    gb1[q] = gb2[q] = gw3[q] = 0.f;
  }
  g1[0] = g1[1] = dup2(0.f);
  __syncthreads();
  for (int s0 = blockIdx.x * kTS; s0 < S; s0 += gridDim.x * kTS) {
    if (t < kTS * kF / 4) {
      const int r = t >> 2, k = (t & 3) * 4;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (s0 + r < S) v = __ldg(reinterpret_cast<const float4*>(X + (size_t)(s0 + r) * kF + k));
      *reinterpret_cast<float4*>(sm + sX + r * kXRow + k) = v;
    }
    __syncthreads();
    // layer 1
    float2 a[2][2];
    const float4 bb1 = *reinterpret_cast<const float4*>(sm + sB1 + u0);
#pragma unroll
    for (int u = 0; u < 2; u++) { a[u][0] = lo2(bb1); a[u][1] = hi2(bb1); }
    tile_product<kF, kRow>(sm + sX + r0 * kXRow, kXRow, sm + sW1t + u0, a);
    float h1[2][4];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      h1[u][0] = tanhf(a[u][0].x); h1[u][1] = tanhf(a[u][0].y);
      h1[u][2] = tanhf(a[u][1].x); h1[u][3] = tanhf(a[u][1].y);
      *reinterpret_cast<float4*>(sm + sH1 + (r0 + u) * kRow + u0) =
          make_float4(h1[u][0], h1[u][1], h1[u][2], h1[u][3]);
    }
    __syncwarp();  // a sample's 64 units belong to 16 lanes of one warp
    // layer 2
    const float4 bb2 = *reinterpret_cast<const float4*>(sm + sB2 + u0);
#pragma unroll
    for (int u = 0; u < 2; u++) { a[u][0] = lo2(bb2); a[u][1] = hi2(bb2); }
    tile_product<kH, kRow>(sm + sH1 + r0 * kRow, kRow, sm + sW2t + u0, a);
    const float4 w3 = *reinterpret_cast<const float4*>(sm + sW3 + u0);
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const float h2[4] = {tanhf(a[u][0].x), tanhf(a[u][0].y), tanhf(a[u][1].x), tanhf(a[u][1].y)};
      float z = fmaf(w3.w, h2[3], fmaf(w3.z, h2[2], fmaf(w3.y, h2[1], w3.x * h2[0])));
#pragma unroll
      for (int o = 8; o; o >>= 1) z += __shfl_xor_sync(kFull, z, o);
      z += b3;
      const int s = s0 + r0 + u;
      const bool live = s < S;
      const float sg = 1.0f / (1.0f + expf(-z));
      const float th = lo + (hi - lo) * sg;
      if (BACK) {
        const float e = live ? th - y[s] : 0.f;
        const float wgt = e > 0.f ? 1.0f + over : 1.0f;
        // d(mean loss)/dz; 0 past the last sample
        const float gz = live ? e * wgt * (hi - lo) * sg * (1.0f - sg) / (float)S : 0.f;
        const float wv[4] = {w3.x, w3.y, w3.z, w3.w};
        float d2[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          d2[q] = gz * wv[q] * (1.0f - h2[q] * h2[q]);
          gw3[q] = fmaf(gz, h2[q], gw3[q]);
          gb2[q] += d2[q];
        }
        *reinterpret_cast<float4*>(sm + sD2 + (r0 + u) * kRow + u0) = make_float4(d2[0], d2[1], d2[2], d2[3]);
        if (u0 == 0) {
          gb3 += gz;
          if (live) loss[s] = 0.5f * e * e * wgt;
        }
      } else if (u0 == 0 && live) {
        pred[s] = th;
      }
    }
    if (BACK) {
      __syncwarp();
      a[0][0] = a[0][1] = a[1][0] = a[1][1] = dup2(0.f);
      tile_product<kH, kH>(sm + sD2 + r0 * kRow, kRow, sm + sW2 + u0, a);
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const float v[4] = {a[u][0].x, a[u][0].y, a[u][1].x, a[u][1].y};
        float d1[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          d1[q] = v[q] * (1.0f - h1[u][q] * h1[u][q]);
          gb1[q] += d1[q];
        }
        *reinterpret_cast<float4*>(sm + sD1 + (r0 + u) * kRow + u0) = make_float4(d1[0], d1[1], d1[2], d1[3]);
      }
      __syncthreads();
#pragma unroll 4
      for (int r = half * (kTS / 2); r < (half + 1) * (kTS / 2); r++) {
        const float4 d = *reinterpret_cast<const float4*>(sm + sD2 + r * kRow + j0);
        const float4 h = *reinterpret_cast<const float4*>(sm + sH1 + r * kRow + i0);
#pragma unroll
        for (int q = 0; q < 4; q++) {
          g2[q][0] = __ffma2_rn(dup2(comp(d, q)), lo2(h), g2[q][0]);
          g2[q][1] = __ffma2_rn(dup2(comp(d, q)), hi2(h), g2[q][1]);
        }
        const float e = sm[sD1 + r * kRow + (t1 >> 2)];
        const float4 x = *reinterpret_cast<const float4*>(sm + sX + r * kXRow + (t1 & 3) * 4);
        g1[0] = __ffma2_rn(dup2(e), lo2(x), g1[0]);
        g1[1] = __ffma2_rn(dup2(e), hi2(x), g1[1]);
      }
    }
    __syncthreads();  // the tile's space is free for the next one
  }
  if (!BACK) return;
  // the two halves' weight tiles added (second half through shared memory)
  float* out = part + (size_t)blockIdx.x * kMlpWeights;
  float* f2 = sm + sH1;
  float* f1 = f2 + kH * kH;
  if (half == 1) {
#pragma unroll
    for (int q = 0; q < 4; q++)
      *reinterpret_cast<float4*>(f2 + (j0 + q) * kH + i0) = make_float4(g2[q][0].x, g2[q][0].y, g2[q][1].x, g2[q][1].y);
    *reinterpret_cast<float4*>(f1 + 4 * t1) = make_float4(g1[0].x, g1[0].y, g1[1].x, g1[1].y);
  }
  __syncthreads();
  if (half == 0) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float4 v = *reinterpret_cast<const float4*>(f2 + (j0 + q) * kH + i0);
      float* o = out + oW2 + (j0 + q) * kH + i0;
      o[0] = g2[q][0].x + v.x; o[1] = g2[q][0].y + v.y; o[2] = g2[q][1].x + v.z; o[3] = g2[q][1].y + v.w;
    }
    const float4 v = *reinterpret_cast<const float4*>(f1 + 4 * t1);
    float* o = out + oW1 + 4 * t1;
    o[0] = g1[0].x + v.x; o[1] = g1[0].y + v.y; o[2] = g1[1].x + v.z; o[3] = g1[1].y + v.w;
  }
  __syncthreads();
  // biases and w3: the 32 sample rows of each unit, in order
  float* fb = sm + sH1;  // [3][32][kH], then [32]
  const int row = t >> 4;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    fb[(0 * 32 + row) * kH + u0 + q] = gb1[q];
    fb[(1 * 32 + row) * kH + u0 + q] = gb2[q];
    fb[(2 * 32 + row) * kH + u0 + q] = gw3[q];
  }
  if (u0 == 0) fb[3 * 32 * kH + row] = gb3;
  __syncthreads();
  if (t < 3 * kH) {
    float acc = 0.f;
    for (int r = 0; r < 32; r++) acc += fb[((t / kH) * 32 + r) * kH + t % kH];
    out[(t < kH ? oB1 : t < 2 * kH ? oB2 : oW3) + t % kH] = acc;
  } else if (t == 3 * kH) {
    float acc = 0.f;
    for (int r = 0; r < 32; r++) acc += fb[3 * 32 * kH + r];
    out[oB3] = acc;
  }
}

// The blocks' partial gradients added in a fixed order (8 runs of blocks per
// weight, then the runs), then Adam on the same weight (m non-null), or the
// gradient itself.
__global__ void __launch_bounds__(256) k_mlp_fold(const float* __restrict__ part, int nb, float* __restrict__ grad,
                                                  float* __restrict__ w, float* __restrict__ m,
                                                  float* __restrict__ v, float lr, float b1, float b2, float c1,
                                                  float c2) {
  __shared__ float sh[8][32];
  const int lane = threadIdx.x & 31, run = threadIdx.x >> 5;
  const int t = blockIdx.x * 32 + lane;
  float acc = 0.f;
  if (t < kMlpWeights) {
    const int b = nb * run / 8, e = nb * (run + 1) / 8;
#pragma unroll 8
    for (int k = b; k < e; k++) acc += part[(size_t)k * kMlpWeights + t];
  }
  sh[run][lane] = acc;
  __syncthreads();
  if (run || t >= kMlpWeights) return;
  float g = 0.f;
#pragma unroll
  for (int q = 0; q < 8; q++) g += sh[q][lane];
  if (grad) grad[t] = g;
  if (!m) return;
  const float mt = b1 * m[t] + (1.f - b1) * g;
  const float vt = b2 * v[t] + (1.f - b2) * g * g;
  m[t] = mt;
  v[t] = vt;
  w[t] -= lr * (mt / c1) / (sqrtf(vt / c2) + 1e-8f);
}

__global__ void k_sum_f(const float* __restrict__ a, int S, double* __restrict__ out) {
  // one block: fixed-order partials, then lane 0 folds them
  __shared__ double sh[256];
  double s = 0;
  for (int i = threadIdx.x; i < S; i += blockDim.x) s += a[i];
  sh[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int i = 0; i < (int)blockDim.x; i++) t += sh[i];
    *out = t;
  }
}

// at most one block per SM of a 148-SM device: past that a block takes several
// tiles, so that the partial gradients stay few
constexpr int kEpochBlocks = 148;
static int epoch_blocks(int S) {
  const int tiles = (S + kTS - 1) / kTS;
  return tiles < kEpochBlocks ? tiles : kEpochBlocks;
}
// the kernel's shared memory exceeds the default limit
template <bool BACK>
static void launch_epoch(const float* X, const float* y, int S, const float* w, float lo, float hi, float over,
                         float* part, float* loss, float* pred, cudaStream_t st) {
  constexpr int bytes = kEpochFloats * (int)sizeof(float);
  cudaFuncSetAttribute(k_mlp_epoch<BACK>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  k_mlp_epoch<BACK><<<epoch_blocks(S), kEpochThreads, bytes, st>>>(X, y, S, w, lo, hi, over, part, loss, pred);
}

// scratch for training: loss (S), the blocks' partial gradients
size_t mlp_train_scratch_floats(int S) { return (size_t)S + (size_t)epoch_blocks(S) * kMlpWeights; }

void mlp_loss_grad(const float* X, const float* y, int S, const float* w, float lo, float hi, float over,
                   float* scratch, float* grad, double* loss_out, cudaStream_t st) {
  float* part = scratch + S;
  launch_epoch<true>(X, y, S, w, lo, hi, over, part, scratch, nullptr, st);
  k_mlp_fold<<<(kMlpWeights + 31) / 32, 256, 0, st>>>(part, epoch_blocks(S), grad, nullptr, nullptr, nullptr, 0.f,
                                                      0.f, 0.f, 1.f, 1.f);
  if (loss_out) k_sum_f<<<1, 256, 0, st>>>(scratch, S, loss_out);
}

void mlp_train_epoch(const float* X, const float* y, int S, float* w, float lo, float hi, float over, float* scratch,
                     float* m, float* v, float lr, int step, cudaStream_t st) {
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  float* part = scratch + S;
  launch_epoch<true>(X, y, S, w, lo, hi, over, part, scratch, nullptr, st);
  k_mlp_fold<<<(kMlpWeights + 31) / 32, 256, 0, st>>>(part, epoch_blocks(S), nullptr, w, m, v, lr, b1, b2, c1, c2);
}

void mlp_predict(const float* X, int S, const float* w, float lo, float hi, float* pred, cudaStream_t st) {
  launch_epoch<false>(X, nullptr, S, w, lo, hi, 0.f, nullptr, nullptr, pred, st);
}

void launch_group_features(const int2* groups, const TreeInfo* info, const float4* ipos,
                           const unsigned long long* ph_sorted, const MpRec* rec, const Box* box, int n, int ncrit,
                           float eps, float* feat, const int* sys_off, int nsys, const int* root_beg,
                           const PrevEval& prev, float* amag, int nblocks, cudaStream_t st) {
  k_group_features<<<nblocks, 256, 0, st>>>(groups, info, ipos, ph_sorted, rec, box, n, ncrit, eps, feat, sys_off,
                                            nsys, root_beg, prev, amag);
}

void launch_mlp_infer(const float* feat, const void* wh, const TreeInfo* info, float lo, float hi, const float* amag,
                      const int* acc_valid, float inv_bound, float inv_fixed, float start_alpha, float* inv, float* tau,
                      int nblocks, cudaStream_t st) {
  k_mlp_infer<<<nblocks, 256, 0, st>>>(feat, static_cast<const __half*>(wh), info, lo, hi, amag, acc_valid,
                                       inv_bound, inv_fixed, start_alpha, inv, tau);
}

void launch_relative_tau(const TreeInfo* info, const float* amag, const int* acc_valid, float alpha, float inv_bound,
                         float inv_fixed, float* inv, float* tau, int nblocks, cudaStream_t st) {
  k_relative_tau<<<nblocks, 256, 0, st>>>(info, amag, acc_valid, alpha, inv_bound, inv_fixed, inv, tau);
}

void launch_weights_to_half(const float* w, void* wh, cudaStream_t st) {
  k_weights_to_half<<<(kMlpWeights + 255) / 256, 256, 0, st>>>(w, static_cast<__half*>(wh));
}

void launch_fill_inv_theta(const TreeInfo* info, const float* theta, float c, float* inv, int nblocks,
                           cudaStream_t st) {
  k_fill_inv_theta<<<nblocks, 256, 0, st>>>(info, theta, c, inv);
}

BONSAI_BOUNDS_ACCESSOR(bounds_word_learned)

}  // namespace bonsai
