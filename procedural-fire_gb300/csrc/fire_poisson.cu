// Standalone pressure Poisson solver: the step's multigrid (src/sim.js:415-495, 576-599) iterated to a
// relative-residual tolerance, in the plain FP32 form or as mixed-precision iterative refinement.
//
// Mixed-precision form (FIRE_POISSON_FP16 / FIRE_POISSON_BF16):
//   x, b and every residual are FP32; the correction equation A e = r is solved approximately by V(2,2)
//   cycles whose level arrays (p and b of every level above the on-chip coarse end) are stored in IEEE half
//   or bfloat16, with all arithmetic in FP32 registers.  Halving the bytes of the fine levels is the point:
//   at 256x512x256 the level-0 arrays of the FP32 form (268 MB) do not fit the 129 MB L2 and every sweep is
//   HBM-bound.  The residual handed to the correction solve is scaled by 1/RMS of the previous residual, so
//   it stays O(1) inside half's range; the scale is undone when the correction is added.  The coarsest
//   level is solved in FP64 (64 red-black sweeps on a double copy in shared memory).
// Loop on the device:
//   pre:   ||b||^2  -> scale 1/RMS(b);  r0 = b - A x0 (written scaled into the level-0 RHS);  test
//   WHILE: V-cycle(s) on (e, r~);  x += e * unscale;  r = b - A x (written scaled);  test
// where each test is one small kernel that sums the residual partials in a fixed order (double-float),
// updates the scales and sets the conditional node's value.  The FP32 form runs the step's own V-cycle on
// (x, b) with the same pre-pass and test.
// The cycles run the step's kernels on the storage types: two sweeps per pass (fire_sweep.cu; each value is rounded to the
// storage type where a colour launch would have stored it), marched transfers (fire_level.cuh), the coarse kernel.  All
// levels are in the plain layout: with one pass per two sweeps a red-black split saves no bytes, and plain pairs serve every
// kernel.  Measured (GB300, whole solves, colour launches on a split level 0 -> this): 256x512x256 with FP32 storage 7.20 ->
// 4.67 ms, 128x256x128 with half 1.38 -> 1.04 ms; FP32 form at 64x64x64 296 -> 285 us.
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <cmath>
#include <cstring>
#include <algorithm>
#include <string>
#include <vector>

#include "../../include/fire_sim.h"
#include "fire_internal.h"
#include "fire_device.cuh"
#include "fire_launch.cuh"
#include "fire_level.cuh"
#include "fire_nvtx.h"

namespace fire {
namespace {

// Loads widen to FP32, stores round to nearest.
template <typename T> __device__ __forceinline__ float ld(const T* p) { return Cells2<T>::one(*p); }
template <typename T> __device__ __forceinline__ void st(T* p, float v) { *p = Cells2<T>::back(v); }

constexpr int GX = 32, GY = 4, GZ = 2, NT = GX * GY * GZ;
constexpr int SMZ = 2;   // cells of one colour per smoother thread (as the step's smoother)
constexpr int RZ = 8;    // z-planes per residual thread
constexpr int SUMSQ_CTAS = 1024;
constexpr int COARSE64_SWEEPS = 64;

// Red-black sweep of one colour (mgSmooth, src/sim.js:417-437) on T storage, for levels the two-sweep kernel does not take.  zero_nbrs:
// the level's current values are taken as zero (the first half-sweep of a correction solve from e = 0: the
// colour being updated never reads its own old value, so the other colour's stale contents are not read).
template <typename T>
__global__ void __launch_bounds__(NT) k_psmooth(T* __restrict__ p, const T* __restrict__ b, int nx, int ny, int nz, float h, int color,
                                                int zero_nbrs) {
  pdl_wait();
  pdl_trigger();
  const int gx = blockIdx.x * GX + threadIdx.x, y = blockIdx.y * GY + threadIdx.y;
  const int zb = (blockIdx.z * GZ + threadIdx.z) * SMZ;
  if (y >= ny) return;
  const float h2 = h * h;
  const int sy = nx, sz = nx * ny;
  float v[SMZ];
#pragma unroll
  for (int k = 0; k < SMZ; ++k) {
    const int z = zb + k;
    const int x = gx * 2 + ((y + z + color) & 1);
    if (z < nz && x < nx) {
      const int c = x + y * sy + z * sz;
      float sum = 0.0f, diag = 6.0f;
      const bool rd = !zero_nbrs;
      if (x > 0) { if (rd) sum += ld(p + c - 1); } else diag += 1.0f;
      if (x < nx - 1) { if (rd) sum += ld(p + c + 1); } else diag += 1.0f;
      if (z > 0) { if (rd) sum += ld(p + c - sz); } else diag += 1.0f;
      if (z < nz - 1) { if (rd) sum += ld(p + c + sz); } else diag += 1.0f;
      if (y > 0) { if (rd) sum += ld(p + c - sy); } else diag -= 1.0f;
      if (y < ny - 1) { if (rd) sum += ld(p + c + sy); } else diag += 1.0f;
      v[k] = __fdividef(sum - h2 * ld(b + c), diag);
    }
  }
#pragma unroll
  for (int k = 0; k < SMZ; ++k) {
    const int z = zb + k;
    const int x = gx * 2 + ((y + z + color) & 1);
    if (z < nz && x < nx) st(p + x + sy * y + sz * z, v[k]);
  }
}
// The transfers between levels of any two storage types (fire_level.cuh).
template <typename TF, typename TC>
__global__ void __launch_bounds__(NT) k_prestrict(const TF* __restrict__ p, const TF* __restrict__ b, int nx, int ny, int nz, float h,
                                                  TC* __restrict__ bc, TC* __restrict__ pc) {
  restrict_march<1, true>(p, b, nx, ny, nz, h, bc, pc, blockIdx);
}
template <int kDepth, typename TF, typename TC>
__global__ void __launch_bounds__(NT) k_pprolong(TF* __restrict__ p, const TC* __restrict__ pc, int nx, int ny, int nz) {
  prolong_march<kDepth, true, false>(p, pc, nx, ny, nz, blockIdx);
}

// Solver state on the device.
struct PState {
  double bb;        // ||b||^2
  double rel;       // last relative residual
  double rel0;      // relative residual before the first cycle
  int iters;        // cycles / refinement steps of this solve
  int pad;
  float sc[2];      // sc[0]: unscale of the correction being solved for; sc[1]: scale of the next residual
};

// Writes the CTA's (x, y, z, w) partial (df64 pairs (rr, bb)) into slot `slot`.
__device__ __forceinline__ void cta_partial(df64 rr, df64 bb, float4* partials, int slot) {
  __shared__ df64 sr[NT / 32], sb[NT / 32];
  const int tid = threadIdx.x + GX * (threadIdx.y + GY * threadIdx.z);
  rr = df_warp_sum(rr);
  bb = df_warp_sum(bb);
  if ((tid & 31) == 0) { sr[tid >> 5] = rr; sb[tid >> 5] = bb; }
  __syncthreads();
  if (tid < 32) {
    rr = tid < NT / 32 ? sr[tid] : df_make(0.0f);
    bb = tid < NT / 32 ? sb[tid] : df_make(0.0f);
    rr = df_warp_sum(rr);
    bb = df_warp_sum(bb);
    if (tid == 0) partials[slot] = make_float4(rr.hi, rr.lo, bb.hi, bb.lo);
  }
}

// ||b||^2 partials over a fixed grid of SUMSQ_CTAS CTAs (grid-stride), deterministic.
__global__ void __launch_bounds__(NT) k_sumsq(const float* __restrict__ b, long long n, float4* __restrict__ partials) {
  pdl_wait();
  pdl_trigger();
  const int tid = threadIdx.x + GX * (threadIdx.y + GY * threadIdx.z);
  float s = 0.0f;
  for (long long i = (long long)blockIdx.x * NT + tid; i < n; i += (long long)gridDim.x * NT) {
    const float v = __ldg(b + i);
    s += v * v;
  }
  cta_partial(df_make(0.0f), df_make(s), partials, blockIdx.x);
}

// Laplacian numerator of one cell written as a sum of neighbour differences, (nb - me) per face with the
// ghost rules (p = 0 faces: ghost - me = -2 me; floor: 0).  Each difference is correctly rounded relative to
// itself, so the sum carries no cancellation of the 6|p| scale against 6 p: the residual of a converged
// solution is computed to its own precision, not to eps |p| / h^2.
__device__ __forceinline__ float lap_diff(float me, float xm, float xp, float ym, float yp, float zm, float zp, bool hxm, bool hxp,
                                          bool hym, bool hyp, bool hzm, bool hzp) {
  const float d2 = -2.0f * me;
  return ((hxm ? xm - me : d2) + (hxp ? xp - me : d2)) + ((hym ? ym - me : 0.0f) + (hyp ? yp - me : d2)) +
         ((hzm ? zm - me : d2) + (hzp ? zp - me : d2));
}
// r = b - A (xh + xl) over RZ planes of column (x, y) (xl may be null); the residual scaled by sc[1] is stored
// into rT (if given).  Partials: (||r||^2, ||b||^2).
template <typename TR>
__global__ void __launch_bounds__(NT) k_pres(const float* __restrict__ xh, const float* __restrict__ xl, const float* __restrict__ b,
                                             TR* __restrict__ rT, const PState* __restrict__ ps, int nx, int ny, int nz, float ih2,
                                             float4* __restrict__ partials) {
  pdl_wait();
  pdl_trigger();
  const int x = blockIdx.x * GX + threadIdx.x, y = blockIdx.y * GY + threadIdx.y;
  const int z0 = (blockIdx.z * GZ + threadIdx.z) * RZ;
  float rr = 0.0f, bb = 0.0f;
  if (x < nx && y < ny && z0 < nz) {
    const float s = rT ? ps->sc[1] : 1.0f;
    const int sy = nx, sz = nx * ny;
    const bool hxm = x > 0, hxp = x < nx - 1, hym = y > 0, hyp = y < ny - 1;
    int t = x + sy * y + sz * z0;
    float prev = z0 > 0 ? __ldg(xh + t - sz) : 0.0f, cur = __ldg(xh + t);
    float lprev = 0.0f, lcur = 0.0f;
    if (xl) { lprev = z0 > 0 ? __ldg(xl + t - sz) : 0.0f; lcur = __ldg(xl + t); }
#pragma unroll
    for (int k = 0; k < RZ; ++k) {
      const int z = z0 + k;
      if (z < nz) {
        const bool hzm = z > 0, hzp = z + 1 < nz;
        const float next = hzp ? __ldg(xh + t + sz) : 0.0f;
        float d = lap_diff(cur, hxm ? __ldg(xh + t - 1) : 0.0f, hxp ? __ldg(xh + t + 1) : 0.0f, hym ? __ldg(xh + t - sy) : 0.0f,
                           hyp ? __ldg(xh + t + sy) : 0.0f, prev, next, hxm, hxp, hym, hyp, hzm, hzp);
        float lnext = 0.0f, dl = 0.0f;
        if (xl) {
          lnext = hzp ? __ldg(xl + t + sz) : 0.0f;
          dl = lap_diff(lcur, hxm ? __ldg(xl + t - 1) : 0.0f, hxp ? __ldg(xl + t + 1) : 0.0f, hym ? __ldg(xl + t - sy) : 0.0f,
                        hyp ? __ldg(xl + t + sy) : 0.0f, lprev, lnext, hxm, hxp, hym, hyp, hzm, hzp);
        }
        const float bv = __ldg(b + t);
        const float r = (bv - d * ih2) - dl * ih2;
        if (rT) st(rT + t, r * s);
        rr += r * r;
        bb += bv * bv;
        prev = cur; cur = next;
        lprev = lcur; lcur = lnext;
        t += sz;
      }
    }
  }
  cta_partial(df_make(rr), df_make(bb), partials, blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z));
}

// k_pres for even nx with one thread per x pair (2 gx, 2 gx + 1) and RZ planes: every load of xh, xl and b
// is a float2 (plus one scalar on each side for the x neighbours), and the two residuals are stored as a pair.
// kFull: nz is a multiple of the planes a CTA covers, so no plane test is needed inside the march.
template <typename TR, bool kFull>
__global__ void __launch_bounds__(NT) k_pres2(const float* __restrict__ xh, const float* __restrict__ xl, const float* __restrict__ b,
                                              TR* __restrict__ rT, const PState* __restrict__ ps, int nx, int ny, int nz, float ih2,
                                              float4* __restrict__ partials) {
  pdl_wait();
  pdl_trigger();
  const int hx = nx >> 1;
  const int gx = blockIdx.x * GX + threadIdx.x, y = blockIdx.y * GY + threadIdx.y;
  const int z0 = (blockIdx.z * GZ + threadIdx.z) * RZ;
  float rr = 0.0f, bb = 0.0f;
  if (gx < hx && y < ny && z0 < nz) {
    const float s = rT ? ps->sc[1] : 1.0f;
    const int sy = nx, sz = nx * ny;
    const bool hxm = gx > 0, hxp = gx < hx - 1, hym = y > 0, hyp = y < ny - 1;
    const float2 zero2 = make_float2(0.0f, 0.0f);
    auto ld2 = [](const float* q) { return __ldg(reinterpret_cast<const float2*>(q)); };
    int t = 2 * gx + sy * y + sz * z0;
    float2 hp = z0 > 0 ? ld2(xh + t - sz) : zero2, hc = ld2(xh + t);
    float2 lp = zero2, lc = zero2;
    if (xl) { lp = z0 > 0 ? ld2(xl + t - sz) : zero2; lc = ld2(xl + t); }
#pragma unroll
    for (int k = 0; k < RZ; ++k) {
      const int z = z0 + k;
      if (kFull || z < nz) {
        const bool hzm = z > 0, hzp = z + 1 < nz;
        const float2 hn = hzp ? ld2(xh + t + sz) : zero2;
        const float hl = hxm ? __ldg(xh + t - 1) : 0.0f, hr = hxp ? __ldg(xh + t + 2) : 0.0f;
        const float2 hym2 = hym ? ld2(xh + t - sy) : zero2, hyp2 = hyp ? ld2(xh + t + sy) : zero2;
        const float d0 = lap_diff(hc.x, hl, hc.y, hym2.x, hyp2.x, hp.x, hn.x, hxm, true, hym, hyp, hzm, hzp);
        const float d1 = lap_diff(hc.y, hc.x, hr, hym2.y, hyp2.y, hp.y, hn.y, true, hxp, hym, hyp, hzm, hzp);
        float dl0 = 0.0f, dl1 = 0.0f;
        float2 ln = zero2;
        if (xl) {
          ln = hzp ? ld2(xl + t + sz) : zero2;
          const float ll = hxm ? __ldg(xl + t - 1) : 0.0f, lr = hxp ? __ldg(xl + t + 2) : 0.0f;
          const float2 lym2 = hym ? ld2(xl + t - sy) : zero2, lyp2 = hyp ? ld2(xl + t + sy) : zero2;
          dl0 = lap_diff(lc.x, ll, lc.y, lym2.x, lyp2.x, lp.x, ln.x, hxm, true, hym, hyp, hzm, hzp);
          dl1 = lap_diff(lc.y, lc.x, lr, lym2.y, lyp2.y, lp.y, ln.y, true, hxp, hym, hyp, hzm, hzp);
        }
        const float2 bv = ld2(b + t);
        const float r0 = (bv.x - d0 * ih2) - dl0 * ih2, r1 = (bv.y - d1 * ih2) - dl1 * ih2;
        if (rT) st2<true>(rT + t, make_float2(r0 * s, r1 * s));
        rr += r0 * r0;
        rr += r1 * r1;
        bb += bv.x * bv.x;
        bb += bv.y * bv.y;
        hp = hc; hc = hn;
        lp = lc; lc = ln;
        t += sz;
      }
    }
  }
  cta_partial(df_make(rr), df_make(bb), partials, blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z));
}

// k_pres2 with four cells of a row per thread, for rows that fill whole warps of them: one 16-byte load where the pair form has two
// 8-byte ones, and the x neighbours of the four come from the neighbouring lanes, so a cell costs three quarters of the L1
// traffic and two thirds of the instructions.  Same arithmetic and order within a cell; the partials' cells are grouped differently.
// Measured (GB300, whole solves, pairs -> this): 256x512x256 with FP32 storage 4.99 -> 4.83 ms, 128x256x128 with half 1.043 -> 1.030.
template <typename TR>
__global__ void __launch_bounds__(NT) k_pres4(const float* __restrict__ xh, const float* __restrict__ xl, const float* __restrict__ b,
                                              TR* __restrict__ rT, const PState* __restrict__ ps, int nx, int ny, int nz, float ih2,
                                              float4* __restrict__ partials) {
  pdl_wait();
  pdl_trigger();
  const int gx = blockIdx.x * GX + threadIdx.x, y = blockIdx.y * GY + threadIdx.y;
  const int z0 = (blockIdx.z * GZ + threadIdx.z) * RZ;
  float rr = 0.0f, rr2 = 0.0f, bb = 0.0f, bb2 = 0.0f;   // as many cells in each FP32 sum as the pair form
  if (y < ny && z0 < nz) {   // uniform over a warp: its 32 lanes share y and z
    const float s = rT ? ps->sc[1] : 1.0f;
    const int sy = nx, sz = nx * ny;
    const bool hxm = gx > 0, hxp = gx < (nx >> 2) - 1, hym = y > 0, hyp = y < ny - 1;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto ld4 = [](const float* q) { return __ldg(reinterpret_cast<const float4*>(q)); };
    int t = 4 * gx + sy * y + sz * z0;
    float4 hp = z0 > 0 ? ld4(xh + t - sz) : zero, hc = ld4(xh + t), lp = zero, lc = zero;
    if (xl) { lp = z0 > 0 ? ld4(xl + t - sz) : zero; lc = ld4(xl + t); }
    const int lane = threadIdx.x;
    auto sides = [&](const float* q, float4 c, float& l, float& r) {
      l = __shfl_up_sync(0xffffffffu, c.w, 1);
      r = __shfl_down_sync(0xffffffffu, c.x, 1);
      if (lane == 0) l = hxm ? __ldg(q + t - 1) : 0.0f;
      if (lane == 31) r = hxp ? __ldg(q + t + 4) : 0.0f;
    };
    auto laps = [&](float4 c, float l, float r, float4 ym, float4 yp, float4 zm, float4 zp, bool hzm, bool hzp) {
      return make_float4(lap_diff(c.x, l, c.y, ym.x, yp.x, zm.x, zp.x, hxm, true, hym, hyp, hzm, hzp),
                         lap_diff(c.y, c.x, c.z, ym.y, yp.y, zm.y, zp.y, true, true, hym, hyp, hzm, hzp),
                         lap_diff(c.z, c.y, c.w, ym.z, yp.z, zm.z, zp.z, true, true, hym, hyp, hzm, hzp),
                         lap_diff(c.w, c.z, r, ym.w, yp.w, zm.w, zp.w, true, hxp, hym, hyp, hzm, hzp));
    };
#pragma unroll
    for (int k = 0; k < RZ; ++k) {
      const int z = z0 + k;
      if (z >= nz) break;
      const bool hzm = z > 0, hzp = z + 1 < nz;
      const float4 hn = hzp ? ld4(xh + t + sz) : zero, ln = xl && hzp ? ld4(xl + t + sz) : zero, bv = ld4(b + t);
      const float4 hym4 = hym ? ld4(xh + t - sy) : zero, hyp4 = hyp ? ld4(xh + t + sy) : zero;
      float l, r;
      sides(xh, hc, l, r);
      const float4 d = laps(hc, l, r, hym4, hyp4, hp, hn, hzm, hzp);
      float4 dl = zero;
      if (xl) {
        const float4 lym = hym ? ld4(xl + t - sy) : zero, lyp = hyp ? ld4(xl + t + sy) : zero;
        sides(xl, lc, l, r);
        dl = laps(lc, l, r, lym, lyp, lp, ln, hzm, hzp);
      }
      const float4 res = make_float4((bv.x - d.x * ih2) - dl.x * ih2, (bv.y - d.y * ih2) - dl.y * ih2, (bv.z - d.z * ih2) - dl.z * ih2,
                                     (bv.w - d.w * ih2) - dl.w * ih2);
      if (rT) {
        st2<true>(rT + t, make_float2(res.x * s, res.y * s));
        st2<true>(rT + t + 2, make_float2(res.z * s, res.w * s));
      }
      rr += res.x * res.x; rr += res.y * res.y; rr2 += res.z * res.z; rr2 += res.w * res.w;
      bb += bv.x * bv.x; bb += bv.y * bv.y; bb2 += bv.z * bv.z; bb2 += bv.w * bv.w;
      hp = hc; hc = hn;
      lp = lc; lc = ln;
      t += sz;
    }
  }
  cta_partial(df_add(df_make(rr), df_make(rr2)), df_add(df_make(bb), df_make(bb2)), partials, blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z));
}

// (xh, xl) += e * sc[0] as a double-float (FP32 pair) update: Knuth's TwoSum then renormalisation, so the
// pair keeps ~44 bits of the solution while every stored array stays FP32.  4 cells per thread.
__device__ __forceinline__ void pair_add(float& hi, float& lo, float d) {
  const float s = __fadd_rn(hi, d);
  const float bp = __fsub_rn(s, hi);
  const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(d, bp));
  const float l2 = __fadd_rn(lo, err);
  hi = __fadd_rn(s, l2);
  lo = __fsub_rn(l2, __fsub_rn(hi, s));
}
// One thread per x pair (2 gx, 2 gx + 1) of a row: the pair is one float2 of xh and xl and one pair of e.
template <typename TE>
__global__ void __launch_bounds__(NT) k_pupdate(float* __restrict__ xh, float* __restrict__ xl, const TE* __restrict__ e,
                                                const PState* __restrict__ ps, int nx, int ny, int nz) {
  pdl_wait();
  pdl_trigger();
  const int gx = blockIdx.x * GX + threadIdx.x, y = blockIdx.y * GY + threadIdx.y, z = blockIdx.z * GZ + threadIdx.z;
  const int x = 2 * gx;
  if (x >= nx || y >= ny || z >= nz) return;
  const float u = ps->sc[0];
  const int t = x + nx * (y + ny * z);
  if ((nx & 1) == 0) {
    float2 hv = *reinterpret_cast<const float2*>(xh + t);
    float2 lv = *reinterpret_cast<const float2*>(xl + t);
    const float2 ev = ld2<true>(e + t);
    pair_add(hv.x, lv.x, __fmul_rn(ev.x, u));
    pair_add(hv.y, lv.y, __fmul_rn(ev.y, u));
    *reinterpret_cast<float2*>(xh + t) = hv;
    *reinterpret_cast<float2*>(xl + t) = lv;
  } else {
    pair_add(xh[t], xl[t], __fmul_rn(ld(e + t), u));
    if (x + 1 < nx) pair_add(xh[t + 1], xl[t + 1], __fmul_rn(ld(e + t + 1), u));
  }
}

// mode 0: ||b||^2 from the sumsq partials; sets the first scale.  mode 1: the residual test (first = 1
// before the loop).  Sets the WHILE condition: continue while rel > tol and iters < max_iters.
__global__ void __launch_bounds__(NT) k_ptest(const float4* __restrict__ partials, int count, PState* __restrict__ ps, int mode, int first,
                                              double tol, int max_iters, double ncells, cudaGraphConditionalHandle h, int set_cond) {
  __shared__ df64 sa[SUMV / 32], sb[SUMV / 32];
  pdl_wait();
  pdl_trigger();
  df64 A, B;
  sum_pairs_fixed<NT>(partials, count, threadIdx.x, sa, sb, A, B);
  if (threadIdx.x != 0) return;
  if (mode == 0) {
    const double bb = df_to_double(B);
    ps->bb = bb;
    ps->sc[0] = 1.0f;
    ps->sc[1] = bb > 0.0 ? (float)(1.0 / sqrt(bb / ncells)) : 1.0f;
    return;
  }
  const double rr = df_to_double(A), bb = ps->bb;
  const double rel = bb > 0.0 ? sqrt(rr / bb) : 0.0;
  ps->rel = rel;
  if (first) { ps->rel0 = rel; ps->iters = 0; } else { ps->iters += 1; }
  ps->sc[0] = 1.0f / ps->sc[1];
  ps->sc[1] = rr > 0.0 ? (float)(1.0 / sqrt(rr / ncells)) : 1.0f;
  if (set_cond) cudaGraphSetConditional(h, (rel > tol && ps->iters < max_iters) ? 1u : 0u);
}

// ---- RHS: sum of Gaussian sources + per-cell normal noise, then the mean removed ----
constexpr int MAX_SOURCES = 256;
__global__ void __launch_bounds__(NT) k_rhs(float* __restrict__ b, int nx, int ny, int nz, const float* __restrict__ src, int ns, float noise,
                                            unsigned seed, float4* __restrict__ partials) {
  __shared__ float s[MAX_SOURCES * 5];
  const int tid = threadIdx.x + GX * (threadIdx.y + GY * threadIdx.z);
  for (int i = tid; i < ns * 5; i += NT) s[i] = src[i];
  __syncthreads();
  const int x = blockIdx.x * GX + threadIdx.x, y = blockIdx.y * GY + threadIdx.y, z = blockIdx.z * GZ + threadIdx.z;
  float v = 0.0f;
  if (x < nx && y < ny && z < nz) {
    const float px = (float)x + 0.5f, py = (float)y + 0.5f, pz = (float)z + 0.5f;
    for (int i = 0; i < ns; ++i) {
      const float dx = px - s[5 * i], dy = py - s[5 * i + 1], dz = pz - s[5 * i + 2], sg = s[5 * i + 3];
      v += s[5 * i + 4] * expf(-(dx * dx + dy * dy + dz * dz) / (2.0f * sg * sg));
    }
    const uint3 hv = pcg3d(make_uint3((unsigned)x, (unsigned)y, (unsigned)z ^ (seed * 0x9E3779B9u)));
    const float u1 = ((float)(hv.x >> 8) + 1.0f) * (1.0f / 16777216.0f);   // (0, 1]
    const float u2 = (float)(hv.y >> 8) * (1.0f / 16777216.0f);            // [0, 1)
    v += noise * sqrtf(-2.0f * logf(u1)) * cosf(6.283185307179586f * u2);
    b[x + nx * (y + ny * z)] = v;
  }
  cta_partial(df_make(0.0f), df_make(v), partials, blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z));
}
__global__ void __launch_bounds__(NT) k_mean(const float4* __restrict__ partials, int count, double ncells, double* __restrict__ mean) {
  __shared__ df64 sa[SUMV / 32], sb[SUMV / 32];
  df64 A, B;
  sum_pairs_fixed<NT>(partials, count, threadIdx.x, sa, sb, A, B);
  if (threadIdx.x == 0) mean[0] = df_to_double(B) / ncells;
}
__global__ void k_sub_mean(float* __restrict__ b, long long n, const double* __restrict__ mean) {
  const float m = (float)mean[0];
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) b[i] -= m;
}

dim3 grid3(int x, int y, int z) { return dim3((x + GX - 1) / GX, (y + GY - 1) / GY, (z + GZ - 1) / GZ); }
const dim3 kBlock(GX, GY, GZ);

}  // namespace
}  // namespace fire

using namespace fire;

// Storage type of a level's arrays.
enum { STO_F32 = 0, STO_F16 = 1, STO_BF16 = 2 };
// One level of the refinement: storage type and device arrays; p2 and sweep as in MGLevel.
struct PLevel {
  int nx, ny, nz;
  float h;
  int sto;
  void* p;
  void* b;
  void* p2;
  SweepPlan sweep;
};

struct FirePoisson {
  int device = 0;
  int res[3] = {0, 0, 0};
  float h = 0;
  int prec = FIRE_POISSON_FP32;
  bool ir = false;              // iterative refinement (every form but FIRE_POISSON_FP32)
  long long cells = 0;
  std::vector<PLevel> levels;
  std::vector<MGLevel> mg;      // float view (levels >= tailFirst are FP32; all levels in the FP32 form)
  int tailFirst = 0;
  bool coarse = false;          // levels [tailFirst, n) run in the register-resident coarse kernel, else in the tail kernel
  int coarseIters = 8;
  void* arena = nullptr;
  float4* partials = nullptr;
  int partialsCount = 0;
  PState* state = nullptr;      // the solve's
  PState* state2 = nullptr;     // fire_poisson_residual's (so it never disturbs a solve's result)
  double* mean = nullptr;
  int* err = nullptr;
  float* src = nullptr;
  float* xlo = nullptr;         // low half of the solution pair when the caller passes none
  double* cinv = nullptr;       // inverse of the coarsest operator (transposed), FP64, or null
  cudaStream_t capStream = nullptr;
  cudaGraphExec_t exec = nullptr;
  // the captured graph's arguments
  const float* gb = nullptr;
  float* gx = nullptr;
  float* gxl = nullptr;
  double gtol = -1;
  int gmax = -1, ginner = -1;
};

namespace {

size_t align_up(size_t v) { return (v + 255) / 256 * 256; }
size_t elem_bytes(int sto) { return sto == STO_F32 ? 4 : 2; }
int storage_of(int prec) { return prec == FIRE_POISSON_FP16 ? STO_F16 : prec == FIRE_POISSON_BF16 ? STO_BF16 : STO_F32; }

// f(T{}) with the level's storage type.
template <typename F>
void with_type(int sto, F&& f) {
  if (sto == STO_F16) f(__half());
  else if (sto == STO_BF16) f(__nv_bfloat16());
  else f(float());
}
void psmooth(const PLevel& L, int color, int zero, cudaStream_t st) {
  with_type(L.sto, [&](auto t) {
    using T = decltype(t);
    launch_pdl(k_psmooth<T>, grid3((L.nx + 1) >> 1, L.ny, (L.nz + SMZ - 1) / SMZ), kBlock, 0, st, (T*)L.p, (const T*)L.b, L.nx, L.ny, L.nz,
               L.h, color, zero);
  });
}
void psweep2(const PLevel& L, const void* p, void* out, bool zero, cudaStream_t st) {
  with_type(L.sto, [&](auto t) {
    using T = decltype(t);
    launch_sweep2_t((const T*)p, (const T*)L.b, (T*)out, L.sweep, L.nx, L.ny, L.nz, L.h, 1.0f, zero, st);
  });
}
// `iters` sweeps in place; pairs of two-sweep launches where the level has a plan (the second of a pair writes p again).
void psweeps(const PLevel& L, int iters, bool zero, cudaStream_t st) {
  int done = 0;
  for (; L.sweep.px > 0 && done + 4 <= iters; done += 4) {
    psweep2(L, L.p, L.p2, zero && done == 0, st);
    psweep2(L, L.p2, L.p, false, st);
  }
  for (; done < iters; ++done) {
    psmooth(L, 0, zero && done == 0, st);
    psmooth(L, 1, 0, st);
  }
}
bool deep(const PLevel& C) { return (long)C.nx * C.ny * C.nz >= TRANSFER_DEEP_CELLS; }
void prestrict(const PLevel& F, const void* p, const PLevel& C, bool clear, cudaStream_t st) {
  with_type(F.sto, [&](auto f) {
    with_type(C.sto, [&](auto c) {
      using TF = decltype(f);
      using TC = decltype(c);
      launch_pdl(k_prestrict<TF, TC>, transfer_grid(C.nx, C.ny, C.nz, 1), kBlock, 0, st, (const TF*)p, (const TF*)F.b, F.nx, F.ny, F.nz, F.h,
                 (TC*)C.b, clear ? (TC*)C.p : (TC*)nullptr);
    });
  });
}
void pprolong(const PLevel& F, void* p, const PLevel& C, cudaStream_t st) {
  with_type(F.sto, [&](auto f) {
    with_type(C.sto, [&](auto c) {
      using TF = decltype(f);
      using TC = decltype(c);
      launch_pdl(deep(C) ? k_pprolong<TRANSFER_DEPTH, TF, TC> : k_pprolong<1, TF, TC>,
                 transfer_grid(C.nx, C.ny, C.nz, deep(C) ? TRANSFER_DEPTH : 1), kBlock, 0, st, (TF*)p, (const TC*)C.p, F.nx, F.ny, F.nz);
    });
  });
}

// The residual kernel's grid: four cells a thread where rows are whole warps of them (k_pres4), x pairs for even nx (k_pres2), single
// cells otherwise (k_pres).
bool pres_four(const PLevel& L) { return L.nx % (4 * GX) == 0; }
dim3 pres_grid(const PLevel& L) {
  const int cols = pres_four(L) ? L.nx / 4 : (L.nx % 2 == 0) ? L.nx / 2 : L.nx;
  return dim3((cols + GX - 1) / GX, (L.ny + GY - 1) / GY, (L.nz + GZ * RZ - 1) / (GZ * RZ));
}

// r = b - A (xh + xl); written scaled into level 0's RHS when `write` (refinement forms); partials for the test.
void pres(FirePoisson* ps, const PState* state, const float* b, const float* xh, const float* xl, bool write, cudaStream_t st) {
  const PLevel& L = ps->levels[0];
  with_type(write ? L.sto : STO_F32, [&](auto t) {
    using TR = decltype(t);
    auto kernel = pres_four(L) ? k_pres4<TR> : L.nx % 2 ? k_pres<TR> : L.nz % (GZ * RZ) ? k_pres2<TR, false> : k_pres2<TR, true>;
    launch_pdl(kernel, pres_grid(L), kBlock, 0, st, xh, xl, b, write ? (TR*)L.b : (TR*)nullptr, state, L.nx, L.ny, L.nz, 1.0f / (L.h * L.h),
               ps->partials);
  });
}
void pupdate(FirePoisson* ps, float* xh, float* xl, cudaStream_t st) {
  const PLevel& L = ps->levels[0];
  with_type(L.sto, [&](auto t) {
    using TE = decltype(t);
    launch_pdl(k_pupdate<TE>, grid3((L.nx + 1) >> 1, L.ny, L.nz), kBlock, 0, st, xh, xl, (const TE*)L.p, (const PState*)ps->state, L.nx, L.ny,
               L.nz);
  });
}
void ptest(FirePoisson* ps, PState* state, int mode, int first, int count, double tol, int max_iters, cudaGraphConditionalHandle h,
           int set_cond, cudaStream_t st) {
  launch_pdl(k_ptest, dim3(1), dim3(NT), 0, st, (const float4*)ps->partials, count, state, mode, first, tol, max_iters,
             (double)ps->cells, h, set_cond);
}
int pres_count(const FirePoisson* ps) {
  const dim3 g = pres_grid(ps->levels[0]);
  return (int)(g.x * g.y * g.z);
}

// One V(2,2) cycle of the correction solve on (levels[0].p, levels[0].b); zero_first: e starts at zero.  The
// coarsest level is solved exactly in FP64 (dense inverse) or, when too large for that, by FP64 sweeps.
void ir_vcycle(FirePoisson* ps, bool zero_first, cudaStream_t st) {
  const int n = (int)ps->levels.size(), T = ps->tailFirst, top = std::min(T, n - 1);
  std::vector<PLevel>& L = ps->levels;
  for (int i = 0; i < top; ++i) {
    const bool two = L[i].sweep.px > 0;
    if (two) psweep2(L[i], L[i].p, L[i].p2, i > 0 || zero_first, st);
    else psweeps(L[i], 2, i > 0 || zero_first, st);
    // a level that is smoothed here next starts from zero without reading its pressure
    prestrict(L[i], two ? L[i].p2 : L[i].p, L[i + 1], i + 1 == top, st);
  }
  if (ps->coarse) {
    launch_coarse(ps->mg.data(), T, n, 2, 2, 0, ps->cinv, 1, ps->err, st);
  } else if (T < n) {
    launch_tail(ps->mg.data(), T, n, 2, 2, COARSE64_SWEEPS, ps->err, st, true, ps->cinv);
  } else {
    psweeps(L[n - 1], ps->coarseIters, n == 1 && zero_first, st);
  }
  for (int i = top - 1; i >= 0; --i) {
    const bool two = L[i].sweep.px > 0;
    pprolong(L[i], two ? L[i].p2 : L[i].p, L[i + 1], st);
    if (two) psweep2(L[i], L[i].p2, L[i].p, false, st);
    else psweeps(L[i], 2, false, st);
  }
}
// The step's V(2,2) cycle (src/sim.js:588-599) on (x, b).
void fp32_vcycle(FirePoisson* ps, cudaStream_t st) {
  const int n = (int)ps->mg.size(), T = ps->tailFirst, top = std::min(T, n - 1);
  launch_down(ps->mg.data(), top, st);
  if (ps->coarse) launch_coarse(ps->mg.data(), T, n, 2, 2, ps->coarseIters, nullptr, 1, ps->err, st);
  else if (T < n) launch_tail(ps->mg.data(), T, n, 2, 2, ps->coarseIters, ps->err, st);
  else launch_sweeps(ps->mg[n - 1], ps->coarseIters, st);
  launch_up(ps->mg.data(), top, st);
}

// Dense inverse of the coarsest operator A (A p = (sum of ghost-ruled neighbours - diag p) / h^2, as the
// smoother's fixed point), by Gauss-Jordan elimination with partial pivoting in FP64; stored transposed
// (column i of the inverse is row i) so a warp's lanes read consecutive addresses.
bool coarse_inverse(const MGLevel& C, std::vector<double>& out) {
  const int nx = C.nx, ny = C.ny, nz = C.nz, n = nx * ny * nz;
  const double ih2 = 1.0 / ((double)C.h * (double)C.h);
  std::vector<double> a((size_t)n * n, 0.0), inv((size_t)n * n, 0.0);
  for (int z = 0; z < nz; ++z)
    for (int y = 0; y < ny; ++y)
      for (int x = 0; x < nx; ++x) {
        const int c = x + nx * (y + ny * z);
        double diag = 6.0;
        auto nb = [&](bool inside, int o, double ghost) {
          if (inside) a[(size_t)c * n + o] += ih2; else diag += ghost;
        };
        nb(x > 0, c - 1, 1.0);
        nb(x < nx - 1, c + 1, 1.0);
        nb(z > 0, c - nx * ny, 1.0);
        nb(z < nz - 1, c + nx * ny, 1.0);
        nb(y > 0, c - nx, -1.0);
        nb(y < ny - 1, c + nx, 1.0);
        a[(size_t)c * n + c] -= diag * ih2;
        inv[(size_t)c * n + c] = 1.0;
      }
  for (int col = 0; col < n; ++col) {
    int piv = col;
    for (int r = col + 1; r < n; ++r)
      if (std::fabs(a[(size_t)r * n + col]) > std::fabs(a[(size_t)piv * n + col])) piv = r;
    if (a[(size_t)piv * n + col] == 0.0) return false;
    if (piv != col)
      for (int k = 0; k < n; ++k) {
        std::swap(a[(size_t)piv * n + k], a[(size_t)col * n + k]);
        std::swap(inv[(size_t)piv * n + k], inv[(size_t)col * n + k]);
      }
    const double d = 1.0 / a[(size_t)col * n + col];
    for (int k = 0; k < n; ++k) { a[(size_t)col * n + k] *= d; inv[(size_t)col * n + k] *= d; }
    for (int r = 0; r < n; ++r) {
      if (r == col) continue;
      const double f = a[(size_t)r * n + col];
      if (f == 0.0) continue;
      for (int k = 0; k < n; ++k) { a[(size_t)r * n + k] -= f * a[(size_t)col * n + k]; inv[(size_t)r * n + k] -= f * inv[(size_t)col * n + k]; }
    }
  }
  out.assign((size_t)n * n, 0.0);
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) out[(size_t)j * n + i] = inv[(size_t)i * n + j];
  return true;
}

#define PCK(call)                                     \
  do {                                                \
    if ((call) != cudaSuccess) return FIRE_ERR_CUDA;  \
  } while (0)

// Captures the whole solve (pre-pass, conditional WHILE loop) for (b, x, x_lo, tol, max_iters, inner).
int build_graph(FirePoisson* ps, const float* b, float* x, float* xl, double tol, int max_iters, int inner) {
  if (ps->exec) { cudaGraphExecDestroy(ps->exec); ps->exec = nullptr; }
  const bool ir = ps->ir;
  if (!ir) { ps->mg[0].p = x; ps->mg[0].b = const_cast<float*>(b); }
  float* lo = ir ? (xl ? xl : ps->xlo) : nullptr;
  cudaStream_t st = ps->capStream;
  cudaGraph_t g = nullptr;
  PCK(cudaGraphCreate(&g, 0));
  PCK(cudaStreamBeginCaptureToGraph(st, g, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
  // tol = 0 asks for exactly max_iters iterations: they are unrolled into the graph (no conditional node,
  // so every kernel node can also be profiled); otherwise the iterations run in a WHILE node
  const bool unroll = tol == 0.0 && max_iters <= 64;
  cudaGraphConditionalHandle h = 0;
  if (!unroll && cudaGraphConditionalHandleCreate(&h, g, 0, cudaGraphCondAssignDefault) != cudaSuccess) {
    cudaGraph_t tmp;
    cudaStreamEndCapture(st, &tmp);
    cudaGraphDestroy(g);
    return FIRE_ERR_CUDA;
  }
  if (ir && !xl) cudaMemsetAsync(ps->xlo, 0, sizeof(float) * (size_t)ps->cells, st);   // the pair starts at (x, 0)
  launch_pdl(k_sumsq, dim3(SUMSQ_CTAS), dim3(NT), 0, st, b, ps->cells, ps->partials);
  ptest(ps, ps->state, 0, 1, SUMSQ_CTAS, tol, max_iters, h, 0, st);
  pres(ps, ps->state, b, x, lo, ir, st);
  ptest(ps, ps->state, 1, 1, pres_count(ps), tol, max_iters, h, unroll ? 0 : 1, st);
  // one iteration: correction cycle(s), update, residual, test
  auto body = [&](cudaStream_t s, int set_cond) {
    if (ir) {
      // the correction solve starts from e = 0: the first half-sweep ignores e's old contents, except when
      // level 0 itself is inside the shared-memory tail, which loads e
      if (ps->tailFirst == 0) cudaMemsetAsync(ps->levels[0].p, 0, sizeof(float) * (size_t)ps->cells, s);
      for (int c = 0; c < inner; ++c) ir_vcycle(ps, c == 0, s);
      pupdate(ps, x, lo, s);
      pres(ps, ps->state, b, x, lo, true, s);
    } else {
      fp32_vcycle(ps, s);
      pres(ps, ps->state, b, x, nullptr, false, s);
    }
    ptest(ps, ps->state, 1, 0, pres_count(ps), tol, max_iters, h, set_cond, s);
  };
  bool bodyOk = true;
  if (unroll) {
    for (int it = 0; it < max_iters; ++it) body(st, 0);
  } else {
    cudaStreamCaptureStatus cs;
    cudaGraph_t cg;
    const cudaGraphNode_t* deps;
    size_t ndeps;
    PCK(cudaStreamGetCaptureInfo(st, &cs, nullptr, &cg, &deps, nullptr, &ndeps));
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    PCK(cudaGraphAddNode(&node, cg, deps, nullptr, ndeps, &cp));
    PCK(cudaStreamUpdateCaptureDependencies(st, &node, nullptr, 1, cudaStreamSetCaptureDependencies));
    cudaStream_t bs = nullptr;
    PCK(cudaStreamCreateWithFlags(&bs, cudaStreamNonBlocking));
    if (cudaStreamBeginCaptureToGraph(bs, cp.conditional.phGraph_out[0], nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal) !=
        cudaSuccess) {
      cudaStreamDestroy(bs);
      return FIRE_ERR_CUDA;
    }
    body(bs, 1);
    cudaGraph_t bodyOut;
    bodyOk = cudaStreamEndCapture(bs, &bodyOut) == cudaSuccess;
    cudaStreamDestroy(bs);
  }
  cudaGraph_t outg;
  const bool ok = cudaStreamEndCapture(st, &outg) == cudaSuccess && bodyOk;
  if (!ok || cudaGetLastError() != cudaSuccess) { cudaGraphDestroy(g); return FIRE_ERR_CUDA; }
  const cudaError_t e = cudaGraphInstantiate(&ps->exec, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) { ps->exec = nullptr; return FIRE_ERR_CUDA; }
  ps->gb = b; ps->gx = x; ps->gxl = xl; ps->gtol = tol; ps->gmax = max_iters; ps->ginner = inner;
  return FIRE_OK;
}

struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    cudaSetDevice(dev);
  }
  ~DeviceGuard() { if (prev >= 0) cudaSetDevice(prev); }
};

constexpr int COARSE_DIRECT_MAX = 512;   // coarsest levels up to this many cells get the dense FP64 inverse

}  // namespace

extern "C" {

int fire_poisson_create(const int res[3], float h, int precision, int device, FirePoisson** out) {
  FIRE_RANGE("fire_poisson_create");
  if (!out) return FIRE_ERR_BAD_ARG;
  *out = nullptr;
  if (!res || res[0] < 2 || res[1] < 2 || res[2] < 2 || !(h > 0.0f)) return FIRE_ERR_BAD_ARG;
  if (precision < FIRE_POISSON_FP32 || precision > FIRE_POISSON_IR32) return FIRE_ERR_BAD_ARG;
  if ((long long)res[0] * res[1] * res[2] >= (1LL << 31)) return FIRE_ERR_BAD_ARG;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) return FIRE_ERR_NO_DEVICE;
  DeviceGuard dg(device);
  FirePoisson* ps = new FirePoisson();
  ps->device = device;
  for (int i = 0; i < 3; ++i) ps->res[i] = res[i];
  ps->h = h;
  ps->prec = precision;
  ps->ir = precision != FIRE_POISSON_FP32;
  ps->cells = (long long)res[0] * res[1] * res[2];
  // level hierarchy and coarse sweeps as FireSim builds them (src/sim.js:79-92)
  {
    int x = res[0], y = res[1], z = res[2];
    double hh = h;
    while (true) {
      ps->mg.push_back(MGLevel{x, y, z, (float)hh, nullptr, nullptr});
      if (x % 2 || y % 2 || z % 2 || std::min(x, std::min(y, z)) <= 6) break;
      x /= 2; y /= 2; z /= 2; hh *= 2;
    }
    const MGLevel& C = ps->mg.back();
    const double PI = 3.14159265358979323846;
    const double mu = (std::cos(PI / C.nx) + std::cos(PI / (2.0 * C.ny)) + std::cos(PI / C.nz)) / 3.0;
    ps->coarseIters = (int)std::max(8.0, std::min(64.0, std::ceil(std::log(0.05) / std::log(mu * mu))));
  }
  const int n = (int)ps->mg.size();
  ps->tailFirst = tail_first(ps->mg.data(), n, ps->ir);
  std::vector<double> cinv;
  const MGLevel& C = ps->mg.back();
  const int ccells = C.nx * C.ny * C.nz;
  // the coarse kernel takes the FP32 cycle, and the refinement's where the coarsest level gets its dense inverse
  const bool small = ccells <= COARSE_DIRECT_MAX;
  const int cf = !ps->ir || small ? coarse_first(ps->mg.data(), n, ps->ir) : n;
  const bool direct = ps->ir && std::min(ps->tailFirst, cf) < n && small && coarse_inverse(C, cinv);
  ps->coarse = cf < n && direct == ps->ir;
  if (ps->coarse) ps->tailFirst = cf;
  // arena: level arrays (level 0 of the FP32 form is the caller's x and b), partials, state
  size_t off = 0;
  std::vector<size_t> pOff(n), bOff(n), p2Off(n);
  ps->levels.resize(n);
  const int sto = storage_of(precision);
  for (int l = 0; l < n; ++l) {
    const MGLevel& M = ps->mg[l];
    PLevel& L = ps->levels[l];
    L.nx = M.nx; L.ny = M.ny; L.nz = M.nz; L.h = M.h;
    L.sto = (ps->ir && l < ps->tailFirst) ? sto : STO_F32;
    // every level that launches smooth: all above the coarse end, and the coarsest itself where none takes it
    // (not of 16-bit rows of an odd length).  The refinement's colour launch takes 3.5 us where the step's takes 1.6 (60x51x47),
    // so there the two-sweep kernel pays at every size: 40 refinements of 64 sweeps there, bfloat16, 18.2 -> 9.3 ms.
    if (l < ps->tailFirst && (L.sto == STO_F32 || M.nx % 2 == 0) && (ps->ir || sweep_pays(M, l == n - 1))) L.sweep = ps->mg[l].sweep = plan_sweep(ps->mg[l]);
    const size_t bytes = align_up((size_t)M.nx * M.ny * M.nz * elem_bytes(L.sto));
    if (l == 0 && !ps->ir) { pOff[l] = bOff[l] = (size_t)-1; continue; }
    pOff[l] = off; off += bytes;
    bOff[l] = off; off += bytes;
  }
  {
    const dim3 g = pres_grid(ps->levels[0]);
    const dim3 gr = grid3(res[0], res[1], res[2]);
    ps->partialsCount = std::max<int>(SUMSQ_CTAS, std::max<int>((int)(g.x * g.y * g.z), (int)(gr.x * gr.y * gr.z)));
  }
  const size_t partOff = off; off = align_up(off + sizeof(float4) * (size_t)ps->partialsCount);
  const size_t stateOff = off; off = align_up(off + 2 * sizeof(PState));
  const size_t meanOff = off; off = align_up(off + sizeof(double));
  const size_t errOff = off; off = align_up(off + sizeof(int));
  const size_t srcOff = off; off = align_up(off + sizeof(float) * MAX_SOURCES * 5);
  const size_t loOff = off; if (ps->ir) off = align_up(off + sizeof(float) * (size_t)ps->cells);
  const size_t cinvOff = off; if (direct) off = align_up(off + sizeof(double) * cinv.size());
  // last, the second pressure arrays of the two-sweep kernel: where only they do not fit, the levels take colour launches
  const size_t without = off;
  for (int l = 0; l < n; ++l)
    if (ps->levels[l].sweep.px > 0) {
      p2Off[l] = off;
      off += align_up((size_t)ps->mg[l].nx * ps->mg[l].ny * ps->mg[l].nz * elem_bytes(ps->levels[l].sto));
    }
  cudaError_t got = cudaMalloc(&ps->arena, off);
  if (got != cudaSuccess && off > without) {
    cudaGetLastError();
    for (int l = 0; l < n; ++l) ps->levels[l].sweep = ps->mg[l].sweep = SweepPlan{};
    off = without;
    got = cudaMalloc(&ps->arena, off);
  }
  if (got != cudaSuccess) { delete ps; return FIRE_ERR_OOM; }
  char* A = (char*)ps->arena;
  for (int l = 0; l < n; ++l) {
    if (ps->levels[l].sweep.px > 0) {
      ps->levels[l].p2 = A + p2Off[l];
      ps->mg[l].p2 = (float*)(A + p2Off[l]);   // used by the FP32 form
    }
    if (pOff[l] == (size_t)-1) continue;
    ps->levels[l].p = A + pOff[l];
    ps->levels[l].b = A + bOff[l];
    if (ps->levels[l].sto == STO_F32) { ps->mg[l].p = (float*)(A + pOff[l]); ps->mg[l].b = (float*)(A + bOff[l]); }
  }
  ps->partials = (float4*)(A + partOff);
  ps->state = (PState*)(A + stateOff);
  ps->state2 = ps->state + 1;
  ps->mean = (double*)(A + meanOff);
  ps->err = (int*)(A + errOff);
  ps->src = (float*)(A + srcOff);
  if (ps->ir) ps->xlo = (float*)(A + loOff);
  if (direct) ps->cinv = (double*)(A + cinvOff);
  if (cudaMemset(ps->arena, 0, off) != cudaSuccess || mg_configure(TAIL_SMEM_BUDGET) != cudaSuccess || coarse_configure() != cudaSuccess ||
      sweep_configure() != cudaSuccess ||
      cudaStreamCreateWithFlags(&ps->capStream, cudaStreamNonBlocking) != cudaSuccess ||
      (direct && cudaMemcpy(ps->cinv, cinv.data(), sizeof(double) * cinv.size(), cudaMemcpyHostToDevice) != cudaSuccess)) {
    fire_poisson_destroy(ps);
    return FIRE_ERR_CUDA;
  }
  *out = ps;
  return FIRE_OK;
}

int fire_poisson_destroy(FirePoisson* ps) {
  if (!ps) return FIRE_ERR_BAD_ARG;
  DeviceGuard dg(ps->device);
  cudaDeviceSynchronize();
  if (ps->exec) cudaGraphExecDestroy(ps->exec);
  if (ps->capStream) cudaStreamDestroy(ps->capStream);
  if (ps->arena) cudaFree(ps->arena);
  delete ps;
  return FIRE_OK;
}

int fire_poisson_solve(FirePoisson* ps, const float* b, float* x, float* x_lo, double tol, int max_iters, int inner_cycles, void* stream) {
  FIRE_RANGE("fire_poisson_solve");
  if (!ps || !b || !x || !(tol >= 0.0) || max_iters < 0 || (const void*)b == (const void*)x) return FIRE_ERR_BAD_ARG;
  if (x_lo && ((const void*)x_lo == (const void*)x || (const void*)x_lo == (const void*)b)) return FIRE_ERR_BAD_ARG;
  if (ps->ir && (inner_cycles < 1 || inner_cycles > 16)) return FIRE_ERR_BAD_ARG;
  if (!ps->ir) { inner_cycles = 1; x_lo = nullptr; }
  // the update and the residual read x, x_lo and b as float2 pairs
  if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(x_lo) | reinterpret_cast<uintptr_t>(b)) & 15u) != 0) return FIRE_ERR_BAD_ARG;
  DeviceGuard dg(ps->device);
  if (!ps->exec || ps->gb != b || ps->gx != x || ps->gxl != x_lo || ps->gtol != tol || ps->gmax != max_iters || ps->ginner != inner_cycles) {
    const int rc = build_graph(ps, b, x, x_lo, tol, max_iters, inner_cycles);
    if (rc) return rc;
  }
  return cudaGraphLaunch(ps->exec, reinterpret_cast<cudaStream_t>(stream)) == cudaSuccess ? FIRE_OK : FIRE_ERR_CUDA;
}

int fire_poisson_result(FirePoisson* ps, FirePoissonResult* out) {
  if (!ps || !out) return FIRE_ERR_BAD_ARG;
  DeviceGuard dg(ps->device);
  if (cudaDeviceSynchronize() != cudaSuccess) return FIRE_ERR_CUDA;
  PState s;
  int err = 0;
  if (cudaMemcpy(&s, ps->state, sizeof s, cudaMemcpyDeviceToHost) != cudaSuccess) return FIRE_ERR_CUDA;
  if (cudaMemcpy(&err, ps->err, sizeof err, cudaMemcpyDeviceToHost) != cudaSuccess) return FIRE_ERR_CUDA;
  if (err) {
    cudaMemset(ps->err, 0, sizeof(int));
    return FIRE_ERR_CUDA;
  }
  out->iterations = s.iters;
  out->rel_residual = s.rel;
  out->rel_residual_initial = s.rel0;
  out->b_norm = std::sqrt(s.bb);
  return FIRE_OK;
}

int fire_poisson_residual(FirePoisson* ps, const float* b, const float* x, const float* x_lo, double* rel) {
  if (!ps || !b || !x || !rel) return FIRE_ERR_BAD_ARG;
  if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(x_lo) | reinterpret_cast<uintptr_t>(b)) & 15u) != 0) return FIRE_ERR_BAD_ARG;
  DeviceGuard dg(ps->device);
  cudaStream_t st = ps->capStream;
  launch_pdl(k_sumsq, dim3(SUMSQ_CTAS), dim3(NT), 0, st, b, ps->cells, ps->partials);
  ptest(ps, ps->state2, 0, 1, SUMSQ_CTAS, 0.0, 0, 0, 0, st);
  pres(ps, ps->state2, b, x, x_lo, false, st);
  ptest(ps, ps->state2, 1, 1, pres_count(ps), 0.0, 0, 0, 0, st);
  if (cudaStreamSynchronize(st) != cudaSuccess) return FIRE_ERR_CUDA;
  PState s;
  if (cudaMemcpy(&s, ps->state2, sizeof s, cudaMemcpyDeviceToHost) != cudaSuccess) return FIRE_ERR_CUDA;
  *rel = s.rel;
  return FIRE_OK;
}

int fire_poisson_set_study(FirePoisson* ps, int coarse_sweeps) {
  if (!ps || ps->ir || coarse_sweeps < 1 || coarse_sweeps > 4096) return FIRE_ERR_BAD_ARG;
  DeviceGuard dg(ps->device);
  if (cudaDeviceSynchronize() != cudaSuccess) return FIRE_ERR_CUDA;
  for (MGLevel& L : ps->mg) { L.study = 1; L.sweep = SweepPlan{}; }   // the study's sweeps are colour launches
  ps->coarseIters = coarse_sweeps;
  ps->tailFirst = tail_first(ps->mg.data(), (int)ps->mg.size(), false);   // single-CTA tails in this variant
  ps->coarse = false;
  if (ps->exec) { cudaGraphExecDestroy(ps->exec); ps->exec = nullptr; }
  return FIRE_OK;
}

int fire_poisson_make_rhs(FirePoisson* ps, float* b, unsigned seed, int n_sources, float noise, void* stream) {
  FIRE_RANGE("fire_poisson_make_rhs");
  if (!ps || !b || n_sources < 0 || n_sources > MAX_SOURCES) return FIRE_ERR_BAD_ARG;
  DeviceGuard dg(ps->device);
  std::vector<float> src((size_t)std::max(1, n_sources) * 5, 0.0f);
  if (n_sources > 0 && fire_poisson_sources(seed, n_sources, ps->res, src.data()) != FIRE_OK) return FIRE_ERR_BAD_ARG;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  // the source table travels by a synchronous copy (it is a few KB, once per right-hand side)
  if (cudaStreamSynchronize(st) != cudaSuccess) return FIRE_ERR_CUDA;
  if (cudaMemcpy(ps->src, src.data(), sizeof(float) * src.size(), cudaMemcpyHostToDevice) != cudaSuccess) return FIRE_ERR_CUDA;
  const dim3 g = grid3(ps->res[0], ps->res[1], ps->res[2]);
  k_rhs<<<g, kBlock, 0, st>>>(b, ps->res[0], ps->res[1], ps->res[2], ps->src, n_sources, noise, seed, ps->partials);
  k_mean<<<1, NT, 0, st>>>(ps->partials, (int)(g.x * g.y * g.z), (double)ps->cells, ps->mean);
  k_sub_mean<<<1024, 256, 0, st>>>(b, ps->cells, ps->mean);
  return cudaGetLastError() == cudaSuccess ? FIRE_OK : FIRE_ERR_CUDA;
}

}  // extern "C"
