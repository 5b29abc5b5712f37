// Transfers between two multigrid levels, for levels stored in FP32, half or bfloat16 (arithmetic in FP32).
//
// Both kernels are bound by bytes: at 256x512x256 the restriction reads p and b once (268 MB) and the prolongation reads and
// writes p (268 MB + 17 MB), at smaller sizes the same out of L2.  A thread owns one column of coarse cells, so one pair of
// fine columns x = 2 cx, 2 cx + 1 in two rows, and marches it up z: every fine value is loaded as part of a pair once per
// thread that needs it (10 pair or side loads per coarse cell and plane pair where a gather per child takes 64), and what two
// coarse planes share stays in registers.
// Measured (GB300, back to back, us, gather per coarse cell -> this; restriction, prolongation): 64x128x64 3.0 -> 1.8,
// 3.2 -> 2.5; 80x120x80 4.5 -> 2.3, 5.2 -> 4.5; 128x256x128 10.1 -> 5.4, 8.9 -> 8.0; 256x512x256 101 -> 56, 72 -> 53 (5.0 and
// 5.4 TB/s).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include "fire_launch.cuh"

namespace fire {

// Two neighbouring cells of a row in storage T, widened to FP32.
template <typename T> struct Cells2;
template <> struct Cells2<float> {
  using V = float2;
  static __device__ __forceinline__ float2 get(V v) { return v; }
  static __device__ __forceinline__ V put(float2 v) { return v; }
  static __device__ __forceinline__ float one(float v) { return v; }
  static __device__ __forceinline__ float back(float v) { return v; }
};
template <> struct Cells2<__half> {
  using V = __half2;
  static __device__ __forceinline__ float2 get(V v) { return __half22float2(v); }
  static __device__ __forceinline__ V put(float2 v) { return __floats2half2_rn(v.x, v.y); }
  static __device__ __forceinline__ float one(__half v) { return __half2float(v); }
  static __device__ __forceinline__ __half back(float v) { return __float2half_rn(v); }
};
template <> struct Cells2<__nv_bfloat16> {
  using V = __nv_bfloat162;
  static __device__ __forceinline__ float2 get(V v) { return __bfloat1622float2(v); }
  static __device__ __forceinline__ V put(float2 v) { return __floats2bfloat162_rn(v.x, v.y); }
  static __device__ __forceinline__ float one(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ __nv_bfloat16 back(float v) { return __float2bfloat16_rn(v); }
};
// kPair: p is aligned to a pair (else two loads).
template <bool kPair, typename T>
__device__ __forceinline__ float2 ld2(const T* p) {
  if (kPair) return Cells2<T>::get(*reinterpret_cast<const typename Cells2<T>::V*>(p));
  return make_float2(Cells2<T>::one(p[0]), Cells2<T>::one(p[1]));
}
template <bool kPair, typename T>
__device__ __forceinline__ void st2(T* p, float2 v) {
  if (kPair) {
    *reinterpret_cast<typename Cells2<T>::V*>(p) = Cells2<T>::put(v);
  } else {
    p[0] = Cells2<T>::back(v.x);
    p[1] = Cells2<T>::back(v.y);
  }
}

constexpr int LX = 32, LY = 4, LZ = 2;   // CTA shape of the transfers (256 threads)

// Fused residual + 8-child restriction (src/sim.js:439-466).  The residual and the sum have the operations and the order of
// restrict_cell (fire_mg.cu), its contractions written out.  pc, where given, is set to zero.
template <int kDepth, bool kPair, typename TF, typename TC>
__device__ __forceinline__ void restrict_march(const TF* __restrict__ p, const TF* __restrict__ b, int nx, int ny, int nz, float h,
                                               TC* __restrict__ bc, TC* __restrict__ pc, uint3 blk) {
  pdl_wait();
  pdl_trigger();
  const int cnx = nx / 2, cny = ny / 2, cnz = nz / 2;
  const int cx = blk.x * LX + threadIdx.x, cy = blk.y * LY + threadIdx.y, cz0 = (blk.z * LZ + threadIdx.z) * kDepth;
  if (cx >= cnx || cy >= cny || cz0 >= cnz) return;
  const float ih2 = 1.0f / (h * h);
  const int plane = nx * ny, at = 2 * cx + nx * 2 * cy + plane * 2 * cz0;
  const bool hxm = cx > 0, hxp = cx < cnx - 1, hym = cy > 0, hyp = cy < cny - 1;
  const float2 none = make_float2(0.0f, 0.0f);
  p += at;
  b += at;
  int t = cx + cnx * (cy + cny * cz0);
  float2 zm[2], c[2];   // the thread's pairs in plane 2 cz - 1 and 2 cz
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    zm[r] = cz0 > 0 ? ld2<kPair>(p - plane + r * nx) : none;
    c[r] = ld2<kPair>(p + r * nx);
  }
#pragma unroll
  for (int k = 0; k < kDepth; ++k) {
    if (k > 0 && cz0 + k >= cnz) break;
    const bool hzm = cz0 + k > 0, hzp = cz0 + k < cnz - 1;
    float2 u[2], w[2], lo[2], hi[2], bv[2][2];
    float xl[2][2], xr[2][2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      u[r] = ld2<kPair>(p + plane + r * nx);
      w[r] = hzp ? ld2<kPair>(p + 2 * plane + r * nx) : none;
    }
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      lo[f] = hym ? ld2<kPair>(p + f * plane - nx) : none;
      hi[f] = hyp ? ld2<kPair>(p + f * plane + 2 * nx) : none;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        xl[f][r] = hxm ? Cells2<TF>::one(p[f * plane + r * nx - 1]) : 0.0f;
        xr[f][r] = hxp ? Cells2<TF>::one(p[f * plane + r * nx + 2]) : 0.0f;
        bv[f][r] = ld2<kPair>(b + f * plane + r * nx);
      }
    }
    float acc = 0.0f;
#pragma unroll
    for (int f = 0; f < 2; ++f)
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          auto pick = [&](float2 v) { return q ? v.y : v.x; };
          const float2 mine = f ? u[r] : c[r];
          const float me = pick(mine);
          const float xm = q ? mine.x : (hxm ? xl[f][r] : -me), xp = q ? (hxp ? xr[f][r] : -me) : mine.y;
          const float ym = r ? pick(f ? u[0] : c[0]) : (hym ? pick(lo[f]) : me), yp = r ? (hyp ? pick(hi[f]) : -me) : pick(f ? u[1] : c[1]);
          const float zl = f ? pick(c[r]) : (hzm ? pick(zm[r]) : -me), zh = f ? (hzp ? pick(w[r]) : -me) : pick(u[r]);
          float sum = __fadd_rn(xm, xp);
          sum = __fadd_rn(sum, ym);
          sum = __fadd_rn(sum, yp);
          sum = __fadd_rn(sum, zl);
          sum = __fadd_rn(sum, zh);
          acc = __fadd_rn(acc, __fmaf_rn(-__fmaf_rn(-6.0f, me, sum), ih2, pick(bv[f][r])));
        }
    bc[t] = Cells2<TC>::back(acc * 0.125f);
    if (pc) pc[t] = Cells2<TC>::back(0.0f);
    t += cnx * cny;
    p += 2 * plane;
    b += 2 * plane;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      zm[r] = u[r];
      c[r] = w[r];
    }
  }
}

// Trilinear prolongation with mirror ghosts (src/sim.js:468-495; kClamp: clamped to the edge without sign flips), added to p.
// A fine cell reads the coarse offsets -1 and 0 or 0 and 1 per axis, an offset's weight being 0.75 for 0 and 0.25 for the others
// whichever child reads it; so each coarse value is weighted once (x, then y, exactly as each child's product
// v * wx * wy * wz starts) for all the children that use it, and a child takes eight FMAs in prolong_cell's order.
template <int kDepth, bool kPair, bool kClamp, typename TF, typename TC>
__device__ __forceinline__ void prolong_march(TF* __restrict__ p, const TC* __restrict__ pc, int nx, int ny, int nz, uint3 blk) {
  pdl_wait();
  pdl_trigger();
  const int ncx = nx / 2, ncy = ny / 2, ncz = nz / 2;
  const int cx = blk.x * LX + threadIdx.x, cy = blk.y * LY + threadIdx.y, cz0 = (blk.z * LZ + threadIdx.z) * kDepth;
  if (cx >= ncx || cy >= ncy || cz0 >= ncz) return;
  // offsets of the clamped 3 x 3 neighbourhood and the flips outside
  const int ox[3] = {max(cx - 1, 0), cx, min(cx + 1, ncx - 1)};
  const int oy[3] = {ncx * max(cy - 1, 0), ncx * cy, ncx * min(cy + 1, ncy - 1)};
  const float wx[3] = {!kClamp && cx == 0 ? -0.25f : 0.25f, 0.75f, !kClamp && cx == ncx - 1 ? -0.25f : 0.25f};
  const float wy[3] = {0.25f, 0.75f, !kClamp && cy == ncy - 1 ? -0.25f : 0.25f};
  float m[3][3][3];   // weighted values of planes cz - 1, cz, cz + 1
  auto load = [&](float (&o)[3][3], int z) {
    const TC* q = pc + ncx * ncy * min(max(z, 0), ncz - 1);
    const bool flip = !kClamp && (z < 0 || z >= ncz);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float v = Cells2<TC>::one(q[ox[c] + oy[r]]);
        o[r][c] = __fmul_rn(__fmul_rn(flip ? -v : v, wx[c]), wy[r]);
      }
  };
  load(m[0], cz0 - 1);
  load(m[1], cz0);
  p += 2 * cx + nx * (2 * cy) + nx * ny * (2 * cz0);
#pragma unroll
  for (int k = 0; k < kDepth; ++k) {
    if (k > 0 && cz0 + k >= ncz) break;
    float2 old[2][2];
#pragma unroll
    for (int dz = 0; dz < 2; ++dz)
#pragma unroll
      for (int dy = 0; dy < 2; ++dy) old[dz][dy] = ld2<kPair>(p + nx * dy + nx * ny * dz);
    load(m[2], cz0 + k + 1);
#pragma unroll
    for (int dz = 0; dz < 2; ++dz)
#pragma unroll
      for (int dy = 0; dy < 2; ++dy) {
        float v[2];
#pragma unroll
        for (int dx = 0; dx < 2; ++dx) {
          float acc = 0.0f;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int a = dz + (q >> 2);
            acc = __fmaf_rn(m[a][dy + ((q >> 1) & 1)][dx + (q & 1)], a == 1 ? 0.75f : 0.25f, acc);
          }
          v[dx] = acc;
        }
        st2<kPair>(p + nx * dy + nx * ny * dz, make_float2(__fadd_rn(old[dz][dy].x, v[0]), __fadd_rn(old[dz][dy].y, v[1])));
      }
    p += 2 * nx * ny;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        m[0][r][c] = m[1][r][c];
        m[1][r][c] = m[2][r][c];
      }
  }
}

// Coarse planes a thread marches: the prolongation four where that still leaves each of the 152 SMs eight CTAs, else one
// (256x512x256: 63 us with one, 55 with two, 53 with four, 57 with eight); the restriction one (56, 56, 62, 65: the compiler
// spreads a longer march's loads out); in a batch both four, since a CTA first has to find its simulation.
constexpr int TRANSFER_DEPTH = 4;
constexpr long TRANSFER_DEEP_CELLS = 152L * 8 * LX * LY * LZ * TRANSFER_DEPTH;
inline dim3 transfer_grid(int cnx, int cny, int cnz, int depth) {
  return dim3((cnx + LX - 1) / LX, (cny + LY - 1) / LY, (cnz + LZ * depth - 1) / (LZ * depth));
}

}  // namespace fire
