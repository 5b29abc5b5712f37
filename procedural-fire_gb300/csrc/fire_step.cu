// Per-step stencil kernels of the fire simulation: MacCormack advection, curl + forces (fused),
// divergence and projection.  Each kernel restates one WGSL compute shader of src/sim.js; the line
// ranges are given per kernel.  One thread per cell; CTAs cover 32 x 4 x 2 bricks so the gathers of
// the semi-Lagrangian back-trace and the 7-point stencils hit L1.  Fields are dense float4 arrays, x fastest, so every warp
// reads and writes 512 contiguous bytes per field.
#include <type_traits>
#include "fire_device.cuh"
#include "fire_launch.cuh"

namespace fire {

constexpr int BX = 32, BY = 4, BZ = 2;
// Minimum resident CTAs per SM requested from the register allocator for the gather-heavy kernels
// (latency-bound: more resident warps hide more of the dependent back-trace loads).
#ifndef FIRE_ADV_MIN_CTAS
#define FIRE_ADV_MIN_CTAS 4
#endif
#ifndef FIRE_FORCES_MIN_CTAS
#define FIRE_FORCES_MIN_CTAS 4
#endif

struct CellId { int i, j, k; bool ok; };
// Every stencil kernel starts here: wait for the predecessor grid (programmatic dependent launch), let the
// successor's launch begin, and locate this thread's cell.
// `blk` is the CTA's position in the simulation's grid: blockIdx for a per-simulation launch, or the
// position a batched launch derived from its flat block index (BatchMap).
// Cell tiles a stage can run with: the per-simulation kernels use Tile0; the batched (ensemble) kernels are
// instantiated for every CELL_TILES entry and the ensemble's autotuner picks one per stage.
template <int TX, int TY, int TZ> struct Tile { static constexpr int X = TX, Y = TY, Z = TZ; };
using Tile0 = Tile<BX, BY, BZ>;
// K: consecutive z cells of a thread (id.k is the first).
template <class T = Tile0, int K = 1>
__device__ __forceinline__ CellId cell_id(Dims d, uint3 blk) {
  pdl_wait();
  pdl_trigger();
  CellId c;
  c.i = blk.x * T::X + threadIdx.x;
  c.j = blk.y * T::Y + threadIdx.y;
  c.k = (blk.z * T::Z + threadIdx.z) * K;
  c.ok = c.i < d.nx && c.j < d.ny && c.k < d.nz;
  return c;
}
__device__ __forceinline__ CellId cell_id(Dims d) { return cell_id<Tile0>(d, blockIdx); }
static dim3 grid_for(Dims d, int depth = 1) {
  return dim3((d.nx + BX - 1) / BX, (d.ny + BY - 1) / BY, (d.nz + BZ * depth - 1) / (BZ * depth));
}
static dim3 block_shape() { return dim3(BX, BY, BZ); }


// ---------------- adv1 (src/sim.js:142-157) ----------------
template <class TileT = Tile0>
__device__ __forceinline__ void adv1_body(const float* __restrict__ P, const Fields& f, Dims d, uint3 blk) {
  CellId id = cell_id<TileT>(d, blk);
  if (!id.ok) return;
  const float dt = __ldg(P + P_dt), dx = __ldg(P + P_dx);
  const size_t ci = cell(id.i, id.j, id.k, d.nx, d.ny);
  f3 c = mk3((float)id.i + 0.5f, (float)id.j + 0.5f, (float)id.k + 0.5f);
  f3 b = backtrace(f.vel, c, xyz(__ldg(f.vel + ci)), dt, dx, d);
  float fade = outside_fade(b, d);
  float ws = sstep(0.03f, 0.4f, b.y * dx);
  f3 wind = mk3(__ldg(P + P_windX) * ws, 0.0f * ws, __ldg(P + P_windZ) * ws);
  Tap t = make_tap(b, d);
  f3 sv = xyz(sample(f.vel, t, d));
  f.velX[ci] = make_float4(mixf(wind.x, sv.x, fade), mixf(wind.y, sv.y, fade), mixf(wind.z, sv.z, fade), 0.0f);
  f.SX[ci] = mul4(sample(f.S, t, d), fade);
  f.S2X[ci] = mul4(sample(f.S2, t, d), fade);
}

// ---- adv1 with two cells a thread ----
// adv1 is bound by the L1's data path (177 wavefronts per warp and cell, 72 % of its rate, at 128x256x128): a float4 texel of
// a row costs four to five, and a trilinear sample eight texels.  A thread with two cells, one above the other, mostly samples
// points one cell apart, so the upper four texels of the first sample are the lower four of the second: they are kept, and
// loaded again only where the two floors differ.  A sample is formed from the same texels by the same operations as sample() in
// adv1_body, plane by plane; which product of a lerp the compiler rounds there (measured: of a x lerp of velocities the
// first, elsewhere, and in the mix with the wind, the second) is written out, so the results are the same bits.
// adv2, whose stencils' ranges double the arithmetic, gains nothing from it (256x512x256: 1469 -> 1508 us).
struct Corner { int o, dx, dy, dz; };   // offset of a 2 x 2 x 2 stencil's first cell and the steps to the second ones (0 at a clamped edge)
struct Weights { float x, y, z; };
__device__ __forceinline__ void corner_of(const Tap& t, Dims d, Corner& c, Weights& w) {
  const int sy = d.nx, sz = d.nx * d.ny;
  c.o = t.x0 + t.y0 * sy + t.z0 * sz;
  c.dx = t.x1 - t.x0;
  c.dy = (t.y1 - t.y0) * sy;
  c.dz = (t.z1 - t.z0) * sz;
  w.x = t.fx; w.y = t.fy; w.z = t.fz;
}
struct Quad { float4 a, b, c, e; };     // (x0, y0), (x1, y0), (x0, y1), (x1, y1) of one plane
__device__ __forceinline__ void load_quad(Quad& q, const float4* __restrict__ f, int o, const Corner& c) {
  q.a = __ldg(f + o);
  q.b = __ldg(f + (o + c.dx));
  q.c = __ldg(f + (o + c.dy));
  q.e = __ldg(f + (o + c.dy + c.dx));
}
// Whether the upper plane of stencil a is the lower plane of stencil b.
__device__ __forceinline__ bool same_plane(const Corner& a, const Corner& b) { return a.o + a.dz == b.o && a.dx == b.dx && a.dy == b.dy; }
// a (1 - t) + b t with one product inside an FMA: the first one, or (kSecond) the second.
template <bool kSecond>
__device__ __forceinline__ float4 lerp_as(const float4& a, const float4& b, float t) {
  const float s = 1.0f - t;
  auto one = [&](float p, float q) { return kSecond ? __fmaf_rn(q, t, __fmul_rn(p, s)) : __fmaf_rn(p, s, __fmul_rn(q, t)); };
  return make_float4(one(a.x, b.x), one(a.y, b.y), one(a.z, b.z), one(a.w, b.w));
}
template <bool kVel>
__device__ __forceinline__ float4 bilinear(const Quad& q, const Weights& w) {
  return lerp_as<false>(lerp_as<kVel>(q.a, q.b, w.x), lerp_as<kVel>(q.c, q.e, w.x), w.y);
}
// K samples of a field, K stencils one above the other.
template <bool kVel, int K>
__device__ __forceinline__ void sample_column(float4 (&out)[K], const float4* __restrict__ f, const Corner (&c)[K], const Weights (&w)[K]) {
  Quad q;
  load_quad(q, f, c[0].o, c[0]);
#pragma unroll
  for (int k = 0; k < K; ++k) {
    if (k > 0 && !same_plane(c[k > 0 ? k - 1 : 0], c[k])) load_quad(q, f, c[k].o, c[k]);
    const float4 lo = bilinear<kVel>(q, w[k]);
    load_quad(q, f, c[k].o + c[k].dz, c[k]);
    out[k] = lerp_as<false>(lo, bilinear<kVel>(q, w[k]), w[k].z);
  }
}
template <class TileT, int K>
__device__ __forceinline__ void adv1_column(const float* __restrict__ P, const Fields& f, Dims d, uint3 blk) {
  CellId id = cell_id<TileT, K>(d, blk);
  if (!id.ok) return;
  const float dt = __ldg(P + P_dt), dx = __ldg(P + P_dx);
  const unsigned plane = (unsigned)(d.nx * d.ny), c0 = (unsigned)(id.i + d.nx * id.j) + plane * (unsigned)id.k;
  unsigned ci[K];   // a cell above the domain repeats the top one and is not stored
  f3 c[K], v[K], b[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int z = min(id.k + k, d.nz - 1);
    ci[k] = c0 + plane * (unsigned)(z - id.k);
    c[k] = mk3((float)id.i + 0.5f, (float)id.j + 0.5f, (float)z + 0.5f);
    v[k] = xyz(__ldg(f.vel + ci[k]));
  }
  Corner at[K];
  Weights w[K];
  float4 s[K];
#pragma unroll
  for (int k = 0; k < K; ++k) corner_of(make_tap(c[k] - v[k] * (0.5f * dt) / dx, d), d, at[k], w[k]);
  sample_column<true>(s, f.vel, at, w);
  float fade[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    b[k] = c[k] - xyz(s[k]) * dt / dx;
    fade[k] = outside_fade(b[k], d);
    corner_of(make_tap(b[k], d), d, at[k], w[k]);
  }
  sample_column<true>(s, f.vel, at, w);
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const float ws = sstep(0.03f, 0.4f, b[k].y * dx);
    const float4 wind = make_float4(__ldg(P + P_windX) * ws, 0.0f * ws, __ldg(P + P_windZ) * ws, 0.0f);
    const f3 v = xyz(lerp_as<false>(wind, s[k], fade[k]));
    if (id.k + k < d.nz) f.velX[ci[k]] = make_float4(v.x, v.y, v.z, 0.0f);
  }
  sample_column<false>(s, f.S, at, w);
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (id.k + k < d.nz) f.SX[ci[k]] = mul4(s[k], fade[k]);
  sample_column<false>(s, f.S2, at, w);
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (id.k + k < d.nz) f.S2X[ci[k]] = mul4(s[k], fade[k]);
}

// ---------------- adv2 (src/sim.js:159-197) ----------------
template <class TileT = Tile0>
__device__ __forceinline__ void adv2_body(const float* __restrict__ P, const Fields& f, Dims d, uint3 blk) {
  CellId id = cell_id<TileT>(d, blk);
  if (!id.ok) return;
  const float dt = __ldg(P + P_dt), dx = __ldg(P + P_dx);
  const size_t ci = cell(id.i, id.j, id.k, d.nx, d.ny);
  f3 c = mk3((float)id.i + 0.5f, (float)id.j + 0.5f, (float)id.k + 0.5f);
  f3 v = xyz(__ldg(f.vel + ci));
  // reverse advection of the forward result
  f3 fw = c + v * dt / dx;
  f3 vH = xyz(__ldg(f.velX + ci));
  float4 sH = __ldg(f.SX + ci);
  float4 s2H = __ldg(f.S2X + ci);
  Tap tf = make_tap(fw, d);
  f3 vN = vH + (v - xyz(sample(f.velX, tf, d))) * 0.5f;
  float4 sN = add4(sH, mul4(sub4(__ldg(f.S + ci), sample(f.SX, tf, d)), 0.5f));
  float4 s2N = add4(s2H, mul4(sub4(__ldg(f.S2 + ci), sample(f.S2X, tf, d)), 0.5f));
  // clamp to the range of the source stencil at the back-traced point (Selle et al. 2008)
  f3 bt = backtrace(f.vel, c, v, dt, dx, d);
  f3 b = mk3(bt.x - 0.5f, bt.y - 0.5f, bt.z - 0.5f);
  int b0x = (int)floorf(clampf(b.x, -2.0f, (float)(d.nx + 1)));
  int b0y = (int)floorf(clampf(b.y, -2.0f, (float)(d.ny + 1)));
  int b0z = (int)floorf(clampf(b.z, -2.0f, (float)(d.nz + 1)));
  f3 vmn = mk3(1e9f, 1e9f, 1e9f), vmx = mk3(-1e9f, -1e9f, -1e9f);
  float4 smn = make_float4(1e9f, 1e9f, 1e9f, 1e9f), smx = make_float4(-1e9f, -1e9f, -1e9f, -1e9f);
  float4 tmn = smn, tmx = smx;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    int qx = b0x + (q & 1), qy = b0y + ((q >> 1) & 1), qz = b0z + ((q >> 2) & 1);
    f3 vv = xyz(ldc(f.vel, qx, qy, qz, d));
    float4 ss = ldc(f.S, qx, qy, qz, d);
    float4 tt = ldc(f.S2, qx, qy, qz, d);
    vmn = fmin3(vmn, vv); vmx = fmax3(vmx, vv);
    smn = fmin4(smn, ss); smx = fmax4(smx, ss);
    tmn = fmin4(tmn, tt); tmx = fmax4(tmx, tt);
  }
  if (outside_fade(mk3(b.x + 0.5f, b.y + 0.5f, b.z + 0.5f), d) < 1.0f) { vN = vH; sN = sH; s2N = s2H; }
  vN = fmin3(fmax3(vN, fmin3(vmn, vH)), fmax3(vmx, vH));
  sN = fmin4(fmax4(sN, fmin4(smn, sH)), fmax4(smx, sH));
  s2N = fmin4(fmax4(s2N, fmin4(tmn, s2H)), fmax4(tmx, s2H));
  const float4 z0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  f.velY[ci] = make_float4(vN.x, vN.y, vN.z, 0.0f);
  f.SY[ci] = fmax4(sN, z0);
  f.S2Y[ci] = fmax4(s2N, z0);
}

// ---------------- curl (src/sim.js:200-211) ----------------
__global__ void __launch_bounds__(256) k_curl(Fields f, Dims d) {
  CellId id = cell_id(d);
  if (!id.ok) return;
  f.vort[cell(id.i, id.j, id.k, d.nx, d.ny)] = curl_at(f.velY, id.i, id.j, id.k, d);
}

// ---------------- forces (src/sim.js:214-396), with the curl recomputed in place ----------------
// The reference runs a separate curl dispatch into a vorticity texture and reads 7 taps of it here.
// This kernel computes those 7 vorticity values from velY directly (the taps are clamped to the
// domain exactly as `ld` clamps them), and only in the cells whose confinement gate is open.
// Most cells of a domain are cold and burn nothing, and the kernel is bound by its instructions.  Where a factor is exactly 0,
// what it multiplies is left out: combustion below the ignition window, confinement and turbulence below 450 K without heat
// release, the age of gas that has none, the speed limit's root.  Only the sign of a zero can differ.  (Gates on the soot
// oxidation and the cooling cost more in a burning warp than they save.)
// A column march through shared memory, which formed every cell's vorticity once (870 instructions a cell, 65 % of the issue slots),
// lost to this as soon as the gates were there.  Measured (GB300, us, march without gates, with, this): 50x98x50 30.3, 28.9,
// 21.2; 80x120x80 50.6, 50.1, 39.3; 96x192x96 91.8, 90.8, 60.3; 128x256x128 185, 184, 103; 256x512x256 1103, 990, 621.  Where hot
// cells are strewn over the whole domain (82 % of 128x256x128 at random) it is 222 against 209.
// Per-cell physics.  The cell's own SY, S2Y and geometry values are passed in.
// Readers of the per-step parameter block for the forces physics: from global memory (batched, eager and
// adjoint launches), or from the kernel's own parameter space (the step graph's launch, whose block is set on
// the instantiated graph before every step), where each read is a constant-bank operand instead of a load.
struct ParamsGlobal {
  const float* __restrict__ P;
  __device__ __forceinline__ float operator[](int i) const { return __ldg(P + i); }
};
struct ParamsByValue {
  const ParamBlock& b;
  __device__ __forceinline__ float operator[](int i) const { return b.v[i]; }
};
// The cell's neighbourhood of velY.  The vorticity and its gradient are wanted only where confinement acts, in hot gas, a small
// part of a domain; there the seven curls are formed from their 42 velY cells, which the L1 holds.  Offsets along an axis: the
// clamped cells at -2, -1, 0, +1, +2, and what lies above the clamped -1 and below the clamped +1 (the cell itself, or at
// an edge its only neighbour: a tap outside the domain is the clamped cell's, with that cell's own neighbours).
struct Axis { int m2, m1, c, p1, p2, above_m1, below_p1; };
__device__ __forceinline__ Axis axis_of(int i, int n, int stride) {
  const int m1 = max(i - 1, 0), p1 = min(i + 1, n - 1);
  return Axis{stride * max(m1 - 1, 0), stride * m1, stride * i, stride * p1, stride * min(p1 + 1, n - 1),
              stride * min(m1 + 1, n - 1), stride * max(p1 - 1, 0)};
}
// sqrt(x^2 + y^2 + z^2) with the first (kSecond: the second) of the inner two squares rounded before it is added.
template <bool kSecond>
__device__ __forceinline__ float length_as(f3 a) {
  return sqrtf(__fmaf_rn(a.z, a.z, kSecond ? __fmaf_rn(a.x, a.x, __fmul_rn(a.y, a.y)) : __fmaf_rn(a.y, a.y, __fmul_rn(a.x, a.x))));
}
__device__ __forceinline__ f3 cross_as(f3 a, f3 b) {
  return mk3(__fmaf_rn(a.y, b.z, -__fmul_rn(a.z, b.y)), __fmaf_rn(a.z, b.x, -__fmul_rn(a.x, b.z)), __fmaf_rn(a.x, b.y, -__fmul_rn(a.y, b.x)));
}
struct VelNb {
  const float4* __restrict__ v;
  Dims d;
  int i, j, k;
  __device__ f3 at(int o) const { return xyz(__ldg(v + o)); }
  // the curl from the six neighbours' offsets
  __device__ f3 curl(int xm, int xp, int ym, int yp, int zm, int zp) const {
    const f3 L = at(xm), R = at(xp), B = at(ym), T = at(yp), K = at(zm), F = at(zp);
    return mk3((T.z - B.z) - (F.y - K.y), (F.x - K.x) - (R.z - L.z), (R.y - L.y) - (T.x - B.x)) * 0.5f;
  }
  __device__ float4 vel_center() const { return __ldg(v + cell(i, j, k, d.nx, d.ny)); }
  // The vorticity w, and in g the gradient of its length.
  __device__ f3 vorticity(f3& g) const {
    const Axis X = axis_of(i, d.nx, 1), Y = axis_of(j, d.ny, d.nx), Z = axis_of(k, d.nz, d.nx * d.ny);
    const int yz = Y.c + Z.c, xz = X.c + Z.c, xy = X.c + Y.c;
    auto side = [&](int xm, int xp, int ym, int yp, int zm, int zp) { return length_as<false>(curl(xm, xp, ym, yp, zm, zp)); };
    g.x = side(X.below_p1 + yz, X.p2 + yz, X.p1 + Y.m1 + Z.c, X.p1 + Y.p1 + Z.c, X.p1 + Y.c + Z.m1, X.p1 + Y.c + Z.p1) -
          side(X.m2 + yz, X.above_m1 + yz, X.m1 + Y.m1 + Z.c, X.m1 + Y.p1 + Z.c, X.m1 + Y.c + Z.m1, X.m1 + Y.c + Z.p1);
    g.y = side(X.m1 + Y.p1 + Z.c, X.p1 + Y.p1 + Z.c, Y.below_p1 + xz, Y.p2 + xz, X.c + Y.p1 + Z.m1, X.c + Y.p1 + Z.p1) -
          side(X.m1 + Y.m1 + Z.c, X.p1 + Y.m1 + Z.c, Y.m2 + xz, Y.above_m1 + xz, X.c + Y.m1 + Z.m1, X.c + Y.m1 + Z.p1);
    g.z = side(X.m1 + Y.c + Z.p1, X.p1 + Y.c + Z.p1, X.c + Y.m1 + Z.p1, X.c + Y.p1 + Z.p1, Z.below_p1 + xy, Z.p2 + xy) -
          side(X.m1 + Y.c + Z.m1, X.p1 + Y.c + Z.m1, X.c + Y.m1 + Z.m1, X.c + Y.p1 + Z.m1, Z.m2 + xy, Z.above_m1 + xy);
    return curl(X.m1 + yz, X.p1 + yz, Y.m1 + xz, Y.p1 + xz, Z.m1 + xy, Z.p1 + xy);
  }
  __device__ f3 lap_v() const {   // src/sim.js:340-343, same summation order
    f3 l = xyz(ldc(v, i + 1, j, k, d)) + xyz(ldc(v, i - 1, j, k, d));
    l = l + xyz(ldc(v, i, j + 1, k, d));
    l = l + xyz(ldc(v, i, j - 1, k, d));
    l = l + xyz(ldc(v, i, j, k + 1, d));
    l = l + xyz(ldc(v, i, j, k - 1, d));
    return l - xyz(vel_center()) * 6.0f;
  }
};
template <class PA>
__device__ __forceinline__ void forces_cell(const PA& pa, const Fields& f, const uint2* __restrict__ noiseT,
                                            const uint2* __restrict__ curlT, Dims d, int i, int j, int k, unsigned ci,
                                            const VelNb& nb, float4 s, float4 s2, const float4 geo) {
  const float dt = pa[P_dt], dx = pa[P_dx], I = pa[P_intensity];
  const float seed = pa[P_seed], time = pa[P_time];
  f3 p = mk3(pa[P_ox], pa[P_oy], pa[P_oz]) + mk3((float)i + 0.5f, (float)j + 0.5f, (float)k + 0.5f) * dx;
  float4 v4 = nb.vel_center();
  f3 v = xyz(v4);

  // ---- sources: pyrolysis on the hot log surfaces + the coal bed (src/sim.js:246-284)
  float src = 0.0f, anchor = 0.0f;
  if (geo.x > 0.001f) {
    f3 qa = p * pa[P_anchorFreq] + mk3(seed * 0.37f, 0.0f, 0.11f);
    anchor = sstep(-0.05f, 0.25f, noise4(noiseT, qa).z);
    f3 qn = p * (pa[P_srcFreq] * 0.06f) + mk3(seed * 0.131f, 0.0f, time * pa[P_srcSpeed]);
    const float th = pa[P_srcThresh];
    float pulse = sstep_inv(th - 0.25f, pa[P_STRIDE + E_invPulse], noise4(noiseT, qn).x);
    src = clampf(geo.x * pa[P_logSrc] * (pa[P_srcFloor] + pa[P_anchorGain] * anchor) * mixf(0.55f, 1.0f, pulse) * 1.2f,
                 0.0f, 1.0f) * I;
    src *= 1.0f - geo.z;
  }
  // Gaussian pyrolysis spots (build-defined extension; none by default)
  const int nSpots = (int)pa[P_STRIDE + E_nSpots];
  if (nSpots > 0 && p.y < pa[P_STRIDE + E_spotTop]) {   // above every spot's 4-sigma reach the sum is exactly 0
    const float spotRef = pa[P_STRIDE + E_spotRef];
    float acc = 0.0f;
    for (int q = 0; q < nSpots; ++q) {
      const int sp = P_STRIDE + E_SPOTS + SPOT_STRIDE * q;
      f3 dd = p - mk3(pa[sp + 0], pa[sp + 1], pa[sp + 2]);
      float sg = pa[sp + 3];
      float d2 = dot3(dd, dd);
      if (d2 < 16.0f * sg * sg) acc += (pa[sp + 4] / spotRef) * expf(-d2 / (2.0f * sg * sg));
    }
    src = fmaxf(src, clampf(acc, 0.0f, 1.0f) * I);
  }
  const float srcW = fminf(src, 1.0f);
  const float bedHot = geo.y;
  float bed = geo.y * clampf(I * 1.4f, 0.3f, 1.0f);
  if (bed > 0.001f) {
    f3 qb = p * 2.4f + mk3(0.17f, -time * 0.12f, time * 0.05f);
    bed *= sstep(0.0f, 0.3f, noise4(noiseT, qb).y);
  }
  s.y = fmaxf(s.y, src * pa[P_fuelSrc]);
  s.y = fmaxf(s.y, bed * pa[P_bedFuel]);
  s.x = fmaxf(s.x, src * pa[P_srcTemp]);
  s.x = fmaxf(s.x, bedHot * pa[P_bedTemp]);
  const float srcAll = fmaxf(srcW, bed);
  s2.w = mixf(s2.w, 1.0f, bed * (1.0f - srcW));
  s2.w = mixf(s2.w, 0.0f, srcW);
  s2.y = s2.y * (1.0f - srcAll);
  s2.x = fmaxf(s2.x, (1.0f - s.y) * srcW);
  s2.x = fmaxf(s2.x, (1.0f - s.y) * bed * 0.6f);
  // pow(1, y) = 1 exactly, so cells without a source skip the pow (here and for the sponge/top factors below)
  const float wsa = clampf(srcW + bed * 0.4f, 0.0f, 1.0f);
  float wsrc = wsa > 0.0f ? 1.0f - powf(1.0f - wsa * 0.5f, dt * 90.0f) : 0.0f;
  v.y = mixf(v.y, fmaxf(v.y, pa[P_srcVel]), wsrc);
  s2.z += geo.x * (1.0f - anchor) * pa[P_smolder] * dt * I;

  // ---- burst (src/sim.js:288-296)
  const float burstAmt = pa[P_burstAmt];
  if (burstAmt > 0.0f) {
    float bd = len3(p - mk3(pa[P_burstX], pa[P_burstY], pa[P_burstZ]));
    float bw = clampf(expf(-bd * bd / 0.006f) * burstAmt, 0.0f, 1.0f);
    s.y = fmaxf(s.y, 0.17f * bw);
    s.x = fmaxf(s.x, 0.9f * bw);
    s2.x *= 1.0f - bw;
    s2.w *= 1.0f - bw;
    s2.y = fmaxf(s2.y, 0.05f * bw * clampf(s.y + s2.x, 0.0f, 1.0f));
  }
  float ageF = s2.y != 0.0f ? s2.y / fmaxf(s.y + s2.x, 1e-4f) : s2.y;

  // ---- mixing-limited combustion (src/sim.js:299-309)
  const float T0 = 293.0f + 1000.0f * s.x;
  const float o = clampf(1.0f - s.y - s2.x, 0.0f, 1.0f);
  const float ignT = pa[P_ignT], rs = pa[P_rs];
  const float ign = sstep_inv(ignT - 50.0f, pa[P_STRIDE + E_invIgn], T0);
  const float kMix = pa[P_kMix], heatOut = pa[P_heatOut], expansion = pa[P_expansion];
  auto finite = [](float x) { return fabsf(x) <= 3.4028235e38f; };
  // without finite uniforms a product with an exact 0 need not be 0
  const bool plain = finite(kMix) && finite(heatOut) && finite(expansion) && rs > 0.0f && finite(rs) && dt > 0.0f && finite(dt);
  float b = 0.0f, T = T0, q = 0.0f, phi = 0.0f;
  if (plain && ign == 0.0f && T0 > 0.0f) {
    s2.x = fminf(s2.x, 1.0f);
  } else {
    b = fminf(s.y, o / rs) * (1.0f - expf(-kMix * ign * dt));
    s.y -= b;
    s2.x = fminf(s2.x + (1.0f + rs) * b, 1.0f);
    const float dT = fminf(heatOut * b, fmaxf(2100.0f - T0, 0.0f));
    T = T0 + dT;
    q = dT / dt;
    phi = geo.z > 0.5f ? 0.0f : fminf(expansion * q / T, 60.0f);
  }

  // ---- soot (src/sim.js:312-318); the age gate bounds come from the extension block
  const float sootOx = pa[P_sootOx];
  ageF = fminf(ageF + dt, 4.0f);
  s.z += pa[P_sootForm] * b * sstep_inv(pa[P_STRIDE + E_sootAge0], pa[P_STRIDE + E_invSootAge], ageF) * sstep(1000.0f, 1400.0f, T) * (1.0f - s2.w);
  s.z *= expf(-sootOx * (0.25f + o) * sstep(1100.0f, 1400.0f, T) * dt);
  s.z *= expf(-sootOx * 0.5f * o * sstep(850.0f, 1100.0f, T) * (1.0f - sstep(1100.0f, 1300.0f, T)) * dt);
  s.z *= pa[P_STRIDE + E_decaySoot];   // exp(-sootDissip dt), the same for every cell (host-evaluated)

  // ---- cooling (src/sim.js:321-330)
  const float th = T * 0.001f;
  T -= fminf(pa[P_radCool] * 970.0f * s.z * th * th * (th * th * th * th - 0.00737f), 6000.0f) * dt;
  const float notBurning = 1.0f - sstep(500.0f, 5000.0f, q);
  T = 293.0f + fmaxf(T - 293.0f, 0.0f) * expf(-pa[P_coolRate] * notBurning * dt);
  s.x = (T - 293.0f) * 0.001f;
  s.w = q * 1e-4f;
  s.y *= pa[P_STRIDE + E_decayFuel];    // exp(-fuelDissip dt)
  s2.x *= pa[P_STRIDE + E_decayVit];    // exp(-vitDecay dt)
  s2.z *= pa[P_STRIDE + E_decaySmoke];  // exp(-smokeDissip dt)
  s2.y = ageF * clampf(s.y + s2.x, 0.0f, 1.0f);

  // ---- buoyancy (src/sim.js:333)
  v.y += pa[P_buoyancy] * s.x * dt;

  // ---- hot-gas viscosity (src/sim.js:339-346)
  const float visc = pa[P_visc];
  if (visc > 0.0f) {
    f3 lapV = nb.lap_v();
    float nu = visc * 1.5e-5f * powf(fmaxf(T, 293.0f) / 293.0f, 1.7f);
    v = v + lapV * fminf(nu * dt / (dx * dx), 0.15f);
  }
  // ---- laminar flame base (src/sim.js:350); both gates below are 0 in cold gas without heat release
  if (T > 450.0f || s.w != 0.0f) {
    const float lamAge = pa[P_lamAge];
    const float lam = lamAge > 0.0f ? sstep(0.5f * lamAge, fmaxf(lamAge, 1e-3f), ageF) : 1.0f;

    // ---- vorticity confinement (src/sim.js:353-361).  Where the gate is exactly 0 (gas below 450 K, the
    // sources, the floor layer) the increment is a signed zero, so it is skipped; only the sign of a zero
    // velocity component can differ.
    const float gate = sstep(450.0f, 900.0f, T) * (1.0f - srcAll) * sstep(0.02f, 0.08f, p.y) * lam;
    if (gate != 0.0f) {
      f3 g;
      const f3 w = nb.vorticity(g);
      const float gl = length_as<true>(g);
      if (gl > 1e-6f) v = v + cross_as(g / gl, w) * (pa[P_vortEps] * gate) * dt;
    }

    // ---- sub-grid turbulence: rising, evolving curl noise (src/sim.js:364-368); skipped the same way where
    // its gate is exactly 0 (below 500 K with no heat release: most of the domain), which saves the table sample
    const float tgate = fmaxf(sstep(500.0f, 1100.0f, T), sstep(0.0f, 3.0f, s.w)) * (1.0f - srcAll) *
                        mixf(0.6f, 1.8f, sstep(0.2f, 0.75f, p.y)) * lam;
    if (tgate != 0.0f) {
      f3 tq = (p - mk3(0.0f, time * pa[P_turbRise], 0.0f)) * pa[P_turbFreq] + mk3(0.0f, 0.0f, time * pa[P_turbEvolve]);
      f3 cn = xyz(sample_table(curlT, tq));
      v = v + cn * pa[P_STRIDE + E_turbK] * tgate * dt * 10.0f;   // E_turbK = turbAmp / 12
    }
  }

  // ---- wind above the logs (src/sim.js:372-375)
  const float windX = pa[P_windX], windZ = pa[P_windZ];
  const float windK = sstep(0.05f, 0.5f, p.y) * (1.0f + pa[P_gust]);
  v.x += (windX * windK - v.x) * dt * 0.35f * windK;
  v.z += (windZ * windK - v.z) * dt * 0.35f * windK;
  v = v * pa[P_STRIDE + E_decayVel];    // exp(-velDissip dt)

  // ---- solids & sponge layers (src/sim.js:378-388)
  if (geo.z > 0.5f) { v = mk3(0.0f, 0.0f, 0.0f); s.y = 0.0f; s2.y = 0.0f; }
  f3 fp = mk3((float)i + 0.5f, (float)j + 0.5f, (float)k + 0.5f);
  float side = fminf(fminf(fp.x, (float)d.nx - fp.x), fminf(fp.z, (float)d.nz - fp.z));
  float sp = (1.0f - sstep(0.0f, 5.0f, side)) * pa[P_sponge];
  float wsy = sstep(0.03f, 0.4f, p.y);
  float wSx = windX * wsy, wSz = windZ * wsy;
  const float spc = clampf(sp, 0.0f, 1.0f);
  float ks = spc > 0.0f ? 1.0f - powf(1.0f - 0.15f * spc, dt * 90.0f) : 0.0f;
  v.x = mixf(v.x, wSx, ks);
  v.z = mixf(v.z, wSz, ks);
  float top = sstep((float)d.ny - 10.0f, (float)d.ny, fp.y);
  float kt = top > 0.0f ? powf(1.0f - 0.1f * top, dt * 90.0f) : 1.0f;
  s.z *= kt;
  s2.z *= kt;

  const float vv = dot3(v, v);
  if (vv > 224.0f) {   // sqrt(224) < 15
    const float vl = sqrtf(vv);
    if (vl > 15.0f) v = v * (15.0f / vl);
  }
  bool bad = isnan(s.x) || isnan(s.y) || isnan(s.z) || isnan(s.w) || isnan(s2.x) || isnan(s2.y) || isnan(s2.z) ||
             isnan(s2.w) || isnan(v.x) || isnan(v.y) || isnan(v.z);
  if (bad) {
    s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    s2 = s;
    v = mk3(0.0f, 0.0f, 0.0f);
  }
  f.velX[ci] = make_float4(v.x, v.y, v.z, phi);
  f.S[ci] = s;
  f.S2[ci] = s2;
}

template <class TileT = Tile0, class PA>
__device__ __forceinline__ void forces_body(const PA& pa, const Fields& f, const uint2* __restrict__ noiseT, const uint2* __restrict__ curlT,
                                            Dims d, uint3 blk) {
  CellId id = cell_id<TileT>(d, blk);
  if (!id.ok) return;
  const VelNb nb{f.velY, d, id.i, id.j, id.k};
  const size_t ci = cell(id.i, id.j, id.k, d.nx, d.ny);
  forces_cell(pa, f, noiseT, curlT, d, id.i, id.j, id.k, (unsigned)ci, nb, __ldg(f.SY + ci), __ldg(f.S2Y + ci), __ldg(f.geo + ci));
}

// ---------------- divergence minus the expansion target (src/sim.js:399-413) ----------------
// The z neighbours of a thread's K cells are its own cells.
template <class TileT = Tile0, int K = 1>
__device__ __forceinline__ void div_body(const float* __restrict__ P, const float4* __restrict__ velX, float* __restrict__ b0, Dims d,
                                         uint3 blk) {
  CellId id = cell_id<TileT, K>(d, blk);
  if (!id.ok) return;
  const int i = id.i, j = id.j;
  const float dx = __ldg(P + P_dx);
  const int plane = d.nx * d.ny;
  int ci = i + d.nx * j + plane * id.k;
  const int xm = i > 0 ? -1 : 0, xp = i < d.nx - 1 ? 1 : 0, ym = j > 0 ? -d.nx : 0, yp = j < d.ny - 1 ? d.nx : 0;
  float4 me = __ldg(velX + ci);
  float below = id.k > 0 ? __ldg(velX + (ci - plane)).z : me.z;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    if (k > 0 && id.k + k >= d.nz) break;
    const float4 above = id.k + k < d.nz - 1 ? __ldg(velX + (ci + plane)) : me;
    const float L = __ldg(velX + (ci + xm)).x, R = __ldg(velX + (ci + xp)).x;
    float B = __ldg(velX + (ci + ym)).y;
    const float T = __ldg(velX + (ci + yp)).y;
    if (j == 0) B = -me.y;   // solid floor
    b0[ci] = ((R - L) + (T - B) + (above.z - below)) / (2.0f * dx) - me.w;
    below = me.z;
    me = above;
    ci += plane;
  }
}

// ---------------- projection (src/sim.js:526-550) ----------------
// Ghosts: open sides and top, p = 0 on the face (-me); floor, Neumann (me).  The z neighbours of a thread's K cells are its own.
template <class TileT = Tile0, int K = 1>
__device__ __forceinline__ void project_body(const float* __restrict__ P, const float4* __restrict__ velX, const float* __restrict__ p0,
                                             const unsigned char* __restrict__ solid, float4* __restrict__ vel, Dims d, uint3 blk) {
  CellId id = cell_id<TileT, K>(d, blk);
  if (!id.ok) return;
  const int i = id.i, j = id.j;
  const float dx = __ldg(P + P_dx);
  const int plane = d.nx * d.ny;
  int ci = i + d.nx * j + plane * id.k;
  float me = __ldg(p0 + ci);
  float below = id.k > 0 ? __ldg(p0 + (ci - plane)) : -me;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    if (k > 0 && id.k + k >= d.nz) break;
    const float above = id.k + k < d.nz - 1 ? __ldg(p0 + (ci + plane)) : -me;
    const float xm = i > 0 ? __ldg(p0 + (ci - 1)) : -me, xp = i < d.nx - 1 ? __ldg(p0 + (ci + 1)) : -me;
    const float ym = j > 0 ? __ldg(p0 + (ci - d.nx)) : me, yp = j < d.ny - 1 ? __ldg(p0 + (ci + d.nx)) : -me;
    const f3 g = mk3(xp - xm, yp - ym, above - below) / (2.0f * dx);
    f3 v = xyz(__ldg(velX + ci)) - g;
    if (__ldg(solid + ci)) v = mk3(0.0f, 0.0f, 0.0f);   // geo.b > 0.5
    if (j == 0) v.y = fmaxf(v.y, 0.0f);
    const float vv = dot3(v, v);
    if (!(vv <= 399.0f)) {   // sqrt(399) < 20
      const float vl = sqrtf(vv);
      if (vl > 20.0f || isnan(vl)) v = isnan(vl) ? mk3(0.0f, 0.0f, 0.0f) : v * 20.0f / vl;
    }
    vel[ci] = make_float4(v.x, v.y, v.z, 0.0f);
    below = me;
    me = above;
    ci += plane;
  }
}

// ---------------- per-simulation kernels ----------------
__global__ void __launch_bounds__(256, FIRE_ADV_MIN_CTAS) k_adv1(const float* __restrict__ P, Fields f, Dims d) { adv1_body(P, f, d, blockIdx); }
__global__ void __launch_bounds__(256, FIRE_ADV_MIN_CTAS) k_adv1_column(const float* __restrict__ P, Fields f, Dims d) {
  adv1_column<Tile0, ADV1_DEPTH>(P, f, d, blockIdx);
}
__global__ void __launch_bounds__(256, FIRE_ADV_MIN_CTAS) k_adv2(const float* __restrict__ P, Fields f, Dims d) { adv2_body(P, f, d, blockIdx); }
__global__ void __launch_bounds__(256, FIRE_FORCES_MIN_CTAS) k_forces(const float* __restrict__ P, Fields f, const uint2* __restrict__ noiseT,
                                                                      const uint2* __restrict__ curlT, Dims d) {
  forces_body(ParamsGlobal{P}, f, noiseT, curlT, d, blockIdx);
}
__global__ void __launch_bounds__(256, FIRE_FORCES_MIN_CTAS) k_forces_pb(const __grid_constant__ ParamBlock pb, Fields f,
                                                                         const uint2* __restrict__ noiseT, const uint2* __restrict__ curlT,
                                                                         Dims d) {
  forces_body(ParamsByValue{pb}, f, noiseT, curlT, d, blockIdx);
}
// mg_counter (the residual-driven step graph only, else null): the solve that follows counts its V-cycles
// from zero, so this kernel clears the count instead of a separate launch.
template <int K>
__global__ void __launch_bounds__(256) k_div(const float* __restrict__ P, const float4* __restrict__ velX, float* __restrict__ b0, Dims d,
                                             int* __restrict__ mg_counter) {
  div_body<Tile0, K>(P, velX, b0, d, blockIdx);
  if (mg_counter && (blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.x | threadIdx.y | threadIdx.z) == 0) *mg_counter = 0;
}
template <int K>
__global__ void __launch_bounds__(256) k_project(const float* __restrict__ P, const float4* __restrict__ velX, const float* __restrict__ p0,
                                                 const unsigned char* __restrict__ solid, float4* __restrict__ vel, Dims d) {
  project_body<Tile0, K>(P, velX, p0, solid, vel, d, blockIdx);
}

// ---------------- batched kernels: one grid over many independent simulations ----------------
// Each CTA finds its simulation and its position in that simulation's grid from the flat block index
// (BatchMap), then runs the same body as the per-simulation kernel: the arithmetic, and so the results,
// are those of stepping each simulation alone.
template <class T, int K>
__global__ void __launch_bounds__(256, FIRE_ADV_MIN_CTAS) k_adv1_b(const __grid_constant__ BatchMap m, const __grid_constant__ StepBatch I) {
  uint3 blk; int i;
  batch_locate(m, blk, i);
  if (K > 1) adv1_column<T, K>(I.s[i].P, I.s[i].f, I.s[i].d, blk);
  else adv1_body<T>(I.s[i].P, I.s[i].f, I.s[i].d, blk);
}
template <class T>
__global__ void __launch_bounds__(256, FIRE_ADV_MIN_CTAS) k_adv2_b(const __grid_constant__ BatchMap m, const __grid_constant__ StepBatch I) {
  uint3 blk; int i;
  batch_locate(m, blk, i);
  adv2_body<T>(I.s[i].P, I.s[i].f, I.s[i].d, blk);
}
template <class T>
__global__ void __launch_bounds__(256, FIRE_FORCES_MIN_CTAS) k_forces_b(const __grid_constant__ BatchMap m, const __grid_constant__ StepBatch I,
                                                                        const uint2* __restrict__ noiseT, const uint2* __restrict__ curlT) {
  uint3 blk; int i;
  batch_locate(m, blk, i);
  forces_body<T>(ParamsGlobal{I.s[i].P}, I.s[i].f, noiseT, curlT, I.s[i].d, blk);
}
template <class T, int K>
__global__ void __launch_bounds__(256) k_div_b(const __grid_constant__ BatchMap m, const __grid_constant__ StepBatch I) {
  uint3 blk; int i;
  batch_locate(m, blk, i);
  div_body<T, K>(I.s[i].P, I.s[i].f.velX, I.s[i].b0, I.s[i].d, blk);
}
template <class T, int K>
__global__ void __launch_bounds__(256) k_project_b(const __grid_constant__ BatchMap m, const __grid_constant__ StepBatch I) {
  uint3 blk; int i;
  batch_locate(m, blk, i);
  project_body<T, K>(I.s[i].P, I.s[i].f.velX, I.s[i].p0, I.s[i].f.solid, I.s[i].f.vel, I.s[i].d, blk);
}

// The tile candidates of the batched stages: CELL_TILES cell tiles (256 threads each; x stays 32 or 64 wide
// for coalescing); the forces stage takes the first FORCES_TILES of them.
template <class F> void with_cell_tile(int v, F&& f) {
  switch (v) {
    case 1: f(Tile<32, 8, 1>{}); break;
    case 2: f(Tile<32, 2, 4>{}); break;
    case 3: f(Tile<64, 4, 1>{}); break;
    default: f(Tile0{}); break;
  }
}
static_assert(CELL_TILES == 4, "with_cell_tile lists every cell tile");
static_assert(FORCES_TILES <= CELL_TILES, "the forces stage's candidates are cell tiles");

// ---------------- launchers ----------------
// A thread takes several cells along z where enough threads remain to fill the SMs.  Measured (GB300, us, one cell -> several):
// adv1 50x98x50 16.8 -> 17.5, 64x128x64 22.0 -> 22.5, 80x120x80 30.5 -> 29.1, 96x192x96 56.1 -> 51.4, 128x256x128 119 -> 106,
// 256x512x256 873 -> 755; div and project together 64x128x64 16.4 -> 18.3, 80x120x80 20.4 -> 18.8, 128x256x128 61.4 -> 57.5,
// 256x512x256 390 -> 354.  In a batch all members count: a CTA of one cell a thread is short against finding its
// simulation (64x128x64 and 96x192x96 together: adv1 75 -> 63, div 19 -> 12.5, project 31 -> 16).
constexpr long ADV1_DEEP_CELLS = 600000, FLOW_DEEP_CELLS = 700000;
static long cells_of(Dims d) { return (long)d.nx * d.ny * d.nz; }
int adv1_depth(long cells) { return cells >= ADV1_DEEP_CELLS ? ADV1_DEPTH : 1; }
int flow_depth(long cells) { return cells >= FLOW_DEEP_CELLS ? FLOW_DEPTH : 1; }
void launch_adv1(const float* P, Fields f, Dims d, cudaStream_t st) {
  const int K = adv1_depth(cells_of(d));
  launch_pdl(K > 1 ? k_adv1_column : k_adv1, grid_for(d, K), block_shape(), 0, st, P, f, d);
}
void launch_adv2(const float* P, Fields f, Dims d, cudaStream_t st) { launch_pdl(k_adv2, grid_for(d), block_shape(), 0, st, P, f, d); }
void launch_curl(Fields f, Dims d, cudaStream_t st) { launch_pdl(k_curl, grid_for(d), block_shape(), 0, st, f, d); }
void launch_forces(const float* P, Fields f, const uint2* noise, const uint2* curl, Dims d, cudaStream_t st) {
  launch_pdl(k_forces, grid_for(d), block_shape(), 0, st, P, f, noise, curl, d);
}
void launch_forces_pb(const ParamBlock& pb, Fields f, const uint2* noise, const uint2* curl, Dims d, cudaStream_t st) {
  launch_pdl(k_forces_pb, grid_for(d), block_shape(), 0, st, pb, f, noise, curl, d);
}
cudaError_t forces_pb_set(cudaGraphExec_t exec, cudaGraphNode_t node, const ParamBlock& pb, Fields f, const uint2* noise,
                          const uint2* curl, Dims d) {
  void* args[] = {(void*)&pb, (void*)&f, (void*)&noise, (void*)&curl, (void*)&d};
  cudaKernelNodeParams kp = {};
  kp.func = (void*)k_forces_pb;
  kp.gridDim = grid_for(d);
  kp.blockDim = block_shape();
  kp.sharedMemBytes = 0;
  kp.kernelParams = args;
  return cudaGraphExecKernelNodeSetParams(exec, node, &kp);
}
// Block grids of the batched stages for a simulation of dims d with tile candidate `tile`.
dim3 step_grid(Dims d, int tile, int depth) {
  dim3 g;
  with_cell_tile(tile, [&](auto t) {
    using T = decltype(t);
    g = dim3((d.nx + T::X - 1) / T::X, (d.ny + T::Y - 1) / T::Y, (d.nz + T::Z * depth - 1) / (T::Z * depth));
  });
  return g;
}
void launch_adv1_batch(const BatchMap& m, const StepBatch& I, int tile, int depth, cudaStream_t st) {
  with_cell_tile(tile, [&](auto t) {
    using T = decltype(t);
    launch_pdl(depth > 1 ? k_adv1_b<T, ADV1_DEPTH> : k_adv1_b<T, 1>, dim3(m.prefix[m.n]), dim3(T::X, T::Y, T::Z), 0, st, m, I);
  });
}
void launch_adv2_batch(const BatchMap& m, const StepBatch& I, int tile, cudaStream_t st) {
  with_cell_tile(tile, [&](auto t) {
    using T = decltype(t);
    launch_pdl(k_adv2_b<T>, dim3(m.prefix[m.n]), dim3(T::X, T::Y, T::Z), 0, st, m, I);
  });
}
void launch_forces_batch(const BatchMap& m, const StepBatch& I, const uint2* noise, const uint2* curl, int tile, cudaStream_t st) {
  with_cell_tile(tile, [&](auto t) {
    using T = decltype(t);
    launch_pdl(k_forces_b<T>, dim3(m.prefix[m.n]), dim3(T::X, T::Y, T::Z), 0, st, m, I, noise, curl);
  });
}
void launch_div_batch(const BatchMap& m, const StepBatch& I, int tile, int depth, cudaStream_t st) {
  with_cell_tile(tile, [&](auto t) {
    using T = decltype(t);
    launch_pdl(depth > 1 ? k_div_b<T, FLOW_DEPTH> : k_div_b<T, 1>, dim3(m.prefix[m.n]), dim3(T::X, T::Y, T::Z), 0, st, m, I);
  });
}
void launch_project_batch(const BatchMap& m, const StepBatch& I, int tile, int depth, cudaStream_t st) {
  with_cell_tile(tile, [&](auto t) {
    using T = decltype(t);
    launch_pdl(depth > 1 ? k_project_b<T, FLOW_DEPTH> : k_project_b<T, 1>, dim3(m.prefix[m.n]), dim3(T::X, T::Y, T::Z), 0, st, m, I);
  });
}
void launch_div(const float* P, Fields f, float* b0, Dims d, cudaStream_t st, int* mg_counter) {
  const int K = flow_depth(cells_of(d));
  launch_pdl(K > 1 ? k_div<FLOW_DEPTH> : k_div<1>, grid_for(d, K), block_shape(), 0, st, P, (const float4*)f.velX, b0, d, mg_counter);
}
void launch_project(const float* P, Fields f, const float* p0, Dims d, cudaStream_t st) {
  const int K = flow_depth(cells_of(d));
  launch_pdl(K > 1 ? k_project<FLOW_DEPTH> : k_project<1>, grid_for(d, K), block_shape(), 0, st, P, (const float4*)f.velX, p0, (const unsigned char*)f.solid, f.vel, d);
}

}  // namespace fire

namespace fire {
// Verifies that this library carries a kernel image for the current device.
cudaError_t kernels_probe() {
  cudaFuncAttributes a;
  return cudaFuncGetAttributes(&a, k_div<1>);
}
}  // namespace fire
