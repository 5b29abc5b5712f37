// Two red-black sweeps of a multigrid level (four colour passes) in one pass over its arrays.
//
// Why it looks like this.  A colour sweep as its own launch reads both colours' cache lines of p and b and writes p: at
// 128x256x128 it moves 88 MB of L2 traffic (9.6 us, the L2's rate), at 256x512x256 400 MB of DRAM traffic (70 us, the
// DRAM's rate), four times for the two sweeps of a visit.  Here a CTA marches a tile of columns up z and runs the four colour
// passes as a pipeline: with plane k just loaded, colour 0 of plane k-1, colour 1 of k-2, colour 0 again of k-3 and
// colour 1 of k-4, which is final and is written.  The four cells are the same column's (the colours alternate with z), so a
// thread's z neighbours are its own registers; it owns a pair of columns x = 2 px, 2 px + 1 in two rows, and in every
// step one column of each pair works while the other only serves as neighbour.  What neighbours need of a working
// column is one float4, its planes k .. k-3 after the step, which they read in the next step, when it rests: two float4 reads
// and one write per four updates, one barrier per plane.
// The tile's outermost four columns and rows, and four planes below and above a chunk, are computed from incomplete neighbours and
// not written (the next tile computes them); the result goes to another buffer, because other tiles read the old values.
// Each update has the arithmetic and the order of rb_update (fire_mg.cu): a neighbour outside the domain is a zero (added to a sum that
// starts at +0), the diagonal's reciprocal is exact for 3..9 in the sense of __fdividef (see fire_coarse.cu), so the
// result is bit-identical to the four launches.
//
// Measured (GB300, two sweeps back to back, us, four colour launches -> this): 64x128x64 8.6 -> 6.5, 80x120x80 13.2 -> 7.4,
// 96x192x96 19.0 -> 10.7, 128x256x128 28.0 -> 18.3, 256x512x256 270 -> 111 (402 MB there: 3.6 TB/s).  A step costs 0.3-0.5 us
// whatever the tile: about 130 instructions a warp behind a chain of reads, four dependent updates, a write and a barrier;
// registers and the halo keep it to one or two CTAs an SM.
// Grids without coarser levels (an odd side) run all their sweeps here; rows of an odd length copy their cells one by one.  Steps of two
// cycles with 64 sweeps each, us, colour launches -> this: 101x90x95 886 -> 731, 131x211x120 2491 -> 1709.
// Tried and slower: loads into register slots two planes ahead instead of the ring (16x16x16 2.9 -> 4.8, 256x512x256 123 -> 152:
// two steps do not cover a load, and 16 unrolled steps miss the instruction cache), four rows a thread (123 -> 134: spills).
#include <algorithm>
#include "fire_device.cuh"
#include "fire_launch.cuh"
#include "fire_level.cuh"

namespace fire {
namespace {

constexpr int SW_ROWS = 2;        // rows a thread owns
constexpr int SW_HALO = 4;
constexpr int SW_THREADS = 512;   // 128 registers a thread
constexpr int SW_AHEAD = 4;       // planes of p and b in flight: a step takes about 0.3 us, a load from L2 0.4 and more
constexpr int SW_RING = 7;        // entries a thread's ring is long: six planes, and one more so that 32 lanes hit all banks

// Asynchronous copy of one pair, or (kOdd: rows of an odd length, whose pairs are not aligned) of its two cells one by one; zeros
// where it lies outside the domain, and for the second cell where only that does.
template <bool kOdd, typename V>
__device__ __forceinline__ void copy_pair(V* dst, const void* src, bool in, bool second) {
  if (kOdd) {
    static_assert(!kOdd || sizeof(V) == 8, "cells of four bytes");
    const unsigned to = (unsigned)__cvta_generic_to_shared(dst);
    const char* from = static_cast<const char*>(src);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to), "l"(from), "r"(in ? 4 : 0) : "memory");
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to + 4), "l"(in && second ? from + 4 : from), "r"(in && second ? 4 : 0) : "memory");
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "n"((int)sizeof(V)), "r"(in ? (int)sizeof(V) : 0) : "memory");
  }
}

// A column of a thread as rings over the planes: plane k - j of the march's step k = i (mod 6) sits at slot (i - j) mod 6, so
// nothing is moved when the march advances.
struct Col { float v[6], b[6]; };
__host__ __device__ constexpr int slot(int i, int j) { return (i - j + 12) % 6; }
struct Sweeper {
  int nz;
  float h2, omega;
  float rd[SW_ROWS][2], rdz[SW_ROWS][2];   // reciprocal diagonals, and at the bottom and top planes
  float4* S;                                // published columns: [parity][row + 1][pair + 1], at this thread's first row
  int par, pitch;                           // float4 strides of a parity and of a row
  bool live;                                // the columns lie inside the domain
  bool both, wide;                          // and so do the second row and (rows of an odd length) the second column
};
template <bool kRelax>
__device__ __forceinline__ float update(const Sweeper& w, float old, float own, float far, float zm, float zp, float ym, float yp, float b, float rd) {
  float sum = __fadd_rn(own, far);   // x-, x+ in either order
  sum = __fadd_rn(sum, zm);
  sum = __fadd_rn(sum, zp);
  sum = __fadd_rn(sum, ym);
  sum = __fadd_rn(sum, yp);
  const float t = __fmaf_rn(-w.h2, b, sum);
  // relaxed: the change t rd - old takes one rounding, as the colour launches' contracted form does (two lose half a digit of p)
  return kRelax ? __fmaf_rn(w.omega, __fmaf_rn(t, rd, -old), old) : __fmul_rn(t, rd);
}
// Step k = I (mod 6) of the march.  kEdge: some of the planes k-4 .. k-1 lie outside the domain or touch its bottom or top.
template <typename T, bool kRelax, bool kOdd, int I, bool kEdge>
__device__ __forceinline__ void step(const Sweeper& w, Col (&c)[SW_ROWS][2], int k) {
  constexpr int a0 = (I & 1) ? 0 : 1;   // working column of row 0: (x + y + k - 1) even, y even; row 1's is the other
  float4 far[SW_ROWS];
#pragma unroll
  for (int r = 0; r < SW_ROWS; ++r) {
    const int a = (a0 + r) & 1;
    far[r] = w.S[r * w.pitch + (a ? 1 : w.par - 1)];   // x + 1 of an odd column, x - 1 of an even one
  }
  const float4 ylo = w.S[a0 * w.par - w.pitch];
  const float4 yhi = w.S[((a0 + SW_ROWS - 1) & 1) * w.par + SW_ROWS * w.pitch];
  const float lo[4] = {ylo.x, ylo.y, ylo.z, ylo.w}, hi[4] = {yhi.x, yhi.y, yhi.z, yhi.w};
#pragma unroll
  for (int j = 1; j <= 4; ++j) {
    const int z = k - j;
#pragma unroll
    for (int r = 0; r < SW_ROWS; ++r) {
      const int a = (a0 + r) & 1;
      Col& m = c[r][a];
      const float f[4] = {far[r].x, far[r].y, far[r].z, far[r].w};
      const float ym = r > 0 ? c[r > 0 ? r - 1 : 0][a].v[slot(I, j)] : lo[j - 1];
      const float yp = r + 1 < SW_ROWS ? c[r + 1 < SW_ROWS ? r + 1 : r][a].v[slot(I, j)] : hi[j - 1];
      float rd = w.rd[r][a];
      if (kEdge && (z == 0 || z == w.nz - 1)) rd = w.rdz[r][a];
      float v = update<kRelax>(w, m.v[slot(I, j)], c[r][1 - a].v[slot(I, j)], f[j - 1], m.v[slot(I, j + 1)], m.v[slot(I, j - 1)], ym, yp,
                                     m.b[slot(I, j)], rd);
      v = Cells2<T>::one(Cells2<T>::back(v));   // what a colour launch would have stored
      if ((r == 1 && !w.both) || (kOdd && a == 1 && !w.wide)) v = 0.0f;   // whatever its neighbours hold, also an infinity
      if (!kEdge || (unsigned)z < (unsigned)w.nz) m.v[slot(I, j)] = v;
    }
  }
  if (w.live) {
#pragma unroll
    for (int r = 0; r < SW_ROWS; ++r) {
      const int a = (a0 + r) & 1;
      const Col& m = c[r][a];
      w.S[r * w.pitch + a * w.par] = make_float4(m.v[slot(I, 0)], m.v[slot(I, 1)], m.v[slot(I, 2)], m.v[slot(I, 3)]);
    }
  }
}

// One tile: [x0, x1) x [y0, y1) x [z0, z1) is written; block of px pairs x ty thread rows.
struct SweepTile { int lx, ly, x0, x1, y0, y1, z0, z1; };
template <typename T, bool kZero, bool kRelax, bool kOdd = false>
__device__ __forceinline__ void sweep2_body(const T* __restrict__ p, const T* __restrict__ b, T* __restrict__ out, int nx, int ny, int nz,
                                            float h, float omega, int PX, int TY, const SweepTile& t) {
  extern __shared__ float4 sw_smem[];
  const bool work = (int)threadIdx.x < PX * TY;
  const int tid = threadIdx.x, ty = work ? tid / PX : 0, px = work ? tid - ty * PX : 0;   // a surplus thread reads thread 0's neighbours
  Sweeper w;
  w.nz = nz;
  w.h2 = h * h;
  w.omega = omega;
  w.pitch = PX + 2;
  w.par = w.pitch * (SW_ROWS * TY + 2);
  w.S = sw_smem + w.pitch * (SW_ROWS * ty + 1) + px + 1;
  for (int i = tid; i < 2 * w.par; i += blockDim.x) sw_smem[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const int x = t.lx + 2 * px, y = t.ly + SW_ROWS * ty;
  w.live = work && x < nx && y < ny;   // of an odd nx or ny the last pair or thread row has one column or row in the domain
  const bool wide = w.wide = !kOdd || x + 1 < nx;
  const bool both = w.both = y + 1 < ny;
  const bool core = w.live && x >= t.x0 && x < t.x1 && y >= t.y0 && y < t.y1;
  Col c[SW_ROWS][2];
#pragma unroll
  for (int r = 0; r < SW_ROWS; ++r)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const float d = 6.0f + (x + q == 0 ? 1.0f : 0.0f) + (x + q == nx - 1 ? 1.0f : 0.0f) + (y + r == ny - 1 ? 1.0f : 0.0f) - (y + r == 0 ? 1.0f : 0.0f);
      asm("rcp.approx.f32 %0, %1;" : "=f"(w.rd[r][q]) : "f"(d));
      asm("rcp.approx.f32 %0, %1;" : "=f"(w.rdz[r][q]) : "f"(d + 1.0f));
#pragma unroll
      for (int j = 0; j < 6; ++j) c[r][q].v[j] = c[r][q].b[j] = 0.0f;
    }
  const int plane = nx * ny, kend = t.z1 - 1 + SW_HALO;
  int k = max(t.z0 - SW_HALO, 0);
  const int kfirst = k;
  // the thread's rings of planes in flight, read only by itself: [p row 0, p row 1, b row 0, b row 1], plane k at entry I
  using V = typename Cells2<T>::V;
  V* ring[2 * SW_ROWS];
#pragma unroll
  for (int q = 0; q < 2 * SW_ROWS; ++q) ring[q] = reinterpret_cast<V*>(sw_smem + 2 * w.par) + (q * blockDim.x + tid) * SW_RING;
  const int first = w.live ? x + nx * (y + ny * k) : 0, row = w.live && both ? nx : 0;
  const T *pq = p + first, *bq = b + first;   // the plane to ask for next
  T* oq = out + first;                        // plane k - 4, once it is inside the chunk
  const int ahead = w.live ? plane : 0;
  pdl_wait();
  pdl_trigger();
  auto fetch = [&](int q, int entry) {
    const bool in = w.live && q < nz && q <= kend;
#pragma unroll
    for (int r = 0; r < SW_ROWS; ++r) {
      const bool here = in && (r == 0 || both);
      if (!kZero) copy_pair<kOdd>(ring[r] + entry, pq + r * row, here, wide);
      copy_pair<kOdd>(ring[SW_ROWS + r] + entry, bq + r * row, here, wide);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (q + 1 < nz) { pq += ahead; bq += ahead; }
  };
#pragma unroll
  for (int q = 0; q < SW_AHEAD; ++q) fetch(k + q, q);
  __syncthreads();
  // a step: plane k has arrived; plane k + SW_AHEAD is asked for once the step's own reads are under way
  auto advance = [&](auto index, auto edge) {
    constexpr int I = decltype(index)::value;
    constexpr bool kEdge = decltype(edge)::value;
    asm volatile("cp.async.wait_group %0;" ::"n"(SW_AHEAD - 1) : "memory");
#pragma unroll
    for (int r = 0; r < SW_ROWS; ++r) {
      if (!kZero) {
        const float2 v = Cells2<T>::get(ring[r][I]);
        c[r][0].v[slot(I, 0)] = v.x;
        c[r][1].v[slot(I, 0)] = v.y;
      } else {
        c[r][0].v[slot(I, 0)] = c[r][1].v[slot(I, 0)] = 0.0f;
      }
    }
    step<T, kRelax, kOdd, I, kEdge>(w, c, k);
#pragma unroll
    for (int r = 0; r < SW_ROWS; ++r) {   // b of plane k: used from the next step on; its slot held plane k - 6's
      const float2 v = Cells2<T>::get(ring[SW_ROWS + r][I]);
      c[r][0].b[slot(I, 0)] = v.x;
      c[r][1].b[slot(I, 0)] = v.y;
    }
    fetch(k + SW_AHEAD, (I + SW_AHEAD) % 6);
    if (k - SW_HALO >= kfirst) {
      if (core && k - SW_HALO >= t.z0)
#pragma unroll
        for (int r = 0; r < SW_ROWS; ++r)
          if (r == 0 || both) {
            const float2 v = make_float2(c[r][0].v[slot(I, 4)], c[r][1].v[slot(I, 4)]);
            if (!kOdd) {
              *reinterpret_cast<V*>(oq + r * nx) = Cells2<T>::put(v);
            } else {
              oq[r * nx] = Cells2<T>::back(v.x);
              if (wide) oq[r * nx + 1] = Cells2<T>::back(v.y);
            }
          }
      oq += plane;
    }
    ++k;
    __syncthreads();
  };
  // the march starts at an even plane, so I fixes the parity of k
  while (true) {
    if (k > SW_HALO && k + 5 < nz && k + 5 <= kend) {
      advance(std::integral_constant<int, 0>{}, std::false_type{});
      advance(std::integral_constant<int, 1>{}, std::false_type{});
      advance(std::integral_constant<int, 2>{}, std::false_type{});
      advance(std::integral_constant<int, 3>{}, std::false_type{});
      advance(std::integral_constant<int, 4>{}, std::false_type{});
      advance(std::integral_constant<int, 5>{}, std::false_type{});
      if (k > kend) break;
    } else {
      advance(std::integral_constant<int, 0>{}, std::true_type{}); if (k > kend) break;
      advance(std::integral_constant<int, 1>{}, std::true_type{}); if (k > kend) break;
      advance(std::integral_constant<int, 2>{}, std::true_type{}); if (k > kend) break;
      advance(std::integral_constant<int, 3>{}, std::true_type{}); if (k > kend) break;
      advance(std::integral_constant<int, 4>{}, std::true_type{}); if (k > kend) break;
      advance(std::integral_constant<int, 5>{}, std::true_type{}); if (k > kend) break;
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

__device__ __forceinline__ SweepTile tile_of(const SweepPlan& P, int nx, int ny, int nz, int blk) {
  SweepTile t;
  const int tx = blk % P.ntx, q = blk / P.ntx, ty = q % P.nty, tz = q / P.nty;
  t.x0 = tx * P.cx; t.x1 = min(nx, t.x0 + P.cx);
  t.y0 = ty * P.cy; t.y1 = min(ny, t.y0 + P.cy);
  t.z0 = tz * P.cz; t.z1 = min(nz, t.z0 + P.cz);
  t.lx = max(0, t.x0 - SW_HALO);
  t.ly = max(0, t.y0 - SW_HALO);
  return t;
}
template <typename T, bool kZero, bool kRelax, bool kOdd = false>
__global__ void __launch_bounds__(SW_THREADS, 1) k_sweep2(const T* __restrict__ p, const T* __restrict__ b, T* __restrict__ out, int nx, int ny,
                                                          int nz, float h, float omega, SweepPlan P) {
  sweep2_body<T, kZero, kRelax, kOdd>(p, b, out, nx, ny, nz, h, omega, P.px, P.ty, tile_of(P, nx, ny, nz, blockIdx.x));
}

// Measured (GB300, ensemble of 16 grids from 32x64x32 to 96x192x96, 4 cycles): 8 launches per level and cycle of batched colour
// sweeps, 1245 us of a step's 2978, became 2 and the step takes 2486; CTAs of 256 or 448 threads give the same within 1 %.
// With both bodies (omega 1 and not) in one kernel 160 bytes of registers spilled: a step 2244, with one body 2032.
// A level of every simulation of a batch: down from p (kZero: from zero) into p2, else back from p2 into p.
// kMixed: some member's omega is not 1 (a second body, which costs registers).
template <bool kZero, bool kMixed>
__global__ void __launch_bounds__(SW_THREADS, 1) k_sweep2_b(const __grid_constant__ BatchMap m, const __grid_constant__ LevelBatch L, int down) {
  uint3 blk; int i;
  batch_locate(m, blk, i);
  const MGLevel& v = L.l[i];
  const SweepTile t = tile_of(v.sweep, v.nx, v.ny, v.nz, blk.x);
  const float* p = down ? v.p : v.p2;
  float* out = down ? v.p2 : v.p;
  if (!kMixed || v.omega == 1.0f) sweep2_body<float, kZero, false>(p, v.b, out, v.nx, v.ny, v.nz, v.h, v.omega, v.sweep.px, v.sweep.ty, t);
  else sweep2_body<float, kZero, true>(p, v.b, out, v.nx, v.ny, v.nz, v.h, v.omega, v.sweep.px, v.sweep.ty, t);
}

constexpr size_t SW_SMEM = 200 * 1024;
int sweep_threads(const SweepPlan& P) { return std::max(64, (P.px * P.ty + 31) / 32 * 32); }
size_t sweep_smem(const SweepPlan& P, int threads) {
  return sizeof(float4) * 2 * (size_t)(P.px + 2) * (SW_ROWS * P.ty + 2) + sizeof(float2) * 2 * SW_ROWS * SW_RING * (size_t)threads;
}

}  // namespace

// The cut that costs least by a model of the kernel: a step of a resident set of CTAs takes the larger of a step's least (one
// warp's chain of four updates, the shared-memory reads and the barrier) and SW_WARP cycles per resident warp (its instructions
// on one of four schedulers); a CTA runs its planes and eight more, and about SW_START cycles around them.  On levels of
// SW_LARGE_CELLS and more a step takes SW_ADD besides, and 6 % more where a row of pairs ends inside eight lanes: fitted to 9638
// plans of ten levels, the choice is within 3.5 % of the fastest everywhere (256x512x256: 111 us, 124 without).  On small levels
// those terms choose narrower rows, as fast back to back but slower in whole solves (64x64x64 and 50x98x50 2 %, 128x256x128 0.3 %).
constexpr double SW_STEP = 300.0, SW_STEP_LARGE = 200.0, SW_ADD = 200.0, SW_WARP = 30.0, SW_START = 1500.0;
constexpr long SW_LARGE_CELLS = 5000000;
SweepPlan plan_sweep(const MGLevel& L, int sms, int block) {
  const int nx = L.nx, ny = L.ny, nz = L.nz;
  SweepPlan best{};
  if (L.study || nx < 8 || ny < 4 || nz < 4) return best;
  const bool large = (long)nx * ny * nz >= SW_LARGE_CELLS;
  double cost = 1e30;
  auto even = [](int v) { return (v + 1) & ~1; };
  for (int ntx = 1; ntx <= 16; ++ntx) {
    const int cx = even((nx + ntx - 1) / ntx);
    if ((nx + cx - 1) / cx != ntx || (cx < 16 && ntx > 1)) continue;
    const int px = (std::min(nx, cx + SW_HALO * std::min(ntx - 1, 2)) + 1) / 2;
    for (int nty = 1; nty <= 128; ++nty) {
      const int cy = even((ny + nty - 1) / nty);
      if (cy < 8 && nty > 1) break;
      if ((ny + cy - 1) / cy != nty) continue;
      const int ty = (std::min(ny, cy + SW_HALO * std::min(nty - 1, 2)) + SW_ROWS - 1) / SW_ROWS;
      SweepPlan P{px, ty, ntx, nty, 1, cx, cy, nz};
      if (px * ty > (block ? block : SW_THREADS)) continue;
      const int threads = block ? block : sweep_threads(P);
      if (sweep_smem(P, threads) > SW_SMEM) continue;
      const int occ = std::max(1, std::min({65536 / (128 * threads), (int)(SW_SMEM / sweep_smem(P, threads)), 8}));
      int last = 0;
      for (int waves = 1; waves <= 8; ++waves) {   // chunks in z that fill whole waves of the SMs
        const int want = std::max(1, std::min(sms * occ * waves / (ntx * nty), nz / 4));
        const int cz = even((nz + want - 1) / want), ntz = (nz + cz - 1) / cz;
        if (ntz == last) continue;
        last = ntz;
        const long ctas = (long)ntx * nty * ntz, w = (ctas + (long)sms * occ - 1) / ((long)sms * occ);
        const int resident = (int)std::min<long>(occ, (ctas + sms - 1) / sms);
        const double warps = SW_WARP * resident * threads / 32.0;
        const double step = large ? (SW_ADD + std::max(SW_STEP_LARGE, warps)) * (px % 8 ? 1.06 : 1.0) : std::max(SW_STEP, warps);
        const double c = w * ((std::min(nz, cz + SW_HALO * std::min(ntz, 2)) + 1) * step + SW_START);
        if (c < cost) { cost = c; best = P; best.ntz = ntz; best.cz = cz; }
      }
    }
  }
  return best;
}

// Where a launch of this kernel is faster than the four colour launches it replaces, from whole-level times (GB300, us, this against
// four): odd rows 61x111x57 8.5 / 7.2, 71x131x67 8.3 / 12.5; a coarsest level (odd in y or z) 50x91x49 6.9 / 6.6, 56x101x60 5.8 /
// 7.3; a level with coarser ones 42x84x42 7.0 / 6.3, 46x92x44 5.9 / 6.4.  (In a batch all members' levels share the launch.)
bool sweep_pays(const MGLevel& L, bool coarsest) {
  return (long)L.nx * L.ny * L.nz >= (L.nx % 2 ? 500000 : coarsest ? 280000 : 150000);
}

template <typename T>
cudaError_t launch_sweep2_t(const T* p, const T* b, T* out, const SweepPlan& P, int nx, int ny, int nz, float h, float omega, bool zero,
                            cudaStream_t st) {
  if (P.px == 0) return cudaErrorInvalidValue;
  const dim3 grid(P.ntx * P.nty * P.ntz), block(sweep_threads(P));
  const size_t smem = sweep_smem(P, (int)block.x);
  auto go = [&](auto kernel) { return launch_pdl(kernel, grid, block, smem, st, p, b, out, nx, ny, nz, h, omega, P); };
  if (nx % 2) {
    if constexpr (sizeof(T) != sizeof(float)) return cudaErrorInvalidValue;   // 16-bit rows of an odd length: colour launches
    else if (omega == 1.0f) return zero ? go(k_sweep2<T, true, false, true>) : go(k_sweep2<T, false, false, true>);
    else return zero ? go(k_sweep2<T, true, true, true>) : go(k_sweep2<T, false, true, true>);
  }
  if (omega == 1.0f) return zero ? go(k_sweep2<T, true, false>) : go(k_sweep2<T, false, false>);
  if constexpr (sizeof(T) != sizeof(float)) return cudaErrorInvalidValue;   // the refinement's sweeps are Gauss-Seidel
  else return zero ? go(k_sweep2<T, true, true>) : go(k_sweep2<T, false, true>);
}
cudaError_t launch_sweep2(const MGLevel& L, const float* p, float* out, bool zero, cudaStream_t st) {
  return launch_sweep2_t<float>(p, L.b, out, L.sweep, L.nx, L.ny, L.nz, L.h, L.omega, zero, st);
}

cudaError_t launch_sweep2_batch(const BatchMap& m, const LevelBatch& L, bool down, bool zero, cudaStream_t st) {
  size_t smem = 0;
  for (int k = 0; k < m.n; ++k) smem = std::max(smem, sweep_smem(L.l[m.inst[k]].sweep, SW_BATCH_THREADS));
  bool mixed = false;
  for (int k = 0; k < m.n; ++k) mixed = mixed || L.l[m.inst[k]].omega != 1.0f;
  return launch_pdl(mixed ? (zero ? k_sweep2_b<true, true> : k_sweep2_b<false, true>) : zero ? k_sweep2_b<true, false> : k_sweep2_b<false, false>,
                    dim3(m.prefix[m.n]), dim3(SW_BATCH_THREADS), smem, st, m, L, (int)down);
}

template cudaError_t launch_sweep2_t<float>(const float*, const float*, float*, const SweepPlan&, int, int, int, float, float, bool, cudaStream_t);
template cudaError_t launch_sweep2_t<__half>(const __half*, const __half*, __half*, const SweepPlan&, int, int, int, float, float, bool,
                                             cudaStream_t);
template cudaError_t launch_sweep2_t<__nv_bfloat16>(const __nv_bfloat16*, const __nv_bfloat16*, __nv_bfloat16*, const SweepPlan&, int, int, int,
                                                    float, float, bool, cudaStream_t);

cudaError_t launch_sweeps(const MGLevel& L, int iters, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  int done = 0;
  for (; L.sweep.px > 0 && done + 4 <= iters && e == cudaSuccess; done += 4) {   // p -> p2 -> p
    e = launch_sweep2(L, L.p, L.p2, false, st);
    if (e == cudaSuccess) e = launch_sweep2(L, L.p2, L.p, false, st);
  }
  for (; done < iters && e == cudaSuccess; ++done) {
    e = launch_smooth(L, 0, st);
    if (e == cudaSuccess) e = launch_smooth(L, 1, st);
  }
  return e;
}
static MGLevel on_p2(MGLevel L) {
  L.p = L.p2;
  return L;
}
cudaError_t launch_down(const MGLevel* levels, int top, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  for (int i = 0; i < top && e == cudaSuccess; ++i) {
    const MGLevel& L = levels[i];
    const bool two = L.sweep.px > 0;
    e = two ? launch_sweep2(L, L.p, L.p2, i > 0, st) : launch_sweeps(L, 2, st);
    // a level that starts with the two-sweep kernel does not read its pressure
    if (e == cudaSuccess) e = launch_restrict(two ? on_p2(L) : L, levels[i + 1], st, i + 1 == top || levels[i + 1].sweep.px == 0);
  }
  return e;
}
cudaError_t launch_up(const MGLevel* levels, int top, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  for (int i = top - 1; i >= 0 && e == cudaSuccess; --i) {
    const MGLevel& L = levels[i];
    const bool two = L.sweep.px > 0;
    e = launch_prolong(two ? on_p2(L) : L, levels[i + 1], st);
    if (e == cudaSuccess) e = two ? launch_sweep2(L, L.p2, L.p, false, st) : launch_sweeps(L, 2, st);
  }
  return e;
}
cudaError_t sweep_configure() {
  cudaError_t e = cudaSuccess;
  auto opt_in = [&](auto k) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SW_SMEM);
  };
  opt_in(k_sweep2<float, false, false>);
  opt_in(k_sweep2<float, true, false>);
  opt_in(k_sweep2<float, false, true>);
  opt_in(k_sweep2<float, true, true>);
  opt_in(k_sweep2<float, false, false, true>);
  opt_in(k_sweep2<float, true, false, true>);
  opt_in(k_sweep2<float, false, true, true>);
  opt_in(k_sweep2<float, true, true, true>);
  opt_in(k_sweep2_b<false, false>);
  opt_in(k_sweep2_b<true, false>);
  opt_in(k_sweep2_b<false, true>);
  opt_in(k_sweep2_b<true, true>);
  opt_in(k_sweep2<__half, false, false>);
  opt_in(k_sweep2<__half, true, false>);
  opt_in(k_sweep2<__nv_bfloat16, false, false>);
  opt_in(k_sweep2<__nv_bfloat16, true, false>);
  return e;
}

}  // namespace fire
