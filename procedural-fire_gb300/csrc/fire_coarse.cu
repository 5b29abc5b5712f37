// The coarse end of the multigrid V-cycle in one launch, each thread owning a fixed block of cells.
//
// Why it looks like this.  The levels below the ones that fill the GPU are bound by latency, not by bytes: a
// level of 32x64x32 holds 0.5 MB, and a V-cycle visits it in ten dependent phases.  As one launch per phase a
// phase cost 2.1-2.6 us; as a phase of a kernel that recomputes its cells' positions and re-reads every
// neighbour it cost 0.4 us in one CTA and 2.6 us over a cluster.  Here
//   * a thread owns 2 x 4 x 1 cells (2 x 1 x 1 on the smallest levels): both colours at half-index gx, four rows of y, one z.  Their
//     pressure, right-hand side and reciprocal diagonal stay in registers through all phases of a visit, and so do
//     the y neighbours inside the four rows and one x neighbour of every cell;
//   * the pressure is stored split by colour, the four rows of a (gx, z) as one 16-byte element (rows in the order
//     0 2 1 3), so a phase of four updates reads two 8-byte x neighbours, two 16-byte z neighbours and two scalars,
//     all with unit stride over the lanes, and stores one element.  Elements of zeros frame every level in z and
//     y, and an x neighbour outside the row is redirected to one: no face test, a missing neighbour adds 0;
//   * a level of more than CO_LOCAL_CELLS cells is split by rows of y over a thread-block cluster of up to 16 CTAs.  A
//     CTA sends the rows its neighbours read straight into their shared memory right after updating them
//     (st.async, completing on an mbarrier of the receiver), so a phase waits for its two neighbours' rows and not for
//     a barrier of the cluster, whose release costs 0.7 us with the stores in flight;
//   * the levels below are gathered on CTA 0 and synchronised by a named barrier over just the warps that own cells; the
//     coarse rows a CTA's prolongation reads are copied back once.
// The arithmetic of every update, residual and prolongation is that of the launch-per-phase kernels of
// fire_mg.cu, in the same order, written with explicit FMAs, so the cycle is bit-identical to theirs:
// __fdividef(a, d) equals a * rcp.approx(d) bit for bit for the diagonals 3..9 (checked over 2^30 values of a
// for each), and a zero added for a missing neighbour does not change a sum that starts at +0.
//
// Measured (GB300, back to back, us; the forms this replaces: one launch per phase, the single-CTA or 8-CTA tail):
//   one V(2,2) cycle from 32x64x32            21.2   (46: level 0 in launches, tail from 16x32x16)
//   four cycles of it in one launch           73.6   (186)
//   one cycle from 20x30x20, 43 coarse sweeps 24.3; with 40x60x40 on top 42.3 (66): that level runs in launches, see coarse_first
//   64 sweeps of a 25x49x25 coarsest level    59.6   (190: two launches a sweep)
// A phase costs about 0.15 us on one CTA (LDS - six adds - store - barrier) and 0.3 us on a split level, of which half is
// the neighbours' rows in flight; nothing here is near a byte or FLOP limit.
#include <algorithm>
#include <cstring>
#include "fire_device.cuh"
#include "fire_launch.cuh"

namespace fire {
cudaError_t coarse_configure();
namespace {

constexpr int CO_MAX = 12;         // levels
constexpr int CO_SMEM = 224 * 1024;
constexpr int CO_CLUSTER = 16;     // CTAs of the largest cluster (non-portable size; 8 where it cannot be scheduled)
constexpr int CO_LOCAL_CELLS = 2048;

struct CoLevel {
  int nx, ny, nz;
  float h;
  int p;        // float4 offset of the level's pressure (two colours of `arr` elements)
  int b;        // float4 offset of its right-hand side (two colours of `items` elements, one per owning thread)
  int k;        // rows a thread owns: 4, or 1 on a level of one CTA that has the threads for it (shorter phases)
  int runs;     // groups of k rows a CTA's arrays hold
  int halo;     // split levels: float offset of the rows below and above this CTA's (two colours of each)
  int team;     // threads that own cells (or work on a coarser level of the same CTA), rounded up to a warp
  int plain;    // float offset of the pressure in plain order ([row][z][x]; split levels with a row below and above), for the
                // prolongation onto the finer level
  float rhx, rnz;   // 1 / half-row, 1 / nz: (t + 0.5) times them truncates to the quotient exactly for t < 1024
};
struct CoDesc {
  int n;                 // levels
  int nd;                // the first nd are split over the cluster
  int nact;              // CTAs that hold rows of them
  int csize;             // CTAs of the cluster
  CoLevel l[CO_MAX];
  short bound[CO_CLUSTER + 1];   // rows [bound[r], bound[r + 1]) of level `base` are CTA r's
  int base;
  int gather;            // float offset of the right-hand side of level nd in plain order on CTA 0
  int stage;             // float offset of a copy of the rows of level nd's plain pressure that this CTA's prolongation reads
  int scratch;           // float offset: restriction partials, two per thread
  int dsum;              // float offset (even) of the direct solve's partials; its plain right-hand side follows
  float* gp;             // the first level in global memory
  const float* gb;
  int vec;               // gp and gb allow float2 accesses (even nx, 8-byte aligned)
  float omega;
  int coarse;            // sweeps of the coarsest level
  const double* cinv;    // or its dense inverse (transposed), applied in FP64
  int* err;              // set to 1 when a bounded wait runs out
  int polls;             // its limit
};

extern __shared__ float4 co_smem4[];
__device__ __forceinline__ float* co_smem() { return reinterpret_cast<float*>(co_smem4); }   // every function names the array itself, so its accesses are shared-memory ones

// ---- cluster primitives ----
__device__ __forceinline__ unsigned smem32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned map_rank(unsigned addr, unsigned rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster(unsigned addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
// Asynchronous store into another CTA's shared memory that completes 4 bytes on that CTA's mbarrier.
__device__ __forceinline__ void st_async(unsigned addr, float v, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(__float_as_uint(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ float ld_cluster(unsigned addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float rcp_approx(float d) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(d));
  return r;
}
// Rows from the neighbouring CTAs.  Every exchange (one colour after a phase, or both after a load or a prolongation)
// uses the barrier pair of its parity: a neighbour sends exchange i + 1 only after it has received this CTA's exchange i, which
// this CTA sends after arming exchange i's barriers, and it sends i + 2 only after this CTA has finished waiting for i.  The
// threads that read the received rows are those that send the next ones, so a row is never overwritten before it is read.
// Every wait is bounded.  A CTA whose wait runs out reports it and is dead from then on: it runs through the remaining phases on
// what it has and takes part in every barrier of its team and of the cluster, but it arms no barrier (a phase of it may be
// incomplete), waits for no row, stores nothing and, from the next visit of a level on, sends none (until then at most 128 exchanges
// of 4 KB, well inside a barrier's 2^20 pending bytes).  Its neighbours miss its rows and end the same way, sooner than
// their limits, as a late wait looks for a report.  Rows that arrive at a dead CTA are waited for by nobody, so it holds its
// shared memory for CO_LANDING_NS after the cluster's last barrier, when nothing is sent any more.
__shared__ alignas(8) unsigned long long co_bar[2][2];   // [from below, from above][parity]
__shared__ int co_limit;   // polls of a wait; -1: dead (thread 0 sets it before the team's barrier of the phase)
__shared__ int* co_err;
constexpr unsigned long long CO_LANDING_NS = 50000000ull;
__device__ __forceinline__ int wait_limit() { return *(volatile int*)&co_limit; }
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void bar_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_test(unsigned bar, unsigned parity) {
  unsigned done;
  asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
               : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
// Up to `polls` polls, about a second, and 64 polls where a timeout has been reported already.
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity, int polls) {
  if (bar_test(bar, parity) && polls > 0) return true;
  const unsigned long long t0 = global_ns();
  for (int i = 1; i < polls; ++i) {
    if (bar_test(bar, parity)) return true;
    if ((i & 63) == 63 && (global_ns() - t0 > 1000000000ull || *(volatile int*)co_err)) break;
  }
  return false;
}
__device__ __forceinline__ void team_sync(int bar, int team) {
  asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(team) : "memory");
}

// Position of row j of a four-row run inside its element: rows 0 2 1 3.
__device__ __forceinline__ int row_slot(int j) { return ((j & 1) << 1) | ((j >> 1) & 1); }
// Shared memory by byte offset.
__device__ __forceinline__ float* sm_at(int off) { return reinterpret_cast<float*>(reinterpret_cast<char*>(co_smem4) + off); }
// The K rows of an element.
template <int K> __device__ __forceinline__ void sm_read(float (&v)[K], int off) {
  if (K == 4) {
    const float4 q = *reinterpret_cast<const float4*>(sm_at(off));
    v[0] = q.x; v[K > 2 ? 2 : 0] = q.y; v[K > 1 ? 1 : 0] = q.z; v[K > 3 ? 3 : 0] = q.w;
  } else {
    v[0] = *sm_at(off);
  }
}
template <int K> __device__ __forceinline__ void sm_write(const float (&v)[K], int off) {
  if (K == 4) *reinterpret_cast<float4*>(sm_at(off)) = make_float4(v[0], v[K > 2 ? 2 : 0], v[K > 1 ? 1 : 0], v[K > 3 ? 3 : 0]);
  else *sm_at(off) = v[0];
}

// This CTA's part of one level.  Element of (gx, z, run) of colour c: c arr + gx + hx (z + 1 + (nz + 2)(run + 1)), in
// elements of 4 K bytes from byte offset P.
struct Slab {
  int nx, ny, nz, hx, n;   // n: columns (gx, z)
  int plane, arr, items;
  int R, y0, runs;         // rows held, first row, groups of rows
  float h, h2, ih2, omega, rhx, rnz;
  int plain;               // float offset
  int P, B, halo;          // byte offsets; halo (split levels): rows below [c][z][gx], then rows above, in plain order, so that a
                           // warp's remote stores fill whole sectors
  int bar, team;
  unsigned lo, hi;         // shared-memory addresses of the halo rows this CTA's edge rows go to (0: none)
  unsigned lo_bar, hi_bar; // and of the receivers' barriers (parity 0)
};
__shared__ Slab co_slab[CO_MAX];   // one thread per level fills it in, once per launch
__device__ __forceinline__ int row_bound(const CoDesc& D, int l, int r) { return (int)D.bound[min(r, D.nact)] << (D.base - l); }
__device__ __forceinline__ Slab make_slab(const CoDesc& D, int l, int r) {
  const CoLevel& L = D.l[l];
  Slab s;
  s.nx = L.nx; s.ny = L.ny; s.nz = L.nz;
  s.hx = (L.nx + 1) >> 1;
  s.n = s.hx * L.nz;
  s.plane = s.hx * (L.nz + 2);
  s.arr = s.plane * (L.runs + 2);
  s.items = s.n * L.runs;
  s.h = L.h;
  s.h2 = L.h * L.h;
  s.ih2 = 1.0f / (L.h * L.h);
  s.omega = D.omega;
  s.rhx = L.rhx; s.rnz = L.rnz;
  s.plain = L.plain;
  s.P = 16 * L.p;
  s.B = 16 * L.b;
  s.halo = 4 * L.halo;
  s.bar = l + 1;
  s.team = L.team;
  s.lo = s.hi = s.lo_bar = s.hi_bar = 0;
  if (l < D.nd) {
    s.y0 = row_bound(D, l, r);
    s.R = row_bound(D, l, r + 1) - s.y0;
    const unsigned a = smem32(sm_at(s.halo));
    if (r > 0 && r < D.nact) {   // row 0 lies above the CTA below
      s.lo = map_rank(a, r - 1) + 8u * (unsigned)s.n;
      s.lo_bar = map_rank(smem32(&co_bar[1][0]), r - 1);
    }
    if (r + 1 < D.nact) {        // the last row lies below the CTA above
      s.hi = map_rank(a, r + 1);
      s.hi_bar = map_rank(smem32(&co_bar[0][0]), r + 1);
    }
  } else {
    s.y0 = 0;
    s.R = L.ny;
  }
  s.runs = (s.R + L.k - 1) / L.k;
  return s;
}
// Arms exchange `ex` for `colours` colours from each neighbour (thread 0, before this CTA sends its own rows).
template <bool kSplit>
__device__ __forceinline__ void exchange_arm(const Slab& L, int colours, int ex, int limit) {
  if (!kSplit || threadIdx.x != 0 || limit < 0) return;
  const unsigned bytes = 4u * (unsigned)(colours * L.n);
  if (L.lo) bar_expect(smem32(&co_bar[0][ex & 1]), bytes);
  if (L.hi) bar_expect(smem32(&co_bar[1][ex & 1]), bytes);
}
// The end of a phase: the neighbours' rows of exchange `ex` have arrived (warp 0 waits for them; thread 0's wait decides whether
// this CTA is dead), and this CTA's cells and those rows are visible to the level's threads.  limit: the thread's copy of co_limit.
// (A call in place of the inlined loops costs 30 ns a phase.)
template <bool kSplit>
__device__ __forceinline__ void level_sync(const Slab& L, int& ex, int& limit) {
  if (kSplit) {
    if (threadIdx.x < 32) {
      if (limit >= 0) {
        const unsigned parity = (unsigned)(ex >> 1) & 1u;
        if ((L.lo && !bar_wait(smem32(&co_bar[0][ex & 1]), parity, limit)) || (L.hi && !bar_wait(smem32(&co_bar[1][ex & 1]), parity, limit))) {
          limit = -1;
          if (threadIdx.x == 0) {
            *(volatile int*)&co_limit = -1;
            *(volatile int*)co_err = 1;
          }
        }
      }
    }
    ++ex;
  }
  team_sync(L.bar, L.team);
}

// A thread's cells of one level: colour c of row j0 + k at [c][k], x = 2 gx + ((y + z + c) & 1).
template <int K>
struct Own {
  float p[2][K], b[2][K], rd[2][K];
  int gx, z, j0, nv;   // nv: rows owned (0: none)
  int e, item;         // byte offsets of the element in P (colour 0) and in B
  int ex, ey;          // element offsets of the x neighbours of the cells with parity s0 / 1 - s0 (or of an element of zeros)
  int ylo[2], yhi[2];  // byte offsets of the values below row 0 and above row nv - 1, by colour
  int col;             // gx + hx z
  int s0;              // (y0 + j0 + z) & 1: the x parity of colour c at row k is (s0 + k + c) & 1
  bool odd;            // the row ends at an even x: the cell of x parity 1 does not exist
  unsigned mask;       // bit c K + k: the cell exists
  unsigned lo, hi;     // where row 0 / the last row of colour 0 goes in the neighbouring CTA (0: nowhere)
};
template <int K, bool kSplit>
__device__ __forceinline__ void own_cells(Own<K>& o, const Slab& L, int tid) {
  const int q = (int)(((float)tid + 0.5f) * L.rhx);
  o.gx = tid - q * L.hx;
  const int run = (int)(((float)q + 0.5f) * L.rnz);
  o.z = q - run * L.nz;
  o.j0 = run * K;
  o.item = tid;
  o.nv = run < L.runs ? min(K, L.R - o.j0) : 0;
  const bool idle = o.nv == 0;
  if (idle) { o.gx = 0; o.z = 0; o.j0 = 0; o.item = 0; }   // surplus thread: reads stay inside the arrays, nothing is written
  constexpr int S = 4 * K;   // bytes of an element
  const int e = o.gx + L.hx * (o.z + 1) + L.plane * (o.j0 / K + 1);
  const int zero = e - L.hx * (o.z + 1);
  const int left = o.gx > 0 ? e - 1 : zero, right = o.gx < L.hx - 1 ? e + 1 : zero;
  o.e = L.P + S * e;
  o.item = L.B + S * o.item;
  o.s0 = (L.y0 + o.j0 + o.z) & 1;
  o.ex = L.P + S * (o.s0 ? right : left);
  o.ey = L.P + S * (o.s0 ? left : right);
  o.odd = (L.nx & 1) && o.gx == L.hx - 1;
  o.mask = 0u;
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (k < o.nv && !(o.odd && ((o.s0 + k + c) & 1))) o.mask |= 1u << (c * K + k);
  o.col = o.gx + L.hx * o.z;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    o.ylo[c] = L.P + S * (c * L.arr + e - L.plane) + 4 * (K - 1);
    o.yhi[c] = L.P + S * (c * L.arr + e + L.plane);
    if (kSplit && o.j0 == 0) o.ylo[c] = L.halo + 4 * (c * L.n + o.col);
    if (kSplit && o.j0 + o.nv == L.R) o.yhi[c] = L.halo + 4 * ((2 + c) * L.n + o.col);
  }
  const unsigned col = 4u * (unsigned)o.col;
  o.lo = L.lo && !idle && o.j0 == 0 ? L.lo + col : 0u;
  o.hi = L.hi && !idle && o.j0 + o.nv == L.R ? L.hi + col : 0u;
}
// Reciprocal diagonals: open sides and top add 1 to 6, the floor subtracts 1 (rb_update's ghost rules).
template <int K>
__device__ __forceinline__ void own_diag(Own<K>& o, const Slab& L) {
  const float dz = 6.0f + (o.z == 0 ? 1.0f : 0.0f) + (o.z == L.nz - 1 ? 1.0f : 0.0f);
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int y = L.y0 + o.j0 + k;
    const float dy = dz + (y == L.ny - 1 ? 1.0f : 0.0f) - (y == 0 ? 1.0f : 0.0f);
    const float d0 = dy + (o.gx == 0 ? 1.0f : 0.0f) + (2 * o.gx == L.nx - 1 ? 1.0f : 0.0f);   // at the even x
    const float d1 = dy + (2 * o.gx + 1 == L.nx - 1 ? 1.0f : 0.0f);
    const bool s = (o.s0 + k) & 1;   // colour 0 sits at the odd x
    const float r0 = rcp_approx(d0), r1 = rcp_approx(d1);
    o.rd[0][k] = s ? r1 : r0;
    o.rd[1][k] = s ? r0 : r1;
  }
}
template <int K>
__device__ __forceinline__ void own_zero(Own<K>& o) {
#pragma unroll
  for (int k = 0; k < K; ++k) o.p[0][k] = o.p[1][k] = 0.0f;
}
template <int K>
__device__ __forceinline__ void own_read_p(Own<K>& o, const Slab& L) {
  sm_read<K>(o.p[0], o.e);
  sm_read<K>(o.p[1], o.e + 4 * K * L.arr);
  if (o.nv == 0) own_zero(o);
}
template <int K>
__device__ __forceinline__ void own_read_b(const CoDesc& D, int l, Own<K>& o, const Slab& L) {
  if (l == D.nd && l > 0) {   // the gathered level: the right-hand side arrived in plain order
    const float* G = co_smem() + D.gather;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      float v[2] = {0.0f, 0.0f};
      if (k < o.nv) {
        const float* g = G + 2 * o.gx + L.nx * (o.z + L.nz * (o.j0 + k));
        v[0] = g[0];
        if (!o.odd) v[1] = g[1];
      }
      const bool s = (o.s0 + k) & 1;   // colour 0 sits at the odd x
      o.b[0][k] = s ? v[1] : v[0];
      o.b[1][k] = s ? v[0] : v[1];
    }
  } else {
    sm_read<K>(o.b[0], o.item);
    sm_read<K>(o.b[1], o.item + 4 * K * L.items);
  }
}
// The level's pressure in plain order for the prolongation onto the finer level; on a split level with the neighbouring CTAs' rows.
template <int K, bool kSplit>
__device__ __forceinline__ void publish(const Own<K>& o, const Slab& L) {
  if (o.nv == 0) return;
  float* G = co_smem() + L.plain;
  const int row = L.nx * L.nz, at = 2 * o.gx + L.nx * o.z;
  auto put = [&](int r, float a, float b) {   // the cells of even and odd x
    G[at + row * r] = a;
    if (!o.odd) G[at + row * r + 1] = b;
  };
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (k < o.nv) {
      const bool s = (o.s0 + k) & 1;   // colour 0 sits at the odd x
      put(o.j0 + k + (kSplit ? 1 : 0), s ? o.p[1][k] : o.p[0][k], s ? o.p[0][k] : o.p[1][k]);
    }
  if (kSplit) {
    const float* H = sm_at(L.halo) + o.col;
    if (o.j0 == 0) {
      const bool s = !(o.s0 & 1);   // row -1
      put(0, s ? H[L.n] : H[0], s ? H[0] : H[L.n]);
    }
    if (o.j0 + o.nv == L.R) {
      const bool s = (o.s0 + o.nv) & 1;
      put(L.R + 1, s ? H[3 * L.n] : H[2 * L.n], s ? H[2 * L.n] : H[3 * L.n]);
    }
  }
}
// Writes colour c (cells that do not exist as zeros) and sends a split level's edge rows to the neighbouring CTAs.
template <int K, bool kSplit>
__device__ __forceinline__ void own_write(Own<K>& o, const Slab& L, int c, int ex) {
  float last = o.p[c][K - 1];
  if (o.mask != (1u << (2 * K)) - 1u) {
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (!(o.mask & (1u << (c * K + k)))) o.p[c][k] = 0.0f;
    if (K == 4 && kSplit) last = o.nv == 4 ? o.p[c][K - 1] : o.nv == 3 ? o.p[c][K > 2 ? 2 : 0] : o.nv == 2 ? o.p[c][K > 1 ? 1 : 0] : o.p[c][0];
  }
  if (o.nv > 0) sm_write<K>(o.p[c], o.e + 4 * K * c * L.arr);
  if (kSplit) {
    const unsigned ca = 4u * (unsigned)(c * L.n), par = 8u * (unsigned)(ex & 1);
    if (o.lo) st_async(o.lo + ca, o.p[c][0], L.lo_bar + par);
    if (o.hi) st_async(o.hi + ca, last, L.hi_bar + par);
  }
}
// The neighbours of colour c's cells: the x neighbour away from the thread's own pair, below and above in z and in y.
template <int K>
struct Nbr { float far[K], zm[K], zp[K], ylo, yhi; };
template <int K>
__device__ __forceinline__ void read_nbr(Nbr<K>& n, const Own<K>& o, const Slab& L, int c) {
  const int other = c == 0 ? 4 * K * L.arr : 0;   // the colour that is read
  const int a = (c == 0 ? o.ex : o.ey) + other, b = (c == 0 ? o.ey : o.ex) + other;
  if (K == 4) {   // rows 0 and 2 look to one side, 1 and 3 to the other
    const float2 u = *reinterpret_cast<const float2*>(sm_at(a)), v = *reinterpret_cast<const float2*>(sm_at(b + 8));
    n.far[0] = u.x; n.far[K > 2 ? 2 : 0] = u.y; n.far[K > 1 ? 1 : 0] = v.x; n.far[K > 3 ? 3 : 0] = v.y;
    if (K == 1) n.far[0] = u.x;
  } else {
    n.far[0] = *sm_at(a);
  }
  sm_read<K>(n.zm, o.e + other - 4 * K * L.hx);
  sm_read<K>(n.zp, o.e + other + 4 * K * L.hx);
  n.ylo = *sm_at(o.ylo[1 - c]);
  n.yhi = *sm_at(o.yhi[1 - c]);
}
template <int K>
__device__ __forceinline__ float nbr_ym(const Own<K>& o, const Nbr<K>& n, int c, int k) { return k > 0 ? o.p[1 - c][k > 0 ? k - 1 : 0] : n.ylo; }
template <int K>
__device__ __forceinline__ float nbr_yp(const Own<K>& o, const Nbr<K>& n, int c, int k) {
  return k + 1 == K || k + 1 == o.nv ? n.yhi : o.p[1 - c][k + 1 < K ? k + 1 : k];
}
// One colour of a red-black sweep (mgSmooth, src/sim.js:417-437; the order of rb_update in fire_mg.cu; the sum of the two x
// neighbours, which starts at +0, is the same in either order).  zero: the level's pressure is zero, so only the right-hand side counts.
template <int K, bool kSplit, bool kRelax>
__device__ __forceinline__ void sweep_colour(Own<K>& o, const Slab& L, int c, bool zero, int ex, int limit) {
  exchange_arm<kSplit>(L, 1, ex, limit);
  if (zero) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      float v = __fmul_rn(__fmaf_rn(-L.h2, o.b[c][k], 0.0f), o.rd[c][k]);
      if (kRelax) v = __fmaf_rn(L.omega, v, 0.0f);
      o.p[c][k] = v;
    }
  } else {
    Nbr<K> n;
    read_nbr(n, o, L, c);
#pragma unroll
    for (int k = 0; k < K; ++k) {
      float sum = __fadd_rn(__fadd_rn(0.0f, o.p[1 - c][k]), n.far[k]);
      sum = __fadd_rn(sum, n.zm[k]);
      sum = __fadd_rn(sum, n.zp[k]);
      sum = __fadd_rn(sum, nbr_ym(o, n, c, k));
      sum = __fadd_rn(sum, nbr_yp(o, n, c, k));
      const float t = __fmaf_rn(-L.h2, o.b[c][k], sum);
      // relaxed: the change t rd - p takes one rounding, as the single launches' contracted form does
      o.p[c][k] = kRelax ? __fmaf_rn(L.omega, __fmaf_rn(t, o.rd[c][k], -o.p[c][k]), o.p[c][k]) : __fmul_rn(t, o.rd[c][k]);
    }
  }
  own_write<K, kSplit>(o, L, c, ex);
}
template <int K, bool kSplit, bool kRelax>
__device__ __forceinline__ void sweeps(Own<K>& o, const Slab& L, int iters, bool zero, int& ex, int& limit) {
  for (int it = 0; it < iters; ++it) {
    sweep_colour<K, kSplit, kRelax>(o, L, 0, zero && it == 0, ex, limit);
    level_sync<kSplit>(L, ex, limit);
    sweep_colour<K, kSplit, kRelax>(o, L, 1, false, ex, limit);
    level_sync<kSplit>(L, ex, limit);
  }
}
// The first level between global memory and the threads' registers.
template <int K, bool kSplit>
__device__ __forceinline__ void load_global(const CoDesc& D, Own<K>& o, const Slab& L, int ex, int limit) {
  exchange_arm<kSplit>(L, 2, ex, limit);
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const size_t g = 2 * (size_t)o.gx + (size_t)L.nx * ((L.y0 + o.j0 + k) + (size_t)L.ny * o.z);
    float2 p = make_float2(0.0f, 0.0f), b = p;
    if (k < o.nv) {
      if (D.vec) {
        p = *reinterpret_cast<const float2*>(D.gp + g);
        b = *reinterpret_cast<const float2*>(D.gb + g);
      } else {
        p.x = D.gp[g];
        b.x = D.gb[g];
        if (!o.odd) { p.y = D.gp[g + 1]; b.y = D.gb[g + 1]; }
      }
    }
    const bool s = (o.s0 + k) & 1;   // colour 0 sits at the odd x
    o.p[0][k] = s ? p.y : p.x; o.p[1][k] = s ? p.x : p.y;
    o.b[0][k] = s ? b.y : b.x; o.b[1][k] = s ? b.x : b.y;
  }
  if (o.nv > 0) {
    sm_write<K>(o.b[0], o.item);
    sm_write<K>(o.b[1], o.item + 4 * K * L.items);
  }
  own_write<K, kSplit>(o, L, 0, ex);
  own_write<K, kSplit>(o, L, 1, ex);
}
template <int K>
__device__ __forceinline__ void store_global(const CoDesc& D, const Own<K>& o, const Slab& L) {
#pragma unroll
  for (int k = 0; k < K; ++k) {
    if (k >= o.nv) continue;
    const size_t g = 2 * (size_t)o.gx + (size_t)L.nx * ((L.y0 + o.j0 + k) + (size_t)L.ny * o.z);
    const bool s = (o.s0 + k) & 1;
    const float2 p = make_float2(s ? o.p[1][k] : o.p[0][k], s ? o.p[0][k] : o.p[1][k]);
    if (D.vec) *reinterpret_cast<float2*>(D.gp + g) = p;
    else {
      D.gp[g] = p.x;
      if (!o.odd) D.gp[g + 1] = p.y;
    }
  }
}

// Residual of the thread's cells (restrict_cell's ghosts and order, fire_mg.cu); at [x parity][row].  A level that is
// restricted has an even nx, so both cells of a pair exist.
template <int K>
__device__ __forceinline__ void residuals(const Own<K>& o, const Slab& L, float (&r)[2][K]) {
  const bool z0 = o.z == 0, z1 = o.z == L.nz - 1, y0 = L.y0 + o.j0 == 0, y1 = L.y0 + o.j0 + o.nv == L.ny;
  const bool faces[2] = {o.gx == 0, o.gx == L.hx - 1};   // the far x neighbour of a cell of x parity s lies outside
  const bool face0 = o.s0 ? faces[1] : faces[0], face1 = o.s0 ? faces[0] : faces[1];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    Nbr<K> n;
    read_nbr(n, o, L, c);
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const float me = o.p[c][k];
      const float far = (((k + c) & 1) ? face1 : face0) ? -me : n.far[k];
      const float ym = k == 0 && y0 ? me : nbr_ym(o, n, c, k);
      const float up = nbr_yp(o, n, c, k), yp = y1 && k + 1 == o.nv ? -me : up;
      const float zm = z0 ? -me : n.zm[k], zp = z1 ? -me : n.zp[k];
      const float sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(o.p[1 - c][k], far), ym), yp), zm), zp);
      r[c][k] = __fmaf_rn(-__fmaf_rn(-6.0f, me, sum), L.ih2, o.b[c][k]);
    }
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const bool s = (o.s0 + k) & 1;
    const float t = r[0][k];
    r[0][k] = s ? r[1][k] : t;
    r[1][k] = s ? t : r[1][k];
  }
}
// Where a restricted value goes: the coarse right-hand side of this CTA, or CTA 0's plain array when the coarse level is gathered.
struct CoarseOut {
  int nx, nz, hx, items, k, base;   // byte offset base
  bool gather;
  unsigned remote;
  __device__ __forceinline__ void put(int cx, int cy, int cz, int row, float v) const {
    int i;
    if (gather) i = cx + nx * (cz + nz * cy);
    else {
      const int c = (cx + cy + cz) & 1, col = (cx >> 1) + hx * cz;
      i = k == 4 ? 4 * (c * items + col + hx * nz * (row >> 2)) + row_slot(row & 3) : c * items + col + hx * nz * row;
    }
    if (remote) st_cluster(remote + 4u * (unsigned)i, v);
    else sm_at(base)[i] = v;
  }
};
__device__ __forceinline__ CoarseOut coarse_out(const CoDesc& D, int l, int rank) {
  const CoLevel& C = D.l[l + 1];
  CoarseOut w;
  w.nx = C.nx; w.nz = C.nz; w.hx = (C.nx + 1) >> 1; w.items = w.hx * C.nz * C.runs; w.k = C.k;
  w.gather = l + 1 == D.nd;
  w.base = w.gather ? 4 * D.gather : 16 * C.b;
  w.remote = w.gather && rank != 0 ? map_rank(smem32(sm_at(w.base)), 0) : 0u;
  return w;
}
// Restriction (src/sim.js:439-466): the mean residual of the 8 children, summed x, then y, then z.  K = 4: the x and y
// children of a coarse cell are one thread's; the thread of the odd z continues the even z's partial sum.  K = 1: the
// thread of the odd y and z adds the four threads' pairs.
template <int K, bool kSplit>
__device__ __forceinline__ void restrict_level(const CoDesc& D, int l, const Own<K>& o, const Slab& L, int tid, int rank) {
  float r[2][K];
  residuals(o, L, r);
  float2* part = reinterpret_cast<float2*>(co_smem() + D.scratch);
  const CoarseOut out = coarse_out(D, l, rank);
  if (K == 4) {
    auto add4 = [&](float a, int k) {
      return __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(a, r[0][k % K]), r[1][k % K]), r[0][(k + 1) % K]), r[1][(k + 1) % K]);
    };
    if (!(o.z & 1) && o.nv > 0) part[tid] = make_float2(add4(0.0f, 0), add4(0.0f, 2));
    team_sync(L.bar, L.team);
    if ((o.z & 1) && o.nv > 0) {
      const float2 even = part[tid - L.hx];
      const float sum[2] = {__fmul_rn(add4(even.x, 0), 0.125f), __fmul_rn(add4(even.y, 2), 0.125f)};
#pragma unroll
      for (int m = 0; m < 2; ++m)
        if (2 * m < o.nv) {
          const int cj = (o.j0 >> 1) + m;
          out.put(o.gx, (L.y0 >> 1) + cj, o.z >> 1, cj, sum[m]);
        }
    }
  } else {
    if (o.nv > 0) part[tid] = make_float2(r[0][0], r[1][0]);
    team_sync(L.bar, L.team);
    if ((o.z & 1) && (o.j0 & 1) && o.nv > 0) {
      float a = 0.0f;
#pragma unroll
      for (int q = 0; q < 4; ++q) {   // y fastest
        const float2 v = part[tid - ((q & 1) ? 0 : L.n) - ((q & 2) ? 0 : L.hx)];
        a = __fadd_rn(__fadd_rn(a, v.x), v.y);
      }
      const int cj = o.j0 >> 1;
      out.put(o.gx, (L.y0 >> 1) + cj, o.z >> 1, cj, __fmul_rn(a, 0.125f));
    }
  }
  if (!out.gather) team_sync(L.bar, L.team);   // (a gathered level's rows are waited for by the caller)
}
// Prolongation (src/sim.js:468-495) of the coarse correction onto this thread's cells: prolong_cell's weights, mirror
// signs and order.  G: the coarse pressure in plain order, shifted so that coarse row cy is at G + nx nz cy.
template <int K>
__device__ __forceinline__ void prolong_level(Own<K>& o, const Slab& L, const CoLevel& C, const float* G) {
  constexpr int M = K == 4 ? 4 : 2;   // coarse rows read
  const int y = L.y0 + o.j0, dz = o.z & 1;
  const int j = K == 4 ? (y >> 1) - 1 : (y >> 1) - 1 + (y & 1);
  const float wz[2] = {dz ? 0.75f : 0.25f, dz ? 0.25f : 0.75f};
  const float wy1[2] = {(y & 1) ? 0.75f : 0.25f, (y & 1) ? 0.25f : 0.75f};   // K = 1: the row's own parity
  const int last = (L.y0 >> 1) + (L.R >> 1);   // rows past the one above the CTA's own are not held (and only read by surplus rows)
  const float sx[2] = {o.gx > 0 ? 1.0f : -1.0f, o.gx < C.nx - 1 ? 1.0f : -1.0f};   // mirror signs: -1 outside the sides and the top
  const int xl = max(o.gx - 1, 0), xr = min(o.gx + 1, C.nx - 1);
  float acc[2][K];   // [x parity][row]
#pragma unroll
  for (int k = 0; k < K; ++k) acc[0][k] = acc[1][k] = 0.0f;
#pragma unroll
  for (int oz = 0; oz < 2; ++oz) {
    float v[M][3];
    const int qz = (o.z >> 1) - 1 + dz + oz, cz = min(max(qz, 0), C.nz - 1);
    const float sz = qz == cz ? 1.0f : -1.0f;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int qy = j + m, cy = min(min(max(qy, 0), C.ny - 1), last);
      const float s = qy >= C.ny ? -sz : sz;
      const float* g = G + C.nx * (cz + C.nz * cy);
      v[m][0] = g[xl] * (s * sx[0]);
      v[m][1] = g[o.gx] * s;
      v[m][2] = g[xr] * (s * sx[1]);
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int dx = 0; dx < 2; ++dx)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int ox = q & 1, oy = q >> 1, dy = k & 1;   // child 0: 1/4 below, 3/4 here; child 1: 3/4 here, 1/4 above
          const float wx = dx == ox ? 0.25f : 0.75f, wy = K == 4 ? (dy == oy ? 0.25f : 0.75f) : wy1[oy];
          const int m = K == 4 ? (k >> 1) + dy + oy : oy;
          acc[dx][k] = __fmaf_rn(__fmul_rn(__fmul_rn(v[m][dx + ox], wx), wy), wz[oz], acc[dx][k]);
        }
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const bool s = (o.s0 + k) & 1;
    o.p[0][k] = __fadd_rn(o.p[0][k], s ? acc[1][k] : acc[0][k]);
    o.p[1][k] = __fadd_rn(o.p[1][k], s ? acc[0][k] : acc[1][k]);
  }
}

// Exact coarsest solve in FP64, p = A^-1 b: 1024 / n column chunks per row, their partial sums added in order (the
// arithmetic of tail_direct_fp64_cta in fire_mg.cu, whatever the thread count).  A hierarchy of this one level (5x5x5, 6x12x6) has
// its right-hand side and its result in global memory.
__device__ __noinline__ void coarsest_direct(const CoDesc& D, int tid, int nthreads) {
  const int l = D.n - 1, k4 = D.l[l].k == 4;
  const Slab L = co_slab[l];
  const int n = L.nx * L.ny * L.nz, chunks = 1024 / n;
  const bool plain = l == D.nd && l > 0;   // the gathered level
  double* part = reinterpret_cast<double*>(co_smem() + D.dsum);
  float* b = co_smem() + D.dsum + 2 * 1024;
  for (int t = tid; t < n; t += nthreads) {
    const int x = t % L.nx, q = t / L.nx, y = q % L.ny, z = q / L.ny, c = (x + y + z) & 1, col = (x >> 1) + L.hx * z;
    b[t] = l == 0  ? D.gb[t]
           : plain ? co_smem()[D.gather + x + L.nx * (z + L.nz * y)]
                   : sm_at(L.B)[k4 ? 4 * (c * L.items + col + L.n * (y >> 2)) + row_slot(y & 3) : c * L.items + col + L.n * y];
  }
  team_sync(L.bar, L.team);
  for (int t = tid; t < n * chunks; t += nthreads) {
    const int i = t % n, k = t / n;
    double a0 = 0.0, a1 = 0.0;
    int j = k;
    for (; j + chunks < n; j += 2 * chunks) {
      a0 = fma(__ldg(D.cinv + (size_t)j * n + i), (double)b[j], a0);
      a1 = fma(__ldg(D.cinv + (size_t)(j + chunks) * n + i), (double)b[j + chunks], a1);
    }
    if (j < n) a0 = fma(__ldg(D.cinv + (size_t)j * n + i), (double)b[j], a0);
    part[k * n + i] = a0 + a1;
  }
  team_sync(L.bar, L.team);
  for (int t = tid; t < n; t += nthreads) {
    double s = 0.0;
    for (int k = 0; k < chunks; ++k) s += part[k * n + t];
    const int x = t % L.nx, q = t / L.nx, y = q % L.ny, z = q / L.ny, c = (x + y + z) & 1, col = (x >> 1) + L.hx * (z + 1);
    sm_at(L.P)[k4 ? 4 * (c * L.arr + col + L.plane * ((y >> 2) + 1)) + row_slot(y & 3) : c * L.arr + col + L.plane * (y + 1)] = (float)s;
    if (l > 0) co_smem()[L.plain + x + L.nx * (z + L.nz * y)] = (float)s;
    else D.gp[t] = (float)s;
  }
  team_sync(L.bar, L.team);
}

// Pre-smoothing and restriction of level l, or the coarsest level's sweeps.  Its cells come from global memory (the first level's
// first cycle), from shared memory (its later cycles), or are zero with the restricted right-hand side.
template <int K, bool kSplit, bool kRelax>
__device__ __forceinline__ void down(const CoDesc& D, int l, int tid, int rank, int pre, bool load, bool store, int ex) {
  const Slab L = co_slab[l];
  int limit = kSplit ? wait_limit() : 0;
  Own<K> o;
  own_cells<K, kSplit>(o, L, tid);
  if (limit < 0) o.lo = o.hi = 0u;   // a dead CTA sends no rows any more
  if (load) {
    load_global<K, kSplit>(D, o, L, ex, limit);
  } else {
    if (l == 0) own_read_p(o, L);
    else own_zero(o);
    own_read_b(D, l, o, L);
  }
  own_diag(o, L);
  if (load) level_sync<kSplit>(L, ex, limit);
  const bool last = l == D.n - 1;
  sweeps<K, kSplit, kRelax>(o, L, last ? D.coarse : pre, l > 0, ex, limit);
  if (!last) restrict_level<K, kSplit>(D, l, o, L, tid, rank);
  else if (l > 0) publish<K, kSplit>(o, L);
  if (last && store && (!kSplit || wait_limit() >= 0)) store_global(D, o, L);
}
// Prolongation onto level l and post-smoothing; the first level's pressure goes back to global memory.
template <int K, bool kSplit, bool kRelax>
__device__ __forceinline__ void up(const CoDesc& D, int l, int tid, int rank, int post, bool store, int ex) {
  const Slab L = co_slab[l];
  int limit = kSplit ? wait_limit() : 0;
  Own<K> o;
  own_cells<K, kSplit>(o, L, tid);
  if (limit < 0) o.lo = o.hi = 0u;   // a dead CTA sends no rows any more
  own_read_p(o, L);
  const CoLevel& C = D.l[l + 1];
  // rows from cy0 - 1 on for a split level (the staged copy when the coarse level is gathered), from 0 on otherwise
  const int plain = kSplit && l + 1 == D.nd ? D.stage : C.plain;
  prolong_level(o, L, C, co_smem() + plain - (kSplit ? C.nx * C.nz * ((L.y0 >> 1) - 1) : 0));
  exchange_arm<kSplit>(L, 2, ex, limit);
  own_write<K, kSplit>(o, L, 0, ex);
  own_write<K, kSplit>(o, L, 1, ex);
  own_read_b(D, l, o, L);
  own_diag(o, L);
  level_sync<kSplit>(L, ex, limit);
  sweeps<K, kSplit, kRelax>(o, L, post, false, ex, limit);
  if (l > 0) publish<K, kSplit>(o, L);
  if (store && (!kSplit || wait_limit() >= 0)) store_global(D, o, L);
}

template <bool kRelax>
__device__ __forceinline__ void coarse_body(const CoDesc& D, int smem_floats, int pre, int post, int cycles) {
  const int tid = threadIdx.x, T = blockDim.x, n = D.n, nd = D.nd;
  const int rank = D.csize > 1 ? (int)cluster_rank() : 0;
  if (tid < n) co_slab[tid] = make_slab(D, tid, rank);
  if (tid == 0) {
    co_limit = D.polls;
    co_err = D.err;
    for (int i = 0; i < 4; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem32(&co_bar[i >> 1][i & 1])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int t = tid; t < smem_floats / 4; t += T) co_smem4[t] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);   // frames of zeros
  pdl_wait();
  pdl_trigger();
  if (D.csize > 1) cluster_sync();   // no CTA sends to a neighbour that is still clearing its arrays
  else __syncthreads();
  int ex = 0;   // exchanges so far
  for (int cyc = 0; cyc < cycles; ++cyc) {
    const bool load = cyc == 0, store = cyc == cycles - 1;
    for (int l = 0; l < n; ++l) {
      if (l == nd && nd > 0) cluster_sync();   // the gathered right-hand side is complete
      const int ex0 = ex;   // every thread counts a split level's exchanges, also one that owns no cells of it
      if (l < nd) ex += (load && l == 0 ? 1 : 0) + 2 * (l == n - 1 ? D.coarse : pre);
      if ((l >= nd && rank != 0) || tid >= D.l[l].team) continue;
      if (l == n - 1 && D.cinv) coarsest_direct(D, tid, T);
      else if (l < nd) down<4, true, kRelax>(D, l, tid, rank, pre, load && l == 0, store && n == 1, ex0);
      else if (D.l[l].k == 4) down<4, false, kRelax>(D, l, tid, rank, pre, load && l == 0, store && n == 1, ex0);
      else down<1, false, kRelax>(D, l, tid, rank, pre, load && l == 0, store && n == 1, ex0);
    }
    for (int l = n - 2; l >= 0; --l) {
      if (l == nd - 1) {
        cluster_sync();
        // the coarse rows this CTA's prolongation reads (its own and one on each side): a contiguous piece of CTA 0's array
        const CoLevel& C = D.l[nd];
        const int row = C.nx * C.nz;
        const int y0 = row_bound(D, l, rank) >> 1, y1 = row_bound(D, l, rank + 1) >> 1;
        const int a = max(y0 - 1, 0) * row, b = min(y1 + 1, C.ny) * row;
        const unsigned src = map_rank(smem32(co_smem() + C.plain), 0);
        float* st = co_smem() + D.stage - (y0 - 1) * row;
        if (y1 > y0)
          for (int t = a + tid; t < b; t += T) st[t] = ld_cluster(src + 4u * (unsigned)t);
        __syncthreads();
      }
      const int ex0 = ex;
      if (l < nd) ex += 1 + 2 * post;
      if ((l >= nd && rank != 0) || tid >= D.l[l].team) continue;
      if (l != nd - 1) team_sync(l + 1, D.l[l].team);   // the coarser level's threads are done
      if (l < nd) up<4, true, kRelax>(D, l, tid, rank, post, store && l == 0, ex0);
      else if (D.l[l].k == 4) up<4, false, kRelax>(D, l, tid, rank, post, store && l == 0, ex0);
      else up<1, false, kRelax>(D, l, tid, rank, post, store && l == 0, ex0);
    }
  }
  const bool dead = tid == 0 && wait_limit() < 0;
  if (D.csize > 1) cluster_sync();   // a CTA's shared memory outlives its neighbours' stores into it
  if (dead) {
    const unsigned long long t0 = global_ns();
    for (int i = 0; i < TAIL_WAIT_POLLS && global_ns() - t0 < CO_LANDING_NS; ++i) __nanosleep(1000);
  }
}

// T: the most threads a CTA is launched with, and so its registers per thread (128 / 72 / 64).
template <int T, bool kRelax>
__global__ void __launch_bounds__(T, 1) k_coarse(const __grid_constant__ CoDesc D, int smem_floats, int pre, int post, int cycles) {
  coarse_body<kRelax>(D, smem_floats, pre, post, cycles);
}
// The coarse ends of many simulations, one cluster each; every member has its own omega.
template <int T>
__global__ void __launch_bounds__(T, 1) k_coarse_b(const CoDesc* __restrict__ descs, int csize, int smem_floats, int pre, int post) {
  __shared__ CoDesc D;
  const int* src = reinterpret_cast<const int*>(descs + blockIdx.x / csize);
  for (int t = threadIdx.x; t < (int)(sizeof(CoDesc) / sizeof(int)); t += blockDim.x) reinterpret_cast<int*>(&D)[t] = src[t];
  __syncthreads();
  if (D.omega == 1.0f) coarse_body<false>(D, smem_floats, pre, post, 1);
  else coarse_body<true>(D, smem_floats, pre, post, 1);
}
constexpr int CO_THREADS[3] = {512, 832, 1024};
template <class F> auto with_kernel(int threads, bool relax, F&& f) {
  if (threads <= CO_THREADS[0]) return relax ? f(k_coarse<CO_THREADS[0], true>) : f(k_coarse<CO_THREADS[0], false>);
  if (threads <= CO_THREADS[1]) return relax ? f(k_coarse<CO_THREADS[1], true>) : f(k_coarse<CO_THREADS[1], false>);
  return relax ? f(k_coarse<CO_THREADS[2], true>) : f(k_coarse<CO_THREADS[2], false>);
}

// The largest cluster the device schedules with the kernels' full shared memory: 16 CTAs, a non-portable size, or 8.
int cluster_size() {
  static const int size = [] {
    int best = 1;
    if (coarse_configure() != cudaSuccess) return best;
    for (int c : {8, CO_CLUSTER}) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(c);
      cfg.blockDim = dim3(1024);
      cfg.dynamicSmemBytes = CO_SMEM;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = c;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, k_coarse<CO_THREADS[2], false>, &cfg) == cudaSuccess && clusters > 0) best = c;
      else cudaGetLastError();
    }
    return best;
  }();
  return size;
}

// Lays out levels [first, n) with the first nd split over `csize` CTAs; threads: what the CTA needs.
bool plan_with(const MGLevel* levels, int first, int n, bool direct, int nd, int csize, CoDesc& D, size_t& smem, int& threads) {
  const int cnt = n - first;
  std::memset(&D, 0, sizeof D);
  D.n = cnt; D.nd = nd; D.csize = nd > 0 ? csize : 1;
  D.base = nd < cnt ? nd : cnt - 1;
  const int nb = levels[first + D.base].ny;
  if (nb > 32767) return false;
  D.nact = nd > 0 ? std::min(D.csize, nb) : 1;
  for (int r = 0; r <= D.nact; ++r) D.bound[r] = (short)((long)nb * r / D.nact);
  int off = 0;   // float4 units
  threads = 128;
  for (int l = 0; l < cnt; ++l) {
    const MGLevel& M = levels[first + l];
    CoLevel& L = D.l[l];
    L.nx = M.nx; L.ny = M.ny; L.nz = M.nz; L.h = M.h;
    L.rhx = 1.0f / (float)((M.nx + 1) / 2);
    L.rnz = 1.0f / (float)M.nz;
    const int rows = l < nd ? ((nb + D.nact - 1) / D.nact) << (D.base - l) : M.ny;
    const long columns = (long)((M.nx + 1) / 2) * M.nz;
    L.k = l >= nd && columns * rows <= 512 ? 1 : 4;
    L.runs = (rows + L.k - 1) / L.k;
    if (columns * L.runs > 1024) return false;
    L.team = (int)(columns * L.runs + 31) / 32 * 32;
    threads = std::max(threads, L.team);
    L.p = off;
    auto float4s = [&](long elements) { return (int)((elements * L.k + 3) / 4); };
    off += float4s(2L * ((M.nx + 1) / 2) * (M.nz + 2) * (L.runs + 2));
    L.b = off;
    off += float4s(2 * columns * L.runs);
    if (l < nd) {
      L.halo = 4 * off;
      off += (int)columns;
    }
    if (l > 0) {
      L.plain = 4 * off;
      off += (M.nx * M.nz * (rows + (l < nd ? 2 : 0)) + 3) / 4;
    }
  }
  for (int l = cnt - 2; l >= 0; --l)
    if (l != nd - 1) D.l[l].team = std::max(D.l[l].team, D.l[l + 1].team);
  if (direct) {   // the whole CTA applies the inverse
    threads = std::max(threads, 512);
    for (int l = nd; l < cnt; ++l) D.l[l].team = threads;
  }
  off *= 4;      // floats from here on
  if (nd > 0 && nd < cnt) {
    const MGLevel& M = levels[first + nd];
    D.gather = off;
    off += M.nx * M.ny * M.nz;
    D.stage = off;
    off += ((nb + D.nact - 1) / D.nact + 2) * M.nx * M.nz;
  }
  off = (off + 3) & ~3;
  D.scratch = off;
  off += 2 * threads;
  if (direct) {
    D.dsum = off;
    off += 2 * 1024 + 512;
  }
  off = (off + 3) & ~3;
  smem = sizeof(float) * (size_t)off;
  return smem <= CO_SMEM;
}
// The plan for [first, n): levels of more than CO_LOCAL_CELLS cells split over the cluster, more when they do not fit.
// (8192 cells of 16x32x16 on one CTA: 0.7 us a phase, the SM's issue rate; split over 16: 0.3.  1024 cells of 8x16x8: 0.14
// on one CTA.)
bool make_plan(const MGLevel* levels, int first, int n, bool direct, CoDesc& D, size_t& smem, int& threads) {
  const int cnt = n - first;
  if (first < 0 || cnt < 1 || cnt > CO_MAX || levels[first].study) return false;
  if (direct && (long)levels[n - 1].nx * levels[n - 1].ny * levels[n - 1].nz > 512) return false;
  auto cells = [&](int l) { return (long)levels[first + l].nx * levels[first + l].ny * levels[first + l].nz; };
  int nd = 0;
  if (cluster_size() >= 2)
    while (nd < cnt && cells(nd) > CO_LOCAL_CELLS && !(direct && nd == cnt - 1)) ++nd;
  for (; nd <= cnt; ++nd) {
    if (nd > 0 && cluster_size() < 2) return false;
    if (nd == cnt && direct) return false;   // the inverse is applied by one CTA
    if (plan_with(levels, first, n, direct, nd, cluster_size(), D, smem, threads)) return true;
  }
  return false;
}
void fill_plan(CoDesc& D, const MGLevel* levels, int first, int coarse, const double* cinv, int* err, int polls) {
  D.err = err;
  D.polls = polls;
  D.gp = levels[first].p;
  D.gb = levels[first].b;
  D.vec = levels[first].nx % 2 == 0 && ((reinterpret_cast<uintptr_t>(D.gp) | reinterpret_cast<uintptr_t>(D.gb)) & 7u) == 0;
  D.omega = levels[first].omega;
  D.coarse = coarse;
  D.cinv = cinv;
}
template <class K, class... A>
cudaError_t launch_clusters(K kernel, int csize, int count, int threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(csize * count);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = csize;
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = csize > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace

int coarse_first(const MGLevel* levels, int n, bool direct) {
  CoDesc D;
  size_t smem;
  int threads, first = n;
  // A level that needs more than 512 threads a CTA leaves a thread too few registers: 40x60x40 on top of 20x30x20 costs 18 us a
  // cycle here and 14 in launches.  It stays where it is the coarsest level (one launch for all its sweeps) or the finest: one launch
  // for all cycles outweighs the loss where a simulation alone runs a fixed number of them; to a tolerance, in the solver and in
  // an ensemble, which launch every cycle, a finest level of that size pays those 4 us.
  while (first > 0 && make_plan(levels, first - 1, n, direct, D, smem, threads) && (threads <= CO_THREADS[0] || first == 1 || first == n)) --first;
  return first;
}
cudaError_t launch_coarse(const MGLevel* levels, int first, int n, int pre, int post, int coarse, const double* cinv, int cycles,
                          int* err, cudaStream_t st, int wait_polls) {
  CoDesc D;
  size_t smem = 0;
  int threads = 0;
  if (!make_plan(levels, first, n, cinv != nullptr, D, smem, threads)) return cudaErrorInvalidValue;
  fill_plan(D, levels, first, coarse, cinv, err, wait_polls);
  const int floats = (int)(smem / sizeof(float));
  return with_kernel(threads, D.omega != 1.0f, [&](auto kernel) {
    return launch_clusters(kernel, D.csize, 1, threads, smem, st, D, floats, pre, post, cycles);
  });
}
bool coarse_fits(const MGLevel* levels, int first, int n, bool direct) {
  CoDesc D;
  size_t smem;
  int threads;
  return first < n && make_plan(levels, first, n, direct, D, smem, threads);
}
bool coarse_waits(const MGLevel* levels, int first, int n) {
  CoDesc D;
  size_t smem;
  int threads;
  return first < n && make_plan(levels, first, n, false, D, smem, threads) && D.nd > 0 && D.nact > 1;
}

// ---- batched form: members are grouped by cluster and CTA size ----
size_t coarse_desc_size() { return sizeof(CoDesc); }
int coarse_desc_fill(const MGLevel* levels, int first, int n, int coarse, int* err, void* out, size_t* smem) {
  CoDesc D;
  int threads = 0;
  if (!make_plan(levels, first, n, false, D, *smem, threads)) return -1;
  fill_plan(D, levels, first, coarse, nullptr, err, TAIL_WAIT_POLLS);
  std::memcpy(out, &D, sizeof D);
  return (D.csize > 1 ? 1 : 0) + (threads <= CO_THREADS[0] ? 0 : 2);
}
cudaError_t launch_coarse_batch(int kind, const void* descs, int count, size_t smem, int pre, int post, cudaStream_t st) {
  if (count <= 0) return cudaSuccess;
  const int csize = (kind & 1) ? cluster_size() : 1, floats = (int)(smem / sizeof(float));
  const CoDesc* d = static_cast<const CoDesc*>(descs);
  return (kind & 2) ? launch_clusters(k_coarse_b<CO_THREADS[2]>, csize, count, CO_THREADS[2], smem, st, d, csize, floats, pre, post)
                    : launch_clusters(k_coarse_b<CO_THREADS[0]>, csize, count, CO_THREADS[0], smem, st, d, csize, floats, pre, post);
}

// Opts the kernels into their shared memory and cluster size on the current device.
cudaError_t coarse_configure() {
  cudaError_t e = cudaSuccess;
  auto opt_in = [&](auto k) -> int {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, CO_SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return 0;
  };
  for (int t : CO_THREADS)
    for (bool relax : {false, true}) with_kernel(t, relax, opt_in);
  opt_in(k_coarse_b<CO_THREADS[0]>);
  opt_in(k_coarse_b<CO_THREADS[2]>);
  return e;
}

}  // namespace fire
