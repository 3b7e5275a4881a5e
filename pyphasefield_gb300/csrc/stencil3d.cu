// 3-D explicit steps that march along z: Diffusion / Allen-Cahn (7-point)
// and Cahn-Hilliard (radius 2 through an on-chip chemical-potential tile).
//
// Diffusion / Allen-Cahn by default: lean7_kernel, warps without a shared tile.
// Otherwise a CTA owns a TY x TX column of the grid and a chunk of ZC planes. Its
// z-planes (with an xy halo) are staged by TMA tensor loads into a ring of
// shared-memory slots, several planes ahead of the plane being computed, so
// HBM reads overlap the stencil; each plane is read once and written once
// (xy halos are re-read from L2). The TMA box starts 4 columns left of the
// tile (16-byte aligned); cells outside the grid arrive zero-filled and are
// rewritten with the boundary rule on edge tiles only.
//
// Reference: Field.laplacian (field.py:60-67), engine_ExplicitDiffusion
// (Engines/Diffusion.py:198-208), engine_CahnAllenExplicit
// (Engines/CahnAllen.py:128-135), engine_CahnHilliardExplicit
// (Engines/CahnHilliard.py:134-146).
#include <cmath>

#include "ppf_common.cuh"
#include "ppf_pack.cuh"
#include "ppf_rows.cuh"
#include "ppf_tma.cuh"

namespace ppf {
namespace {

constexpr int kThreads = 256;
constexpr int kXOff = 4;  // box starts kXOff columns left of the tile

template <typename T>
struct Diffusion7 {
  T r;
  __device__ __forceinline__ T operator()(T c, T w, T e, T n, T s, T d, T u) const {
    const T lap = fma(T(-6), c, ((w + e) + (n + s)) + (d + u));
    return fma(r, lap, c);
  }
  // two cells: the sums of the west / east, north / south and lower / upper
  // pairs, rounded as above
  __device__ __forceinline__ F2 pair(F2 c, F2 we, F2 ns, F2 du) const {
    return fma2(sp(r), fma2(sp(-6.f), c, (we + ns) + du), c);
  }
};

template <typename T>
struct AllenCahn7 {
  T a, b;
  __device__ __forceinline__ T operator()(T c, T w, T e, T n, T s, T d, T u) const {
    const T lap = fma(T(-6), c, ((w + e) + (n + s)) + (d + u));
    const T fp = c * fma(c, fma(T(4), c, T(-6)), T(2));
    return c + fma(a, lap, -b * fp);
  }
  __device__ __forceinline__ F2 pair(F2 c, F2 we, F2 ns, F2 du) const {
    const F2 lap = fma2(sp(-6.f), c, (we + ns) + du);
    const F2 fp = c * fma2(c, fma2(sp(4.f), c, sp(-6.f)), sp(2.f));
    return c + fma2(sp(a), lap, sp(-b) * fp);
  }
};

// One vector of cells from its neighbours: packed in float, cell by cell in double.
template <typename Op>
__device__ __forceinline__ void advance(const Op& op, const float (&c)[4], float w, float e,
                                        const float (&n)[4], const float (&s)[4],
                                        const float (&d)[4], const float (&u)[4], float (&o)[4]) {
  const F2 a = op.pair(pk(c[0], c[1]), pk(w + c[1], c[0] + c[2]), pk(n[0], n[1]) + pk(s[0], s[1]),
                       pk(d[0], d[1]) + pk(u[0], u[1]));
  const F2 b = op.pair(pk(c[2], c[3]), pk(c[1] + c[3], c[2] + e), pk(n[2], n[3]) + pk(s[2], s[3]),
                       pk(d[2], d[3]) + pk(u[2], u[3]));
  o[0] = lo(a), o[1] = hi(a), o[2] = lo(b), o[3] = hi(b);
}
template <typename Op>
__device__ __forceinline__ void advance(const Op& op, const double (&c)[2], double w, double e,
                                        const double (&n)[2], const double (&s)[2],
                                        const double (&d)[2], const double (&u)[2],
                                        double (&o)[2]) {
  o[0] = op(c[0], w, c[1], n[0], s[0], d[0], u[0]);
  o[1] = op(c[1], c[0], e, n[1], s[1], d[1], u[1]);
}

// Shared-memory plane ring fed by TMA. Plane p (p >= pbase) lives in slot
// (p - pbase) % NS; its k-th use of the slot completes mbarrier phase k.
template <typename T, int NS>
struct PlaneRing {
  T* slots;
  uint64_t* bars;
  int slot_elems;  // elements per slot (BX * BY, padded to 128 bytes)
  int pbase;
  // p >= pbase always: unsigned arithmetic (a mask when NS is a power of two)
  __device__ T* plane(int p) const { return slots + ((unsigned)(p - pbase) % NS) * slot_elems; }
  __device__ uint64_t* bar(int p) const { return bars + (unsigned)(p - pbase) % NS; }
  __device__ uint32_t parity(int p) const { return ((unsigned)(p - pbase) / NS) & 1u; }
};

struct MarchGeom {
  int TX, TY, ZC, H;  // tile, z chunk, halo
  int BX, BY;         // TMA box (BX = TX + 2 * kXOff, BY = TY + 2H)
};

// A plane outside the grid along a non-periodic z axis is a ghost plane:
// its values follow the boundary rule (Neumann offset, Dirichlet value), so
// the fix-up writes all of it.
template <typename T>
__device__ __forceinline__ bool ghost_plane(const Geo& g, const Bc<T>& bc, int p) {
  return (unsigned)p >= (unsigned)g.n[0] && bc.type[0] != PPF_BC_PERIODIC;
}

// Issue (one thread) the load of plane p. A ghost plane is not loaded; its
// barrier phase is completed by a plain arrive instead.
template <typename T, int NS>
__device__ __forceinline__ void issue_plane(const PlaneRing<T, NS>& ring, const CUtensorMap* map,
                                            const Geo& g, const Bc<T>& bc, const MarchGeom& m,
                                            int x0, int y0, int p) {
  uint64_t* b = ring.bar(p);
  const int nz = g.n[0];
  if (ghost_plane(g, bc, p)) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory");
    return;
  }
  const int pz = wrap_index(p, nz);
  fence_proxy_async();
  mbar_expect_tx(b, (uint32_t)(m.BX * m.BY * sizeof(T)));
  tma_load_3d(ring.plane(p), map, x0 - kXOff, y0 - m.H, pz, b);
}

// The cells of a CTA's W x Hh window (W = TX + 2H, Hh = TY + 2H) that lie
// outside the grid: cl / cr columns on the left / right, rt / rb rows at the
// top / bottom, enumerated as the full rows first, then the outside columns
// of the remaining rows.
struct EdgeSet {
  int W, Hh, cl, cr, rt, rb, nrow, ncol, count;
};

__device__ __forceinline__ EdgeSet edge_set(const MarchGeom& m, const Geo& g, int x0, int y0) {
  EdgeSet E;
  E.W = m.TX + 2 * m.H;
  E.Hh = m.TY + 2 * m.H;
  E.cl = min(E.W, max(0, m.H - x0));
  E.cr = min(E.W - E.cl, max(0, x0 - m.H + E.W - g.n[2]));
  E.rt = min(E.Hh, max(0, m.H - y0));
  E.rb = min(E.Hh - E.rt, max(0, y0 - m.H + E.Hh - g.n[1]));
  E.nrow = (E.rt + E.rb) * E.W;
  E.ncol = E.cl + E.cr;
  E.count = E.nrow + (E.Hh - E.rt - E.rb) * E.ncol;
  return E;
}

// Window coordinates (ly, lx) of edge cell e < E.count.
__device__ __forceinline__ void edge_cell(const EdgeSet& E, int e, int& ly, int& lx) {
  if (e < E.nrow) {
    const int r = e / E.W;
    ly = r < E.rt ? r : E.Hh - E.rb + (r - E.rt);
    lx = e - r * E.W;
  } else {
    const int e2 = e - E.nrow;
    const int r = e2 / E.ncol, c = e2 - r * E.ncol;
    ly = E.rt + r;
    lx = c < E.cl ? c : E.W - E.cr + (c - E.cl);
  }
}

// Edge cells per thread held in registers between the fetch of a plane's
// edge values and their store into its slot.
constexpr int kEdgeRegs = 2;

// Fetch (boundary rule, global loads) the edge values of plane p into
// registers: issued one plane ahead, the loads overlap the stencil of the
// current plane.
template <typename T>
__device__ __forceinline__ void edge_load(const EdgeSet& E, const T* __restrict__ in,
                                          const Geo& g, const Bc<T>& bc, const MarchGeom& m,
                                          int x0, int y0, int p, T (&v)[kEdgeRegs]) {
  const int tid = threadIdx.x + 32 * threadIdx.y;
#pragma unroll
  for (int k = 0; k < kEdgeRegs; ++k) {
    const int e = tid + k * kThreads;
    if (e < E.count) {
      int ly, lx;
      edge_cell(E, e, ly, lx);
      v[k] = fetch<T, 3>(in, g, bc, 0, p, y0 - m.H + ly, x0 - m.H + lx);
    }
  }
}

// Store the edge values of plane p (after its TMA load landed); cells
// beyond kEdgeRegs per thread are fetched here.
template <typename T, int NS>
__device__ __forceinline__ void edge_store(const EdgeSet& E, const PlaneRing<T, NS>& ring,
                                           const T* __restrict__ in, const Geo& g,
                                           const Bc<T>& bc, const MarchGeom& m, int x0, int y0,
                                           int p, const T (&v)[kEdgeRegs]) {
  T* dst = ring.plane(p) + (kXOff - m.H);
  const int tid = threadIdx.x + 32 * threadIdx.y;
#pragma unroll
  for (int k = 0; k < kEdgeRegs; ++k) {
    const int e = tid + k * kThreads;
    if (e < E.count) {
      int ly, lx;
      edge_cell(E, e, ly, lx);
      dst[ly * m.BX + lx] = v[k];
    }
  }
  for (int e = tid + kEdgeRegs * kThreads; e < E.count; e += kThreads) {
    int ly, lx;
    edge_cell(E, e, ly, lx);
    dst[ly * m.BX + lx] = fetch<T, 3>(in, g, bc, 0, p, y0 - m.H + ly, x0 - m.H + lx);
  }
}

// Rewrite the cells of plane p that the TMA box could not supply: the edge
// cells of an edge tile, or the whole of a ghost plane, by the generic
// boundary rule.
template <typename T, int NS>
__device__ __forceinline__ void fixup_plane(const PlaneRing<T, NS>& ring, const T* __restrict__ in,
                                            const Geo& g, const Bc<T>& bc, const MarchGeom& m,
                                            int x0, int y0, int p, bool xy_edge) {
  const bool zfixed = ghost_plane(g, bc, p);
  if (!xy_edge && !zfixed) return;
  T* dst = ring.plane(p);
  const int W = m.TX + 2 * m.H, Hh = m.TY + 2 * m.H;
  if (zfixed) {
    for (int ly = threadIdx.y; ly < Hh; ly += kThreads / 32) {
      const int gy = y0 - m.H + ly;
      for (int lx = threadIdx.x; lx < W; lx += 32) {
        const int gx = x0 - m.H + lx;
        dst[ly * m.BX + (gx - x0 + kXOff)] = fetch<T, 3>(in, g, bc, 0, p, gy, gx);
      }
    }
    return;
  }
  const EdgeSet E = edge_set(m, g, x0, y0);
  for (int e = threadIdx.x + 32 * threadIdx.y; e < E.count; e += kThreads) {
    int ly, lx;
    edge_cell(E, e, ly, lx);
    dst[ly * m.BX + lx + (kXOff - m.H)] =
        fetch<T, 3>(in, g, bc, 0, p, y0 - m.H + ly, x0 - m.H + lx);
  }
}

// Asynchronous copy of one element from global to shared memory (the
// issuing thread waits for its copies with cp_async_wait_all).
template <typename T>
__device__ __forceinline__ void cp_async_elem(T* dst, const T* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(dst)), "l"(src),
               "n"((int)sizeof(T))
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Bounded wait by every thread; returns false (uniformly) if any timed out.
__device__ __forceinline__ bool wait_all(uint64_t* bar, uint32_t parity, int* abort_flag) {
  if (!mbar_wait(bar, parity)) *abort_flag = 1;
  __syncthreads();
  return *abort_flag == 0;
}

template <typename T>
__device__ __forceinline__ void report_timeout(int* status) {
  if (threadIdx.x == 0 && threadIdx.y == 0) atomicOr(status, PPF_STATUS_TIMEOUT);
}

// After a timeout: wait (bounded) for every plane still in flight so that no
// TMA write lands in shared memory after the CTA has exited.
template <typename T, int NS>
__device__ void drain(const PlaneRing<T, NS>& ring, int first, int last) {
  if (threadIdx.x == 0 && threadIdx.y == 0)
    for (int p = first; p <= last; ++p) mbar_wait(ring.bar(p), ring.parity(p));
  __syncthreads();
}

// First 128-byte aligned address at or after p (the dynamic shared memory
// base). The offset is added to p itself, not to an integer copy of it, so
// the compiler keeps the shared address space and emits shared loads.
template <typename T>
__device__ __forceinline__ T* align128(unsigned char* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  return reinterpret_cast<T*>(p + ((128u - (a & 127u)) & 127u));
}

// ------------------------------------------------------------- 7-point
constexpr int kNS7 = 5;  // planes z-1, z, z+1 in use; z+2, z+3 in flight

template <typename T, typename Op>
__global__ void __launch_bounds__(kThreads)
    march7_kernel(const __grid_constant__ CUtensorMap map, Op op, Geo g, Bc<T> bc,
                  const T* __restrict__ in, T* __restrict__ out, MarchGeom m, int slot_elems,
                  int* status) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bars[kNS7];
  __shared__ int abort_flag;
  const int x0 = blockIdx.x * m.TX, y0 = blockIdx.y * m.TY, z0 = blockIdx.z * m.ZC;
  const int nz = g.n[0], ny = g.n[1], nx = g.n[2];
  const int z1 = min(z0 + m.ZC, nz);
  const bool xy_edge = x0 - 1 < 0 || y0 - 1 < 0 || x0 + m.TX + 1 > nx || y0 + m.TY + 1 > ny ||
                       x0 - kXOff < 0 || x0 + m.TX + kXOff > nx;
  PlaneRing<T, kNS7> ring{align128<T>(smem_raw), bars, slot_elems, z0 - 1};
  const bool leader = threadIdx.x == 0 && threadIdx.y == 0;

  if (leader) {
    for (int i = 0; i < kNS7; ++i) mbar_init(&bars[i], 1);
    mbar_init_fence();
    abort_flag = 0;
  }
  __syncthreads();
  pdl_wait();
  pdl_launch_next();
  const int last = z1;  // last plane needed
  if (leader)
    for (int p = z0 - 1; p <= min(z0 + 2, last); ++p) issue_plane(ring, &map, g, bc, m, x0, y0, p);
  int issued = min(z0 + 2, last);

  for (int p = z0 - 1; p <= z0; ++p) {
    if (!wait_all(ring.bar(p), ring.parity(p), &abort_flag)) {
      report_timeout<T>(status);
      drain(ring, p, issued);
      return;
    }
    fixup_plane(ring, in, g, bc, m, x0, y0, p, xy_edge);
  }
  const int W = m.BX;
  for (int z = z0; z < z1; ++z) {
    if (leader && z + 3 <= last) {
      issue_plane(ring, &map, g, bc, m, x0, y0, z + 3);
      issued = z + 3;
    }
    if (!wait_all(ring.bar(z + 1), ring.parity(z + 1), &abort_flag)) {
      report_timeout<T>(status);
      if (leader) issued = min(z + 3, last);
      drain(ring, z + 1, min(z + 3, last));
      return;
    }
    fixup_plane(ring, in, g, bc, m, x0, y0, z + 1, xy_edge);
    __syncthreads();
    const T* pd = ring.plane(z - 1);
    const T* pc = ring.plane(z);
    const T* pu = ring.plane(z + 1);
    for (int ly = 1 + threadIdx.y; ly <= m.TY; ly += kThreads / 32) {
      const int gy = y0 + ly - 1;
      if (gy >= ny) break;
      T* orow = out + (int64_t)z * g.plane + (int64_t)gy * g.pitch;
      for (int lx = threadIdx.x; lx < m.TX; lx += 32) {
        const int gx = x0 + lx;
        if (gx >= nx) break;
        const int i = ly * W + lx + kXOff;
        orow[gx] = op(pc[i], pc[i - 1], pc[i + 1], pc[i - W], pc[i + W], pd[i], pu[i]);
      }
    }
    __syncthreads();
  }
}

// Lean 7-point kernel (the default): a warp owns 32 V columns (V cells of one
// 16-byte vector per lane; LX = 16 or 8 lanes a row, and groups of lanes on rows of
// their own, where x is short) and R rows and marches along z with planes z - 1, z
// and z + 1 of its rows in registers; west / east cells come by shuffles. A
// lane copies its own vectors of the band and of the two rows beside it, D - 1
// planes ahead, into a ring in shared memory (cp.async) and is the only one to
// read them back: no barrier, and a warp waits for its own copies alone. The
// grid's edges take the same path: a ghost row or plane is copied from its
// source and fixed after the read (AxisRule), a ghost column one of the strip's side
// cells (ColumnRule), and of a vector that reaches past nx the cells below it.
//
// Bound: HBM beyond L2 (512^3: 6.3 TB/s), instruction latency below. us per step
// against the 32 x 32 shared-memory tiles this replaced, whose edge tiles
// rewrote their window every plane behind a barrier: Allen-Cahn 320 x 200 x 250
// no-flux 86 -> 30, diffusion 64^3 22.9 -> 3.8, 256^3 38.2 -> 25.8, 384^3 104 ->
// 79, 512^3 221 -> 170; float64 200^3 309 -> 260.
constexpr int kLWarps = 4;

// Row bands a launch holds (gridDim.y); a grid with more takes several launches,
// each from its first row y_first on.
constexpr int kMaxBands = 65535;

template <typename T, int R, int LX>
struct Lean7Slot {
  static constexpr int V = Vec16<T>::n;
  static constexpr int side = (R + 2) * 32 * V;  // per group: west cells, then east cells
  static constexpr int elems = (side + 2 * R * (32 / LX) + V - 1) / V * V;
};

template <typename T, typename Op, int R, int D, int LX>
__global__ void __launch_bounds__(32 * kLWarps)
    lean7_kernel(Op op, const __grid_constant__ Geo g, const __grid_constant__ Bc<T> bc,
                 const T* __restrict__ in, T* __restrict__ out, int zc, int y_first) {
  constexpr int V = Vec16<T>::n;
  constexpr int G = 32 / LX;  // groups of lanes, each with R rows of its own
  constexpr int RS = 32 * V;  // elements of a row of the slot
  using VT = typename Vec16<T>::type;
  using Slot = Lean7Slot<T, R, LX>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x, lx = G > 1 ? lane % LX : lane;
  const int group = G > 1 ? lane / LX : 0;
  T* ring = reinterpret_cast<T*>(smem_raw) + threadIdx.y * D * Slot::elems;
  const int x0 = blockIdx.x * (LX * V);
  const int yw = y_first + (blockIdx.y * kLWarps + threadIdx.y) * (R * G);
  const int y0 = yw + group * R;
  const int z0 = blockIdx.z * zc;
  const int nz = g.n[0], ny = g.n[1], nx = g.n[2];
  pdl_wait();
  pdl_launch_next();
  if (yw >= ny) return;  // whole warp; no block-wide barrier follows
  const int z1 = min(z0 + zc, nz);
  const int x = x0 + lx * V;
  const bool vec = x + V <= nx;
  const bool full_x = x0 + LX * V <= nx;
  // bytes a lane copies of a row: the cells below nx, the rest of its vector
  // reads zero
  const uint32_t bytes = (uint32_t)max(0, min(V, nx - x)) * (uint32_t)sizeof(T);
  const bool rows_in = yw >= 1 && yw + R * G + 1 <= ny;     // uniform across the warp
  const bool first = lx == 0;                               // uses the west neighbours
  const bool last = x < nx && (lx == LX - 1 || x + V >= nx);  // uses the east neighbours
  const ColumnRule<T, 1, 2> wr(g, bc, x0 - 1), er(g, bc, min(x0 + LX * V, nx));
  const bool x_ghost = wr.ghost || er.ghost;  // uniform across the warp
  const bool full_y = yw + R * G <= ny;
  const int64_t out_off = (int64_t)y0 * g.pitch;
  // this lane's element of each row of a plane (planes below 2^31 elements)
  const uint32_t xs = x < nx ? x : 0;
  uint32_t off[R + 2];
#pragma unroll
  for (int j = 0; j < R + 2; ++j)
    // rows past the ghost row feed outputs that are not stored
    off[j] = (uint32_t)(rows_in ? y0 - 1 + j : AxisRule<T>(g, bc, 1, min(y0 - 1 + j, ny)).src) *
                 (uint32_t)g.pitch +
             xs;
  // lane j < 2 R of a group copies one side cell: west of row j, east of row j - R
  uint32_t side_off = 0;
  const int side_at = Slot::side + group * (2 * R);
#pragma unroll
  for (int j = 0; j < R; ++j) {
    if (lx == j) side_off = off[j + 1] - xs + (uint32_t)wr.xi;
    if (lx == R + j) side_off = off[j + 1] - xs + (uint32_t)er.xi;
  }

  // plane p: the band's own rows, and for a plane that is advanced the rows
  // and columns beside them
  auto issue = [&](int p, int slot) {
    T* s = ring + slot * Slot::elems;
    const int zs = (unsigned)p < (unsigned)nz ? p : AxisRule<T>(g, bc, 0, p).src;
    const T* src = in + (int64_t)zs * g.plane;
    const bool beside = p >= z0 && p < z1;
    const uint32_t d = smem_addr(s + lane * V);
#pragma unroll
    for (int j = 0; j < R + 2; ++j)
      if ((j >= 1 && j <= R) || beside)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                         d + (uint32_t)(j * RS * sizeof(T))),
                     "l"(src + off[j]), "r"(bytes)
                     : "memory");
    if (beside && lx < 2 * R) cp_async_elem(s + side_at + lx, src + side_off);
  };
  auto read_row = [&](const T* s, int j, T (&v)[V]) {
    const VT q = *reinterpret_cast<const VT*>(s + j * RS + lane * V);
    const T* pq = reinterpret_cast<const T*>(&q);
#pragma unroll
    for (int e = 0; e < V; ++e) v[e] = pq[e];
  };
  auto read_own = [&](int z, const T* s, T (&v)[R][V]) {
#pragma unroll
    for (int j = 0; j < R; ++j) read_row(s, j + 1, v[j]);
    if ((unsigned)z >= (unsigned)nz) {
      const AxisRule<T> zr(g, bc, 0, z);
#pragma unroll
      for (int j = 0; j < R; ++j)
#pragma unroll
        for (int e = 0; e < V; ++e) v[j][e] = zr.value(v[j][e]);
    }
  };

  // one group per plane, empty ones past the end, so that the count of groups
  // in flight is the same in every iteration
#pragma unroll
  for (int q = 0; q < D; ++q) {
    if (z0 - 1 + q <= z1) issue(z0 - 1 + q, q);
    cp_async_commit();
  }
  T cm[R][V], c0[R][V];
  asm volatile("cp.async.wait_group %0;" ::"n"(D - 2) : "memory");
  read_own(z0 - 1, ring, cm);
  read_own(z0, ring + Slot::elems, c0);
  int sm = 0;  // slot of plane z - 1
  for (int z = z0; z < z1; ++z) {
    // planes up to z + D - 2 are issued: z + 1 has landed when D - 3 are pending
    // (the side cells are other lanes' copies)
    asm volatile("cp.async.wait_group %0;" ::"n"(D - 3) : "memory");
    __syncwarp();
    if (z + D - 1 <= z1) issue(z + D - 1, sm);
    cp_async_commit();
    const int s0 = sm + 1 == D ? 0 : sm + 1, sp = s0 + 1 == D ? 0 : s0 + 1;
    const T* S0 = ring + s0 * Slot::elems;
    T cp[R][V], c[R + 2][V], side[2 * R];
    read_own(z + 1, ring + sp * Slot::elems, cp);
    read_row(S0, 0, c[0]);
    read_row(S0, R + 1, c[R + 1]);
#pragma unroll
    for (int j = 0; j < R; ++j)
#pragma unroll
      for (int e = 0; e < V; ++e) c[j + 1][e] = c0[j][e];
#pragma unroll
    for (int q = 0; q < 2 * R / V; ++q) {
      const VT v = *reinterpret_cast<const VT*>(S0 + side_at + q * V);
      const T* pv = reinterpret_cast<const T*>(&v);
#pragma unroll
      for (int e = 0; e < V; ++e) side[q * V + e] = pv[e];
    }
    if (!rows_in) {  // ghost rows
#pragma unroll
      for (int j = 0; j < R + 2; ++j) {
        const AxisRule<T> r(g, bc, 1, min(y0 - 1 + j, ny));
        if (r.ghost) {
#pragma unroll
          for (int e = 0; e < V; ++e) c[j][e] = r.value(c[j][e]);
        }
      }
    }
    if (x_ghost) {
#pragma unroll
      for (int j = 0; j < R; ++j) {
        side[j] = wr.value(0, side[j]);
        side[R + j] = er.value(0, side[R + j]);
      }
    }
    T* orow = out + (int64_t)z * g.plane + out_off;
#pragma unroll
    for (int j = 1; j <= R; ++j) {
      const T wv = side[j - 1], ev = side[R + j - 1];
      if (!full_x) {  // the ghost column inside the last lane's vector
#pragma unroll
        for (int e = 1; e < V; ++e)
          if (x + e == nx) c[j][e] = ev;
      }
      T wl = __shfl_up_sync(0xffffffffu, c[j][V - 1], 1);
      T ee = __shfl_down_sync(0xffffffffu, c[j][0], 1);
      if (first) wl = wv;
      if (last) ee = ev;
      T o[V];
      advance(op, c[j], wl, ee, c[j - 1], c[j + 1], cm[j - 1], cp[j - 1], o);
      if (full_y || y0 + j - 1 < ny) store_cells<T, V>(orow, x, nx, vec, o);
      orow += g.pitch;
    }
#pragma unroll
    for (int j = 0; j < R; ++j)
#pragma unroll
      for (int e = 0; e < V; ++e) cm[j][e] = c0[j][e], c0[j][e] = cp[j][e];
    sm = s0;
  }
  cp_async_wait_all();
}

// ------------------------------------------------------------- Cahn-Hilliard
// mu~ = -(eps^2/dx^2) lap'(c) + f'(c), lap' the unscaled 7-point sum;
// c' = c + sum over the 6 faces of F = a (mu~_nbr - mu~_c), a = dt M/dx^2.
// With QUANT each face flux is rounded to a multiple of q (a power of two).
// F(A->B) = -F(B->A) bit for bit (the same mu~ values enter both cells and
// rounding to nearest is odd-symmetric), so the float field conserves its
// sum exactly while every value stays a multiple of q below 2^24 q.
template <typename T>
struct ChCoef {
  T kap;         // eps^2/dx^2
  T a;           // dt*M/dx^2
  T aiq;         // a / q (QUANT only; exact: q is a power of two)
  T q, iq;       // quantum and its inverse (QUANT only)
  T range;       // 2^24 q: |c| beyond this loses exactness (QUANT only)
  int centered;  // field holds u = c - 1/2
};

// f'(c) - kap lap(c), f' = 4c^3 - 6c^2 + 2c, or in the centered variable 4u^3 - u. In
// float the multiply-adds are written out, so that the scalar and the packed form round
// alike; in double, which has no packed form, the compiler's own give the same bits and
// up to 3 % more speed (one line of 977253 cells, us per step: 4417 against 4575).
__device__ __forceinline__ float ch_mu(const ChCoef<float>& k, float c, float w, float e, float n,
                                       float s, float d, float u) {
  const float lap = fmaf(-6.f, c, ((w + e) + (n + s)) + (d + u));
  const float wl = k.centered ? fmaf(4.f * c, c, -1.f) : fmaf(c, fmaf(4.f, c, -6.f), 2.f);
  return fmaf(c, wl, -k.kap * lap);
}
__device__ __forceinline__ double ch_mu(const ChCoef<double>& k, double c, double w, double e,
                                        double n, double s, double d, double u) {
  const double lap = ((w + e) + (n + s)) + (d + u) - 6.0 * c;
  const double fp = k.centered ? c * (4.0 * c * c - 1.0) : c * (2.0 + c * (-6.0 + 4.0 * c));
  return fp - k.kap * lap;
}

template <typename T>
__device__ __forceinline__ T ch_flux(const ChCoef<T>& k, T mn, T mc) {
  return k.a * (mn - mc);
}

constexpr int kNSC = 7;  // c planes z..z+2 read, z+3 .. z+5 in flight
constexpr int kMuSlots = 3;  // mu planes z - 1, z, z + 1
// Cahn-Hilliard tile (double): 32 x 32 cells, 256 threads; thread (tx, ty) owns the
// kCQ = 4 xy-columns (ty + 8q, tx) and keeps, per column, c(z), c(z+1),
// mu(z) and the flux through the face below plane z in registers while
// marching along z (the flux through a face is computed once: the cell
// above takes it negated, bit for bit). mu of the tile plus a one-cell ring
// lives in a three-plane shared ring for the xy fluxes (one block barrier
// per plane: the one that publishes mu(z + 1)); the kRingN ring
// positions are computed by threads 0..kRingN-1. Every shared index is a
// compile-time offset from a per-thread base.
constexpr int kCTX = 32;
constexpr int kCTY = 32;
constexpr int kCQ = kCTY / 8;
constexpr int kCW = kCTX + 2 * kXOff;     // c plane row length (TMA box width)
constexpr int kCH = kCTY + 4;             // c plane rows (halo 2)
constexpr int kCSlot = kCW * kCH;         // 1440 elements, a multiple of 128 bytes
constexpr int kMW = kCTX + 2;
constexpr int kMH = kCTY + 2;
constexpr int kMN = kMW * kMH;
constexpr int kRingN = kMN - kCTX * kCTY;  // 132

// Ring position i -> mu-region coordinates (ly, lx) on the border.
__device__ __forceinline__ void ring_pos(int i, int& ly, int& lx) {
  if (i < kMW) {
    ly = 0;
    lx = i;
  } else if (i < 2 * kMW) {
    ly = kMH - 1;
    lx = i - kMW;
  } else if (i < 2 * kMW + kCTY) {
    ly = 1 + (i - 2 * kMW);
    lx = 0;
  } else {
    ly = 1 + (i - 2 * kMW - kCTY);
    lx = kMW - 1;
  }
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
    cahn_hilliard_kernel(const __grid_constant__ CUtensorMap map, ChCoef<T> k, Geo g, Bc<T> bc,
                         const T* __restrict__ in, T* __restrict__ out, double* __restrict__ mass,
                         int* __restrict__ status, MarchGeom m, int slot_elems,
                         int* __restrict__ lib_status) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bars[kNSC];
  __shared__ int abort_flag;
  __shared__ double red[kThreads / 32];
  const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + 32 * ty;
  const int x0 = blockIdx.x * kCTX, y0 = blockIdx.y * kCTY, z0 = blockIdx.z * m.ZC;
  const int nz = g.n[0], ny = g.n[1], nx = g.n[2];
  const int z1 = min(z0 + m.ZC, nz);
  const bool xy_edge = x0 - kXOff < 0 || y0 - 2 < 0 || x0 + kCTX + kXOff > nx ||
                       y0 + kCTY + 2 > ny;
  PlaneRing<T, kNSC> ring{align128<T>(smem_raw), bars, kCSlot, z0 - 2};
  // kMuSlots mu planes: in iteration z a thread writes mu(z + 1) while
  // others may still read mu(z - 1) (nothing but the one barrier per plane
  // orders the iterations), so mu(z - 1), mu(z), mu(z + 1) need three slots
  T* const mring = ring.slots + kNSC * kCSlot;
  const bool leader = tid == 0;
  (void)slot_elems;

  // own cells q: c-plane index ci + q * 8 * kCW, mu-plane index mi + q * 8 * kMW
  const int ci = (ty + 2) * kCW + tx + kXOff;
  const int mi = (ty + 1) * kMW + tx + 1;
  const bool has_ring = tid < kRingN;
  int rci = 0, rmi = 0;
  if (has_ring) {
    int ly, lx;
    ring_pos(tid, ly, lx);
    rci = (ly + 1) * kCW + lx + (kXOff - 1);
    rmi = ly * kMW + lx;
  }

  if (leader) {
    for (int i = 0; i < kNSC; ++i) mbar_init(&bars[i], 1);
    mbar_init_fence();
    abort_flag = 0;
  }
  __syncthreads();
  pdl_wait();
  pdl_launch_next();
  const int last = z1 + 1;
  if (leader)
    for (int p = z0 - 2; p <= min(z0 + kNSC - 3, last); ++p)
      issue_plane(ring, &map, g, bc, m, x0, y0, p);
  for (int p = z0 - 2; p <= z0 + 1; ++p) {
    if (!wait_all(ring.bar(p), ring.parity(p), &abort_flag)) {
      report_timeout<T>(lib_status);
      drain(ring, p, min(z0 + kNSC - 3, last));
      return;
    }
    fixup_plane(ring, in, g, bc, m, x0, y0, p, xy_edge);
  }
  __syncthreads();

  auto mu_at = [&](const T* cd, const T* cc, const T* cu, int i) {
    return ch_mu(k, cc[i], cc[i - 1], cc[i + 1], cc[i - kCW], cc[i + kCW], cd[i], cu[i]);
  };
  T c0[kCQ], c1[kCQ], mu0[kCQ], fup[kCQ];
  {
    const T* Pm2 = ring.plane(z0 - 2);
    const T* Pm1 = ring.plane(z0 - 1);
    const T* P0 = ring.plane(z0);
    const T* P1 = ring.plane(z0 + 1);
    T* M0 = mring;
#pragma unroll
    for (int q = 0; q < kCQ; ++q) {
      const int i = ci + q * 8 * kCW;
      const T mum = mu_at(Pm2, Pm1, P0, i);
      mu0[q] = mu_at(Pm1, P0, P1, i);
      M0[mi + q * 8 * kMW] = mu0[q];
      c0[q] = P0[i];
      c1[q] = P1[i];
      // flux through the face below z0, stored negated as "flux into the
      // cell below from above": the loop takes fd = -fup
      fup[q] = -ch_flux(k, mum, mu0[q]);
    }
    if (has_ring) M0[rmi] = mu_at(Pm1, P0, P1, rci);
  }
  // the first iteration's load goes into the slot of plane z0 - 2, read
  // just above
  __syncthreads();

  T* optr = out + (int64_t)z0 * g.plane + (int64_t)(y0 + ty) * g.pitch + x0 + tx;
  const int64_t qstride = (int64_t)8 * g.pitch;
  const bool xin = x0 + tx < nx;
  int nq = 0;  // own rows inside the grid: rows ty + 8q < ny - y0
#pragma unroll
  for (int q = 0; q < kCQ; ++q) nq += (xin && y0 + ty + 8 * q < ny) ? 1 : 0;
  // CTA-uniform: the whole tile lies inside the grid (no per-cell checks)
  const bool full = x0 + kCTX <= nx && y0 + kCTY <= ny;

  double acc = 0.0;
  T vmax = T(0), vsum = T(0);
  int m0i = 0;  // mu slot of plane z
  // edge tiles: the boundary-rule values of plane z + 2 are fetched into
  // registers during iteration z - 1
  const EdgeSet E = edge_set(m, g, x0, y0);
  const bool has_edge = xy_edge && E.count > 0;
  T pre[kEdgeRegs];
  if (has_edge && z0 + 2 <= last && !ghost_plane(g, bc, z0 + 2))
    edge_load(E, in, g, bc, m, x0, y0, z0 + 2, pre);
  for (int z = z0; z < z1; ++z) {
    // plane z + kNSC - 2 reuses the slot of plane z - 2, last read in
    // iteration z - 2 (c plane p is read in iterations p - 2 .. p), before
    // the barriers of iteration z - 1
    if (leader && z + kNSC - 2 <= last) issue_plane(ring, &map, g, bc, m, x0, y0, z + kNSC - 2);
    // every thread waits for plane z + 2 itself; a timeout is acted on, by
    // all threads alike, after the barrier below
    if (!mbar_wait(ring.bar(z + 2), ring.parity(z + 2))) abort_flag = 1;
    if (ghost_plane(g, bc, z + 2)) {
      fixup_plane(ring, in, g, bc, m, x0, y0, z + 2, xy_edge);
      __syncthreads();
    } else if (has_edge) {
      edge_store(E, ring, in, g, bc, m, x0, y0, z + 2, pre);
      __syncthreads();
    }
    if (has_edge && z + 3 <= last && !ghost_plane(g, bc, z + 3))
      edge_load(E, in, g, bc, m, x0, y0, z + 3, pre);
    const T* P0 = ring.plane(z);
    const T* P1 = ring.plane(z + 1);
    const T* P2 = ring.plane(z + 2);
    const int m1i = m0i == kMuSlots - 1 ? 0 : m0i + 1;
    T* M1 = mring + m1i * kMN;
    T c2[kCQ], mup[kCQ];
#pragma unroll
    for (int q = 0; q < kCQ; ++q) {
      const int i = ci + q * 8 * kCW;
      c2[q] = P2[i];
      mup[q] = ch_mu(k, c1[q], P1[i - 1], P1[i + 1], P1[i - kCW], P1[i + kCW], c0[q], c2[q]);
      M1[mi + q * 8 * kMW] = mup[q];
    }
    if (has_ring) M1[rmi] = mu_at(P0, P1, P2, rci);
    __syncthreads();
    if (abort_flag) {
      report_timeout<T>(lib_status);
      drain(ring, z + 2, min(z + kNSC - 2, last));
      return;
    }
    const T* M0 = mring + m0i * kMN;
    m0i = m1i;
#pragma unroll
    for (int q = 0; q < kCQ; ++q) {
      const int i = mi + q * 8 * kMW;
      const T m0 = mu0[q];
      const T fw = ch_flux(k, M0[i - 1], m0);
      const T fe = ch_flux(k, M0[i + 1], m0);
      const T fn = ch_flux(k, M0[i - kMW], m0);
      const T fs = ch_flux(k, M0[i + kMW], m0);
      const T fu = ch_flux(k, mup[q], m0);
      const T fd = -fup[q];
      const T v = c0[q] + (((fw + fe) + (fn + fs)) + (fd + fu));
      if (full || q < nq) {
        optr[q * qstride] = v;
        acc += (double)v;
        vmax = fmax(vmax, fabs(v));
        vsum += v;
      }
      c0[q] = c1[q];
      c1[q] = c2[q];
      mu0[q] = mup[q];
      fup[q] = fu;
    }
    optr += g.plane;
  }
  int flags = 0;
  if (!isfinite(vsum) || !isfinite(vmax)) flags |= PPF_STATUS_NONFINITE;
  if (status && flags) atomicOr(status, flags);
  if (mass) {
    double v = acc;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (tx == 0) red[ty] = v;
    __syncthreads();
    if (ty == 0) {
      double s = tx < kThreads / 32 ? red[tx] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (tx == 0) atomicAdd(mass, s);
    }
  }
}

// ------------------------------------------------------------- Cahn-Hilliard, float
// A warp owns 128 columns (4 per lane) and kHR rows and marches along z, as
// lean7_kernel does: c planes come by cp.async into a ring of its own, mu(z) and
// mu(z + 1) of its rows and the rows beside them stay in registers, and every
// face flux is computed once by the cell west, north or below of it and taken
// negated by the other (x across lanes through the neighbour's mu). The columns
// beside the strip come as 24 side cells per plane, from which lanes 0 .. 7 form
// the eight mu values the strip's outer faces need. Nothing but a warp's own
// copies is waited for. The arithmetic is packed (FP32x2) and rounds as ch_mu and
// ch_flux do.
//
// Bound: instruction issue and latency at 12 warps per SM (registers, shared
// memory); 26.5 M warp instructions per 256^3 step where the shared-memory tiles
// of cahn_hilliard_kernel, which this replaced in float, took 62.5 M and a block
// barrier per plane. us per step: 256^3 87 -> 42, 384^3 235 -> 130, 128^3 33 ->
// 12, one plane of 1500 x 2000 40 -> 13.
constexpr int kHR = 4;              // rows per warp
constexpr int kHWarps = 4;
constexpr int kHRow = 128;          // elements of a row in a slot
constexpr int kHRows = kHR + 4;     // c rows y0 - 2 .. y0 + kHR + 1
constexpr int kHSideRows = kHR + 2; // side rows y0 - 1 .. y0 + kHR
constexpr int kHSide = kHRows * kHRow;           // side cells: 4 columns x kHSideRows
constexpr int kHSlot = kHSide + 32;
static_assert(4 * kHSideRows <= 32 && 2 * kHR <= 8, "one side cell and one side mu per lane");
constexpr int kHD = 4;                           // ring: planes z .. z + 2 in use, one coming
template <bool FLAT>  // the ring and two sets of eight side mu values
constexpr int kHWarpElems = (FLAT ? 1 : kHD) * kHSlot + 16;

struct Quad {  // four adjacent cells of a lane
  F2 a, b;
};
__device__ __forceinline__ Quad operator+(Quad x, Quad y) { return {x.a + y.a, x.b + y.b}; }
__device__ __forceinline__ Quad operator-(Quad x, Quad y) { return {x.a - y.a, x.b - y.b}; }
__device__ __forceinline__ Quad quad(const float4& v) { return {pk(v.x, v.y), pk(v.z, v.w)}; }

__device__ __forceinline__ F2 ch_mu2(const ChCoef<float>& k, F2 c, F2 we, F2 ns, F2 du) {
  const F2 lap = fma2(sp(-6.f), c, (we + ns) + du);
  const F2 w = k.centered ? fma2(sp(4.f) * c, c, sp(-1.f))
                          : fma2(c, fma2(sp(4.f), c, sp(-6.f)), sp(2.f));
  return fma2(c, w, sp(-k.kap) * lap);
}

// Fluxes from the differences of mu across the faces, as ch_flux; QUANT: rounded to the
// quantum ((a d) / q == (a / q) d bit for bit: scaling by a power of two is exact).
template <bool QUANT>
__device__ __forceinline__ float ch_scale(const ChCoef<float>& k, float d) {
  return QUANT ? rintf(k.aiq * d) * k.q : k.a * d;
}
template <bool QUANT>
__device__ __forceinline__ Quad ch_scale4(const ChCoef<float>& k, Quad d) {
  if (!QUANT) return {sp(k.a) * d.a, sp(k.a) * d.b};
  const F2 x = sp(k.aiq) * d.a, y = sp(k.aiq) * d.b;
  return {pk(rintf(lo(x)), rintf(hi(x))) * sp(k.q), pk(rintf(lo(y)), rintf(hi(y))) * sp(k.q)};
}
template <bool QUANT>
__device__ __forceinline__ Quad ch_flux4(const ChCoef<float>& k, Quad mn, Quad mc) {
  return ch_scale4<QUANT>(k, mn - mc);
}

// FLAT: a single plane, its own neighbour along z (no march, no z fluxes). Off holds
// an element's offset within a plane; 64 bits make the general form, for grids beyond
// 2^31 elements a plane or kMaxBands row bands and for outputs off a 16-byte boundary
// (y_first is 0 and out is aligned in the other, whose registers are all taken: the
// row's start alone cost 1 % of 256^3).
template <bool QUANT, bool FLAT, typename Off>
__global__ void __launch_bounds__(32 * kHWarps, 3)
    ch_march_kernel(const __grid_constant__ ChCoef<float> k, const __grid_constant__ Geo g,
                    const __grid_constant__ Bc<float> bc, const float* __restrict__ in,
                    float* __restrict__ out, double* __restrict__ mass, int* __restrict__ status,
                    int zc, int y_first) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x;
  float* ring = reinterpret_cast<float*>(smem_raw) + threadIdx.y * kHWarpElems<FLAT>;
  float* smu = ring + (FLAT ? 1 : kHD) * kHSlot;
  const int nz = g.n[0], ny = g.n[1], nx = g.n[2];
  const int x0 = blockIdx.x * kHRow;
  const int y0 = (sizeof(Off) == 8 ? y_first : 0) + (blockIdx.y * kHWarps + threadIdx.y) * kHR;
  const int z0 = blockIdx.z * zc;
  pdl_wait();
  pdl_launch_next();
  if (y0 >= ny) return;  // whole warp; no block-wide barrier follows
  const int z1 = min(z0 + zc, nz);
  const int x = x0 + 4 * lane;
  // source elements within a plane; rows and columns further out than two ghost
  // cells feed nothing that is stored
  Off off[kHRows];
#pragma unroll
  for (int j = 0; j < kHRows; ++j)
    off[j] = (Off)AxisRule<float>(g, bc, 1, min(y0 - 2 + j, ny + 1)).src * (Off)g.pitch;
  const bool vec = x + 4 <= nx;
  uint32_t col[4];  // a lane whose vector reaches past nx copies cell by cell
#pragma unroll
  for (int e = 0; e < 4; ++e) col[e] = AxisRule<float>(g, bc, 2, min(x + e, nx + 1)).src;
  const bool used = x < nx + 2;
  // side cell `lane`: columns x0 - 2, x0 - 1, x0 + 128, x0 + 129, kHSideRows each
  Off side_off = 0;
  const bool has_side = lane < 4 * kHSideRows;
  {
    const int q = lane / kHSideRows, j = lane - q * kHSideRows;
    const int xc = q < 2 ? x0 - 2 + q : x0 + kHRow - 2 + q;
    const uint32_t c = AxisRule<float>(g, bc, 2, min(xc, nx + 1)).src;
#pragma unroll
    for (int r = 0; r < kHSideRows; ++r)
      if (r == j) side_off = off[r + 1] + c;
  }

  auto issue = [&](int p, int slot) {
    float* s = ring + slot * kHSlot;
    const int zs = (unsigned)p < (unsigned)nz ? p : AxisRule<float>(g, bc, 0, p).src;
    const float* src = in + (int64_t)zs * g.plane;
    if (vec) {
      const uint32_t d = smem_addr(s + 4 * lane);
#pragma unroll
      for (int j = 0; j < kHRows; ++j)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 4 * j * kHRow),
                     "l"(src + off[j] + x)
                     : "memory");
    } else if (used) {
#pragma unroll
      for (int j = 0; j < kHRows; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          cp_async_elem(s + j * kHRow + 4 * lane + e, src + off[j] + col[e]);
    }
    if (has_side) cp_async_elem(s + kHSide + lane, src + side_off);
  };
  auto row = [&](const float* s, int j) {
    return quad(*reinterpret_cast<const float4*>(s + j * kHRow + 4 * lane));
  };

  // mu of the rows y0 - 1 .. y0 + kHR of plane S1 (below it S0, above it S2);
  // lanes 0 .. 3: of column x0 - 1, lanes 4 .. 7: of column x0 + 128, own rows
  auto mu_rows = [&](const float* S0, const float* S1, const float* S2, Quad (&m)[kHR + 2],
                     float& ms) {
    Quad n = row(S1, 0), c = row(S1, 1);
    // the columns beside the strip, for lane 0 (west) and lane 31 (east)
    const float* sc = S1 + kHSide + (lane == 31 ? 2 : 1) * kHSideRows;
#pragma unroll
    for (int i = 0; i < kHR + 2; ++i) {
      const Quad s = row(S1, i + 2);
      const Quad du = FLAT ? c + c : row(S0, i + 1) + row(S2, i + 1);
      const float beside = sc[i];
      const float c0 = lo(c.a), c1 = hi(c.a), c2 = lo(c.b), c3 = hi(c.b);
      float wl = __shfl_up_sync(0xffffffffu, c3, 1);
      float er = __shfl_down_sync(0xffffffffu, c0, 1);
      if (lane == 0) wl = beside;
      if (lane == 31) er = beside;
      const Quad ns = n + s;
      m[i].a = ch_mu2(k, c.a, pk(wl + c1, c0 + c2), ns.a, du.a);
      m[i].b = ch_mu2(k, c.b, pk(c1 + c3, c2 + er), ns.b, du.b);
      n = c;
      c = s;
    }
    if (lane < 2 * kHR) {
      const int e = lane / kHR, j = lane - e * kHR;
      const int q = (e ? 2 : 1) * kHSideRows + j + 1;  // the cell among the side cells
      const float inner = S1[(j + 2) * kHRow + (e ? kHRow - 1 : 0)];
      const float outer = S1[kHSide + (e ? 3 : 0) * kHSideRows + j + 1];
      const float c1 = S1[kHSide + q];
      ms = ch_mu(k, c1, e ? inner : outer, e ? outer : inner, S1[kHSide + q - 1],
                 S1[kHSide + q + 1], FLAT ? c1 : S0[kHSide + q], FLAT ? c1 : S2[kHSide + q]);
    }
  };

  Quad mu[kHR + 2], fup[kHR];
  float ms = 0.f;
  int s0 = 0;  // slot of plane z
  if (FLAT) {
    issue(0, 0);
    cp_async_commit();
    cp_async_wait_all();
    __syncwarp();
    mu_rows(ring, ring, ring, mu, ms);
  } else {
    // planes z0 - 2 .. z0 + 1 into slots 0 .. 3
#pragma unroll
    for (int q = 0; q < kHD; ++q) {
      issue(z0 - 2 + q, q);
      cp_async_commit();
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    Quad ml[kHR + 2];
    float unused = 0.f;
    mu_rows(ring, ring + kHSlot, ring + 2 * kHSlot, ml, unused);  // mu(z0 - 1)
    __syncwarp();
    issue(z0 + 2, 0);
    cp_async_commit();
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    mu_rows(ring + kHSlot, ring + 2 * kHSlot, ring + 3 * kHSlot, mu, ms);  // mu(z0)
#pragma unroll
    for (int j = 0; j < kHR; ++j) fup[j] = ch_flux4<QUANT>(k, mu[j + 1], ml[j + 1]);
    s0 = 2;
  }
  const bool full = x0 + kHRow <= nx && y0 + kHR <= ny &&
                    (sizeof(Off) == 4 || ((uintptr_t)out & 15) == 0);
  float vmax = 0.f;
  F2 vsum = sp(0.f);
  long long acc_q = 0;
  double acc = 0.0;
  float* orow0 = out + (int64_t)z0 * g.plane + (int64_t)y0 * g.pitch + x;
  for (int z = z0; z < z1; ++z, orow0 += g.plane) {
    const float* S0 = ring + s0 * kHSlot;
    // this plane's side mu to the lanes that use them
    if (lane < 2 * kHR) smu[(z & 1) * 8 + lane] = ms;
    Quad mun[kHR + 2];
    if (!FLAT) {
      const int sa = (s0 + 1) & (kHD - 1), sb = (s0 + 2) & (kHD - 1);
      asm volatile("cp.async.wait_group 0;" ::: "memory");  // plane z + 2
      __syncwarp();  // every lane is done with plane z - 1, whose slot is refilled
      if (z + 1 < z1) {
        issue(z + 3, (s0 + 3) & (kHD - 1));
        cp_async_commit();
      }
      mu_rows(S0, ring + sa * kHSlot, ring + sb * kHSlot, mun, ms);
    } else {
      __syncwarp();
    }
    const float4 side = *reinterpret_cast<const float4*>(smu + (z & 1) * 8 + (lane == 31 ? 4 : 0));
    const float sm[4] = {side.x, side.y, side.z, side.w};
    Quad fs = ch_flux4<QUANT>(k, mu[1], mu[0]);  // the face north of row 0
    int32_t quanta = 0;
    float* orow = orow0;
#pragma unroll
    for (int j = 0; j < kHR; ++j, orow += g.pitch) {
      const Quad m = mu[j + 1];
      const float m0 = lo(m.a), m1 = hi(m.a), m2 = lo(m.b), m3 = hi(m.b);
      float mw = __shfl_up_sync(0xffffffffu, m3, 1);
      float me = __shfl_down_sync(0xffffffffu, m0, 1);
      if (lane == 0) mw = sm[j];
      if (lane == 31) me = sm[j];
      // the faces east of the cells and west of the first
      const Quad fe = ch_scale4<QUANT>(k, {pk(m1 - m0, m2 - m1), pk(m3 - m2, me - m3)});
      const float fw = ch_scale<QUANT>(k, m0 - mw);
      const float e0 = lo(fe.a), e1 = hi(fe.a), e2 = lo(fe.b), e3 = hi(fe.b);
      const Quad fx = {pk(e0 - fw, e1 - e0), pk(e2 - e1, e3 - e2)};
      const Quad fn = fs;
      fs = ch_flux4<QUANT>(k, mu[j + 2], m);
      const Quad c = row(S0, j + 2);
      Quad sum = fx + (fs - fn);
      if (!FLAT) {
        const Quad fu = ch_flux4<QUANT>(k, mun[j + 1], m);
        sum = sum + (fu - fup[j]);
        fup[j] = fu;
      }
      const Quad v = c + sum;
      const float o[4] = {lo(v.a), hi(v.a), lo(v.b), hi(v.b)};
      if (full) {
        *reinterpret_cast<float4*>(orow) = make_float4(o[0], o[1], o[2], o[3]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          vmax = fmaxf(vmax, fabsf(o[e]));
          if (!QUANT) acc += (double)o[e];
        }
        if (QUANT) {  // exact: |v / q| < 2^24
          const F2 qa = v.a * sp(k.iq), qb = v.b * sp(k.iq);
          quanta += __float2int_rn(lo(qa)) + __float2int_rn(hi(qa));
          quanta += __float2int_rn(lo(qb)) + __float2int_rn(hi(qb));
        }
        vsum = vsum + (v.a + v.b);
      } else if (y0 + j < ny) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (x + e < nx) {
            orow[e] = o[e];
            vmax = fmaxf(vmax, fabsf(o[e]));
            if (QUANT) quanta += __float2int_rn(o[e] * k.iq);
            else acc += (double)o[e];
            vsum = vsum + pk(o[e], 0.f);
          }
      }
    }
    acc_q += quanta;
    if (!FLAT) {
#pragma unroll
      for (int i = 0; i < kHR + 2; ++i) mu[i] = mun[i];
      s0 = (s0 + 1) & (kHD - 1);
    }
  }
  cp_async_wait_all();
  int flags = 0;
  const float vs = lo(vsum) + hi(vsum);
  if (QUANT && !(vmax < k.range)) flags |= PPF_STATUS_RANGE;
  if (!isfinite(vs) || !isfinite(vmax)) flags |= PPF_STATUS_NONFINITE;
  if (status && flags) atomicOr(status, flags);
  if (mass) {
    // QUANT: whole quanta (|sum| < 2^53): the same total in any order
    double v = QUANT ? (double)acc_q : acc;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) atomicAdd(mass, QUANT ? v * (double)k.q : v);
  }
}

// ------------------------------------------------------------- host side
template <typename T>
int32_t plan3d(const PpfTiling* t, const Geo& g, int halo, int nslots, int mu_planes,
               MarchGeom* m, int* slot_elems, size_t* smem) {
  m->TX = t && t->tile_x ? t->tile_x : 64;
  m->TY = t && t->tile_y ? t->tile_y : 16;
  m->H = halo;
  if (t && t->depth > 1)
    return fail(PPF_ERR_UNSUPPORTED, "3-D steps advance one step per pass (depth=%d)", t->depth);
  if (m->TX < 4 || m->TX > 256 - 2 * kXOff || (m->TX % 4) != 0 || m->TY < 1 ||
      m->TY + 2 * halo > 256)
    return fail(PPF_ERR_INVALID, "tile %dx%d invalid (tile_x multiple of 4, <= %d)", m->TX,
                m->TY, 256 - 2 * kXOff);
  m->BX = m->TX + 2 * kXOff;
  m->BY = m->TY + 2 * halo;
  if (t && t->zchunk < 0) return fail(PPF_ERR_INVALID, "zchunk must be >= 0");
  m->ZC = 0;  // set by the caller (zchunk_of)
  const size_t slot_bytes = ((size_t)m->BX * m->BY * sizeof(T) + 127) / 128 * 128;
  *slot_elems = (int)(slot_bytes / sizeof(T));
  *smem = 128 + (size_t)nslots * slot_bytes +
          (size_t)mu_planes * (m->TX + 2) * (m->TY + 2) * sizeof(T);
  if (*smem > 200 * 1024)
    return fail(PPF_ERR_INVALID, "tile needs %zu bytes of shared memory", *smem);
  return PPF_OK;
}

// Planes per CTA along z when the caller leaves it open: short chunks (many
// CTAs in flight over a compact stretch of z) measured fastest on GB300 for
// both 3-D kernels (384^3 and 512^3: 8-16 planes beat 32-64 by 1.3-1.9x, and
// sizing the chunks to one wave of CTAs was slower still).
constexpr int kDefaultZChunk = 12;

int zchunk_of(const PpfTiling* t, const Geo& g) {
  const int zc = t && t->zchunk > 0 ? t->zchunk : kDefaultZChunk;
  return zc < g.n[0] ? zc : g.n[0];
}

// The same for the lean 7-point kernel: a chunk of zc planes copies zc + 2, and a
// warp advances one plane after the other, so chunks are as short as it takes to
// have a dozen warps per SM (float, us per step with 2 / 4 / 8 planes: 64^3 3.8 /
// 5.7 / 9.4, 128^3 5.2 / 5.7 / 7.9, 256^3 30 / 29 / 26, 512^3 196 / 178 / 170,
// 16 planes 176). More where gridDim.z would not hold the chunks.
int lean_zchunk(long warps, int nz) {
  int zc = 8;
  while (zc > 2 && warps * ((nz + zc - 1) / zc) < 2048) zc /= 2;
  if (zc < (nz + 65534) / 65535) zc = (nz + 65534) / 65535;
  return zc < nz ? zc : nz;
}

template <typename T>
int32_t plane_map(CUtensorMap* map, const T* base, const Geo& g, const MarchGeom& m) {
  const uint64_t dims[3] = {(uint64_t)g.n[2], (uint64_t)g.n[1], (uint64_t)g.n[0]};
  const uint64_t strides[2] = {(uint64_t)g.pitch * sizeof(T), (uint64_t)g.plane * sizeof(T)};
  const uint32_t box[3] = {(uint32_t)m.BX, (uint32_t)m.BY, 1u};
  return tensor_map(map, base, (int)sizeof(T), 3, dims, strides, box);
}

// A 2-D grid runs as a single-plane 3-D grid with a periodic z axis (the
// z neighbours are the cell itself and cancel in the Laplacian).
int32_t as3d(const PpfGrid* in, const PpfBoundary* bin, PpfGrid* g3, PpfBoundary* b3) {
  if (!in) return fail(PPF_ERR_INVALID, "grid is NULL");
  if (!bin) return fail(PPF_ERR_INVALID, "boundary is NULL");
  *g3 = *in;
  *b3 = *bin;
  if (in->ndim == 2) {
    g3->ndim = 3;
    g3->shape[2] = in->shape[1];
    g3->shape[1] = in->shape[0];
    g3->shape[0] = 1;
    b3->type[2] = bin->type[1];
    b3->type[1] = bin->type[0];
    b3->type[0] = PPF_BC_PERIODIC;
    for (int f = 0; f < 2; ++f)
      for (int s = 0; s < 2; ++s) {
        b3->value[f][2][s] = bin->value[f][1][s];
        b3->value[f][1][s] = bin->value[f][0][s];
        b3->value[f][0][s] = 0.0;
      }
  }
  return PPF_OK;
}

// Rows per lane: four re-read half a row per row, two a whole one; in double, where
// the FP64 units bind, fewer registers win (200^3: 4 %).
template <typename T>
constexpr int kLeanRows = sizeof(T) == 4 ? 4 : 2;

template <typename T>
long lean_warps(const Geo& g, int lx) {
  const int ww = lx * Vec16<T>::n, rows = kLeanRows<T> * (32 / lx);
  return (long)((g.n[2] + ww - 1) / ww) * ((g.n[1] + rows - 1) / rows);
}

// Lanes per row: 32, or 16 or 8 where a row of 32 vectors would reach far past nx:
// the fewest warps, each weighed by what its shorter rows cost (more rows and side
// cells read beside them). In double the FP64 units bind and idle lanes cost as much
// as busy ones: 300 x 400 x 24, us per step with 32 / 16 / 8 lanes: 208 / 115 / 116,
// 300 x 300 x 200 566 / 493 / 468, 300 x 200 x 50 114 / 114 / 125 (the 32 x 32 tiles
// before: 166, 581, 176). In float: 300 x 400 x 24 27 / 19 / 13, 200 x 200 x 180
// 21.2 / 17.4 / 20.7, but 300 x 300 x 200 38.9 / 46 / 52 (48, 65, 98).
template <typename T>
int lean_lanes(const Geo& g) {
  const bool f = sizeof(T) == 4;
  const double c32 = lean_warps<T>(g, 32), c16 = (f ? 1.2 : 1.08) * lean_warps<T>(g, 16),
               c8 = (f ? 1.5 : 1.12) * lean_warps<T>(g, 8);
  return c32 <= c16 && c32 <= c8 ? 32 : c16 <= c8 ? 16 : 8;
}

template <typename T, typename Op, int LX>
int32_t launch_lean7(Op op, const Geo& g, const Bc<T>& bc, const T* in, T* out, int zc, bool pdl,
                     cudaStream_t s) {
  constexpr int R = kLeanRows<T>, D = 4, WW = LX * Vec16<T>::n, rows = R * (32 / LX) * kLWarps;
  const int strips = (g.n[2] + WW - 1) / WW, bands = (g.n[1] + rows - 1) / rows;
  if (!zc) zc = lean_zchunk((long)strips * bands * kLWarps, g.n[0]);
  auto kern = lean7_kernel<T, Op, R, D, LX>;
  const size_t smem = (size_t)kLWarps * D * Lean7Slot<T, R, LX>::elems * sizeof(T);
  PPF_TRY_CUDA(allow_smem(kern, smem));
  for (int band = 0; band < bands; band += kMaxBands) {
    const dim3 gd(strips, min(bands - band, kMaxBands), (g.n[0] + zc - 1) / zc);
    PPF_TRY_CUDA(launch(kern, gd, dim3(32, kLWarps), smem, s, pdl, op, g, bc, in, out, zc,
                        band * rows));
  }
  return PPF_OK;
}

template <typename T, typename Op>
int32_t run_march7(Op op, double dx, const PpfGrid* grid, const PpfBoundary* b, const T* in,
                   T* out, const PpfTiling* tiling, void* stream) {
  Geo g;
  int32_t rc = make_geo(grid, 3, 3, &g);
  if (rc) return rc;
  if (!in || !out) return fail(PPF_ERR_INVALID, "NULL field pointer");
  if (in == out) return fail(PPF_ERR_INVALID, "in and out must differ");
  Bc<T> bc;
  if ((rc = make_bc<T>(b, g, dx, 1, 1, &bc))) return rc;
  MarchGeom m;
  int slot_elems;
  size_t smem;
  int* st = status_ptr();
  if (!st) return fail(PPF_ERR_CUDA, "status word unavailable");
  const bool own = !tiling || ((tiling->tile_x == 0 || tiling->tile_x == 32) &&
                               (tiling->tile_y == 0 || tiling->tile_y == 32));
  if (own && g.plane < (1LL << 31) && (uintptr_t)out % 16 == 0) {
    PpfTiling lt{};
    lt.depth = tiling ? tiling->depth : 0;
    if ((rc = plan3d<T>(&lt, g, 1, kNS7, 0, &m, &slot_elems, &smem))) return rc;
    if ((uintptr_t)in % 16) return fail(PPF_ERR_INVALID, "field base not 16-byte aligned");
    const cudaStream_t st7 = (cudaStream_t)stream;
    const bool pdl = tiling && tiling->pdl;
    const int zc = tiling && tiling->zchunk > 0 ? zchunk_of(tiling, g) : 0;
    switch (lean_lanes<T>(g)) {
      case 8: return launch_lean7<T, Op, 8>(op, g, bc, in, out, zc, pdl, st7);
      case 16: return launch_lean7<T, Op, 16>(op, g, bc, in, out, zc, pdl, st7);
      default: return launch_lean7<T, Op, 32>(op, g, bc, in, out, zc, pdl, st7);
    }
  }
  // tiles: asked for, or outputs off a 16-byte boundary and planes beyond 32-bit offsets
  PpfTiling tt{};
  if (tiling) tt = *tiling;
  if (own) tt.tile_x = tt.tile_y = 32, tt.zchunk = 0;  // (its sign is not looked at here)
  if ((rc = plan3d<T>(&tt, g, 1, kNS7, 0, &m, &slot_elems, &smem))) return rc;
  m.ZC = zchunk_of(tiling, g);
  CUtensorMap map;
  if ((rc = plane_map<T>(&map, in, g, m))) return rc;
  auto kern = march7_kernel<T, Op>;
  PPF_TRY_CUDA(allow_smem(kern, smem));
  dim3 gd((g.n[2] + m.TX - 1) / m.TX, (g.n[1] + m.TY - 1) / m.TY, (g.n[0] + m.ZC - 1) / m.ZC);
  PPF_TRY_CUDA(launch(kern, gd, dim3(32, kThreads / 32), smem, (cudaStream_t)stream,
                      tiling && tiling->pdl, map, op, g, bc, in, out, m, slot_elems, st));
  return PPF_OK;
}

// Planes per warp: one wave of CTAs (three per SM: registers and shared memory)
// where 2 to 32 planes make one, since a warp's planes follow one another and a
// second wave that is nearly empty costs a whole one (256^3, us per step: 42.3 with
// 19 planes, 46.8 with 12, 47.6 with 8, 65.6 with 32; 384^3: 130 with 32, 141 with 8).
int32_t run_ch_march(const ChCoef<float>& k, const Geo& g, const Bc<float>& bc, const float* in,
                     float* out, double* mass, int* status, const PpfTiling* tiling, bool quant,
                     bool pdl, cudaStream_t s) {
  const bool flat = g.n[0] == 1 && bc.type[0] == PPF_BC_PERIODIC;
  const int strips = (g.n[2] + kHRow - 1) / kHRow;
  const int bands = (g.n[1] + kHR * kHWarps - 1) / (kHR * kHWarps);
  int zc = tiling && tiling->zchunk > 0 ? tiling->zchunk : 0;
  if (!zc) {
    int dev = 0, sms = 0;
    PPF_TRY_CUDA(cudaGetDevice(&dev));
    PPF_TRY_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const long fit = 3L * sms / ((long)strips * bands);  // chunks of one wave
    zc = fit > 0 ? (int)((g.n[0] + fit - 1) / fit) : 32;
    zc = zc < 2 ? 2 : zc > 32 ? 32 : zc;
  }
  zc = zc < g.n[0] ? zc : g.n[0];
  const size_t smem = (size_t)kHWarps * (flat ? kHWarpElems<true> : kHWarpElems<false>) * sizeof(float);
  auto pick = [&](auto off) {
    using Off = decltype(off);
    return quant ? (flat ? ch_march_kernel<true, true, Off> : ch_march_kernel<true, false, Off>)
                 : (flat ? ch_march_kernel<false, true, Off> : ch_march_kernel<false, false, Off>);
  };
  const bool small = g.plane < (1LL << 31) && bands <= kMaxBands && (uintptr_t)out % 16 == 0;
  auto kern = small ? pick(uint32_t{}) : pick(int64_t{});
  PPF_TRY_CUDA(allow_smem(kern, smem));
  for (int band = 0; band < bands; band += kMaxBands) {
    const dim3 gd(strips, min(bands - band, kMaxBands), (g.n[0] + zc - 1) / zc);
    PPF_TRY_CUDA(launch(kern, gd, dim3(32, kHWarps), smem, s, pdl, k, g, bc, in, out, mass, status,
                        zc, band * kHR * kHWarps));
  }
  return PPF_OK;
}

template <typename T>
int32_t cahn_hilliard(const PpfCahnHilliardParams* p, const PpfGrid* grid_in,
                      const PpfBoundary* b_in, const T* in, T* out, double* mass,
                      int32_t* status, const PpfTiling* tiling, void* stream) {
  clear_error();
  if (!p) return fail(PPF_ERR_INVALID, "params is NULL");
  if (!(p->dx > 0)) return fail(PPF_ERR_INVALID, "dx must be > 0");
  PpfGrid grid;
  PpfBoundary b;
  int32_t rc = as3d(grid_in, b_in, &grid, &b);
  if (rc) return rc;
  Geo g;
  if ((rc = make_geo(&grid, 3, 3, &g))) return rc;
  if (!in || !out) return fail(PPF_ERR_INVALID, "NULL field pointer");
  if (in == out) return fail(PPF_ERR_INVALID, "in and out must differ");
  for (int a = 0; a < 3; ++a) {
    if (b.type[a] == PPF_BC_DIRCHLET)
      return fail(PPF_ERR_UNSUPPORTED, "Cahn-Hilliard supports PERIODIC and NEUMANN axes only");
    if (b.type[a] == PPF_BC_NEUMANN && (b.value[0][a][0] != 0.0 || b.value[0][a][1] != 0.0))
      return fail(PPF_ERR_UNSUPPORTED, "Cahn-Hilliard NEUMANN axes must be no-flux (gradient 0)");
  }
  Bc<T> bc;
  if ((rc = make_bc<T>(&b, g, p->dx, 1, 2, &bc))) return rc;
  MarchGeom m;
  int slot_elems;
  size_t smem;
  if (tiling && ((tiling->tile_x && tiling->tile_x != kCTX) ||
                 (tiling->tile_y && tiling->tile_y != kCTY)))
    return fail(PPF_ERR_UNSUPPORTED, "Cahn-Hilliard tiles are %dx%d", kCTX, kCTY);
  PpfTiling ct{};
  ct.depth = tiling ? tiling->depth : 0;
  ct.tile_x = kCTX;
  ct.tile_y = kCTY;
  if ((rc = plan3d<T>(&ct, g, 2, kNSC, kMuSlots, &m, &slot_elems, &smem))) return rc;
  ChCoef<T> k;
  k.kap = (T)(p->epsilon * p->epsilon / (p->dx * p->dx));
  k.a = (T)(p->dt * p->M / (p->dx * p->dx));
  const bool quant = p->quantum > 0;
  if (quant) {
    int e;
    const double mant = std::frexp(p->quantum, &e);
    if (mant != 0.5 || sizeof(T) != 4)
      return fail(PPF_ERR_INVALID, "quantum must be a power of two and needs the float path");
  }
  k.q = (T)(quant ? p->quantum : 0.0);
  k.iq = (T)(quant ? 1.0 / p->quantum : 0.0);
  k.aiq = (T)(quant ? (double)k.a * (1.0 / p->quantum) : 0.0);
  k.range = (T)(quant ? std::ldexp(p->quantum, 24) : 0.0);
  if (p->centered != 0 && p->centered != 1)
    return fail(PPF_ERR_INVALID, "centered must be 0 or 1");
  k.centered = p->centered;
  const bool pdl = tiling && tiling->pdl;
  if constexpr (sizeof(T) == 4) {
    if ((uintptr_t)in % 16) return fail(PPF_ERR_INVALID, "field base not 16-byte aligned");
    return run_ch_march(k, g, bc, in, out, mass, (int*)status, tiling, quant, pdl,
                        (cudaStream_t)stream);
  } else {
    if (slot_elems != kCSlot || m.BX != kCW || m.BY != kCH)
      return fail(PPF_ERR_INVALID, "Cahn-Hilliard plane slot mismatch");
    CUtensorMap map;
    if ((rc = plane_map<T>(&map, in, g, m))) return rc;
    int* st = status_ptr();
    if (!st) return fail(PPF_ERR_CUDA, "status word unavailable");
    m.ZC = zchunk_of(tiling, g);
    const dim3 gd((g.n[2] + m.TX - 1) / m.TX, (g.n[1] + m.TY - 1) / m.TY,
                  (g.n[0] + m.ZC - 1) / m.ZC);
    auto kern = cahn_hilliard_kernel<T>;
    PPF_TRY_CUDA(allow_smem(kern, smem));
    PPF_TRY_CUDA(launch(kern, gd, dim3(32, kThreads / 32), smem, (cudaStream_t)stream, pdl, map, k,
                        g, bc, in, out, mass, (int*)status, m, slot_elems, st));
  }
  return PPF_OK;
}

}  // namespace

int32_t diffusion3d_f32(const PpfDiffusionParams* p, const PpfGrid* g, const PpfBoundary* b,
                        const float* in, float* out, const PpfTiling* t, void* s) {
  clear_error();
  if (!p || !(p->dx > 0)) return fail(PPF_ERR_INVALID, "bad params");
  return run_march7<float>(Diffusion7<float>{(float)(p->dt * p->D / (p->dx * p->dx))}, p->dx, g,
                           b, in, out, t, s);
}
int32_t diffusion3d_f64(const PpfDiffusionParams* p, const PpfGrid* g, const PpfBoundary* b,
                        const double* in, double* out, const PpfTiling* t, void* s) {
  clear_error();
  if (!p || !(p->dx > 0)) return fail(PPF_ERR_INVALID, "bad params");
  return run_march7<double>(Diffusion7<double>{p->dt * p->D / (p->dx * p->dx)}, p->dx, g, b, in,
                            out, t, s);
}
int32_t allen_cahn3d_f32(const PpfAllenCahnParams* p, const PpfGrid* g, const PpfBoundary* b,
                         const float* in, float* out, const PpfTiling* t, void* s) {
  clear_error();
  if (!p || !(p->dx > 0)) return fail(PPF_ERR_INVALID, "bad params");
  AllenCahn7<float> op{(float)(p->dt * p->M * p->epsilon * p->epsilon / (p->dx * p->dx)),
                       (float)(p->dt * p->M * 16.0 * p->W)};
  return run_march7<float>(op, p->dx, g, b, in, out, t, s);
}
int32_t allen_cahn3d_f64(const PpfAllenCahnParams* p, const PpfGrid* g, const PpfBoundary* b,
                         const double* in, double* out, const PpfTiling* t, void* s) {
  clear_error();
  if (!p || !(p->dx > 0)) return fail(PPF_ERR_INVALID, "bad params");
  AllenCahn7<double> op{p->dt * p->M * p->epsilon * p->epsilon / (p->dx * p->dx),
                        p->dt * p->M * 16.0 * p->W};
  return run_march7<double>(op, p->dx, g, b, in, out, t, s);
}

}  // namespace ppf

using namespace ppf;

extern "C" {

int32_t ppf_cahn_hilliard_step_f32(const PpfCahnHilliardParams* p, const PpfGrid* g,
                                   const PpfBoundary* bc, const float* in, float* out,
                                   double* mass_accum, int32_t* status, const PpfTiling* tiling,
                                   void* stream) {
  return cahn_hilliard<float>(p, g, bc, in, out, mass_accum, status, tiling, stream);
}
int32_t ppf_cahn_hilliard_step_f64(const PpfCahnHilliardParams* p, const PpfGrid* g,
                                   const PpfBoundary* bc, const double* in, double* out,
                                   double* mass_accum, int32_t* status, const PpfTiling* tiling,
                                   void* stream) {
  return cahn_hilliard<double>(p, g, bc, in, out, mass_accum, status, tiling, stream);
}

}  // extern "C"
