// Implicit and Crank-Nicolson diffusion: pyphasefield's engines
// engine_ImplicitDiffusion{1,2,3}D[_ADI], engine_CrankNicolsonDiffusion{1,2,3}D[_ADI]
// and their *_GMRES twins (Engines/Diffusion.py:210-633), on periodic
// interior grids (the reference's matrices are periodic, Diffusion.py:18-196).
//
// Line solves (1-D engines and the ADI engines). Along one axis every line
// solves the periodic system (1 + 2a) x_i - a (x_{i-1} + x_{i+1}) = d_i. With
// r in (0, 1) the root of a r^2 - (1 + 2a) r + a = 0 the operator factors as
// (a / r)(I - r S)(I - r S^-1), S the cyclic shift, so
//   y_i = (r / a) d_i + r y_{i-1}   (cyclic forward recurrence)
//   x_i = y_i + r x_{i+1}           (cyclic backward recurrence)
// Both recurrences contract (|r| < 1). Each line is cut into segments; a
// segment's local sums with zero carry (pass 1), a short per-line pass that
// closes the cyclic carries in the field's type, from constants formed in double
// (pass 2), and a pass that recomputes each segment from its true carries (pass 3)
// give the exact solution with three streaming kernels (12 bytes of traffic per
// cell and float). Lines of up to 4096 cells run the three passes in one launch
// (line_fused) where that is as exact (alpha up to 128) and faster (three_launches).
//   - lines along y or z: one thread per (column, 32-cell segment), threads
//     of a warp on adjacent columns, so every load and store is coalesced;
//   - lines along x: one warp per 256-cell segment, cell i of a 32-cell
//     chunk in lane i, the recurrence across lanes as a weighted warp scan.
// The Crank-Nicolson explicit half step (1 - 2a) c + a (c[-e] + c[+e]) along
// any axis e is folded into the right-hand side loads.
//
// Full systems (2-D and 3-D engines without ADI): the reference factors the
// dense N x N matrix. Here the Chebyshev semi-iteration runs on the 2d+1
// point operator, whose spectrum [1, 1 + 4 d a] is known in closed form, so
// the iteration count for a given error bound is fixed before the first
// iteration: one fused stencil kernel per iteration, no reductions.
#include <math.h>

#include "ppf_lines.cuh"

namespace ppf {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kSeg = 32;      // lines along y/z: cells per thread segment
constexpr int kLineThreads = 128;

template <typename T>
struct V2;
template <>
struct V2<float> {
  using type = float2;
};
template <>
struct V2<double> {
  using type = double2;
};

// Lines of one solve. Physical axes: x (contiguous), y (rows), z (planes).
struct Lines {
  int n;           // cells per line
  int nseg;        // segments per line
  int seglen;      // kSeg or kXSegV
  int nlines;
  int64_t stride;  // elements between consecutive cells of a line
  // lines along y or z: line = o * nx + x, o the remaining axis
  int nx, no;
  int64_t ostride;
  // lines along x: line = z * ny + y
  int ny;
  int64_t pitch, plane;
  // explicit part of the right-hand side
  int expl;        // 0 none, 1 along the solved axis, 2 along another axis
  int e_is_x;      // expl == 2 on y/z lines: the other axis is x (else the remaining one)
  int e_is_y;      // expl == 2 on x lines: the other axis is y (else z)
  int ne;          // extent of the explicit axis
  int64_t estride;
};

template <typename T>
struct LineCoef {
  T r, kappa;   // recurrence root and r / a (the recurrences run on d,
                // the solution is kappa times their result)
  T w0, w1;     // rhs = w0 c + w1 (c[-e] + c[+e])
  T rpow[33];   // r^0 .. r^32 (compile-time indices only)
  T rbit[8];    // r^1, r^2, r^4, ..., r^128
};

template <typename T>
struct CarryCoef {
  T R, G;       // r^L and sum_{k<L} r^(2k+1) of a full segment
  T Rl, Gl;     // the same for the last segment
  T inv_close;  // 1 / (1 - r^n)
  T Rp[6];      // R^1, R^2, R^4, R^8, R^16, R^32
};

// p[b] = q^(2^b), b < NB (compile-time indices only: a lane-dependent index
// into kernel parameters would serialise the warp on the constant cache).
// Returns q^e for 0 <= e < 2^NB.
template <int NB, typename T>
__device__ __forceinline__ T pow_bits(const T* p, int e) {
  T v = T(1);
#pragma unroll
  for (int b = 0; b < NB; ++b)
    if ((e >> b) & 1) v *= p[b];
  return v;
}

// Offsets of the two neighbours of coordinate q along an axis of extent n
// and stride st, periodic.
__device__ __forceinline__ void wrap_offsets(int q, int n, int64_t st, int64_t& om,
                                             int64_t& op) {
  om = (q == 0 ? (int64_t)(n - 1) : (int64_t)-1) * st;
  op = (q == n - 1 ? (int64_t)(1 - n) : (int64_t)1) * st;
}

// ---------------------------------------------------------------- y/z lines
// A thread takes one 32-cell segment of two adjacent columns (x, x + 1): one
// 8- or 16-byte load per cell pair, two independent recurrences.
struct StridedIdx {
  int x, o, s;
  int64_t base;
  bool ok, pair;
};

__device__ __forceinline__ StridedIdx strided_index(const Lines& L) {
  StridedIdx r;
  r.x = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
  const int64_t so = (int64_t)blockIdx.y + (int64_t)gridDim.y * blockIdx.z;
  r.ok = r.x < L.nx && so < (int64_t)L.nseg * L.no;
  r.pair = r.x + 1 < L.nx;
  r.s = (int)(so % L.nseg);
  r.o = (int)(so / L.nseg);
  r.base = r.x + (int64_t)r.o * L.ostride;
  return r;
}

// Two adjacent cells (the second 0 when the column does not exist); the
// offset is even, so the vector load is aligned where the field is (VEC).
template <bool VEC, typename T>
__device__ __forceinline__ void load2(const T* __restrict__ p, bool pair, T (&v)[2]) {
  if (VEC && pair) {
    if constexpr (sizeof(T) == 4) {
      const float2 q = __ldg(reinterpret_cast<const float2*>(p));
      v[0] = q.x, v[1] = q.y;
    } else {
      const double2 q = __ldg(reinterpret_cast<const double2*>(p));
      v[0] = q.x, v[1] = q.y;
    }
  } else {
    v[0] = __ldg(p);
    v[1] = !VEC && pair ? __ldg(p + 1) : T(0);
  }
}

template <bool VEC, typename T>
__device__ __forceinline__ void store2(T* p, bool pair, T a, T b) {
  if (VEC && pair) {
    if constexpr (sizeof(T) == 4)
      *reinterpret_cast<float2*>(p) = make_float2(a, b);
    else
      *reinterpret_cast<double2*>(p) = make_double2(a, b);
  } else {
    *p = a;
    if (!VEC && pair) p[1] = b;
  }
}

// Offsets of the explicit part's neighbours, per column.
struct EOff {
  int64_t m[2], p[2];
};

template <int EXPL>
__device__ __forceinline__ EOff strided_eoffsets(const Lines& L, const StridedIdx& id) {
  EOff e{};
  if (EXPL == 2) {
    if (L.e_is_x) {
      wrap_offsets(id.x, L.ne, 1, e.m[0], e.p[0]);
      wrap_offsets(id.x + 1 < L.ne ? id.x + 1 : 0, L.ne, 1, e.m[1], e.p[1]);
    } else {
      wrap_offsets(id.o, L.ne, L.estride, e.m[0], e.p[0]);
      e.m[1] = e.m[0], e.p[1] = e.p[0];
    }
  }
  return e;
}

// Right-hand side of the cell pair at line position i (pointer p).
template <typename T, int EXPL, bool VEC>
__device__ __forceinline__ void rhs2(const T* __restrict__ p, const Lines& L,
                                     const LineCoef<T>& k, const StridedIdx& id, int i,
                                     const EOff& e, T (&d)[2]) {
  load2<VEC>(p, id.pair, d);
  if (EXPL == 0) return;
  T a[2], b[2];
  if (EXPL == 1) {
    int64_t om, op;
    wrap_offsets(i, L.n, L.stride, om, op);
    load2<VEC>(p + om, id.pair, a);
    load2<VEC>(p + op, id.pair, b);
  } else if (L.e_is_x) {
    a[0] = __ldg(p + e.m[0]);
    b[0] = __ldg(p + e.p[0]);
    a[1] = id.pair ? __ldg(p + 1 + e.m[1]) : T(0);
    b[1] = id.pair ? __ldg(p + 1 + e.p[1]) : T(0);
  } else {
    load2<VEC>(p + e.m[0], id.pair, a);
    load2<VEC>(p + e.p[0], id.pair, b);
  }
#pragma unroll
  for (int c = 0; c < 2; ++c) d[c] = k.w0 * d[c] + k.w1 * (a[c] + b[c]);
}

// Pass 1: per segment, y's end value with zero carry (F) and the sum of
// r^(i - start) y_i over the segment (Bu).
template <typename T, int EXPL, bool VEC>
__global__ void __launch_bounds__(kLineThreads)
    line_sums_yz(Lines L, LineCoef<T> k, const T* __restrict__ in,
                 typename V2<T>::type* __restrict__ seg) {
  pdl_wait();
  pdl_launch_next();
  const StridedIdx id = strided_index(L);
  if (!id.ok) return;
  const EOff e = strided_eoffsets<EXPL>(L, id);
  const int i0 = id.s * kSeg;
  const int len = min(kSeg, L.n - i0);
  const T* p = in + id.base + (int64_t)i0 * L.stride;
  T d[kSeg][2];
  if (len == kSeg) {
#pragma unroll
    for (int j = 0; j < kSeg; ++j) rhs2<T, EXPL, VEC>(p + (int64_t)j * L.stride, L, k, id, i0 + j, e, d[j]);
  } else {
#pragma unroll
    for (int j = 0; j < kSeg; ++j) {
      if (j < len)
        rhs2<T, EXPL, VEC>(p + (int64_t)j * L.stride, L, k, id, i0 + j, e, d[j]);
      else
        d[j][0] = d[j][1] = T(0);
    }
  }
  T u0 = 0, u1 = 0, b0 = 0, b1 = 0;
#pragma unroll
  for (int j = 0; j < kSeg; ++j) {
    if (j < len) {
      u0 = fma(k.r, u0, d[j][0]);
      u1 = fma(k.r, u1, d[j][1]);
      b0 = fma(k.rpow[j], u0, b0);
      b1 = fma(k.rpow[j], u1, b1);
    }
  }
  typename V2<T>::type* q = seg + (int64_t)id.s * L.nlines + (int64_t)id.o * L.nx + id.x;
  q[0] = {u0, b0};
  if (id.pair) q[1] = {u1, b1};
}

// Pass 3: the segment again, from its true carries.
template <typename T, int EXPL, bool VEC>
__global__ void __launch_bounds__(kLineThreads)
    line_solve_yz(Lines L, LineCoef<T> k, const T* __restrict__ in,
                  const typename V2<T>::type* __restrict__ seg, T* __restrict__ out) {
  pdl_wait();
  pdl_launch_next();
  const StridedIdx id = strided_index(L);
  if (!id.ok) return;
  const EOff e = strided_eoffsets<EXPL>(L, id);
  const int i0 = id.s * kSeg;
  const int len = min(kSeg, L.n - i0);
  const int64_t off0 = id.base + (int64_t)i0 * L.stride;
  const typename V2<T>::type* q = seg + (int64_t)id.s * L.nlines + (int64_t)id.o * L.nx + id.x;
  const typename V2<T>::type c0 = q[0];
  const typename V2<T>::type c1 = id.pair ? q[1] : c0;
  T y[kSeg][2];
  if (len == kSeg) {
#pragma unroll
    for (int j = 0; j < kSeg; ++j)
      rhs2<T, EXPL, VEC>(in + off0 + (int64_t)j * L.stride, L, k, id, i0 + j, e, y[j]);
  } else {
#pragma unroll
    for (int j = 0; j < kSeg; ++j) {
      if (j < len)
        rhs2<T, EXPL, VEC>(in + off0 + (int64_t)j * L.stride, L, k, id, i0 + j, e, y[j]);
      else
        y[j][0] = y[j][1] = T(0);
    }
  }
  T y0 = c0.x, y1 = c1.x;
#pragma unroll
  for (int j = 0; j < kSeg; ++j) {
    y0 = fma(k.r, y0, y[j][0]);
    y1 = fma(k.r, y1, y[j][1]);
    y[j][0] = y0;
    y[j][1] = y1;
  }
  T x0 = c0.y, x1 = c1.y;
#pragma unroll
  for (int j = kSeg - 1; j >= 0; --j) {
    if (j < len) {
      x0 = fma(k.r, x0, y[j][0]);
      x1 = fma(k.r, x1, y[j][1]);
      store2<VEC>(out + off0 + (int64_t)j * L.stride, id.pair, k.kappa * x0, k.kappa * x1);
    }
  }
}

// ---------------------------------------------------------------- x lines
// A warp takes a 512-cell segment of a row as 4 chunks of 128 cells, lane j
// holding cells 4j .. 4j+3 of a chunk (one 16-byte load). Within a lane the
// recurrence runs over its 4 cells; across lanes it is a warp scan with
// weights r^4, r^8, ... (5 shuffles per 4 cells).
constexpr int kXC = 4;            // chunks per segment
constexpr int kXSegV = 128 * kXC;  // cells per segment

struct XIdx {
  int line, s, lane;
  int64_t row;
  bool ok;
};

__device__ __forceinline__ XIdx x_index(const Lines& L) {
  XIdx r;
  r.lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * (kLineThreads / 32) + (threadIdx.x >> 5);
  r.ok = w < (int64_t)L.nlines * L.nseg;  // uniform across the warp
  r.line = (int)(w / L.nseg);
  r.s = (int)(w % L.nseg);
  const int yy = r.line % L.ny, zz = r.line / L.ny;
  r.row = (int64_t)zz * L.plane + (int64_t)yy * L.pitch;
  return r;
}

// Cells i .. i+3 of a row (i a multiple of 4, so the 16 or 32 bytes are
// aligned where the field is, VEC: the pitch is a multiple of 4). Cells at or past n
// read 0; a vector that starts below n lies inside the row's pitch.
template <bool VEC, typename T>
__device__ __forceinline__ void load4(const T* __restrict__ row, int i, int n, T (&v)[4]) {
  if constexpr (!VEC) {
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = i + k < n ? __ldg(row + i + k) : T(0);
    return;
  }
  if (i >= n) {
    v[0] = v[1] = v[2] = v[3] = T(0);
    return;
  }
  if constexpr (sizeof(T) == 4) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(row + i));
    v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
  } else {
    const double2 a = __ldg(reinterpret_cast<const double2*>(row + i));
    const double2 b = __ldg(reinterpret_cast<const double2*>(row + i + 2));
    v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
  }
#pragma unroll
  for (int k = 1; k < 4; ++k)
    if (i + k >= n) v[k] = T(0);
}

// Right-hand side of the segment's cells: d[c][k] = cell 128c + 4 lane + k.
template <typename T, int EXPL, bool VEC>
__device__ __forceinline__ void x_rhs(const T* __restrict__ in, const Lines& L,
                                      const LineCoef<T>& k, const XIdx& id,
                                      T (&d)[kXC][4]) {
  const T* row = in + id.row;
  const int i0 = id.s * kXSegV;
#pragma unroll
  for (int c = 0; c < kXC; ++c) load4<VEC>(row, i0 + 128 * c + 4 * id.lane, L.n, d[c]);
  if (EXPL == 0) return;
  if (EXPL == 2) {
    int64_t em, ep;
    const int yy = id.line % L.ny, zz = id.line / L.ny;
    wrap_offsets(L.e_is_y ? yy : zz, L.ne, L.estride, em, ep);
#pragma unroll
    for (int c = 0; c < kXC; ++c) {
      T a[4], b[4];
      const int i = i0 + 128 * c + 4 * id.lane;
      load4<VEC>(row + em, i, L.n, a);
      load4<VEC>(row + ep, i, L.n, b);
#pragma unroll
      for (int q = 0; q < 4; ++q) d[c][q] = k.w0 * d[c][q] + k.w1 * (a[q] + b[q]);
    }
    return;
  }
  // along the row itself: neighbours inside the lane, from the lanes and
  // chunks beside, or (segment and line ends) from memory; every lane takes
  // part in every shuffle
  const T lo_edge = __ldg(row + (i0 == 0 ? L.n - 1 : i0 - 1));
  const T hi_edge = __ldg(row + (i0 + kXSegV < L.n ? i0 + kXSegV : 0));
  const T first = __ldg(row);
  T left[kXC], right[kXC];
#pragma unroll
  for (int c = 0; c < kXC; ++c) {
    const T up = __shfl_up_sync(kFull, d[c][3], 1);
    const T dn = __shfl_down_sync(kFull, d[c][0], 1);
    const T prev_last = __shfl_sync(kFull, d[c > 0 ? c - 1 : 0][3], 31);
    const T next_first = __shfl_sync(kFull, d[c < kXC - 1 ? c + 1 : 0][0], 0);
    left[c] = id.lane > 0 ? up : (c > 0 ? prev_last : lo_edge);
    right[c] = id.lane < 31 ? dn : (c < kXC - 1 ? next_first : hi_edge);
  }
#pragma unroll
  for (int c = 0; c < kXC; ++c) {
    const int i = i0 + 128 * c + 4 * id.lane;
    T v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const T l = q > 0 ? d[c][q > 0 ? q - 1 : 0] : left[c];
      T rr = q < 3 ? d[c][q < 3 ? q + 1 : 0] : right[c];
      if (i + q == L.n - 1) rr = first;
      v[q] = i + q < L.n ? k.w0 * d[c][q] + k.w1 * (l + rr) : T(0);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) d[c][q] = v[q];
  }
}

// Inclusive scans over lanes with weight r^(4 * distance).
template <typename T>
__device__ __forceinline__ T scan4_up(T t, const LineCoef<T>& k, int lane) {
#pragma unroll
  for (int b = 0; b < 5; ++b) {
    const T o = __shfl_up_sync(kFull, t, 1 << b);
    if (lane >= (1 << b)) t = fma(k.rbit[b + 2], o, t);
  }
  return t;
}

template <typename T>
__device__ __forceinline__ T scan4_down(T t, const LineCoef<T>& k, int lane) {
#pragma unroll
  for (int b = 0; b < 5; ++b) {
    const T o = __shfl_down_sync(kFull, t, 1 << b);
    if (lane + (1 << b) < 32) t = fma(k.rbit[b + 2], o, t);
  }
  return t;
}

// Forward recurrence u_i = d_i + r u_{i-1} over one chunk entered with
// `carry` (the u before the chunk); returns the chunk's u in u[4] and the u
// of its last valid cell (nv valid cells, 1..128).
template <typename T>
__device__ __forceinline__ T x_forward(const T (&d)[4], T carry, int nv, T w4j,
                                       const LineCoef<T>& k, int lane, T (&u)[4]) {
  u[0] = d[0];
  u[1] = fma(k.r, u[0], d[1]);
  u[2] = fma(k.r, u[1], d[2]);
  u[3] = fma(k.r, u[2], d[3]);
  const T S = scan4_up(u[3], k, lane);
  const T prev = __shfl_up_sync(kFull, S, 1);
  const T yin = fma(w4j, carry, lane > 0 ? prev : T(0));  // u before the lane's cells
  T rp = k.r;
#pragma unroll
  for (int q = 0; q < 4; ++q, rp *= k.r) u[q] = fma(rp, yin, u[q]);
  if (nv == 128) return __shfl_sync(kFull, u[3], 31);
  const int q = (nv - 1) & 3;
  const T sel = q == 0 ? u[0] : q == 1 ? u[1] : q == 2 ? u[2] : u[3];
  return __shfl_sync(kFull, sel, (nv - 1) >> 2);
}

template <typename T, int EXPL, bool VEC>
__global__ void __launch_bounds__(kLineThreads)
    line_sums_x(Lines L, LineCoef<T> k, const T* __restrict__ in,
                typename V2<T>::type* __restrict__ seg) {
  pdl_wait();
  pdl_launch_next();
  const XIdx id = x_index(L);
  if (!id.ok) return;
  T d[kXC][4];
  x_rhs<T, EXPL, VEC>(in, L, k, id, d);
  const int i0 = id.s * kXSegV;
  const T w4j = pow_bits<5>(k.rbit + 2, id.lane);  // r^(4 lane)
  T carry = 0, bu = 0, pwk = 1;
#pragma unroll
  for (int c = 0; c < kXC; ++c) {
    const int nv = min(128, L.n - (i0 + 128 * c));
    if (nv > 0) {
      T u[4];
      const T last = x_forward(d[c], carry, nv, w4j, k, id.lane, u);
      const int base = 4 * id.lane;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (base + q >= nv) u[q] = T(0);
      T h = fma(k.r, u[3], u[2]);
      h = fma(k.r, h, u[1]);
      h = fma(k.r, h, u[0]);
      bu = fma(pwk * w4j, h, bu);
      carry = last;
      pwk *= k.rbit[7];
    }
  }
#pragma unroll
  for (int sh = 16; sh > 0; sh >>= 1) bu += __shfl_xor_sync(kFull, bu, sh);
  if (id.lane == 0) seg[(int64_t)id.s * L.nlines + id.line] = {carry, bu};
}

template <typename T, int EXPL, bool VEC>
__global__ void __launch_bounds__(kLineThreads)
    line_solve_x(Lines L, LineCoef<T> k, const T* __restrict__ in,
                 const typename V2<T>::type* __restrict__ seg, T* __restrict__ out) {
  pdl_wait();
  pdl_launch_next();
  const XIdx id = x_index(L);
  if (!id.ok) return;
  T y[kXC][4];
  x_rhs<T, EXPL, VEC>(in, L, k, id, y);
  const typename V2<T>::type cr = seg[(int64_t)id.s * L.nlines + id.line];
  const int i0 = id.s * kXSegV;
  const int base = 4 * id.lane;
  const T w4j = pow_bits<5>(k.rbit + 2, id.lane);        // r^(4 lane)
  const T w4t = pow_bits<5>(k.rbit + 2, 31 - id.lane);   // r^(4 (31 - lane))
  T carry = cr.x;
#pragma unroll
  for (int c = 0; c < kXC; ++c) {
    const int nv = min(128, L.n - (i0 + 128 * c));
    if (nv > 0) {
      T u[4];
      carry = x_forward(y[c], carry, nv, w4j, k, id.lane, u);
#pragma unroll
      for (int q = 0; q < 4; ++q) y[c][q] = base + q < nv ? u[q] : T(0);
    }
  }
  T* row = out + id.row;
  carry = cr.y;  // x just after the segment
#pragma unroll
  for (int c = kXC - 1; c >= 0; --c) {
    const int nv = min(128, L.n - (i0 + 128 * c));
    if (nv > 0) {
      T v[4];
      v[3] = y[c][3];
      v[2] = fma(k.r, v[3], y[c][2]);
      v[1] = fma(k.r, v[2], y[c][1]);
      v[0] = fma(k.r, v[1], y[c][0]);
      const T W = scan4_down(v[0], k, id.lane);
      const T nxt = __shfl_down_sync(kFull, W, 1);
      T after = id.lane < 31 ? nxt : T(0);  // x after the lane's cells, carry excluded
      if (nv == 128) after = fma(w4t, carry, after);
      T x[4];
      T rp = k.r;
#pragma unroll
      for (int q = 3; q >= 0; --q, rp *= k.r) x[q] = fma(rp, after, v[q]);
      if (nv < 128) {  // the carry enters after the last valid cell
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (base + q < nv) x[q] = fma(pow_bits<8>(k.rbit, nv - (base + q)), carry, x[q]);
      }
      carry = __shfl_sync(kFull, x[0], 0);
      const int i = i0 + 128 * c + base;
      if (VEC && base + 3 < nv) {
        if constexpr (sizeof(T) == 4) {
          *reinterpret_cast<float4*>(row + i) =
              make_float4(k.kappa * x[0], k.kappa * x[1], k.kappa * x[2], k.kappa * x[3]);
        } else {
          *reinterpret_cast<double2*>(row + i) = make_double2(k.kappa * x[0], k.kappa * x[1]);
          *reinterpret_cast<double2*>(row + i + 2) = make_double2(k.kappa * x[2], k.kappa * x[3]);
        }
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (base + q < nv) row[i + q] = k.kappa * x[q];
      }
    }
  }
}

// ---------------------------------------------------------------- carries
// Pass 2, one warp per line: closes the two cyclic recurrences over the
// segments. In: (F_s, Bu_s). Out: (y just before segment s, x just after it).
// Over the segments the recurrences are Y_s = F_s + R Y_{s-1} and
// X_s = Bv_s + R X_{s+1} with Bv_s = Bu_s + G Y_{s-1} (the last segment has
// its own Rl, Gl); the warp runs them as weighted scans, 32 segments at a
// time, in the field's precision (both recurrences contract).
template <typename T>
__device__ __forceinline__ T wscan_up(T v, const T* Rp, int lane) {
#pragma unroll
  for (int b = 0; b < 5; ++b) {
    const T o = __shfl_up_sync(kFull, v, 1 << b);
    if (lane >= (1 << b)) v = fma(Rp[b], o, v);
  }
  return v;
}

template <typename T>
__device__ __forceinline__ T wscan_down(T v, const T* Rp, int lane) {
#pragma unroll
  for (int b = 0; b < 5; ++b) {
    const T o = __shfl_down_sync(kFull, v, 1 << b);
    if (lane + (1 << b) < 32) v = fma(Rp[b], o, v);
  }
  return v;
}

template <typename T>
__global__ void __launch_bounds__(128)
    line_carry(Lines L, CarryCoef<T> cc, typename V2<T>::type* __restrict__ seg) {
  pdl_wait();
  pdl_launch_next();
  const int lane = threadIdx.x & 31;
  const int line = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (line >= L.nlines) return;  // uniform across the warp
  const int m = L.nseg, mc = m - 1;  // segments 0 .. mc-1 share R and G
  auto at = [&](int s) -> typename V2<T>::type& { return seg[(int64_t)s * L.nlines + line]; };
  const T up_w = pow_bits<6>(cc.Rp, lane + 1);   // R^(lane+1)
  const T dn_w = pow_bits<6>(cc.Rp, 32 - lane);  // R^(32-lane)
  // forward chain from `start` (the y before segment 0); calls f(s, y_before)
  auto forward = [&](T start, auto&& f) -> T {
    T carry = start;
    for (int b0 = 0; b0 < mc; b0 += 32) {
      const int s = b0 + lane;
      const int nv = min(32, mc - b0);
      const T v = s < mc ? at(s).x : 0.0;
      const T y = fma(up_w, carry, wscan_up(v, cc.Rp, lane));
      const T prev = __shfl_up_sync(kFull, y, 1);  // every lane takes part
      const T before = lane == 0 ? carry : prev;
      if (s < mc) f(s, before);
      carry = __shfl_sync(kFull, y, nv - 1);
    }
    return carry;  // y before the last segment
  };
  // the y of the line's last cell with zero start, then the true start
  const T y_mc0 = forward(0.0, [](int, T) {});
  const T ystart = (at(mc).x + cc.Rl * y_mc0) * cc.inv_close;
  const T y_mc = forward(ystart, [&](int s, T before) {
    typename V2<T>::type& v = at(s);
    v.y = (v.y + before * cc.G);  // Bu -> Bv
    v.x = before;                          // F -> y before the segment
  });
  __syncwarp();
  {
    typename V2<T>::type& v = at(mc);
    if (lane == 0) {
      v.y = (v.y + y_mc * cc.Gl);
      v.x = y_mc;
    }
  }
  __syncwarp();
  // backward chain over segments mc-1 .. 0 from `start` (the x after
  // segment mc-1, i.e. the first x of the last segment); calls g(s, x_after)
  auto backward = [&](T start, auto&& g) -> T {
    T carry = start;
    for (int top = mc; top > 0; top -= 32) {
      const int s = top - 32 + lane;  // batches end at top; padding at the low end
      const int first = max(0, top - 32) - (top - 32);  // first valid lane
      const T v = s >= 0 ? at(s).y : 0.0;
      const T x = fma(dn_w, carry, wscan_down(v, cc.Rp, lane));
      const T next = __shfl_down_sync(kFull, x, 1);  // every lane takes part
      const T after = lane == 31 ? carry : next;
      if (s >= 0) g(s, after);
      carry = __shfl_sync(kFull, x, first);
    }
    return carry;  // x of the line's first cell
  };
  const T bv_last = at(mc).y;
  // zero start after the line's end: x_0 = (sum ...) / (1 - r^n)
  const T x_first0 = backward(bv_last, [](int, T) {});
  const T x0 = x_first0 * cc.inv_close;
  const T x_last = bv_last + cc.Rl * x0;  // first x of the last segment
  __syncwarp();
  backward(x_last, [&](int s, T after) { at(s).y = after; });
  if (lane == 0) at(mc).y = x0;
}

// The same pass with the line's (F, Bu) held in registers: B batches of 32
// segments per lane, one load and one store round (lines of up to 32 B + 1
// segments). Batches are aligned at segment 0; the top batch may be partial
// (nv valid lanes), so the backward chain enters it at lane nv - 1.
template <typename T, int B>
__global__ void __launch_bounds__(128)
    line_carry_reg(Lines L, CarryCoef<T> cc, typename V2<T>::type* __restrict__ seg) {
  pdl_wait();
  pdl_launch_next();
  const int lane = threadIdx.x & 31;
  const int line = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (line >= L.nlines) return;  // uniform across the warp
  const int mc = L.nseg - 1;     // segments 0 .. mc-1 share R and G
  const int nb = (mc + 31) / 32;
  typename V2<T>::type* col = seg + line;
  const int64_t st = L.nlines;
  T F[B], Bv[B], Yin[B], Xin[B];
#pragma unroll
  for (int b = 0; b < B; ++b) {
    const int s = 32 * b + lane;
    F[b] = Bv[b] = T(0);
    if (b < nb && s < mc) {
      const typename V2<T>::type v = col[s * st];
      F[b] = v.x;
      Bv[b] = v.y;
    }
  }
  const typename V2<T>::type last = col[(int64_t)mc * st];
  const T up_w = pow_bits<6>(cc.Rp, lane + 1);   // R^(lane+1)
  const T dn_w = pow_bits<6>(cc.Rp, 32 - lane);  // R^(32-lane)
  T carry = T(0);
#pragma unroll
  for (int b = 0; b < B; ++b) {
    if (b < nb) {
      const int nv = min(32, mc - 32 * b);
      const T y = fma(up_w, carry, wscan_up(F[b], cc.Rp, lane));
      carry = __shfl_sync(kFull, y, nv - 1);
    }
  }
  const T ystart = (last.x + cc.Rl * carry) * cc.inv_close;  // y of the line's last cell
  carry = ystart;
#pragma unroll
  for (int b = 0; b < B; ++b) {
    if (b < nb) {
      const int nv = min(32, mc - 32 * b);
      const T y = fma(up_w, carry, wscan_up(F[b], cc.Rp, lane));
      const T prev = __shfl_up_sync(kFull, y, 1);
      Yin[b] = lane == 0 ? carry : prev;
      if (32 * b + lane < mc) Bv[b] = fma(Yin[b], cc.G, Bv[b]);
      carry = __shfl_sync(kFull, y, nv - 1);
    }
  }
  const T y_mc = carry;                          // y before the last segment
  const T bv_last = last.y + y_mc * cc.Gl;
  auto backward = [&](T start, bool keep) -> T {
    T c = start;
#pragma unroll
    for (int b = B - 1; b >= 0; --b) {
      if (b < nb) {
        const int nv = min(32, mc - 32 * b);
        const T w = nv == 32 ? dn_w : (lane < nv ? pow_bits<6>(cc.Rp, nv - lane) : T(0));
        const T x = fma(w, c, wscan_down(Bv[b], cc.Rp, lane));
        const T nxt = __shfl_down_sync(kFull, x, 1);
        if (keep) Xin[b] = lane == nv - 1 ? c : nxt;
        c = __shfl_sync(kFull, x, 0);
      }
    }
    return c;
  };
  const T x0 = backward(bv_last, false) * cc.inv_close;  // x of the line's first cell
  backward(bv_last + cc.Rl * x0, true);
#pragma unroll
  for (int b = 0; b < B; ++b) {
    const int s = 32 * b + lane;
    if (b < nb && s < mc) col[s * st] = {Yin[b], Xin[b]};
  }
  if (lane == 0) col[(int64_t)mc * st] = {y_mc, x0};
}

// ---------------------------------------------------------------- whole lines
// Lines of up to kFusedSegs segments in one launch: a CTA holds whole lines in
// registers (a thread one segment of LS cells), so a cell is read once and
// written once, its right-hand side is formed once, and the segment carries
// close through shared memory.
//   pass 1  every thread: the segment's local sums F, Bu (as line_sums_yz)
//   pass 2  a warp per line: the cyclic carries, one weighted scan up and one
//           down over the segments, closed afterwards by what the closing
//           adds (R^(s+1) times the start value) instead of a second scan; lines
//           of few segments by a thread each (carry_serial)
//   pass 3  every thread: the segment from its true carries
// Lines along y / z: `nl` adjacent columns per CTA (at least one 32-byte sector
// wide), read and written directly. Lines along x: rows come through shared
// memory (cp.async, 16 bytes; segments padded to LS + V elements, so that
// both the 16-byte row accesses and the threads' 16-byte segment accesses are
// free of bank conflicts).
//
// Bound: in double the FP64 units (seven operations per cell with a divided
// explicit half step, five without), busy for half of a 1024 x 1400 solve's time,
// and the threads' chains at a quarter of the SMs' warps in one wave and a
// remainder; latency and L2 in float. us per solve with the
// explicit half step, three launches -> one: 256^2 float 11.2 -> 2.3 (along
// x 5.4 -> 2.5) and double 32.8 -> 5.0 (13.9 -> 6.4), 1024^2 float 11.9 ->
// 4.0 (8.3 -> 4.9) and double 44.5 -> 21.4 (58.8 -> 24.8), 256^3 float 82 ->
// 30 (90 -> 44) and double 588 -> 307 (953 -> 312).
constexpr int kFusedSegs = 128;
// The root's rounding to the field's type shifts alpha by sqrt(alpha) ulps, and
// line_fused takes every constant from the rounded root, where the three launches
// take the carries' from the root in double. Errors against extended precision on
// fields of zero mean, one launch / three: at most 1.6 (float) and 2.1 (double) up
// to alpha 175, 3.7 and 3.3 at 700, 15 and 7 at 1e5, 50 and 30 at 1e7; from 1e15 the
// rounded float root is 1. (On fields with a mean the one launch is the more
// accurate throughout.)
constexpr double kFusedMaxAlpha = 128.0;
constexpr int kCarryW = 36;  // 33 weights, a multiple of 16 bytes

// W[k] = R^k, k <= 32, in shared memory; B batches of 32 segments.
template <typename T, int B>
__device__ __forceinline__ void carry_scan(int mc, const CarryCoef<T>& cc, int lane,
                                           const T* __restrict__ W, T* F, T* Bu) {
  const int nb = (mc + 31) / 32;  // segments 0 .. mc - 1 share R and G; mc is the last
  const T up_w = W[lane + 1];
  T y[B], bv[B];
  T carry = T(0);
#pragma unroll
  for (int b = 0; b < B; ++b) {
    y[b] = bv[b] = T(0);
    if (b < nb) {
      const int q = 32 * b + lane;
      bv[b] = q < mc ? Bu[q] : T(0);
      y[b] = wscan_up(q < mc ? F[q] : T(0), cc.Rp, lane);
      if (b > 0) y[b] = fma(up_w, carry, y[b]);
      carry = __shfl_sync(kFull, y[b], min(32, mc - 32 * b) - 1);
    }
  }
  const T ystart = (F[mc] + cc.Rl * carry) * cc.inv_close;  // y of the line's last cell
  const T blast = Bu[mc];
  __syncwarp();
  T add = ystart, before = ystart;  // what closing adds to the y before the batch
#pragma unroll
  for (int b = 0; b < B; ++b) {
    if (b < nb) {
      const int q = 32 * b + lane;
      const T yt = fma(up_w, add, y[b]);
      const T prev = __shfl_up_sync(kFull, yt, 1);
      const T yin = lane == 0 ? before : prev;  // y just before the segment
      if (q < mc) {
        bv[b] = fma(yin, cc.G, bv[b]);
        F[q] = yin;
      }
      before = __shfl_sync(kFull, yt, min(32, mc - 32 * b) - 1);
      if (b + 1 < nb) add *= cc.Rp[5];
    }
  }
  if (lane == 0) F[mc] = before;
  // backward: x of segment s with zero x past the line's end
  const T bv_last = blast + before * cc.Gl;
  carry = bv_last;
#pragma unroll
  for (int b = B - 1; b >= 0; --b) {
    if (b < nb) {
      const int nv = min(32, mc - 32 * b);
      y[b] = wscan_down(bv[b], cc.Rp, lane);
      if (lane < nv) y[b] = fma(W[nv - lane], carry, y[b]);
      carry = __shfl_sync(kFull, y[b], 0);
    }
  }
  const T x0 = carry * cc.inv_close;  // x of the line's first cell
  add = cc.Rl * x0;
  T after = bv_last + add;
#pragma unroll
  for (int b = B - 1; b >= 0; --b) {
    if (b < nb) {
      const int nv = min(32, mc - 32 * b);
      const int q = 32 * b + lane;
      T xt = y[b];
      if (lane < nv) xt = fma(W[nv - lane], add, xt);
      const T nxt = __shfl_down_sync(kFull, xt, 1);
      if (q < mc) Bu[q] = lane == nv - 1 ? after : nxt;  // x just past the segment
      after = __shfl_sync(kFull, xt, 0);
      if (b > 0) add *= W[nv];
    }
  }
  if (lane == 0) Bu[mc] = x0;
}

// The same by one thread, for lines of few segments: a warp would scan 32 / nseg of
// them one after the other, most of its lanes idle. us per solve with the scan /
// with this (three launches): 30 x 16 double 20.4 / 4.4 (8.7), 1000 x 16 float 7.0 / 2.4
// (4.9), 20 x 100000 columns in double 153 / 33 (125).
constexpr int kSerialSegs = 8;
template <typename T>
__device__ __forceinline__ void carry_serial(int mc, const CarryCoef<T>& cc, T* F, T* Bu) {
  T y = T(0);
  for (int s = 0; s < mc; ++s) y = fma(cc.R, y, F[s]);
  y = (F[mc] + cc.Rl * y) * cc.inv_close;  // y of the line's last cell
  for (int s = 0; s < mc; ++s) {
    const T next = fma(cc.R, y, F[s]);
    Bu[s] = fma(y, cc.G, Bu[s]);
    F[s] = y;
    y = next;
  }
  F[mc] = y;
  const T last = Bu[mc] + y * cc.Gl;
  T x = last;  // with zero x past the line's end
  for (int s = mc - 1; s >= 0; --s) x = fma(cc.R, x, Bu[s]);
  x *= cc.inv_close;  // x of the line's first cell
  Bu[mc] = x;
  x = fma(cc.Rl, x, last);
  for (int s = mc - 1; s >= 0; --s) {
    const T next = fma(cc.R, x, Bu[s]);
    Bu[s] = x;
    x = next;
  }
}

// Right-hand side c + ea (ab - 2 c) from c and its neighbours' sum ab: a uniform
// field comes back unchanged whatever ea is. DIVIDED: by ea, one operation less
// (kappa scales the solution back). The weight 1/ea - 2 is rounded, an error of ea
// ulps in every mode but the uniform one, so that form is for small ea (kMaxDivided),
// and for double, where every operation counts: 1024 x 1400 Crank-Nicolson ADI, one
// call of 20 steps 1014 us against 1102.
template <bool DIVIDED, typename T>
__device__ __forceinline__ T half_step(const LineCoef<T>& k, T c, T ab) {
  return DIVIDED ? fma(k.w0, c, ab) : fma(k.w1, fma(T(-2), c, ab), c);
}
constexpr double kMaxDivided = 4.0;

// The half step along another axis than x for rows_in: a row's cells and those of the
// two rows beside it, as vectors (cell by cell 4096^2 in float took 66.7 us, the three
// launches 58.5; now 52.4).
template <bool DIVIDED, typename T>
struct HalfStep {
  const Lines& L;
  const LineCoef<T>& k;
  __device__ __forceinline__ void offsets(int line, int64_t& em, int64_t& ep) const {
    wrap_offsets(L.e_is_y ? line % L.ny : line / L.ny, L.ne, L.estride, em, ep);
  }
  __device__ __forceinline__ T at(const T* row, int line, int i) const {
    int64_t em, ep;
    offsets(line, em, ep);
    return half_step<DIVIDED>(k, __ldg(row + i), __ldg(row + em + i) + __ldg(row + ep + i));
  }
  __device__ __forceinline__ void vec(const T* row, int line, int i, T* v) const {
    using VT = typename LineVec<T>::type;
    int64_t em, ep;
    offsets(line, em, ep);
    const VT c = __ldg(reinterpret_cast<const VT*>(row + i));
    const VT a = __ldg(reinterpret_cast<const VT*>(row + em + i));
    const VT b = __ldg(reinterpret_cast<const VT*>(row + ep + i));
#pragma unroll
    for (int e = 0; e < 16 / (int)sizeof(T); ++e)
      v[e] = half_step<DIVIDED>(k, reinterpret_cast<const T*>(&c)[e],
                                reinterpret_cast<const T*>(&a)[e] +
                                    reinterpret_cast<const T*>(&b)[e]);
  }
};

// B: batches of 32 segments in pass 2's scan, 0: a thread per line.
// MODE: 0 no explicit part, 1 along the solved axis, 2 along another one; 3 and 4 as
// 1 and 2 with the divided half step.
template <typename T, int LS, int B, int MODE, bool X>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 1024 : 512)
    line_fused(const __grid_constant__ Lines L, const __grid_constant__ LineCoef<T> k,
               const __grid_constant__ CarryCoef<T> cc, const T* __restrict__ in,
               T* __restrict__ out, int nl, int vec_ok) {
  constexpr int V = 16 / (int)sizeof(T);
  constexpr int EXPL = MODE > 2 ? MODE - 2 : MODE;
  constexpr bool DIVIDED = MODE > 2;
  constexpr int PS = LS + V;  // a segment's elements in shared memory (x lines)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, nt = blockDim.x;
  const int ns = L.nseg;
  T* W = reinterpret_cast<T*>(smem_raw);  // R^0 .. R^32
  T* sF = W + kCarryW;
  T* sB = sF + nl * ns;
  T* tile = sF + (2 * nl * ns + V - 1) / V * V;
  if (B > 0 && tid < 33) W[tid] = pow_bits<6>(cc.Rp, tid);
  pdl_wait();
  pdl_launch_next();

  // this thread's line and segment
  int ln, sg;
  int64_t base = 0;  // strided: the line's first cell
  bool ok;
  int x = 0, o = 0, line0 = 0;
  if constexpr (X) {
    ln = tid / ns;
    sg = tid - ln * ns;
    line0 = blockIdx.x * nl;
    ok = ln < nl && line0 + ln < L.nlines;
  } else {
    const int cb = (L.nx + nl - 1) / nl;
    o = blockIdx.x / cb;
    ln = tid & (nl - 1);  // nl is a power of two
    sg = tid / nl;
    x = (blockIdx.x - o * cb) * nl + ln;
    ok = sg < ns && x < L.nx;
    base = x + (int64_t)o * L.ostride;
  }
  const int i0 = sg * LS;
  const int len = ok ? min(LS, L.n - i0) : 0;
  T d[LS];
  T cm = T(0), cp = T(0);  // the explicit part's cells beside the segment

  if constexpr (X) {
    rows_in<T, LS, EXPL != 2>(tile, in, line0, nl, L.nlines, L.n, ns, L.ny, L.pitch, L.plane,
                              vec_ok, HalfStep<DIVIDED, T>{L, k});
    if (ok) {
      segment_in<T, LS>(tile + (ln * ns + sg) * PS, len, d);
      if (EXPL == 1) {
        const T* l0 = tile + ln * ns * PS;
        const int im = i0 == 0 ? L.n - 1 : i0 - 1, ip = i0 + len == L.n ? 0 : i0 + len;
        cm = l0[im / LS * PS + im % LS];
        cp = l0[ip / LS * PS + ip % LS];
      }
    } else {
#pragma unroll
      for (int j = 0; j < LS; ++j) d[j] = T(0);
    }
  } else {
    const T* p = in + base + (int64_t)i0 * L.stride;
    if (len == LS) {
#pragma unroll
      for (int j = 0; j < LS; ++j) d[j] = __ldg(p + (int64_t)j * L.stride);
    } else {
#pragma unroll
      for (int j = 0; j < LS; ++j) d[j] = j < len ? __ldg(p + (int64_t)j * L.stride) : T(0);
    }
    if (EXPL == 1 && ok) {
      cm = __ldg(in + base + (int64_t)(i0 == 0 ? L.n - 1 : i0 - 1) * L.stride);
      cp = __ldg(in + base + (int64_t)(i0 + len == L.n ? 0 : i0 + len) * L.stride);
    }
    if (EXPL == 2 && ok) {
      int64_t em, ep;
      if (L.e_is_x)
        wrap_offsets(x, L.ne, 1, em, ep);
      else
        wrap_offsets(o, L.ne, L.estride, em, ep);
#pragma unroll
      for (int j = 0; j < LS; ++j)
        if (j < len)
          d[j] = half_step<DIVIDED>(k, d[j], __ldg(p + (int64_t)j * L.stride + em) +
                                                 __ldg(p + (int64_t)j * L.stride + ep));
    }
  }
  if (EXPL == 1) {
    T prev = cm;
#pragma unroll
    for (int j = 0; j < LS; ++j) {
      const T cur = d[j];
      const T nxt = j + 1 < LS ? d[j + 1 < LS ? j + 1 : j] : cp;
      if (j < len) d[j] = half_step<DIVIDED>(k, cur, prev + (j + 1 == len ? cp : nxt));
      prev = cur;
    }
  }

  // pass 1
  T u = T(0), bu = T(0);
#pragma unroll
  for (int j = 0; j < LS; ++j) {
    if (j < len) {
      u = fma(k.r, u, d[j]);
      bu = fma(k.rpow[j], u, bu);
    }
  }
  if (ok) {
    sF[ln * ns + sg] = u;
    sB[ln * ns + sg] = bu;
  }
  __syncthreads();
  // pass 2
  if constexpr (B == 0) {
    for (int q = tid; q < nl; q += nt) carry_serial(ns - 1, cc, sF + q * ns, sB + q * ns);
  } else {
    for (int q = tid >> 5; q < nl; q += nt >> 5)
      carry_scan<T, B>(ns - 1, cc, tid & 31, W, sF + q * ns, sB + q * ns);
  }
  __syncthreads();
  // pass 3
  T y = ok ? sF[ln * ns + sg] : T(0);
  T xv = ok ? sB[ln * ns + sg] : T(0);
#pragma unroll
  for (int j = 0; j < LS; ++j) {
    y = fma(k.r, y, d[j]);
    d[j] = y;
  }
  if constexpr (X) {
#pragma unroll
    for (int j = LS - 1; j >= 0; --j) {
      if (j < len) {
        xv = fma(k.r, xv, d[j]);
        d[j] = k.kappa * xv;
      }
    }
    if (ok) segment_out<T, LS>(tile + (ln * ns + sg) * PS, d);
    __syncthreads();
    rows_out<T, LS>(tile, out, line0, nl, L.nlines, L.n, ns, L.ny, L.pitch, L.plane, vec_ok);
  } else {
    T* p = out + base + (int64_t)i0 * L.stride;
#pragma unroll
    for (int j = LS - 1; j >= 0; --j) {
      if (j < len) {
        xv = fma(k.r, xv, d[j]);
        p[(int64_t)j * L.stride] = k.kappa * xv;
      }
    }
  }
}

// ---------------------------------------------------------------- Chebyshev
// One iteration: y_new = y_prev + omega (y + gamma (b - A y) - y_prev), or
// y + gamma (b - A y) for the first. A y = diag y - a sum(neighbours of y);
// b = c, or for Crank-Nicolson w0 c + w1 sum(neighbours of c). y_new may
// alias y_prev (each cell reads its own y_prev only).
template <typename T>
struct ChebStep {
  T diag, a, w0, w1, gamma, omega;
  int first;
};

template <typename T, int ND, bool CN>
__global__ void __launch_bounds__(256)
    chebyshev_kernel(Geo g, ChebStep<T> k, const T* __restrict__ c, const T* __restrict__ y,
                     const T* yprev, T* ynew) {
  pdl_wait();
  pdl_launch_next();
  const int nx = g.n[ND - 1], ny = g.n[ND - 2];
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= nx) return;
  const int z = ND == 3 ? blockIdx.z : 0;
  const int xm = x == 0 ? nx - 1 : x - 1, xp = x == nx - 1 ? 0 : x + 1;
  int64_t zm = 0, zp = 0;
  if (ND == 3) {
    const int nz = g.n[0];
    zm = (int64_t)(z == 0 ? nz - 1 : z - 1) * g.plane;
    zp = (int64_t)(z == nz - 1 ? 0 : z + 1) * g.plane;
  }
  const int64_t zb = (int64_t)z * g.plane;
  for (int yy = blockIdx.y; yy < ny; yy += gridDim.y) {
    const int64_t ym = (int64_t)(yy == 0 ? ny - 1 : yy - 1) * g.pitch;
    const int64_t yp = (int64_t)(yy == ny - 1 ? 0 : yy + 1) * g.pitch;
    const int64_t yb = (int64_t)yy * g.pitch;
    const int64_t i = zb + yb + x;
    T sy = __ldg(y + zb + yb + xm) + __ldg(y + zb + yb + xp) + __ldg(y + zb + ym + x) +
           __ldg(y + zb + yp + x);
    if (ND == 3) sy += __ldg(y + zm + yb + x) + __ldg(y + zp + yb + x);
    const T yc = __ldg(y + i);
    T b = __ldg(c + i);
    if (CN) {
      T sc = __ldg(c + zb + yb + xm) + __ldg(c + zb + yb + xp) + __ldg(c + zb + ym + x) +
             __ldg(c + zb + yp + x);
      if (ND == 3) sc += __ldg(c + zm + yb + x) + __ldg(c + zp + yb + x);
      b = k.w0 * b + k.w1 * sc;
    }
    const T rich = yc + k.gamma * (b - (k.diag * yc - k.a * sy));
    ynew[i] = k.first ? rich : yprev[i] + k.omega * (rich - yprev[i]);
  }
}

// ---------------------------------------------------------------- host side
int phys_axis(const Geo& g, int axis) { return axis + (3 - g.ndim); }  // 0 z, 1 y, 2 x

struct Extents {
  int n[3];        // z, y, x
  int64_t st[3];   // strides
};

Extents extents(const Geo& g) {
  Extents e;
  e.n[0] = g.ndim == 3 ? g.n[0] : 1;
  e.n[1] = g.n[g.ndim - 2];
  e.n[2] = g.n[g.ndim - 1];
  e.st[0] = g.ndim == 3 ? g.plane : (int64_t)g.pitch * e.n[1];
  e.st[1] = g.pitch;
  e.st[2] = 1;
  return e;
}

Lines make_lines(const Geo& g, int axis) {
  const Extents e = extents(g);
  const int p = phys_axis(g, axis);
  Lines L{};
  L.n = e.n[p];
  L.stride = e.st[p];
  L.pitch = g.pitch;
  L.plane = e.st[0];
  L.ny = e.n[1];
  L.nx = e.n[2];
  if (p == 2) {
    L.seglen = kXSegV;
    L.nlines = e.n[0] * e.n[1];
  } else {
    L.seglen = kSeg;
    const int o = p == 1 ? 0 : 1;  // the remaining axis
    L.no = e.n[o];
    L.ostride = e.st[o];
    L.nlines = e.n[2] * L.no;
  }
  L.nseg = (L.n + L.seglen - 1) / L.seglen;
  return L;
}

size_t line_scratch_bytes(const Geo& g, int axis, int elem_bytes) {
  const Lines L = make_lines(g, axis);
  return (size_t)L.nlines * L.nseg * 2 * elem_bytes;
}

double recurrence_root(double a) { return 2.0 * a / (1.0 + 2.0 * a + sqrt(1.0 + 4.0 * a)); }

template <typename T>
int32_t copy_field(const Geo& g, const T* in, T* out, cudaStream_t st) {
  const Extents e = extents(g);
  const size_t bytes = (size_t)e.st[0] * e.n[0] * sizeof(T);
  PPF_TRY_CUDA(cudaMemcpyAsync(out, in, bytes, cudaMemcpyDeviceToDevice, st));
  return PPF_OK;
}

template <typename T>
cudaError_t launch_carry(const Lines& L, const CarryCoef<T>& cc, typename V2<T>::type* seg,
                         cudaStream_t st) {
  const dim3 grid((L.nlines + 3) / 4), block(128);
  const int nb = (L.nseg - 1 + 31) / 32;
  if (nb <= 1) return launch(line_carry_reg<T, 1>, grid, block, 0, st, true, L, cc, seg);
  if (nb <= 2) return launch(line_carry_reg<T, 2>, grid, block, 0, st, true, L, cc, seg);
  if (nb <= 4) return launch(line_carry_reg<T, 4>, grid, block, 0, st, true, L, cc, seg);
  if (nb <= 8) return launch(line_carry_reg<T, 8>, grid, block, 0, st, true, L, cc, seg);
  if (nb <= 16) return launch(line_carry_reg<T, 16>, grid, block, 0, st, true, L, cc, seg);
  return launch(line_carry<T>, grid, block, 0, st, true, L, cc, seg);
}

template <typename T, int EXPL, bool VEC>
int32_t launch_line(const Lines& L, const LineCoef<T>& k, const CarryCoef<T>& cc, const T* in,
                    T* out, typename V2<T>::type* seg, cudaStream_t st) {
  if (L.seglen == kXSegV) {
    const int64_t warps = (int64_t)L.nlines * L.nseg;
    const dim3 grid((unsigned)((warps + kLineThreads / 32 - 1) / (kLineThreads / 32)));
    if (grid.x > 0x7fffffffu) return fail(PPF_ERR_INVALID, "grid too large");
    PPF_TRY_CUDA(
        launch(line_sums_x<T, EXPL, VEC>, grid, dim3(kLineThreads), 0, st, true, L, k, in, seg));
    PPF_TRY_CUDA(launch_carry<T>(L, cc, seg, st));
    PPF_TRY_CUDA(launch(line_solve_x<T, EXPL, VEC>, grid, dim3(kLineThreads), 0, st, true, L, k,
                        in, seg, out));
    return PPF_OK;
  }
  const int64_t so = (int64_t)L.nseg * L.no;
  const unsigned gy = (unsigned)(so < 65535 ? so : 65535);
  const unsigned gz = (unsigned)((so + gy - 1) / gy);
  if (gz > 65535) return fail(PPF_ERR_INVALID, "grid too large for the line solver");
  const int pairs = (L.nx + 1) / 2;
  const dim3 grid((pairs + kLineThreads - 1) / kLineThreads, gy, gz);
  PPF_TRY_CUDA(
      launch(line_sums_yz<T, EXPL, VEC>, grid, dim3(kLineThreads), 0, st, true, L, k, in, seg));
  PPF_TRY_CUDA(launch_carry<T>(L, cc, seg, st));
  PPF_TRY_CUDA(launch(line_solve_yz<T, EXPL, VEC>, grid, dim3(kLineThreads), 0, st, true, L, k, in,
                      seg, out));
  return PPF_OK;
}

// The same with vectors of two cells (columns) or four (x, as 16 bytes each) where the
// fields lie on their boundary, else cell by cell.
template <typename T, int EXPL>
int32_t launch_line_any(const Lines& L, const LineCoef<T>& k, const CarryCoef<T>& cc, const T* in,
                        T* out, typename V2<T>::type* seg, cudaStream_t st) {
  const uintptr_t need = L.seglen == kXSegV ? 16 : 2 * sizeof(T);
  const bool vec = (uintptr_t)in % need == 0 && (uintptr_t)out % need == 0;
  return vec ? launch_line<T, EXPL, true>(L, k, cc, in, out, seg, st)
             : launch_line<T, EXPL, false>(L, k, cc, in, out, seg, st);
}

template <typename T>
void carry_coef(double r, int n, int seglen, int nseg, CarryCoef<T>& cc) {
  const int Ll = n - (nseg - 1) * seglen;
  const double R = pow(r, seglen);
  cc.R = (T)R;
  cc.Rl = (T)pow(r, Ll);
  cc.G = (T)(r * (1.0 - pow(r, 2.0 * seglen)) / (1.0 - r * r));
  cc.Gl = (T)(r * (1.0 - pow(r, 2.0 * Ll)) / (1.0 - r * r));
  cc.inv_close = (T)(1.0 / (1.0 - pow(r, n)));
  for (int b = 0; b < 6; ++b) cc.Rp[b] = (T)pow(R, (double)(1 << b));
}

template <typename T, int LS, int MAXB, int MODE, bool X>
int32_t launch_fused(Lines L, const LineCoef<T>& k, double r, const T* in, T* out,
                     cudaStream_t st) {
  constexpr int V = 16 / (int)sizeof(T);
  L.seglen = LS;
  L.nseg = (L.n + LS - 1) / LS;
  CarryCoef<T> cc{};
  carry_coef(r, L.n, LS, L.nseg, cc);
  // lines per CTA: a sector of columns or a row, more where lines are short
  int nl = X ? 1 : 32 / (int)sizeof(T);
  while (nl * L.nseg < 128 && nl < 128) nl *= 2;
  const int threads = (nl * L.nseg + 31) / 32 * 32;
  size_t smem = (size_t)(kCarryW + 2 * nl * L.nseg + V) * sizeof(T);
  if (X) smem += (size_t)nl * L.nseg * (LS + V) * sizeof(T);
  const int64_t ctas = X ? ((int64_t)L.nlines + nl - 1) / nl
                         : (int64_t)((L.nx + nl - 1) / nl) * L.no;
  if (ctas > 0x7fffffff) return fail(PPF_ERR_INVALID, "grid too large for the line solver");
  const int vec_ok = ((uintptr_t)in) % 16 == 0 && ((uintptr_t)out) % 16 == 0;
  auto kern = L.nseg <= 33 ? line_fused<T, LS, 1, MODE, X> : line_fused<T, LS, 2, MODE, X>;
  if constexpr (MAXB == 4)
    if (L.nseg > 65) kern = line_fused<T, LS, 4, MODE, X>;
  if constexpr (LS < 32)
    if (L.nseg <= kSerialSegs) kern = line_fused<T, LS, 0, MODE, X>;
  PPF_TRY_CUDA(allow_smem(kern, smem));
  PPF_TRY_CUDA(launch(kern, dim3((unsigned)ctas), dim3(threads), smem, st, true, L, k, cc, in, out,
                      nl, vec_ok));
  return PPF_OK;
}

// Cells per thread. Short segments give small grids more threads and a shorter
// chain per thread (and code: a kernel that runs once per warp waits for its
// instructions), long ones fewer carries per line; above 96 segments the scan
// and the CTA's size cost more than they give. us per solve with 8 / 16 / 32:
// 256^2 float 2.2 / 2.7 / 4.1 and double 4.4 / 7.3 / 13.1, 1024^2 float 4.7 /
// 3.7 / 3.6 and double 19.6 / 16.4 / 15.6 (along x 5.2 / 4.6 / 5.4 and 20.8 /
// 20.1 / 21.1), 256^3 float 42 / 31 / 28, double 249 / 244 / 257.
template <typename T>
int fused_segment(const Lines& L, bool x) {
  const int64_t cells = (int64_t)L.nlines * L.n;
  if (L.n <= 512 && cells < (1 << 20)) return 8;
  if (L.n > (x && L.nlines < 300 ? 2048 : 1536)) return 32;
  if (sizeof(T) == 4 && (cells >= (1 << 22) || (!x && L.n > 1024))) return 32;
  return 16;
}

// Where the three launches are the faster ones: long lines of which a CTA holds one
// (x) or a sector of columns, with too few of them to hide a thread's chain of 32
// cells, or so many cells that loads bind. us per solve, one launch / three:
//   x, beyond 2048 cells: double 30 x 3000 18.6 / 17.3, 30 x 4000 23.5 / 18.2,
//     60 x 4000 20.5 / 18.1 but 100 x 4000 23.5 / 24.6, 500 x 3000 9 / 24; float
//     without an explicit part 30 x 4000 6.7 / 6.2, 1000 x 2500 12.7 / 10.9 but
//     300 x 4000 6.9 / 7.3. (A line alone takes one launch: 1 x 3000 1.2 times faster.)
//   columns without an explicit part: float 3000^2 21.4 / 18.9, 2048^2 8.0 / 14.0,
//     1500 x 8000 1.3 times slower than three; double 4000 x 30 31.2 / 22.6, 3000 x
//     100 23.6 / 21.7, 2300 x 100 faster, 3000 x 8000 331 / 299, 1300 x 16000 1.23
//     times slower, 700 x 16000 faster. With one: double 4000 x 30 40.9 / 36.4.
template <typename T>
bool three_launches(const Lines& L, int mode) {
  const int64_t cells = (int64_t)L.nlines * L.n;
  if (L.seglen == kXSegV) {
    if (L.n <= 2048 || L.nlines == 1) return false;
    return sizeof(T) == 8 ? L.nlines < 64 : mode == 0 && (L.nlines < 100 || L.nlines > 600);
  }
  if (mode == 2) return false;
  if (sizeof(T) == 4) return mode == 0 && L.n > (cells > (1 << 23) ? 1200 : 2048);
  if (mode == 1) return L.n > 3500 && L.nlines < 128;
  return (L.n > 2560 && L.nlines < 256) || (L.n > 800 && cells > (1 << 23));
}

template <typename T, int MODE>
int32_t launch_fused_axis(const Lines& L, const LineCoef<T>& k, double r, const T* in, T* out,
                          cudaStream_t st) {
  const bool x = L.seglen == kXSegV;
  switch (fused_segment<T>(L, x)) {
    case 8:
      return x ? launch_fused<T, 8, 2, MODE, true>(L, k, r, in, out, st)
               : launch_fused<T, 8, 2, MODE, false>(L, k, r, in, out, st);
    case 16:
      return x ? launch_fused<T, 16, 4, MODE, true>(L, k, r, in, out, st)
               : launch_fused<T, 16, 4, MODE, false>(L, k, r, in, out, st);
    default:
      return x ? launch_fused<T, 32, 4, MODE, true>(L, k, r, in, out, st)
               : launch_fused<T, 32, 4, MODE, false>(L, k, r, in, out, st);
  }
}

// One periodic line solve along `axis` (C order) with an optional explicit
// half step along `eaxis` (-1: none) folded into the right-hand side.
template <typename T>
int32_t line_sweep(const Geo& g, int axis, double a, int eaxis, double ea, const T* in, T* out,
                   void* scratch, size_t scratch_bytes, cudaStream_t st) {
  if (axis < 0 || axis >= g.ndim) return fail(PPF_ERR_INVALID, "axis %d out of range", axis);
  if (eaxis >= g.ndim) return fail(PPF_ERR_INVALID, "explicit axis %d out of range", eaxis);
  if (!(a >= 0) || !isfinite(a) || !(ea >= 0) || !isfinite(ea))
    return fail(PPF_ERR_INVALID, "alpha must be finite and >= 0");
  Lines L = make_lines(g, axis);
  if (L.n < 3)
    return fail(PPF_ERR_INVALID,
                "periodic line solves need >= 3 cells along the solved axis (got %d)", L.n);
  if (eaxis >= 0 && in == out)
    return fail(PPF_ERR_INVALID, "in and out must differ when an explicit part is folded in");
  const size_t need = line_scratch_bytes(g, axis, sizeof(T));
  if (!scratch || scratch_bytes < need)
    return fail(PPF_ERR_INVALID, "scratch of %zu bytes needed (got %zu)", need, scratch_bytes);
  const Extents e = extents(g);
  LineCoef<T> k{};
  int mode = 0;
  k.w0 = T(1);
  k.w1 = T(0);
  if (eaxis >= 0) {
    const int pe = phys_axis(g, eaxis), pa = phys_axis(g, axis);
    if (e.n[pe] < 3 && pe != pa)
      return fail(PPF_ERR_INVALID, "the explicit axis needs >= 3 cells (got %d)", e.n[pe]);
    k.w0 = (T)(1.0 - 2.0 * ea);
    k.w1 = (T)ea;
    mode = pe == pa ? 1 : 2;
    L.ne = e.n[pe];
    L.estride = e.st[pe];
    L.e_is_x = pe == 2;
    L.e_is_y = pe == 1;
  }
  L.expl = mode;
  if (a == 0.0) {
    if (mode == 0) return in == out ? PPF_OK : copy_field(g, in, out, st);
    // the explicit half step alone: a line solve with a vanishing implicit part
  }
  const double r = a > 0 ? recurrence_root(a) : 0.0;
  k.r = (T)r;
  k.kappa = (T)(a > 0 ? r / a : 1.0);
  double pw = 1.0;
  for (int i = 0; i <= 32; ++i, pw *= r) k.rpow[i] = (T)pw;
  CarryCoef<T> cc{};
  carry_coef(r, L.n, L.seglen, L.nseg, cc);
  for (int b = 0; b < 8; ++b) k.rbit[b] = (T)pow(r, (double)(1 << b));
  // whole lines in one launch while a line's segments fit a CTA, the root is not close
  // to 1 and the three launches are not the faster ones (they need the scratch aligned)
  const bool seg_ok = (uintptr_t)scratch % (2 * sizeof(T)) == 0;
  if (L.n <= 32 * kFusedSegs && a <= kFusedMaxAlpha &&
      !(seg_ok && three_launches<T>(L, mode))) {
    // every constant from the root as rounded to T, and kappa from the gain the
    // constants give a uniform field, so that it comes back unscaled: a
    // rounding of kappa itself would add up over the steps
    LineCoef<T> kf = k;
    const double rt = (double)(T)r;
    const bool divided = sizeof(T) == 8 && mode != 0 && ea >= 1e-3 && ea <= kMaxDivided;
    if (divided) kf.w0 = (T)((1.0 - 2.0 * ea) / ea);
    const double gain = divided ? (double)kf.w0 + 2.0 : 1.0;
    kf.kappa = (T)((1.0 - rt) * (1.0 - rt) / gain);
    pw = 1.0;
    for (int i = 0; i <= 32; ++i, pw *= rt) kf.rpow[i] = (T)pw;
    if constexpr (sizeof(T) == 8) {
      if (divided)
        return mode == 1 ? launch_fused_axis<T, 3>(L, kf, rt, in, out, st)
                         : launch_fused_axis<T, 4>(L, kf, rt, in, out, st);
    }
    switch (mode) {
      case 0: return launch_fused_axis<T, 0>(L, kf, rt, in, out, st);
      case 1: return launch_fused_axis<T, 1>(L, kf, rt, in, out, st);
      default: return launch_fused_axis<T, 2>(L, kf, rt, in, out, st);
    }
  }
  if (!seg_ok)
    return fail(PPF_ERR_INVALID, "scratch must be %zu-byte aligned", 2 * sizeof(T));
  auto* seg = static_cast<typename V2<T>::type*>(scratch);
  switch (mode) {
    case 0: return launch_line_any<T, 0>(L, k, cc, in, out, seg, st);
    case 1: return launch_line_any<T, 1>(L, k, cc, in, out, seg, st);
    default: return launch_line_any<T, 2>(L, k, cc, in, out, seg, st);
  }
}

struct ChebPlan {
  int iters;
  double gamma, rho;
};

ChebPlan chebyshev_plan(double a, int ndim, double tol) {
  ChebPlan p{};
  const double lmax = 1.0 + 4.0 * ndim * a;
  p.gamma = 2.0 / (lmax + 1.0);
  p.rho = (lmax - 1.0) / (lmax + 1.0);
  if (p.rho <= 0) return p;
  const double need = 2.0 * fmax(1.0, 8.0 * ndim * a) / tol;
  p.iters = (int)ceil(acosh(need) / acosh(1.0 / p.rho));
  if (p.iters < 1) p.iters = 1;
  return p;
}

// Solve (1 + 2 d a) x - a sum(neighbours of x) = b on the periodic grid,
// b = in (rhs_a = 0) or (1 - 2 d rhs_a) in + rhs_a sum(neighbours of in).
template <typename T>
int32_t periodic_solve(const Geo& g, double a, double rhs_a, double tol, const T* in, T* out,
                       T* tmp, int32_t* iterations, cudaStream_t st) {
  if (!(a >= 0) || !isfinite(a) || !(rhs_a >= 0) || !isfinite(rhs_a))
    return fail(PPF_ERR_INVALID, "alpha must be finite and >= 0");
  if (!(tol > 0) || !(tol < 1)) return fail(PPF_ERR_INVALID, "tol must be in (0, 1)");
  for (int ax = 0; ax < g.ndim; ++ax)
    if (g.n[ax] < 3)
      return fail(PPF_ERR_INVALID, "periodic solves need >= 3 cells per axis (axis %d has %d)",
                  ax, g.n[ax]);
  if (!tmp || tmp == in || tmp == out || in == out)
    return fail(PPF_ERR_INVALID, "in, out and tmp must be three distinct buffers");
  const ChebPlan plan = chebyshev_plan(a, g.ndim, tol);
  const int d = g.ndim;
  ChebStep<T> k{};
  k.diag = (T)(1.0 + 2.0 * d * a);
  k.a = (T)a;
  k.w0 = (T)(1.0 - 2.0 * d * rhs_a);
  k.w1 = (T)rhs_a;
  k.gamma = (T)plan.gamma;
  const bool cn = rhs_a != 0.0;
  const Extents e = extents(g);
  const dim3 grid((e.n[2] + 255) / 256, (unsigned)(e.n[1] < 65535 ? e.n[1] : 65535),
                  (unsigned)e.n[0]);
  if (e.n[0] > 65535) return fail(PPF_ERR_INVALID, "too many planes");
  if (iterations) *iterations = plan.iters;
  auto run = [&](const ChebStep<T>& kk, const T* y, const T* yp, T* yn) -> int32_t {
    cudaError_t err;
    if (d == 2)
      err = cn ? launch(chebyshev_kernel<T, 2, true>, grid, dim3(256), 0, st, true, g, kk, in, y,
                        yp, yn)
               : launch(chebyshev_kernel<T, 2, false>, grid, dim3(256), 0, st, true, g, kk, in,
                        y, yp, yn);
    else
      err = cn ? launch(chebyshev_kernel<T, 3, true>, grid, dim3(256), 0, st, true, g, kk, in, y,
                        yp, yn)
               : launch(chebyshev_kernel<T, 3, false>, grid, dim3(256), 0, st, true, g, kk, in,
                        y, yp, yn);
    PPF_TRY_CUDA(err);
    return PPF_OK;
  };
  if (plan.iters == 0) {  // a = 0: x = b, as one step y + (b - y) from y = in
    ChebStep<T> k0 = k;
    k0.diag = T(1);
    k0.a = T(0);
    k0.gamma = T(1);
    k0.first = 1;
    return run(k0, in, nullptr, out);
  }
  // iterations j = 1..K; y_j lands in out when K - j is even, else in tmp
  const T* prev = nullptr;
  const T* cur = in;
  double om = 1.0;
  const double rho2 = plan.rho * plan.rho;
  for (int j = 1; j <= plan.iters; ++j) {
    if (j == 2)
      om = 2.0 / (2.0 - rho2);
    else if (j > 2)
      om = 1.0 / (1.0 - rho2 * om / 4.0);
    T* dst = ((plan.iters - j) % 2 == 0) ? out : tmp;
    ChebStep<T> kj = k;
    kj.first = j == 1;
    kj.omega = (T)om;
    const int32_t rc = run(kj, cur, prev, dst);
    if (rc) return rc;
    prev = cur;
    cur = dst;
  }
  return PPF_OK;
}

template <typename T>
int32_t implicit_step(const PpfImplicitDiffusionParams* p, const PpfGrid* grid, const T* in,
                      T* out, T* tmp, void* scratch, size_t scratch_bytes, int32_t* iterations,
                      void* stream) {
  clear_error();
  if (!p) return fail(PPF_ERR_INVALID, "params is NULL");
  Geo g;
  int32_t rc = make_geo(grid, 2, 3, &g);
  if (rc) return rc;
  if (!in || !out) return fail(PPF_ERR_INVALID, "NULL field pointer");
  if (in == out) return fail(PPF_ERR_INVALID, "in and out must differ");
  if (!(p->dx > 0) || !(p->dt >= 0) || !(p->D >= 0) || !isfinite(p->dx) || !isfinite(p->dt) ||
      !isfinite(p->D))
    return fail(PPF_ERR_INVALID, "dx > 0, dt >= 0 and D >= 0 are required");
  const bool cn = p->solver == PPF_SOLVER_CRANK_NICOLSON;
  if (!cn && p->solver != PPF_SOLVER_IMPLICIT)
    return fail(PPF_ERR_INVALID, "solver must be PPF_SOLVER_IMPLICIT or PPF_SOLVER_CRANK_NICOLSON");
  const double a = (cn ? 0.5 : 1.0) * p->D * p->dt / (p->dx * p->dx);
  cudaStream_t st = (cudaStream_t)stream;
  if (iterations) *iterations = 0;
  const bool oned = g.ndim == 2 && g.n[0] == 1;
  if (oned) {  // engine_*Diffusion1D: one line along x
    return line_sweep<T>(g, 1, a, cn ? 1 : -1, a, in, out, scratch, scratch_bytes, st);
  }
  if (!p->adi) {
    const double tol = p->tol > 0 ? p->tol : (sizeof(T) == 4 ? 1e-7 : 1e-14);
    return periodic_solve<T>(g, a, cn ? a : 0.0, tol, in, out, tmp, iterations, st);
  }
  // ADI: the reference's axis order (Diffusion.py:428-431, 474-482, 527-533, 580-591)
  int sweeps[3][2];
  int ns = 0;
  if (!cn) {
    for (int ax = g.ndim - 1; ax >= 0; --ax) sweeps[ns][0] = ax, sweeps[ns][1] = -1, ++ns;
  } else if (g.ndim == 2) {
    sweeps[0][0] = 0, sweeps[0][1] = 0;
    sweeps[1][0] = 1, sweeps[1][1] = 1;
    ns = 2;
  } else {
    sweeps[0][0] = 1, sweeps[0][1] = 0;
    sweeps[1][0] = 0, sweeps[1][1] = 1;
    sweeps[2][0] = 2, sweeps[2][1] = 2;
    ns = 3;
  }
  if (cn && (!tmp || tmp == in || tmp == out))
    return fail(PPF_ERR_INVALID, "Crank-Nicolson ADI needs a tmp field distinct from in and out");
  const T* src = in;
  for (int i = 0; i < ns; ++i) {
    // without an explicit part a sweep may run in place: every thread reads
    // only the cells it writes after pass 1 has read them all
    T* dst = cn ? (((ns - 1 - i) % 2 == 0) ? out : tmp) : out;
    rc = line_sweep<T>(g, sweeps[i][0], a, sweeps[i][1], a, src, dst, scratch, scratch_bytes, st);
    if (rc) return rc;
    src = dst;
  }
  return PPF_OK;
}

}  // namespace
}  // namespace ppf

using namespace ppf;

extern "C" {

int32_t ppf_implicit_scratch_bytes(const PpfGrid* grid, int32_t elem_bytes, size_t* bytes) {
  clear_error();
  Geo g;
  int32_t rc = make_geo(grid, 2, 3, &g);
  if (rc) return rc;
  if (!bytes) return fail(PPF_ERR_INVALID, "bytes is NULL");
  if (elem_bytes != 4 && elem_bytes != 8) return fail(PPF_ERR_INVALID, "elem_bytes must be 4 or 8");
  size_t m = 0;
  for (int ax = 0; ax < g.ndim; ++ax) {
    const size_t b = line_scratch_bytes(g, ax, elem_bytes);
    m = b > m ? b : m;
  }
  *bytes = m;
  return PPF_OK;
}

int32_t ppf_line_solve_f32(const PpfGrid* grid, int32_t axis, double alpha, int32_t expl_axis,
                           double expl_alpha, const float* in, float* out, void* scratch,
                           size_t scratch_bytes, void* stream) {
  clear_error();
  Geo g;
  int32_t rc = make_geo(grid, 2, 3, &g);
  if (rc) return rc;
  if (!in || !out) return fail(PPF_ERR_INVALID, "NULL field pointer");
  return line_sweep<float>(g, axis, alpha, expl_axis, expl_alpha, in, out, scratch, scratch_bytes,
                           (cudaStream_t)stream);
}

int32_t ppf_line_solve_f64(const PpfGrid* grid, int32_t axis, double alpha, int32_t expl_axis,
                           double expl_alpha, const double* in, double* out, void* scratch,
                           size_t scratch_bytes, void* stream) {
  clear_error();
  Geo g;
  int32_t rc = make_geo(grid, 2, 3, &g);
  if (rc) return rc;
  if (!in || !out) return fail(PPF_ERR_INVALID, "NULL field pointer");
  return line_sweep<double>(g, axis, alpha, expl_axis, expl_alpha, in, out, scratch,
                            scratch_bytes, (cudaStream_t)stream);
}

int32_t ppf_periodic_solve_f32(const PpfGrid* grid, double alpha, double rhs_alpha, double tol,
                               const float* in, float* out, float* tmp, int32_t* iterations,
                               void* stream) {
  clear_error();
  Geo g;
  int32_t rc = make_geo(grid, 2, 3, &g);
  if (rc) return rc;
  if (!in || !out) return fail(PPF_ERR_INVALID, "NULL field pointer");
  return periodic_solve<float>(g, alpha, rhs_alpha, tol, in, out, tmp, iterations,
                               (cudaStream_t)stream);
}

int32_t ppf_periodic_solve_f64(const PpfGrid* grid, double alpha, double rhs_alpha, double tol,
                               const double* in, double* out, double* tmp, int32_t* iterations,
                               void* stream) {
  clear_error();
  Geo g;
  int32_t rc = make_geo(grid, 2, 3, &g);
  if (rc) return rc;
  if (!in || !out) return fail(PPF_ERR_INVALID, "NULL field pointer");
  return periodic_solve<double>(g, alpha, rhs_alpha, tol, in, out, tmp, iterations,
                                (cudaStream_t)stream);
}

int32_t ppf_diffusion_implicit_step_f32(const PpfImplicitDiffusionParams* p, const PpfGrid* g,
                                        const float* in, float* out, float* tmp, void* scratch,
                                        size_t scratch_bytes, int32_t* iterations, void* stream) {
  return implicit_step<float>(p, g, in, out, tmp, scratch, scratch_bytes, iterations, stream);
}

int32_t ppf_diffusion_implicit_step_f64(const PpfImplicitDiffusionParams* p, const PpfGrid* g,
                                        const double* in, double* out, double* tmp, void* scratch,
                                        size_t scratch_bytes, int32_t* iterations, void* stream) {
  return implicit_step<double>(p, g, in, out, tmp, scratch, scratch_bytes, iterations, stream);
}

}  // extern "C"
