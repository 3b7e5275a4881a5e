// Warp-wide rows of a field: 16-byte vectors of cells, their loads and stores
// at the ends of a row, and the boundary rule of a whole row or plane.
#pragma once

#include "ppf_common.cuh"

namespace ppf {

template <typename T>
struct Vec16;
template <>
struct Vec16<float> {
  using type = float4;
  static constexpr int n = 4;
};
template <>
struct Vec16<double> {
  using type = double2;
  static constexpr int n = 2;
};

// fetch's rule for a whole row or plane at coordinate i of one axis (field 0):
// the row it is read from, and what becomes of the cells after the load.
template <typename T>
struct AxisRule {
  int src;
  bool ghost, fixed;
  T add;  // Dirichlet value, or the shift added to the loaded value
  __device__ __forceinline__ AxisRule(const Geo& g, const Bc<T>& bc, int axis, int i) {
    const int n = g.n[axis];
    src = i;
    ghost = (unsigned)i >= (unsigned)n;
    fixed = false;
    add = T(0);
    if (!ghost) return;
    const int side = i < 0 ? 0 : 1;
    if (bc.type[axis] == PPF_BC_PERIODIC) {
      src = wrap_index(i, n);
    } else if (bc.type[axis] == PPF_BC_NEUMANN) {
      src = mirror_index(i, n);
      add = bc.shift[0][axis][side];
    } else {
      src = i < 0 ? 0 : n - 1;
      fixed = true;
      add = bc.shift[0][axis][side];
    }
  }
  __device__ __forceinline__ T value(T loaded) const { return fixed ? add : loaded + add; }
};

// A lane's V cells x .. x + V - 1 of one row: a vector where it lies inside
// the row and the rows are 16-byte aligned, else the cells below nx one by
// one (zeros past them).
template <typename T, int V>
__device__ __forceinline__ void load_cells(const T* __restrict__ row, int x, int nx, bool vec,
                                           T (&v)[V]) {
  using VT = typename Vec16<T>::type;
  if (vec) {
    const VT q = __ldg(reinterpret_cast<const VT*>(row + x));
    const T* pq = reinterpret_cast<const T*>(&q);
#pragma unroll
    for (int e = 0; e < V; ++e) v[e] = pq[e];
  } else {
#pragma unroll
    for (int e = 0; e < V; ++e) v[e] = x + e < nx ? __ldg(row + x + e) : T(0);
  }
}

template <typename T, int V>
__device__ __forceinline__ void store_cells(T* row, int x, int nx, bool vec, const T (&v)[V]) {
  using VT = typename Vec16<T>::type;
  if (vec) {
    VT q;
    T* pq = reinterpret_cast<T*>(&q);
#pragma unroll
    for (int e = 0; e < V; ++e) pq[e] = v[e];
    *reinterpret_cast<VT*>(row + x) = q;
  } else {
#pragma unroll
    for (int e = 0; e < V; ++e)
      if (x + e < nx) row[x + e] = v[e];
  }
}

}  // namespace ppf
