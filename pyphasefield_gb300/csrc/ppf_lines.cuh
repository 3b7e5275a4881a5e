// Rows of a field in shared memory for the line solvers that hold whole lines
// in a CTA: a thread owns one segment of LS consecutive cells, segments
// padded to LS + V elements (V elements are 16 bytes), so that the 16-byte
// accesses along a row and the threads' 16-byte accesses to their segments
// are both free of bank conflicts.
#pragma once

#include "ppf_common.cuh"

namespace ppf {

template <typename T>
struct LineVec;  // 16 bytes
template <>
struct LineVec<float> {
  using type = float4;
};
template <>
struct LineVec<double> {
  using type = double2;
};

template <typename T>
__device__ __forceinline__ void copy16_async(T* dst, const T* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

// Rows line0 .. line0 + nl - 1 (those below nlines; row = z * ny + y) of n cells
// to the tile, `ns` segments per row. vec_ok: 16-byte aligned rows (a vector
// that starts below n lies inside the row's pitch, a multiple of 4).
// COPY: the cells themselves; else cell.at(row, line, i), or cell.vec(row, line, i, v)
// for a whole vector.
template <typename T, int LS, bool COPY, typename Cell>
__device__ __forceinline__ void rows_in(T* tile, const T* __restrict__ in, int line0, int nl,
                                        int nlines, int n, int ns, int ny, int64_t pitch,
                                        int64_t plane, int vec_ok, Cell cell) {
  constexpr int V = 16 / (int)sizeof(T), PS = LS + V;
  const int nv = (n + V - 1) / V;
  for (int i = threadIdx.x; i < nl * nv; i += blockDim.x) {
    const int r = i / nv, c0 = (i - r * nv) * V;
    const int line = line0 + r;
    if (line >= nlines) break;
    const T* row = in + (int64_t)(line / ny) * plane + (int64_t)(line % ny) * pitch;
    T* dst = tile + (r * ns + c0 / LS) * PS + c0 % LS;
    if (COPY && vec_ok) {
      copy16_async(dst, row + c0);
    } else if (!COPY && vec_ok && c0 + V <= n) {
      typename LineVec<T>::type v;
      cell.vec(row, line, c0, reinterpret_cast<T*>(&v));
      *reinterpret_cast<typename LineVec<T>::type*>(dst) = v;
    } else {
#pragma unroll
      for (int e = 0; e < V; ++e)
        if (c0 + e < n) dst[e] = COPY ? __ldg(row + c0 + e) : cell.at(row, line, c0 + e);
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
}

// The tile back to the rows (after a barrier that orders its writers).
template <typename T, int LS>
__device__ __forceinline__ void rows_out(const T* tile, T* __restrict__ out, int line0, int nl,
                                         int nlines, int n, int ns, int ny, int64_t pitch,
                                         int64_t plane, int vec_ok) {
  constexpr int V = 16 / (int)sizeof(T), PS = LS + V;
  using VT = typename LineVec<T>::type;
  const int nv = (n + V - 1) / V;
  for (int i = threadIdx.x; i < nl * nv; i += blockDim.x) {
    const int r = i / nv, c0 = (i - r * nv) * V;
    const int line = line0 + r;
    if (line >= nlines) break;
    T* row = out + (int64_t)(line / ny) * plane + (int64_t)(line % ny) * pitch;
    const T* src = tile + (r * ns + c0 / LS) * PS + c0 % LS;
    if (vec_ok && c0 + V <= n) {
      *reinterpret_cast<VT*>(row + c0) = *reinterpret_cast<const VT*>(src);
    } else {
#pragma unroll
      for (int e = 0; e < V; ++e)
        if (c0 + e < n) row[c0 + e] = src[e];
    }
  }
}

// A thread's segment between the tile and its registers (cells at or past
// `len` read 0).
template <typename T, int LS>
__device__ __forceinline__ void segment_in(const T* s, int len, T (&d)[LS]) {
  constexpr int V = 16 / (int)sizeof(T);
  using VT = typename LineVec<T>::type;
#pragma unroll
  for (int q = 0; q < LS / V; ++q) {
    const VT v = *reinterpret_cast<const VT*>(s + q * V);
    const T* pv = reinterpret_cast<const T*>(&v);
#pragma unroll
    for (int e = 0; e < V; ++e) d[q * V + e] = q * V + e < len ? pv[e] : T(0);
  }
}

template <typename T, int LS>
__device__ __forceinline__ void segment_out(T* s, const T (&d)[LS]) {
  constexpr int V = 16 / (int)sizeof(T);
  using VT = typename LineVec<T>::type;
#pragma unroll
  for (int q = 0; q < LS / V; ++q) {
    VT v;
    T* pv = reinterpret_cast<T*>(&v);
#pragma unroll
    for (int e = 0; e < V; ++e) pv[e] = d[q * V + e];
    *reinterpret_cast<VT*>(s + q * V) = v;
  }
}

}  // namespace ppf
