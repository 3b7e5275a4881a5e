// Kernels of the learned surrogate (a convolutional encoder-decoder that
// advances the Warren1995 (phi, c) state by k stencil steps): a BF16
// tensor-core GEMM with FP32 accumulation whose operand loaders and result
// storers implement the patchify / unpatchify implicit-GEMM convolutions and
// the 1x1 convolutions (forward, data gradient, weight gradient), plus
// depthwise 3x3 convolution, bias, GELU, loss and Adam kernels.
//
// Activations are channels-last: token t = (sample, row, col) of the patch
// grid, channel n contiguous. Weights of a 1x1 / patch convolution are
// W[out][in] (bf16 copy for the GEMM, fp32 master for Adam).
//
// Tensor-core path: mma.sync.m16n8k16 (bf16 x bf16 -> f32). A 64x64 output
// tile per CTA of 4 warps (32x32 each), k in steps of 32 staged in shared
// memory (A row-major, B stored transposed so every fragment register is one
// 32-bit shared load).
#include <cuda_bf16.h>
#include <math.h>

#include <initializer_list>
#include <type_traits>

#include "ppf_common.cuh"
#include "ppf_tma.cuh"

namespace ppf {
namespace {

// Every kernel of the network waits for the one before (pdl_wait) before it touches
// memory and is launched while that one still runs: a pass is a chain of some 100
// launches of about 10 us, whose starts are then hidden (one gradient evaluation of
// 8 x 512 x 512: 1186 -> 1032 us).
template <typename... KArgs, typename... Args>
cudaError_t sg_launch(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                      Args... args) {
  return launch(kern, grid, block, smem, s, true, args...);
}

constexpr int BM = 64, BN = 64, BK = 32;
constexpr int kGemmThreads = 128;
constexpr int kPad = 8;  // shared row padding (bf16 elements)

// ---------------------------------------------------------------- loaders
// A(m, k) and B(k, n) element accessors (return float; converted to bf16).
struct StridedBf16 {  // element (i, j) = x[i * si + j * sj]
  const __nv_bfloat16* x;
  long long si, sj;
};

// Patch gather of a 2-channel state field stack: rows are tokens
// (b, ty, tx), columns are (ch, py, px) of the P x P patch; fields are fp32
// [b][ch][H][pitch] and are normalised by `scale[ch]` on the fly.
struct PatchGather {
  const float* f;
  int P, H, W, pitch, gh, gw;  // image H x W, patch grid gh x gw
  float o0, s0, o1, s1;        // input normalisation (v - o) * s per channel
  __device__ float operator()(long long t, long long k) const {
    const int per = gh * gw;
    const int b = (int)(t / per);
    const int r = (int)(t - (long long)b * per);
    const int ty = r / gw, tx = r - ty * gw;
    const int ch = (int)(k / (P * P));
    const int q = (int)(k - (long long)ch * P * P);
    const int py = q / P, px = q - py * P;
    const float v = f[(((long long)b * 2 + ch) * H + ty * P + py) * pitch + tx * P + px];
    return ch == 0 ? (v - o0) * s0 : (v - o1) * s1;
  }
};

// The same gather seen as B(k = token, n = (ch, py, px)) for weight grads.
struct PatchGatherT {
  PatchGather g;
  __device__ float operator()(long long k, long long n) const { return g(k, n); }
};

// ---------------------------------------------------------------- storers
// C(m, n) epilogues. All receive the fp32 accumulator. pre() is what the
// storer reads of the element beforehand (0 where it reads nothing): kernels
// fetch it for a batch of elements before they store any, since a store that
// might alias the next load would chain one round trip per element. put2 / pre2:
// elements n, n + 1 (n even) at once, where pairs() holds.
__device__ __forceinline__ void put_pair(float* p, float a, float b) {
  *reinterpret_cast<float2*>(p) = make_float2(a, b);
}
__device__ __forceinline__ void put_pair(__nv_bfloat16* p, float a, float b) {
  *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b);
}
inline bool pair_ok(const void* p, int elem) { return (uintptr_t)p % (2 * elem) == 0; }

struct StoreF32 {  // y[m * ld + n] (= or +=) acc + bias[n]
  float* y;
  const float* bias;
  long long ld;
  int accumulate;
  bool pairs() const { return pair_ok(y, 4) && ld % 2 == 0; }
  __device__ float pre(long long m, long long n) const {
    return accumulate ? y[m * ld + n] : 0.f;
  }
  __device__ float2 pre2(long long m, long long n) const {
    return accumulate ? *reinterpret_cast<const float2*>(y + m * ld + n) : make_float2(0.f, 0.f);
  }
  __device__ float value(long long n, float v, float e) const {
    if (bias) v += bias[n];
    return accumulate ? e + v : v;
  }
  __device__ void put(long long m, long long n, float v, float e) const {
    y[m * ld + n] = value(n, v, e);
  }
  __device__ void put2(long long m, long long n, float v, float w, float2 e) const {
    put_pair(y + m * ld + n, value(n, v, e.x), value(n + 1, w, e.y));
  }
  __device__ void operator()(long long m, long long n, float v) const { put(m, n, v, pre(m, n)); }
};

struct StoreBf16Pair {  // fp32 and bf16 copies of acc + bias (no activation)
  float* y;
  __nv_bfloat16* yb;
  const float* bias;
  long long ld;
  bool pairs() const { return pair_ok(y, 4) && pair_ok(yb, 2) && ld % 2 == 0; }
  __device__ float pre(long long, long long) const { return 0.f; }
  __device__ float2 pre2(long long, long long) const { return make_float2(0.f, 0.f); }
  __device__ void put(long long m, long long n, float v, float) const {
    if (bias) v += bias[n];
    y[m * ld + n] = v;
    yb[m * ld + n] = __float2bfloat16(v);
  }
  __device__ void put2(long long m, long long n, float v, float w, float2) const {
    if (bias) v += bias[n], w += bias[n + 1];
    put_pair(y + m * ld + n, v, w);
    put_pair(yb + m * ld + n, v, w);
  }
  __device__ void operator()(long long m, long long n, float v) const { put(m, n, v, 0.f); }
};

__device__ __forceinline__ float gelu(float x) {
  return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f));
}
__device__ __forceinline__ float gelu_grad(float x) {
  return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) +
         x * 0.39894228040143268f * expf(-0.5f * x * x);
}

struct StoreGelu {  // pre = acc + bias (fp32), act = gelu(pre) (bf16)
  float* out;
  __nv_bfloat16* act;
  const float* bias;
  long long ld;
  bool pairs() const { return pair_ok(out, 4) && pair_ok(act, 2) && ld % 2 == 0; }
  __device__ float pre(long long, long long) const { return 0.f; }
  __device__ float2 pre2(long long, long long) const { return make_float2(0.f, 0.f); }
  __device__ void put(long long m, long long n, float v, float) const {
    v += bias[n];
    out[m * ld + n] = v;
    act[m * ld + n] = __float2bfloat16(gelu(v));
  }
  __device__ void put2(long long m, long long n, float v, float w, float2) const {
    v += bias[n], w += bias[n + 1];
    put_pair(out + m * ld + n, v, w);
    put_pair(act + m * ld + n, gelu(v), gelu(w));
  }
  __device__ void operator()(long long m, long long n, float v) const { put(m, n, v, 0.f); }
};

struct StoreGeluGrad {  // d_pre = acc * gelu'(pre), bf16
  const float* x;
  __nv_bfloat16* dpre;
  long long ld;
  bool pairs() const { return pair_ok(x, 4) && pair_ok(dpre, 2) && ld % 2 == 0; }
  __device__ float pre(long long m, long long n) const { return x[m * ld + n]; }
  __device__ float2 pre2(long long m, long long n) const {
    return *reinterpret_cast<const float2*>(x + m * ld + n);
  }
  __device__ void put(long long m, long long n, float v, float e) const {
    dpre[m * ld + n] = __float2bfloat16(v * gelu_grad(e));
  }
  __device__ void put2(long long m, long long n, float v, float w, float2 e) const {
    put_pair(dpre + m * ld + n, v * gelu_grad(e.x), w * gelu_grad(e.y));
  }
  __device__ void operator()(long long m, long long n, float v) const { put(m, n, v, pre(m, n)); }
};

struct StoreResidual {  // y = yin + acc + bias (yin may be y), and a bf16 copy of y
  const float* yin;
  float* y;
  __nv_bfloat16* yb;
  const float* bias;
  long long ld;
  bool pairs() const {
    return pair_ok(yin, 4) && pair_ok(y, 4) && pair_ok(yb, 2) && ld % 2 == 0;
  }
  __device__ float pre(long long m, long long n) const { return yin[m * ld + n]; }
  __device__ float2 pre2(long long m, long long n) const {
    return *reinterpret_cast<const float2*>(yin + m * ld + n);
  }
  __device__ void put(long long m, long long n, float v, float e) const {
    const float r = e + v + bias[n];
    y[m * ld + n] = r;
    yb[m * ld + n] = __float2bfloat16(r);
  }
  __device__ void put2(long long m, long long n, float v, float w, float2 e) const {
    const float r = e.x + v + bias[n], q = e.y + w + bias[n + 1];
    put_pair(y + m * ld + n, r, q);
    put_pair(yb + m * ld + n, r, q);
  }
  __device__ void operator()(long long m, long long n, float v) const { put(m, n, v, pre(m, n)); }
};

struct StoreAtomic {  // y[m * ld + n] += acc (split-k weight gradients)
  float* y;
  long long ld;
  bool pairs() const { return true; }
  __device__ float pre(long long, long long) const { return 0.f; }
  __device__ float2 pre2(long long, long long) const { return make_float2(0.f, 0.f); }
  __device__ void put(long long m, long long n, float v, float) const { (*this)(m, n, v); }
  __device__ void put2(long long m, long long n, float v, float w, float2) const {
    atomicAdd(y + m * ld + n, v);
    atomicAdd(y + m * ld + n + 1, w);
  }
  __device__ void operator()(long long m, long long n, float v) const {
    atomicAdd(y + m * ld + n, v);
  }
};

// ---------------------------------------------------------------- GEMM
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4],
                                         const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Shared tile fill (64 rows x BK columns): S[r][c] = operand element
// (row r0 + r, column c0 + c); zero outside rows < R, columns < ce.
// Generic loaders: consecutive threads take consecutive loader columns
// (the patch gather's pixel index), i.e. tile columns for A, rows for B.
template <typename LD, bool kTransposed>
__device__ __forceinline__ void fill_tile(__nv_bfloat16 (*S)[BK + kPad], const LD& ld, long long r0,
                                          long long R, long long c0, long long ce, int tid) {
  for (int i = tid; i < 64 * BK; i += kGemmThreads) {
    const int r = kTransposed ? i % 64 : i / BK;
    const int c = kTransposed ? i / 64 : i % BK;
    const long long gr = r0 + r, gc = c0 + c;
    float v = 0.f;
    if (gr < R && gc < ce) v = kTransposed ? ld(gc, gr) : ld(gr, gc);
    S[r][c] = __float2bfloat16(v);
  }
}

// Strided bf16 operands: element (r, c) = x[r * rs + c * cs]. Unit column
// stride: 16-byte vector loads where aligned; unit row stride: consecutive
// threads take consecutive rows (coalesced), otherwise scalar.
__device__ __forceinline__ void fill_strided(__nv_bfloat16 (*S)[BK + kPad],
                                             const __nv_bfloat16* __restrict__ x, long long rs,
                                             long long cs, long long r0, long long R, long long c0,
                                             long long ce, int tid) {
  const __nv_bfloat16 zero = __float2bfloat16(0.f);
  if (cs == 1) {
    const bool vec = (rs & 7) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    for (int i = tid; i < 64 * (BK / 8); i += kGemmThreads) {
      const int r = i / (BK / 8), c = (i - r * (BK / 8)) * 8;
      const long long gr = r0 + r, gc = c0 + c;
      if (vec && gr < R && gc + 8 <= ce) {
        *reinterpret_cast<uint4*>(&S[r][c]) = *reinterpret_cast<const uint4*>(x + gr * rs + gc);
      } else {
#pragma unroll
        for (int q = 0; q < 8; ++q) S[r][c + q] = (gr < R && gc + q < ce) ? x[gr * rs + gc + q] : zero;
      }
    }
  } else {
    for (int i = tid; i < 64 * BK; i += kGemmThreads) {
      const int c = i / 64, r = i - c * 64;
      const long long gr = r0 + r, gc = c0 + c;
      S[r][c] = (gr < R && gc < ce) ? x[gr * rs + gc * cs] : zero;
    }
  }
}

template <typename LA>
__device__ __forceinline__ void fill_a(__nv_bfloat16 (*S)[BK + kPad], const LA& la, long long m0,
                                       long long M, long long k0, long long ke, int tid) {
  fill_tile<LA, false>(S, la, m0, M, k0, ke, tid);
}
__device__ __forceinline__ void fill_a(__nv_bfloat16 (*S)[BK + kPad], const StridedBf16& la,
                                       long long m0, long long M, long long k0, long long ke,
                                       int tid) {
  fill_strided(S, la.x + m0 * la.si + k0 * la.sj, la.si, la.sj, 0, M - m0, 0, ke - k0, tid);
}
// B tiles are stored transposed: S[n - n0][k - k0] = B(k, n).
template <typename LB>
__device__ __forceinline__ void fill_b(__nv_bfloat16 (*S)[BK + kPad], const LB& lb, long long n0,
                                       long long N, long long k0, long long ke, int tid) {
  fill_tile<LB, true>(S, lb, n0, N, k0, ke, tid);
}
__device__ __forceinline__ void fill_b(__nv_bfloat16 (*S)[BK + kPad], const StridedBf16& lb,
                                       long long n0, long long N, long long k0, long long ke,
                                       int tid) {
  fill_strided(S, lb.x + k0 * lb.si + n0 * lb.sj, lb.sj, lb.si, 0, N - n0, 0, ke - k0, tid);
}

// Patch gather, 4 consecutive patch columns (px .. px + 3 of one patch row,
// P a multiple of 4) per 16-byte load: (token t, column k) -> fields
// offset; the columns of a 4-group share channel and patch row.
__device__ __forceinline__ long long patch_offset(const PatchGather& p, long long t, int k) {
  const int per = p.gh * p.gw;
  const int b = (int)(t / per);
  const int r = (int)(t - (long long)b * per);
  const int ty = r / p.gw, tx = r - ty * p.gw;
  const int ch = k / (p.P * p.P);
  const int q = k - ch * p.P * p.P;
  const int py = q / p.P, px = q - py * p.P;
  return (((long long)b * 2 + ch) * p.H + ty * p.P + py) * p.pitch + tx * p.P + px;
}

__device__ __forceinline__ void fill_a(__nv_bfloat16 (*S)[BK + kPad], const PatchGather& la,
                                       long long m0, long long M, long long k0, long long ke,
                                       int tid) {
  if ((la.P & 3) || (la.pitch & 3) || (reinterpret_cast<uintptr_t>(la.f) & 15)) {
    fill_tile<PatchGather, false>(S, la, m0, M, k0, ke, tid);
    return;
  }
  for (int i = tid; i < 64 * (BK / 4); i += kGemmThreads) {
    const int r = i / (BK / 4), c = (i - r * (BK / 4)) * 4;
    const long long m = m0 + r, k = k0 + c;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (m < M && k + 4 <= ke) {
      const float4 x = *reinterpret_cast<const float4*>(la.f + patch_offset(la, m, (int)k));
      const bool c0 = k < (long long)la.P * la.P;  // channel 0 (the group shares it)
      const float o = c0 ? la.o0 : la.o1, sc = c0 ? la.s0 : la.s1;
      v[0] = (x.x - o) * sc;
      v[1] = (x.y - o) * sc;
      v[2] = (x.z - o) * sc;
      v[3] = (x.w - o) * sc;
    } else if (m < M) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (k + q < ke) v[q] = la(m, k + q);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) S[r][c + q] = __float2bfloat16(v[q]);
  }
}

// B(k = token, n = patch column) of the patch weight gradient: 4
// consecutive n per load, stored transposed (S[n][k]).
__device__ __forceinline__ void fill_b(__nv_bfloat16 (*S)[BK + kPad], const PatchGatherT& lb,
                                       long long n0, long long N, long long k0, long long ke,
                                       int tid) {
  const PatchGather& g = lb.g;
  if ((g.P & 3) || (g.pitch & 3) || (reinterpret_cast<uintptr_t>(g.f) & 15)) {
    fill_tile<PatchGatherT, true>(S, lb, n0, N, k0, ke, tid);
    return;
  }
  for (int i = tid; i < (64 / 4) * BK; i += kGemmThreads) {
    const int c = i / (64 / 4), r = (i - c * (64 / 4)) * 4;  // token column c, n rows r..r+3
    const long long k = k0 + c, n = n0 + r;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (k < ke && n + 4 <= N) {
      const float4 x = *reinterpret_cast<const float4*>(g.f + patch_offset(g, k, (int)n));
      const bool c0 = n < (long long)g.P * g.P;
      const float o = c0 ? g.o0 : g.o1, sc = c0 ? g.s0 : g.s1;
      v[0] = (x.x - o) * sc;
      v[1] = (x.y - o) * sc;
      v[2] = (x.z - o) * sc;
      v[3] = (x.w - o) * sc;
    } else if (k < ke) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (n + q < N) v[q] = g(k, n + q);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) S[r + q][c] = __float2bfloat16(v[q]);
  }
}

// C(M x N) = sum over k in [k0, k1) of A(m, k) B(k, n); blockIdx.z splits k.
template <typename LA, typename LB, typename ST>
__global__ void __launch_bounds__(kGemmThreads)
    gemm_kernel(LA la, LB lb, ST st, long long M, long long N, long long K, long long kchunk) {
  __shared__ __align__(16) __nv_bfloat16 As[BM][BK + kPad];
  __shared__ __align__(16) __nv_bfloat16 Bt[BN][BK + kPad];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long m0 = (long long)blockIdx.y * BM, n0 = (long long)blockIdx.x * BN;
  const long long kb = (long long)blockIdx.z * kchunk;
  const long long ke = kb + kchunk < K ? kb + kchunk : K;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  const int g = lane >> 2, t = lane & 3;
  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.f;

  pdl_wait();
  pdl_launch_next();
  for (long long k0 = kb; k0 < ke; k0 += BK) {
    fill_a(As, la, m0, M, k0, ke, tid);
    fill_b(Bt, lb, n0, N, k0, ke, tid);
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; kk += 16) {
      uint32_t a[2][4], b[4][2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = wm + i * 16 + g;
        a[i][0] = *reinterpret_cast<const uint32_t*>(&As[r][kk + 2 * t]);
        a[i][1] = *reinterpret_cast<const uint32_t*>(&As[r + 8][kk + 2 * t]);
        a[i][2] = *reinterpret_cast<const uint32_t*>(&As[r][kk + 2 * t + 8]);
        a[i][3] = *reinterpret_cast<const uint32_t*>(&As[r + 8][kk + 2 * t + 8]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = wn + j * 8 + g;
        b[j][0] = *reinterpret_cast<const uint32_t*>(&Bt[c][kk + 2 * t]);
        b[j][1] = *reinterpret_cast<const uint32_t*>(&Bt[c][kk + 2 * t + 8]);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_bf16(acc[i][j], a[i], b[j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const long long m = m0 + wm + i * 16 + g + (r >= 2 ? 8 : 0);
        const long long n = n0 + wn + j * 8 + 2 * t + (r & 1);
        if (m < M && n < N) st(m, n, acc[i][j][r]);
      }
}

// ---------------------------------------------------------------- pipelined
// The same GEMM for bf16 operands with one contiguous axis each, 16-byte
// aligned: tiles come by cp.async, kPStages - 1 ahead, in the order they have
// in memory (A as [m][k] or [k][m], B as [n][k] or [k][n]), and ldmatrix, with
// .trans where the contiguous axis is not k, gives the fragments. The
// accumulators see the k steps in gemm_kernel's order: the same bits.
//
// gemm_kernel transposes a tile whose contiguous axis is not k element by
// element on its way into shared memory and waits for each tile's loads before
// the next: latency-bound (8192 tokens, us: dW of 384 x 192 66 -> 8.7, its input's
// gradient 8192 x 384 x 192 with the GELU derivative 50 -> 15.7, 8192 x 192 x 384
// 46 -> 10.9).
constexpr int kPStages = 4;
constexpr int kRowK = BK + 8;   // row of a tile stored with k contiguous (80 bytes)
constexpr int kRowM = 64 + 8;   // row of a tile stored with m or n contiguous (144 bytes)
constexpr int kPTile = 64 * kRowK > BK * kRowM ? 64 * kRowK : BK * kRowM;

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldmatrix4t(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

// One operand's 64 x BK tile at (r0, k0) of x: KC: element (r, k) at r * ld + k,
// else at k * ld + r; zero outside R rows and below ke.
template <bool KC>
__device__ __forceinline__ void copy_tile(__nv_bfloat16* s, const __nv_bfloat16* __restrict__ x,
                                          long long ld, long long r0, long long R, long long k0,
                                          long long ke, int tid) {
#pragma unroll
  for (int q = 0; q < 64 * BK / 8 / kGemmThreads; ++q) {
    const int i = tid + q * kGemmThreads;
    const int row = KC ? i / (BK / 8) : i / 8;
    const int c = (KC ? i % (BK / 8) : i % 8) * 8;
    const long long r = r0 + (KC ? row : c), k = k0 + (KC ? c : row);
    const bool in = r < R && k < ke;
    const __nv_bfloat16* src = x + (in ? (KC ? r * ld + k : k * ld + r) : 0);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(s + row * (KC ? kRowK : kRowM) + c)),
                 "l"(src), "r"(in ? 16 : 0)
                 : "memory");
  }
}

// A warp's 32 x 32 accumulators to C at (m0, n0), eight pairs' reads before their
// stores.
template <typename ST>
__device__ __forceinline__ void store_pairs(const float (&acc)[2][4][4], const ST& st,
                                            long long m0, long long n0, long long M, long long N,
                                            int lane) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    float2 e[4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const long long m = m0 + i * 16 + g + 8 * h, n = n0 + j * 8 + 2 * t;
        e[j][h] = m < M && n < N ? st.pre2(m, n) : make_float2(0.f, 0.f);
      }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const long long m = m0 + i * 16 + g + 8 * h, n = n0 + j * 8 + 2 * t;
        if (m < M && n < N) st.put2(m, n, acc[i][j][2 * h], acc[i][j][2 * h + 1], e[j][h]);
      }
  }
}

template <bool AK, bool BKC, typename ST>
__global__ void __launch_bounds__(kGemmThreads)
    gemm_pipe_kernel(const __nv_bfloat16* __restrict__ a, long long lda,
                     const __nv_bfloat16* __restrict__ b, long long ldb, ST st, long long M,
                     long long N, long long K, long long kchunk) {
  __shared__ __align__(16) __nv_bfloat16 As[kPStages][kPTile];
  __shared__ __align__(16) __nv_bfloat16 Bs[kPStages][kPTile];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long m0 = (long long)blockIdx.y * BM, n0 = (long long)blockIdx.x * BN;
  const long long kb = (long long)blockIdx.z * kchunk;
  const long long ke = kb + kchunk < K ? kb + kchunk : K;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  const int nk = (int)((ke - kb + BK - 1) / BK);
  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.f;
  pdl_wait();
  pdl_launch_next();
  auto issue = [&](int kt) {
    if (kt < nk) {
      const int q = kt % kPStages;
      copy_tile<AK>(As[q], a, lda, m0, M, kb + (long long)kt * BK, ke, tid);
      copy_tile<BKC>(Bs[q], b, ldb, n0, N, kb + (long long)kt * BK, ke, tid);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int kt = 0; kt < kPStages - 1; ++kt) issue(kt);
  const int mi = lane >> 3, mr = lane & 7;  // ldmatrix: matrix and row of this lane
  for (int kt = 0; kt < nk; ++kt) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kPStages - 2) : "memory");
    __syncthreads();  // tile kt is here, and every warp is done with tile kt - 1
    issue(kt + kPStages - 1);
    const __nv_bfloat16* A = As[kt % kPStages];
    const __nv_bfloat16* B = Bs[kt % kPStages];
#pragma unroll
    for (int kk = 0; kk < BK; kk += 16) {
      uint32_t fa[2][4], fb[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int m = wm + i * 16 + (mi & 1) * 8, k = kk + (mi >> 1) * 8;
        if (AK)
          ldmatrix4(fa[i], A + (m + mr) * kRowK + k);
        else
          ldmatrix4t(fa[i], A + (k + mr) * kRowM + m);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int n = wn + j * 16 + (mi >> 1) * 8, k = kk + (mi & 1) * 8;
        if (BKC)
          ldmatrix4(fb[j], B + (n + mr) * kRowK + k);
        else
          ldmatrix4t(fb[j], B + (k + mr) * kRowM + n);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t bb[2] = {fb[j >> 1][(j & 1) * 2], fb[j >> 1][(j & 1) * 2 + 1]};
          mma_bf16(acc[i][j], fa[i], bb);
        }
    }
  }
  store_pairs(acc, st, m0 + wm, n0 + wn, M, N, lane);
}

// Whether the pipelined kernel applies to one operand of R rows: unit stride
// along k or along the rows, whole 16-byte vectors.
inline bool pipe_operand(const void* x, long long sr, long long sk, long long R, long long K) {
  if (reinterpret_cast<uintptr_t>(x) & 15) return false;
  if (sk == 1) return (sr & 7) == 0 && (K & 7) == 0;
  return sr == 1 && (sk & 7) == 0 && (R & 7) == 0;
}

template <typename ST>
cudaError_t launch_pipe(const StridedBf16& la, const StridedBf16& lb, const ST& st, long long M,
                        long long N, long long K, long long kchunk, dim3 grid, cudaStream_t s) {
  const bool ak = la.sj == 1, bk = lb.si == 1;
  const long long lda = ak ? la.si : la.sj, ldb = bk ? lb.sj : lb.si;
  auto kern = ak ? (bk ? gemm_pipe_kernel<true, true, ST> : gemm_pipe_kernel<true, false, ST>)
                 : (bk ? gemm_pipe_kernel<false, true, ST> : gemm_pipe_kernel<false, false, ST>);
  return sg_launch(kern, grid, kGemmThreads, 0, s, la.x, lda, lb.x, ldb, st, M, N, K, kchunk);
}

// The patch embedding and its weight gradient: gemm_pipe_kernel with the patch
// gather as one operand, whose raw floats come by cp.async too (P a multiple of 4:
// four patch columns are 16 aligned bytes, and 16 of them share a channel) and are
// normalised and rounded as the fragments are read. FWD: A(m = token, k = patch
// column), x the [n][k] weights. Else B(k = token, n = patch column), x the tokens'
// gradient, [k][m]. gemm_kernel's k order and roundings: the same bits. Latency-bound
// like gemm_kernel, whose loads each wait for the tile before: 8192 tokens of P 16,
// 192 channels, us: embedding 73.5 -> 18.9, weight gradient 92.3 -> 21.6.
constexpr int kGStages = 3;

template <bool FWD, typename ST>
__global__ void __launch_bounds__(kGemmThreads)
    gemm_gather_kernel(const PatchGather g, const __nv_bfloat16* __restrict__ x, long long ldx,
                       ST st, long long M, long long N, long long K, long long kchunk) {
  constexpr int kRow = FWD ? BK + 8 : 64 + 4;  // floats: no bank conflicts in the fragments
  constexpr int kGroups = (FWD ? BK : 64) / 4;  // 16-byte groups of a row
  __shared__ __align__(16) float Gs[kGStages][(FWD ? 64 : BK) * kRow];
  __shared__ __align__(16) __nv_bfloat16 Xs[kGStages][kPTile];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long m0 = (long long)blockIdx.y * BM, n0 = (long long)blockIdx.x * BN;
  const long long kb = (long long)blockIdx.z * kchunk;
  const long long ke = kb + kchunk < K ? kb + kchunk : K;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  const int nk = (int)((ke - kb + BK - 1) / BK);
  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.f;
  // this thread's groups: one group column, four rows of the tile
  const int gc = tid % kGroups * 4, gr = tid / kGroups;
  constexpr int kStep = kGemmThreads / kGroups;
  const int per = g.gh * g.gw, pp = g.P * g.P;
  auto token = [&](int b, int r) {  // offset of token r of sample b
    const int ty = r / g.gw, tx = r - ty * g.gw;
    return ((long long)b * 2 * g.H + ty * g.P) * g.pitch + tx * g.P;
  };
  auto column = [&](int k) {  // offset of a patch column within its token
    const int ch = k >= pp, q = k - ch * pp, py = q / g.P;
    return ((long long)ch * g.H + py) * g.pitch + (q - py * g.P);
  };
  long long fixed[FWD ? 4 : 1];  // the tokens' (FWD) or the column's offset; -1: outside
  int b0 = 0, r0 = 0;            // sample and token within it of the first k (not FWD)
  if (FWD) {
#pragma unroll
    for (int q = 0; q < (FWD ? 4 : 1); ++q) {
      const long long m = m0 + gr + q * kStep;
      const int b = (int)(m / per);
      fixed[q] = m < M ? token(b, (int)(m - (long long)b * per)) : -1;
    }
  } else {
    fixed[0] = n0 + gc < N ? column((int)n0 + gc) : -1;
    b0 = (int)(kb / per);
    r0 = (int)(kb - (long long)b0 * per);
  }
  pdl_wait();
  pdl_launch_next();
  auto issue = [&](int kt) {
    if (kt < nk) {
      const int s = kt % kGStages;
      const long long k0 = kb + (long long)kt * BK;
      const bool kin = k0 + gc < ke;
      const long long col = FWD ? (kin ? column((int)k0 + gc) : 0) : fixed[0];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int row = gr + q * kStep;
        long long off;
        bool in;
        if (FWD) {
          in = kin && fixed[FWD ? q : 0] >= 0;
          off = fixed[FWD ? q : 0] + col;
        } else {
          const int r = r0 + kt * BK + row, b = r / per;
          in = col >= 0 && k0 + row < ke;
          off = token(b0 + b, r - b * per) + col;
        }
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(Gs[s] + row * kRow + gc)),
                     "l"(g.f + (in ? off : 0)), "r"(in ? 16 : 0)
                     : "memory");
      }
      copy_tile<FWD>(Xs[s], x, ldx, FWD ? n0 : m0, FWD ? N : M, k0, ke, tid);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int kt = 0; kt < kGStages - 1; ++kt) issue(kt);
  const int mi = lane >> 3, mr = lane & 7;
  const int fg = lane >> 2, ft = lane & 3;
  auto pack = [&](float u, float v, bool ch) {
    const float o = ch ? g.o1 : g.o0, sc = ch ? g.s1 : g.s0;
    const __nv_bfloat162 h = __floats2bfloat162_rn((u - o) * sc, (v - o) * sc);
    return *reinterpret_cast<const uint32_t*>(&h);
  };
  for (int kt = 0; kt < nk; ++kt) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kGStages - 2) : "memory");
    __syncthreads();
    issue(kt + kGStages - 1);
    const float* G = Gs[kt % kGStages];
    const __nv_bfloat16* X = Xs[kt % kGStages];
#pragma unroll
    for (int kk = 0; kk < BK; kk += 16) {
      uint32_t fa[2][4], fb[4][2];
      if (FWD) {
        const bool ch = kb + (long long)kt * BK + kk >= pp;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int r = 0; r < 4; ++r) {  // rows fg, fg + 8; columns 2 ft, 2 ft + 8
            const float2 v = *reinterpret_cast<const float2*>(
                G + (wm + i * 16 + fg + (r & 1) * 8) * kRow + kk + 2 * ft + (r >> 1) * 8);
            fa[i][r] = pack(v.x, v.y, ch);
          }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          uint32_t r[4];
          ldmatrix4(r, X + (wn + j * 16 + (mi >> 1) * 8 + mr) * kRowK + kk + (mi & 1) * 8);
          fb[2 * j][0] = r[0], fb[2 * j][1] = r[1];
          fb[2 * j + 1][0] = r[2], fb[2 * j + 1][1] = r[3];
        }
      } else {
#pragma unroll
        for (int i = 0; i < 2; ++i)
          ldmatrix4t(fa[i], X + (kk + (mi >> 1) * 8 + mr) * kRowM + wm + i * 16 + (mi & 1) * 8);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool ch = n0 + wn + j * 8 >= pp;
#pragma unroll
          for (int r = 0; r < 2; ++r) {  // rows 2 ft, 2 ft + 1 (+ 8); column fg
            const float* v = G + (kk + 2 * ft + r * 8) * kRow + wn + j * 8 + fg;
            fb[j][r] = pack(v[0], v[kRow], ch);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) mma_bf16(acc[i][j], fa[i], fb[j]);
    }
  }
  store_pairs(acc, st, m0 + wm, n0 + wn, M, N, lane);
}

// Whether gemm_gather_kernel applies to the gather; k indexes and token numbers
// within a split stay below 2^31.
inline bool gather_operand(const PatchGather& g, long long cols, long long kspan) {
  return g.P % 4 == 0 && g.pitch % 4 == 0 && !(reinterpret_cast<uintptr_t>(g.f) & 15) &&
         cols < (1LL << 31) && kspan + (long long)g.gh * g.gw + BK < (1LL << 31);
}

// ---------------------------------------------------------------- tcgen05
// The tcgen05 path is on by default for GEMMs of at least kTcMinRows rows
// (the training batches, N 384, K 192: 4096 tokens take 8.2 us here and on
// mma.sync, 8192 tokens 8.3 and 12.3, 65536 tokens 41 and 59); below that (the
// 1024-token prediction) its few tiles leave most SMs idle and mma.sync's
// 64 x 64 tiles win. ppf_sg_set_tensor_path(0) selects mma.sync everywhere.
int g_tc_enabled = 1;
constexpr long long kTcMinRows = 4096;
bool tc_enabled() { return g_tc_enabled != 0; }

// 5th-generation tensor-core GEMM for the GEMMs whose operands are both
// K-contiguous bf16 (A[m][k], B stored as [n][k]): the forward 1x1
// convolutions and the output head. One CTA (8 warps) owns a 128 x TN
// output tile whose FP32 accumulator lives in tensor memory (128 lanes x
// TN columns, allocated by warp 0); k advances in 64-wide tiles staged in
// shared memory in the K-major 128-byte-swizzled layout (8-row x 128-byte
// atoms, 1024 bytes apart along the rows: row r's 16-byte chunk j of k at
// (r / 8) * 1024 + (r % 8) * 128 + ((j ^ (r % 8)) * 16), see tc_desc and
// tc_load_tile). Two stages: the tile for kt + 1 is
// loaded while the tensor core works on kt. One thread issues
// tcgen05.mma (kind::f16, BF16 x BF16 -> F32, M = 128, N = TN, K = 16 per
// instruction) and tcgen05.commit arrives on the stage's mbarrier; the
// epilogue reads the accumulator with tcgen05.ld (warp w: lanes
// 32 (w % 4) .. + 31 = rows, half of the columns) and applies the storer. Every
// mbarrier wait is bounded; a timeout sets PPF_STATUS_TIMEOUT, lets the issued MMAs
// finish (bounded) and frees the tensor memory.
//
// TN is 64, but 128 where N is a multiple of 128 from 512 on. Tiles of 64 columns
// spread a batch more evenly over the SMs and pad N = 192 less, but read A more often.
// us with 64 / 128 columns: 8192 x 384 8.3 / 10.2, 65536 x 192 30.8 / 36.0,
// 65536 x 384 41.0 / 43.0, 131072 x 384 77.7 / 77.8; 8192 x 512 11.3 / 10.3,
// 65536 x 512 (K 512) 70.4 / 67.5.
constexpr int TCM = 128, TCK = 64, kTcThreads = 256;
template <int TN>
constexpr int kTcStage = (TCM + TN) * TCK * 2;  // bytes of one A + B stage
template <int TN>
constexpr uint32_t kTcIdesc = (1u << 4)                        // D: F32
                              | (1u << 7) | (1u << 10)         // A, B: BF16, K-major
                              | ((uint32_t)(TN >> 3) << 17)    // N / 8
                              | ((uint32_t)(TCM >> 4) << 24);  // M / 16

__device__ __forceinline__ uint32_t tc_smem(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// shared-memory matrix descriptor: K-major, 128-byte swizzle (8-row x
// 128-byte atoms, stride byte offset 1024 between atoms along M / N; the
// leading offset is implied by the swizzle), descriptor version 1, the tile
// 1024-byte aligned. Stepping K by 16 elements moves the start by 32 bytes.
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)1 << 16) |
         ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ bool tc_wait(uint64_t* bar, uint32_t parity, uint32_t limit) {
  const uint32_t a = tc_smem(bar);
  for (uint32_t i = 0; i < limit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 20000;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Pipeline: a producer thread (warp 0) streams the k-tiles of A (128 rows)
// and B (TN columns) into kTcStages shared-memory stages with TMA tensor
// loads (cp.async.bulk.tensor.2d, 128-byte swizzle: the K-major SW128 layout
// the descriptors describe), completing on the stage's `full` mbarrier; an
// MMA thread (warp 1) waits for a stage, issues its four tcgen05.mma (K = 16
// each) into the TMEM accumulator and commits onto the stage's `empty`
// mbarrier, which frees the stage for the producer; a final commit onto
// `done` releases the warps into the epilogue. With three stages
// of 24 or 32 KB two or three CTAs share an SM, so one CTA's epilogue overlaps
// another's loads.
// Every wait is bounded; a timeout sets PPF_STATUS_TIMEOUT, the issued MMAs
// and loads are waited for (bounded) and the tensor memory is freed.
constexpr int kTcStages = 3;

__device__ __forceinline__ void tc_tma_load(void* dst, const CUtensorMap* map, int x, int y,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(tc_smem(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(tc_smem(bar))
      : "memory");
}

template <int TN, typename ST>
__global__ void __launch_bounds__(kTcThreads)
    tc_gemm_kernel(const __grid_constant__ CUtensorMap map_a,
                   const __grid_constant__ CUtensorMap map_b, ST st, long long M, long long N,
                   long long K, int* __restrict__ lib_status) {
  extern __shared__ __align__(1024) uint8_t tc_stage[];
  __shared__ __align__(8) uint64_t full[kTcStages], empty[kTcStages], done;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag, consumed;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long m0 = (long long)blockIdx.y * TCM, n0 = (long long)blockIdx.x * TN;
  uint8_t* const base = tc_stage + ((1024 - (tc_smem(tc_stage) & 1023)) & 1023);
  auto sa = [&](int st_) { return base + st_ * kTcStage<TN>; };
  auto sb = [&](int st_) { return base + st_ * kTcStage<TN> + TCM * TCK * 2; };
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(tc_smem(&tmem_base)), "r"(TN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < kTcStages; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&full[i])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&empty[i])) : "memory");
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&done)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_flag = 0;
    consumed = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base;
  pdl_wait();
  pdl_launch_next();
  const int nk = (int)((K + TCK - 1) / TCK);
  constexpr uint32_t kLimit = 1u << 15;
  int issued = 0;
  if (warp == 0 && lane == 0) {  // producer
    for (int kt = 0; kt < nk; ++kt) {
      const int s = kt % kTcStages;
      if (kt >= kTcStages &&
          !tc_wait(&empty[s], (uint32_t)((kt / kTcStages - 1) & 1), kLimit)) {
        atomicExch(&abort_flag, 1);
        break;
      }
      if (*(volatile int*)&abort_flag) break;
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                   ::"r"(tc_smem(&full[s])), "r"((uint32_t)kTcStage<TN>) : "memory");
      tc_tma_load(sa(s), &map_a, kt * TCK, (int)m0, &full[s]);
      tc_tma_load(sb(s), &map_b, kt * TCK, (int)n0, &full[s]);
      issued = kt + 1;
    }
  } else if (warp == 1 && lane == 0) {  // MMA issuer
    int kt = 0;
    for (; kt < nk; ++kt) {
      const int s = kt % kTcStages;
      if (!tc_wait(&full[s], (uint32_t)((kt / kTcStages) & 1), kLimit)) {
        atomicExch(&abort_flag, 1);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int kk = 0; kk < TCK / 16; ++kk) {
        const uint64_t da = tc_desc(tc_smem(sa(s)) + kk * 32);
        const uint64_t db = tc_desc(tc_smem(sb(s)) + kk * 32);
        const uint32_t acc = (kt > 0 || kk > 0) ? 1u : 0u;
        asm volatile(
            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
            ::"r"(tmem), "l"(da), "l"(db), "r"(kTcIdesc<TN>), "r"(acc) : "memory");
      }
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
          ::"r"(tc_smem(&empty[s])) : "memory");
    }
    consumed = kt;
    // completes once every MMA issued above has (also after an abort)
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
        ::"r"(tc_smem(&done)) : "memory");
  }
  bool ok = tc_wait(&done, 0u, kLimit);
  ok = !__syncthreads_or(!ok || abort_flag);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (ok) {
    // lane = row of the accumulator; 32 columns per round go through a
    // per-warp 32 x 33 shared tile so that the storer runs with consecutive
    // lanes on consecutive columns (coalesced global writes)
    // (a warp reads the 32 accumulator rows of its number modulo four; warps w
    // and w + 4 take half of the columns each)
    const int q4 = warp & 3;
    float* tile = reinterpret_cast<float*>(base) + warp * 32 * 33;
#pragma unroll 1
    for (int c0 = (warp >> 2) * (TN / 2); c0 < (warp >> 2) * (TN / 2) + TN / 2; c0 += 32) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t r[16];
        const uint32_t taddr = tmem + ((uint32_t)(q4 * 32) << 16) + (uint32_t)(c0 + 16 * h);
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,"
            "%13,%14,%15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
              "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
              "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr)
            : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 16; ++j) tile[lane * 33 + 16 * h + j] = __uint_as_float(r[j]);
      }
      __syncwarp();
      const long long n = n0 + c0 + lane;
      // eight rows at a time: their reads first, then their stores. The residual
      // storer at 8192 x 192: 66 us a row at a time, 26.7 like this on four warps,
      // 16.3 on eight (the GELU storer at 8192 x 384: 20.9 on four, 16.1), both at 128
      // columns; 13.7 and 13.4 at 64
#pragma unroll 1
      for (int r0 = 0; r0 < 32; r0 += 8) {
        float e[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const long long m = m0 + q4 * 32 + r0 + q;
          e[q] = m < M && n < N ? st.pre(m, n) : 0.f;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const long long m = m0 + q4 * 32 + r0 + q;
          if (m < M && n < N) st.put(m, n, tile[(r0 + q) * 33 + lane], e[q]);
        }
      }
      __syncwarp();
    }
  } else {
    if (tid == 0) atomicOr(lib_status, PPF_STATUS_TIMEOUT);
    // the MMAs: `done` completes when they have; the loads issued but not
    // consumed: their stages' `full` phases
    if (tid == 0) tc_wait(&done, 0u, kLimit);
    if (warp == 0 && lane == 0)
      for (int kt = consumed; kt < issued; ++kt)
        tc_wait(&full[kt % kTcStages], (uint32_t)((kt / kTcStages) & 1), kLimit);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TN)
                 : "memory");
}

// Whether the tcgen05 kernel applies: both operands K-contiguous with rows
// on 16-byte boundaries, K a multiple of 8, enough rows to fill the GPU
// with its tiles of 128 rows.
bool tc_eligible(const StridedBf16& la, const StridedBf16& lb, long long M, long long K) {
  return la.sj == 1 && lb.si == 1 && (la.si & 7) == 0 && (lb.sj & 7) == 0 && (K & 7) == 0 &&
         (reinterpret_cast<uintptr_t>(la.x) & 15) == 0 &&
         (reinterpret_cast<uintptr_t>(lb.x) & 15) == 0 && M >= kTcMinRows;
}

template <int TN, typename ST>
int32_t tc_gemm(const StridedBf16& la, const StridedBf16& lb, ST st, long long M, long long N,
                long long K, cudaStream_t s) {
  int* status = status_ptr();
  if (!status) return fail(PPF_ERR_CUDA, "status word unavailable");
  if (M > (1LL << 31) - 1 || N > (1LL << 31) - 1 || K > (1LL << 31) - 1)
    return fail(PPF_ERR_INVALID, "GEMM too large");
  CUtensorMap ma, mb;
  int32_t rc = tensor_map_bf16_sw128(&ma, la.x, (uint64_t)K, (uint64_t)M,
                                     (uint64_t)la.si * 2, TCK, TCM);
  if (rc) return rc;
  if ((rc = tensor_map_bf16_sw128(&mb, lb.x, (uint64_t)K, (uint64_t)N, (uint64_t)lb.sj * 2, TCK,
                                  TN)))
    return rc;
  const size_t smem = (size_t)kTcStages * kTcStage<TN> + 1024;
  auto kern = tc_gemm_kernel<TN, ST>;
  PPF_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  dim3 grid((unsigned)((N + TN - 1) / TN), (unsigned)((M + TCM - 1) / TCM));
  if (grid.y > 65535) return fail(PPF_ERR_INVALID, "GEMM too large");
  PPF_TRY_CUDA(sg_launch(kern, grid, dim3(kTcThreads), smem, s, ma, mb, st, M, N, K, status));
  return PPF_OK;
}

template <typename LA, typename LB, typename ST>
int32_t gemm(LA la, LB lb, ST st, long long M, long long N, long long K, int splits,
             cudaStream_t s) {
  if (M < 1 || N < 1 || K < 1) return fail(PPF_ERR_INVALID, "empty GEMM");
  if constexpr (std::is_same<LA, StridedBf16>::value && std::is_same<LB, StridedBf16>::value) {
    if (splits <= 1 && tc_enabled() && tc_eligible(la, lb, M, K))
      return N >= 512 && N % 128 == 0 ? tc_gemm<128>(la, lb, st, M, N, K, s)
                                      : tc_gemm<64>(la, lb, st, M, N, K, s);
  }
  if (splits < 1) splits = 1;
  long long kchunk = (K + splits - 1) / splits;
  kchunk = (kchunk + BK - 1) / BK * BK;
  const long long nz = (K + kchunk - 1) / kchunk;
  dim3 grid((unsigned)((N + BN - 1) / BN), (unsigned)((M + BM - 1) / BM), (unsigned)nz);
  if (grid.y > 65535 || nz > 65535) return fail(PPF_ERR_INVALID, "GEMM too large");
  if constexpr (std::is_same<LA, StridedBf16>::value && std::is_same<LB, StridedBf16>::value) {
    if (N % 2 == 0 && st.pairs() && pipe_operand(la.x, la.si, la.sj, M, K) &&
        pipe_operand(lb.x, lb.sj, lb.si, N, K)) {
      PPF_TRY_CUDA(launch_pipe(la, lb, st, M, N, K, kchunk, grid, s));
      return PPF_OK;
    }
  }
  if constexpr (std::is_same<LA, PatchGather>::value && std::is_same<LB, StridedBf16>::value) {
    if (N % 2 == 0 && st.pairs() && gather_operand(la, K, kchunk) && lb.si == 1 &&
        pipe_operand(lb.x, lb.sj, lb.si, N, K)) {
      PPF_TRY_CUDA(sg_launch(gemm_gather_kernel<true, ST>, grid, kGemmThreads, 0, s, la, lb.x,
                             lb.sj, st, M, N, K, kchunk));
      return PPF_OK;
    }
  }
  if constexpr (std::is_same<LA, StridedBf16>::value && std::is_same<LB, PatchGatherT>::value) {
    if (N % 2 == 0 && st.pairs() && gather_operand(lb.g, N, kchunk) && la.si == 1 &&
        la.sj != 1 && pipe_operand(la.x, la.si, la.sj, M, K)) {
      PPF_TRY_CUDA(sg_launch(gemm_gather_kernel<false, ST>, grid, kGemmThreads, 0, s, lb.g, la.x,
                             la.sj, st, M, N, K, kchunk));
      return PPF_OK;
    }
  }
  PPF_TRY_CUDA(sg_launch(gemm_kernel<LA, LB, ST>, grid, kGemmThreads, 0, s, la, lb, st, M, N, K,
                         kchunk));
  return PPF_OK;
}

// ---------------------------------------------------------------- split-k
// Weight gradients are GEMMs over the token axis (k = tokens, thousands),
// split across CTAs. Each split writes its partial tile to one of two fixed
// library arrays (16 MiB each) with plain stores, and grad_tail_kernel adds the
// splits into the gradient: far fewer memory operations than one atomic per
// split and element. The arrays are shared by every call, so weight-gradient
// calls must not overlap on the GPU (the network's passes run on one stream).
constexpr long long kSplitkCap = 4LL << 20;  // floats
__device__ float g_splitk[2 * kSplitkCap];

struct StorePartial {  // part[split][m][n] = acc
  float* part;
  long long ld, zstride;
  bool pairs() const { return pair_ok(part, 4) && ld % 2 == 0 && zstride % 2 == 0; }
  __device__ float pre(long long, long long) const { return 0.f; }
  __device__ float2 pre2(long long, long long) const { return make_float2(0.f, 0.f); }
  __device__ void put(long long m, long long n, float v, float) const { (*this)(m, n, v); }
  __device__ void put2(long long m, long long n, float v, float w, float2) const {
    put_pair(part + blockIdx.z * zstride + m * ld + n, v, w);
  }
  __device__ void operator()(long long m, long long n, float v) const {
    part[blockIdx.z * zstride + m * ld + n] = v;
  }
};

// Device address of g_splitk on the current device (per device and
// context, see SymbolCache); nullptr if the lookup failed.
float* splitk_buffer() {
  static SymbolCache cache;
  void* p = nullptr;
  if (symbol_address(g_splitk, cache, &p) != PPF_OK) {
    cudaGetLastError();
    return nullptr;
  }
  return (float*)p;
}

// What is left of a weight gradient after its GEMM: y[mn] += the sum of nz splits.
struct SplitSum {
  const float* part;
  float* y;
  long long mn;
  int nz;  // 0: nothing
};
// A bias gradient: db[n] += sum_m x[m * N + n] (x NULL: of the bf16 xb).
struct ColSum {
  const float* x;
  const __nv_bfloat16* xb;
  float* db;
  long long M;
  int N;
};
constexpr int kTailThreads = 256;
constexpr int kColChunk = 32;  // rows added up by a thread before its atomic

// The split sums and column sums of up to two weight gradients in one launch:
// blocks of each job follow those of the job before (e0, e1, e2: where jobs 0 to 2
// end). Each alone is a few us of latency: at 8192 tokens, 192 and 384 channels
// a block's four were 23.2 us in four launches, 12.5 in this one (with 16 loads a
// thread in flight; 19.5 with eight).
__global__ void __launch_bounds__(kTailThreads)
    grad_tail_kernel(SplitSum s0, SplitSum s1, ColSum c0, ColSum c1, unsigned e0, unsigned e1,
                     unsigned e2) {
  pdl_wait();
  pdl_launch_next();
  unsigned blk = blockIdx.x;
  if (blk < e1) {
    const bool first = blk < e0;
    const SplitSum& s = first ? s0 : s1;
    if (!first) blk -= e0;
    const long long stride = (long long)(first ? e0 : e1 - e0) * kTailThreads;
    for (long long i = (long long)blk * kTailThreads + threadIdx.x; i < s.mn; i += stride) {
      float acc = 0.f;
#pragma unroll 16
      for (int z = 0; z < s.nz; ++z) acc += __ldg(s.part + z * s.mn + i);
      s.y[i] += acc;
    }
    return;
  }
  const bool first = blk < e2;
  const ColSum& c = first ? c0 : c1;
  const long long i = (long long)(blk - (first ? e1 : e2)) * kTailThreads + threadIdx.x;
  const long long chunk = i / c.N;
  const int n = (int)(i - chunk * c.N);
  const long long m0 = chunk * kColChunk;
  if (m0 >= c.M) return;
  const int rows = (int)(c.M - m0 < kColChunk ? c.M - m0 : kColChunk);
  float acc = 0.f;
  constexpr int NR = 16;  // rows in flight
  for (int r = 0; r < rows; r += NR) {
    float v[NR];
    if (c.x) {
#pragma unroll
      for (int q = 0; q < NR; ++q)
        v[q] = r + q < rows ? __ldg(c.x + (m0 + r + q) * c.N + n) : 0.f;
    } else {
#pragma unroll
      for (int q = 0; q < NR; ++q)
        v[q] = r + q < rows ? __bfloat162float(c.xb[(m0 + r + q) * c.N + n]) : 0.f;
    }
#pragma unroll
    for (int q = 0; q < NR; ++q) acc += v[q];
  }
  atomicAdd(c.db + n, acc);
}

// Blocks of the two jobs of one weight gradient.
inline long long tail_blocks(const SplitSum& s) {
  const long long b = s.nz ? (s.mn + kTailThreads - 1) / kTailThreads : 0;
  return b > 4096 ? 4096 : b;
}
inline long long tail_blocks(const ColSum& c) {
  const long long t = (c.M + kColChunk - 1) / kColChunk * c.N;
  return (t + kTailThreads - 1) / kTailThreads;
}

int32_t grad_tail(const SplitSum& s0, const ColSum& c0, const SplitSum& s1, const ColSum& c1,
                  cudaStream_t s) {
  const long long e0 = tail_blocks(s0), e1 = e0 + tail_blocks(s1), e2 = e1 + tail_blocks(c0),
                  e3 = e2 + tail_blocks(c1);
  if (e3 > (1LL << 31) - 1 || c0.M > 65535LL * kColChunk)
    return fail(PPF_ERR_INVALID, "size out of range");
  PPF_TRY_CUDA(sg_launch(grad_tail_kernel, (unsigned)e3, kTailThreads, 0, s, s0, s1, c0, c1,
                         (unsigned)e0, (unsigned)e1, (unsigned)e2));
  return PPF_OK;
}

// y[M x N] += A B with k = tokens (about 256 per split). What the splits leave in
// array `slot` (0 or 1) is *left, for grad_tail.
template <typename LA, typename LB>
int32_t gemm_wgrad(LA la, LB lb, float* y, long long M, long long N, long long K, int slot,
                   SplitSum* left, cudaStream_t s) {
  *left = SplitSum{nullptr, y, M * N, 0};
  long long splits = K / 256;
  const long long cap = kSplitkCap / (M * N);
  if (splits > cap) splits = cap;
  if (splits > 1024) splits = 1024;
  float* part = splits > 1 ? splitk_buffer() : nullptr;
  if (splits <= 1 || !part) return gemm(la, lb, StoreF32{y, nullptr, N, 1}, M, N, K, 1, s);
  part += slot * kSplitkCap;
  long long kchunk = (K + splits - 1) / splits;
  kchunk = (kchunk + BK - 1) / BK * BK;
  left->part = part;
  left->nz = (int)((K + kchunk - 1) / kchunk);
  return gemm(la, lb, StorePartial{part, N, M * N}, M, N, K, (int)splits, s);
}

// ---------------------------------------------------------------- others
// Depthwise 3x3 convolution over the patch grid (zero padding at each
// sample's edge): h[t, c] = bd[c] + sum w[c][dy][dx] y[(row+dy-1, col+dx-1), c].
__global__ void dwconv_fwd_kernel(const float* __restrict__ y, const float* __restrict__ w,
                                  const float* __restrict__ bd, float* __restrict__ h,
                                  __nv_bfloat16* __restrict__ hb, long long T, int C, int gh,
                                  int gw) {
  pdl_wait();
  pdl_launch_next();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T * C) return;
  const long long t = i / C;
  const int c = (int)(i - t * C);
  const int per = gh * gw;
  const int r = (int)(t % per), row = r / gw, col = r - row * gw;
  float acc = bd[c];
#pragma unroll
  for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
    for (int dx = -1; dx <= 1; ++dx) {
      const int rr = row + dy, cc = col + dx;
      if ((unsigned)rr < (unsigned)gh && (unsigned)cc < (unsigned)gw)
        acc += w[c * 9 + (dy + 1) * 3 + (dx + 1)] * y[(t + (long long)dy * gw + dx) * C + c];
    }
  h[i] = acc;
  hb[i] = __float2bfloat16(acc);
}

// dY[t, c] += sum w[c][dy][dx] dh[(row-dy+1, col-dx+1), c]
__global__ void dwconv_bwd_data_kernel(const float* __restrict__ dh, const float* __restrict__ w,
                                       float* __restrict__ dy_out, long long T, int C, int gh,
                                       int gw) {
  pdl_wait();
  pdl_launch_next();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T * C) return;
  const long long t = i / C;
  const int c = (int)(i - t * C);
  const int per = gh * gw;
  const int r = (int)(t % per), row = r / gw, col = r - row * gw;
  float acc = 0.f;
#pragma unroll
  for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
    for (int dx = -1; dx <= 1; ++dx) {
      const int rr = row - dy, cc = col - dx;
      if ((unsigned)rr < (unsigned)gh && (unsigned)cc < (unsigned)gw)
        acc += w[c * 9 + (dy + 1) * 3 + (dx + 1)] * dh[(t - (long long)dy * gw - dx) * C + c];
    }
  dy_out[i] += acc;
}

// dW[c][dy][dx] += sum_t dh[t, c] y[t + off, c];  dB[c] += sum_t dh[t, c].
// Thread = channel (consecutive threads read consecutive channels of a
// token: coalesced), CTA = a chunk of tokens; per-thread sums, then one
// atomic per (CTA, channel, tap).
__global__ void dwconv_bwd_weight_kernel(const float* __restrict__ dh, const float* __restrict__ y,
                                         float* __restrict__ dw, float* __restrict__ db,
                                         long long T, int C, int gh, int gw, long long chunk) {
  pdl_wait();
  pdl_launch_next();
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const long long t0 = (long long)blockIdx.x * chunk;
  const long long t1 = t0 + chunk < T ? t0 + chunk : T;
  const int per = gh * gw;
  float acc[10];
#pragma unroll
  for (int q = 0; q < 10; ++q) acc[q] = 0.f;
  int r = (int)(t0 % per), row = r / gw, col = r - row * gw;
#pragma unroll 4
  for (long long t = t0; t < t1; ++t) {
    const float d = dh[t * C + c];
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
      for (int dx = -1; dx <= 1; ++dx) {
        const int rr = row + dy, cc = col + dx;
        if ((unsigned)rr < (unsigned)gh && (unsigned)cc < (unsigned)gw)
          acc[(dy + 1) * 3 + (dx + 1)] += d * y[(t + (long long)dy * gw + dx) * C + c];
      }
    acc[9] += d;
    if (++col == gw) {  // next token: (row, col) of the patch grid
      col = 0;
      if (++row == gh) row = 0;
    }
  }
#pragma unroll
  for (int q = 0; q < 9; ++q) atomicAdd(dw + c * 9 + q, acc[q]);
  atomicAdd(db + c, acc[9]);
}

// Two channels of kDwTokens tokens in a row per thread (C even, 8-byte aligned rows):
// a segment's tokens take 18 loads of y instead of 36, and the weights one per
// CTA, tap by tap in shared memory (in memory a channel's nine taps are together, and
// a warp's reads of them cost more than its tokens). The same sums in the same order.
// DATA: dy = dy_in + the transposed convolution of x (dwconv_bwd_data_kernel) and,
// with outb, its bf16 copy; else h = the convolution of x and its bf16 copy
// (dwconv_fwd_kernel). Bound: L2 traffic and latency; 8192 x 192, us: 16.2 ->
// 9.8, the gradient 16.1 and a copy of dy -> 10.4.
constexpr int kDwTokens = 4;
constexpr int kDwMaxC = 1344;  // 9 C floats of shared memory
template <bool DATA>
__global__ void __launch_bounds__(256)
    dwconv2_kernel(const float* __restrict__ x, const float* __restrict__ w,
                   const float* __restrict__ bd, const float* dy_in, float* out,
                   __nv_bfloat16* __restrict__ outb, long long n, int C, int gh, int gw) {
  pdl_wait();
  pdl_launch_next();
  extern __shared__ float wt[];  // [tap][channel]
  const int c2 = C / 2, segs = (gw + kDwTokens - 1) / kDwTokens;
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  const long long s = i / c2;  // segment
  const int c = (int)(i - s * c2) * 2;
  const long long line = s / segs;  // row of a sample
  const int col = (int)(s - line * segs) * kDwTokens, row = (int)(line % gh);
  const long long t = line * gw + col;
  const bool live = i < n;
  float2 v[3][kDwTokens + 2];
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int q = 0; q < kDwTokens + 2; ++q) {
      const bool in = live && (unsigned)(row + j - 1) < (unsigned)gh &&
                      (unsigned)(col + q - 1) < (unsigned)gw;
      v[j][q] = in ? __ldg(reinterpret_cast<const float2*>(
                         x + (t + (long long)(j - 1) * gw + q - 1) * C + c))
                   : make_float2(0.f, 0.f);
    }
  for (int k = threadIdx.x; k < 9 * C; k += 256) wt[k % 9 * C + k / 9] = __ldg(w + k);
  __syncthreads();
  if (!live) return;
  float2 acc[kDwTokens];
  const float2 b0 = DATA ? make_float2(0.f, 0.f) : *reinterpret_cast<const float2*>(bd + c);
#pragma unroll
  for (int q = 0; q < kDwTokens; ++q) acc[q] = b0;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int j = DATA ? 2 - k / 3 : k / 3, d = DATA ? 2 - k % 3 : k % 3;
    const float2 wk = *reinterpret_cast<const float2*>(wt + k * C + c);
    if ((unsigned)(row + j - 1) < (unsigned)gh) {
#pragma unroll
      for (int q = 0; q < kDwTokens; ++q)
        if ((unsigned)(col + q + d - 1) < (unsigned)gw) {
          acc[q].x += wk.x * v[j][q + d].x;
          acc[q].y += wk.y * v[j][q + d].y;
        }
    }
  }
  float2 base[kDwTokens];
  if (DATA) {  // dy may be dy_in: read before any is stored
#pragma unroll
    for (int q = 0; q < kDwTokens; ++q)
      if (col + q < gw) base[q] = *reinterpret_cast<const float2*>(dy_in + (t + q) * C + c);
  }
#pragma unroll
  for (int q = 0; q < kDwTokens; ++q)
    if (col + q < gw) {
      const long long o = (t + q) * C + c;
      if (DATA) acc[q] = make_float2(base[q].x + acc[q].x, base[q].y + acc[q].y);
      put_pair(out + o, acc[q].x, acc[q].y);
      if (!DATA || outb) put_pair(outb + o, acc[q].x, acc[q].y);
    }
}

// Depthwise weight and bias gradients, two channels per lane and a row of the
// patch grid per warp: the 3 x 3 window of y moves along the row in registers
// (three loads a token instead of nine), kDwRows rows are added up in shared
// memory, and one atomic per CTA, channel and tap remains. The loads of eight tokens
// are in flight together. 8192 x 192: 51.8 us -> 12.0 (20.9 a token at a time).
constexpr int kDwRows = 4;
__global__ void __launch_bounds__(32 * kDwRows)
    dwconv2_bwd_weight_kernel(const float* __restrict__ dh, const float* __restrict__ y,
                              float* __restrict__ dw, float* __restrict__ db, long long nrows,
                              int C, int gh, int gw) {
  pdl_wait();
  pdl_launch_next();
  __shared__ float2 part[kDwRows][10][32];
  const int lane = threadIdx.x, wid = threadIdx.y;
  const int c = blockIdx.y * 64 + 2 * lane;
  const long long pr = (long long)blockIdx.x * kDwRows + wid;  // (sample, patch row)
  float2 acc[10];
#pragma unroll
  for (int q = 0; q < 10; ++q) acc[q] = make_float2(0.f, 0.f);
  if (pr < nrows && c < C) {
    const int row = (int)(pr % gh);
    const long long t0 = pr * gw;
    const float2 zero = make_float2(0.f, 0.f);
    auto at = [&](int j, int col) {  // y of row `row + j - 1`, column col
      return (unsigned)(row + j - 1) < (unsigned)gh && col < gw
                 ? __ldg(reinterpret_cast<const float2*>(
                       y + (t0 + (long long)(j - 1) * gw + col) * C + c))
                 : zero;
    };
    float2 left[3], mid[3];  // columns col - 1 and col
#pragma unroll
    for (int j = 0; j < 3; ++j) left[j] = zero, mid[j] = at(j, 0);
    constexpr int NT = 8;  // tokens whose loads are in flight together
    for (int c0 = 0; c0 < gw; c0 += NT) {
      float2 d[NT], next[3][NT];
#pragma unroll
      for (int q = 0; q < NT; ++q) {
        d[q] = c0 + q < gw ? __ldg(reinterpret_cast<const float2*>(dh + (t0 + c0 + q) * C + c))
                           : zero;
#pragma unroll
        for (int j = 0; j < 3; ++j) next[j][q] = at(j, c0 + q + 1);
      }
#pragma unroll
      for (int q = 0; q < NT; ++q) {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const float2 win[3] = {left[j], mid[j], next[j][q]};
#pragma unroll
          for (int p = 0; p < 3; ++p) {
            acc[3 * j + p].x = fmaf(d[q].x, win[p].x, acc[3 * j + p].x);
            acc[3 * j + p].y = fmaf(d[q].y, win[p].y, acc[3 * j + p].y);
          }
          left[j] = mid[j];
          mid[j] = next[j][q];
        }
        acc[9].x += d[q].x;
        acc[9].y += d[q].y;
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 10; ++q) part[wid][q][lane] = acc[q];
  __syncthreads();
  if (c >= C) return;
  for (int q = wid; q < 10; q += kDwRows) {
    float2 v = part[0][q][lane];
    for (int r = 1; r < kDwRows; ++r) {
      v.x += part[r][q][lane].x;
      v.y += part[r][q][lane].y;
    }
    float* p = q < 9 ? dw + c * 9 + q : db + c;
    atomicAdd(p, v.x);
    atomicAdd(p + (q < 9 ? 9 : 1), v.y);
  }
}

// Loss on the network output out[t, (ch, py, px)] against the normalised
// target change: d = out - (new - old) * scale[ch]; loss += d^2 / count;
// grad (bf16) = 2 d / count.
//
// V consecutive elements per thread (4: P and the pitch multiples of 4, whole 16-byte
// vectors; else 1). The loss: each 32 elements in float, in the order of a warp's
// xor tree over them, then in double. A CTA adds up its elements and issues one
// atomic: one per 256 elements, all on one address, was the bound. 8 x 512 x 512,
// us: 42.5 -> 15.8.
constexpr int kMseThreads = 256;
template <int V>
__global__ void __launch_bounds__(kMseThreads)
    mse_kernel(const float* __restrict__ out, const float* __restrict__ f_old,
               const float* __restrict__ f_new, __nv_bfloat16* __restrict__ grad,
               double* __restrict__ loss, long long T, int P, int H, int pitch, int gh, int gw,
               float s0, float s1, float inv_count) {
  pdl_wait();
  pdl_launch_next();
  const int K = 2 * P * P;
  const long long n = T * K, stride = (long long)gridDim.x * kMseThreads * V;
  double sum = 0.0;
  for (long long base = (long long)blockIdx.x * kMseThreads * V; base < n; base += stride) {
    const long long i = base + threadIdx.x * V;
    float v[V];
#pragma unroll
    for (int e = 0; e < V; ++e) v[e] = 0.f;
    if (i < n) {  // (n and K are multiples of V)
      const long long t = i / K;
      const int k = (int)(i - t * K);
      const int per = gh * gw;
      const int b = (int)(t / per), r = (int)(t - (long long)b * per);
      const int ty = r / gw, tx = r - ty * gw;
      const int ch = k / (P * P), q = k - ch * P * P, py = q / P, px = q - py * P;
      const long long o = (((long long)b * 2 + ch) * H + ty * P + py) * pitch + tx * P + px;
      const float sc = ch == 0 ? s0 : s1;
      float a[V], x[V], y[V], d[V];
      if (V == 4) {
        *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(out + i);
        *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(f_new + o);
        *reinterpret_cast<float4*>(y) = *reinterpret_cast<const float4*>(f_old + o);
      } else {
        a[0] = out[i], x[0] = f_new[o], y[0] = f_old[o];
      }
#pragma unroll
      for (int e = 0; e < V; ++e) {
        d[e] = a[e] - (x[e] - y[e]) * sc;
        v[e] = d[e] * d[e] * inv_count;
      }
      if (V == 4) {
        put_pair(grad + i, 2.f * d[0] * inv_count, 2.f * d[1] * inv_count);
        put_pair(grad + i + 2, 2.f * d[V - 2] * inv_count, 2.f * d[V - 1] * inv_count);
      } else {
        grad[i] = __float2bfloat16(2.f * d[0] * inv_count);
      }
    }
#pragma unroll
    for (int o = 16 / V; o > 0; o >>= 1)
#pragma unroll
      for (int e = 0; e < V; ++e) v[e] += __shfl_xor_sync(0xffffffffu, v[e], o);
    sum += V == 4 ? (v[0] + v[V / 2]) + (v[V / 4] + v[V - 1]) : v[0];
  }
  // every lane of a group of 32 / V holds the group's sum
  if (threadIdx.x & (32 / V - 1)) sum = 0.0;
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  __shared__ double part[kMseThreads / 32];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kMseThreads / 32; ++w) sum += part[w];
    if (sum != 0.0) atomicAdd(loss, sum);
  }
}

// new = old + out / scale[ch] (the surrogate's k-step prediction), fields
// [b][ch][H][pitch], out [token][(ch, py, px)].
__global__ void apply_kernel(const float* __restrict__ out, const float* __restrict__ f_old,
                             float* __restrict__ f_new, long long T, int P, int H, int pitch,
                             int gh, int gw, float inv_s0, float inv_s1, float lo0, float hi0,
                             float lo1, float hi1) {
  pdl_wait();
  pdl_launch_next();
  const int K = 2 * P * P;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T * K) return;
  const long long t = i / K;
  const int k = (int)(i - t * K);
  const int per = gh * gw;
  const int b = (int)(t / per), r = (int)(t - (long long)b * per);
  const int ty = r / gw, tx = r - ty * gw;
  const int ch = k / (P * P), q = k - ch * P * P, py = q / P, px = q - py * P;
  const long long o = (((long long)b * 2 + ch) * H + ty * P + py) * pitch + tx * P + px;
  const float v = f_old[o] + out[i] * (ch == 0 ? inv_s0 : inv_s1);
  const float lo = ch == 0 ? lo0 : lo1, hi = ch == 0 ? hi0 : hi1;
  f_new[o] = v < lo ? lo : (v > hi ? hi : v);  // a NaN stays NaN for the check to see
}

// Adam (bias-corrected) on fp32 master weights; refreshes the bf16 copy.
__global__ void adam_kernel(float* __restrict__ w, __nv_bfloat16* __restrict__ wb,
                            const float* __restrict__ g, float* __restrict__ m1,
                            float* __restrict__ m2, long long n, float lr, float b1, float b2,
                            float eps, float c1, float c2, float wd) {
  pdl_wait();
  pdl_launch_next();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float a = b1 * m1[i] + (1.f - b1) * gi;
  const float v = b2 * m2[i] + (1.f - b2) * gi * gi;
  m1[i] = a;
  m2[i] = v;
  const float upd = (a / c1) / (sqrtf(v / c2) + eps) + wd * w[i];
  const float nw = w[i] - lr * upd;
  w[i] = nw;
  if (wb) wb[i] = __float2bfloat16(nw);
}

__global__ void cast_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ y,
                            long long n) {
  pdl_wait();
  pdl_launch_next();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = __float2bfloat16(x[i]);
}

// Window check of a k-step prediction p from state u, given s = one stencil
// step from p. Per sample b (fields [b][ch][H][pitch], phi = channel 0):
//   out[3b]   += sum over phi cells of (k (s - p) - (p - u))^2
//   out[3b+1] += sum over phi cells of p^2
//   out[3b+2] += number of cells where p or s holds a non-finite value
__global__ void residual_kernel(const float* __restrict__ u, const float* __restrict__ p,
                                const float* __restrict__ sp, int H, int W, int pitch, float k,
                                double* __restrict__ out) {
  pdl_wait();
  pdl_launch_next();
  const int b = blockIdx.y;
  const long long plane = (long long)H * pitch;
  const float* u0 = u + (long long)b * 2 * plane;
  const float* p0 = p + (long long)b * 2 * plane;
  const float* s0 = sp + (long long)b * 2 * plane;
  double num = 0.0, den = 0.0, bad = 0.0;
  const long long n = (long long)H * W;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const long long row = i / W;
    const long long o = row * pitch + (i - row * W);
    const float pv = p0[o], pc = p0[plane + o], sv = s0[o], sc = s0[plane + o];
    const float r = k * (sv - pv) - (pv - u0[o]);
    num += (double)r * r;
    den += (double)pv * pv;
    bad += (isfinite(pv) && isfinite(pc) && isfinite(sv) && isfinite(sc)) ? 0.0 : 1.0;
  }
  for (int off = 16; off > 0; off >>= 1) {
    num += __shfl_xor_sync(0xffffffffu, num, off);
    den += __shfl_xor_sync(0xffffffffu, den, off);
    bad += __shfl_xor_sync(0xffffffffu, bad, off);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(out + 3 * b, num);
    atomicAdd(out + 3 * b + 1, den);
    if (bad != 0.0) atomicAdd(out + 3 * b + 2, bad);
  }
}

// Channels in whole vectors of `n` floats (or halves), 16-byte aligned rows.
bool dw_vec(int C, int n, std::initializer_list<const void*> ptrs) {
  for (const void* p : ptrs)
    if ((uintptr_t)p & 15) return false;
  return C % n == 0;
}

// Whether dwconv2_kernel applies (bf16 may be NULL), and its threads.
bool dw_two(const PpfSgShape* s, std::initializer_list<const void*> ptrs, const void* bf16) {
  for (const void* p : ptrs)
    if ((uintptr_t)p & 7) return false;
  return s->C % 2 == 0 && s->C <= kDwMaxC && pair_ok(bf16, 2);
}
long long dw_threads(const PpfSgShape* s) {
  const int gh = s->H / s->P, gw = s->W / s->P;
  return (long long)s->B * gh * ((gw + kDwTokens - 1) / kDwTokens) * (s->C / 2);
}

int32_t grid1d(long long n, unsigned* blocks) {
  const long long b = (n + 255) / 256;
  if (b < 1 || b > (1LL << 31) - 1) return fail(PPF_ERR_INVALID, "size out of range");
  *blocks = (unsigned)b;
  return PPF_OK;
}

}  // namespace
}  // namespace ppf

using namespace ppf;

extern "C" {

// C[M, N] = A[M, K] B[K, N] with bf16 operands given by element strides
// (A(m, k) = a[m*sam + k*sak], B(k, n) = b[k*sbk + n*sbn]) and fp32 result
// y[m*ldy + n] (= or += when accumulate) + bias[n]. splits > 1 splits k
// over CTAs and requires accumulate (atomic adds).
int32_t ppf_sg_gemm(const void* a, long long sam, long long sak, const void* b, long long sbk,
                    long long sbn, float* y, long long ldy, const float* bias, int32_t accumulate,
                    long long M, long long N, long long K, int32_t splits, void* stream) {
  clear_error();
  if (!a || !b || !y) return fail(PPF_ERR_INVALID, "NULL operand");
  StridedBf16 la{(const __nv_bfloat16*)a, sam, sak};
  StridedBf16 lb{(const __nv_bfloat16*)b, sbk, sbn};
  if (splits > 1) {
    if (!accumulate || bias) return fail(PPF_ERR_INVALID, "split-k needs accumulate, no bias");
    return gemm(la, lb, StoreAtomic{y, ldy}, M, N, K, splits, (cudaStream_t)stream);
  }
  return gemm(la, lb, StoreF32{y, bias, ldy, accumulate}, M, N, K, 1, (cudaStream_t)stream);
}

}  // extern "C"

// Network-level entry points (used by pyphasefield_gb300/surrogate.py);
// PpfSgShape is declared in ppf_gb300.h.
extern "C" {

static int32_t sg_check(const PpfSgShape* s) {
  if (!s) return fail(PPF_ERR_INVALID, "shape is NULL");
  if (s->B < 1 || s->P < 1 || s->H % s->P || s->W % s->P || s->pitch < s->W || s->C < 1 ||
      s->E < 1)
    return fail(PPF_ERR_INVALID, "bad surrogate shape");
  return PPF_OK;
}

// Patch embedding: y = patches(fields) Win^T + b, with fp32 and bf16 copies.
int32_t ppf_sg_patch_fwd(const PpfSgShape* s, const float* fields, const void* w_in_bf16,
                         const float* b_in, float* y, void* y_bf16, void* stream) {
  clear_error();
  int32_t rc = sg_check(s);
  if (rc) return rc;
  const int gh = s->H / s->P, gw = s->W / s->P;
  const long long T = (long long)s->B * gh * gw, K = 2LL * s->P * s->P;
  PatchGather la{fields, s->P, s->H, s->W, s->pitch, gh, gw, s->in_off0, s->in_sc0,
                 s->in_off1, s->in_sc1};
  StridedBf16 lb{(const __nv_bfloat16*)w_in_bf16, 1, K};
  return gemm(la, lb, StoreBf16Pair{y, (__nv_bfloat16*)y_bf16, b_in, s->C}, T, s->C, K, 1,
              (cudaStream_t)stream);
}

// dWin += dy^T patches(fields) (split-k over tokens), db_in += column sums
// of dy.
int32_t ppf_sg_patch_bwd_weight(const PpfSgShape* s, const float* fields, const void* dy_bf16,
                                float* dw_in, float* db_in, void* stream) {
  clear_error();
  int32_t rc = sg_check(s);
  if (rc) return rc;
  const int gh = s->H / s->P, gw = s->W / s->P;
  const long long T = (long long)s->B * gh * gw, K = 2LL * s->P * s->P;
  StridedBf16 la{(const __nv_bfloat16*)dy_bf16, 1, s->C};  // A(m = out ch, k = token)
  PatchGatherT lb{{fields, s->P, s->H, s->W, s->pitch, gh, gw, s->in_off0, s->in_sc0,
                   s->in_off1, s->in_sc1}};
  cudaStream_t st = (cudaStream_t)stream;
  SplitSum left;
  if ((rc = gemm_wgrad(la, lb, dw_in, s->C, K, T, 0, &left, st))) return rc;
  return grad_tail(left, ColSum{nullptr, (const __nv_bfloat16*)dy_bf16, db_in, T, s->C},
                   SplitSum{}, ColSum{}, st);
}

// Depthwise conv + pointwise expand + GELU: h = dw(y), pre = h W1^T + b1,
// act = gelu(pre) (bf16).
int32_t ppf_sg_block_fwd(const PpfSgShape* s, const float* y, const float* w_dw, const float* b_dw,
                         float* h, void* h_bf16, const void* w1_bf16, const float* b1, float* pre,
                         void* act_bf16, const void* w2_bf16, const float* b2, float* y_out,
                         void* y_out_bf16, void* stream) {
  clear_error();
  int32_t rc = sg_check(s);
  if (rc) return rc;
  const int gh = s->H / s->P, gw = s->W / s->P;
  const long long T = (long long)s->B * gh * gw;
  cudaStream_t st = (cudaStream_t)stream;
  unsigned blocks;
  const bool two = dw_two(s, {y, b_dw, h}, h_bf16);
  if ((rc = grid1d(two ? dw_threads(s) : T * s->C, &blocks))) return rc;
  if (two)
    PPF_TRY_CUDA(sg_launch(dwconv2_kernel<false>, blocks, 256, 9 * s->C * sizeof(float), st, y,
                           w_dw, b_dw, nullptr, h, (__nv_bfloat16*)h_bf16, dw_threads(s), s->C,
                           gh, gw));
  else
    PPF_TRY_CUDA(sg_launch(dwconv_fwd_kernel, blocks, 256, 0, st, y, w_dw, b_dw, h,
                           (__nv_bfloat16*)h_bf16, T, s->C, gh, gw));
  StridedBf16 ha{(const __nv_bfloat16*)h_bf16, s->C, 1};
  StridedBf16 w1{(const __nv_bfloat16*)w1_bf16, 1, s->C};  // B(k=c, n=e) = W1[e][c]
  if ((rc = gemm(ha, w1, StoreGelu{pre, (__nv_bfloat16*)act_bf16, b1, s->E}, T, s->E, s->C, 1,
                 st)))
    return rc;
  StridedBf16 aa{(const __nv_bfloat16*)act_bf16, s->E, 1};
  StridedBf16 w2{(const __nv_bfloat16*)w2_bf16, 1, s->E};  // B(k=e, n=c) = W2[c][e]
  // y_out = y + act W2^T + b2 (y_out may alias y)
  return gemm(aa, w2, StoreResidual{y, y_out, (__nv_bfloat16*)y_out_bf16, b2, s->C}, T, s->C,
              s->E, 1, st);
}

// Backward of ppf_sg_block_fwd given dy_out (fp32, also bf16 copy):
// dW2, db2, dW1, db1, dWdw, dbdw accumulate; dy (fp32) = dy_out + dwconv^T(dh), and its
// bf16 copy where dy_bf16 is not NULL (dy_bf16 may be dy_out_bf16).
int32_t ppf_sg_block_bwd_pair(const PpfSgShape* s, const float* y, const void* h_bf16,
                              const float* pre, const void* act_bf16, const void* w1_bf16,
                              const void* w2_bf16, const float* w_dw, const float* dy_out,
                              const void* dy_out_bf16, void* dpre_bf16, float* dh,
                              void* dh_bf16, float* dy, void* dy_bf16, float* dw1, float* db1,
                              float* dw2, float* db2, float* dw_dw, float* db_dw,
                              void* stream) {
  clear_error();
  int32_t rc = sg_check(s);
  if (rc) return rc;
  const int gh = s->H / s->P, gw = s->W / s->P;
  const long long T = (long long)s->B * gh * gw;
  cudaStream_t st = (cudaStream_t)stream;
  // dW2[c][e] += sum_t dy_out[t][c] act[t][e]
  StridedBf16 dyT{(const __nv_bfloat16*)dy_out_bf16, 1, s->C};
  StridedBf16 act{(const __nv_bfloat16*)act_bf16, s->E, 1};
  SplitSum left2, left1;
  if ((rc = gemm_wgrad(dyT, act, dw2, s->C, s->E, T, 0, &left2, st))) return rc;
  // d_act = dy_out W2 ; d_pre = d_act * gelu'(pre)
  StridedBf16 dyA{(const __nv_bfloat16*)dy_out_bf16, s->C, 1};
  StridedBf16 w2{(const __nv_bfloat16*)w2_bf16, s->E, 1};  // B(k=c, n=e) = W2[c][e]
  if ((rc = gemm(dyA, w2, StoreGeluGrad{pre, (__nv_bfloat16*)dpre_bf16, s->E}, T, s->E, s->C, 1,
                 st)))
    return rc;
  // dW1[e][c] += sum_t dpre[t][e] h[t][c], and both bias gradients
  StridedBf16 dpT{(const __nv_bfloat16*)dpre_bf16, 1, s->E};
  StridedBf16 hh{(const __nv_bfloat16*)h_bf16, s->C, 1};
  if ((rc = gemm_wgrad(dpT, hh, dw1, s->E, s->C, T, 1, &left1, st))) return rc;
  if ((rc = grad_tail(left2, ColSum{dy_out, nullptr, db2, T, s->C}, left1,
                      ColSum{nullptr, (const __nv_bfloat16*)dpre_bf16, db1, T, s->E}, st)))
    return rc;
  // dh = dpre W1
  StridedBf16 dpA{(const __nv_bfloat16*)dpre_bf16, s->E, 1};
  StridedBf16 w1{(const __nv_bfloat16*)w1_bf16, s->C, 1};  // B(k=e, n=c) = W1[e][c]
  if ((rc = gemm(dpA, w1, StoreBf16Pair{dh, (__nv_bfloat16*)dh_bf16, nullptr, s->C}, T, s->C,
                 s->E, 1, st)))
    return rc;
  // depthwise: weight/bias grads, then dy = dy_out + dwconv^T(dh)
  if (dw_vec(s->C, 2, {dh, y})) {
    const long long nrows = (long long)s->B * gh;
    dim3 wg((unsigned)((nrows + kDwRows - 1) / kDwRows), (unsigned)((s->C + 63) / 64));
    PPF_TRY_CUDA(sg_launch(dwconv2_bwd_weight_kernel, wg, dim3(32, kDwRows), 0, st, dh, y, dw_dw,
                           db_dw, nrows, s->C, gh, gw));
  } else {
    const long long wchunk = 32;
    dim3 wg((unsigned)((T + wchunk - 1) / wchunk), (unsigned)((s->C + 127) / 128));
    PPF_TRY_CUDA(sg_launch(dwconv_bwd_weight_kernel, wg, 128, 0, st, dh, y, dw_dw, db_dw, T, s->C,
                           gh, gw, wchunk));
  }
  const bool two = dw_two(s, {dh, dy, dy_out}, dy_bf16);
  unsigned blocks;
  if ((rc = grid1d(two ? dw_threads(s) : T * s->C, &blocks))) return rc;
  if (two) {
    PPF_TRY_CUDA(sg_launch(dwconv2_kernel<true>, blocks, 256, 9 * s->C * sizeof(float), st, dh,
                           w_dw, nullptr, dy_out, dy, (__nv_bfloat16*)dy_bf16, dw_threads(s),
                           s->C, gh, gw));
  } else {
    if (dy != dy_out)
      PPF_TRY_CUDA(cudaMemcpyAsync(dy, dy_out, T * s->C * sizeof(float), cudaMemcpyDeviceToDevice,
                                   st));
    PPF_TRY_CUDA(sg_launch(dwconv_bwd_data_kernel, blocks, 256, 0, st, dh, w_dw, dy, T, s->C, gh,
                           gw));
    if (dy_bf16)
      PPF_TRY_CUDA(sg_launch(cast_kernel, blocks, 256, 0, st, dy, (__nv_bfloat16*)dy_bf16,
                             T * s->C));
  }
  return PPF_OK;
}

int32_t ppf_sg_block_bwd(const PpfSgShape* s, const float* y, const void* h_bf16,
                         const float* pre, const void* act_bf16, const void* w1_bf16,
                         const void* w2_bf16, const float* w_dw, const float* dy_out,
                         const void* dy_out_bf16, void* dpre_bf16, float* dh, void* dh_bf16,
                         float* dy, float* dw1, float* db1, float* dw2, float* db2, float* dw_dw,
                         float* db_dw, void* stream) {
  return ppf_sg_block_bwd_pair(s, y, h_bf16, pre, act_bf16, w1_bf16, w2_bf16, w_dw, dy_out,
                               dy_out_bf16, dpre_bf16, dh, dh_bf16, dy, nullptr, dw1, db1, dw2,
                               db2, dw_dw, db_dw, stream);
}

// Output head: out = y Wout^T + bout, out [token][2 P P].
int32_t ppf_sg_head_fwd(const PpfSgShape* s, const void* y_bf16, const void* w_out_bf16,
                        const float* b_out, float* out, void* stream) {
  clear_error();
  int32_t rc = sg_check(s);
  if (rc) return rc;
  const int gh = s->H / s->P, gw = s->W / s->P;
  const long long T = (long long)s->B * gh * gw, K = 2LL * s->P * s->P;
  StridedBf16 la{(const __nv_bfloat16*)y_bf16, s->C, 1};
  StridedBf16 lb{(const __nv_bfloat16*)w_out_bf16, 1, s->C};  // B(k=c, n=o) = Wout[o][c]
  return gemm(la, lb, StoreF32{out, b_out, K, 0}, T, K, s->C, 1, (cudaStream_t)stream);
}

// Head backward: dWout += dout^T y, dbout, dy = dout Wout (fp32 and bf16).
int32_t ppf_sg_head_bwd(const PpfSgShape* s, const void* y_bf16, const void* w_out_bf16,
                        const void* dout_bf16, float* dw_out, float* db_out, float* dy,
                        void* dy_bf16, void* stream) {
  clear_error();
  int32_t rc = sg_check(s);
  if (rc) return rc;
  const int gh = s->H / s->P, gw = s->W / s->P;
  const long long T = (long long)s->B * gh * gw, K = 2LL * s->P * s->P;
  cudaStream_t st = (cudaStream_t)stream;
  StridedBf16 doT{(const __nv_bfloat16*)dout_bf16, 1, K};
  StridedBf16 yy{(const __nv_bfloat16*)y_bf16, s->C, 1};
  SplitSum left;
  if ((rc = gemm_wgrad(doT, yy, dw_out, K, s->C, T, 0, &left, st))) return rc;
  if ((rc = grad_tail(left, ColSum{nullptr, (const __nv_bfloat16*)dout_bf16, db_out, T, (int)K},
                      SplitSum{}, ColSum{}, st)))
    return rc;
  StridedBf16 doA{(const __nv_bfloat16*)dout_bf16, K, 1};
  StridedBf16 w{(const __nv_bfloat16*)w_out_bf16, s->C, 1};  // B(k=o, n=c) = Wout[o][c]
  return gemm(doA, w, StoreBf16Pair{dy, (__nv_bfloat16*)dy_bf16, nullptr, s->C}, T, s->C, K, 1,
              st);
}

int32_t ppf_sg_mse(const PpfSgShape* s, const float* out, const float* f_old, const float* f_new,
                   void* grad_bf16, double* loss, void* stream) {
  clear_error();
  int32_t rc = sg_check(s);
  if (rc) return rc;
  const int gh = s->H / s->P, gw = s->W / s->P;
  const long long T = (long long)s->B * gh * gw, K = 2LL * s->P * s->P;
  unsigned blocks;
  if ((rc = grid1d(T * K, &blocks))) return rc;
  const bool four = dw_vec(s->P, 4, {out, f_old, f_new}) && s->pitch % 4 == 0 &&
                    pair_ok(grad_bf16, 2);
  const long long per = kMseThreads * (four ? 4 : 1), need = (T * K + per - 1) / per;
  const unsigned grid = (unsigned)(need < 1216 ? need : 1216);  // 8 CTAs per SM over 152 SMs
  auto kern = four ? mse_kernel<4> : mse_kernel<1>;
  PPF_TRY_CUDA(sg_launch(kern, grid, kMseThreads, 0, (cudaStream_t)stream, out, f_old, f_new,
                         (__nv_bfloat16*)grad_bf16, loss, T, s->P, s->H, s->pitch, gh, gw, s->s0,
                         s->s1, 1.0f / (float)(T * K)));
  return PPF_OK;
}

int32_t ppf_sg_apply(const PpfSgShape* s, const float* out, const float* f_old, float* f_new,
                     void* stream) {
  clear_error();
  int32_t rc = sg_check(s);
  if (rc) return rc;
  const int gh = s->H / s->P, gw = s->W / s->P;
  const long long T = (long long)s->B * gh * gw, K = 2LL * s->P * s->P;
  unsigned blocks;
  if ((rc = grid1d(T * K, &blocks))) return rc;
  PPF_TRY_CUDA(sg_launch(apply_kernel, blocks, 256, 0, (cudaStream_t)stream, out, f_old, f_new, T,
                         s->P, s->H, s->pitch, gh, gw, 1.0f / s->s0, 1.0f / s->s1, s->lo0,
                         s->hi0, s->lo1, s->hi1));
  return PPF_OK;
}

// out[3 B] is overwritten.
int32_t ppf_sg_residual(const PpfSgShape* s, const float* u, const float* pred,
                        const float* stepped, int32_t k, double* out, void* stream) {
  clear_error();
  int32_t rc = sg_check(s);
  if (rc) return rc;
  if (!u || !pred || !stepped || !out || k < 1) return fail(PPF_ERR_INVALID, "bad residual args");
  const long long n = (long long)s->H * s->W;
  long long bx = (n + 255) / 256;
  if (bx > 1216) bx = 1216;  // 8 CTAs of 256 per SM over 152 SMs
  dim3 grid((unsigned)bx, (unsigned)s->B);
  PPF_TRY_CUDA(cudaMemsetAsync(out, 0, sizeof(double) * 3 * s->B, (cudaStream_t)stream));
  PPF_TRY_CUDA(sg_launch(residual_kernel, grid, 256, 0, (cudaStream_t)stream, u, pred, stepped,
                         s->H, s->W, s->pitch, (float)k, out));
  return PPF_OK;
}

// 1: GEMMs with K-contiguous operands run on tcgen05 (default); 0: mma.sync.
int32_t ppf_sg_set_tensor_path(int32_t tcgen05) {
  clear_error();
  g_tc_enabled = tcgen05 ? 1 : 0;
  return PPF_OK;
}

int32_t ppf_sg_cast_bf16(const float* x, void* y, long long n, void* stream) {
  clear_error();
  if (!x || !y) return fail(PPF_ERR_INVALID, "NULL pointer");
  unsigned blocks;
  int32_t rc = grid1d(n, &blocks);
  if (rc) return rc;
  PPF_TRY_CUDA(sg_launch(cast_kernel, blocks, 256, 0, (cudaStream_t)stream, x, (__nv_bfloat16*)y,
                         n));
  return PPF_OK;
}

int32_t ppf_sg_adam(float* w, void* w_bf16, const float* g, float* m1, float* m2, long long n,
                    float lr, float b1, float b2, float eps, int32_t step, float weight_decay,
                    void* stream) {
  clear_error();
  if (!w || !g || !m1 || !m2 || step < 1) return fail(PPF_ERR_INVALID, "bad Adam arguments");
  unsigned blocks;
  int32_t rc = grid1d(n, &blocks);
  if (rc) return rc;
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  PPF_TRY_CUDA(sg_launch(adam_kernel, blocks, 256, 0, (cudaStream_t)stream, w,
                         (__nv_bfloat16*)w_bf16, g, m1, m2, n, lr, b1, b2, eps, c1, c2,
                         weight_decay));
  return PPF_OK;
}

}  // extern "C"
