// Two-step column transforms of the Cartesian operator (yfull.cuh), device code.
//
// H = N1 N2, y = j + N2 i, kappa = (ky - sy) mod H = k1 + N1 k2: thread
// (tx, j) transforms its N1 values, the twiddled results change hands through
// shared memory, and thread (tx, k1) transforms N2 of them; of the results
// only the sampled rows are stored, and the adjoint reads only those (the next
// coil's ahead of the barrier).  A column costs the same whatever the number
// of sampled rows, which beats the class sums of yfft.cu from about 2.5 N1
// rows on while the second step is short: 160 x 128 (16 x 8), 24 frames, 12
// coils, 64 rows 27 + 42 us with the class sums, 23 + 22 here; 160 x 160 (16 x
// 10), 40 rows 25 + 33 and 24 + 23; at the line 128 x 112 (14 x 8), 37 rows
// 24 + 31 and 25 + 25, 200 x 200 (20 x 10), 67 rows 39 + 58 and 51 + 46.  With a longer second step the registers
// of the two (128 to 166 a thread) leave too few warps: 192 x 192 (16 x 12),
// 48 rows 43 + 56 and 54 + 65; 320 x 320 (20 x 16), 53 rows 321 + 435 and 525
// + 509.
#pragma once

#include "regfft.cuh"
#include "yfull.cuh"

namespace avx {

template <int N1, int N2>
struct ColSplit {
  static constexpr int H = N1 * N2, XT = 8, JP = (N1 + 1) * XT, E = (N1 + 1) / 2 * 2;
  static constexpr int NW = (XT * N2 + 31) / 32;  // warps that hold image values (and maps)
  static constexpr int NT = (XT * N1 + 31) / 32 * 32;
};

template <int N1, int N2>
AVX_D void col_twiddles(float2* tw, const float2* __restrict__ w) {
  for (int e = threadIdx.x; e < N1 * N2; e += blockDim.x) {
    const int k1 = e / N2, j = e - k1 * N2;
    tw[e] = w[k1 * j];
  }
}
// the thread's map values of one coil, in the fragment order of yfft_maps_kernel
template <int E>
AVX_D void col_maps(const float4* __restrict__ p, float2 (&m)[E]) {
#pragma unroll
  for (int i = 0; i < E / 2; ++i) {
    const float4 v = __ldg(p + 32 * i);
    m[2 * i] = make_float2(v.x, v.y);
    m[2 * i + 1] = make_float2(v.z, v.w);
  }
}

template <int N1, int N2>
__global__ void __launch_bounds__(ColSplit<N1, N2>::NT, N1 > 16 ? 3 : 4) yfull_kernel(KArgs a, int cpz) {
  using SP = ColSplit<N1, N2>;
  constexpr int XT = SP::XT, JP = SP::JP, E = SP::E;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tw = reinterpret_cast<float2*>(smem_raw);
  float2* buf = tw + SP::H;  // [2][N2][JP]
  const CartGeomDev& g = a.g;
  const int W = g.W, C = g.C, t = blockIdx.y;
  const int r0 = g.row_off[t], S = g.row_off[t + 1] - r0;
  const int tid = threadIdx.x, tx = tid & (XT - 1), l = tid / XT;
  const int x = blockIdx.x * XT + tx;
  col_twiddles<N1, N2>(tw, g.twy);
  int row[N2];  // compact rows of kappa = l + N1 k2
  bool any = false;
#pragma unroll
  for (int k = 0; k < N2; ++k) {
    const bool in = l < N1 && x < W;
    row[k] = in ? a.yw_inv[(long long)t * SP::H + l + N1 * k] : -1;
    any = any || row[k] >= 0;
  }
  pdl_wait();
  pdl_trigger();
  if (a.st && a.st->stop) return;
  const int cb = blockIdx.z * cpz, ce = min(C, cb + cpz);
  const bool first = l < N2;
  const float4* __restrict__ maps = reinterpret_cast<const float4*>(a.b1t) +
                                    (((size_t)cb * gridDim.x + blockIdx.x) * SP::NW + (tid >> 5)) * (E / 2) * 32 + (tid & 31);
  const size_t mstep = (size_t)gridDim.x * SP::NW * 32 * (E / 2);
  float2 u[N1], m[E];
  if (first) {
    col_maps<E>(maps, m);
    const float2* in = a.in + ((long long)t * SP::H + l) * W + (x < W ? x : 0);
#pragma unroll
    for (int i = 0; i < N1; ++i) u[i] = x < W ? in[(long long)(N2 * i) * W] : czero();
  }
  __syncthreads();
  for (int c = cb; c < ce; ++c) {
    float2* b = buf + (c & 1) * N2 * JP;
    if (first) {
      float2 v[N1];
#pragma unroll
      for (int i = 0; i < N1; ++i) v[i] = cmul(m[i], u[i]);
      maps += mstep;
      if (c + 1 < ce) col_maps<E>(maps, m);
      reg_dft<N1, +1>(v);
      b[l * JP + tx] = v[0];
#pragma unroll
      for (int k = 1; k < N1; ++k) b[l * JP + k * XT + tx] = cmul(v[k], tw[k * N2 + l]);
    }
    __syncthreads();
    if (any) {
      float2 v[N2];
#pragma unroll
      for (int j = 0; j < N2; ++j) v[j] = b[j * JP + l * XT + tx];
      reg_dft<N2, +1>(v);
      float2* out = a.qp + (long long)r0 * C * W + (long long)c * S * W + x;
#pragma unroll
      for (int k = 0; k < N2; ++k)
        if (row[k] >= 0) out[(long long)row[k] * W] = cmul(v[k], __ldg(a.yw_phase + l + N1 * k));
    }
  }
}

template <int N1, int N2>
__global__ void __launch_bounds__(ColSplit<N1, N2>::NT, N1 > 16 ? 3 : 4) yfull_adj_kernel(KArgs a, float2* img) {
  using SP = ColSplit<N1, N2>;
  constexpr int XT = SP::XT, JP = SP::JP, E = SP::E;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tw = reinterpret_cast<float2*>(smem_raw);
  float2* buf = tw + SP::H;
  const CartGeomDev& g = a.g;
  const int W = g.W, C = g.C, t = blockIdx.y;
  const int r0 = g.row_off[t], S = g.row_off[t + 1] - r0;
  const int tid = threadIdx.x, tx = tid & (XT - 1), l = tid / XT;
  const int x = blockIdx.x * XT + tx;
  col_twiddles<N1, N2>(tw, g.twy);
  int row[N2];
#pragma unroll
  for (int k = 0; k < N2; ++k) row[k] = l < N1 && x < W ? a.yw_inv[(long long)t * SP::H + l + N1 * k] : -1;
  pdl_wait();
  pdl_trigger();
  if (a.st && a.st->stop) return;
  const bool first = l < N2;
  const float4* __restrict__ maps = reinterpret_cast<const float4*>(a.b1t) +
                                    ((size_t)blockIdx.x * SP::NW + (tid >> 5)) * (E / 2) * 32 + (tid & 31);
  const size_t mstep = (size_t)gridDim.x * SP::NW * 32 * (E / 2);
  const float2* __restrict__ q = a.qp + (long long)r0 * C * W + x;
  float2 acc[N1], v[N2];
#pragma unroll
  for (int i = 0; i < N1; ++i) acc[i] = czero();
  auto load = [&] {  // the next coil's sampled rows
#pragma unroll
    for (int k = 0; k < N2; ++k) v[k] = row[k] >= 0 ? q[(long long)row[k] * W] : czero();
    q += (long long)S * W;
  };
  load();
  __syncthreads();
  for (int c = 0; c < C; ++c) {
    float2* b = buf + (c & 1) * N2 * JP;
    if (l < N1) {
#pragma unroll
      for (int k = 0; k < N2; ++k)
        if (row[k] >= 0) v[k] = cmulc(__ldg(a.yw_phase + l + N1 * k), v[k]);
      reg_dft<N2, -1>(v);
      b[l * XT + tx] = v[0];
#pragma unroll
      for (int j = 1; j < N2; ++j) b[j * JP + l * XT + tx] = cmulc(tw[l * N2 + j], v[j]);
    }
    if (c + 1 < C) load();
    __syncthreads();
    if (first) {
      float2 w[N1], m[E];
      col_maps<E>(maps, m);
      maps += mstep;
#pragma unroll
      for (int k = 0; k < N1; ++k) w[k] = b[l * JP + k * XT + tx];
      reg_dft<N1, -1>(w);
#pragma unroll
      for (int i = 0; i < N1; ++i) {
        acc[i].x = fmaf(m[i].x, w[i].x, fmaf(m[i].y, w[i].y, acc[i].x));
        acc[i].y = fmaf(m[i].x, w[i].y, fmaf(-m[i].y, w[i].x, acc[i].y));
      }
    }
  }
  if (first && x < W) {
    float2* out = img + ((long long)t * SP::H + l) * W + x;
#pragma unroll
    for (int i = 0; i < N1; ++i) out[(long long)(N2 * i) * W] = acc[i];
  }
}

// kernel `what` (0 forward, 1 adjoint) of one split
template <int N1, int N2>
void yfull_run(int what, const KArgs& k, float2* img, cudaStream_t s) {
  using SP = ColSplit<N1, N2>;
  const int tiles = (k.g.W + SP::XT - 1) / SP::XT, C = k.g.C;
  const size_t sm = sizeof(float2) * (SP::H + 2 * (size_t)N2 * SP::JP);
  if (what == 0) {
    // parts of the coils: enough warps for 14 an SM
    const long long warps = (long long)tiles * k.g.T * (SP::NT / 32);
    const int z = warps >= 148 * 14 ? 1 : (int)((148 * 14 + warps - 1) / warps);
    const int cpz = (C + (z < C ? z : C) - 1) / (z < C ? z : C);
    launch_dependent(yfull_kernel<N1, N2>, dim3(tiles, k.g.T, (C + cpz - 1) / cpz), SP::NT, sm, s, k, cpz);
  } else {
    launch_dependent(yfull_adj_kernel<N1, N2>, dim3(tiles, k.g.T), SP::NT, sm, s, k, img);
  }
}
template <int N1, int N2>
cudaError_t yfull_set() {
  const int sm = (int)(sizeof(float2) * (N1 * N2 + 2 * (size_t)N2 * ColSplit<N1, N2>::JP));
  cudaError_t e = cudaFuncSetAttribute(yfull_kernel<N1, N2>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(yfull_adj_kernel<N1, N2>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
  return e;
}

#define YFULL_DECLARE(F)                                                                   \
  int yfull_first_##F(int H);                                                              \
  bool yfull_run_##F(int what, const KArgs& k, float2* img, cudaStream_t s);               \
  cudaError_t yfull_set_##F(int H);
YFULL_DECLARE(a)
YFULL_DECLARE(b)
// The heights built, in two files: the splits of fftsplits.cuh whose second step has at most 10 points (see above).
// Other heights, such as 63, 81 or 135, take the class sums at any number of rows.
#define YFULL_SPLITS_A(X) X(12, 8) X(14, 7) X(10, 10) X(13, 8) X(12, 9) X(11, 10) X(14, 8) X(12, 10)
#define YFULL_SPLITS_B(X) X(14, 9) X(16, 8) X(13, 10) X(14, 10) X(15, 10) X(16, 10) X(18, 9) X(20, 10)
#define YFULL_FIRST_CASE(N1, N2) \
  case N1 * N2: return N1;
#define YFULL_CASE(N1, N2) \
  case N1 * N2: yfull_run<N1, N2>(what, k, img, s); return true;
#define YFULL_SET_CASE(N1, N2) \
  case N1 * N2: return yfull_set<N1, N2>();
#define YFULL_DEFINE(F, SPLITS)                                                            \
  int yfull_first_##F(int H) {                                                             \
    switch (H) { SPLITS(YFULL_FIRST_CASE) default: return 0; }                             \
  }                                                                                        \
  bool yfull_run_##F(int what, const KArgs& k, float2* img, cudaStream_t s) {              \
    switch (k.g.H) { SPLITS(YFULL_CASE) default: return false; }                           \
  }                                                                                        \
  cudaError_t yfull_set_##F(int H) {                                                       \
    switch (H) { SPLITS(YFULL_SET_CASE) default: return cudaSuccess; }                     \
  }

}  // namespace avx
