// Radial grid transforms (radfft.cuh), device code.
//
// A length G = N1 N2 is transformed in two register steps as in
// rowfft_impl.cuh: thread j < N2 takes the values j + N2 i through an N1-point
// FFT and the twiddles, thread k1 < N1 then holds k1 + N1 k2.  The padding's
// zeros are not stored or read: the y pass runs on the image columns alone
// and reads the image rows alone, the x pass pads in registers.  The x pass
// of the forward transform keeps its rows in shared memory and interpolates
// the samples of those rows from there, so that the full grid is never
// written; the adjoint's x pass writes only the image columns.
//
// Before, four passes over the whole grid (Stockham FFTs through shared
// memory) and a gather per sample.  128 x 128, 40 frames, 12 coils, 21 spokes
// of 256 samples, grid 192 x 192: forward transform and interpolation 252 ->
// 148 us, adjoint transform 176 -> 98; 104 x 90, 23 frames, 5 coils, 13 spokes
// of 208, grid 208 x 180 (a run-time plan with radix 13 before): 107 -> 47 and
// 136 -> 55 with the spreading (of spread.cu).
#pragma once

#include "fftsplits.cuh"
#include "radfft.cuh"
#include "regfft.cuh"

namespace avx {

template <int N1, int N2>
struct RadSplit {
  static_assert(N1 >= N2, "the first step is the longer one");
  static constexpr int G = N1 * N2;
  static constexpr int P = N2 | 1;       // odd pitch of the exchanged rows
  static constexpr int ROW = N1 * P;     // a row: position (i, j) = (n / N2, n % N2) at i P + j
  static constexpr int XT = 8;           // columns per CTA of the y passes
};

// grid index -> image index along one axis, or -1 in the padding
AVX_D int rad_img(int m, int d, int G) {
  const int h = d / 2;
  if (m < d - h) return m + h;
  if (m >= G - h) return m - G + h;
  return -1;
}

template <int N1, int N2>
AVX_D void rad_twiddles(float2* tw, const float2* __restrict__ w) {
  for (int e = threadIdx.x; e < N1 * N2; e += blockDim.x) {
    const int k1 = e / N2, j = e - k1 * N2;
    tw[e] = w[k1 * j];
  }
}

// Forward y pass: CTA (8 image columns, frame, part of the coils).  The
// frame's deapodised column values stay in registers over the coils; two
// exchange buffers, one barrier a coil.
template <int N1, int N2>
__global__ void __launch_bounds__(8 * N1) rad_cols_fwd_kernel(RArgs a, int cpz) {
  using SP = RadSplit<N1, N2>;
  constexpr int XT = SP::XT, JP = (N1 + 1) * XT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tw = reinterpret_cast<float2*>(smem_raw);
  float2* buf = tw + SP::G;  // [2][N2][N1 + 1][XT]
  const RadialGeomDev& g = a.g;
  const int W = g.W, H = g.H;
  const int f = blockIdx.y, tx = threadIdx.x & (XT - 1), l = threadIdx.x / XT;
  const int x = blockIdx.x * XT + tx;
  rad_twiddles<N1, N2>(tw, g.twgy);
  pdl_wait();
  pdl_trigger();
  if (a.st && a.st->stop) return;
  const bool first = l < N2 && x < W;
  float2 u[N1];
  int off[N1];
#pragma unroll
  for (int i = 0; i < N1; ++i) {
    const int n = first ? rad_img(l + N2 * i, H, SP::G) : -1;
    off[i] = n < 0 ? -1 : n * W + x;
    u[i] = czero();
    if (n >= 0) {
      const long long p = (long long)f * H * W + off[i];
      float2 v = a.in[p];
      if (a.in2) v = csub(v, a.in2[p]);
      u[i] = cscale(v, g.inv_psi_y[n] * g.inv_psi_x[x]);
    }
  }
  const int cb = blockIdx.z * cpz, ce = min(g.C, cb + cpz);
  __syncthreads();
  for (int c = cb; c < ce; ++c) {
    float2* b = buf + (c & 1) * N2 * JP;
    if (first) {
      const float2* __restrict__ b1 = a.b1 + (long long)c * H * W;
      float2 v[N1];
#pragma unroll
      for (int i = 0; i < N1; ++i) v[i] = off[i] >= 0 ? __ldg(b1 + off[i]) : czero();
#pragma unroll
      for (int i = 0; i < N1; ++i) v[i] = cmul(v[i], u[i]);
      reg_dft<N1, -1>(v);
      b[l * JP + tx] = v[0];
#pragma unroll
      for (int k = 1; k < N1; ++k) b[l * JP + k * XT + tx] = cmulc(tw[k * N2 + l], v[k]);
    }
    __syncthreads();
    if (x < W) {
      float2 v[N2];
#pragma unroll
      for (int j = 0; j < N2; ++j) v[j] = b[j * JP + l * XT + tx];
      reg_dft<N2, -1>(v);
      float2* out = a.grid + (((long long)f * g.C + c) * SP::G + l) * g.Gx + x;
#pragma unroll
      for (int k = 0; k < N2; ++k) out[(long long)(N1 * k) * g.Gx] = v[k];
    }
  }
}

// rows of the grid that the samples of sector rows [sr0, sr1) reach beyond them
AVX_HD int rad_halo_low(float J) { return (int)floorf(0.5f * J) + 1; }
AVX_HD int rad_halo_high(float J) { return (int)floorf(ceilf(J) - 0.5f * J) + 1; }

// what the interpolation reads of one sample
template <int NW>
struct RadSample {
  int s;
  int2 g0;
  float wx[NW], wy[NW], sc;
  float2 z, d;
};
template <int NW>
AVX_D void rad_load_sample(const RArgs& a, int fc, int f, int s, bool zd, RadSample<NW>& o) {
  const RadialGeomDev& g = a.g;
  const long long fs = (long long)f * g.S + s;
  o.s = s;
  o.g0 = __ldg(g.win0 + fs);
  if constexpr (NW == 4) {  // a sample's eight weights are one aligned sector
    const float4* w4 = reinterpret_cast<const float4*>(g.winw) + fs * 2;
    const float4 p = __ldg(w4), q = __ldg(w4 + 1);
    o.wx[0] = p.x, o.wx[1] = p.y, o.wx[2] = p.z, o.wx[3] = p.w;
    o.wy[0] = q.x, o.wy[1] = q.y, o.wy[2] = q.z, o.wy[3] = q.w;
  } else {
#pragma unroll
    for (int k = 0; k < NW; ++k) {
      o.wx[k] = __ldg(g.winw + fs * 2 * NW + k);
      o.wy[k] = __ldg(g.winw + fs * 2 * NW + NW + k);
    }
  }
  o.sc = __ldg(g.sqrt_w + fs);
  if (zd) {
    o.z = a.z[(long long)fc * g.S + s];
    o.d = a.d[(long long)fc * g.S + s];
  }
}

// Forward x pass and interpolation: CTA (block of sector rows, frame and
// coil).  The block's grid rows and their halo are transformed into shared
// memory, then each thread interpolates samples of the block's sectors.
// 32 rows a block: the halo of 4 costs an eighth of the transforms, and three
// CTAs' tiles fit an SM.  Bound by LSU wavefronts and issue slots (67 % and
// 47 %, 105 us at the 192 x 192 problem); without the requests a round ahead
// 110, with scalar loads of the weights 122.
template <int N1, int N2, int NW>
__global__ void __launch_bounds__(256) rad_rows_interp_kernel(RArgs a, int mode, int srb) {
  using SP = RadSplit<N1, N2>;
  constexpr int G = SP::G, RP = 256 / N1;  // rows per pass
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tw = reinterpret_cast<float2*>(smem_raw);
  float2* tile = tw + G;  // [rows][ROW]
  const RadialGeomDev& g = a.g;
  const int fc = blockIdx.y, f = fc / g.C;
  const int sr0 = blockIdx.x * srb, sr1 = min(g.nsy, sr0 + srb);
  const int y0 = sr0 * g.sw - rad_halo_low(g.J);
  const int rows = min(g.Gy, sr1 * g.sw) + rad_halo_high(g.J) - y0;
  const int W = g.W;
  rad_twiddles<N1, N2>(tw, g.twgx);
  pdl_wait();
  pdl_trigger();
  if (a.st && a.st->stop && mode != 3) return;
  __syncthreads();
  // the block's samples; each thread's next one is requested a round ahead (the first before the transforms), its
  // index two rounds, so that the two dependent latencies pass behind the arithmetic
  const int* st = g.sec_start + (long long)f * (g.nsx * g.nsy + 1);
  const int* order = g.order + (long long)f * g.S;
  int q = st[sr0 * g.nsx] + threadIdx.x;
  const int q1 = st[sr1 * g.nsx];
  const bool zd = mode == 0 || mode == 2;
  RadSample<NW> nx;
  int s_next = 0;
  if (q < q1) rad_load_sample<NW>(a, fc, f, order[q], zd, nx);
  if (q + 256 < q1) s_next = order[q + 256];
  const float2* src = a.grid + (long long)fc * g.Gy * G;
  const int r = threadIdx.x / N1, l = threadIdx.x - r * N1;
  const int m_low = W - W / 2 - l, m_high = G - W / 2 - l;
  for (int k0 = 0; k0 < rows; k0 += RP) {
    const int rr = k0 + r;
    const bool live = r < RP && rr < rows;
    float2* row = tile + rr * SP::ROW;
    if (live && l < N2) {
      int y = y0 + rr;
      y = y < 0 ? y + g.Gy : (y >= g.Gy ? y - g.Gy : y);
      const float2* p = src + (long long)y * G;
      float2 v[N1];
      // grid positions m = l + N2 i below W - h hold x = m + h, those from G - h on x = m - G + h (h = W / 2)
      const float2* pa = p + W / 2 + l;
      const float2* pb = pa - G;
#pragma unroll
      for (int i = 0; i < N1; ++i) {
        v[i] = czero();
        if (N2 * i < m_low) v[i] = pa[N2 * i];
        if (N2 * i >= m_high) v[i] = pb[N2 * i];
      }
      reg_dft<N1, -1>(v);
      row[l] = v[0];
#pragma unroll
      for (int k = 1; k < N1; ++k) row[k * SP::P + l] = cmulc(tw[k * N2 + l], v[k]);
    }
    __syncthreads();
    if (live) {
      float2 v[N2];
#pragma unroll
      for (int j = 0; j < N2; ++j) v[j] = row[l * SP::P + j];
      reg_dft<N2, -1>(v);
#pragma unroll
      for (int k = 0; k < N2; ++k) row[l * SP::P + k] = v[k];  // kx = l + N1 k, in place
    }
  }
  __syncthreads();
  const float sig = a.st ? (float)a.st->sigma : 0.f;
  const float zscale = (mode == 0) ? (float)(1.0 / (1.0 + a.st->sigma / (double)a.lam)) : 1.f;
  double acc[3] = {0.0, 0.0, 0.0};
  for (; q < q1; q += 256) {
    const RadSample<NW> o = nx;
    if (q + 256 < q1) rad_load_sample<NW>(a, fc, f, s_next, zd, nx);
    if (q + 512 < q1) s_next = order[q + 512];
    int px[NW];
#pragma unroll
    for (int k = 0; k < NW; ++k) {
      int kx = o.g0.x + k;
      kx = kx < 0 ? kx + G : (kx >= G ? kx - G : kx);
      px[k] = (kx % N1) * SP::P + kx / N1;
    }
    // the window's first row within the tile: its unwrapped start lies at most a grid away from the block's
    int ly = o.g0.y - y0;
    ly = ly < 0 ? ly + g.Gy : (ly >= g.Gy ? ly - g.Gy : ly);
    const long long zi = (long long)fc * g.S + o.s;
    float2 v = czero();
    if (ly + NW <= rows) {
      const float2* t = tile + ly * SP::ROW;
#pragma unroll
      for (int oy = 0; oy < NW; ++oy) {
        float2 rowv = czero();
#pragma unroll
        for (int ox = 0; ox < NW; ++ox) rowv = fma2(make_float2(o.wx[ox], o.wx[ox]), t[oy * SP::ROW + px[ox]], rowv);
        v = fma2(make_float2(o.wy[oy], o.wy[oy]), rowv, v);
      }
    }
    const float2 k = cscale(v, o.sc * g.norm);
    if (mode == 0) {
      // z += sigma K x; z = (z - sigma d) / (1 + sigma / lambda)   (tgv2.cpp:254-264)
      float2 zn = make_float2(o.z.x + sig * k.x, o.z.y + sig * k.y);
      zn = make_float2(zn.x - sig * o.d.x, zn.y - sig * o.d.y);
      a.z[zi] = cscale(zn, zscale);
    } else if (mode == 1) {
      acc[0] += (double)cabs2(k);
    } else if (mode == 2) {
      acc[0] += (double)cabs2(csub(k, o.d));
      acc[1] += (double)o.d.x * o.z.x + (double)o.d.y * o.z.y;
      acc[2] += (double)cabs2(o.z);
    } else {
      a.out[zi] = k;
    }
  }
  if (mode == 1 || mode == 2) {
    __shared__ double red[32 * 3];
    block_sum<3>(acc, red);
    if (threadIdx.x == 0) {
      const int nb = gridDim.x * gridDim.y, b = blockIdx.y * gridDim.x + blockIdx.x;
      for (int k = 0; k < 3; ++k) a.partial[k * nb + b] = acc[k];
    }
  }
}

// Adjoint x pass: rows of the grid (any frame and coil), cropped to the image
// columns at the row's start.  Each row is read before the exchange and
// written after it by the same CTA, so in place.
template <int N1, int N2>
__global__ void __launch_bounds__(256) rad_rows_inv_kernel(RArgs a, long long nrows) {
  using SP = RadSplit<N1, N2>;
  constexpr int G = SP::G, RP = 256 / N1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tw = reinterpret_cast<float2*>(smem_raw);
  float2* tile = tw + G;  // [RP][ROW]
  const RadialGeomDev& g = a.g;
  rad_twiddles<N1, N2>(tw, g.twgx);
  pdl_wait();
  pdl_trigger();
  if (a.st && a.st->stop) return;
  __syncthreads();
  const int r = threadIdx.x / N1, l = threadIdx.x - r * N1;
  const long long rr = (long long)blockIdx.x * RP + r;
  const bool live = r < RP && rr < nrows;
  float2* row = tile + r * SP::ROW;
  float2* p = a.grid + rr * G;
  if (live && l < N2) {
    float2 v[N1];
#pragma unroll
    for (int i = 0; i < N1; ++i) v[i] = p[l + N2 * i];
    reg_dft<N1, +1>(v);
    row[l] = v[0];
#pragma unroll
    for (int k = 1; k < N1; ++k) row[k * SP::P + l] = cmul(v[k], tw[k * N2 + l]);
  }
  __syncthreads();
  if (live) {
    float2 v[N2];
#pragma unroll
    for (int j = 0; j < N2; ++j) v[j] = row[l * SP::P + j];
    reg_dft<N2, +1>(v);
#pragma unroll
    for (int k = 0; k < N2; ++k) {
      const int x = rad_img(l + N1 * k, g.W, G);
      if (x >= 0) p[x] = v[k];
    }
  }
}

// Adjoint y pass: CTA (8 image columns, frame), all coils; thread (tx, k1)
// accumulates the image rows of grid rows k1 + N1 k2.  The next coil's column
// values are requested before the barrier, and registers are held to five
// CTAs an SM: 172 registers and no request ahead took 77 us at the 192 x 192
// problem, this 61 (96 MB read).
template <int N1, int N2>
__global__ void __launch_bounds__(8 * N1, N1 > 16 ? 3 : 5) rad_cols_inv_kernel(RArgs a, float2* img) {
  using SP = RadSplit<N1, N2>;
  constexpr int XT = SP::XT, JP = (N1 + 1) * XT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tw = reinterpret_cast<float2*>(smem_raw);
  float2* buf = tw + SP::G;
  const RadialGeomDev& g = a.g;
  const int W = g.W, H = g.H;
  const int f = blockIdx.y, tx = threadIdx.x & (XT - 1), l = threadIdx.x / XT;
  const int x = blockIdx.x * XT + tx;
  rad_twiddles<N1, N2>(tw, g.twgy);
  pdl_wait();
  pdl_trigger();
  if (a.st && a.st->stop) return;
  float2 acc[N2], v[N1];
#pragma unroll
  for (int k = 0; k < N2; ++k) acc[k] = czero();
  const bool first = l < N2 && x < W;
  const float2* in = a.grid + ((long long)f * g.C * SP::G + l) * g.Gx + x;
  auto load = [&] {  // the next coil's column values
    if (first)
#pragma unroll
      for (int i = 0; i < N1; ++i) v[i] = in[(long long)(N2 * i) * g.Gx];
    in += (long long)SP::G * g.Gx;
  };
  load();
  __syncthreads();
  for (int c = 0; c < g.C; ++c) {
    float2* b = buf + (c & 1) * N2 * JP;
    if (first) {
      reg_dft<N1, +1>(v);
      b[l * JP + tx] = v[0];
#pragma unroll
      for (int k = 1; k < N1; ++k) b[l * JP + k * XT + tx] = cmul(v[k], tw[k * N2 + l]);
    }
    if (c + 1 < g.C) load();
    __syncthreads();
    if (x < W) {
      const float2* __restrict__ b1 = a.b1 + (long long)c * H * W + x;
      float2 w[N2];
#pragma unroll
      for (int j = 0; j < N2; ++j) w[j] = b[j * JP + l * XT + tx];
      reg_dft<N2, +1>(w);
#pragma unroll
      for (int k = 0; k < N2; ++k) {
        const int n = rad_img(l + N1 * k, H, SP::G);
        if (n >= 0) {
          const float2 m = __ldg(b1 + n * W);
          acc[k].x = fmaf(m.x, w[k].x, fmaf(m.y, w[k].y, acc[k].x));
          acc[k].y = fmaf(m.x, w[k].y, fmaf(-m.y, w[k].x, acc[k].y));
        }
      }
    }
  }
  if (x < W)
#pragma unroll
    for (int k = 0; k < N2; ++k) {
      const int n = rad_img(l + N1 * k, H, SP::G);
      if (n >= 0) img[((long long)f * H + n) * W + x] = cscale(acc[k], g.inv_psi_y[n] * g.inv_psi_x[x]);
    }
}

template <int N1, int N2>
size_t rad_cols_smem() {
  return sizeof(float2) * (N1 * N2 + 2 * (size_t)N2 * (N1 + 1) * 8);
}
// sector rows per block of the interpolating pass: 32 grid rows or one sector row
inline int rad_block_sectors(const RadialGeomDev& g) { return g.sw >= 32 ? 1 : 32 / g.sw; }
template <int N1, int N2>
size_t rad_interp_smem(const RadialGeomDev& g) {
  const int rows = rad_block_sectors(g) * g.sw + rad_halo_low(g.J) + rad_halo_high(g.J);
  return sizeof(float2) * (N1 * N2 + (size_t)rows * RadSplit<N1, N2>::ROW);
}

// kernel instances of one split, by the kernel's number: 0 y forward, 1 x
// forward with interpolation, 2 x adjoint, 3 y adjoint; configure: attributes
template <int N1, int N2>
void radfft_run(int what, const RArgs& a, int mode, float2* img, cudaStream_t s) {
  const RadialGeomDev& g = a.g;
  const int tiles = (g.W + 7) / 8;
  if (what == 0) {
    // parts of the coils: enough warps for 14 an SM
    const long long warps = (long long)tiles * g.T * (8 * N1 / 32);
    const int z = (int)(warps >= 148 * 14 ? 1 : (148 * 14 + warps - 1) / warps);
    const int cpz = (g.C + (z < g.C ? z : g.C) - 1) / (z < g.C ? z : g.C);
    launch_dependent(rad_cols_fwd_kernel<N1, N2>, dim3(tiles, g.T, (g.C + cpz - 1) / cpz), 8 * N1,
                     rad_cols_smem<N1, N2>(), s, a, cpz);
  } else if (what == 1) {
    const int srb = rad_block_sectors(g);
    const dim3 gr((g.nsy + srb - 1) / srb, g.C * g.T);
    const size_t sm = rad_interp_smem<N1, N2>(g);
    if (g.nw == 4)
      launch_dependent(rad_rows_interp_kernel<N1, N2, 4>, gr, 256, sm, s, a, mode, srb);
    else if (g.nw == 3)
      launch_dependent(rad_rows_interp_kernel<N1, N2, 3>, gr, 256, sm, s, a, mode, srb);
    else
      launch_dependent(rad_rows_interp_kernel<N1, N2, 5>, gr, 256, sm, s, a, mode, srb);
  } else if (what == 2) {
    const long long rows = (long long)g.T * g.C * g.Gy;
    constexpr int RP = 256 / N1;
    launch_dependent(rad_rows_inv_kernel<N1, N2>, (unsigned)((rows + RP - 1) / RP), 256,
                     sizeof(float2) * (N1 * N2 + (size_t)RP * RadSplit<N1, N2>::ROW), s, a, rows);
  } else {
    launch_dependent(rad_cols_inv_kernel<N1, N2>, dim3(tiles, g.T), 8 * N1, rad_cols_smem<N1, N2>(), s, a, img);
  }
}
template <int N1, int N2>
cudaError_t radfft_set(const RadialGeomDev& g) {
  const cudaFuncAttribute dyn = cudaFuncAttributeMaxDynamicSharedMemorySize;
  cudaError_t e = cudaSuccess;
  if (g.Gy == N1 * N2) {
    e = cudaFuncSetAttribute(rad_cols_fwd_kernel<N1, N2>, dyn, AVX_DYN_SMEM_MAX);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(rad_cols_inv_kernel<N1, N2>, dyn, AVX_DYN_SMEM_MAX);
  }
  if (e == cudaSuccess && g.Gx == N1 * N2) {
    auto interp = g.nw == 4   ? rad_rows_interp_kernel<N1, N2, 4>
                  : g.nw == 3 ? rad_rows_interp_kernel<N1, N2, 3>
                              : rad_rows_interp_kernel<N1, N2, 5>;
    e = cudaFuncSetAttribute(interp, dyn, AVX_DYN_SMEM_MAX);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(rad_rows_inv_kernel<N1, N2>, dyn, AVX_DYN_SMEM_MAX);
  }
  return e;
}

#define RADFFT_DECLARE(F)                                                                              \
  bool radfft_run_##F(int G, int what, const RArgs* a, int mode, float2* img, cudaStream_t s);         \
  cudaError_t radfft_set_##F(const RadialGeomDev& g);                                                  \
  size_t radfft_interp_smem_##F(const RadialGeomDev& g);
RADFFT_DECLARE(a)
RADFFT_DECLARE(b)
RADFFT_DECLARE(c)
RADFFT_DECLARE(d)

// runs kernel `what` of length G when this file has its split (a == nullptr: only says whether it has)
#define RADFFT_CASE(N1, N2) \
  case N1 * N2: if (a) radfft_run<N1, N2>(what, *a, mode, img, s); return true;
#define RADFFT_SMEM_CASE(N1, N2) \
  case N1 * N2: return rad_interp_smem<N1, N2>(g);
#define RADFFT_SET_CASE(N1, N2) \
  if (e == cudaSuccess) e = radfft_set<N1, N2>(g);
#define RADFFT_DEFINE(F, SPLITS)                                                                       \
  bool radfft_run_##F(int G, int what, const RArgs* a, int mode, float2* img, cudaStream_t s) {        \
    switch (G) { SPLITS(RADFFT_CASE) default: return false; }                                          \
  }                                                                                                    \
  size_t radfft_interp_smem_##F(const RadialGeomDev& g) {                                              \
    switch (g.Gx) { SPLITS(RADFFT_SMEM_CASE) default: return 0; }                                      \
  }                                                                                                    \
  cudaError_t radfft_set_##F(const RadialGeomDev& g) {                                                 \
    cudaError_t e = cudaSuccess;                                                                       \
    SPLITS(RADFFT_SET_CASE)                                                                            \
    return e;                                                                                          \
  }

}  // namespace avx
