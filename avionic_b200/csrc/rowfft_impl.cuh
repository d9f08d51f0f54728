// Row FFTs of the Cartesian operator's compact rows (rowfft.cuh), device code.
//
// A row of W = N1 N2 values is transformed by L = max(N1, N2) threads in two
// steps with one exchange through shared memory: thread j < N2 takes the
// values x = j + N2 i through an N1-point register FFT and the twiddles
// w^{j k1}; after the exchange thread k1 < N1 takes them through an N2-point
// FFT and holds kx = k1 + N1 k2, where the pointwise stage (mask, z-prox,
// gap or norm sums) happens in registers with neighbouring threads on
// neighbouring kx.  The inverse transform runs the same two steps back.  The
// Stockham passes of rows_kernel move every value through shared memory
// eight times per forward and inverse pair; here it is twice.
//
// Bound by the latency of a pass's phases (load, exchange, pointwise,
// exchange, store) at 15 to 20 warps an SM; a quarter of the issue slots are
// used, DRAM runs at 3 TB/s at 320 x 320.  z and d arrive by cp.async in one
// contiguous run per pass: requesting them into registers needs 168 registers
// (301 us), loading them where they are used serialises their latency (324).
// 102 registers at most (two CTAs of 320 threads): 134 take 276 us, 68 spill
// (339).  Stage time, rows_kernel -> here: 320 x 320, 48 frames, 32 coils, 53
// rows 341 -> 246 us; 192 x 192, 30 frames, 16 coils, 16 rows 25 -> 20;
// 160 x 128, 24 frames, 12 coils, 64 rows 47 -> 26; 150 x 131, 13 frames, 7
// coils (rows_kernel has only a run-time plan) 40 -> 16.
#pragma once

#include "regfft.cuh"
#include "rowfft.cuh"

namespace avx {

template <int N1, int N2>
struct RowSplit {
  static constexpr int W = N1 * N2, L = N1 > N2 ? N1 : N2;
  static constexpr int P1 = N2 | 1, P2 = N1 | 1;  // odd pitches: strided 64-bit reads hit every bank once
  static constexpr int ROW = ((N1 * P1 > N2 * P2 ? N1 * P1 : N2 * P2) + 1) & ~1;
};

// position n of the transform's sequences holds index n + sx (mod W) of a row
template <int W, bool CENT>
AVX_D int row_index(int n, int sx) {
  if (!CENT) return n;
  n += sx;
  return n >= W ? n - W : n;
}

// PD: mode 0 (the primal-dual step) alone, else the mode is read at run time.
// CENT: centred transform; without it every access of a thread is one base
// pointer plus a constant.
template <int N1, int N2, bool PD, bool CENT>
__global__ void __launch_bounds__(320, 2) rowfft_kernel(KArgs a, int mode_rt, int kc) {
  using SP = RowSplit<N1, N2>;
  constexpr int W = SP::W, L = SP::L;
  const int mode = PD ? 0 : mode_rt;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const CartGeomDev& g = a.g;
  const int C = g.C;
  const int c = blockIdx.x % C, t = blockIdx.x / C;
  const int r0 = g.row_off[t], S = g.row_off[t + 1] - r0;
  const long long zb = kbase(g, t, c, r0, r0 + S);
  float2* tw = reinterpret_cast<float2*>(smem_raw);  // [N1][N2] w^{j k1}
  float2* buf = tw + W + (W & 1);                    // [kc][ROW]
  float2* zs = buf + kc * SP::ROW;                   // PD: [kc][W] of z, then of d
  float2* ds = zs + kc * W;
  const int tid = threadIdx.x;  // kc L threads, and idle ones up to a whole warp
  for (int e = tid; e < W; e += blockDim.x) {
    const int k1 = e / N2, j = e - k1 * N2;
    tw[e] = g.twx[k1 * j];
  }
  pdl_wait();
  pdl_trigger();
  if (a.st && a.st->stop && (PD || (mode != 3 && mode != 5))) return;
  const int r = tid / L, l = tid - r * L;
  float2* row = buf + r * SP::ROW;
  const int sx = g.sx;
  const float sig = a.st ? (float)a.st->sigma : 0.f;
  const float zscale = mode == 0 ? (float)(1.0 / (1.0 + a.st->sigma / (double)a.lam)) : 1.f;
  double acc[3] = {0.0, 0.0, 0.0};
  for (int k0 = 0; k0 < S; k0 += kc) {
    const int kk = k0 + r;
    const bool live = r < kc && kk < S;
    const long long base = zb + (long long)kk * W;
    const bool first = live && l < N2, second = live && l < N1;
    __syncthreads();  // the twiddles are staged; the previous pass has read its rows
    if (PD) {
      // the pass's z and d, one contiguous run each, are in flight during the first step
      const long long b0 = zb + (long long)k0 * W;
      const int n = min(kc, S - k0) * W;
      const unsigned sz = (unsigned)__cvta_generic_to_shared(zs), sd = (unsigned)__cvta_generic_to_shared(ds);
      if constexpr (W % 2 == 0) {
        for (int e = 2 * tid; e < n; e += 2 * blockDim.x) {
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sz + 8 * e), "l"(a.z + b0 + e) : "memory");
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sd + 8 * e), "l"(a.d + b0 + e) : "memory");
        }
      } else {
        for (int e = tid; e < n; e += blockDim.x) {
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sz + 8 * e), "l"(a.z + b0 + e) : "memory");
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sd + 8 * e), "l"(a.d + b0 + e) : "memory");
        }
      }
    }
    float2 X[N2];
    if (PD || mode != 5) {
      if (first) {
        float2 v[N1];
#pragma unroll
        for (int i = 0; i < N1; ++i) {
          const int x = row_index<W, CENT>(l + N2 * i, sx);
          v[i] = a.qp[base + x];
        }
        reg_dft<N1, +1>(v);
        row[l] = v[0];
#pragma unroll
        for (int k = 1; k < N1; ++k) row[k * SP::P1 + l] = cmul(v[k], tw[k * N2 + l]);
      }
    }
    if (PD) asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (second) {
      const float* mr = g.mrow + (long long)(r0 + kk) * W;
      if (PD || mode != 5) {
#pragma unroll
        for (int j = 0; j < N2; ++j) X[j] = row[l * SP::P1 + j];
        reg_dft<N2, +1>(X);
      } else {
        const float2* src = a.dense_in + (((long long)t * C + c) * g.H + g.rows[r0 + kk]) * W;
#pragma unroll
        for (int k = 0; k < N2; ++k) {
          const int kx = row_index<W, CENT>(l + N1 * k, sx);
          X[k] = src[kx];
        }
      }
      if (PD) {
#pragma unroll
        for (int k = 0; k < N2; ++k) {
          const int kx = row_index<W, CENT>(l + N1 * k, sx);
          const float m = __ldg(mr + kx);
          const float2 mX = cscale(cscale(X[k], g.inv_sqrt_w), m);
          const float2 zo = zs[r * W + kx], dv = ds[r * W + kx];
          // z += sigma * (mask X); z = (z - sigma d) / (1 + sigma / lambda); z *= mask
          float2 zn = make_float2(zo.x + sig * mX.x, zo.y + sig * mX.y);
          zn = make_float2(zn.x - sig * dv.x, zn.y - sig * dv.y);
          zn = cscale(zn, zscale);
          zn = cscale(zn, m);
          a.z[base + kx] = zn;
          X[k] = zn;
        }
      } else if (mode != 5) {
#pragma unroll
        for (int k = 0; k < N2; ++k) {
          const int kx = row_index<W, CENT>(l + N1 * k, sx);
          const float m = mr[kx];
          const float2 mX = cscale(cscale(X[k], g.inv_sqrt_w), m);
          if (mode == 1) {
            acc[0] += (double)cabs2(mX);
          } else if (mode == 2) {
            const float2 zo = a.z[base + kx], dv = a.d[base + kx];
            acc[0] += (double)cabs2(csub(mX, dv));
            acc[1] += (double)dv.x * zo.x + (double)dv.y * zo.y;
            acc[2] += (double)cabs2(zo);
            const float2 zm = cscale(zo, m);
            if (!a.binary_mask) a.z[base + kx] = zm;
            X[k] = zm;
          } else if (mode == 4) {
            X[k] = cscale(mX, m);
          } else {
            a.dense_out[(((long long)t * C + c) * g.H + g.rows[r0 + kk]) * W + kx] = mX;
          }
        }
      }
    }
    if (!PD && (mode == 1 || mode == 3)) continue;
    __syncthreads();  // every thread has read its first-step values
    if (second) {
      reg_dft<N2, -1>(X);
#pragma unroll
      for (int j = 0; j < N2; ++j) row[j * SP::P2 + l] = cmulc(tw[l * N2 + j], X[j]);
    }
    __syncthreads();
    if (first) {
      float2 v[N1];
#pragma unroll
      for (int k = 0; k < N1; ++k) v[k] = row[l * SP::P2 + k];
      reg_dft<N1, -1>(v);
#pragma unroll
      for (int i = 0; i < N1; ++i) {
        const int x = row_index<W, CENT>(l + N2 * i, sx);
        a.qp[base + x] = cscale(v[i], g.inv_sqrt_w);
      }
    }
  }
  if (!PD && (mode == 1 || mode == 2)) {
    __shared__ double red[32 * 3];
    block_sum<3>(acc, red);
    if (tid == 0) {
      const int nb = gridDim.x;
      a.partial[0 * nb + blockIdx.x] = acc[0];
      a.partial[1 * nb + blockIdx.x] = acc[1];
      a.partial[2 * nb + blockIdx.x] = acc[2];
    }
  }
}

template <int N1, int N2>
void rowfft_launch(const KArgs& k, int mode, cudaStream_t s) {
  using SP = RowSplit<N1, N2>;
  const int kc = k.rows_kc ? k.rows_kc : 16;  // rows per pass: 8, 12 or 16
  const size_t sm = sizeof(float2) * (SP::W + (SP::W & 1) + (size_t)kc * (SP::ROW + (mode == 0 ? 2 * SP::W : 0)));
  const int nt = (kc * SP::L + 31) / 32 * 32;  // block_sum's shuffles need whole warps
  if (mode != 0)
    launch_dependent(rowfft_kernel<N1, N2, false, true>, k.g.C * k.g.T, nt, sm, s, k, mode, kc);
  else if (k.g.sx)
    launch_dependent(rowfft_kernel<N1, N2, true, true>, k.g.C * k.g.T, nt, sm, s, k, 0, kc);
  else
    launch_dependent(rowfft_kernel<N1, N2, true, false>, k.g.C * k.g.T, nt, sm, s, k, 0, kc);
}

template <int N1, int N2>
cudaError_t rowfft_configure() {
  using SP = RowSplit<N1, N2>;
  const int sm = (int)(sizeof(float2) * (SP::W + 1 + (size_t)16 * (SP::ROW + 2 * SP::W)));
  const cudaFuncAttribute dyn = cudaFuncAttributeMaxDynamicSharedMemorySize;
  cudaError_t e = cudaFuncSetAttribute(rowfft_kernel<N1, N2, true, true>, dyn, sm);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(rowfft_kernel<N1, N2, true, false>, dyn, sm);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(rowfft_kernel<N1, N2, false, true>, dyn, sm);
  return e;
}

// Short rows (rowfft_e.cu): lengths 20 to 32 of 5 to 13 by 2 to 5 points, and
// longer ones of 7 to 16 by 5 to 7.  Such a pass is all latency: two register
// steps have one exchange where the Stockham plan has two to four, and the
// kernel can be a dependent launch.  A whole TGV2 iteration, run-time plan and
// here: 24 x 20, 6 frames, 4 coils 19.5 and 15.7 us; 50 x 64, 10 frames, 6
// coils, 16 rows 33.3 and 19.2; 72 x 131, 12 frames, 8 coils 58.0 and 45.5;
// 40 x 97, 10 frames, 8 coils 37.8 and 29.5.  Below 20 the plan's two steps
// are as short, and other splits (an N2 under 5 at longer rows) leave most
// lanes idle in one step.
bool rowfft_short_split(int W, int* n1, int* n2);
void rowfft_launch_short(int n1, int n2, const KArgs& k, int mode, cudaStream_t s);
cudaError_t rowfft_configure_short(int n1, int n2);

// one translation unit per first length, so that the instances build in parallel
#define ROWFFT_DECLARE(N1)                                                       \
  void rowfft_launch_##N1(int n2, const KArgs& k, int mode, cudaStream_t s);     \
  cudaError_t rowfft_configure_##N1(int n2);
ROWFFT_DECLARE(8)
ROWFFT_DECLARE(9)
ROWFFT_DECLARE(10)
ROWFFT_DECLARE(11)
ROWFFT_DECLARE(12)
ROWFFT_DECLARE(13)
ROWFFT_DECLARE(14)
ROWFFT_DECLARE(15)
ROWFFT_DECLARE(16)
ROWFFT_DECLARE(20)

template <int N1, int N2>
void rowfft_launch_rec(int n2, const KArgs& k, int mode, cudaStream_t s) {
  if constexpr (N2 >= 8) {
    if (n2 == N2)
      rowfft_launch<N1, N2>(k, mode, s);
    else
      rowfft_launch_rec<N1, N2 - 1>(n2, k, mode, s);
  }
}
template <int N1, int N2>
cudaError_t rowfft_configure_rec(int n2) {
  if constexpr (N2 >= 8) return n2 == N2 ? rowfft_configure<N1, N2>() : rowfft_configure_rec<N1, N2 - 1>(n2);
  return cudaSuccess;
}
#define ROWFFT_DEFINE(N1)                                                        \
  void rowfft_launch_##N1(int n2, const KArgs& k, int mode, cudaStream_t s) {    \
    rowfft_launch_rec<N1, (N1 < 16 ? N1 : 16)>(n2, k, mode, s);                  \
  }                                                                              \
  cudaError_t rowfft_configure_##N1(int n2) { return rowfft_configure_rec<N1, (N1 < 16 ? N1 : 16)>(n2); }

}  // namespace avx
