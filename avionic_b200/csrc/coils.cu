// Variational H1 coil-sensitivity estimation kernels (reference:
// CUDA/src/coil_construction.cpp:55-556, cartesian_coil_construction.cpp:23-86).
//
// Images are single W x H slices (coil images stacked [coil][H][W]); the 2D
// stencils are the (x, y) restriction of the 3D ones: gradient (D+x, D+y),
// symmetrised gradient (xx, yy, xy with 1/2 on the off-diagonal),
// divergences as their negative adjoints (utils.cpp:156-181, 525-568,
// 664-684, 817-844, 1078-1117).
#include <algorithm>

#include <cooperative_groups.h>

#include "coils.cuh"
#include "regfft.cuh"
#include "stencil.cuh"

namespace avx {

struct P2 {
  int x, y, W, H;
  long long i;
};

AVX_D P2 p2_of(int idx, int W, int H) {
  P2 p;
  p.x = idx % W;
  p.y = idx / W;
  p.W = W;
  p.H = H;
  p.i = idx;
  return p;
}

AVX_D void grad2(const float2* u, const P2& p, float2 (&g)[2]) {
  g[0] = d_fwd(u, p.i, p.x, p.W, 1);
  g[1] = d_fwd(u, p.i, p.y, p.H, p.W);
}
AVX_D float2 div2(const float2* y0, const float2* y1, const P2& p) {
  const float2 a = cadd(d_fwd_t(y0, p.i, p.x, p.W, 1), d_fwd_t(y1, p.i, p.y, p.H, p.W));
  return make_float2(-a.x, -a.y);
}
// SymmetricGradient2D (utils.cpp:525-556): (D-x v0, D-y v1, (D-y v0 + D-x v1) / 2)
AVX_D void symgrad2(const float2* v0, const float2* v1, const P2& p, float2 (&e)[3]) {
  e[0] = d_bwd(v0, p.i, p.x, p.W, 1);
  e[1] = d_bwd(v1, p.i, p.y, p.H, p.W);
  e[2] = cadd(cscale(d_bwd(v0, p.i, p.y, p.H, p.W), 0.5f), cscale(d_bwd(v1, p.i, p.x, p.W, 1), 0.5f));
}
// SymmetricDivergence2D (utils.cpp:1078-1117)
AVX_D void symdiv2(const float2* w0, const float2* w1, const float2* w2, const P2& p, float2 (&d)[2]) {
  float2 a = cadd(d_bwd_t(w0, p.i, p.x, p.W, 1), d_bwd_t(w2, p.i, p.y, p.H, p.W));
  d[0] = make_float2(-a.x, -a.y);
  a = cadd(d_bwd_t(w2, p.i, p.x, p.W, 1), d_bwd_t(w1, p.i, p.y, p.H, p.W));
  d[1] = make_float2(-a.x, -a.y);
}

// ---------------------------------------------------------------------------
// time-averaged reconstruction
// ---------------------------------------------------------------------------

__global__ void ta_sum_kernel(const float2* kdata, const float* mask, float2* out, int HW, int C, int T) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= (long long)C * HW) return;
  const int c = (int)(i / HW), p = (int)(i % HW);
  float2 s = czero();
  float m = 0.f;
  for (int t = 0; t < T; ++t) {
    s = cadd(s, kdata[((long long)t * C + c) * HW + p]);
    m += mask ? mask[(long long)t * HW + p] : 1.f;
  }
  m = fmaxf(m, 1.f);
  out[i] = make_float2(s.x / m, s.y / m);
}

__global__ void ta_combine_kernel(float2* crec, float2* u, int HW, int C, float scale, int apply_phase) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= HW) return;
  float s = 0.f;
  float2 sum = czero();
  for (int c = 0; c < C; ++c) {
    const float2 v = cscale(crec[(long long)c * HW + p], scale);
    crec[(long long)c * HW + p] = v;
    s += cabs2(v);
    sum = cadd(sum, v);
  }
  float2 r = make_float2(sqrtf(s), 0.f);
  if (apply_phase) {
    const float ang = atan2f(sum.y, sum.x);
    r = cmul(r, make_float2(cosf(ang), sinf(ang)));
  }
  u[p] = r;
}

// ---------------------------------------------------------------------------
// H1 solve: (mu |u|^2 - Laplace_periodic) x = conj(u) mu |crec_c|, complex CG
// in FP64 (cg_forward_operation.h:47-70)
// ---------------------------------------------------------------------------

AVX_D double2 h1_apply(const double2* v, const double* muu, int x, int y, int W, int H) {
  const int i = y * W + x;
  const int xp = x + 1 == W ? 0 : x + 1, xm = x == 0 ? W - 1 : x - 1;
  const int yp = y + 1 == H ? 0 : y + 1, ym = y == 0 ? H - 1 : y - 1;
  const double2 c = v[i];
  const double2 a = v[y * W + xp], b = v[y * W + xm], d = v[yp * W + x], e = v[ym * W + x];
  const double m = muu[i] + 4.0;
  return make_double2(m * c.x - a.x - b.x - d.x - e.x, m * c.y - a.y - b.y - d.y - e.y);
}

template <int NT>
AVX_D double block_dsum(double v, double* red) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  double r = 0.0;
  for (int k = 0; k < NT / 32; ++k) r += red[k];
  return r;
}

// Each coil's system is solved by a cluster of H1_CLUSTER CTAs (contiguous
// blocks of pixels per CTA).  The vectors stay in global
// memory; the stencil reads its neighbours there after a cluster barrier
// (release/acquire at cluster scope).  Every inner product is a block sum per
// CTA, the CTA sums written into a slot of every CTA's shared memory, and one
// cluster barrier, after which each CTA adds the slots in rank order: every
// CTA holds the same value, so all take the same branch of the stopping test.
#define H1_CLUSTER 8

__global__ void __cluster_dims__(H1_CLUSTER, 1, 1) __launch_bounds__(1024)
    h1_cg_cluster_kernel(const float2* u, const float2* crec, double mu, int W, int H, int max_it, double rel_tol,
                         double2* work, double* muu_buf, float2* out, int* iters) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ double red[32];
  __shared__ double slots[2][H1_CLUSTER];  // the CTA sums of the two most recent reductions
  const int rank = (int)cl.block_rank();
  const int c = blockIdx.x / H1_CLUSTER;
  const int N = W * H;
  const int i0 = (int)((long long)N * rank / H1_CLUSTER), i1 = (int)((long long)N * (rank + 1) / H1_CLUSTER);
  double2* x = work + (size_t)c * 4 * N;
  double2* r = x + N;
  double2* p = r + N;
  double2* q = p + N;
  double* muu = muu_buf + (size_t)c * N;
  int nred = 0;
  auto csum = [&](double v) {
    v = block_dsum<1024>(v, red);
    double* buf = slots[nred & 1];
    if (threadIdx.x == 0)
      for (int k = 0; k < H1_CLUSTER; ++k) cl.map_shared_rank(buf, k)[rank] = v;
    cl.sync();
    double t = 0.0;
    for (int k = 0; k < H1_CLUSTER; ++k) t += buf[k];
    ++nred;
    return t;
  };
  double rr = 0.0;
  for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
    const float2 uu = u[i];
    const double au2 = (double)uu.x * uu.x + (double)uu.y * uu.y;
    muu[i] = mu * au2;
    const float2 cr = crec[(size_t)c * N + i];
    const double ac = mu * sqrt((double)cr.x * cr.x + (double)cr.y * cr.y);
    const double2 y = make_double2((double)uu.x * ac, -(double)uu.y * ac);
    x[i] = make_double2(0.0, 0.0);
    r[i] = y;
    p[i] = y;
    rr += y.x * y.x + y.y * y.y;
  }
  rr = csum(rr);  // the barrier also publishes p and muu to the cluster
  const double rr0 = rr;
  int it = 0;
  for (; it < max_it && rr > rel_tol * rel_tol * rr0 && rr > 0.0; ++it) {
    double pq = 0.0;
    for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
      const double2 a = h1_apply(p, muu, i % W, i / W, W, H);
      q[i] = a;
      const double2 pv = p[i];
      pq += pv.x * a.x + pv.y * a.y;
    }
    pq = csum(pq);
    const double alpha = rr / pq;
    double rn = 0.0;
    for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
      const double2 pv = p[i], qv = q[i];
      double2 xv = x[i], rv = r[i];
      xv.x += alpha * pv.x;
      xv.y += alpha * pv.y;
      rv.x -= alpha * qv.x;
      rv.y -= alpha * qv.y;
      x[i] = xv;
      r[i] = rv;
      rn += rv.x * rv.x + rv.y * rv.y;
    }
    rn = csum(rn);
    const double beta = rn / rr;
    rr = rn;
    for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
      const double2 rv = r[i], pv = p[i];
      p[i] = make_double2(rv.x + beta * pv.x, rv.y + beta * pv.y);
    }
    cl.sync();  // the new p before any CTA applies the stencil to it
  }
  for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) out[(size_t)c * N + i] = make_float2((float)x[i].x, (float)x[i].y);
  if (rank == 0 && threadIdx.x == 0 && iters) iters[c] = it;
}


// The same solve with the vectors on chip, for images whose block of rows a
// CTA holds at PX pixels a thread: x, r, q and the diagonal in registers, p in
// shared memory with one halo row above and below, which the neighbouring
// CTAs write.  In global memory an iteration's three phases each waited for
// L2 (12 coils of 128 x 128: 5.2 ms, FP64 pipe 9 % active; here 2.4 ms, the
// cluster barriers of the two reductions and the stencil).
template <int PX>
__global__ void __launch_bounds__(1024)
    h1_cg_resident_kernel(const float2* u, const float2* crec, double mu, int W, int H, int max_it, double rel_tol,
                          float2* out, int* iters, int rows_max) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* p = reinterpret_cast<double2*>(smem_raw);  // [rows_max + 2][W]
  __shared__ double red[32];
  __shared__ double slots[2][H1_CLUSTER];
  const int rank = (int)cl.block_rank();
  const int c = blockIdx.x / H1_CLUSTER;
  const int y0 = (int)((long long)H * rank / H1_CLUSTER), y1 = (int)((long long)H * (rank + 1) / H1_CLUSTER);
  const int n = (y1 - y0) * W;
  const int up = rank == 0 ? H1_CLUSTER - 1 : rank - 1, down = rank + 1 == H1_CLUSTER ? 0 : rank + 1;  // periodic
  const int up_rows = (int)((long long)H * (up + 1) / H1_CLUSTER) - (int)((long long)H * up / H1_CLUSTER);
  double2* p_up = cl.map_shared_rank(p, up) + (size_t)(up_rows + 1) * W;  // lower halo of the CTA above
  double2* p_down = cl.map_shared_rank(p, down);                          // upper halo of the CTA below
  int nred = 0;
  auto csum = [&](double v) {
    v = block_dsum<1024>(v, red);
    double* buf = slots[nred & 1];
    if (threadIdx.x < H1_CLUSTER) cl.map_shared_rank(buf, threadIdx.x)[rank] = v;
    cl.sync();
    double t = 0.0;
    for (int k = 0; k < H1_CLUSTER; ++k) t += buf[k];
    ++nred;
    return t;
  };
  auto put = [&](int idx, double2 v) {
    p[idx + W] = v;
    if (idx < W) p_up[idx] = v;
    if (idx >= n - W) p_down[idx - (n - W)] = v;
  };
  double2 x[PX], r[PX], q[PX];
  double m[PX];
  int xl[PX], xr[PX];  // horizontal neighbours, wrapped
  double rr = 0.0;
  cl.sync();  // every CTA of the cluster runs before its shared memory is written
#pragma unroll
  for (int k = 0; k < PX; ++k) {
    const int idx = threadIdx.x + k * 1024;
    x[k] = r[k] = q[k] = make_double2(0.0, 0.0);
    m[k] = 0.0;
    xl[k] = xr[k] = 0;
    if (idx < n) {
      const int i = y0 * W + idx, px = idx % W;
      xl[k] = px == 0 ? idx + W - 1 : idx - 1;
      xr[k] = px + 1 == W ? idx - (W - 1) : idx + 1;
      const float2 uu = u[i];
      const double au2 = (double)uu.x * uu.x + (double)uu.y * uu.y;
      m[k] = mu * au2 + 4.0;
      const float2 cr = crec[(size_t)c * W * H + i];
      const double ac = mu * sqrt((double)cr.x * cr.x + (double)cr.y * cr.y);
      r[k] = make_double2((double)uu.x * ac, -(double)uu.y * ac);
      put(idx, r[k]);
      rr += r[k].x * r[k].x + r[k].y * r[k].y;
    }
  }
  rr = csum(rr);  // the barrier also publishes p to the cluster
  const double rr0 = rr;
  int it = 0;
  for (; it < max_it && rr > rel_tol * rel_tol * rr0 && rr > 0.0; ++it) {
    double pq = 0.0;
#pragma unroll
    for (int k = 0; k < PX; ++k) {
      const int idx = threadIdx.x + k * 1024;
      if (idx < n) {
        const double2 pc = p[idx + W], a = p[xr[k] + W], b = p[xl[k] + W], d = p[idx + 2 * W], e = p[idx];
        q[k] = make_double2(m[k] * pc.x - a.x - b.x - d.x - e.x, m[k] * pc.y - a.y - b.y - d.y - e.y);
        pq += pc.x * q[k].x + pc.y * q[k].y;
      }
    }
    pq = csum(pq);
    const double alpha = rr / pq;
    double rn = 0.0;
#pragma unroll
    for (int k = 0; k < PX; ++k) {
      const int idx = threadIdx.x + k * 1024;
      if (idx < n) {
        const double2 pc = p[idx + W];
        x[k].x += alpha * pc.x;
        x[k].y += alpha * pc.y;
        r[k].x -= alpha * q[k].x;
        r[k].y -= alpha * q[k].y;
        rn += r[k].x * r[k].x + r[k].y * r[k].y;
      }
    }
    rn = csum(rn);
    const double beta = rn / rr;
    rr = rn;
#pragma unroll
    for (int k = 0; k < PX; ++k) {
      const int idx = threadIdx.x + k * 1024;
      if (idx < n) {
        const double2 pc = p[idx + W];
        put(idx, make_double2(r[k].x + beta * pc.x, r[k].y + beta * pc.y));
      }
    }
    cl.sync();  // the new p before any CTA applies the stencil to it
  }
#pragma unroll
  for (int k = 0; k < PX; ++k) {
    const int idx = threadIdx.x + k * 1024;
    if (idx < n) out[(size_t)c * W * H + y0 * W + idx] = make_float2((float)x[k].x, (float)x[k].y);
  }
  if (rank == 0 && threadIdx.x == 0 && iters) iters[c] = it;
}

// b1 <- |b1_c / sqrt(sum_c |b1_c|^2)| (coil_construction.cpp:428-444)
__global__ void h1_normalize_kernel(float2* b1, int HW, int C) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= HW) return;
  float s = 0.f;
  for (int c = 0; c < C; ++c) s += cabs2(b1[(long long)c * HW + p]);
  const float n = sqrtf(s);
  for (int c = 0; c < C; ++c) {
    const float2 v = b1[(long long)c * HW + p];
    const float2 w = make_float2(v.x / n, v.y / n);
    b1[(long long)c * HW + p] = make_float2(sqrtf(cabs2(w)), 0.f);
  }
}

// ---------------------------------------------------------------------------
// UTGV2Recon (coil_construction.cpp:75-215)
// ---------------------------------------------------------------------------

__global__ void utgv_prep_kernel(const float2* b10, const float2* crec0, const int* inds, int ninds, float tau, int HW,
                                 float2* Lw, float2* Ib) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= HW) return;
  float2 lw = czero(), sb = czero();
  for (int k = 0; k < ninds; ++k) {
    const float2 b = b10[(long long)inds[k] * HW + p];
    const float2 cr = crec0[(long long)inds[k] * HW + p];
    lw = cadd(lw, cmulc(b, cr));
    sb = cadd(sb, cmulc(b, b));
  }
  Lw[p] = lw;
  // Ib = 1 / (1 + tau sumB1) (complex division of 1 by a real-valued complex)
  const float2 den = make_float2(1.f + tau * sb.x, tau * sb.y);
  const float dd = cabs2(den);
  Ib[p] = make_float2(den.x / dd, -den.y / dd);
}

// One UTGV2Recon iteration (coil_construction.cpp:75-215) in one kernel: the
// dual update (y1 += sigma (grad x1bar - x2bar), y2 += sigma E x2bar, each
// projected onto its ball) at this pixel and at the neighbours the primal
// update reads (the divergence: x - 1, y - W; the symmetrised divergence:
// x + 1, y + W), recomputed from the old extragradients and duals, then the
// primal update (x1 <- (x1 + tau (div y1 + Lw)) Ib, x2 += tau (y1 + div_sym
// y2), extragradients 2 new - old).  The extragradients and the duals are
// double-buffered; x1 and x2 are updated in place by their own thread.
__global__ void utgv_fused_kernel(CoilPD a, UtgvBuffers b) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= a.W * a.H) return;
  const P2 p = p2_of(idx, a.W, a.H);
  // the dual update at pixel (qx, qy)
  auto dual = [&](int qx, int qy, float2 (&y1)[2], float2 (&y2)[3]) {
    P2 q;
    q.x = qx;
    q.y = qy;
    q.W = a.W;
    q.H = a.H;
    q.i = (long long)qy * a.W + qx;
    float2 g[2], e[3];
    grad2(b.ext1_in, q, g);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const float2 d = csub(g[k], ldc(b.ext2_in[k], q.i));
      const float2 v = ldc(b.y1_in[k], q.i);
      y1[k] = make_float2(v.x + a.sigma * d.x, v.y + a.sigma * d.y);
    }
    symgrad2(b.ext2_in[0], b.ext2_in[1], q, e);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float2 v = ldc(b.y2_in[k], q.i);
      y2[k] = make_float2(v.x + a.sigma * e[k].x, v.y + a.sigma * e[k].y);
    }
    const float n1 = sqrtf(cabs2(y1[0]) + cabs2(y1[1]));
    const float n2 = sqrtf(cabs2(y2[0]) + cabs2(y2[1]) + 2.f * cabs2(y2[2]));
    const float d1 = fmaxf(1.f, a.s1 * n1), d2 = fmaxf(1.f, a.s2 * n2);
#pragma unroll
    for (int k = 0; k < 2; ++k) y1[k] = make_float2(y1[k].x / d1, y1[k].y / d1);
#pragma unroll
    for (int k = 0; k < 3; ++k) y2[k] = make_float2(y2[k].x / d2, y2[k].y / d2);
  };
  float2 y1[2], y2[3];
  dual(p.x, p.y, y1, y2);
#pragma unroll
  for (int k = 0; k < 2; ++k) b.y1_out[k][idx] = y1[k];
#pragma unroll
  for (int k = 0; k < 3; ++k) b.y2_out[k][idx] = y2[k];
  float2 n1[2], n2[3];
  // div2 (d_fwd_t along x of y1_0, along y of y1_1), negated
  float2 xm = czero(), ym = czero();
  if (p.x > 0) {
    dual(p.x - 1, p.y, n1, n2);
    xm = n1[0];
  }
  if (p.y > 0) {
    dual(p.x, p.y - 1, n1, n2);
    ym = n1[1];
  }
  const float2 ax = csub(xm, p.x < a.W - 1 ? y1[0] : czero());
  const float2 ay = csub(ym, p.y < a.H - 1 ? y1[1] : czero());
  const float2 s2 = cadd(ax, ay);
  const float2 dv = make_float2(-s2.x, -s2.y);
  const float2 xo = a.x1[idx];
  float2 x1n = make_float2(xo.x + a.tau * dv.x, xo.y + a.tau * dv.y);
  const float2 lw = a.Lw[idx];
  x1n = make_float2(x1n.x + a.tau * lw.x, x1n.y + a.tau * lw.y);
  x1n = cmul(x1n, a.Ib[idx]);
  a.x1[idx] = x1n;
  b.ext1_out[idx] = make_float2(2.f * x1n.x - xo.x, 2.f * x1n.y - xo.y);
  // symdiv2 (d_bwd_t: w0 and w2 along x, w2 and w1 along y), negated
  float2 w0p = czero(), w2x = czero(), w2y = czero(), w1p = czero();
  if (p.x < a.W - 1) {
    dual(p.x + 1, p.y, n1, n2);
    w0p = n2[0];
    w2x = n2[2];
  }
  if (p.y < a.H - 1) {
    dual(p.x, p.y + 1, n1, n2);
    w1p = n2[1];
    w2y = n2[2];
  }
  const float2 z = czero();
  float2 sd[2];
  float2 t0 = cadd(p.x < a.W - 1 ? csub(y2[0], w0p) : z, p.y < a.H - 1 ? csub(y2[2], w2y) : z);
  sd[0] = make_float2(-t0.x, -t0.y);
  t0 = cadd(p.x < a.W - 1 ? csub(y2[2], w2x) : z, p.y < a.H - 1 ? csub(y2[1], w1p) : z);
  sd[1] = make_float2(-t0.x, -t0.y);
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float2 r = cadd(y1[k], sd[k]);
    const float2 x2 = a.x2[k][idx];
    const float2 m = make_float2(x2.x + a.tau * r.x, x2.y + a.tau * r.y);
    a.x2[k][idx] = m;
    b.ext2_out[k][idx] = make_float2(2.f * m.x - x2.x, 2.f * m.y - x2.y);
  }
}

// ---------------------------------------------------------------------------
// B1Recon (coil_construction.cpp:217-361)
// ---------------------------------------------------------------------------

__global__ void absmax_kernel(const float2* v, int n, unsigned* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  float m = 0.f;
  if (i < n) m = sqrtf(cabs2(v[i]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
  // non-negative floats order like their bit patterns
  if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(m));
}

__global__ void b1r_prep_kernel(const float2* u0, const unsigned* umax, const float2* crec, int coils, int HW,
                                float tau, float2* Lw, float2* Iu) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= HW) return;
  const float mx = __uint_as_float(*umax);
  const float2 un = make_float2(u0[p].x / mx, u0[p].y / mx);
  const float2 sumU = make_float2(1.f + tau * cabs2(un), 0.f);
  const float2 iu = make_float2(1.f / sumU.x, 0.f);
  for (int c = 0; c < coils; ++c) {
    Lw[(long long)c * HW + p] = cmulc(un, crec[(long long)c * HW + p]);
    Iu[(long long)c * HW + p] = iu;
  }
}

// One B1Recon iteration (coil_construction.cpp:217-361) in one kernel: the
// dual update (y = (y + sigma grad xbar) / (1 + sigma / mu)) at this pixel and
// at the neighbours the divergence reads (x - 1 for the x component, x - W for
// the y component), recomputed from the old extragradient and duals, then the
// primal update (x <- (x + tau (div y + Lw)) Iu, extragradient 2 new - old).
// The extragradient and the duals are double-buffered (neighbouring threads
// read the old values while the owner writes the new ones); x is updated in
// place (read and written by its own thread only).
__global__ void b1r_fused_kernel(CoilPD a, int coils, B1Buffers b) {
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int HW = a.W * a.H;
  if (idx >= (long long)coils * HW) return;
  const int c = (int)(idx / HW);
  const int pix = (int)(idx % HW);
  const P2 p = p2_of(pix, a.W, a.H);
  const long long cb = (long long)c * HW;
  const float2* e = b.ext_in + cb;
  const float sc = 1.f / (1.f + a.sigma / a.mu);
  // dual component k at coil pixel q
  auto dual = [&](int k, int qx, int qy) {
    const long long q = (long long)qy * a.W + qx;
    const float2 g = k == 0 ? d_fwd(e, q, qx, a.W, 1) : d_fwd(e, q, qy, a.H, a.W);
    const float2 v = (k == 0 ? b.y0_in : b.y1_in)[cb + q];
    return cscale(make_float2(v.x + a.sigma * g.x, v.y + a.sigma * g.y), sc);
  };
  const float2 y0 = dual(0, p.x, p.y), y1 = dual(1, p.x, p.y);
  b.y0_out[idx] = y0;
  b.y1_out[idx] = y1;
  // divergence (div2 of coils.cu) from the new duals
  const float2 y0m = p.x > 0 ? dual(0, p.x - 1, p.y) : czero();
  const float2 y1m = p.y > 0 ? dual(1, p.x, p.y - 1) : czero();
  const float2 ax = csub(y0m, p.x < a.W - 1 ? y0 : czero());
  const float2 ay = csub(y1m, p.y < a.H - 1 ? y1 : czero());
  const float2 s2 = cadd(ax, ay);
  const float2 dv = make_float2(-s2.x, -s2.y);
  const float2 xo = a.x1[idx];
  float2 n1 = make_float2(xo.x + a.tau * dv.x, xo.y + a.tau * dv.y);
  const float2 lw = a.Lw[idx];
  n1 = cmul(make_float2(n1.x + a.tau * lw.x, n1.y + a.tau * lw.y), a.Ib[idx]);
  a.x1n[idx] = n1;
  b.ext_out[idx] = make_float2(2.f * n1.x - xo.x, 2.f * n1.y - xo.y);
}

__global__ void b1r_normalize_kernel(const float2* x, float2* out, int HW, int coils) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= HW) return;
  float s = 0.f;
  for (int c = 0; c < coils; ++c) s += cabs2(x[(long long)c * HW + p]);
  const float n = sqrtf(s);
  for (int c = 0; c < coils; ++c) {
    const float2 v = x[(long long)c * HW + p];
    out[(long long)c * HW + p] = make_float2(v.x / n, v.y / n);
  }
}

// b1 = |absb1| * exp(i angle(x1))
__global__ void phase_apply_kernel(const float2* absb1, const float2* x1, float2* out, int HW) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= HW) return;
  const float ang = atan2f(x1[p].y, x1[p].x);
  out[p] = cmul(absb1[p], make_float2(cosf(ang), sinf(ang)));
}

// w = sqrt(w*w + conj(b) b); crec_abs products and sums for the greedy order
__global__ void weight_update_kernel(float2* w, const float2* b, int HW) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= HW) return;
  const float2 ww = cmul(w[p], w[p]);
  const float2 s = cadd(ww, cmulc(b[p], b[p]));
  // complex square root of a value with zero imaginary part here
  const float r = sqrtf(sqrtf(cabs2(s)));
  const float th = 0.5f * atan2f(s.y, s.x);
  w[p] = make_float2(r * cosf(th), r * sinf(th));
}

// u_in = absb1 * u * w; crec_in = crec * w
__global__ void greedy_inputs_kernel(const float2* absb1, const float2* u, const float2* w, const float2* crec,
                                     float2* u_in, float2* crec_in, int HW) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= HW) return;
  u_in[p] = cmul(cmul(absb1[p], u[p]), w[p]);
  crec_in[p] = cmul(crec[p], w[p]);
}

// FP64 sums over a coil image of |a| (b == null) or |a| |b|
__global__ void abs_sum_kernel(const float2* a, const float2* b, int HW, double* partial) {
  __shared__ double red[32];
  double acc[1] = {0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < HW; i += gridDim.x * blockDim.x) {
    float v = sqrtf(cabs2(a[i]));
    if (b) v *= sqrtf(cabs2(b[i]));
    acc[0] += (double)v;
  }
  block_sum<1>(acc, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = acc[0];
}

// ---------------------------------------------------------------------------
// Whole loops in one launch.  A coil image is cut into blocks of rows, one per
// CTA of a cluster; the fields live in registers and shared memory, boundary
// rows are written into the neighbouring CTAs' shared memory, and one (B1) or
// two (UTGV2) cluster barriers order an iteration.  The loops are thousands of
// iterations over one or a few 128 x 128 images: as one kernel per iteration
// they cost 4.5 us each, almost all of it launch and L2 latency; a cluster
// loop with the fields in global memory was no faster.  At 128 x 128 a B1
// iteration of one coil takes 0.85 us here (16 CTAs), of 12 coils 1.2 us (8
// CTAs each), a UTGV2 iteration 3.6 us: bound by the barriers and the chain of
// loads, roots and divisions between them on 16 SMs (packed arithmetic changed
// nothing; storing after all pixels were computed was slower, 4.1).
// ---------------------------------------------------------------------------

#define COIL_NT 512  // threads per CTA: up to 128 registers each for the pixels they hold

struct CoilTile {
  int W, H, y0, n, rank, size;  // image, first row, pixels of this CTA, rank in the cluster
};
AVX_D CoilTile coil_tile(int W, int H) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  CoilTile t;
  t.W = W;
  t.H = H;
  t.rank = (int)cl.block_rank();
  t.size = (int)cl.num_blocks();
  t.y0 = (int)((long long)H * t.rank / t.size);
  t.n = ((int)((long long)H * (t.rank + 1) / t.size) - t.y0) * W;
  return t;
}
// writes v at pixel idx of the CTA's block into field f ([rows + 2][W], one
// halo row above and below) and, on boundary rows, into the neighbours' halos
template <bool UP, bool DOWN>
AVX_D void coil_put(const CoilTile& t, float2* f, int idx, float2 v) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  f[idx + t.W] = v;
  if (UP && idx < t.W && t.rank > 0) {  // first row: the lower halo of the CTA above
    const int above = (t.y0 - (int)((long long)t.H * (t.rank - 1) / t.size)) * t.W;
    cl.map_shared_rank(f, t.rank - 1)[idx + above + t.W] = v;
  }
  if (DOWN && idx >= t.n - t.W && t.rank + 1 < t.size)  // last row: the upper halo of the CTA below
    cl.map_shared_rank(f, t.rank + 1)[idx - (t.n - t.W)] = v;
}

// B1Recon's loop (the arithmetic of b1r_fused_kernel): the extragradient is
// double-buffered in shared memory; each thread also carries the two
// neighbouring dual values its divergence reads (left and upper), which it
// recomputes from the same inputs as their owner does.
template <int PX>
__global__ void __launch_bounds__(COIL_NT) b1r_cluster_kernel(CoilPD a, unsigned iters, int rows_max) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  namespace cg = cooperative_groups;
  const CoilTile t = coil_tile(a.W, a.H);
  const int W = a.W, field = (rows_max + 2) * W;
  float2* ext = reinterpret_cast<float2*>(smem_raw);  // [2][rows_max + 2][W]
  const long long cb = (long long)(blockIdx.x / t.size) * a.W * a.H + (long long)t.y0 * W;
  for (int e = threadIdx.x; e < 2 * field; e += COIL_NT) ext[e] = czero();
  float2 x[PX], y0[PX], y0l[PX], y1[PX], y1u[PX], lw[PX], ib[PX];
  unsigned at[PX];  // pixel index, bits 28..31: has a right, lower, left, upper neighbour
#pragma unroll
  for (int k = 0; k < PX; ++k) {
    const int idx = threadIdx.x + k * COIL_NT;
    x[k] = y0[k] = y0l[k] = y1[k] = y1u[k] = lw[k] = ib[k] = czero();
    at[k] = 0u;
    if (idx < t.n) {
      const int px = idx % W, py = t.y0 + idx / W;
      at[k] = (unsigned)idx | (px < W - 1 ? 1u << 28 : 0u) | (py < a.H - 1 ? 1u << 29 : 0u) | (px > 0 ? 1u << 30 : 0u) |
              (py > 0 ? 1u << 31 : 0u);
      lw[k] = a.Lw[cb + idx];
      ib[k] = a.Ib[cb + idx];
    }
  }
  const float sc = 1.f / (1.f + a.sigma / a.mu);
  cg::this_cluster().sync();
  for (unsigned it = 0; it < iters; ++it) {
    const float2* e = ext + (it & 1u) * field + W;
    float2* en = ext + ((it + 1u) & 1u) * field;
#pragma unroll
    for (int k = 0; k < PX; ++k) {
      const int idx = (int)(at[k] & 0x0FFFFFFFu);
      if ((int)threadIdx.x + k * COIL_NT < t.n) {
        const bool r = at[k] & 1u << 28, d = at[k] & 1u << 29, l = at[k] & 1u << 30, u = at[k] & 1u << 31;
        const float2 c = e[idx];
        auto dual = [&](float2 y, float2 g) {
          return scale2(fma2(make_float2(a.sigma, a.sigma), g, y), sc);
        };
        y0[k] = dual(y0[k], r ? sub2(e[idx + 1], c) : czero());
        y1[k] = dual(y1[k], d ? sub2(e[idx + W], c) : czero());
        if (l) y0l[k] = dual(y0l[k], sub2(c, e[idx - 1]));
        if (u) y1u[k] = dual(y1u[k], sub2(c, e[idx - W]));
        const float2 ax = sub2(y0l[k], r ? y0[k] : czero());
        const float2 ay = sub2(y1u[k], d ? y1[k] : czero());
        const float2 s2 = add2(ax, ay);
        const float2 dv = make_float2(-s2.x, -s2.y);
        const float2 xo = x[k];
        float2 n1 = fma2(make_float2(a.tau, a.tau), dv, xo);
        n1 = cmul(fma2(make_float2(a.tau, a.tau), lw[k], n1), ib[k]);
        x[k] = n1;
        coil_put<true, true>(t, en, idx, fma2(make_float2(2.f, 2.f), n1, make_float2(-xo.x, -xo.y)));
      }
    }
    cg::this_cluster().sync();
  }
#pragma unroll
  for (int k = 0; k < PX; ++k) {
    const int idx = threadIdx.x + k * COIL_NT;
    if (idx < t.n) a.x1[cb + idx] = x[k];
  }
}

// UTGV2Recon's loop (the arithmetic of utgv_fused_kernel): extragradients and
// duals in shared memory, the duals written before a first barrier, the
// primal update and its extragradients before a second.
template <int PX>
__global__ void __launch_bounds__(COIL_NT) utgv_cluster_kernel(CoilPD a, unsigned iters, int rows_max) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  namespace cg = cooperative_groups;
  const CoilTile t = coil_tile(a.W, a.H);
  const int W = a.W, field = (rows_max + 2) * W;
  float2* f = reinterpret_cast<float2*>(smem_raw);  // ext1, ext2[2], y1[2], y2[3], each [rows_max + 2][W]
  float2 *ext1 = f, *e20 = f + field, *e21 = f + 2 * field;
  float2 *s10 = f + 3 * field, *s11 = f + 4 * field, *s20 = f + 5 * field, *s21 = f + 6 * field, *s22 = f + 7 * field;
  const long long cb = (long long)t.y0 * W;
  for (int e = threadIdx.x; e < 8 * field; e += COIL_NT) f[e] = czero();
  cg::this_cluster().sync();
  float2 x1[PX], x20[PX], x21[PX], y10[PX], y11[PX], y20[PX], y21[PX], y22[PX], lw[PX], ib[PX];
  bool right[PX], low[PX], left[PX], up[PX];  // has that neighbour
#pragma unroll
  for (int k = 0; k < PX; ++k) {
    const int idx = threadIdx.x + k * COIL_NT;
    const int px = idx % W, py = t.y0 + idx / W;
    right[k] = px < W - 1;
    low[k] = py < a.H - 1;
    left[k] = px > 0;
    up[k] = py > 0;
    x1[k] = x20[k] = x21[k] = y10[k] = y11[k] = y20[k] = y21[k] = y22[k] = lw[k] = ib[k] = czero();
    if (idx < t.n) {
      x1[k] = a.x1[cb + idx];
      lw[k] = a.Lw[cb + idx];
      ib[k] = a.Ib[cb + idx];
      coil_put<true, true>(t, ext1, idx, x1[k]);
    }
  }
  cg::this_cluster().sync();
  for (unsigned it = 0; it < iters; ++it) {
#pragma unroll
    for (int k = 0; k < PX; ++k) {
      const int idx = threadIdx.x + k * COIL_NT;
      if (idx < t.n) {
        const int i = idx + W;
        const bool r = right[k], d = low[k], l = left[k], u = up[k];
        const float2 z = czero(), c = ext1[i], p0 = e20[i], p1 = e21[i];
        // y1 += sigma (grad x1bar - x2bar)
        const float2 g0 = sub2(r ? sub2(ext1[i + 1], c) : z, p0), g1 = sub2(d ? sub2(ext1[i + W], c) : z, p1);
        float2 a0 = fma2(make_float2(a.sigma, a.sigma), g0, y10[k]);
        float2 a1 = fma2(make_float2(a.sigma, a.sigma), g1, y11[k]);
        const float d1 = a.s1 * sqrtf(cabs2(a0) + cabs2(a1));
        if (d1 > 1.f) {  // outside the ball
          a0 = make_float2(a0.x / d1, a0.y / d1);
          a1 = make_float2(a1.x / d1, a1.y / d1);
        }
        y10[k] = a0;
        y11[k] = a1;
        // y2 += sigma E x2bar (backward differences)
        const float2 p0r = r ? p0 : z, p0d = d ? p0 : z, p1r = r ? p1 : z, p1d = d ? p1 : z;
        const float2 p0l = l ? e20[i - 1] : z, p0u = u ? e20[i - W] : z, p1l = l ? e21[i - 1] : z, p1u = u ? e21[i - W] : z;
        const float2 b0 = sub2(p0r, p0l), b1 = sub2(p1d, p1u);
        const float2 b2 = add2(scale2(sub2(p0d, p0u), 0.5f), scale2(sub2(p1r, p1l), 0.5f));
        float2 q0 = fma2(make_float2(a.sigma, a.sigma), b0, y20[k]);
        float2 q1 = fma2(make_float2(a.sigma, a.sigma), b1, y21[k]);
        float2 q2 = fma2(make_float2(a.sigma, a.sigma), b2, y22[k]);
        const float d2 = a.s2 * sqrtf(cabs2(q0) + cabs2(q1) + 2.f * cabs2(q2));
        if (d2 > 1.f) {
          q0 = make_float2(q0.x / d2, q0.y / d2);
          q1 = make_float2(q1.x / d2, q1.y / d2);
          q2 = make_float2(q2.x / d2, q2.y / d2);
        }
        y20[k] = q0;
        y21[k] = q1;
        y22[k] = q2;
        s10[i] = y10[k];
        coil_put<false, true>(t, s11, idx, y11[k]);  // read by the row below
        s20[i] = y20[k];
        coil_put<true, false>(t, s21, idx, y21[k]);  // read by the row above
        coil_put<true, false>(t, s22, idx, y22[k]);
      }
    }
    cg::this_cluster().sync();
#pragma unroll
    for (int k = 0; k < PX; ++k) {
      const int idx = threadIdx.x + k * COIL_NT;
      if (idx < t.n) {
        const int i = idx + W;
        const bool r = right[k], d = low[k], l = left[k], u = up[k];
        const float2 z = czero();
        const float2 ax = sub2(l ? s10[i - 1] : z, r ? y10[k] : z), ay = sub2(u ? s11[i - W] : z, d ? y11[k] : z);
        const float2 s2 = add2(ax, ay);
        const float2 dv = make_float2(-s2.x, -s2.y);
        const float2 xo = x1[k];
        float2 n1 = fma2(make_float2(a.tau, a.tau), dv, xo);
        n1 = fma2(make_float2(a.tau, a.tau), lw[k], n1);
        n1 = cmul(n1, ib[k]);
        x1[k] = n1;
        coil_put<true, false>(t, ext1, idx, fma2(make_float2(2.f, 2.f), n1, make_float2(-xo.x, -xo.y)));  // read by the row above
        // x2 += tau (y1 + div_sym y2)
        float2 t0 = add2(r ? sub2(y20[k], s20[i + 1]) : z, d ? sub2(y22[k], s22[i + W]) : z);
        const float2 sd0 = make_float2(-t0.x, -t0.y);
        t0 = add2(r ? sub2(y22[k], s22[i + 1]) : z, d ? sub2(y21[k], s21[i + W]) : z);
        const float2 sd1 = make_float2(-t0.x, -t0.y);
        const float2 r0 = add2(y10[k], sd0), r1 = add2(y11[k], sd1);
        const float2 o0 = x20[k], o1 = x21[k];
        const float2 m0 = fma2(make_float2(a.tau, a.tau), r0, o0);
        const float2 m1 = fma2(make_float2(a.tau, a.tau), r1, o1);
        x20[k] = m0;
        x21[k] = m1;
        coil_put<false, true>(t, e20, idx, fma2(make_float2(2.f, 2.f), m0, make_float2(-o0.x, -o0.y)));
        coil_put<false, true>(t, e21, idx, fma2(make_float2(2.f, 2.f), m1, make_float2(-o1.x, -o1.y)));
      }
    }
    cg::this_cluster().sync();
  }
#pragma unroll
  for (int k = 0; k < PX; ++k) {
    const int idx = threadIdx.x + k * COIL_NT;
    if (idx < t.n) a.x1[cb + idx] = x1[k];
  }
}

static inline unsigned nb256(long long n) { return (unsigned)((n + 255) / 256); }

void launch_ta_sum(const float2* kdata, const float* mask, float2* out, int HW, int C, int T, cudaStream_t s) {
  ta_sum_kernel<<<nb256((long long)C * HW), 256, 0, s>>>(kdata, mask, out, HW, C, T);
}
void launch_ta_combine(float2* crec, float2* u, int HW, int C, float scale, int apply_phase, cudaStream_t s) {
  ta_combine_kernel<<<nb256(HW), 256, 0, s>>>(crec, u, HW, C, scale, apply_phase);
}
void launch_h1_cg(const float2* u, const float2* crec, double mu, int W, int H, int C, int max_it, double rel_tol,
                  double2* work, double* muu, float2* out, int* iters, cudaStream_t s) {
  const int rows = (H + H1_CLUSTER - 1) / H1_CLUSTER;
  const int px = (rows * W + 1023) / 1024;
  const size_t sm = sizeof(double2) * (size_t)(rows + 2) * W;
  if (H >= H1_CLUSTER && W > 1 && px <= 2 && sm <= 200 * 1024) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C * H1_CLUSTER);
    cfg.blockDim = dim3(1024);
    cfg.dynamicSmemBytes = sm;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = H1_CLUSTER;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    auto kernel = px == 1 ? h1_cg_resident_kernel<1> : h1_cg_resident_kernel<2>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaLaunchKernelEx(&cfg, kernel, u, crec, mu, W, H, max_it, rel_tol, out, iters, rows);
    return;
  }
  h1_cg_cluster_kernel<<<C * H1_CLUSTER, 1024, 0, s>>>(u, crec, mu, W, H, max_it, rel_tol, work, muu, out, iters);
}
void launch_h1_normalize(float2* b1, int HW, int C, cudaStream_t s) {
  h1_normalize_kernel<<<nb256(HW), 256, 0, s>>>(b1, HW, C);
}
void launch_utgv_prep(const float2* b10, const float2* crec0, const int* inds, int ninds, float tau, int HW,
                      float2* Lw, float2* Ib, cudaStream_t s) {
  utgv_prep_kernel<<<nb256(HW), 256, 0, s>>>(b10, crec0, inds, ninds, tau, HW, Lw, Ib);
}
void launch_utgv_fused(const CoilPD& a, const UtgvBuffers& b, cudaStream_t s) {
  utgv_fused_kernel<<<nb256((long long)a.W * a.H), 256, 0, s>>>(a, b);
}
void launch_absmax(const float2* v, int n, unsigned* out, cudaStream_t s) {
  absmax_kernel<<<nb256(n), 256, 0, s>>>(v, n, out);
}
void launch_b1r_prep(const float2* u0, const unsigned* umax, const float2* crec, int coils, int HW, float tau,
                     float2* Lw, float2* Iu, cudaStream_t s) {
  b1r_prep_kernel<<<nb256(HW), 256, 0, s>>>(u0, umax, crec, coils, HW, tau, Lw, Iu);
}
void launch_b1r_fused(const CoilPD& a, int coils, const B1Buffers& b, cudaStream_t s) {
  const long long n = (long long)coils * a.W * a.H;
  b1r_fused_kernel<<<nb256(n), 256, 0, s>>>(a, coils, b);
}
// launches kernel PX of `kernels` (pixels a thread holds, 1 .. n) for an image
// cut over `size` CTAs; false when it does not fit
template <class K, size_t N>
static bool launch_coil_cluster(K (&kernels)[N], const CoilPD& a, int coils, unsigned iters, int fields, int size,
                                cudaStream_t s) {
  if (a.H < size) return false;
  const int rows = (a.H + size - 1) / size;
  const int px = (rows * a.W + COIL_NT - 1) / COIL_NT;
  const size_t sm = sizeof(float2) * (size_t)fields * (rows + 2) * a.W;
  if (px > (int)N || sm > AVX_DYN_SMEM_MAX) return false;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(coils * size);
  cfg.blockDim = dim3(COIL_NT);
  cfg.dynamicSmemBytes = sm;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = size;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const K kernel = kernels[px - 1];
  int fits = 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AVX_DYN_SMEM_MAX) != cudaSuccess ||
      cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&fits, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();  // a cluster this large cannot be resident on this device
    return false;
  }
  if (fits < 1) return false;
  if (cudaLaunchKernelEx(&cfg, kernel, a, iters, rows) == cudaSuccess) return true;
  cudaGetLastError();
  return false;
}

static void (*const kB1Cluster[])(CoilPD, unsigned, int) = {b1r_cluster_kernel<1>, b1r_cluster_kernel<2>,
                                                            b1r_cluster_kernel<3>, b1r_cluster_kernel<4>,
                                                            b1r_cluster_kernel<5>, b1r_cluster_kernel<6>};
static void (*const kUtgvCluster[])(CoilPD, unsigned, int) = {utgv_cluster_kernel<1>, utgv_cluster_kernel<2>,
                                                              utgv_cluster_kernel<3>, utgv_cluster_kernel<4>};

// A single image is spread over 16 CTAs where the device holds such a cluster
// (half the pixels per CTA of a portable one, and the other SMs idle anyway),
// several coils over 8 each, so that 16 coils run at once.
bool launch_b1r_cluster(const CoilPD& a, int coils, unsigned iters, cudaStream_t s) {
  return (coils == 1 && launch_coil_cluster(kB1Cluster, a, coils, iters, 2, 16, s)) ||
         launch_coil_cluster(kB1Cluster, a, coils, iters, 2, 8, s);
}
bool launch_utgv_cluster(const CoilPD& a, unsigned iters, cudaStream_t s) {
  return launch_coil_cluster(kUtgvCluster, a, 1, iters, 8, 16, s) ||
         launch_coil_cluster(kUtgvCluster, a, 1, iters, 8, 8, s);
}

void launch_b1r_normalize(const float2* x, float2* out, int HW, int coils, cudaStream_t s) {
  b1r_normalize_kernel<<<nb256(HW), 256, 0, s>>>(x, out, HW, coils);
}
void launch_phase_apply(const float2* absb1, const float2* x1, float2* out, int HW, cudaStream_t s) {
  phase_apply_kernel<<<nb256(HW), 256, 0, s>>>(absb1, x1, out, HW);
}
void launch_weight_update(float2* w, const float2* b, int HW, cudaStream_t s) {
  weight_update_kernel<<<nb256(HW), 256, 0, s>>>(w, b, HW);
}
void launch_greedy_inputs(const float2* absb1, const float2* u, const float2* w, const float2* crec, float2* u_in,
                          float2* crec_in, int HW, cudaStream_t s) {
  greedy_inputs_kernel<<<nb256(HW), 256, 0, s>>>(absb1, u, w, crec, u_in, crec_in, HW);
}
void launch_abs_sum(const float2* a, const float2* b, int HW, double* partial, int nblocks, cudaStream_t s) {
  abs_sum_kernel<<<nblocks, 256, 0, s>>>(a, b, HW, partial);
}

// v *= f (agile::scale of the data normalisation, raw_data_preparation.cpp:792, 842)
__global__ void cscale_kernel(float2* v, long long n, float f) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float2 a = v[i];
    v[i] = make_float2(a.x * f, a.y * f);
  }
}

void launch_cscale(float2* v, long long n, float f, cudaStream_t s) {
  const long long nb = std::min<long long>((n + 255) / 256, 148 * 16);
  if (nb > 0) cscale_kernel<<<(int)nb, 256, 0, s>>>(v, n, f);
}

}  // namespace avx
