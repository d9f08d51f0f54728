// Partial DFTs along y with register FFTs (see yfft.cuh).
#include <algorithm>
#include <cmath>

#include "regfft.cuh"
#include "tc_dft.cuh"
#include "yfft.cuh"

namespace avx {

namespace {

constexpr int XT = 8;  // image columns per CTA: a row of the tile is two full 32-byte sectors
constexpr int kSms = 148;

// largest CTA: the longer FFTs hold up to 128 registers a thread
constexpr int max_threads(int n1) { return n1 > 8 ? 512 : 1024; }
AVX_HD int tile_warps(int n2) { return (XT * n2 + 31) / 32; }
AVX_HD int coef_pitch(int n2) { return n2 | 1; }    // odd: rows of coefficients start in different banks
constexpr int even(int n) { return n + (n & 1); }

size_t fwd_smem(int n1, int n2, int rows) {
  return (size_t)2 * n2 * (n1 + 1) * XT * sizeof(float2) + (size_t)rows * coef_pitch(n2) * sizeof(float2) +
         (size_t)rows * sizeof(int2);
}
size_t adj_smem(int n1, int n2, int rows, int groups) {
  const size_t nt = (size_t)32 * tile_warps(n2);
  return (size_t)groups * (2 * n1 * nt + 4 * (size_t)rows * XT) * sizeof(float2) + (size_t)rows * n2 * sizeof(float2) +
         (size_t)rows * sizeof(int2);
}

AVX_D void cp_async8(void* dst, const void* src, bool in) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = in ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

// the coil's map values of one thread, y = j + n2 i for i < N1, from the
// fragment-ordered maps (yfft_maps_kernel): 16 bytes a load, warp-contiguous
template <int N1>
AVX_D void load_maps(const float4* __restrict__ p, float2 (&m)[even(N1)]) {
#pragma unroll
  for (int i = 0; i < even(N1) / 2; ++i) {
    const float4 v = __ldg(p + 32 * i);
    m[2 * i] = make_float2(v.x, v.y);
    m[2 * i + 1] = make_float2(v.z, v.w);
  }
}

}  // namespace

// Forward: CTA (column tile, frame, part of the coils), thread (tx, j) holds
// the frame's values u[j + n2 i] of its column in registers, and per pair of
// coils multiplies them by b1, transforms them, and shares the classes'
// values through shared memory; then thread (tx, r) forms the sampled rows
// r, r + n2, ...  The next coil's map values are in flight meanwhile.
//
// Bound by issue slots and shared-memory wavefronts (ncu, cine problem
// 192 x 192, 30 frames, 16 coils, 16 rows a frame: 14.7 M warp instructions,
// 54 % issue-active, 54 % of the LSU data pipe).  8 columns a CTA because the
// small CTAs balance over the SMs (16 columns: 50-56 us, 32: 60); float2
// coefficients (a duplicated float4 costs two more wavefronts a read: 320 x
// 320, 53 rows, 494 us against 394); the maps in fragment order cut 18.2 M
// instructions to 14.7 M (40.6 -> 32.4 us).  Cine: 52.7 us with the
// tensor-core partial DFT, 32.4 here; 320 x 320, 48 frames, 32 coils, 53 rows:
// 2332 us with the dense fp32 sums, 319 here; 160 x 128, 24 frames, 12 coils,
// 64 rows: 139 -> 27 (23 by yfull_impl.cuh, which takes it); 128 x 128, 20 frames, 8 coils, 16 rows: 20.7 -> 13.7.
template <int N1>
__global__ void __launch_bounds__(max_threads(N1)) yfft_kernel(KArgs a, int cpz) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const CartGeomDev& g = a.g;
  const int W = g.W, H = g.H, C = g.C, n2 = H / N1;
  const int t = blockIdx.y;
  const int r0 = g.row_off[t], S = g.row_off[t + 1] - r0;
  if (S == 0) {
    pdl_wait();
    return;
  }
  constexpr int JP = (N1 + 1) * XT, E = even(N1);
  const int tid = threadIdx.x, nt = blockDim.x;  // nt = 32 tile_warps(n2) >= XT n2
  const int tx = tid & (XT - 1), j = tid / XT;
  const bool act = j < n2;
  const int x = blockIdx.x * XT + tx;
  const bool in = act && x < W;
  const int pitch = coef_pitch(n2);
  float2* buf = reinterpret_cast<float2*>(smem_raw);  // [2][n2][N1 + 1][XT]
  float2* coef = buf + (size_t)2 * n2 * JP;           // [S][pitch]
  int2* oc = reinterpret_cast<int2*>(coef + (size_t)S * pitch);
  for (int e = tid; e < S * n2; e += nt) {
    const int p = e / n2;
    coef[p * pitch + (e - p * n2)] = a.yf_coef[(size_t)r0 * n2 + e];
  }
  for (int e = tid; e < S; e += nt) oc[e] = a.yf_order[r0 + e];
  pdl_wait();
  pdl_trigger();
  if (a.st && a.st->stop) return;
  const int cb = blockIdx.z * cpz, ce = min(C, cb + cpz);
  const float4* __restrict__ maps =
      reinterpret_cast<const float4*>(a.b1t) +
      (((size_t)cb * gridDim.x + blockIdx.x) * (nt >> 5) + (tid >> 5)) * (E / 2) * 32 + (tid & 31);
  const size_t mstep = (size_t)gridDim.x * nt * (E / 2);
  float2 u[N1], m[E];
  load_maps<N1>(maps, m);
  {
    const float2* in_p = a.in + (long long)t * W * H + (in ? (long long)j * W + x : 0);
    const long long step = in ? (long long)n2 * W : 0;
#pragma unroll
    for (int i = 0; i < N1; ++i) u[i] = in_p[i * step];
  }
  const long long kb = (long long)r0 * C * W + x;
  float2* mine = buf + (act ? j : 0) * JP + tx;
  for (int c0 = cb; c0 < ce; c0 += 2) {
    const int nc = min(2, ce - c0);
    __syncthreads();  // the previous pair's values are read (and, first, the tables are staged)
#pragma unroll 1
    for (int q = 0; q < nc; ++q) {
      float2 v[N1];
#pragma unroll
      for (int i = 0; i < N1; ++i) v[i] = cmul(m[i], u[i]);
      maps += mstep;
      if (c0 + q + 1 < ce) load_maps<N1>(maps, m);
      reg_dft<N1, +1>(v);
      float2* o = mine + (size_t)q * n2 * JP;
      if (act)
#pragma unroll
        for (int i = 0; i < N1; ++i) o[i * XT] = v[i];
    }
    __syncthreads();
    if (!act) continue;
    for (int p = j; p < S; p += n2) {
      const int2 ocp = oc[p];
      const float2* cf = coef + p * pitch;
      const float2* v0 = buf + ocp.y * XT + tx;
      const float2* v1 = v0 + (size_t)(nc - 1) * n2 * JP;
      float2 a0 = czero(), b0 = czero(), a1 = czero(), b1 = czero();
#pragma unroll 4
      for (int jj = 0; jj < n2; ++jj) {
        const float2 w = cf[jj], q0 = v0[jj * JP], q1 = v1[jj * JP];
        a0 = fma2(make_float2(w.x, w.x), q0, a0);
        b0 = fma2(make_float2(w.y, w.y), q0, b0);
        a1 = fma2(make_float2(w.x, w.x), q1, a1);
        b1 = fma2(make_float2(w.y, w.y), q1, b1);
      }
      if (x < W) {
        float2* out = a.qp + kb + ((long long)c0 * S + ocp.x) * W;
        out[0] = make_float2(a0.x - b0.y, a0.y + b0.x);
        if (nc > 1) out[(long long)S * W] = make_float2(a1.x - b1.y, a1.y + b1.x);
      }
    }
  }
}

// Adjoint: CTA (column tile, frame), its threads in groups that share the
// coils out.  Thread (tx, j) of a group sums the sampled rows of each class
// for two coils (the coils' rows staged in class order, two coils ahead),
// transforms the classes in registers, multiplies by conj(b1) and accumulates
// over its coils the image rows y = j + n2 i of its column.  The class sums
// pass through the thread's own slots of shared memory: one loop over the
// sampled rows with a flush at each class's last row, instead of a loop per
// class.  The groups' sums are added in group order.
//
// Bound as the forward kernel is (cine: 18.3 M warp instructions, 56 %
// issue-active, 59 % of the LSU data pipe).  A loop per class, its length
// read from shared memory, took 33 M instructions and 71.6 us.  Cine: 51.4 us
// with the tensor-core column adjoint, 35.6 here; the 320 x 320 problem above
// 2297 -> 433; 160 x 128 168 -> 41; 128 x 128 16.5 -> 15.4.
template <int N1>
__global__ void __launch_bounds__(max_threads(N1)) yfft_adj_kernel(KArgs a, float2* img, int groups) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const CartGeomDev& g = a.g;
  const int W = g.W, H = g.H, C = g.C, n2 = H / N1;
  const int t = blockIdx.y;
  const int r0 = g.row_off[t], S = g.row_off[t + 1] - r0;
  constexpr int E = even(N1);
  const int nt = 32 * tile_warps(n2);
  const int grp = threadIdx.x / nt, tid = threadIdx.x - grp * nt;
  const int tx = tid & (XT - 1), j = tid / XT;
  const bool act = j < n2;
  const int x0 = blockIdx.x * XT, x = x0 + tx;
  float2* cls0 = reinterpret_cast<float2*>(smem_raw);          // [groups][2][N1][nt]
  float2* rows0 = cls0 + (size_t)groups * 2 * N1 * nt;         // [groups][2][2][S][XT]
  float2* coef = rows0 + (size_t)groups * 4 * S * XT;          // [S][n2]
  int2* oc = reinterpret_cast<int2*>(coef + (size_t)S * n2);   // [S] compact row; slot of the class (last row) or -1
  float2* cls = cls0 + (size_t)grp * 2 * N1 * nt + tid;
  float2* rows = rows0 + (size_t)grp * 4 * S * XT;
  for (int e = threadIdx.x; e < S * n2; e += blockDim.x) coef[e] = a.yf_coef[(size_t)r0 * n2 + e];
  for (int e = threadIdx.x; e < S; e += blockDim.x) {
    const int2 v = a.yf_order[r0 + e];
    const bool last = e + 1 == S || a.yf_order[r0 + e + 1].y != v.y;
    oc[e] = make_int2(v.x, last ? v.y * nt : -1);
  }
  pdl_wait();
  pdl_trigger();
  if (a.st && a.st->stop) return;
  float2 acc[N1];
#pragma unroll
  for (int i = 0; i < N1; ++i) acc[i] = cls[i * nt] = cls[(N1 + i) * nt] = czero();  // empty classes stay zero
  const int rounds = (C + 2 * groups - 1) / (2 * groups);
  const int cb = min(C, grp * 2 * rounds), ce = min(C, cb + 2 * rounds);
  const float2* __restrict__ qp = a.qp + (long long)r0 * C * W;
  const float4* __restrict__ maps =
      reinterpret_cast<const float4*>(a.b1t) +
      (((size_t)cb * gridDim.x + blockIdx.x) * (nt >> 5) + (tid >> 5)) * (E / 2) * 32 + (tid & 31);
  const size_t mstep = (size_t)gridDim.x * nt * (E / 2);
  const float2* cf = coef + (act ? j : 0);
  __syncthreads();
  auto stage = [&](int r) {  // round r's coils cb + 2 r, cb + 2 r + 1
    const int c0 = cb + 2 * r;
    float2* d = rows + (size_t)(r & 1) * 2 * S * XT;
    const int nc = max(0, min(2, ce - c0));
    for (int e = tid; e < nc * S * XT; e += nt) {
      const int ex = e & (XT - 1), p = e / XT;  // p < nc S
      const int q = p >= S ? 1 : 0;
      const bool ok = x0 + ex < W;
      cp_async8(d + e, qp + ((long long)(c0 + q) * S + oc[p - q * S].x) * W + (ok ? x0 + ex : 0), ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (S > 0) {
    stage(0);
    for (int r = 0; r < rounds; ++r) {
      if (r + 1 < rounds) {
        stage(r + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      __syncthreads();
      const int nc = min(2, ce - (cb + 2 * r));  // <= 0: this group has no coils left
      if (nc > 0) {
        const float2* z0 = rows + (size_t)(r & 1) * 2 * S * XT + tx;
        const float2* z1 = z0 + (size_t)(nc - 1) * S * XT;
        float2 a0 = czero(), b0 = czero(), a1 = czero(), b1 = czero();
#pragma unroll 4
        for (int p = 0; p < S; ++p) {
          const float2 w = cf[p * n2], q0 = z0[p * XT], q1 = z1[p * XT];
          a0 = fma2(make_float2(w.x, w.x), q0, a0);
          b0 = fma2(make_float2(w.y, w.y), q0, b0);
          a1 = fma2(make_float2(w.x, w.x), q1, a1);
          b1 = fma2(make_float2(w.y, w.y), q1, b1);
          const int slot = oc[p].y;
          if (slot >= 0) {
            cls[slot] = make_float2(a0.x + b0.y, a0.y - b0.x);
            cls[N1 * nt + slot] = make_float2(a1.x + b1.y, a1.y - b1.x);
            a0 = b0 = a1 = b1 = czero();
          }
        }
      }
#pragma unroll 1
      for (int q = 0; q < nc; ++q) {
        float2 v[N1], m[E];
        load_maps<N1>(maps, m);
        maps += mstep;
#pragma unroll
        for (int i = 0; i < N1; ++i) v[i] = cls[(q * N1 + i) * nt];
        reg_dft<N1, -1>(v);
#pragma unroll
        for (int i = 0; i < N1; ++i) {
          acc[i].x = fmaf(m[i].x, v[i].x, fmaf(m[i].y, v[i].y, acc[i].x));
          acc[i].y = fmaf(m[i].x, v[i].y, fmaf(-m[i].y, v[i].x, acc[i].y));
        }
      }
      __syncthreads();  // the round's stage is refilled next
    }
  }
  if (groups > 1) {
    if (grp > 0)
#pragma unroll
      for (int i = 0; i < N1; ++i) cls[i * nt] = acc[i];
    __syncthreads();
    if (grp > 0) return;
    for (int k = 1; k < groups; ++k)
#pragma unroll
      for (int i = 0; i < N1; ++i) acc[i] = add2(acc[i], cls[(size_t)(2 * k * N1 + i) * nt]);
  }
  if (act && x < W) {
    float2* out = img + ((long long)t * H + j) * W + x;
    const long long step = (long long)n2 * W;
#pragma unroll
    for (int i = 0; i < N1; ++i) out[i * step] = acc[i];
  }
}

// fragment order of the coil maps: [coil][column tile][warp][i / 2][lane][i % 2]
// holds b1[coil][y = j + n2 i][x] of thread 32 warp + lane = XT j + tx; zero
// where the thread or the column does not exist
__global__ void yfft_maps_kernel(const float2* __restrict__ b1, float2* __restrict__ out, int W, int H, int n1, int n2,
                                 int tiles, long long n) {
  const int nw = tile_warps(n2), e2 = (n1 + 1) / 2;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    long long r = e >> 6;
    const int i = 2 * (int)(r % e2) + (int)(e & 1);
    r /= e2;
    const int tid = 32 * (int)(r % nw) + (int)((e >> 1) & 31);
    r /= nw;
    const int x = XT * (int)(r % tiles) + (tid & (XT - 1)), j = tid / XT;
    const int c = (int)(r / tiles);
    out[e] = j < n2 && i < n1 && x < W ? b1[((long long)c * H + j + n2 * i) * W + x] : czero();
  }
}

#define YFFT_DISPATCH(N1, CALL) \
  switch (N1) {                 \
    case 16: CALL(16); break;   \
    case 15: CALL(15); break;   \
    case 14: CALL(14); break;   \
    case 13: CALL(13); break;   \
    case 12: CALL(12); break;   \
    case 11: CALL(11); break;   \
    case 10: CALL(10); break;   \
    case 9: CALL(9); break;     \
    case 8: CALL(8); break;     \
    case 7: CALL(7); break;     \
    case 6: CALL(6); break;     \
    case 5: CALL(5); break;     \
    default: CALL(4); break;    \
  }

// The longest register FFT that divides the height and leaves n2 >= 4 (a
// whole warp of 8 columns x n2 threads: 92 x 28, 19 coils, took 1.2 times as
// long with n1 = 14, n2 = 2), else the longest at all: each step down trades
// register butterflies for class sums.  At n1 = 4 the class sums are H / 4
// long and the tensor-core partial DFT is faster where it applies (192 x 316,
// 20 frames, 8 coils, 20 rows a frame: 93 us for both of its directions
// against 117; n1 = 5 at 305 rows: 79 against 92), so 4 serves only the
// frames with more rows than that form takes.
int yfft_n1(int H, int max_rows) {
  for (int least : {4, 1})
    for (int n1 = 16; n1 >= (2 * max_rows > TC_MAX_NP ? 4 : 5); --n1) {
      const int n2 = H / n1;
      if (H % n1 || n2 < least || 32 * tile_warps(n2) > max_threads(n1)) continue;
      if (fwd_smem(n1, n2, max_rows) > AVX_DYN_SMEM_MAX || adj_smem(n1, n2, max_rows, 1) > AVX_DYN_SMEM_MAX) continue;
      return n1;
    }
  return 0;
}

size_t yfft_maps_count(int W, int H, int C, int n1) {
  return (size_t)C * ((W + XT - 1) / XT) * tile_warps(H / n1) * even(n1) * 32;
}

void launch_yfft_maps(const float2* b1, float2* out, int W, int H, int C, int n1, cudaStream_t s) {
  const long long n = (long long)yfft_maps_count(W, H, C, n1);
  const int blocks = (int)std::min<long long>((n + 255) / 256, kSms * 16);
  yfft_maps_kernel<<<blocks, 256, 0, s>>>(b1, out, W, H, n1, H / n1, (W + XT - 1) / XT, n);
}

void yfft_build(int H, int T, int sy, int n1, const int* rows, const int* row_off, int2* order_cls, float2* coef) {
  const int n2 = H / n1;
  const double inv = 1.0 / std::sqrt((double)H);
  for (int t = 0; t < T; ++t) {
    const int r0 = row_off[t], S = row_off[t + 1] - r0;
    int p = 0;
    for (int k1 = 0; k1 < n1; ++k1)
      for (int s = 0; s < S; ++s) {
        const int kappa = ((rows[r0 + s] - sy) % H + H) % H;
        if (kappa % n1 != k1) continue;
        order_cls[r0 + p] = make_int2(s, k1);
        for (int j = 0; j < n2; ++j) {
          const double ang = 2.0 * M_PI * (double)((long long)kappa * (j - sy + H) % H) / H;
          coef[(size_t)(r0 + p) * n2 + j] = make_float2((float)(std::cos(ang) * inv), (float)(std::sin(ang) * inv));
        }
        ++p;
      }
  }
}

void launch_yfft(const KArgs& k, cudaStream_t s) {
  const int n2 = k.g.H / k.yf_n1, nt = 32 * tile_warps(n2), tiles = (k.g.W + XT - 1) / XT;
  // parts of the coils: enough warps for 14 an SM, at least two coils a part
  const long long warps = (long long)tiles * k.g.T * (nt / 32);
  const int z = (int)std::max<long long>(1, std::min<long long>((k.g.C + 1) / 2, (kSms * 14 + warps - 1) / warps));
  const int cpz = 2 * ((k.g.C + 2 * z - 1) / (2 * z));
  dim3 gr(tiles, k.g.T, (k.g.C + cpz - 1) / cpz);
  const size_t sm = fwd_smem(k.yf_n1, n2, k.yf_rows);
#define CALL_Y(N) launch_dependent(yfft_kernel<N>, gr, nt, sm, s, k, cpz)
  YFFT_DISPATCH(k.yf_n1, CALL_Y)
#undef CALL_Y
}

void launch_yfft_adjoint(const KArgs& k, float2* img, cudaStream_t s) {
  const int n2 = k.g.H / k.yf_n1, nt = 32 * tile_warps(n2), tiles = (k.g.W + XT - 1) / XT;
  const long long warps = (long long)tiles * k.g.T * (nt / 32);
  // groups that share a CTA's coils: for 14 warps an SM, as far as threads and shared memory allow
  int grp = 1;
  while (2 * grp <= (k.g.C + 1) / 2 && grp * warps < kSms * 14 && 2 * grp * nt <= 512 &&
         2 * adj_smem(k.yf_n1, n2, k.yf_rows, 2 * grp) <= AVX_DYN_SMEM_MAX)
    grp *= 2;
  dim3 gr(tiles, k.g.T);
  const size_t sm = adj_smem(k.yf_n1, n2, k.yf_rows, grp);
#define CALL_A(N) launch_dependent(yfft_adj_kernel<N>, gr, nt * grp, sm, s, k, img, grp)
  YFFT_DISPATCH(k.yf_n1, CALL_A)
#undef CALL_A
}

cudaError_t configure_yfft(int n1) {
  cudaError_t e = cudaSuccess;
#define SET_Y(N)                                                                                                \
  e = cudaFuncSetAttribute(yfft_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, AVX_DYN_SMEM_MAX);       \
  if (e == cudaSuccess)                                                                                          \
    e = cudaFuncSetAttribute(yfft_adj_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, AVX_DYN_SMEM_MAX)
  YFFT_DISPATCH(n1, SET_Y)
#undef SET_Y
  return e;
}

}  // namespace avx
