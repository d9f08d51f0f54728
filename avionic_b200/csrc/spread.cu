// Gridding of radial samples, sectors of 8 x 8 cells (spread.cuh).
//
// A warp owns half a sector (8 x 4 cells, one a lane, CC coils' sums in
// registers) and walks the sector's work list in batches of NB samples, which
// the warp stages by cp.async into its own two slots of shared memory: while
// one batch is summed the next one's values and weights, and the list entries
// of the one after, are in flight, across sector boundaries too.
//
// A sector has 18 samples on average at 128 x 128 (192 x 192 grid, 21 spokes),
// so that a block per sector (rad_spread_kernel) spends its time in the chain
// list -> window -> values -> barrier -> sums.  Here that chain overlaps the
// sums, no warp waits on another, row masks are ballots instead of shared
// atomics, and values lie sample by sample, two coils a load.  128 x 128, 40
// frames, 12 coils: 69.2 -> 53.6 M warp instructions, 108 -> 82 us (64 %
// issue-active, 58 % of the LSU data pipe).  The whole adjoint, block per
// sector and here: 16 coils 311 -> 242 us, 8 coils 156 -> 129; 8 frames, 16
// coils 125 -> 88; 64 x 64, 8 frames, 4 coils 44 -> 26; 160 x 160, 20 frames,
// 20 coils, 30 spokes, osf 2 537 -> 409; 150 x 40, 60 frames, 3 coils 148 ->
// 128.
#include <algorithm>

#include "regfft.cuh"
#include "spread.cuh"

namespace avx {

namespace {

// items a warp walks at most: one item each (no overlap of one's end with the next's start) takes 120 us where 3 take
// 83 and 8 take 81; 16 lengthen the last wave (86)
constexpr int SW = 8, MAX_PER = 8;

AVX_D int wrap1(int a, int n) { return a < 0 ? a + n : (a >= n ? a - n : a); }

AVX_D void async8(void* dst, const void* src, bool in) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = in ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

template <int NW, int CC>
struct Slot {
  // samples a batch: 32 for 12 coils leave fewer warps (85 us against 82), 16 for 8 coils more batches (58 and 55 the
  // adjoint at 104 x 90, 5 coils)
  static constexpr int NB = CC > 8 ? 16 : 32;
  static constexpr int VP = 2 * CC + 4, WP = NW == 5 ? 14 : 10;  // odd multiples of 16 and of 8 bytes
  float v[NB * VP];                                              // [sample][coil] re, im
  float w[NB * WP];                                              // [sample] x weights, y weights times sqrt(w) norm
  int2 r[NB];                                                    // window offset of the sector's first cell
};

// one batch of a sector's list: entries [b0, min(b0 + NB, tot))
struct Batch {
  int n, b0;  // the warp's item, first entry
};

}  // namespace

// PAIRS = 4: the `heavy` longest lists have a block each, whose pairs of warps share them batch by batch
template <int NW, int CC, int PAIRS>
__global__ void __launch_bounds__(64 * PAIRS, PAIRS > 1 ? 3 : CC > 8 ? 12 : 16)
spread8_kernel(RArgs a, const float2* __restrict__ samples, int items, int heavy, int per) {
  if (a.st && a.st->stop) return;
  using SL = Slot<NW, CC>;
  constexpr int NB = SL::NB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const RadialGeomDev& g = a.g;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = warp & 1, pair = warp >> 1;
  SL* slots = reinterpret_cast<SL*>(smem_raw) + 2 * warp;
  const int e0 = lane & (NB - 1), hl = lane / NB;  // the sample this lane stages, and which half of its coils
  const int lx = lane & (SW - 1), ry0 = half * 4, ly = ry0 + lane / SW;
  const int nsec = g.nsx * g.nsy, c0 = blockIdx.y * CC, cc = min(CC, g.C - c0);
  // pair u of the other blocks takes items heavy + u, heavy + u + (number of pairs), ...; lane n holds the n-th one's
  // place
  const bool split = PAIRS > 1 && (int)blockIdx.x < heavy;
  const int item0 = split ? (int)blockIdx.x : heavy + ((int)blockIdx.x - heavy) * PAIRS + pair;
  const int stride = ((int)gridDim.x - heavy) * PAIRS;
  const int cnt = split ? 1 : item0 < items ? min(per, (items - item0 + stride - 1) / stride) : 0;
  const int start = split ? pair * NB : 0, step = split ? PAIRS * NB : NB;
  int my_blk = 0, my_off = 0, my_tot = 0;
  if (lane < cnt) {
    my_blk = g.spread_blocks[item0 + lane * stride];
    my_off = g.spread_off[my_blk];
    my_tot = g.spread_off[my_blk + 1] - my_off;
  }
  auto next = [&](Batch b) {  // the batch after b (n = cnt: none)
    const int tot = __shfl_sync(0xffffffffu, my_tot, b.n & 31);
    return b.b0 + step < tot ? Batch{b.n, b.b0 + step} : Batch{b.n + 1, start};
  };
  auto entry = [&](Batch b) {  // this lane's list entry of the batch, or -1
    const int tot = __shfl_sync(0xffffffffu, my_tot, b.n & 31), off = __shfl_sync(0xffffffffu, my_off, b.n & 31);
    return b.n < cnt && b.b0 + e0 < tot ? g.spread_list[off + b.b0 + e0] : -1;
  };
  int2 g0 = make_int2(0, 0);
  float sc = 0.f;
  auto stage = [&](Batch b, int j, SL& s) {
    const int blk = __shfl_sync(0xffffffffu, my_blk, b.n & 31);
    if (j >= 0) {
      const int f = blk / nsec;
      const long long fj = (long long)f * g.S + j;
      const float2* src = samples + ((long long)f * g.C + c0) * g.S + j;
      constexpr int HC = CC * NB / 32;
#pragma unroll
      for (int k = 0; k < HC; ++k) {
        const int kc = hl * HC + k;
        async8(s.v + e0 * SL::VP + 2 * kc, kc < cc ? src + (long long)kc * g.S : src, kc < cc);
      }
      if (hl == 0) {
#pragma unroll
        for (int o = 0; o < NW; ++o) async8(s.w + e0 * SL::WP + 2 * o, g.winw + fj * 2 * NW + 2 * o, true);
        g0 = g.win0[fj];
        sc = g.sqrt_w[fj];
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  Batch cur{0, start};
  int j = entry(cur);
  stage(cur, j, slots[0]);
  Batch nxt = next(cur);
  int jn = entry(nxt);
  float2 acc[CC];
#pragma unroll
  for (int k = 0; k < CC; ++k) acc[k] = czero();
  int gx = 0, gy = 0;
  float2* out = a.grid;
  auto store = [&] {
    if (gx < g.Gx && gy < g.Gy)
#pragma unroll
      for (int k = 0; k < CC; ++k)
        if (k < cc) out[k * (long long)g.Gy * g.Gx] = acc[k];
  };
  for (int it = 0; cur.n < cnt; ++it) {
    SL& s = slots[it & 1];
    const int blk = __shfl_sync(0xffffffffu, my_blk, cur.n);
    const int f = blk / nsec, sec = blk - f * nsec;
    const int X0 = sec % g.nsx * SW, Y0 = sec / g.nsx * SW;
    gx = X0 + lx, gy = Y0 + ly;
    out = a.grid + (((long long)f * g.C + c0) * g.Gy + gy) * g.Gx + gx;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // window offsets of the sector's first cell and row of this half: 0 <= o + l < NW inside the window
    int rx = wrap1(X0 - g0.x, g.Gx), ry = wrap1(Y0 - g0.y, g.Gy);
    if (rx >= NW) rx -= g.Gx;
    if (ry >= NW) ry -= g.Gy;
    const bool mine = j >= 0 && hl == 0;
    if (mine) {
      s.r[e0] = make_int2(rx, ry);
      float* wy = s.w + e0 * SL::WP + NW;
      const float q = sc * g.norm;
#pragma unroll
      for (int o = 0; o < NW; ++o) wy[o] *= q;
    }
    unsigned m = 0;  // the batch's samples whose window covers this lane's row
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const unsigned b = __ballot_sync(0xffffffffu, mine && (unsigned)(ry + ry0 + y) < (unsigned)NW);
      if (ly - ry0 == y) m = b;
    }
    __syncwarp();  // every lane's copies and offsets; the other slot's last reader is past
    const Batch nn = next(nxt);
    stage(nxt, jn, slots[(it + 1) & 1]);
    const int jnn = entry(nn);
    if (gx >= g.Gx || gy >= g.Gy) m = 0;
    while (m) {
      const int e = __ffs((int)m) - 1;
      m &= m - 1;
      const int2 r = s.r[e];
      const int ox = r.x + lx;
      if ((unsigned)ox < (unsigned)NW) {
        const float* w = s.w + e * SL::WP;
        const float p = w[ox] * w[NW + r.y + ly];
        const float2 pp = make_float2(p, p);
        const float4* v = reinterpret_cast<const float4*>(s.v + e * SL::VP);
#pragma unroll
        for (int k = 0; k < CC / 2; ++k) {
          const float4 q = v[k];
          acc[2 * k] = fma2(pp, make_float2(q.x, q.y), acc[2 * k]);
          acc[2 * k + 1] = fma2(pp, make_float2(q.z, q.w), acc[2 * k + 1]);
        }
      }
    }
    if (!split && nxt.n != cur.n) {
      store();
#pragma unroll
      for (int k = 0; k < CC; ++k) acc[k] = czero();
    }
    cur = nxt;
    j = jn;
    nxt = nn;
    jn = jnn;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (PAIRS == 1 || !split) return;
  float2* red = reinterpret_cast<float2*>(smem_raw) + (threadIdx.x & 63);  // [PAIRS - 1][CC][64]
  __syncthreads();
  if (pair) {
#pragma unroll
    for (int k = 0; k < CC; ++k) red[((pair - 1) * CC + k) * 64] = acc[k];
  }
  __syncthreads();
  if (pair) return;
  for (int p = 0; p < PAIRS - 1; ++p) {
#pragma unroll
    for (int k = 0; k < CC; ++k) acc[k] = add2(acc[k], red[(p * CC + k) * 64]);
  }
  store();
}

// Windows of 3 to 5 points are those of kernel widths up to 4; a side of 32 cells keeps a window from reaching a sector
// from both ends.
bool spread8_applies(const RadialGeomDev& g) {
  return !g.per_sector && g.sw == SW && g.nw >= 3 && g.nw <= 5 && g.Gx >= 32 && g.Gy >= 32;
}

template <int NW, int CC>
static void launch(const RArgs& a, const float2* samples, cudaStream_t s) {
  const int items = a.g.nsx * a.g.nsy * a.g.T, passes = (a.g.C + CC - 1) / CC;
  constexpr size_t sm = 4 * sizeof(Slot<NW, CC>);
  // Fewer than two items for each of the pairs in two waves of 12 to 16 blocks an SM: the longest lists (a sector by
  // the centre of k-space holds 500 samples of 34 spokes) last longer than all the rest, so the 8 longest a frame are
  // shared out.  Adjoint at 96 x 96, 6 frames, 12 coils, 34 spokes 93 us without, 61 with; 128 x 128, 8 frames, 16
  // coils 109 and 88; 64 x 64, 8 frames, 4 coils 34 and 26; 24 a frame 60, 86 and 26.  With more items they end
  // within the first wave, and the larger blocks cost more than they give: 160 x 160, 20 frames, 20 coils 405 and
  // 436, 128 x 128, 40 frames, 12 coils 181 and 190.
  const int per = items / (148 * 32);
  if (per < 2) {
    const int heavy = std::min(items, 8 * a.g.T);
    spread8_kernel<NW, CC, 4>
        <<<dim3(heavy + (items - heavy + 3) / 4, passes), 256, 4 * sm, s>>>(a, samples, items, heavy, 1);
  } else {
    const int n = std::min(per, MAX_PER);
    spread8_kernel<NW, CC, 1><<<dim3((items + n - 1) / n, passes), 64, sm, s>>>(a, samples, items, 0, n);
  }
}

template <int NW>
static void launch_c(const RArgs& a, const float2* samples, cudaStream_t s) {
  if (a.g.C <= 4) launch<NW, 4>(a, samples, s);
  else if (a.g.C <= 8) launch<NW, 8>(a, samples, s);
  else if (a.g.C <= 12) launch<NW, 12>(a, samples, s);
  else launch<NW, 16>(a, samples, s);
}

void launch_spread8(const RArgs& a, const float2* samples, cudaStream_t s) {
  if (a.g.nw == 3) launch_c<3>(a, samples, s);
  else if (a.g.nw == 4) launch_c<4>(a, samples, s);
  else launch_c<5>(a, samples, s);
}

template <int NW>
static cudaError_t configure() {
  cudaError_t e = cudaSuccess;
  for (auto f : {spread8_kernel<NW, 4, 4>, spread8_kernel<NW, 8, 4>, spread8_kernel<NW, 12, 4>, spread8_kernel<NW, 16, 4>})
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, AVX_DYN_SMEM_MAX);
  return e;
}
cudaError_t configure_spread8(const RadialGeomDev& g) {
  return g.nw == 3 ? configure<3>() : g.nw == 4 ? configure<4>() : configure<5>();
}

}  // namespace avx
