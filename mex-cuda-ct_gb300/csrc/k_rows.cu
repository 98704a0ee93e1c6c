// k_rows.cu -- parallel and fan forward projection, all slices of a ray's plane
// at once (CUDAmex_FP.cu:56-247; the OSC forward pass CUDAmex_oscIter.cu:140-271).
//
// A parallel or fan ray stays in one slice, and the rays of a detector column
// take the same (x, y) path through every slice.  The slab kernel walked that
// path once per slice: two samples per voxel, four taps and ~40 instructions
// each.  Here the path is turned into weights once and applied to 128 slices.
//  - The volume is laid out z-fastest, [y][x][z] with a frame of one voxel in
//    x and y (launch_pad_rows): a column of slices is contiguous.
//  - A CTA takes 32 detector columns of V views and 128 rows, and sweeps the
//    planes of the views' dominant axis a (x or y).  All samples of a ray that
//    touch plane p (floor(ta) = p - 1 or p) are merged into one weight per
//    column f they touch; four neighbouring rays share a column list.  All
//    eight warps (a lane per ray) write the weights of the next 8 / V planes,
//    then all apply them: with the weights left to V of the warps beside the
//    others' work, the others waited for them (15.0 ms at 384^3 x 512, 46 % of
//    the stalls at the barrier).
//  - The plane's columns (64 or fewer) come by TMA into one of two buffers.  A
//    warp owns four rays of each view and 128 rows: per column one 16-byte
//    load of data per lane, one broadcast of the four weights, and 8 packed
//    FMAs.
//  - Calls of few views share a tile's planes in a cluster of four or eight CTAs.
// What that moves: a column of shared memory is read once per 4 rays instead
// of 4 taps per sample, and the weights cost ~200 instructions per ray and
// plane for 128 rows.  Measured, slab kernel -> this: 384^3 x 512 parallel
// 52.4 -> 13.4 ms, fan 55.1 -> 14.7 ms; 243^2 x 201 x 361 fan in FP16 9.8 ->
// 3.1 ms; 128^2 x 100 x 360 1.27 -> 0.60 ms; 64^3 x 90 0.107 -> 0.074 ms.
// Volumes of few slices keep the slab kernel (fp_uses_rows).  Error against 64
// bits 2.3e-6 -> 3.7e-7 (shorter sums).  Bound now (four views per CTA): 54 % of
// the issue slots (the weights a fifth of them) and 60 % of the shared / L1 data
// path at 16 warps per SM, which wait on fixed latencies and shared memory.  Also
// measured: weights stored in pairs for the packed FMAs (one more load per
// column) 15.0 ms.
//
// The sum over a ray's samples is the reference's (positions entry + k step
// dir, k < n, binary32 set-up); only its order changes: taps that fall on the
// same voxel are added as weights first.  The result does not depend on V, on
// how a call's views are split into launches (nall), on the slices beside it or
// on whether a plane came from shared memory.  It does depend on SP, whose parts
// are summed apart, and so on the call's views, the detector's columns and the SM
// count: a view by itself can differ in the last bits from the same view in a full
// call, and the objective's integrals (never split) from the residuals'.
// Four rays whose columns of a plane do not fit a list (fans steeper than ~65
// degrees to the sweep axis) add that plane's samples one by one.
// A column list is shared by four rays, so a voxel that is not finite would
// reach rays that give it weight 0: a sum that is not finite is taken again
// sample by sample (rows_slow).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <type_traits>

#include "kernels.h"
#include "tma.cuh"

namespace mexct {

namespace {

constexpr int kRU = 32;      // detector columns per CTA
constexpr int kRF = 64;      // volume columns per staged plane
constexpr int kRZ = 128;     // slices per CTA: four per lane
constexpr int kRC = 16;      // columns of one weight list (even)
constexpr int kRThreads = 256;
constexpr int kRPlans = 2048;  // planes with a planned box; later ones read global memory
constexpr int kStage = kRF * kRZ;  // elements of a staged plane

// ---------------------------------------------------------------------------
// z-fastest padded layout.
// ---------------------------------------------------------------------------
// A frame of one column in x and y: edge copies (clamp addressing) or zeros
// (border).  Block: 32 x-columns of one y, 64 slices.
template <typename T>
__global__ void __launch_bounds__(256) pad_rows_kernel(const T* __restrict__ src,
                                                       T* __restrict__ dst, int W, int H, int Ph,
                                                       int border) {
  __shared__ float tile[64][33];
  const int Ps = W + 2;
  const int x0 = blockIdx.x * 32, yp = blockIdx.y, r0 = blockIdx.z * 64;
  const int tx = threadIdx.x, ty = threadIdx.y;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int z = r0 + ty + 8 * i, xp = x0 + tx;
    float v = 0.f;
    if (xp < Ps && z < H) {
      int x = xp - 1, y = yp - 1;
      if (!border || (x >= 0 && x < W && y >= 0 && y < W)) {
        x = min(max(x, 0), W - 1);
        y = min(max(y, 0), W - 1);
        v = ldf(src + (size_t)x + (size_t)W * ((size_t)y + (size_t)W * z));
      }
    }
    tile[ty + 8 * i][tx] = v;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int xc = ty * 4 + (i >> 1), zc = 32 * (i & 1) + tx;
    if (x0 + xc < Ps && r0 + zc < Ph)
      stf(dst + ((size_t)yp * Ps + x0 + xc) * Ph + r0 + zc, tile[zc][xc]);
  }
}

// ---------------------------------------------------------------------------
// Kernel.
// ---------------------------------------------------------------------------
// Four consecutive values of a column as two packed pairs.
struct Quad {
  float2 lo, hi;
};
__device__ __forceinline__ Quad ld_quad(const float* p) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ Quad ld_quad(const __half* p) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  return {__half22float2(*reinterpret_cast<const __half2*>(&v.x)),
          __half22float2(*reinterpret_cast<const __half2*>(&v.y))};
}
__device__ __forceinline__ Quad ld_quad(const __nv_bfloat16* p) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  return {__bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x)),
          __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y))};
}

struct RowsRay {
  float ta0, da, tf0, df;
  int n;
};

struct RowsMeta {
  int f, n;  // first column and (even) length of a weight list; n < 0: too long
};

template <int V>
struct RowsShared {
  uint64_t bar[4];
  RowsRay ray[V][kRU];
  float4 w[8 / V][V][kRU / 4][kRC];  // weights of a group of planes: four rays each
  RowsMeta meta[8 / V][V][kRU / 4];
  int amin, amax, abort;
  short plan[kRPlans];               // first column of each plane's box, -1: none
  double wsum[kRThreads / 32];
};

// Column index of a voxel column, and the clamp of a tap the slab kernel's
// global path takes.
__device__ __forceinline__ size_t rows_col(int Ps, bool xdom, int a, int f) {
  a = min(max(a, 0), Ps - 1);
  f = min(max(f, 0), Ps - 1);
  return xdom ? (size_t)f * Ps + a : (size_t)a * Ps + f;
}

// A ray's samples in order of rising ta: sample i is k = i (da > 0) or n - 1 -
// i, at fma(k, d, t0).  Counts are floats (exact, and no conversions).
struct RowsWalk {
  float ta0, da, tf0, df, nf, kb, ks;
  __device__ __forceinline__ explicit RowsWalk(const RowsRay& R)
      : ta0(R.ta0), da(R.da), tf0(R.tf0), df(R.df), nf((float)R.n) {
    kb = da > 0.f ? 0.f : nf - 1.0f;
    ks = da > 0.f ? 1.f : -1.f;
  }
  __device__ __forceinline__ float ta(float i) const { return fmaf(fmaf(i, ks, kb), da, ta0); }
  __device__ __forceinline__ float tf(float i) const { return fmaf(fmaf(i, ks, kb), df, tf0); }
  // First i in [0, n] with ta(i) >= a: estimated, then settled on the positions.
  __device__ __forceinline__ float first_at(float a) const {
    float i = fminf(fmaxf(ceilf(__fdividef(a - ta(0.f), fabsf(da))), 0.f), nf);
    while (i > 0.f && ta(i - 1.0f) >= a) i -= 1.0f;
    while (i < nf && ta(i) < a) i += 1.0f;
    return i;
  }
};

// One ray's sum for the four rows at `z` (an element offset in a column),
// sample by sample with bilinear interpolation.
template <typename TV>
__device__ __noinline__ float4 rows_slow(const TV* vol, const RowsRay r, bool xdom, int Ps,
                                         size_t pitch, size_t z) {
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int k = 0; k < r.n; ++k) {
    const float ta = fmaf((float)k, r.da, r.ta0), tf = fmaf((float)k, r.df, r.tf0);
    const float fa = floorf(ta), ff = floorf(tf);
    const float wa = ta - fa, wf = tf - ff;
    const int a = min(max((int)fa, 0), Ps - 2), f = min(max((int)ff, 0), Ps - 2);
    const TV* p[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) p[t] = vol + rows_col(Ps, xdom, a + (t >> 1), f + (t & 1)) * pitch + z;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float v00 = ldp(p[0] + i), v01 = ldp(p[1] + i), v10 = ldp(p[2] + i), v11 = ldp(p[3] + i);
      const float r0 = fmaf(wf, v01 - v00, v00), r1 = fmaf(wf, v11 - v10, v10);
      acc[i] += fmaf(wa, r1 - r0, r0);
    }
  }
  return make_float4(acc[0], acc[1], acc[2], acc[3]);
}

// EPI 0: line integrals (accum: added to the output); 1: OSC residuals; 2:
// objective partials.  V views per CTA, NB staged planes (2: two CTAs per SM;
// 4: one CTA per SM, for grids that leave it alone there).  SP = 4 or 8: a
// cluster of CTAs shares the tile, a part of the planes each; the parts' sums
// are added in order from the CTAs' shared memory, one of a warp's four rays
// (or half of its slices) per CTA.
template <int EPI, typename TV, typename TO, int V, int NB, int SP>
__global__ void __launch_bounds__(kRThreads, 2) fp_rows_kernel(
    const __grid_constant__ RayArgs A, const int geom, const __grid_constant__ CUtensorMap tmx,
    const __grid_constant__ CUtensorMap tmy, const TV* __restrict__ vol, int Ph,
    TO* __restrict__ out, const SlabEpi E) {
  static_assert(SP == 1 || ((SP == 4 || SP == 8) && V == 1 && EPI != 2), "a cluster takes one view");
  constexpr int NG = kRU / 4, PG = 8 / V;  // ray groups; planes whose weights are made at once
  static_assert(NG == kRThreads / 32, "a warp per four rays");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  TV* const buf = reinterpret_cast<TV*>(smem_raw);
  RowsShared<V>& S = *reinterpret_cast<RowsShared<V>*>(smem_raw + NB * kStage * sizeof(TV));
  const int tid = threadIdx.x, lane = tid & 31, g = tid >> 5;
  const int nvg = (A.nviews + V - 1) / V, tiles_u = (A.det_w + kRU - 1) / kRU;
  const int rank = SP > 1 ? (int)(blockIdx.x % SP) : 0, job = (int)(blockIdx.x / SP);
  // the ray of each warp's four and the slices of each lane's four that this
  // CTA finishes
  constexpr int NZ = SP == 8 ? 2 : 4;
  const int ray = SP == 8 ? rank >> 1 : rank, zb = SP == 8 ? 2 * (rank & 1) : 0;
  const int vg = job % nvg, tile = (job / nvg) % tiles_u, chunk = (job / nvg) / tiles_u;
  const int u0 = tile * kRU, v0 = vg * V, nv = min(V, A.nviews - v0);
  const int Ps = A.S + 2;
  const size_t pitch = Ph;
  if (tid == 0) {
    for (int b = 0; b < NB; ++b) mbar_init(&S.bar[b], 1);
    S.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // this lane's four slices; past the column's end it reads the last ones
  // again (not stored)
  const int z0 = chunk * kRZ + 4 * lane;
  const size_t zoff = min(z0, Ph - 4);
  uint32_t phase = 0u;
  uint64_t issued = 0u;  // thread 0: copies per buffer, 16 bits each
  float2 acc[V][4][2];
#pragma unroll
  for (int r = 0; r < V; ++r)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[r][i][0] = acc[r][i][1] = make_float2(0.f, 0.f);

  auto redo = [&](float2* q, const RowsRay& R, bool xdom) {
    const bool bad[4] = {!(q[0].x - q[0].x == 0.f), !(q[0].y - q[0].y == 0.f),
                         !(q[1].x - q[1].x == 0.f), !(q[1].y - q[1].y == 0.f)};
    if (bad[0] || bad[1] || bad[2] || bad[3]) {
      const float4 f = rows_slow(vol, R, xdom, Ps, pitch, zoff);
      if (bad[0]) q[0].x = f.x;
      if (bad[1]) q[0].y = f.y;
      if (bad[2]) q[1].x = f.z;
      if (bad[3]) q[1].y = f.w;
    }
  };
  for (int ax = 0; ax < 2; ++ax) {
    const bool xdom = ax == 0;  // sweep the views whose rays run mostly along x, then y
    bool mine[V], any = false;
#pragma unroll
    for (int r = 0; r < V; ++r) {
      const Trig t = A.trig[v0 + min(r, nv - 1)];
      mine[r] = r < nv && (fabsf(t.c) >= fabsf(t.s)) == xdom;
      any |= mine[r];
    }
    if (!any) continue;
    __syncthreads();
    if (tid == 0) {
      S.amin = 0x7fffffff;
      S.amax = -0x7fffffff;
    }
    __syncthreads();
    // rays: warp r < V sets up view r's 32 rays
    if (g < V) {
      RowsRay R{0.f, 1.f, 0.f, 0.f, 0};
      const Trig t = A.trig[v0 + min(g, nv - 1)];
      const int ix = u0 + lane;
      float s[3], e[3];
      if (geom == 0)
        std_ray<0>(min(ix, A.det_w - 1), 0, A.u0, A.v0, t.s, t.c, A.SR, A.RD, s, e, A.du, A.dv,
                   A.ou, A.ov);
      else
        std_ray<1>(min(ix, A.det_w - 1), 0, A.u0, A.v0, t.s, t.c, A.SR, A.RD, s, e, A.du, A.dv,
                   A.ou, A.ov);
      const Ray c = clip_ray(s[0], s[1], s[2], e[0], e[1], e[2], A.bx, A.by, A.bz, A.step);
      R.ta0 = (xdom ? c.cx - A.bx : c.cy - A.by) + 0.5f;
      R.tf0 = (xdom ? c.cy - A.by : c.cx - A.bx) + 0.5f;
      R.da = xdom ? c.dx : c.dy;
      R.df = xdom ? c.dy : c.dx;
      R.n = c.n;
      // a decoupled detector's columns can miss the volume
      const bool own = A.det_w == A.S && A.du == 1.0f;
      const float sxy[3] = {s[0], s[1], 0.f}, exy[3] = {e[0], e[1], 0.f};
      if (ix >= A.det_w || g >= nv || (fabsf(t.c) >= fabsf(t.s)) != xdom ||
          !(own || hits_box(sxy, exy, A.bx, A.by, A.bz)))
        R.n = 0;
      if (R.n > 0) {
        const int t0 = __float2int_rd(R.ta0);
        const int t1 = __float2int_rd(fmaf((float)(R.n - 1), R.da, R.ta0));
        atomicMin(&S.amin, min(t0, t1));
        atomicMax(&S.amax, max(t0, t1));
      }
      S.ray[g][lane] = R;
    }
    __syncthreads();
    if (S.amax < S.amin) continue;  // no ray of these views meets the volume
    // planes p0 .. p0 + np - 1 (this CTA's share of them)
    const int npa = S.amax - S.amin + 2, first = npa * rank / SP;
    const int p0 = S.amin + first, np = npa * (rank + 1) / SP - first;
    // Boxes: the columns of the outermost rays of each view between planes
    // p - 1 and p + 1 (f is monotone across a view's rays), one more each side.
    for (int j = tid; j < min(np, kRPlans); j += kRThreads) {
      float lo = 3.0e38f, hi = -3.0e38f;
#pragma unroll
      for (int r = 0; r < V; ++r) {
        if (!mine[r]) continue;
        const int last = min(kRU, A.det_w - u0) - 1;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const RowsRay c = S.ray[r][q ? last : 0];
          if (c.n == 0) continue;
          const float m = c.df / c.da;
          const float fa = fmaf((float)(p0 + j - 1) - c.ta0, m, c.tf0);
          const float fb = fmaf((float)(p0 + j + 1) - c.ta0, m, c.tf0);
          lo = fminf(lo, fminf(fa, fb));
          hi = fmaxf(hi, fmaxf(fa, fb));
        }
      }
      const float f0 = fmaxf(floorf(lo) - 1.0f, 0.f), f1 = fminf(floorf(hi) + 2.0f, (float)(Ps - 1));
      // a list outside the box reads global memory, so a box that is not
      // wide enough is still worth staging
      S.plan[j] = f1 >= f0 ? (short)f0 : (short)-1;
    }
    // Weight lists of plane p0 + j for the rays of view g % V, into slot g / V:
    // a lane's samples i0 <= i < i1 lie between planes p - 1 and p + 1.
    auto weights = [&](int j) {
      const int b = g / V, r = g % V, q = lane >> 2;
      const RowsRay R = S.ray[r][lane];
      const float pf = (float)(p0 + j);
      const RowsWalk K(R);
      float i0 = 0.f, i1 = 0.f;
      if (j < np) {
        i0 = K.first_at(pf - 1.0f);
        i1 = K.first_at(pf + 1.0f);
      }
      float lo = 3.0e38f, hi = -3.0e38f;
      if (i1 > i0) {
        const float fx = floorf(K.tf(i0)), fy = floorf(K.tf(i1 - 1.0f));
        lo = fminf(fx, fy);
        hi = fmaxf(fx, fy) + 2.0f;
      }
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      }
      int len = hi > lo ? ((int)(fminf(hi - lo, 4096.f)) + 1) & ~1 : 0;
      if (len > kRC) len = -1;
      if ((lane & 3) == 0) S.meta[b][r][q] = RowsMeta{len ? (int)lo : 0, len};
      if (len > 0) {
        float* t = reinterpret_cast<float*>(&S.w[b][r][q][0]) + (lane & 3);
        float* const end = t + 4 * len;
        const bool frise = (R.df >= 0.f) == (R.da > 0.f);  // f rises with i
        float fc = lo, w0 = 0.f, w1 = 0.f;       // columns fc, fc + 1
        float i = frise ? i0 : i1 - 1.0f;
        const float di = frise ? 1.0f : -1.0f;
        for (float s = i0; s < i1; s += 1.0f, i += di) {
          const float tf = K.tf(i);
          // a sample's share of plane p: 1 - |ta - p|
          const float w = 1.0f - fabsf(K.ta(i) - pf);
          while (tf >= fc + 1.0f) {
            *t = w0;
            t += 4;
            w0 = w1;
            w1 = 0.f;
            fc += 1.0f;
          }
          const float wf = tf - fc;
          w0 = fmaf(w, 1.0f - wf, w0);
          w1 = fmaf(w, wf, w1);
        }
        for (; t < end; t += 4) {
          *t = w0;
          w0 = w1;
          w1 = 0.f;
        }
      }
    };
    const CUtensorMap* tm = xdom ? &tmx : &tmy;
    __syncthreads();  // plans
    auto issue = [&](int j) {  // thread 0: the box of plane p0 + j into buffer j % NB
      if (j >= min(np, kRPlans) || S.plan[j] < 0 || S.abort) return;
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_expect_tx(&S.bar[j % NB], (uint32_t)(kStage * sizeof(TV)));
      const int f = S.plan[j], a = p0 + j;
      tma_load_3d(buf + (size_t)(j % NB) * kStage, tm, chunk * kRZ, xdom ? a : f, xdom ? f : a,
                  &S.bar[j % NB]);
      issued += 1ull << (16 * (j % NB));
    };
    if (tid == 0)
      for (int j = 0; j < min(np, NB); ++j) issue(j);
    auto landed = [&](int j) {
      if (j >= kRPlans || S.plan[j] < 0) return false;
      const bool ok = mbar_wait_bounded(&S.bar[j % NB], (phase >> (j % NB)) & 1u, E.err, &S.abort,
                                        E.wait_us);
      phase ^= 1u << (j % NB);
      return ok;
    };
    for (int j = 0; j < np; ++j) {
      const bool staged = landed(j);
      if (j % PG == 0) {  // the last group's weights are spent
        weights(j + g / V);
        __syncthreads();
      }
      const int f0 = j < kRPlans ? S.plan[j] : -1, slot = j % PG;
      const TV* b = buf + (size_t)(j % NB) * kStage + 4 * lane;
#pragma unroll
      for (int r = 0; r < V; ++r) {
        const RowsMeta m = S.meta[slot][r][g];
        if (m.n < 0) {  // too many columns for a list: the plane's samples in turn
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const RowsWalk K(S.ray[r][4 * g + i]);
            const float pf = (float)(p0 + j), i1 = K.first_at(pf + 1.0f);
            for (float s = K.first_at(pf - 1.0f); s < i1; s += 1.0f) {
              const float tf = K.tf(s), ff = floorf(tf), wf = tf - ff;
              const float w = 1.0f - fabsf(K.ta(s) - pf);
              const float wl = w * (1.0f - wf), wr = w * wf;
              const Quad a = ld_quad(vol + rows_col(Ps, xdom, p0 + j, (int)ff) * pitch + zoff);
              const Quad c = ld_quad(vol + rows_col(Ps, xdom, p0 + j, (int)ff + 1) * pitch + zoff);
              const float2 l2 = make_float2(wl, wl), r2 = make_float2(wr, wr);
              acc[r][i][0] = __ffma2_rn(r2, c.lo, __ffma2_rn(l2, a.lo, acc[r][i][0]));
              acc[r][i][1] = __ffma2_rn(r2, c.hi, __ffma2_rn(l2, a.hi, acc[r][i][1]));
            }
          }
          continue;
        }
        const float4* w = &S.w[slot][r][g][0];
        auto apply = [&](float4 wt, Quad d) {
          const float wu[4] = {wt.x, wt.y, wt.z, wt.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 w2 = make_float2(wu[i], wu[i]);
            acc[r][i][0] = __ffma2_rn(w2, d.lo, acc[r][i][0]);
            acc[r][i][1] = __ffma2_rn(w2, d.hi, acc[r][i][1]);
          }
        };
        if (staged && m.f >= f0 && m.f + m.n <= f0 + kRF) {
          const TV* d = b + (m.f - f0) * kRZ;
#pragma unroll 2
          for (int c = 0; c < m.n; c += 2) {
            const Quad d0 = ld_quad(d + c * kRZ), d1 = ld_quad(d + (c + 1) * kRZ);
            apply(w[c], d0);
            apply(w[c + 1], d1);
          }
        } else {
          for (int c = 0; c < m.n; ++c)
            apply(w[c], ld_quad(vol + rows_col(Ps, xdom, p0 + j, m.f + c) * pitch + zoff));
        }
      }
      __syncthreads();  // buffer j % NB is free
      if (tid == 0 && j + NB < np) issue(j + NB);
    }
    // Sums that are not finite: again, sample by sample, for the rows concerned.
    if constexpr (SP == 1) {
#pragma unroll
      for (int r = 0; r < V; ++r)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (mine[r]) redo(acc[r][i], S.ray[r][4 * g + i], xdom);
    }
  }
  if (tid == 0 && S.abort) slab_drain(S.bar, issued, E.err);
  if constexpr (SP > 1) {
    // every copy has landed: the quarters' sums over the stage buffers
    __syncthreads();
    float* part = reinterpret_cast<float*>(smem_raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float q[4] = {acc[0][i][0].x, acc[0][i][0].y, acc[0][i][1].x, acc[0][i][1].y};
#pragma unroll
      for (int z = 0; z < 4; ++z) part[(4 * i + z) * kRThreads + tid] = q[z];
    }
    cluster_sync();
    float q[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int z = 0; z < 4; ++z) {
      if (z < zb || z >= zb + NZ) continue;
      const float* p = part + (4 * ray + z) * kRThreads + tid;
      q[z] = cluster_ld(p, 0);
#pragma unroll
      for (int c = 1; c < SP; ++c) q[z] += cluster_ld(p, c);
    }
    cluster_sync();  // the other CTAs have read this one's
    acc[0][0][0] = make_float2(q[0], q[1]);
    acc[0][0][1] = make_float2(q[2], q[3]);
    const Trig t = A.trig[v0];
    redo(acc[0][0], S.ray[0][4 * g + ray], fabsf(t.c) >= fabsf(t.s));
  }

  constexpr int NI = SP > 1 ? 1 : 4;  // rays of this thread's warp in each view
  double obj = 0.0;
#pragma unroll
  for (int r = 0; r < V; ++r) {
    if (r >= nv) continue;
    const long long gv = A.view0 + (long long)(v0 + r) * A.vstride;
    const int ix0 = u0 + 4 * g + (SP > 1 ? ray : 0);
    // detector row = slice of the whole volume
    const size_t gi0 = (size_t)gv * A.P + (size_t)(z0 + A.zoff) * A.det_w + ix0;
    auto valid = [&](int z, int i) {
      return z0 + z < A.zrows - 2 && ix0 + i < A.det_w && z >= zb && z < zb + NZ;
    };
    float pre[EPI ? 4 : 1][NI], post[EPI ? 4 : 1][NI];
    if constexpr (EPI != 0) {  // all counts before the first store
#pragma unroll
      for (int z = 0; z < 4; ++z)
#pragma unroll
        for (int i = 0; i < NI; ++i) {
          const size_t gi = gi0 + (size_t)z * A.det_w + i;
          pre[z][i] = valid(z, i) ? __ldg(E.pre + gi) : 0.f;
          post[z][i] = valid(z, i) ? __ldg(E.post + gi) : 0.f;
        }
    }
#pragma unroll
    for (int z = 0; z < 4; ++z) {
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        if (!valid(z, i)) continue;
        const float2 q = acc[r][i][z >> 1];
        const float l = ((z & 1) ? q.y : q.x) * A.step;
        if constexpr (EPI == 0) {
          TO* o = out + gi0 + (size_t)z * A.det_w + i;
          stf(o, A.accum ? ldp(o) + l : l);
        } else {
          const float pv = pre[z][i], qv = post[z][i];
          if constexpr (EPI == 2) {
            obj += (double)(pv * expf(-l)) + (double)qv * (double)l;
          } else {
            // CUDAmex_oscIter.cu:262-268, into the residual views' quads (as the
            // slab kernel's epilogue)
            const float ehat = pv * expf(-l);
            const int Wp = sino_pad_pitch(A.det_w), iy = z0 + z + A.zoff;
            const size_t ri = ((size_t)(v0 + r) * (A.det_h + 2 * kSinoPad) + (iy + kSinoPad)) * Wp +
                              (ix0 + i + kSinoPad);
            const float r0 = ehat - qv, r1 = ehat * l;
            const size_t qd[4] = {4 * ri, 4 * (ri - Wp) + 1, 4 * (ri - 1) + 2,
                                  4 * (ri - Wp - 1) + 3};
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              if constexpr (std::is_same<TO, float>::value) {
                static_cast<float*>(E.rpre)[qd[t]] = r0;
                static_cast<float*>(E.rpost)[qd[t]] = r1;
              } else {
                stf(static_cast<TO*>(E.rpre) + qd[t], r0 * E.rscale);
                stf(static_cast<TO*>(E.rpost) + qd[t], r1 * E.rscale);
              }
            }
          }
        }
      }
    }
  }
  if constexpr (EPI == 2) {  // FP64 in a fixed order: lanes, then warps
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) obj += __shfl_xor_sync(0xffffffffu, obj, o);
    if (lane == 0) S.wsum[g] = obj;
    __syncthreads();
    if (tid == 0) {
      double t = 0.0;
      for (int w = 0; w < kRThreads / 32; ++w) t += S.wsum[w];
      E.obj[blockIdx.x] += t;
    }
  }
}

PFN_cuTensorMapEncodeTiled_v12000 rows_encode() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }();
  return fn;
}

long long rows_ctas(const RayArgs& a, int v) {
  return (long long)((a.nviews + v - 1) / v) * ((a.det_w + kRU - 1) / kRU) *
         ((a.zrows - 2 + kRZ - 1) / kRZ);
}

// CTAs that share each tile's planes as a cluster: four for calls of few views,
// whose CTAs would leave SMs idle (an OSC subset: 84^2 x 76, 25 views per
// subset, an iteration of 5 subsets 568 us without, 350 with), eight where that
// still leaves them idle (64^2 x 40, 3 views, 12 subsets: 366 -> 286 us).  The
// rule does not look at the slices, so a slab of a volume is summed as the whole
// volume is.
int rows_split(const RayArgs& a, int sms) {
  const long long n = (long long)std::max(a.nall, a.nviews) * ((a.det_w + kRU - 1) / kRU);
  return 8 * n <= sms ? 8 : n <= sms ? 4 : 1;
}

// Views per CTA: four or two where the CTAs still fill the GPU and their
// rays' columns of one plane fit the box (neighbouring rays at 45 degrees are
// up to sqrt(2) times the magnification apart; a view shifts by its angle times
// the half diagonal; what does not fit is read from global memory), else one.
int rows_views(int geom, const RayArgs& a, int sms) {
  const double R = 0.7072 * a.S;
  const double mag = geom == 1 ? std::min(1.0 + R / std::max((double)a.SR, 1.0), 2.0) : 1.0;
  const double tile = std::min(kRU, a.det_w) * 1.4143 * mag * a.du;
  double cmin = 1.0;  // cosine of the largest angle between neighbouring views
  for (int i = 0; i + 1 < a.nviews; ++i) {
    const Trig p = a.trig[i], q = a.trig[i + 1];
    cmin = std::min(cmin, (double)p.c * q.c + (double)p.s * q.s);
  }
  const double worst = std::acos(std::max(-1.0, cmin));
  for (int v : {4, 2})
    if (rows_ctas(a, v) >= 2ll * sms && tile + (v - 1) * worst * R + 4.0 <= kRF + 2.0)
      return v;
  return 1;
}

template <int EPI, typename TV, typename TO, int V, int NB, int SP>
cudaError_t rows_go(int geom, const RayArgs& a, const CUtensorMap& mx, const CUtensorMap& my,
                    const void* vol, int Ph, void* out, const SlabEpi& e, cudaStream_t st,
                    bool attr_only) {
  auto k = fp_rows_kernel<EPI, TV, TO, V, NB, SP>;
  const size_t smem = NB * kStage * sizeof(TV) + sizeof(RowsShared<V>) + 16;
  static std::atomic<unsigned long long> done{0};  // devices whose attributes are set
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(done.load() & bit)) {
    err = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err == cudaSuccess)
      err = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared);
    if (err != cudaSuccess) return err;
    done.fetch_or(bit);
  }
  if (attr_only) return cudaSuccess;
  const long long ctas = SP * rows_ctas(a, V);
  if (ctas > 0x7fffffffLL) return cudaErrorInvalidValue;
  if constexpr (SP > 1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(kRThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = SP;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, a, geom, mx, my, (const TV*)vol, Ph, (TO*)out, e);
  } else {
    k<<<(unsigned)ctas, kRThreads, smem, st>>>(a, geom, mx, my, (const TV*)vol, Ph, (TO*)out, e);
    return cudaGetLastError();
  }
}

template <int EPI, typename TV, typename TO>
cudaError_t rows_launch(int geom, const RayArgs& a, const CUtensorMap& mx, const CUtensorMap& my,
                        const void* vol, int Ph, void* out, const SlabEpi& e, cudaStream_t st) {
#define GO(V, NB, SP, only) \
  rows_go<EPI, TV, TO, V, NB, SP>(geom, a, mx, my, vol, Ph, out, e, st, only)
  if (a.nviews <= 0) {  // no work: the kernels' attributes, before a capture
    for (cudaError_t err : {GO(1, 2, 1, true), GO(2, 2, 1, true), GO(4, 2, 1, true)})
      if (err != cudaSuccess) return err;
    if constexpr (EPI != 2)
      for (cudaError_t err : {GO(1, 2, 4, true), GO(1, 4, 4, true), GO(1, 4, 8, true)})
        if (err != cudaSuccess) return err;
    return cudaSuccess;
  }
  // (the objective's partials have room for one CTA per tile)
  if constexpr (EPI != 2) {
    const int sp = rows_split(a, device_sms());
    if (sp == 8) return GO(1, 4, 8, false);
    if (sp == 4) return 4 * rows_ctas(a, 1) > device_sms() ? GO(1, 2, 4, false) : GO(1, 4, 4, false);
  }
  const int v = rows_views(geom, a, device_sms());
  return v == 4 ? GO(4, 2, 1, false) : v == 2 ? GO(2, 2, 1, false) : GO(1, 2, 1, false);
#undef GO
}

}  // namespace

void fp_rows_shape(int geom, const RayArgs& a, int epi, int sms, int* views, int* split) {
  *split = epi == 2 ? 1 : rows_split(a, sms);
  *views = *split > 1 ? 1 : rows_views(geom, a, sms);
}

// A CTA of the rows kernel works on 128 slices whatever nz is; the slab kernel's
// work goes with its tiles of eight rows (the rows of a last, part-filled tile three
// quarters of it).  A plane of the sweep takes a wave of slab CTAs (four per SM)
// 0.29 us and a wave of rows CTAs (two per SM) of 1 / 2 / 4 views 0.75 / 1.36 / 2.0
// us, and a CTA's fixed work stands for 35 planes (slab) and 45 (four views): the
// factors below, fitted to 568 pairs of times of W = 64 .. 512 with 30 .. 720 views
// and 1 .. 128 slices.  The form taken is at most 10 % slower than the other there,
// and 4 % in all but five.  (The OSC epilogue's stores weigh more on the fewer rows
// CTAs: 256^2 x 48, 360 / 6 breaks even at ~50 slices, 1.1.)  Measured, slab ->
// rows at 16, 32, 48, 64 slices: 512^2 x 720 parallel 5.5 -> 11.0, 10.8 -> 11.0,
// 16.1 -> 11.1, 21.4 -> 11.1 ms (one slice: 1.5 -> 11.0); 128^2 x 180 156 -> 326,
// 248 -> 328, 348 -> 330, 447 -> 324 us; 512^2 x 90 0.77 -> 1.98, 1.47 -> 1.98, 2.18
// -> 1.99, 2.88 -> 1.99 ms.
// Clusters (few views) fill idle SMs: an OSC subset of 6 views of 256^2 breaks even
// at eight slices, one of 5 views of 64^2 gains at one.  Line integrals also run in
// batches, whose problems must agree with single calls bit for bit: there other
// problems fill the SMs, the clusters pay from 49 slices on, and each rows problem
// is two launches, which a problem of less than ~10 us of the slab kernel does not
// make up for (64 problems 32^3 x 30: slab 228, rows 603 us).
bool fp_uses_rows(int geom, const RayArgs& a, int nz, int epi, int sms) {
  if ((geom != 0 && geom != 1) || a.nviews <= 0) return false;
  if (sms <= 0) sms = device_sms();
  const long long views = std::max(a.nall, a.nviews), tiles_u = (a.det_w + kRU - 1) / kRU;
  const long long bundles = views * tiles_u, tz = (nz + 7) / 8;
  if (epi == 0 && bundles * tz * (a.S + 2) < 12000) return false;
  int v, split;
  fp_rows_shape(geom, a, epi, sms, &v, &split);
  if (split > 1) return epi == 0 ? tz > 6 : tz > 1 || 4 * bundles <= sms;
  const double wave = (double)((views + v - 1) / v * tiles_u) / (2.0 * sms);
  const double rows = std::max(1.0, 0.1 * wave + 0.9 * std::ceil(wave)) *
                      (v == 4 ? 6.8 * (1.0 + 45.0 / a.S) : v == 2 ? 4.7 : 2.6) *
                      (epi == 1 ? 1.1 : 1.0);
  const double slab = bundles * (0.25 * tz + 0.75 * nz / 8.0) / (4.0 * sms) * (1.0 + 35.0 / a.S);
  return slab > rows;
}

int rows_pitch(int nz, int dtype) {
  const int unit = dtype == kF32 ? 4 : 8;  // 16-byte rows for TMA
  return (nz + unit - 1) / unit * unit;
}

size_t rows_bytes(int W, int nz, int dtype) {
  return (size_t)(W + 2) * (W + 2) * rows_pitch(nz, dtype) * (dtype == kF32 ? 4 : 2);
}

cudaError_t launch_pad_rows(const void* src, int dtype, int W, int nz, bool border, void* dst,
                            cudaStream_t st) {
  const int Ph = rows_pitch(nz, dtype), Ps = W + 2;
  dim3 blk(32, 8), grd((Ps + 31) / 32, Ps, (Ph + 63) / 64);
  const int mode = border ? 1 : 0;
  if (dtype == kF32)
    pad_rows_kernel<float><<<grd, blk, 0, st>>>((const float*)src, (float*)dst, W, nz, Ph, mode);
  else if (dtype == kF16)
    pad_rows_kernel<__half><<<grd, blk, 0, st>>>((const __half*)src, (__half*)dst, W, nz, Ph, mode);
  else
    pad_rows_kernel<__nv_bfloat16><<<grd, blk, 0, st>>>((const __nv_bfloat16*)src,
                                                        (__nv_bfloat16*)dst, W, nz, Ph, mode);
  return cudaGetLastError();
}

cudaError_t make_rows_tmap(CUtensorMap* map, const void* base, int dtype, int W, int nz,
                           bool xdom) {
  PFN_cuTensorMapEncodeTiled_v12000 fn = rows_encode();
  if (!fn) return cudaErrorNotSupported;
  const size_t es = dtype == kF32 ? 4 : 2;
  const cuuint64_t Ph = rows_pitch(nz, dtype), Ps = W + 2;
  cuuint64_t dims[3] = {Ph, Ps, Ps};
  cuuint64_t strides[2] = {Ph * es, Ps * Ph * es};
  cuuint32_t box[3] = {(cuuint32_t)kRZ, (cuuint32_t)(xdom ? 1 : kRF), (cuuint32_t)(xdom ? kRF : 1)};
  cuuint32_t estr[3] = {1, 1, 1};
  const CUtensorMapDataType dt = dtype == kF32   ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                 : dtype == kF16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                                 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  CUresult r = fn(map, dt, 3, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t launch_fp_rows(int geom, int epi, const RayArgs& a, const CUtensorMap& mx,
                           const CUtensorMap& my, const void* vol, int Ph, int vt, void* out,
                           int ot, const SlabEpi& e, cudaStream_t st) {
  if (geom != 0 && geom != 1) return cudaErrorInvalidValue;
#define GO(EP, TV, TO) return rows_launch<EP, TV, TO>(geom, a, mx, my, vol, Ph, out, e, st)
  if (epi == 1) {
    if (ot == kF16 && vt == kF32) GO(1, float, __half);
    if (ot != kF32) return cudaErrorInvalidValue;
    if (vt == kF32) GO(1, float, float);
    if (vt == kF16) GO(1, __half, float);
    GO(1, __nv_bfloat16, float);
  }
  if (epi == 2) {
    if (!e.obj || !e.pre || !e.post) return cudaErrorInvalidValue;
    if (vt == kF32) GO(2, float, float);
    if (vt == kF16) GO(2, __half, float);
    GO(2, __nv_bfloat16, float);
  }
  if (vt == kF32 && ot == kF32) GO(0, float, float);
  if (vt == kF16 && ot == kF16) GO(0, __half, __half);
  if (vt == kF16 && ot == kF32) GO(0, __half, float);
  if (vt == kBF16 && ot == kBF16) GO(0, __nv_bfloat16, __nv_bfloat16);
  if (vt == kBF16 && ot == kF32) GO(0, __nv_bfloat16, float);
#undef GO
  return cudaErrorInvalidValue;
}

}  // namespace mexct
