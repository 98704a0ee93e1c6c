// k_iter.cu -- TV descent, FP64 reductions and the FDK/FBP pre-filter.
//
// TV (CUDAmex_TVmin_3D.cu:101-234).  The reference runs three full-volume
// passes per step (gradient kernel -> thrust norm -> thrust saxpy) and stores
// the gradient.  Here a step is two passes and no gradient volume:
//   tv_norm_kernel   gradient recomputed per voxel, ||g||^2 reduced (FP32 per
//                    thread, FP64 across threads: warp shuffles, per-CTA
//                    partials, last-CTA fixed-order sum: deterministic), step
//                    scale -c/||g|| written to HBM;
//   tv_update_kernel gradient recomputed, y = x + scale*g into the other
//                    buffer of a ping-pong pair.
// Algorithmic traffic is 12 bytes per voxel per step (read x twice, write y).
// Whole FP32 descents take tv_fused_kernel instead, one sweep and one gradient
// per step, where that is faster (tv_fused_pays).  The pair serves the others,
// FP16 / BF16, captured calls, the sub-volume sweeps and the allocation-free form
// (one scratch volume).
// FP32 volumes whose x extent is a multiple of 4 use tv4_kernel (four x-voxels
// per thread, 16-byte loads and stores, packed FP32x2 arithmetic): 512^3 step
// 0.92 -> 0.55 ms, 2.9 TB/s of algorithmic traffic; other volumes tv_sweep.
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdio>

#include "kernels.h"

namespace mexct {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-level FP64 sum with a fixed tree (deterministic); blockDim.x*y*z
// threads, result valid in thread 0.
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double red[32];
  const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
  const int nt = blockDim.x * blockDim.y * blockDim.z;
  v = warp_sum(v);
  if ((tid & 31) == 0) red[tid >> 5] = v;
  __syncthreads();
  double r = 0.0;
  if (tid < 32) {
    r = (tid < (nt + 31) / 32) ? red[tid] : 0.0;
    r = warp_sum(r);
  }
  __syncthreads();
  return r;
}

// Last-CTA finalisation: every CTA stores its partial, the last one to arrive
// sums all partials in index order (deterministic).  Returns true in thread 0
// of the last CTA with *total set.
__device__ __forceinline__ bool finish_partials(double mine, double* partials,
                                                unsigned* counter,
                                                double* total) {
  __shared__ bool last;
  const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
  const int nt = blockDim.x * blockDim.y * blockDim.z;
  const unsigned nb = gridDim.x * gridDim.y * gridDim.z;
  const unsigned bid = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  if (tid == 0) {
    partials[bid] = mine;
    __threadfence();
    last = (atomicAdd(counter, 1u) == nb - 1);
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  double acc = 0.0;
  for (unsigned i = tid; i < nb; i += nt) acc += __ldcg(partials + i);
  acc = block_sum(acc);
  if (tid == 0) {
    *total = acc;
    *counter = 0u;  // ready for the next launch on this stream
  }
  return tid == 0;
}

// ---------------------------------------------------------------------------
// Tiled TV gradient.  With backward differences a_p = x_p - x_{p-1},
// b_p = x_p - x_{p-sy}, c_p = x_p - x_{p-sz} and r_p = 1/(eps + |(a,b,c)_p|),
// the four terms of the reference's gradient at voxel i are
//   g_i = (a+b+c)_i r_i - a_{i+1} r_{i+1} - b_{i+sy} r_{i+sy} - c_{i+sz} r_{i+sz}
// (CUDAmex_TVmin_3D.cu:121-152: the second to fourth terms are the first
// term's components at the +x, +y and +z neighbours), so each voxel's
// (a, b, c, r) is computed once (one reciprocal square root, one reciprocal)
// instead of four times.  A CTA of 32 x 16 threads sweeps a column tile along z:
// thread (tx, ty) computes q at its column in every plane, takes the +x
// neighbour's value by a shuffle, the +y neighbour's from shared memory (one
// barrier per plane) and the +z neighbour's from its next plane, and writes the
// voxel when tx < 31 and ty < 15 (tiles overlap by one column and one row).  The
// next plane's loads are issued before the current plane is computed.
// ---------------------------------------------------------------------------
// 32 x 16 threads (31 x 15 outputs: 91 % of the threads own a voxel, 85 % with
// 32 x 8; 512^3 step 0.978 -> 0.926 ms), 32 planes per CTA
constexpr int kTvBx = 32, kTvBy = 16, kTvZ = 32;
constexpr int kTvOx = kTvBx - 1, kTvOy = kTvBy - 1;  // output voxels per tile row / column

// Sweep of one tile: calls visit(z, x_z, g, out) for every plane z of the
// tile, with x_z the voxel value, g the gradient (0 on the volume border) and
// out whether this thread owns the voxel.
template <typename T, typename F>
__device__ __forceinline__ void tv_sweep(const T* __restrict__ v, int Nx, int Ny, int Nz,
                                         F&& visit) {
  __shared__ float sqb[2][kTvBy][kTvBx];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int gx = blockIdx.x * kTvOx + tx, gy = blockIdx.y * kTvOy + ty;
  const int z0 = blockIdx.z * kTvZ;
  const int zend = min(z0 + kTvZ, Nz);
  const size_t sy = (size_t)Nx, sz = (size_t)Nx * Ny;
  const bool incol = gx < Nx && gy < Ny;
  const bool qcol = incol && gx >= 1 && gy >= 1;  // columns where q exists
  const bool own = incol && tx < kTvOx && ty < kTvOy;
  const size_t ci = (size_t)gx + (size_t)gy * sy;
  // column-invariant parts of the interior test and of the loads
  const bool col_int = gx >= 1 && gy >= 1 && gx < Nx - 1 && gy < Ny - 1;
  const bool ld_y = gy >= 1, ld_m = tx == 0 && gx >= 1;
  const int srow = ty + (ty < kTvOy);  // row of the +y neighbour in sqb
  // value of the plane below the first one, and the first plane's loads
  float xprev = (qcol && z0 >= 1) ? ldf(v + ci + (size_t)(z0 - 1) * sz) : 0.f;
  float xcur = 0.f, xym = 0.f, xxm = 0.f;
  const T* pl = v + ci + (size_t)z0 * sz;  // column at the plane being loaded
  auto load = [&](int p, float& xo, float& yo, float& mo) {
    if (incol && p < Nz) {
      xo = ldf(pl);
      yo = ld_y ? ldf(pl - sy) : 0.f;
      mo = ld_m ? ldf(pl - 1) : 0.f;
    }
    pl += sz;
  };
  load(z0, xcur, xym, xxm);
  float q0p = 0.f, qanp = 0.f, xz = 0.f;  // plane p-1: own q0, +x neighbour's qa, x
  for (int p = z0; p <= zend; ++p) {
    float xn = 0.f, yn = 0.f, mn = 0.f;
    if (p + 1 <= zend) load(p + 1, xn, yn, mn);  // prefetch the next plane
    // x_{p-1} of lane tx is lane tx-1's x_p; lane 0 loaded it
    const float xl = __shfl_up_sync(0xffffffffu, xcur, 1);
    const float xm = tx == 0 ? xxm : xl;
    float q0 = 0.f, qa = 0.f, qb = 0.f, qc = 0.f;
    if (qcol && p >= 1 && p < Nz) {
      const float a = xcur - xm, b = xcur - xym, c = xcur - xprev;
      // |(a,b,c)| from the hardware reciprocal square root and 1/(eps + |.|)
      // from the hardware reciprocal (a few ulp each, far inside the 1e-5
      // bound; the IEEE-rounded forms cost ~4x the instructions of the whole
      // stencil).  s = 0 (flat region) gives |.| = 0 as it must.
      const float s2 = fmaf(c, c, fmaf(b, b, a * a));
      const float nrm = s2 > 0.f ? s2 * rsqrtf(s2) : 0.f;
      const float r = __fdividef(1.0f, 1.0e-6f + nrm);
      q0 = ((a + b) + c) * r;
      qa = a * r;
      qb = b * r;
      qc = c * r;
    }
    if (p > z0) {
      const int z = p - 1;
      const bool interior = col_int && z >= 1 && z < Nz - 1;
      const float g = interior ? ((q0p - qanp) - sqb[(p - 1) & 1][srow][tx]) - qc : 0.f;
      visit(z, xz, g, own && interior, own);
    }
    sqb[p & 1][ty][tx] = qb;
    qanp = __shfl_down_sync(0xffffffffu, qa, 1);
    q0p = q0;
    xz = xcur;
    xprev = xcur;
    xcur = xn;
    xym = yn;
    xxm = mn;
    __syncthreads();
  }
}

template <typename T>
__global__ void __launch_bounds__(kTvBx * kTvBy) tv_norm_kernel(
    const T* __restrict__ x, int Nx, int Ny, int Nz, float c,
    const double* __restrict__ cmul, double* __restrict__ partials,
    unsigned* __restrict__ counter, float* __restrict__ scale,
    double* __restrict__ norm) {
  // ||g||^2: squares and the 32-voxel sum of a thread in FP32, every level
  // above in FP64 (fixed order, deterministic).
  float ss = 0.f;
  tv_sweep(x, Nx, Ny, Nz, [&](int, float, float g, bool interior, bool) {
    if (interior) ss = fmaf(g, g, ss);
  });
  const double blk = block_sum((double)ss);
  double total;
  if (finish_partials(blk, partials, counter, &total)) {
    const double m = sqrt(total);
    // c_eff = c * (*cmul): the OSC-TV driver passes TV_constant * d_a with d_a
    // computed on the device (OSC_TV_recon.m:68).
    const double ce = cmul ? (double)c * __ldcg(cmul) : (double)c;
    *norm = m;
    *scale = (float)(-ce / m);
  }
}

template <typename T>
__global__ void __launch_bounds__(kTvBx * kTvBy) tv_update_kernel(
    const T* __restrict__ x, T* __restrict__ y, int Nx, int Ny, int Nz,
    const float* __restrict__ scale) {
  const float a = __ldg(scale);
  const size_t sy = (size_t)Nx, sz = (size_t)Nx * Ny;
  const size_t ci = (size_t)(blockIdx.x * kTvOx + threadIdx.x) +
                    (size_t)(blockIdx.y * kTvOy + threadIdx.y) * sy;
  tv_sweep(x, Nx, Ny, Nz, [&](int z, float xv, float g, bool, bool own) {
    // x <- a*g + x (thrust saxpy, CUDAmex_TVmin_3D.cu:232); border g = 0.
    if (own) stf(y + ci + (size_t)z * sz, fmaf(a, g, xv));
  });
}

// ---------------------------------------------------------------------------
// TV sweep, four x-voxels per thread (FP32 volumes with Nx % 4 == 0 and
// 16-byte aligned pointers).  Same per-voxel arithmetic as tv_sweep, in the
// same order, with every elementwise step done as two packed FP32x2
// operations and each thread's row segment moved by one 16-byte load or
// store: a thread's per-plane cost (loop, barrier, addresses, predicates) is
// shared by four voxels.  A CTA of 32 x 16 threads covers 128 x 16 columns
// and owns 124 x 15 of them: the last lane's four columns and the last row
// give the +x / +y neighbours' terms (the stride of 124 keeps every segment
// 16-byte aligned).  The norm sums a segment's squares in FP32 and segments as
// two floats (add_squares); everything above is FP64 as in tv_norm_kernel.
// ---------------------------------------------------------------------------
constexpr int kT4Bx = 32, kT4By = 16, kT4Z = 32;
constexpr int kT4Ox = kT4Bx * 4 - 4, kT4Oy = kT4By - 1;  // 124 x 15 outputs

// a - b as one packed fma with -1 (the product is exact, so the result is the
// correctly rounded difference, as a subtraction gives).
__device__ __forceinline__ float2 tv_sub2(float2 a, float2 b) {
  return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a);
}

// Four voxels as two pairs.
struct V4 {
  float2 lo, hi;
};
__device__ __forceinline__ V4 v4(float4 f) { return V4{make_float2(f.x, f.y), make_float2(f.z, f.w)}; }
__device__ __forceinline__ V4 sub4(V4 a, V4 b) { return V4{tv_sub2(a.lo, b.lo), tv_sub2(a.hi, b.hi)}; }
__device__ __forceinline__ V4 add4(V4 a, V4 b) { return V4{__fadd2_rn(a.lo, b.lo), __fadd2_rn(a.hi, b.hi)}; }
__device__ __forceinline__ V4 mul4(V4 a, V4 b) { return V4{__fmul2_rn(a.lo, b.lo), __fmul2_rn(a.hi, b.hi)}; }
__device__ __forceinline__ V4 fma4(V4 a, V4 b, V4 c) {
  return V4{__ffma2_rn(a.lo, b.lo, c.lo), __ffma2_rn(a.hi, b.hi, c.hi)};
}

// 1 / (eps + |(a, b, c)|) of four voxels by the hardware reciprocal square root
// and reciprocal: |.| = s2 rsqrt(s2).  s2 starts from FLT_MIN (no effect beside
// eps), so both arguments are normal and the flush-to-zero forms need no range
// tests.  Each is within its documented error (a few ulp; 1 / x would be correctly
// rounded): the tests hold whole steps to 1e-5 of the oracle.
__device__ __forceinline__ float rsqrt_normal(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rcp_normal(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ V4 tv_recip(V4 a, V4 b, V4 c) {
  const float2 tiny = make_float2(1.17549435e-38f, 1.17549435e-38f);
  const float2 eps = make_float2(1.0e-6f, 1.0e-6f);
  const V4 s2 = fma4(c, c, fma4(b, b, fma4(a, a, V4{tiny, tiny})));
  const V4 rs{make_float2(rsqrt_normal(s2.lo.x), rsqrt_normal(s2.lo.y)),
              make_float2(rsqrt_normal(s2.hi.x), rsqrt_normal(s2.hi.y))};
  const V4 den = fma4(s2, rs, V4{eps, eps});
  return V4{make_float2(rcp_normal(den.lo.x), rcp_normal(den.lo.y)),
            make_float2(rcp_normal(den.hi.x), rcp_normal(den.hi.y))};
}

// Sum of squares of the four voxels of a segment in FP32, added to a running
// sum kept as two floats (the rounding of every addition in lo): a thread's
// sum is good to ~1e-14, so the norm does not depend on which tiles grouped
// the segments, and the kernels that tile differently give the same step scale.
__device__ __forceinline__ void add_squares(float4 g, float2& sum) {
  const float q = fmaf(g.w, g.w, fmaf(g.z, g.z, fmaf(g.y, g.y, g.x * g.x)));
  const float s = sum.x + q, b = s - sum.x;
  sum.y += (sum.x - (s - b)) + (q - b);
  sum.x = s;
}

// mode 0: ||g||^2 reduction (scale / norm written by the last CTA);
// mode 1: y = x + scale*g for the owned voxels.
template <int MODE>
__global__ void __launch_bounds__(kT4Bx * kT4By, 2) tv4_kernel(
    const float* __restrict__ v, float* __restrict__ yout, int Nx, int Ny, int Nz, float c,
    const double* __restrict__ cmul, double* __restrict__ partials,
    unsigned* __restrict__ counter, float* __restrict__ scale, double* __restrict__ norm,
    const float* __restrict__ scale_in) {
  __shared__ float4 qbs[2][kT4By][kT4Bx];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int gx0 = blockIdx.x * kT4Ox + tx * 4, gy = blockIdx.y * kT4Oy + ty;
  const int z0 = blockIdx.z * kT4Z;
  const int zend = min(z0 + kT4Z, Nz);
  // 32-bit element offsets (the volume holds fewer than 2^31 voxels)
  const int sy = Nx, sz = Nx * Ny;
  const bool incol = gx0 < Nx && gy < Ny;  // Nx % 4 == 0: the whole segment is in range
  const bool own = incol && tx < kT4Bx - 1 && ty < kT4Oy;
  const bool ld_y = incol && gy >= 1, ld_l = incol && tx == 0 && gx0 >= 1;
  const bool row_int = gy >= 1 && gy < Ny - 1;
  // interior columns of the segment as 0/1 masks (g is 0 on the volume border)
  float xin[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) xin[e] = (gx0 + e >= 1 && gx0 + e < Nx - 1 && row_int) ? 1.f : 0.f;
  const V4 xmask{make_float2(xin[0], xin[1]), make_float2(xin[2], xin[3])};
  const float a_upd = MODE == 1 ? __ldg(scale_in) : 0.f;
  const float2 a2 = make_float2(a_upd, a_upd);
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  // offset of the column at plane z0 (the row above and the left neighbour are
  // read only where they exist)
  int oc = gx0 + gy * sy + z0 * sz;
  auto ld4 = [&](int o, bool ok) {
    return ok ? __ldg(reinterpret_cast<const float4*>(v + o)) : z4;
  };
  V4 xprev = v4(ld4(oc - sz, incol && z0 >= 1));
  float4 xc4 = ld4(oc, incol && z0 < Nz);
  float4 xy4 = ld4(oc - sy, ld_y && z0 < Nz);
  float xl = (ld_l && z0 < Nz) ? __ldg(v + oc - 1) : 0.f;
  V4 q0p{}, qap{}, xz{};
  float qa_next = 0.f;  // +x neighbour's qa of the previous plane (lane + 1, element 0)
  float2 ss = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int p = z0; p <= zend; ++p) {
    // prefetch the next plane
    const int on = oc + sz;
    const bool nxt = p + 1 <= zend && p + 1 < Nz;
    const float4 xn4 = ld4(on, incol && nxt), yn4 = ld4(on - sy, ld_y && nxt);
    const float ln = (ld_l && nxt) ? __ldg(v + on - 1) : 0.f;
    const V4 xc = v4(xc4), xy = v4(xy4);
    // x - 1 of element 0: lane tx-1's element 3 (lane 0 loaded it)
    const float left = __shfl_up_sync(0xffffffffu, xc4.w, 1);
    const V4 xm{make_float2(tx == 0 ? xl : left, xc4.x), make_float2(xc4.y, xc4.z)};
    const V4 a = sub4(xc, xm), b = sub4(xc, xy), cc = sub4(xc, xprev);
    // 0 where q does not exist
    const float qm = (incol && gy >= 1 && p >= 1 && p < Nz) ? 1.f : 0.f;
    const float2 qm2 = make_float2(qm, qm);
    const V4 r = mul4(V4{qm2, qm2}, tv_recip(a, b, cc));
    const V4 q0 = mul4(add4(add4(a, b), cc), r);
    const V4 qa = mul4(a, r), qb = mul4(b, r), qc = mul4(cc, r);
    if (p > z0) {
      // g of plane p - 1 = q0 - qa(x+1) - qb(y+1) - qc(z+1), 0 on the border
      const int z = p - 1;
      const float zm = (z >= 1 && z < Nz - 1) ? 1.f : 0.f;
      const float4 qbb = qbs[(p - 1) & 1][ty + (ty < kT4By - 1)][tx];
      const V4 qan{make_float2(qap.lo.y, qap.hi.x), make_float2(qap.hi.y, qa_next)};
      V4 g = sub4(sub4(sub4(q0p, qan), v4(qbb)), qc);
      const float2 zm2 = make_float2(zm, zm);
      g = V4{__fmul2_rn(__fmul2_rn(g.lo, xmask.lo), zm2), __fmul2_rn(__fmul2_rn(g.hi, xmask.hi), zm2)};
      if (MODE == 0) {
        if (own) add_squares(make_float4(g.lo.x, g.lo.y, g.hi.x, g.hi.y), ss);
      } else if (own) {
        const float2 lo = __ffma2_rn(a2, g.lo, xz.lo), hi = __ffma2_rn(a2, g.hi, xz.hi);
        *reinterpret_cast<float4*>(yout + (oc - sz)) = make_float4(lo.x, lo.y, hi.x, hi.y);
      }
    }
    oc = on;
    qbs[p & 1][ty][tx] = make_float4(qb.lo.x, qb.lo.y, qb.hi.x, qb.hi.y);
    qa_next = __shfl_down_sync(0xffffffffu, qa.lo.x, 1);
    q0p = q0;
    qap = qa;
    xz = xc;
    xprev = xc;
    xc4 = xn4;
    xy4 = yn4;
    xl = ln;
    __syncthreads();
  }
  if (MODE == 0) {
    const double blk = block_sum((double)ss.x + (double)ss.y);
    double total;
    if (finish_partials(blk, partials, counter, &total)) {
      const double m = sqrt(total);
      const double ce = cmul ? (double)c * __ldg(cmul) : (double)c;
      *norm = m;
      *scale = (float)(-ce / m);
    }
  }
}

// ---------------------------------------------------------------------------
// Fused TV steps (FP32).  tv_norm + tv_update evaluate the gradient twice per
// step.  Here a sweep stores it: step k reads x_k and g_k = g(x_k), forms
// x_{k+1} = x_k + scale_k g_k on its tile and the tile's halo, and in the same
// sweep writes x_{k+1}, g_{k+1} = g(x_{k+1}) and its norm: one gradient per
// step and 16 bytes per voxel instead of two gradients and 12 bytes (the pair
// was issue-bound at 80 % of the issue slots).  Per voxel the operations are
// tv4_kernel's, in its order; only the norm's partial sums are grouped by
// other tiles.
//
// A CTA is 8 rows (7 of them its own) of WX warps of 128 columns.  Tiles do not
// overlap in x: the right neighbour's term crosses warps through shared memory
// with the +y terms, and past the tile's end its last lane evaluates that one
// term itself (at 256^3 tv4_kernel's 124-column tiles covered 372 columns and
// filled 1.4 waves).  Buffers between the steps have rows of a multiple of four
// voxels (the spare columns hold zeros), so any Nx takes this path: only the
// first two sweeps read the caller's rows (XVEC: whole and aligned rows).
// 20 steps, pairs -> fused: 64^3 0.82 -> 0.21 ms, 127^3 0.90 -> 0.30, 256^3
// 1.99 -> 1.26 (60 us a sweep: 240 MB of DRAM traffic, 3.9 TB/s; loads one
// plane ahead in 32 warps of 64 registers per SM is what waits, long
// scoreboard first), 255^2 x 201 2.31 -> 1.28, 384^2 x 300 4.23 -> 3.55,
// 512^3 10.95 -> 9.99.  Measured and not kept: 1024-thread CTAs over 512
// columns (384^2 x 300: 4.53 ms), L2 prefetches four planes ahead (1.93 ms at
// 256^3).
// ---------------------------------------------------------------------------
constexpr int kTfRows = 8, kTfOy = kTfRows - 1;

struct TvFused {
  const float* x;   // x_k: rows of xp voxels
  const float* g;   // g_k (mode 1)
  float* y;         // x_{k+1} (mode 1)
  float* gout;      // g of the sweep's volume
  int xp, gp;       // row pitch of x; of g, y and gout (a multiple of 4)
  int Nx, Ny, Nz, zc;
  float c;
  const double* cmul;
  double* partials;
  unsigned* counter;
  const float* scale_in;
  float* scale_out;
  double* norm;
};

// mode 0: g and norm of x; mode 1: x + scale g, then g and norm of that.
// EDGE: several tiles along x (WX = 1; 80 registers instead of 64).
template <int MODE, int WX, bool XVEC, bool EDGE>
__global__ void __launch_bounds__(32 * WX * kTfRows, EDGE ? 3 : 4 / WX) tv_fused_kernel(const TvFused A) {
  constexpr int TX = 32 * WX;
  __shared__ float4 qbs[2][kTfRows][TX];
  __shared__ float qas[2][kTfRows][WX + 1];
  const int tx = threadIdx.x, ty = threadIdx.y, lane = tx & 31, wx = tx >> 5;
  const int gx0 = blockIdx.x * (4 * TX) + tx * 4, gy = blockIdx.y * kTfOy + ty;
  const int Nx = A.Nx, Ny = A.Ny, Nz = A.Nz;
  const int z0 = blockIdx.z * A.zc, zend = min(z0 + A.zc, Nz);
  const bool incol = gx0 < Nx && gy < Ny;
  const bool own = incol && (ty < kTfOy || gy == Ny - 1);
  // the last lane needs a column past the tile
  const bool rgt = EDGE && lane == 31 && blockIdx.x != gridDim.x - 1;
  const bool row_int = gy >= 1 && gy < Ny - 1;
  bool xin[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) xin[e] = row_int && gx0 + e >= 1 && gx0 + e < Nx - 1;
  const float s = MODE == 1 ? __ldg(A.scale_in) : 0.f;
  const float2 s2v = make_float2(s, s);
  // Loads are unconditional, from the nearest place that exists: a column, row
  // above, left neighbour or plane that does not exist is read by terms that
  // no interior voxel takes.
  const int cx = min(gx0, A.gp - 4), cy = min(gy, Ny - 1), cu = max(cy - 1, 0);
  const int xsz = A.xp * Ny, gsz = A.gp * Ny;
  const float* px = A.x + cx + (size_t)A.xp * cy;
  const float* gx = A.g + cx + (size_t)A.gp * cy;
  const int xup = (cu - cy) * A.xp, gup = (cu - cy) * A.gp, lf = cx > 0 ? -1 : 0;
  auto ldx = [&](const float* p) {  // four voxels of a row (those past its end are 0)
    if (XVEC) return __ldg(reinterpret_cast<const float4*>(p));
    float4 v;
    v.x = __ldg(p);
    v.y = cx + 1 < Nx ? __ldg(p + 1) : 0.f;
    v.z = cx + 2 < Nx ? __ldg(p + 2) : 0.f;
    v.w = cx + 3 < Nx ? __ldg(p + 3) : 0.f;
    return v;
  };
  auto ldg4 = [&](const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); };
  auto step4 = [&](float4 x, float4 g) {  // x + s g
    V4 r{__ffma2_rn(s2v, make_float2(g.x, g.y), make_float2(x.x, x.y)),
         __ffma2_rn(s2v, make_float2(g.z, g.w), make_float2(x.z, x.w))};
    return r;
  };
  // raw values of plane p: own segment, the row above, the left neighbour
  struct Raw {
    float4 x, xu, g, gu;
    float xl, gl;            // left of the warp
    float xr, xru, gr, gru;  // right of the tile, and above that
  };
  auto load = [&](int p) {
    Raw r;
    const int pc = min(max(p, 0), Nz - 1);
    const float* xo = px + (size_t)pc * xsz;
    r.x = ldx(xo);
    r.xu = ldx(xo + xup);
    r.xl = lane == 0 ? __ldg(xo + lf) : 0.f;
    r.xr = r.xru = r.gr = r.gru = 0.f;
    if (EDGE && rgt) {
      r.xr = __ldg(xo + 4);
      r.xru = __ldg(xo + xup + 4);
    }
    if (MODE == 1) {
      const float* go = gx + (size_t)pc * gsz;
      r.g = ldg4(go);
      r.gu = ldg4(go + gup);
      r.gl = lane == 0 ? __ldg(go + lf) : 0.f;
      if (EDGE && rgt) {
        r.gr = __ldg(go + 4);
        r.gru = __ldg(go + gup + 4);
      }
    }
    return r;
  };
  V4 prev;
  float prevr = 0.f;
  {
    const size_t pc = max(z0 - 1, 0);
    const float4 xv = ldx(px + pc * xsz);
    prev = MODE == 1 ? step4(xv, ldg4(gx + pc * gsz)) : v4(xv);
    if (EDGE && rgt) {
      prevr = __ldg(px + pc * xsz + 4);
      if (MODE == 1) prevr = fmaf(s, __ldg(gx + pc * gsz + 4), prevr);
    }
  }
  Raw cur = load(z0);
  int og = gx0 + A.gp * gy + z0 * gsz;  // this plane's segment in y and gout
  V4 q0p{}, qap{};
  float qa_next = 0.f;
  float2 ss = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int p = z0; p <= zend; ++p) {
    const Raw nxt = load(p + 1);
    const V4 xc = MODE == 1 ? step4(cur.x, cur.g) : v4(cur.x);
    const V4 xu = MODE == 1 ? step4(cur.xu, cur.gu) : v4(cur.xu);
    const float xl = MODE == 1 ? fmaf(s, cur.gl, cur.xl) : cur.xl;
    if (MODE == 1 && own && p < zend)
      *reinterpret_cast<float4*>(A.y + og) = make_float4(xc.lo.x, xc.lo.y, xc.hi.x, xc.hi.y);
    const float left = __shfl_up_sync(0xffffffffu, xc.hi.y, 1);
    const V4 xm{make_float2(lane == 0 ? xl : left, xc.lo.x), make_float2(xc.lo.y, xc.hi.x)};
    const V4 a = sub4(xc, xm), b = sub4(xc, xu), cc = sub4(xc, prev);
    const V4 r = tv_recip(a, b, cc);
    const V4 q0 = mul4(add4(add4(a, b), cc), r);
    const V4 qa = mul4(a, r), qb = mul4(b, r), qc = mul4(cc, r);
    if (p > z0) {
      // g of plane z = p - 1; every term it takes exists where it is interior
      const int z = p - 1;
      if (lane == 31) qa_next = qas[z & 1][ty][wx + 1];
      const float4 qbb = qbs[z & 1][min(ty + 1, kTfRows - 1)][tx];
      const V4 qan{make_float2(qap.lo.y, qap.hi.x), make_float2(qap.hi.y, qa_next)};
      const V4 g = sub4(sub4(sub4(q0p, qan), v4(qbb)), qc);
      float4 gm = make_float4(xin[0] ? g.lo.x : 0.f, xin[1] ? g.lo.y : 0.f,
                              xin[2] ? g.hi.x : 0.f, xin[3] ? g.hi.y : 0.f);
      if (z < 1 || z >= Nz - 1) gm = make_float4(0.f, 0.f, 0.f, 0.f);
      if (own) {
        add_squares(gm, ss);
        *reinterpret_cast<float4*>(A.gout + (og - gsz)) = gm;
      }
    }
    qbs[p & 1][ty][tx] = make_float4(qb.lo.x, qb.lo.y, qb.hi.x, qb.hi.y);
    if (lane == 0) qas[p & 1][ty][wx] = qa.lo.x;
    qa_next = __shfl_down_sync(0xffffffffu, qa.lo.x, 1);
    if (EDGE) {  // the term of the first column past the tile, kept for plane p
      const float xr = MODE == 1 ? fmaf(s, cur.gr, cur.xr) : cur.xr;
      const float xru = MODE == 1 ? fmaf(s, cur.gru, cur.xru) : cur.xru;
      const float ar = xr - xc.hi.y, br = xr - xru, cr = xr - prevr;
      const float sr = fmaf(cr, cr, fmaf(br, br, fmaf(ar, ar, 1.17549435e-38f)));
      const float qr = ar * rcp_normal(fmaf(sr, rsqrt_normal(sr), 1.0e-6f));
      if (lane == 31) qas[p & 1][ty][WX] = qr;
      prevr = xr;
    }
    q0p = q0;
    qap = qa;
    prev = xc;
    cur = nxt;
    og += gsz;
    __syncthreads();
  }
  const double blk = block_sum((double)ss.x + (double)ss.y);
  double total;
  if (finish_partials(blk, A.partials, A.counter, &total)) {
    const double m = sqrt(total);
    const double ce = A.cmul ? (double)A.c * __ldcg(A.cmul) : (double)A.c;
    *A.norm = m;
    *A.scale_out = (float)(-ce / m);
  }
}

// out = x + scale g, from rows of xp and gp voxels to the caller's rows of Nx.
// out may be x.
__global__ void __launch_bounds__(256) tv_last_kernel(const float* x, int xp,
                                                      const float* __restrict__ g, int gp,
                                                      float* out, int Nx, long long rows,
                                                      const float* __restrict__ scale) {
  const float s = __ldg(scale);
  const long long step = (long long)gridDim.x * 8;
  for (long long r = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += step)
    for (int i = threadIdx.x & 31; i < Nx; i += 32)
      out[r * Nx + i] = fmaf(s, __ldg(g + r * gp + i), x[r * xp + i]);
}

__global__ void __launch_bounds__(256) tv_last4_kernel(const float4* x,
                                                       const float4* __restrict__ g, float4* out,
                                                       long long n,
                                                       const float* __restrict__ scale) {
  const float s = __ldg(scale);
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
    const float4 a = x[i], b = __ldg(g + i);
    out[i] = make_float4(fmaf(s, b.x, a.x), fmaf(s, b.y, a.y), fmaf(s, b.z, a.z), fmaf(s, b.w, a.w));
  }
}

static int tvf_pitch(int Nx) { return (Nx + 3) & ~3; }
// Warps along x: one or two for rows of one tile, else tiles of one.
static int tvf_wx(int Nx) { return Nx > 128 && Nx <= 256 ? 2 : 1; }

// Tiles of a fused sweep.  Slices per CTA: 32 (one slice in 33 is done twice),
// fewer where the grid would leave SMs idle.
static dim3 tvf_grid(int Nx, int Ny, int Nz, int* zc) {
  const int wx = tvf_wx(Nx);
  const unsigned gx = (Nx + 128 * wx - 1) / (128 * wx);
  const unsigned gy = std::max(1, (Ny - 1 + kTfOy - 1) / kTfOy);
  int z = 32;
  while (z > 4 && 2 * (long long)gx * gy * ((Nz + z - 1) / z) * wx < 7ll * device_sms()) z /= 2;
  *zc = z;
  return dim3(gx, gy, (Nz + z - 1) / z);
}

size_t tv_fused_elems(int Nx, int Ny, int Nz) { return (size_t)tvf_pitch(Nx) * Ny * Nz; }

size_t tv_fused_partials(int Nx, int Ny, int Nz) {
  int zc;
  const dim3 g = tvf_grid(Nx, Ny, Nz, &zc);
  return (size_t)g.x * g.y * g.z;
}

bool tv_fused_ok(int Nx, int Ny, int Nz) {
  int zc;
  const dim3 g = tvf_grid(Nx, Ny, Nz, &zc);
  return g.y <= 65535 && g.z <= 65535 &&
         (long long)tvf_pitch(Nx) * Ny * ((long long)Nz + 2) < (1LL << 31);
}

// Whether the fused steps are the faster form.  Rows that are not whole: always
// (the pair would be the scalar tv_sweep).  Else the pair's tiles of 124 x 15
// columns stand against tiles of 128 x 7, which cost half as much each and move
// more memory: once the pair fills two CTAs on most SMs, a step of the pair takes
// 1.95 times the tiles' ratio of a fused step's time, and the first and last sweep
// of a fused descent add 0.2 steps.  So the columns that the tiles waste decide:
// 20 steps, pair and fused, 512^3 10.95 and 9.95 ms, 384^3 5.36 and 4.46, but 600^2
// x 300 7.38 and 8.15, 372 x 360 x 200 2.15 and 2.48; one step, 512^3 547 and 587
// us.  Below that the pair's latency counts: 256^2 x 16 0.54 and 0.25 ms, 248 x 240
// x 240 1.40 and 1.20.
bool tv_fused_pays(int Nx, int Ny, int Nz, int n_steps, bool whole, int sms) {
  if (!whole) return true;
  if (sms <= 0) sms = device_sms();
  const long long pair = (long long)((Nx + kT4Ox - 1) / kT4Ox) * ((Ny + kT4Oy - 1) / kT4Oy);
  const long long fused = (long long)((Nx + 127) / 128) * std::max(1, (Ny - 1 + kTfOy - 1) / kTfOy);
  if (pair * ((Nz + kT4Z - 1) / kT4Z) * 100 <= 185ll * sms) return true;
  return (n_steps + 0.2) * (double)fused <= 1.95 * n_steps * (double)pair;
}

template <int MODE, bool XVEC>
static cudaError_t tvf_go(const TvFused& a, dim3 grd, cudaStream_t st) {
  const int wx = tvf_wx(a.Nx);
  const dim3 blk(32 * wx, kTfRows);
  if (wx == 2) tv_fused_kernel<MODE, 2, XVEC, false><<<grd, blk, 0, st>>>(a);
  else if (grd.x == 1) tv_fused_kernel<MODE, 1, XVEC, false><<<grd, blk, 0, st>>>(a);
  else tv_fused_kernel<MODE, 1, XVEC, true><<<grd, blk, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_tv_fused(const float* in, float* out, int Nx, int Ny, int Nz, float c,
                            const double* cmul, int n_steps, float* work[4], double* partials,
                            unsigned* counter, float* scale2, double* norm, cudaStream_t st) {
  const int gp = tvf_pitch(Nx);
  // x_1, x_2, ... alternate between work[0] and work[3] (null: the rows are
  // whole, x_2, x_4, ... go to out); g_0, g_1, ... between work[1] and work[2]
  const bool whole = Nx % 4 == 0 && ((uintptr_t)in & 15) == 0 && ((uintptr_t)out & 15) == 0;
  float* xb[2] = {work[0], whole ? out : work[3]};
  // (the last sweep would turn rows of gp voxels into rows of Nx in place)
  if (!xb[1] || (!whole && xb[1] == out && n_steps % 2 != 0)) return cudaErrorInvalidValue;
  TvFused a{};
  a.gp = gp;
  a.Nx = Nx;
  a.Ny = Ny;
  a.Nz = Nz;
  const dim3 grd = tvf_grid(Nx, Ny, Nz, &a.zc);
  a.c = c;
  a.cmul = cmul;
  a.partials = partials;
  a.counter = counter;
  a.norm = norm;
  const float* x = in;
  int xp = Nx;
  for (int k = 0; k < n_steps; ++k) {  // g_k, from x_{k-1} and g_{k-1} for k > 0
    a.x = x;
    a.xp = xp;
    a.gout = work[1 + (k & 1)];
    a.scale_out = scale2 + (k & 1);
    const bool vec = xp % 4 == 0 && ((uintptr_t)x & 15) == 0;
    cudaError_t e;
    if (k == 0) {
      e = vec ? tvf_go<0, true>(a, grd, st) : tvf_go<0, false>(a, grd, st);
    } else {
      a.g = work[1 + ((k - 1) & 1)];
      a.scale_in = scale2 + ((k - 1) & 1);
      a.y = xb[(k - 1) & 1];
      e = vec ? tvf_go<1, true>(a, grd, st) : tvf_go<1, false>(a, grd, st);
      x = a.y;
      xp = gp;
    }
    if (e != cudaSuccess) return e;
  }
  const float* g = work[1 + ((n_steps - 1) & 1)];
  const float* scale = scale2 + ((n_steps - 1) & 1);
  const int ctas = device_sms() * 8;
  if (xp == Nx && gp == Nx && (((uintptr_t)x | (uintptr_t)out) & 15) == 0) {
    tv_last4_kernel<<<ctas, 256, 0, st>>>(reinterpret_cast<const float4*>(x),
                                          reinterpret_cast<const float4*>(g),
                                          reinterpret_cast<float4*>(out),
                                          (long long)Nx / 4 * Ny * Nz, scale);
  } else {
    tv_last_kernel<<<ctas, 256, 0, st>>>(x, xp, g, gp, out, Nx, (long long)Ny * Nz, scale);
  }
  return cudaGetLastError();
}

static bool tv4_ok(const void* x, const void* y, int xt, int Nx, int Ny, int Nz) {
  return xt == kF32 && Nx % 4 == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)y & 15) == 0 &&
         (long long)Nx * Ny * (Nz + 1) < (1LL << 31);
}

static dim3 tv4_grid(int Nx, int Ny, int Nz) {
  return dim3((Nx + kT4Ox - 1) / kT4Ox, (Ny + kT4Oy - 1) / kT4Oy, (Nz + kT4Z - 1) / kT4Z);
}

static dim3 tv_grid(int Nx, int Ny, int Nz) {
  return dim3((Nx + kTvOx - 1) / kTvOx, (Ny + kTvOy - 1) / kTvOy, (Nz + kTvZ - 1) / kTvZ);
}

size_t tv_partials_needed(int Nx, int Ny, int Nz) {
  // the four-voxel grid never has more CTAs than this one
  const dim3 g = tv_grid(Nx, Ny, Nz);
  return (size_t)g.x * g.y * g.z;
}

bool tv_shape_launchable(int Nx, int Ny, int Nz) {
  const long long gx = ((long long)Nx + kTvOx - 1) / kTvOx;
  const long long gy = ((long long)Ny + kTvOy - 1) / kTvOy, gz = ((long long)Nz + kTvZ - 1) / kTvZ;
  return gx <= 0x7fffffffLL && gy <= 65535 && gz <= 65535;
}

static cudaError_t tv_norm_go(const void* x, int xt, int Nx, int Ny, int Nz, float c,
                              const double* cmul, double* partials, unsigned* counter,
                              float* scale, double* norm, cudaStream_t st) {
  if (tv4_ok(x, x, xt, Nx, Ny, Nz)) {
    tv4_kernel<0><<<tv4_grid(Nx, Ny, Nz), dim3(kT4Bx, kT4By), 0, st>>>(
        (const float*)x, nullptr, Nx, Ny, Nz, c, cmul, partials, counter, scale, norm, nullptr);
    return cudaGetLastError();
  }
  dim3 blk(kTvBx, kTvBy), grd = tv_grid(Nx, Ny, Nz);
  if (xt == kF32)
    tv_norm_kernel<float><<<grd, blk, 0, st>>>((const float*)x, Nx, Ny, Nz, c, cmul,
                                               partials, counter, scale, norm);
  else if (xt == kF16)
    tv_norm_kernel<__half><<<grd, blk, 0, st>>>((const __half*)x, Nx, Ny, Nz, c, cmul,
                                                partials, counter, scale, norm);
  else
    tv_norm_kernel<__nv_bfloat16><<<grd, blk, 0, st>>>(
        (const __nv_bfloat16*)x, Nx, Ny, Nz, c, cmul, partials, counter, scale, norm);
  return cudaGetLastError();
}

cudaError_t launch_tv_norm(const void* x, int xt, int Nx, int Ny, int Nz,
                           float c, double* partials, unsigned* counter,
                           float* scale, double* norm, cudaStream_t st) {
  return tv_norm_go(x, xt, Nx, Ny, Nz, c, nullptr, partials, counter, scale, norm, st);
}

cudaError_t launch_tv_norm_scaled(const void* x, int xt, int Nx, int Ny, int Nz,
                                  float c, const double* cmul, double* partials,
                                  unsigned* counter, float* scale, double* norm,
                                  cudaStream_t st) {
  return tv_norm_go(x, xt, Nx, Ny, Nz, c, cmul, partials, counter, scale, norm, st);
}

cudaError_t launch_tv_update(const void* x, void* y, int xt, int Nx, int Ny,
                             int Nz, const float* scale, cudaStream_t st) {
  if (tv4_ok(x, y, xt, Nx, Ny, Nz)) {
    tv4_kernel<1><<<tv4_grid(Nx, Ny, Nz), dim3(kT4Bx, kT4By), 0, st>>>(
        (const float*)x, (float*)y, Nx, Ny, Nz, 0.f, nullptr, nullptr, nullptr, nullptr, nullptr,
        scale);
    return cudaGetLastError();
  }
  dim3 blk(kTvBx, kTvBy), grd = tv_grid(Nx, Ny, Nz);
  if (xt == kF32)
    tv_update_kernel<float><<<grd, blk, 0, st>>>((const float*)x, (float*)y,
                                                 Nx, Ny, Nz, scale);
  else if (xt == kF16)
    tv_update_kernel<__half><<<grd, blk, 0, st>>>((const __half*)x,
                                                  (__half*)y, Nx, Ny, Nz, scale);
  else
    tv_update_kernel<__nv_bfloat16><<<grd, blk, 0, st>>>(
        (const __nv_bfloat16*)x, (__nv_bfloat16*)y, Nx, Ny, Nz, scale);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// ||a - b||^2 in FP64 with NaN differences dropped and, optionally, a[0]
// taken as 0 (OSC_TV_recon.m:45,65-67: mu_old(1) = 0, mu_old(isnan) = 0).
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) ssd_kernel(
    const T* __restrict__ a, const T* __restrict__ b, long long n,
    int zero_first, double* partials, unsigned* counter, double* out) {
  double ss = 0.0;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += stride) {
    const float av = (zero_first && i == 0) ? 0.f : ldf(a + i);
    const float d = av - ldf(b + i);
    if (!isnan(d)) ss += (double)d * (double)d;
  }
  const double blk = block_sum(ss);
  double total;
  if (finish_partials(blk, partials, counter, &total)) *out = sqrt(total);
}

__global__ void __launch_bounds__(1024) sum_partials_kernel(const double* __restrict__ p,
                                                           long long n, double* __restrict__ out) {
  double acc = 0.0;
  for (long long i = threadIdx.x; i < n; i += blockDim.x) acc += p[i];
  acc = block_sum(acc);
  if (threadIdx.x == 0) *out = acc;
}

cudaError_t launch_sum_partials(const double* partials, long long n, double* out,
                                cudaStream_t st) {
  sum_partials_kernel<<<1, 1024, 0, st>>>(partials, n, out);
  return cudaGetLastError();
}

// Norms of the parts of a volume (z-slabs) combined in index order:
// out = sqrt(sum parts[i]^2); with scale non-null also the TV step scale
// -c * (*cmul) / out, as the last CTA of the norm kernel writes it.
__global__ void combine_norms_kernel(const double* __restrict__ parts, int n,
                                     double* __restrict__ out, float c,
                                     const double* __restrict__ cmul, float* __restrict__ scale) {
  double s = 0.0;
  for (int i = 0; i < n; ++i) s += parts[i] * parts[i];
  const double m = sqrt(s);
  *out = m;
  if (scale) {
    const double ce = cmul ? (double)c * *cmul : (double)c;
    *scale = (float)(-ce / m);
  }
}

cudaError_t launch_combine_norms(const double* parts, int n, double* out, float c,
                                 const double* cmul, float* scale, cudaStream_t st) {
  combine_norms_kernel<<<1, 1, 0, st>>>(parts, n, out, c, cmul, scale);
  return cudaGetLastError();
}

int device_sms() {
  static std::atomic<int> cache[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    cudaGetLastError();
    dev = 0;
  }
  int n = cache[dev].load(std::memory_order_relaxed);
  if (n > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) {
    cudaGetLastError();
    n = 1;
  }
  cache[dev].store(n, std::memory_order_relaxed);
  return n;
}

size_t ssd_partials_needed() { return (size_t)device_sms() * 4; }

cudaError_t launch_ssd(const void* a, const void* b, int dt, long long n,
                       int zero_first, double* partials, unsigned* counter,
                       double* out, cudaStream_t st) {
  const int blocks = (int)ssd_partials_needed();
  if (dt == kF32)
    ssd_kernel<float><<<blocks, 256, 0, st>>>((const float*)a, (const float*)b,
                                              n, zero_first, partials, counter, out);
  else if (dt == kF16)
    ssd_kernel<__half><<<blocks, 256, 0, st>>>((const __half*)a,
                                               (const __half*)b, n, zero_first,
                                               partials, counter, out);
  else
    ssd_kernel<__nv_bfloat16><<<blocks, 256, 0, st>>>(
        (const __nv_bfloat16*)a, (const __nv_bfloat16*)b, n, zero_first,
        partials, counter, out);
  return cudaGetLastError();
}

template <typename T>
__global__ void finite_kernel(T* x, long long n) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += stride) {
    const float v = ldp(x + i);
    if (!isfinite(v)) stf(x + i, 0.f);
  }
}

cudaError_t launch_finite(void* x, int dt, long long n, cudaStream_t st) {
  const int blocks = device_sms() * 8;
  if (dt == kF32) finite_kernel<float><<<blocks, 256, 0, st>>>((float*)x, n);
  else if (dt == kF16) finite_kernel<__half><<<blocks, 256, 0, st>>>((__half*)x, n);
  else finite_kernel<__nv_bfloat16><<<blocks, 256, 0, st>>>((__nv_bfloat16*)x, n);
  return cudaGetLastError();
}

template <typename T>
__global__ void fill_kernel(T* x, long long n, float v) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += stride)
    stf(x + i, v);
}

cudaError_t launch_fill(void* x, int dt, long long n, float v,
                        cudaStream_t st) {
  const int blocks = device_sms() * 8;
  if (dt == kF32) fill_kernel<float><<<blocks, 256, 0, st>>>((float*)x, n, v);
  else if (dt == kF16) fill_kernel<__half><<<blocks, 256, 0, st>>>((__half*)x, n, v);
  else fill_kernel<__nv_bfloat16><<<blocks, 256, 0, st>>>((__nv_bfloat16*)x, n, v);
  return cudaGetLastError();
}

// OSC_TV_recon.m:35-37: x(x < eps) = eps (NaN stays NaN, as in MATLAB).
__global__ void clamp_copy_kernel(const float* __restrict__ s, float* __restrict__ d,
                                  long long n, float eps) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const float v = s[i];
    d[i] = (v < eps) ? eps : v;
  }
}

cudaError_t launch_clamp_copy(const float* src, float* dst, long long n, float eps,
                              cudaStream_t st) {
  clamp_copy_kernel<<<device_sms() * 8, 256, 0, st>>>(src, dst, n, eps);
  return cudaGetLastError();
}

// Largest finite value of n FP32 values as an order-preserving integer key
// (atomicMax on the bits of a non-negative float orders like the float; a
// negative or NaN value counts as 0).  *out must start at 0.
__global__ void max_nonneg_kernel(const float* __restrict__ x, long long n,
                                  unsigned* __restrict__ out) {
  unsigned m = 0;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const float v = x[i];
    if (v > 0.f && v <= 3.4028235e38f) m = max(m, __float_as_uint(v));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

cudaError_t launch_max_nonneg(const float* x, long long n, unsigned* out, cudaStream_t st) {
  max_nonneg_kernel<<<device_sms() * 8, 256, 0, st>>>(x, n, out);
  return cudaGetLastError();
}

template <typename S, typename D>
__global__ void convert_kernel(const S* __restrict__ s, D* __restrict__ d,
                               long long n) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += stride)
    stf(d + i, ldp(s + i));
}

cudaError_t launch_convert(const void* src, int st_, void* dst, int dt,
                           long long n, cudaStream_t st) {
  const int blocks = device_sms() * 8;
#define CV(SA, DA) convert_kernel<SA, DA><<<blocks, 256, 0, st>>>((const SA*)src, (DA*)dst, n)
  if (st_ == kF32 && dt == kF16) CV(float, __half);
  else if (st_ == kF32 && dt == kBF16) CV(float, __nv_bfloat16);
  else if (st_ == kF16 && dt == kF32) CV(__half, float);
  else if (st_ == kBF16 && dt == kF32) CV(__nv_bfloat16, float);
  else if (st_ == kF32 && dt == kF32) CV(float, float);
  else return cudaErrorInvalidValue;
#undef CV
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// FDK/FBP pre-filter: per detector row, the cosine weight
// (preFilterSinogram.m:38-57, 1-based U/V as written), the Parker window of
// the row element (parker_weight.m:216-226, a host-built [nP, W] table), the
// zero-padded ramp x window filter as a direct linear convolution with the
// spatial kernel real(ifft(H)) (preFilterSinogram.m:72-78: padding to
// order >= 2W makes the circular convolution linear), and the dbeta/2 factor
// (:80-84).  Optional FBP_recon.m:26-28 log transform on load.
// ---------------------------------------------------------------------------
constexpr int kFiltRows = 4;

__global__ void __launch_bounds__(256) prefilter_kernel(
    const FiltArgs A, const float* __restrict__ sino,
    const float* __restrict__ pre, const float* __restrict__ parker,
    const float* __restrict__ dbeta, const float* __restrict__ kern,
    float* __restrict__ out) {
  extern __shared__ float sm[];
  float* ks = sm;                       // order
  float* xs = sm + A.order;             // kFiltRows * W
  const int view = blockIdx.y;
  const int v0 = blockIdx.x * kFiltRows;
  const int W = A.W, H = A.H;
  for (int i = threadIdx.x; i < A.order; i += blockDim.x) ks[i] = __ldg(kern + i);
  const size_t vbase = (size_t)view * W * H;
  const float db = __ldg(dbeta + view);
  for (int r = 0; r < kFiltRows; ++r) {
    const int v = v0 + r;
    for (int u = threadIdx.x; u < W; u += blockDim.x) {
      float w = 0.f;
      if (v < H) {
        const size_t gi = vbase + (size_t)v * W + u;
        float s = __ldg(sino + gi);
        if (A.log_input) {
          s = -logf(s / __ldg(pre + gi));
          if (!isfinite(s)) s = 0.f;
        }
        const float U = (float)(u + 1) - (float)(W - 1) * 0.5f;
        const float V = (float)(v + 1) - (float)(H - 1) * 0.5f;
        if (A.geom == 1) s *= A.sad / sqrtf(A.sad * A.sad + U * U);
        if (A.geom == 2) s *= A.sad / sqrtf(A.sad * A.sad + U * U + V * V);
        w = s * __ldg(parker + (size_t)view * W + u);
      }
      xs[r * W + u] = w;
    }
  }
  __syncthreads();
  const int mask = A.order - 1;
  for (int u = threadIdx.x; u < W; u += blockDim.x) {
    float acc[kFiltRows];
#pragma unroll
    for (int r = 0; r < kFiltRows; ++r) acc[r] = 0.f;
    for (int j = 0; j < W; ++j) {
      const float k = ks[(u - j) & mask];
#pragma unroll
      for (int r = 0; r < kFiltRows; ++r) acc[r] = fmaf(xs[r * W + j], k, acc[r]);
    }
#pragma unroll
    for (int r = 0; r < kFiltRows; ++r) {
      const int v = v0 + r;
      if (v < H) out[vbase + (size_t)v * W + u] = acc[r] * db;
    }
  }
}

// Weighted input sample of the pre-filter (log transform, cosine weight,
// Parker weight), as prefilter_kernel stages it.
__device__ __forceinline__ float prefilter_input(const FiltArgs& A, const float* __restrict__ sino,
                                                 const float* __restrict__ pre,
                                                 const float* __restrict__ parker, int view,
                                                 int v, int u) {
  const size_t gi = ((size_t)view * A.H + v) * A.W + u;
  float s = __ldg(sino + gi);
  if (A.log_input) {
    s = -logf(s / __ldg(pre + gi));
    if (!isfinite(s)) s = 0.f;
  }
  const float U = (float)(u + 1) - (float)(A.W - 1) * 0.5f;
  const float V = (float)(v + 1) - (float)(A.H - 1) * 0.5f;
  if (A.geom == 1) s *= A.sad / sqrtf(A.sad * A.sad + U * U);
  if (A.geom == 2) s *= A.sad / sqrtf(A.sad * A.sad + U * U + V * V);
  return s * __ldg(parker + (size_t)view * A.W + u);
}

// Register-blocked form of prefilter_kernel: a block filters 8*RG detector
// rows of one view, each thread 8 rows x 8 consecutive columns.  The rows are
// staged in shared memory (zero-padded to a multiple of 8 columns); the
// thread keeps the 15 kernel taps k[(u0 - j0 - 7 + m) & mask] its 8 columns
// need for 8 consecutive j in registers, so 64 FMAs take 8 row loads
// (broadcasts) and 15/8 tap loads.  Each output is the same FMA chain over
// j = 0 .. W-1 as in prefilter_kernel: the results are bit-identical.
template <int RG>
__global__ void __launch_bounds__(256) prefilter_tiled_kernel(
    const FiltArgs A, const float* __restrict__ sino, const float* __restrict__ pre,
    const float* __restrict__ parker, const float* __restrict__ dbeta,
    const float* __restrict__ kern, float* __restrict__ out) {
  constexpr int ROWS = 8 * RG, UG = 256 / RG;  // rows per block, column groups
  extern __shared__ float sm[];
  const int W = A.W, H = A.H, Wj = (W + 7) & ~7;
  float* ks = sm;            // order (circular kernel)
  float* xs = sm + A.order;  // ROWS x Wj, row-major
  const int view = blockIdx.y;
  const int v0 = blockIdx.x * ROWS;
  for (int i = threadIdx.x; i < A.order; i += 256) ks[i] = __ldg(kern + i);
  for (int i = threadIdx.x; i < ROWS * Wj; i += 256) {
    const int r = i / Wj, j = i - r * Wj, v = v0 + r;
    xs[i] = (v < H && j < W) ? prefilter_input(A, sino, pre, parker, view, v, j) : 0.f;
  }
  __syncthreads();
  const int mask = A.order - 1;
  const int ug = threadIdx.x % UG, rg = threadIdx.x / UG;
  const float* xr = xs + (size_t)rg * 8 * Wj;
  const float db = __ldg(dbeta + view);
  for (int u0 = 8 * ug; u0 < W; u0 += 8 * UG) {
    float acc[8][8];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[r][i] = 0.f;
    for (int j0 = 0; j0 < Wj; j0 += 8) {
      float kw[15];
#pragma unroll
      for (int m = 0; m < 15; ++m) kw[m] = ks[(u0 - j0 - 7 + m) & mask];
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) {
        float x[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) x[r] = xr[r * Wj + j0 + jj];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float k = kw[i - jj + 7];  // k[(u0 + i - j) & mask]
#pragma unroll
          for (int r = 0; r < 8; ++r) acc[r][i] = fmaf(x[r], k, acc[r][i]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int v = v0 + rg * 8 + r;
      if (v >= H) continue;
      float* o = out + ((size_t)view * H + v) * W;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (u0 + i < W) o[u0 + i] = acc[r][i] * db;
    }
  }
}

// ---------------------------------------------------------------------------
// FFT form of the pre-filter (order 64 .. 4096, i.e. W <= 2048).  The ramp
// kernel is as long as the row, so the direct form costs 2 W flops per output
// (58 GFLOP at 384^2 x 512 views, 2.47 ms); one transform pair costs ~60
// whatever W is.  Two detector rows travel as the real and imaginary part of
// one complex row: the filter's spectrum is real and even, so it acts on both
// at once.  A thread keeps 16 complex elements in registers; N / 16 threads
// share a transform of N = R1 R2 R3 points, done in place with decimation in
// frequency forward and the mirrored decimation in time back, so the spectrum
// stays in digit-reversed order (the host lays the filter out in that order)
// and the last forward and the first inverse pass meet in registers: 4 trips
// through shared memory for 3 radices.  The zero half of the padded row
// (W <= N / 2) is never loaded, and only the first half is transformed back.
// Rows move through memory once: 8 bytes per pixel.  384^2 x 512 views, cone,
// Hamming: 2.47 -> 0.50 ms (1.2 TB/s: issue slots 70 % and the shared / L1 data
// path 61 %, not the memory, bound it); 3 CTAs of 80 registers per SM.  With so
// few warps the order of the loads counts: tables laid out so that a warp reads
// neighbours took it from 0.70 to 0.63 ms (the spectrum, 64 bytes apart, had
// cost as many L1 wavefronts as all exchanges), a row's loads all before its
// arithmetic and table loads before the barriers to 0.49.
//
// The filter all but removes a smooth row, so a transform's rounding (relative
// to the row) would stand out against the output: 2.2e-6 of it at 384 columns,
// Hamming, against 1.8e-6 for the direct sum.  So the row's differences x[u] -
// x[u-1] are transformed and the spectrum is divided by 1 - exp(-i w): what is
// transformed is as small as the output.  The sum of a row, which differences
// lose, is taken beside them and is the transform's element 0.
//
// The twiddle products mix the two rows of a pair, so rounding is relative to
// the larger one: each row is scaled by the power of two that brings its largest
// magnitude into [1, 2) and back at the store (exact, so a pair of like rows
// gives the bits that it gives unscaled; without it a row beside one 1e4 times
// larger was off by 4e-4; 12 us of 499 at 384^2 x 512).  A row of zeros stores
// zeros.
//
// A row with a value that is not finite or above 1e30 would reach its partner
// (and could overflow in a sum the direct form does not take): such rows enter
// the transform as zeros and are convolved directly afterwards.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 c_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 c_sub(float2 a, float2 b) { return tv_sub2(a, b); }
__device__ __forceinline__ float2 c_mul(float2 a, float2 w) {
  return make_float2(fmaf(a.x, w.x, -(a.y * w.y)), fmaf(a.x, w.y, a.y * w.x));
}
template <bool INV>
__device__ __forceinline__ float2 c_rot(float2 a) {  // times -i (forward), i (inverse)
  return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}
template <bool INV>
__device__ __forceinline__ float2 c_conj_if(float2 w) {
  return INV ? make_float2(w.x, -w.y) : w;
}

template <bool INV>
__device__ __forceinline__ void dft4(float2& a, float2& b, float2& c, float2& d) {
  const float2 t0 = c_add(a, c), t1 = c_sub(a, c), t2 = c_add(b, d), t3 = c_rot<INV>(c_sub(b, d));
  a = c_add(t0, t2);
  b = c_add(t1, t3);
  c = c_sub(t0, t2);
  d = c_sub(t1, t3);
}

// R-point transform of v[0 .. R-1], natural order in and out.
template <int R, bool INV>
__device__ __forceinline__ void dft(float2* v) {
  if constexpr (R == 4) {
    dft4<INV>(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 8) {
    constexpr float h = 0.70710678118654752f;
    float2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    dft4<INV>(e[0], e[1], e[2], e[3]);
    dft4<INV>(o[0], o[1], o[2], o[3]);
    o[1] = c_mul(o[1], c_conj_if<INV>(make_float2(h, -h)));
    o[2] = c_rot<INV>(o[2]);
    o[3] = c_mul(o[3], c_conj_if<INV>(make_float2(-h, -h)));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = c_add(e[k], o[k]);
      v[k + 4] = c_sub(e[k], o[k]);
    }
  } else {
    static_assert(R == 16, "radix 4, 8 or 16");
    // cos / sin of pi/8
    constexpr float c1 = 0.92387953251128676f, s1 = 0.38268343236508977f, h = 0.70710678118654752f;
    float2 y[4][4];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
#pragma unroll
      for (int a = 0; a < 4; ++a) y[b][a] = v[4 * a + b];
      dft4<INV>(y[b][0], y[b][1], y[b][2], y[b][3]);
    }
    // twiddles exp(-2 pi i b k / 16)
    y[1][1] = c_mul(y[1][1], c_conj_if<INV>(make_float2(c1, -s1)));
    y[1][2] = c_mul(y[1][2], c_conj_if<INV>(make_float2(h, -h)));
    y[1][3] = c_mul(y[1][3], c_conj_if<INV>(make_float2(s1, -c1)));
    y[2][1] = c_mul(y[2][1], c_conj_if<INV>(make_float2(h, -h)));
    y[2][2] = c_rot<INV>(y[2][2]);
    y[2][3] = c_mul(y[2][3], c_conj_if<INV>(make_float2(-h, -h)));
    y[3][1] = c_mul(y[3][1], c_conj_if<INV>(make_float2(s1, -c1)));
    y[3][2] = c_mul(y[3][2], c_conj_if<INV>(make_float2(-h, -h)));
    y[3][3] = c_mul(y[3][3], c_conj_if<INV>(make_float2(-c1, s1)));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      dft4<INV>(y[0][k], y[1][k], y[2][k], y[3][k]);
#pragma unroll
      for (int q = 0; q < 4; ++q) v[k + 4 * q] = y[q][k];
    }
  }
}

// v[k] *= w^k for k < R: the powers 1, 2, 4, 8 of w from the table, rows of
// `pitch` elements so that a warp reads neighbours, the others as products of
// those (loading every power took 745 us where this took 625 at 384^2 x 512).
template <int R>
__device__ __forceinline__ void twiddle_load(float2* w, const float2* __restrict__ tw, int pitch) {
#pragma unroll
  for (int k = 0; k < (R > 8 ? 4 : R > 4 ? 3 : 2); ++k) w[k] = __ldg(tw + k * pitch);
}
template <int R, bool INV>
__device__ __forceinline__ void twiddle(float2* v, const float2* w) {
  float2 p[R];
  p[1] = c_conj_if<INV>(w[0]);
  p[2] = c_conj_if<INV>(w[1]);
  if constexpr (R > 4) p[4] = c_conj_if<INV>(w[2]);
  if constexpr (R > 8) p[8] = c_conj_if<INV>(w[3]);
#pragma unroll
  for (int k = 1; k < R; ++k) {
    if (k > 8) p[k] = c_mul(p[8], p[k - 8]);
    else if (k > 4 && k < 8) p[k] = c_mul(p[4], p[k - 4]);
    else if (k == 3) p[k] = c_mul(p[2], p[1]);
    v[k] = c_mul(v[k], p[k]);
  }
}

// One spare element per 8 keeps the stride-R passes off each other's banks.
__device__ __forceinline__ int fft_slot(int i) { return i + (i >> 3); }

// Weighted input sample as prefilter_input, the cosine weight by a reciprocal
// square root with one Newton step.
__device__ __forceinline__ float prefilter_fast_input(const FiltArgs& A, float s, float pre, int v,
                                                      int u, float pk) {
  if (A.log_input) {
    s = -logf(s / pre);
    if (!isfinite(s)) s = 0.f;
  }
  if (A.geom != 0) {
    const float U = (float)(u + 1) - (float)(A.W - 1) * 0.5f;
    const float V = (float)(v + 1) - (float)(A.H - 1) * 0.5f;
    const float q = A.geom == 2 ? A.sad * A.sad + U * U + V * V : A.sad * A.sad + U * U;
    const float r = rsqrtf(q);
    s *= A.sad * (r * fmaf(-0.5f * q * r, r, 1.5f));
  }
  return s * pk;
}

// 2^-e and 2^e of a row's largest magnitude m = 2^e (1 .. 2), e >= -126; for a
// row of zeros 2^e is 0.
// Magnitudes as their bits, which integers order alike (a NaN, whose row is kept out
// of the transform, above all others).
__device__ __forceinline__ unsigned magnitude(float x) { return __float_as_uint(x) & 0x7fffffffu; }
__device__ __forceinline__ unsigned row_exp(unsigned m) { return min(max(m >> 23, 1u), 253u); }
__device__ __forceinline__ float row_scale(unsigned m) {
  return __uint_as_float((254u - row_exp(m)) << 23);
}
__device__ __forceinline__ float row_unscale(unsigned m) {
  return m ? __uint_as_float(row_exp(m) << 23) : 0.f;
}

constexpr int kFftThreads = 256, kFftElems = 16 * kFftThreads;  // complex elements per CTA

template <int R1, int R2, int R3>
__global__ void __launch_bounds__(kFftThreads, 3) prefilter_fft_kernel(
    const FiltArgs A, const float* __restrict__ sino, const float* __restrict__ pre,
    const float* __restrict__ parker, const float* __restrict__ dbeta,
    const float* __restrict__ kern, float* __restrict__ out, long long pairs) {
  constexpr int N = R1 * R2 * R3, TF = N / 16, NF = kFftThreads / TF;
  static_assert(R1 == 16 && kFftThreads % TF == 0, "16 elements per thread");
  __shared__ float2 sm[kFftElems + kFftElems / 8];
  __shared__ int bad[2 * NF];  // rows kept out of the transform
  constexpr int TW = TF < 32 ? TF : 32, NWF = TF / TW;  // lanes and warps per transform
  __shared__ float2 psum[NF * NWF], edge[8 * NF * NWF];
  __shared__ uint2 pmax[NF * NWF];
  // after the spatial kernel: the differences' spectrum and the twiddles
  const float2* spec = reinterpret_cast<const float2*>(kern + N);
  const float2 *tw1 = spec + N, *tw2 = tw1 + 4 * TF;
  const int n = threadIdx.x % TF, q = threadIdx.x / TF;
  float2* x = sm + q * (N + N / 8);
  const int W = A.W, H = A.H, hp = (H + 1) >> 1;
  const long long pair = (long long)blockIdx.x * NF + q;
  const bool live = pair < pairs;
  int view = 0, v0 = 0;
  if (live) {
    view = pairs <= 0x7fffffffLL ? (int)((unsigned)pair / (unsigned)hp) : (int)(pair / hp);
    v0 = 2 * (int)(pair - (long long)view * hp);
  }
  const bool two = v0 + 1 < H;
  const size_t row0 = ((size_t)view * H + v0) * W;
  if (threadIdx.x < 2 * NF) bad[threadIdx.x] = 0;
  __syncthreads();
  float2 e[16];
  bool b0 = false, b1 = false;
  {
    // all loads first, the lower row's twice where the upper is missing
    float2 raw[8], r0[8];
    float pk[8];
    const size_t up = two ? W : 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int u = n + j * TF;
      raw[j] = r0[j] = make_float2(0.f, 0.f);
      pk[j] = 0.f;
      if (live && u < W) {
        raw[j] = make_float2(__ldg(sino + row0 + u), __ldg(sino + row0 + up + u));
        if (A.log_input) r0[j] = make_float2(__ldg(pre + row0 + u), __ldg(pre + row0 + up + u));
        pk[j] = __ldg(parker + (size_t)view * W + u);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int u = n + j * TF;
      float2 s = make_float2(0.f, 0.f);
      if (live && u < W) {
        s.x = prefilter_fast_input(A, raw[j].x, r0[j].x, v0, u, pk[j]);
        if (two) s.y = prefilter_fast_input(A, raw[j].y, r0[j].y, v0 + 1, u, pk[j]);
      }
      b0 |= !(fabsf(s.x) <= 1.0e30f);
      b1 |= !(fabsf(s.y) <= 1.0e30f);
      e[j] = s;
      e[j + 8] = make_float2(0.f, 0.f);
    }
    if (b0) bad[2 * q] = 1;
    if (b1) bad[2 * q + 1] = 1;
  }
  // row sums and largest magnitudes, and each element's left neighbour: lane n -
  // 1, whose warp leaves its last lane's elements in edge
  const int wq = q * NWF + n / TW;
  float2 sum = make_float2(0.f, 0.f), left[8];
  uint2 big = make_uint2(0u, 0u);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    sum = c_add(sum, e[j]);
    big = make_uint2(max(big.x, magnitude(e[j].x)), max(big.y, magnitude(e[j].y)));
  }
  const unsigned lanes = TW == 32 ? 0xffffffffu : ((1u << (TW & 31)) - 1u) << (threadIdx.x & 31 & ~(TW - 1));
  big = make_uint2(__reduce_max_sync(lanes, big.x), __reduce_max_sync(lanes, big.y));
#pragma unroll
  for (int o = TW / 2; o > 0; o >>= 1) {
    sum.x += __shfl_xor_sync(0xffffffffu, sum.x, o);
    sum.y += __shfl_xor_sync(0xffffffffu, sum.y, o);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    left[j].x = __shfl_up_sync(0xffffffffu, e[j].x, 1, TW);
    left[j].y = __shfl_up_sync(0xffffffffu, e[j].y, 1, TW);
  }
  if (n % TW == 0) {
    psum[wq] = sum;
    pmax[wq] = big;
  }
  if (n % TW == TW - 1) {
#pragma unroll
    for (int j = 0; j < 8; ++j) edge[8 * wq + j] = e[j];
  }
  const bool any = __syncthreads_or(b0 || b1) != 0;
  const bool bad0 = bad[2 * q] != 0, bad1 = bad[2 * q + 1] != 0;
  // 2^-e of both rows, or 2^e (back); read again at the store instead of kept
  auto scales = [&](bool back) {
    uint2 m = pmax[q * NWF];
#pragma unroll
    for (int w = 1; w < NWF; ++w) {
      const uint2 b = pmax[q * NWF + w];
      m = make_uint2(max(m.x, b.x), max(m.y, b.y));
    }
    return back ? make_float2(row_unscale(m.x), row_unscale(m.y))
                : make_float2(row_scale(m.x), row_scale(m.y));
  };
  const float2 scale = scales(false);
  float2 past = make_float2(0.f, 0.f);  // element N / 2 of the differences (thread 0)
  if (n % TW == 0) {
    const float2* ed = edge + 8 * (n == 0 ? q * NWF + NWF - 1 : wq - 1);
#pragma unroll
    for (int j = 0; j < 8; ++j)
      left[j] = n ? ed[j] : (j ? ed[j - 1] : make_float2(0.f, 0.f));
    if (n == 0) past = make_float2(-ed[7].x, -ed[7].y);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) e[j] = __fmul2_rn(c_sub(e[j], left[j]), scale);
  e[8] = __fmul2_rn(past, scale);
  if (any) {
#pragma unroll
    for (int j = 0; j <= 8; ++j) {
      if (bad0) e[j].x = 0.f;
      if (bad1) e[j].y = 0.f;
    }
  }
  // radix R1, stride TF
  float2 w1[4], w2[4];
  twiddle_load<R1>(w1, tw1 + n, TF);
  dft<R1, false>(e);
  twiddle<R1, false>(e, w1);
#pragma unroll
  for (int j = 0; j < 16; ++j) x[fft_slot(n + j * TF)] = e[j];
  // table loads go out before the barriers they would wait behind
  const int t = n % R3;  // (n + i TF) % R3
  if constexpr (R3 > 1) twiddle_load<R2>(w2, tw2 + t, R3);
  __syncthreads();
  if constexpr (R3 > 1) {  // radix R2, stride R3
#pragma unroll
    for (int i = 0; i < 16 / R2; ++i) {
      const int base = ((n + i * TF) / R3) * (R2 * R3) + t;
#pragma unroll
      for (int j = 0; j < R2; ++j) e[j] = x[fft_slot(base + j * R3)];
      dft<R2, false>(e);
      twiddle<R2, false>(e, w2);
#pragma unroll
      for (int j = 0; j < R2; ++j) x[fft_slot(base + j * R3)] = e[j];
    }
  }
  {  // last radix, filter, first inverse radix
    constexpr int RL = R3 > 1 ? R3 : R2;
    float2 sp[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) sp[i] = __ldg(spec + i % RL * (N / RL) + n + i / RL * TF);
    if constexpr (R3 > 1) __syncthreads();
#pragma unroll
    for (int i = 0; i < 16 / RL; ++i) {
      const int base = (n + i * TF) * RL;
#pragma unroll
      for (int j = 0; j < RL; ++j) e[j] = x[fft_slot(base + j)];
      dft<RL, false>(e);
      if (base == 0) {  // frequency 0: the row sums (element 0 of the spectrum is real)
        e[0] = psum[q * NWF];
#pragma unroll
        for (int w = 1; w < NWF; ++w) e[0] = c_add(e[0], psum[q * NWF + w]);
        e[0] = __fmul2_rn(e[0], scales(false));
        if (bad0) e[0].x = 0.f;
        if (bad1) e[0].y = 0.f;
      }
#pragma unroll
      for (int j = 0; j < RL; ++j) e[j] = c_mul(e[j], sp[i * RL + j]);
      dft<RL, true>(e);
#pragma unroll
      for (int j = 0; j < RL; ++j) x[fft_slot(base + j)] = e[j];
    }
    if constexpr (R3 > 1) twiddle_load<R2>(w2, tw2 + t, R3);
    else twiddle_load<R1>(w1, tw1 + n, TF);
    __syncthreads();
  }
  if constexpr (R3 > 1) {
#pragma unroll
    for (int i = 0; i < 16 / R2; ++i) {
      const int base = ((n + i * TF) / R3) * (R2 * R3) + t;
#pragma unroll
      for (int j = 0; j < R2; ++j) e[j] = x[fft_slot(base + j * R3)];
      twiddle<R2, true>(e, w2);
      dft<R2, true>(e);
#pragma unroll
      for (int j = 0; j < R2; ++j) x[fft_slot(base + j * R3)] = e[j];
    }
    twiddle_load<R1>(w1, tw1 + n, TF);
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < 16; ++j) e[j] = x[fft_slot(n + j * TF)];
  twiddle<R1, true>(e, w1);
  dft<R1, true>(e);
  const float db = live ? __ldg(dbeta + view) : 0.f;
  // one factor: where it underflows, so does what it scales
  float2 back = scales(true);
  back = make_float2(back.x * db, back.y * db);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int u = n + j * TF;
    if (live && u < W) {
      if (!bad0) out[row0 + u] = e[j].x * back.x;
      if (two && !bad1) out[row0 + W + u] = e[j].y * back.y;
    }
  }
  if (any) {  // rows kept out: the direct sum, from staged inputs (out may be sino)
    __syncthreads();
    for (int u = n; live && u < W; u += TF)
      x[u] = make_float2(bad0 ? prefilter_input(A, sino, pre, parker, view, v0, u) : 0.f,
                         bad1 ? prefilter_input(A, sino, pre, parker, view, v0 + 1, u) : 0.f);
    __syncthreads();
    for (int u = n; live && (bad0 || bad1) && u < W; u += TF) {
      float2 acc = make_float2(0.f, 0.f);
      for (int j = 0; j < W; ++j) {
        const float k = __ldg(kern + ((u - j) & (N - 1)));
        acc = make_float2(fmaf(x[j].x, k, acc.x), fmaf(x[j].y, k, acc.y));
      }
      if (bad0) out[row0 + u] = acc.x * db;
      if (bad1) out[row0 + W + u] = acc.y * db;
    }
  }
}

template <int R1, int R2, int R3>
static cudaError_t prefilter_fft_go(const FiltArgs& a, const float* sino, const float* pre,
                                    const float* parker, const float* dbeta, const float* kern,
                                    float* out, cudaStream_t st) {
  constexpr int NF = kFftElems / (R1 * R2 * R3);
  const long long pairs = (long long)a.nP * ((a.H + 1) / 2), ctas = (pairs + NF - 1) / NF;
  if (ctas > 0x7fffffffLL) return cudaErrorInvalidValue;
  prefilter_fft_kernel<R1, R2, R3><<<(unsigned)ctas, kFftThreads, 0, st>>>(
      a, sino, pre, parker, dbeta, kern, out, pairs);
  return cudaGetLastError();
}

// Radices of the transform of `order` points: r[0] * r[1] * r[2]; false where
// the direct form serves (W > 2048).
bool prefilter_fft_radices(int order, int r[3]) {
  static const int tab[7][3] = {{16, 4, 1},  {16, 8, 1},  {16, 16, 1}, {16, 8, 4},
                                {16, 8, 8},  {16, 16, 8}, {16, 16, 16}};
  for (const auto& t : tab)
    if (t[0] * t[1] * t[2] == order) {
      for (int i = 0; i < 3; ++i) r[i] = t[i];
      return true;
    }
  return false;
}

template <int RG>
static cudaError_t prefilter_tiled_go(const FiltArgs& a, size_t smem, const float* sino,
                                      const float* pre, const float* parker, const float* dbeta,
                                      const float* kern, float* out, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(prefilter_tiled_kernel<RG>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  dim3 grd((a.H + 8 * RG - 1) / (8 * RG), a.nP);
  prefilter_tiled_kernel<RG><<<grd, 256, smem, st>>>(a, sino, pre, parker, dbeta, kern, out);
  return cudaGetLastError();
}

cudaError_t launch_prefilter(const FiltArgs& a, const float* sino,
                             const float* pre, const float* parker,
                             const float* dbeta, const float* kern, bool fft, float* out,
                             cudaStream_t st) {
  if (fft) {
#define FFT(R1, R2, R3)          \
  if (a.order == R1 * R2 * R3)   \
  return prefilter_fft_go<R1, R2, R3>(a, sino, pre, parker, dbeta, kern, out, st)
    FFT(16, 4, 1);
    FFT(16, 8, 1);
    FFT(16, 16, 1);
    FFT(16, 8, 4);
    FFT(16, 8, 8);
    FFT(16, 16, 8);
    FFT(16, 16, 16);
#undef FFT
    return cudaErrorInvalidValue;
  }
  // rows too long for the transform (W > 2048): the register-blocked direct
  // form with the most rows per block whose rows and kernel fit 200 KB of
  // shared memory
  const size_t Wj = (size_t)((a.W + 7) & ~7);
  for (int rg : {2, 1}) {
    const size_t smem = sizeof(float) * ((size_t)a.order + (size_t)8 * rg * Wj);
    if (smem > 200 * 1024) continue;
    if (rg == 2) return prefilter_tiled_go<2>(a, smem, sino, pre, parker, dbeta, kern, out, st);
    return prefilter_tiled_go<1>(a, smem, sino, pre, parker, dbeta, kern, out, st);
  }
  dim3 grd((a.H + kFiltRows - 1) / kFiltRows, a.nP);
  const size_t smem = sizeof(float) * ((size_t)a.order + (size_t)kFiltRows * a.W);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(
        prefilter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  prefilter_kernel<<<grd, 256, smem, st>>>(a, sino, pre, parker, dbeta, kern, out);
  return cudaGetLastError();
}

}  // namespace mexct
