// FourierSlice: the central-slice operator pair on ONELINE's geometry.
//
// SPIDER's BP 3F inserts each image's spectrum into the 3D Fourier grid as a
// central slice with Kaiser-Bessel weights (ONELINE, oneline.f:38-200) and has
// no extraction with the same kernel.  This file adds the pair a
// differentiable reconstruction needs (no counterpart in the reference):
//
//   E   (forward, extraction):  grid X -> slices T, the exact real-linear
//       adjoint of the insertion below;
//   E^T (adjoint, insertion):   slices T -> grid X, ONELINE's X += BTQ * W
//       with the weight grid dropped;
//   E^T E + lam I (normal):     E into a slice buffer and E^T of it, or,
//       without a buffer, one pass that gathers each pixel's taps and
//       scatters the sum back over the same taps.
//
// Grid: complex float2 [2nx][2nx][nx+1] (i fastest, Fortran X(0:NX,N,N)).
// Slices: float2 [nslice][2nx][nx+1] in the layout and sign of the staged
// spectra the back-projection inserts (cuFFT R2C of the padded, shifted
// image; ONELINE's BI is its conjugate).  Every tap (voxel, table weight,
// Hermitian flip for x < 0, reflected point, oneline.f:118-150) is that of the
// back-projection's insertion.  E is fs_extract.cuh, E^T the column insertion of
// slab.cuh; E^T of few slices and the normal operators without a buffer take four
// lanes per pixel over the nonzero window of the table.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../include/spider_b200.h"
#include "ctx.h"
#include "fs_extract.cuh"
#include "slab.cuh"

namespace spi {

__device__ __forceinline__ int fs_nint_pos(float v) {  // Fortran NINT, v >= 0
  const float f = floorf(v);
  return (int)f + ((__fsub_rn(v, f) >= 0.5f) ? 1 : 0);
}
__device__ __forceinline__ float fs_tap(const float* tab, float v, int k, float fltb) {
  return tab[fs_nint_pos(__fmul_rn(fabsf(__fsub_rn(v, (float)k)), fltb))];
}

// The tap window of pixel (I, J) for lane q of its four-lane group (lanes
// gl..gl+3 share the pixel): x tap xs + q, the 4 x 4 (y, z) windows starting
// at ys, zs.  Called by all 32 lanes (the y/z weights are exchanged by
// shuffles).  `ok` is false when the pixel has no taps.
struct FsWin {
  bool ok, flipped;
  int xs, ys, zs;
  float tx;
  float ty[4], tz[4];
};

// LS: lanes per x tap (the y/z weight of window position l lives in lane gl + l * LS).
template <int LS = 1>
__device__ __forceinline__ void fs_window(const SliceDesc& sd, int I, int J, int nx, const float* tab, float fltb,
                                          int q, int gl, FsWin& w) {
  const int N = 2 * nx, N2 = nx, LN2 = 2, NN4 = N * N / 4;
  const float fN = (float)N;
  bool ok = I <= N2 && (I * I + J * J) < NN4 && !(I == 0 && J < 0);
  const float fI = (float)I, fJ = (float)J;
  float xnew = __fadd_rn(__fmul_rn(fI, sd.dm[0]), __fmul_rn(fJ, sd.dm[3]));
  float ynew = __fadd_rn(__fmul_rn(fI, sd.dm[1]), __fmul_rn(fJ, sd.dm[4]));
  float znew = __fadd_rn(__fmul_rn(fI, sd.dm[2]), __fmul_rn(fJ, sd.dm[5]));
  w.flipped = xnew < 0.0f;
  if (w.flipped) {
    xnew = -xnew; ynew = -ynew; znew = -znew;
  }
  const int ixn = __float2int_rz(__fadd_rn(__fadd_rn(xnew, 0.5f), fN)) - N;
  const int iyn = __float2int_rz(__fadd_rn(__fadd_rn(ynew, 0.5f), fN)) - N;
  const int izn = __float2int_rz(__fadd_rn(__fadd_rn(znew, 0.5f), fN)) - N;
  ok = ok && ixn <= (N2 - LN2 - 1) && iyn >= (-N2 + 2 + LN2) && iyn <= (N2 - LN2 - 1) && izn >= (-N2 + 2 + LN2) &&
       izn <= (N2 - LN2 - 1);
  if (!ok) { xnew = ynew = znew = 0.0f; }   // keeps the lookups below in range; no taps follow
  const int ix0 = ok ? ixn : 0, iy0 = ok ? iyn : 0, iz0 = ok ? izn : 0;
  w.xs = fs_tap(tab, xnew, ix0 - 2, fltb) != 0.0f ? ix0 - 2 : ix0 - 1;
  w.ys = fs_tap(tab, ynew, iy0 - 2, fltb) != 0.0f ? iy0 - 2 : iy0 - 1;
  w.zs = fs_tap(tab, znew, iz0 - 2, fltb) != 0.0f ? iz0 - 2 : iz0 - 1;
  w.tx = fs_tap(tab, xnew, w.xs + q, fltb);
  const float tyq = fs_tap(tab, ynew, w.ys + q, fltb);
  const float tzq = fs_tap(tab, znew, w.zs + q, fltb);
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    w.ty[l] = __shfl_sync(0xffffffffu, tyq, gl + l * LS);
    w.tz[l] = __shfl_sync(0xffffffffu, tzq, gl + l * LS);
  }
  w.ok = ok && w.tx != 0.0f;
}

// Grid index of tap (q, ly, lz) of window w: main tap (ixp, iyp, izp), or
// for ixp < 0 the reflected point (-ixp, -iyp, -izp) (refl = true).
__device__ __forceinline__ size_t fs_voxel(const FsWin& w, int q, int ly, int lz, int nx, bool& refl) {
  const int N = 2 * nx;
  const int ixp = w.xs + q, iyp = w.ys + ly, izp = w.zs + lz;
  const bool r = ixp < 0;
  const int ixa = r ? -ixp : ixp;
  const int iya = r ? ((iyp > 0) ? N - iyp : -iyp) : ((iyp >= 0) ? iyp : N + iyp);
  const int iza = r ? ((izp > 0) ? N - izp : -izp) : ((izp >= 0) ? izp : N + izp);
  refl = r;
  return ((size_t)iza * N + iya) * (size_t)(nx + 1) + ixa;
}

__device__ __forceinline__ float2 fs_cmul(float2 v, float wg, bool conj_) {
  return make_float2(__fmul_rn(v.x, wg), conj_ ? -__fmul_rn(v.y, wg) : __fmul_rn(v.y, wg));
}

// Sum over the lane's 16 taps of wg * X (conj(X) at reflected points)
__device__ __forceinline__ float2 fs_gather(const float2* __restrict__ X, const FsWin& w, int q, int nx) {
  float2 acc = make_float2(0.0f, 0.0f);
  if (!w.ok) return acc;
#pragma unroll
  for (int lz = 0; lz < 4; ++lz) {
    if (w.tz[lz] == 0.0f) continue;
#pragma unroll
    for (int ly = 0; ly < 4; ++ly) {
      const float tyz = __fmul_rn(w.ty[ly], w.tz[lz]);
      if (tyz == 0.0f) continue;
      const float wg = __fmul_rn(w.tx, tyz);
      if (wg == 0.0f) continue;
      bool refl;
      const float2 v = __ldg(X + fs_voxel(w, q, ly, lz, nx, refl));
      const float2 t = fs_cmul(v, wg, refl);
      acc.x = __fadd_rn(acc.x, t.x);
      acc.y = __fadd_rn(acc.y, t.y);
    }
  }
  return acc;
}

// X[v] += wg * b over the lane's taps (conj(b) at reflected points)
__device__ __forceinline__ void fs_scatter(float2* __restrict__ X, const FsWin& w, int q, int nx, float2 b) {
  if (!w.ok) return;
#pragma unroll
  for (int lz = 0; lz < 4; ++lz) {
    if (w.tz[lz] == 0.0f) continue;
#pragma unroll
    for (int ly = 0; ly < 4; ++ly) {
      const float tyz = __fmul_rn(w.ty[ly], w.tz[lz]);
      if (tyz == 0.0f) continue;
      const float wg = __fmul_rn(w.tx, tyz);
      if (wg == 0.0f) continue;
      bool refl;
      const size_t v = fs_voxel(w, q, ly, lz, nx, refl);
      atomicAdd(X + v, fs_cmul(b, wg, refl));
    }
  }
}

// The same into an FP64 grid, the real (h = 0) or the imaginary part b of the value
__device__ __forceinline__ void fs_scatter_part(double* __restrict__ X, const FsWin& w, int q, int h, int nx, double b) {
  if (!w.ok) return;
#pragma unroll
  for (int lz = 0; lz < 4; ++lz) {
    if (w.tz[lz] == 0.0f) continue;
#pragma unroll
    for (int ly = 0; ly < 4; ++ly) {
      const float tyz = __fmul_rn(w.ty[ly], w.tz[lz]);
      if (tyz == 0.0f) continue;
      const float wg = __fmul_rn(w.tx, tyz);
      if (wg == 0.0f) continue;
      bool refl;
      const size_t v = fs_voxel(w, q, ly, lz, nx, refl);
      const double t = __dmul_rn(b, (double)wg);
      atomicAdd(X + 2 * v + h, h && refl ? -t : t);
    }
  }
}

// E^T tap by tap, for plans too small for the columns (fs_small): a warp takes
// one row J of one slice and adds every tap with a reduction of its own.  X += E^T
// of the slices.  FP32: eight pixels at a time, four lanes per pixel.  FP64: four
// pixels, eight lanes, so that one instruction adds both parts of four
// consecutive voxels (64 contiguous bytes): 256 slices at 16^3 66 us, 91 with four lanes.
template <bool D>
__global__ void __launch_bounds__(256) fs_taps_kernel(const float2* __restrict__ in, void* __restrict__ out,
                                                      const SliceDesc* __restrict__ slices, int nslices, int nx,
                                                      const float* __restrict__ kbtab, float fltb) {
  extern __shared__ float tab[];
  for (int i = threadIdx.x; i < 5000; i += blockDim.x) tab[i] = kbtab[i];
  __syncthreads();
  constexpr int kLanes = D ? 8 : 4;
  const int N = 2 * nx, NN4 = nx * nx;
  const int lane = threadIdx.x & 31;
  const int g = lane / kLanes, q = lane % kLanes / (kLanes / 4), h = lane & 1, gl = lane & ~(kLanes - 1);
  const long long nitems = (long long)nslices * N;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long item = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); item < nitems;
       item += warps) {
    const SliceDesc sd = slices[item / N];
    const int J = (int)(item % N) - nx + 1;
    const float2* row = in + ((size_t)sd.img * N + (J >= 0 ? J : N + J)) * (size_t)(nx + 1);
    for (int I0 = 0; I0 * I0 + J * J < NN4; I0 += 32 / kLanes) {   // warp-uniform
      FsWin w;
      fs_window<kLanes / 4>(sd, I0 + g, J, nx, tab, fltb, q, gl, w);
      // BTQ = BI = conj(T), or conj(BI) = T for a flipped pixel
      float2 b = make_float2(0.0f, 0.0f);
      if (w.ok) {
        const float2 t = row[I0 + g];
        b = make_float2(t.x, w.flipped ? t.y : -t.y);
      }
      if (D) fs_scatter_part(static_cast<double*>(out), w, q, h, nx, (double)(h ? b.y : b.x));
      else fs_scatter(static_cast<float2*>(out), w, q, nx, b);
    }
  }
}

__device__ __forceinline__ float2 group_sum4(float2 v) {   // sum over the four lanes of a pixel, in every lane
  v.x = __fadd_rn(v.x, __shfl_xor_sync(0xffffffffu, v.x, 1));
  v.y = __fadd_rn(v.y, __shfl_xor_sync(0xffffffffu, v.y, 1));
  v.x = __fadd_rn(v.x, __shfl_xor_sync(0xffffffffu, v.x, 2));
  v.y = __fadd_rn(v.y, __shfl_xor_sync(0xffffffffu, v.y, 2));
  return v;
}

// The normal operator E^T E without a slice buffer (P -> Q, Q pre-set to lam *
// P), for callers that give none: a warp takes one row J of one slice (rows
// handed out in slice-major order by a grid stride), eight pixels at a time,
// gathers each pixel's taps and scatters the sum back over them.
__global__ void __launch_bounds__(256) fs_normal_kernel(const float2* __restrict__ in, float2* __restrict__ out,
                                                        const SliceDesc* __restrict__ slices, int nslices, int nx,
                                                        const float* __restrict__ kbtab, float fltb) {
  extern __shared__ float tab[];
  for (int i = threadIdx.x; i < 5000; i += blockDim.x) tab[i] = kbtab[i];
  __syncthreads();
  const int N = 2 * nx, NN4 = nx * nx;
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, q = lane & 3, gl = lane & ~3;
  const long long nitems = (long long)nslices * N;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long item = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); item < nitems;
       item += warps) {
    const SliceDesc sd = slices[item / N];
    const int J = (int)(item % N) - nx + 1;
    for (int I0 = 0; I0 * I0 + J * J < NN4; I0 += 8) {   // warp-uniform
      FsWin w;
      fs_window(sd, I0 + g, J, nx, tab, fltb, q, gl, w);
      // extraction then insertion of the same pixel: the flips cancel
      const float2 sum = group_sum4(fs_gather(in, w, q, nx));
      fs_scatter(out, w, q, nx, sum);
    }
  }
}

// The normal operator in FP64: the same taps and FP32 table weights, with the
// grids, the pixel sums and the scatter (FP64 atomics) in double precision.
// Late CG iterations apply E^T E to directions whose image is much smaller
// than ||E^T E|| ||p||; FP32 sums would lose that many digits there.
// The lane's 16 voxel offsets come from four plane and
// four row terms computed once per pixel (32-bit: a grid has < 2^32 voxels up
// to nx = 512) and serve both the gather and the scatter (measured 2-3%
// faster than computing each tap's index twice, 48 instead of 57 registers).
__global__ void __launch_bounds__(256) fs_normal64_kernel(const double2* __restrict__ in, double2* __restrict__ out,
                                                          const SliceDesc* __restrict__ slices, int nslices, int nx,
                                                          const float* __restrict__ kbtab, float fltb) {
  extern __shared__ float tab[];
  for (int i = threadIdx.x; i < 5000; i += blockDim.x) tab[i] = kbtab[i];
  __syncthreads();
  const int N = 2 * nx;
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, q = lane & 3, gl = lane & ~3;
  const long long nitems = (long long)nslices * N;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long item = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); item < nitems;
       item += warps) {
    const SliceDesc sd = slices[item / N];
    const int J = (int)(item % N) - nx + 1;
    for (int I0 = 0; I0 * I0 + J * J < nx * nx; I0 += 8) {   // warp-uniform
      FsWin w;
      fs_window(sd, I0 + g, J, nx, tab, fltb, q, gl, w);
      double2 v;
      {
        const int ixp = w.xs + q;
        const bool refl = ixp < 0;
        const unsigned ixa = (unsigned)(refl ? -ixp : ixp);
        unsigned zoff[4], yoff[4];
#pragma unroll
        for (int l = 0; l < 4; ++l) {
          const int izp = w.zs + l, iyp = w.ys + l;
          const int iza = refl ? ((izp > 0) ? N - izp : -izp) : ((izp >= 0) ? izp : N + izp);
          const int iya = refl ? ((iyp > 0) ? N - iyp : -iyp) : ((iyp >= 0) ? iyp : N + iyp);
          zoff[l] = (unsigned)iza * (unsigned)N * (unsigned)(nx + 1);
          yoff[l] = (unsigned)iya * (unsigned)(nx + 1) + ixa;
        }
        v = make_double2(0.0, 0.0);
        if (w.ok) {
#pragma unroll
          for (int lz = 0; lz < 4; ++lz) {
            if (w.tz[lz] == 0.0f) continue;
#pragma unroll
            for (int ly = 0; ly < 4; ++ly) {
              const float tyz = __fmul_rn(w.ty[ly], w.tz[lz]);
              if (tyz == 0.0f) continue;
              const float wg = __fmul_rn(w.tx, tyz);
              if (wg == 0.0f) continue;
              const double2 x = in[zoff[lz] + yoff[ly]];
              const double d = (double)wg;
              v.x = __dadd_rn(v.x, __dmul_rn(x.x, d));
              v.y = refl ? __dsub_rn(v.y, __dmul_rn(x.y, d)) : __dadd_rn(v.y, __dmul_rn(x.y, d));
            }
          }
        }
        v.x = __dadd_rn(v.x, __shfl_xor_sync(0xffffffffu, v.x, 1));
        v.y = __dadd_rn(v.y, __shfl_xor_sync(0xffffffffu, v.y, 1));
        v.x = __dadd_rn(v.x, __shfl_xor_sync(0xffffffffu, v.x, 2));
        v.y = __dadd_rn(v.y, __shfl_xor_sync(0xffffffffu, v.y, 2));
        if (!w.ok) continue;
#pragma unroll
        for (int lz = 0; lz < 4; ++lz) {
          if (w.tz[lz] == 0.0f) continue;
#pragma unroll
          for (int ly = 0; ly < 4; ++ly) {
            const float tyz = __fmul_rn(w.ty[ly], w.tz[lz]);
            if (tyz == 0.0f) continue;
            const float wg = __fmul_rn(w.tx, tyz);
            if (wg == 0.0f) continue;
            double* o = reinterpret_cast<double*>(out + (zoff[lz] + yoff[ly]));
            const double d = (double)wg;
            atomicAdd(o, __dmul_rn(v.x, d));
            atomicAdd(o + 1, refl ? -__dmul_rn(v.y, d) : __dmul_rn(v.y, d));
          }
        }
      }
    }
  }
}

// E^T: the column insertion into complex grids (slab.cuh).  us per slice, with
// per-tap reductions -> now: FP32 128^3 2.96 -> 2.03, 256^3 12.1 -> 7.75; FP64
// 7.26 -> 3.33 and 29.4 -> 12.6.  The FP64 normal operator (E and E^T through
// the buffer): 9.50 -> 6.40 and 43.8 -> 27.0; FP32 6.56 -> 4.2 and 34.6 -> 17.3.
template <class F>
__global__ void __launch_bounds__(kSlabThreads + 32, F::D ? kSlabBlocks64 : kSlabBlocks)
    fs_insert_kernel(const __grid_constant__ SlabArgs P, unsigned long long* __restrict__ work) {
  slab_main<F>(P, work);
}

__global__ void fs_scale64_kernel(const double2* __restrict__ p, double lam, double2* __restrict__ q, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const double2 v = p[i];
    q[i] = make_double2(__dmul_rn(lam, v.x), __dmul_rn(lam, v.y));
  }
}

__global__ void fs_scale_kernel(const float2* __restrict__ p, float lam, float2* __restrict__ q, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float2 v = p[i];
    q[i] = make_float2(__fmul_rn(lam, v.x), __fmul_rn(lam, v.y));
  }
}

// Volume of a grid of spectrum coefficients.  The grid models the volume's
// spectrum as V(k) = sum_v X_v K(k - v) (E samples exactly that), so the
// volume is the inverse transform of X times the transform of the separable
// Kaiser-Bessel kernel, |WKB| of WINDKB2A (bp32f.f:964-1005), where the
// direct gridding of BP 3F divides by it.  Plane i = 0 holds each voxel and
// its Friedel mate; its Hermitian part (X(0,j,k) + conj X(0,-j,-k)) / 2 is
// used.  Then the phase (-1)^(i+j+k), SPIDER's inverse sign (conjugate) and a
// C2R transform; the centred nx^3 is cropped, scaled by 1/n^3 and multiplied
// by |WKB(LR)| inside radius nx/2 and set to zero outside.
__global__ void fs_vol_prep_kernel(const float2* __restrict__ X, float2* __restrict__ out, int nx) {
  const int N = 2 * nx;
  const size_t h = (size_t)(nx + 1);
  const size_t nvox = h * N * N;
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < nvox; q += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(q % h);
    const size_t t = q / h;
    const int j = (int)(t % N), k = (int)(t / N);
    float2 v = X[q];
    if (i == 0) {
      const int jm = (N - j) % N, km = (N - k) % N;
      const float2 m = X[((size_t)km * N + jm) * h];
      v = make_float2(__fmul_rn(0.5f, __fadd_rn(v.x, m.x)), __fmul_rn(0.5f, __fsub_rn(v.y, m.y)));
    }
    const float s = ((i + j + k) & 1) ? -1.0f : 1.0f;
    float2 r = make_float2(s * v.x, -(s * v.y));
    if (q == 0) r.y = 0.0f;
    out[q] = r;
  }
}

__global__ void fs_vol_out_kernel(const float* __restrict__ R, int nx, int ip, float pix, const float* __restrict__ wkb,
                                  float* __restrict__ vol) {
  const int N = 2 * nx, c = nx / 2 + 1;
  const int l2 = (nx / 2) * (nx / 2);
  const size_t total = (size_t)nx * nx * nx;
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < total; q += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(q % nx);
    const size_t t = q / nx;
    const int j = (int)(t % nx), k = (int)(t / nx);
    const int lr = (k + 1 - c) * (k + 1 - c) + (j + 1 - c) * (j + 1 - c) + (i + 1 - c) * (i + 1 - c);
    float o = 0.0f;
    if (lr <= l2) o = __fmul_rn(__fmul_rn(R[((size_t)(ip + k) * N + (ip + j)) * N + (ip + i)], pix), wkb[lr]);
    vol[q] = o;
  }
}

}  // namespace spi

using namespace spi;

struct spi_fslice_plan {
  spi_ctx* ctx = nullptr;
  int device = 0, nx = 0, n = 0, nang = 0, sm_count = 148;
  SliceDesc* sl = nullptr;        // [nang]
  float* tab = nullptr;        // KB table, 5000 floats
  float fltb = 0.0f;
  float* wkb = nullptr;        // |WKB(LR)|, LR = 0..(nx/2)^2
  // staging and volume buffers (made on first use; not part of the capturable calls)
  cufftHandle r2c = 0, c2r = 0, r2c_tail = 0;
  int r2c_batch = 0, r2c_tail_batch = 0;
  float* padded = nullptr;     // [r2c_batch][n][n]
  float2* cplx = nullptr;      // [n][n][nx+1]
  float* real3 = nullptr;      // [n][n][n]
};

namespace {

int fs_blocks(const spi_fslice_plan* p) { return p->sm_count * 3; }
int fs_grid_blocks(const spi_fslice_plan* p, size_t work) {
  size_t b = (work + 255) / 256, cap = (size_t)p->sm_count * 8;
  return (int)std::max<size_t>(1, std::min(b, cap));
}
size_t fs_grid_elems(const spi_fslice_plan* p) { return (size_t)(p->nx + 1) * p->n * p->n; }
constexpr size_t kFsSmem = 5000 * sizeof(float);
// work counters of the normal operator's insertion launches, `chunk` slices each
long long fs_counter_bytes(const spi_fslice_plan* p, long long chunk) {
  return (p->nang + chunk - 1) / chunk * (long long)sizeof(unsigned long long);
}
size_t fs_plane(const spi_fslice_plan* p) { return (size_t)p->n * (p->nx + 1); }

// per-device attributes of the extraction and insertion kernels
int fs_set_attributes(int device) {
  static std::atomic<unsigned long long> done{0};
  const unsigned long long bit = 1ull << (device & 63);
  if (done.load() & bit) return 0;
  auto set = [](auto kern, size_t smem) {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  };
  SPI_CUDA(set(fs_insert_kernel<SlabFs>, sizeof(SlabSmem<SlabFs>)));
  SPI_CUDA(set(fs_insert_kernel<SlabFs64>, sizeof(SlabSmem<SlabFs64>)));
  SPI_CUDA(set(fs_insert_kernel<SlabFs64d>, sizeof(SlabSmem<SlabFs64d>)));
  done.fetch_or(bit);
  return 0;
}

template <class F>
int fs_insert(const spi_fslice_plan* p, const void* slices, void* grid, int first, int count, unsigned long long* work,
              cudaStream_t s);

// Is E^T of the plan's slices faster tap by tap?  A column tile takes 10 to 20 us
// from its fetch to its sums, whatever the launch (steep slices most); in small
// boxes the reductions of few slices are over before.  us tap by tap / by columns,
// FP32: 16^3 with 1, 64, 256, 512 slices 21/34, 26/45, 57/57, 84/72; 64^3 with 1,
// 16, 64, 96 33/32, 39/57, 77/80, 100/98; 80^3 with 16, 64 52/63, 113/98; 96^3 with 1,
// 8, 16 44/33, 50/61, 62/58.  FP64: 16^3 with 64, 256, 512 32/60, 66/83, 104/96; 32^3
// with 1, 64, 128 34/31, 60/73, 93/88; 48^3 with 4, 16, 48 43/39, 53/55, 92/78; 64^3
// with 1, 16, 32 52/35, 67/84, 95/91.
bool fs_small(const spi_fslice_plan* p, bool fp64) {
  return p->nx < (fp64 ? 64 : 96) && p->nang <= 256 &&
         (long long)p->nang * p->nx * p->nx <= (fp64 ? 1 << 16 : 1 << 18);
}

// grid = E^T of all slices.  The work counter of the launch is a voxel of the
// output that no tap reaches, (x, y, z) = (NX, 0, 0): the plan may run on
// several streams at once, so the counter has to be the call's own.
template <class F>
int fs_adjoint(const spi_fslice_plan* p, const void* slices, void* grid, size_t voxel, cudaStream_t s) {
  SPI_CUDA(cudaMemsetAsync(grid, 0, fs_grid_elems(p) * voxel, s));
  if (fs_small(p, F::D)) {
    const long long rows = ((long long)p->nang * p->n + 7) / 8;
    fs_taps_kernel<F::D><<<(int)std::min<long long>(rows, fs_blocks(p)), 256, kFsSmem, s>>>(
        static_cast<const float2*>(slices), grid, p->sl, p->nang, p->nx, p->tab, p->fltb);
    SPI_TRY(check_kernel("fs_taps_kernel"));
    p->ctx->count();
    return 0;
  }
  auto* work = reinterpret_cast<unsigned long long*>(static_cast<char*>(grid) + (size_t)p->nx * voxel);
  SPI_TRY(fs_insert<F>(p, slices, grid, 0, p->nang, work, s));
  SPI_CUDA(cudaMemsetAsync(work, 0, sizeof(*work), s));
  return 0;
}

// E of slices [first, first + count) of the plan into out (its first slice first)
template <class T2>
int fs_extract(const spi_fslice_plan* p, const void* grid, void* out, int first, int count, cudaStream_t s) {
  const long long rows = ((long long)count * p->n + kExThreads / 32 - 1) / (kExThreads / 32);
  const int blocks = (int)std::min<long long>(rows, (long long)p->sm_count * ExBlocks<T2>::value);
  fs_extract_kernel<T2><<<blocks, kExThreads, 0, s>>>(static_cast<const T2*>(grid), static_cast<T2*>(out), p->sl + first,
                                                      count, p->nx, p->tab, p->fltb);
  SPI_TRY(check_kernel("fs_extract_kernel"));
  p->ctx->count();
  return 0;
}

// grid += E^T of slices [first, first + count), whose values start at
// `slices`; *work (device) is zero
template <class F>
int fs_insert(const spi_fslice_plan* p, const void* slices, void* grid, int first, int count, unsigned long long* work,
              cudaStream_t s) {
  SlabArgs a{};
  a.ncls = 1;
  SlabClass& m = a.cls[0];
  // descriptors hold the slices' indices in the plan
  m.spec = static_cast<const typename F::Raw*>(slices) - (ptrdiff_t)first * (ptrdiff_t)fs_plane(p);
  m.slices = p->sl + first;
  m.g0 = m.g1 = grid;
  m.tab = p->tab;
  m.nx = p->nx;
  m.nslices = count;
  m.fltb = p->fltb;
  const long long most = (long long)p->sm_count * (F::D ? kSlabBlocks64 : kSlabBlocks);
  a.nitems = slab_items(most, a.cls, 1);
  fs_insert_kernel<F><<<(int)std::min(most, a.nitems), kSlabThreads + 32, sizeof(SlabSmem<F>), s>>>(a, work);
  SPI_TRY(check_kernel("fs_insert_kernel"));
  p->ctx->count();
  return 0;
}

}  // namespace

extern "C" {

int spi_fslice_plan_create(spi_ctx* ctx, int nx, const float* angles, int nang, spi_fslice_plan** out) {
  if (!ctx || !out) return fail(kInvalid, "spi_fslice_plan_create: NULL argument");
  *out = nullptr;
  if (nx < 8 || nx > 512) return fail(kInvalid, "spi_fslice_plan_create: nx = %d must be 8..512", nx);
  if (nang < 1 || !angles) return fail(kInvalid, "spi_fslice_plan_create: %d angles", nang);
  SPI_CUDA(cudaSetDevice(ctx->device));
  KBTab kb;
  fill_kb(2 * nx, kb);
  {
    // zero from distance 1.805 on, as FILLBESSIL's tables are
    const int i0 = std::max(0, (int)std::floor(1.805 * kb.fltb));
    for (int i = i0; i < 5000; ++i)
      if (kb.tab[i] != 0.0f)
        return fail(kInvalid, "spi_fslice_plan_create: the interpolation table of nx = %d has more than four "
                              "nonzero taps per axis", nx);
  }
  SPI_TRY(fs_set_attributes(ctx->device));
  std::vector<SliceDesc> hs(nang);
  for (int a = 0; a < nang; ++a) {
    float dm[9];
    cang(angles[3 * a + 2], angles[3 * a + 1], angles[3 * a + 0], dm);   // BUILDM1 (bp3f.f:1287)
    std::memcpy(hs[a].dm, dm, 6 * sizeof(float));
    hs[a].img = a;
    hs[a].grid = 0;
  }
  std::vector<float> wkb;
  windkb_table(nx, kb, wkb);
  auto* p = new spi_fslice_plan();
  p->ctx = ctx;
  p->device = ctx->device;
  p->sm_count = ctx->sm_count;
  p->nx = nx;
  p->n = 2 * nx;
  p->nang = nang;
  p->fltb = kb.fltb;
  cudaError_t e = cudaMalloc(&p->sl, sizeof(SliceDesc) * nang);
  if (e == cudaSuccess) e = cudaMalloc(&p->tab, sizeof(kb.tab));
  if (e == cudaSuccess) e = cudaMalloc(&p->wkb, wkb.size() * sizeof(float));
  if (e == cudaSuccess) e = cudaMemcpy(p->sl, hs.data(), sizeof(SliceDesc) * nang, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(p->tab, kb.tab, sizeof(kb.tab), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(p->wkb, wkb.data(), wkb.size() * sizeof(float), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    spi_fslice_plan_destroy(p);
    return fail(kAlloc, "spi_fslice_plan_create: %s", cudaGetErrorString(e));
  }
  *out = p;
  return 0;
}

int spi_fslice_plan_destroy(spi_fslice_plan* p) {
  if (!p) return 0;
  cudaSetDevice(p->device);
  if (p->r2c) cufftDestroy(p->r2c);
  if (p->r2c_tail) cufftDestroy(p->r2c_tail);
  if (p->c2r) cufftDestroy(p->c2r);
  cudaFree(p->sl);
  cudaFree(p->tab);
  cudaFree(p->wkb);
  cudaFree(p->padded);
  cudaFree(p->cplx);
  cudaFree(p->real3);
  delete p;
  return 0;
}

int spi_fslice_stage(spi_fslice_plan* p, const float* imgs, float* slices, void* stream) {
  if (!p || !imgs || !slices) return fail(kInvalid, "spi_fslice_stage: NULL argument");
  SPI_CUDA(cudaSetDevice(p->device));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int nx = p->nx, n = p->n;
  if (!p->r2c) {
    p->r2c_batch = (int)std::max<size_t>(1, std::min<size_t>((size_t)p->nang, (512ull << 20) / ((size_t)n * n * 4)));
    SPI_CUDA(cudaMalloc(&p->padded, (size_t)p->r2c_batch * n * n * sizeof(float)));
    int dims[2] = {n, n};
    SPI_CUFFT(cufftPlanMany(&p->r2c, 2, dims, nullptr, 1, n * n, nullptr, 1, n * (n / 2 + 1), CUFFT_R2C,
                            p->r2c_batch));
  }
  SPI_CUFFT(cufftSetStream(p->r2c, s));
  const size_t plane = (size_t)n * (nx + 1);
  for (int a0 = 0; a0 < p->nang; a0 += p->r2c_batch) {
    const int nb = std::min(p->r2c_batch, p->nang - a0);
    SPI_TRY(stage_images(p->ctx, s, imgs + (size_t)a0 * nx * nx, nx, nb, p->padded));
    cufftHandle plan = p->r2c;
    if (nb < p->r2c_batch) {   // a shorter last batch has a plan of its own
      if (p->r2c_tail_batch != nb) {
        if (p->r2c_tail) cufftDestroy(p->r2c_tail);
        p->r2c_tail = 0;
        p->r2c_tail_batch = 0;
        int dims[2] = {n, n};
        SPI_CUFFT(cufftPlanMany(&p->r2c_tail, 2, dims, nullptr, 1, n * n, nullptr, 1, n * (n / 2 + 1), CUFFT_R2C, nb));
        p->r2c_tail_batch = nb;
      }
      plan = p->r2c_tail;
      SPI_CUFFT(cufftSetStream(plan, s));
    }
    SPI_CUFFT(cufftExecR2C(plan, p->padded, reinterpret_cast<cufftComplex*>(slices) + (size_t)a0 * plane));
  }
  p->ctx->count();
  return 0;
}

int spi_fslice_forward(const spi_fslice_plan* p, const float* grid, float* slices, void* stream) {
  if (!p || !grid || !slices) return fail(kInvalid, "spi_fslice_forward: NULL argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return fs_extract<float2>(p, grid, slices, 0, p->nang, s);
}

int spi_fslice_adjoint(const spi_fslice_plan* p, const float* slices, float* grid, void* stream) {
  if (!p || !grid || !slices) return fail(kInvalid, "spi_fslice_adjoint: NULL argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return fs_adjoint<SlabFs>(p, slices, grid, sizeof(float2), s);
}

int spi_fslice_normal(const spi_fslice_plan* p, const float* grid_in, float lam, float* grid_out, void* stream) {
  if (!p || !grid_in || !grid_out) return fail(kInvalid, "spi_fslice_normal: NULL argument");
  if (grid_in == grid_out) return fail(kInvalid, "spi_fslice_normal: input and output must differ");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t ne = fs_grid_elems(p);
  fs_scale_kernel<<<fs_grid_blocks(p, ne), 256, 0, s>>>(reinterpret_cast<const float2*>(grid_in), lam,
                                                        reinterpret_cast<float2*>(grid_out), ne);
  SPI_TRY(check_kernel("fs_scale_kernel"));
  fs_normal_kernel<<<fs_blocks(p), 256, kFsSmem, s>>>(reinterpret_cast<const float2*>(grid_in),
                                                   reinterpret_cast<float2*>(grid_out), p->sl, p->nang, p->nx, p->tab,
                                                   p->fltb);
  SPI_TRY(check_kernel("fs_normal_kernel"));
  p->ctx->count(2);
  return 0;
}

int spi_fslice_normal64(const spi_fslice_plan* p, const double* grid_in, double lam, double* grid_out, void* stream) {
  if (!p || !grid_in || !grid_out) return fail(kInvalid, "spi_fslice_normal64: NULL argument");
  if (grid_in == grid_out) return fail(kInvalid, "spi_fslice_normal64: input and output must differ");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t ne = fs_grid_elems(p);
  fs_scale64_kernel<<<fs_grid_blocks(p, ne), 256, 0, s>>>(reinterpret_cast<const double2*>(grid_in), lam,
                                                          reinterpret_cast<double2*>(grid_out), ne);
  SPI_TRY(check_kernel("fs_scale64_kernel"));
  fs_normal64_kernel<<<fs_blocks(p), 256, kFsSmem, s>>>(reinterpret_cast<const double2*>(grid_in),
                                                        reinterpret_cast<double2*>(grid_out), p->sl, p->nang, p->nx,
                                                        p->tab, p->fltb);
  SPI_TRY(check_kernel("fs_normal64_kernel"));
  p->ctx->count(2);
  return 0;
}

int spi_fslice_forward64(const spi_fslice_plan* p, const double* grid, double* slices, void* stream) {
  if (!p || !grid || !slices) return fail(kInvalid, "spi_fslice_forward64: NULL argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return fs_extract<double2>(p, grid, slices, 0, p->nang, s);
}

int spi_fslice_adjoint64(const spi_fslice_plan* p, const float* slices, double* grid, void* stream) {
  if (!p || !grid || !slices) return fail(kInvalid, "spi_fslice_adjoint64: NULL argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return fs_adjoint<SlabFs64>(p, slices, grid, sizeof(double2), s);
}

int spi_fslice_normal_ws_bytes(const spi_fslice_plan* p, int fp64, long long* bytes) {
  if (!p || !bytes) return fail(kInvalid, "spi_fslice_normal_ws_bytes: NULL argument");
  const long long per = (long long)fs_plane(p) * (fp64 ? sizeof(double2) : sizeof(float2));
  // about 128 MB of slices: 242 of 128^3 in FP64, 0.6 ms of work per pair of launches
  const long long chunk = std::max(1LL, std::min<long long>(p->nang, (128LL << 20) / per));
  *bytes = per * chunk + fs_counter_bytes(p, chunk);
  return 0;
}

int spi_fslice_normal_ws(const spi_fslice_plan* p, const void* grid_in, double lam, void* grid_out, int fp64, void* ws,
                         long long ws_bytes, void* stream) {
  if (!p || !grid_in || !grid_out || !ws) return fail(kInvalid, "spi_fslice_normal_ws: NULL argument");
  if (grid_in == grid_out) return fail(kInvalid, "spi_fslice_normal_ws: input and output must differ");
  const long long per = (long long)fs_plane(p) * (fp64 ? sizeof(double2) : sizeof(float2));
  // as many slices as fit beside one work counter per insertion launch
  long long chunk = std::min<long long>(p->nang, ws_bytes / per);
  while (chunk > 0 && chunk * per + fs_counter_bytes(p, chunk) > ws_bytes) --chunk;
  if (chunk < 1)
    return fail(kInvalid, "spi_fslice_normal_ws: workspace of %lld bytes, one slice and the counters take %lld", ws_bytes,
                per + fs_counter_bytes(p, 1));
  if (reinterpret_cast<uintptr_t>(ws) % 16)
    return fail(kInvalid, "spi_fslice_normal_ws: the workspace must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t ne = fs_grid_elems(p);
  if (fp64)
    fs_scale64_kernel<<<fs_grid_blocks(p, ne), 256, 0, s>>>(static_cast<const double2*>(grid_in), lam,
                                                            static_cast<double2*>(grid_out), ne);
  else
    fs_scale_kernel<<<fs_grid_blocks(p, ne), 256, 0, s>>>(static_cast<const float2*>(grid_in), (float)lam,
                                                          static_cast<float2*>(grid_out), ne);
  SPI_TRY(check_kernel("fs_scale_kernel"));
  p->ctx->count();
  auto* work = reinterpret_cast<unsigned long long*>(static_cast<char*>(ws) + chunk * per);
  SPI_CUDA(cudaMemsetAsync(work, 0, (size_t)fs_counter_bytes(p, chunk), s));
  for (int a = 0; a < p->nang; a += (int)chunk, ++work) {
    const int n = std::min((int)chunk, p->nang - a);
    if (fp64) {
      SPI_TRY((fs_extract<double2>(p, grid_in, ws, a, n, s)));
      SPI_TRY(fs_insert<SlabFs64d>(p, ws, grid_out, a, n, work, s));
    } else {
      SPI_TRY((fs_extract<float2>(p, grid_in, ws, a, n, s)));
      SPI_TRY(fs_insert<SlabFs>(p, ws, grid_out, a, n, work, s));
    }
  }
  return 0;
}

int spi_fslice_volume(spi_fslice_plan* p, const float* grid, float* vol_out, void* stream) {
  if (!p || !grid || !vol_out) return fail(kInvalid, "spi_fslice_volume: NULL argument");
  SPI_CUDA(cudaSetDevice(p->device));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int nx = p->nx, n = p->n;
  if (!p->c2r) {
    SPI_CUDA(cudaMalloc(&p->cplx, fs_grid_elems(p) * sizeof(float2)));
    SPI_CUDA(cudaMalloc(&p->real3, (size_t)n * n * n * sizeof(float)));
    SPI_CUFFT(cufftPlan3d(&p->c2r, n, n, n, CUFFT_C2R));
  }
  SPI_CUFFT(cufftSetStream(p->c2r, s));
  const size_t ne = fs_grid_elems(p);
  fs_vol_prep_kernel<<<fs_grid_blocks(p, ne), 256, 0, s>>>(reinterpret_cast<const float2*>(grid), p->cplx, nx);
  SPI_TRY(check_kernel("fs_vol_prep_kernel"));
  SPI_CUFFT(cufftExecC2R(p->c2r, reinterpret_cast<cufftComplex*>(p->cplx), p->real3));
  const int ip = (n - nx) / 2 + nx % 2;
  const float pix = 1.0f / (float)((long long)n * n * n);
  fs_vol_out_kernel<<<fs_grid_blocks(p, (size_t)nx * nx * nx), 256, 0, s>>>(p->real3, nx, ip, pix, p->wkb, vol_out);
  SPI_TRY(check_kernel("fs_vol_out_kernel"));
  p->ctx->count(2);
  return 0;
}

}  // extern "C"
