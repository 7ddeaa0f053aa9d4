// Central-slice extraction E (the exact adjoint of the column insertion) from
// complex grids in FP32 and FP64, on sm_100a.  Included by fslice.cu.
//
// A warp takes one row J of one slice, eight pixels at a time, four lanes per
// pixel: lane q reads x tap FX + q of the four-voxel window at its 4 x 4 (y, z)
// voxels, so a pixel's reads for one (y, z) are 32 (FP64: 64) contiguous
// bytes and neighbouring pixels find each other's voxels in L1.  The lane's 16
// voxels are four plane and four row offsets in 32 bits, made once per pixel;
// the window starts come from the coordinates (slab_first), not from table
// look-ups, and an index rounds by two additions (slab_nint).
//
// Bound by L1 (a pixel's 16 reads touch 16 lines) and issue.  Before, with the
// window starts looked up in the table and every tap's 64-bit index and
// reflection made anew, and now, us per slice: FP32 64^3 1.17 -> 0.51, 128^3
// 4.42 -> 2.02, 150^3 6.41 -> 2.42, 256^3 25.0 -> 8.7.
// Staging a tile's voxel columns in shared memory, each once, and summing 64
// taps per thread from there was measured too (16 x 16 pixels in FP32, 16 x 8
// with two threads per pixel in FP64): a tile's columns, their addresses and
// two barriers cost more than the reads they save (FP32 3.2, FP64 6.2 us per slice at
// 128^3).
#pragma once

#include "slab.cuh"

namespace spi {

constexpr int kExThreads = 256;
// CTAs per SM launched, measured with 2 to 8: FP32 (5 resident) 8 is best at 64^3, 150^3 and
// 256^3 (0.51, 2.42, 8.7 us per slice; 4: 0.55, 2.62, 10.4) and 4 at 128^3 (1.89 against
// 2.02); the FP64 normal operator is best with 4 at 128^3 and 256^3 (6.4 and 27.0 us; 8: 6.6 and 27.6)
template <class T2>
struct ExBlocks {
  static constexpr int value = sizeof(T2) == 8 ? 8 : 4;
};
constexpr int kExTab = 3336;   // a pixel's window reaches distances below 2, entry 3,333

__device__ __forceinline__ void ex_add(float2& a, float2 x, float w, bool conj_) {
  a.x = fmaf(x.x, w, a.x);
  a.y = fmaf(conj_ ? -x.y : x.y, w, a.y);
}
__device__ __forceinline__ void ex_add(double2& a, double2 x, float w, bool conj_) {
  const double d = (double)w;
  a.x = fma(x.x, d, a.x);
  a.y = fma(conj_ ? -x.y : x.y, d, a.y);
}

// Slices [0, nslices): slice s of the launch goes to out + s * 2 NX * (NX + 1)
template <class T2>
__global__ void __launch_bounds__(kExThreads) fs_extract_kernel(const T2* __restrict__ X, T2* __restrict__ out,
                                                                const SliceDesc* __restrict__ slices, int nslices,
                                                                int nx, const float* __restrict__ kbtab, float fltb) {
  __shared__ float tab[kExTab];
  for (int i = threadIdx.x; i < kExTab; i += kExThreads) tab[i] = kbtab[i];
  __syncthreads();
  const int N = 2 * nx, lane = threadIdx.x & 31;
  const int g = lane >> 2, q = lane & 3, gl = lane & ~3;
  const unsigned rl = (unsigned)(nx + 1), pl = (unsigned)N * rl;
  const long long nitems = (long long)nslices * N;
  const long long warps = (long long)gridDim.x * (kExThreads >> 5);
  auto tap = [&](float c, int k) { return tab[slab_nint(__fmul_rn(fabsf(__fsub_rn(c, (float)k)), fltb))]; };
  for (long long item = (long long)blockIdx.x * (kExThreads >> 5) + (threadIdx.x >> 5); item < nitems; item += warps) {
    const int s = (int)(item / N), J = (int)(item % N) - nx + 1;
    const SliceDesc sd = slices[s];
    T2* row = out + ((size_t)s * N + (J >= 0 ? J : N + J)) * rl;
    const float fj = (float)J;
    const float xj = __fmul_rn(fj, sd.dm[3]), yj = __fmul_rn(fj, sd.dm[4]), zj = __fmul_rn(fj, sd.dm[5]);
    // a matrix that is not a rotation's (an angle that is not finite) has no taps: its rows are zero
    const bool rotation = slab_rotation(sd.dm);
    int I0 = 0;
    for (; rotation && I0 <= nx && I0 * I0 + J * J < nx * nx; I0 += 8) {   // warp-uniform
      const int I = I0 + g;
      float x, y, z;
      bool flip;
      const bool ok = slab_extract_pixel(sd.dm, xj, yj, zj, I, J, nx, x, y, z, flip);
      const int fx = slab_first(x), fy = slab_first(y), fz = slab_first(z);
      const float tx = tap(x, fx + q), tyq = tap(y, fy + q), tzq = tap(z, fz + q);
      // main tap (ixp, iyp, izp), or for ixp < 0 the reflected point with the conjugate value
      const int ixp = fx + q;
      const bool refl = ixp < 0;
      float ty[4], tz[4];
      unsigned yo[4], zo[4];
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        ty[l] = __shfl_sync(0xffffffffu, tyq, gl + l);
        tz[l] = __shfl_sync(0xffffffffu, tzq, gl + l);
        const int iy = refl ? -(fy + l) : fy + l, iz = refl ? -(fz + l) : fz + l;
        yo[l] = (unsigned)(iy < 0 ? N + iy : iy) * rl + (unsigned)(refl ? -ixp : ixp);
        zo[l] = (unsigned)(iz < 0 ? N + iz : iz) * pl;
      }
      T2 a;
      a.x = a.y = 0;
      if (ok && tx != 0.0f) {
#pragma unroll
        for (int lz = 0; lz < 4; ++lz)
#pragma unroll
          for (int ly = 0; ly < 4; ++ly) {
            const float wg = __fmul_rn(tx, __fmul_rn(ty[ly], tz[lz]));
            if (wg != 0.0f) ex_add(a, __ldg(X + (size_t)(zo[lz] + yo[ly])), wg, refl);
          }
      }
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
        a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
      }
      // BI_adj = the sum (conjugated for a flipped pixel); T = conj(BI_adj)
      if (!flip) a.y = -a.y;
      if (q == 0 && I <= nx) row[I] = a;
    }
    for (int I = I0 + lane; I <= nx; I += 32) row[I] = T2{0, 0};
  }
}

}  // namespace spi
