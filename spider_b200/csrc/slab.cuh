// Column insertion of central slices (ONELINE, oneline.f:38-200) on sm_100a.
// Used by bp.cu (grids of {Re X, Im X, W, 0}) and fslice.cu (complex grids in
// FP32 and FP64, without W); the geometry is in slab_geom.h.
//
// A form that adds every tap with its own 16-byte L2 reduction (47 taps per
// pixel, 13 of one slice on every voxel, four lanes per pixel over the four
// nonzero taps of each axis) is bound by those reductions and the instructions
// around them: 15.7 ms per 1,024 images at 256^3, L2 atomic input 54% busy.
// Here a voxel's taps of one slice are summed in registers and go out as one
// reduction, 0.08 per tap.  A CTA takes a tile of 16 x 16 voxel columns of one
// slice: it stages the tile's pixels in shared memory (position, value, the
// four weights along w), then every thread walks the pixels that reach its two
// columns and adds (value, 1) times the weight along u and v times each
// of the four along w to the columns' voxels, kept in registers by their
// residue modulo 8 (12 for steep slices, 20% of orientations), two voxels per
// instruction (fma.rn.f32x2).
//
// What bounds it: shared memory reads (wavefronts 84% of their peak while
// active, ncu at 256^3) and instruction issue (2.7 per cycle); L2 atomic input
// is at 13%.  Measured (images/s, insertion alone, before -> after): 64^3
// 1.04M -> 1.72M, 128^3 267k -> 492k, 192^3 116k -> 229k, 256^3 65.3k -> 135.7k.
// The choices, each measured at 256^3 (ms per 1,024 images, 7.5 as it stands):
// two columns per thread (one: 9.3; a 2 x 2 block: 9.8, its registers leave 12
// warps per SM); weights along u and v looked up per column instead of staged
// per pixel (fewer bytes per pixel read, 12 -> 4 look-ups in the staging); the
// next pixel's reads and look-ups ahead of this one's products (8.5 without);
// a producer warp that fetches the next tile's spectrum values while this one is
// gathered (9.0 with every warp fetching its own); steep slices one column
// at a time, which leaves registers for four CTAs per SM (8.8 with three).
#pragma once

#include <cuda_bf16.h>

#include <type_traits>

#include "slab_geom.h"

namespace spi {

struct SliceDesc {
  float dm[6];  // DMS(1:6): first two columns of the (symmetrised) rotation
  int img;      // index of the slice's values in the launch
  int grid;     // target grid (BP 32F half set)
};
static_assert(sizeof(SliceDesc) == 32, "slice descriptor is 32 bytes");

// What a column insertion reads and adds: slice values of type Raw, a weight
// grid or not, sums in FP32 or FP64.
template <class Raw_, bool W_, bool D_>
struct SlabForm {
  using Raw = Raw_;
  static constexpr bool W = W_, D = D_;
};
using SlabBp = SlabForm<float2, true, false>;              // float4 grid {Re X, Im X, W, 0}
using SlabBpBf16 = SlabForm<__nv_bfloat162, true, false>;  // the same from BF16 spectra
using SlabFs = SlabForm<float2, false, false>;             // float2 grid
using SlabFs64 = SlabForm<float2, false, true>;            // double2 grid from FP32 slices
using SlabFs64d = SlabForm<double2, false, true>;          // double2 grid from FP64 slices

// G[i] += v as one 16-byte reduction in L2 (red.global.add.v4.f32).  The
// address is converted to the global window explicitly: the kernel takes its
// grid pointer from shared memory, and on such a generic pointer
// atomicAdd(float4*) was not compiled to the vector reduction (measured:
// 1.9x the instructions and no L2 reduction requests).
__device__ __forceinline__ void red_add_v4(float4* p, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(__cvta_generic_to_global(p)), "f"(v.x),
               "f"(v.y), "f"(v.z), "f"(v.w));
}
// voxel i of the form's grid += (re, im) and its weight
template <class F>
__device__ __forceinline__ void slab_red(void* grid, size_t i, float re, float im, float w) {
  if (F::W) {
    red_add_v4(static_cast<float4*>(grid) + i, make_float4(re, im, w, 0.0f));
  } else {
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(__cvta_generic_to_global(static_cast<float2*>(grid) + i)),
                 "f"(re), "f"(im));
  }
}
__device__ __forceinline__ void slab_red64(void* grid, size_t i, double re, double im) {
  const auto a = __cvta_generic_to_global(static_cast<double2*>(grid) + i);
  asm volatile("red.global.add.f64 [%0], %1;" ::"l"(a), "d"(re));
  asm volatile("red.global.add.f64 [%0+8], %1;" ::"l"(a), "d"(im));
}

constexpr int kSlabMaxClass = 16;
constexpr int kSlabThreads = kSlabTile * kSlabTile / 2;   // consumers: two columns each, neighbours along v
constexpr int kSlabBlocks = 4;                            // CTAs per SM (96 registers, 54 KB each)
constexpr int kSlabBlocks64 = 3;                          // the same with FP64 sums (128 registers, 48-59 KB)

struct SlabClass {
  const void* spec;            // spectra of the class's images in this launch
  const SliceDesc* slices;
  void* g0;                    // grids the taps go to (half-set 1 and 2)
  void* g1;
  const float* tab;            // interpolation table (5,000 entries)
  long long item0;             // first work item of the class
  int nx, nslices;
  int parts;                   // items per row of tiles
  float fltb;
};
struct SlabArgs {
  SlabClass cls[kSlabMaxClass];
  long long nitems;
  int ncls;
};

// A tile as the producer warp hands it over
struct SlabTile {
  SlabFrame f;
  void* g;                     // grid of its slice
  float fltb;
  int banks;                   // 0: no tile is left
  int u0, v0, jlo, nr, nx, cls;
  int4 rows[kSlabRows];        // {first staged pixel - lo, lo, hi, 0}
};
template <class F>
struct SlabSmem {
  typename std::conditional<F::D, float2, float4>::type pix[kSlabPix];   // {u, v, Re, Im}; FP64: {u, v}, the value in raw
  float4 t[kSlabPix];          // weights along w by residue modulo 4
  int code[kSlabPix];          // slab_masks, kSlabMate, kSlabRep
  SlabTile tile[2];
  typename F::Raw raw[2][kSlabPix];   // slice values
  float tab[kSlabTab];
};
// an SM's 228 KB hold kSlabBlocks (kSlabBlocks64) of them, with the kilobyte that each CTA takes besides
static_assert(sizeof(SlabSmem<SlabBp>) <= (228 / kSlabBlocks - 1) * 1024, "four CTAs per SM");
static_assert(sizeof(SlabSmem<SlabFs64d>) <= (228 / kSlabBlocks64 - 1) * 1024, "three CTAs per SM");

__device__ __forceinline__ unsigned long long slab_pack(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 slab_unpack(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
// barrier ID among n threads of the CTA
template <int ID>
__device__ __forceinline__ void slab_bar(int n) {
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "r"(n) : "memory");
}
// acc += a * b on both halves
__device__ __forceinline__ void slab_fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// Rows of the tile and their places among its staged pixels, by one warp
__device__ __forceinline__ void slab_setup(SlabTile& T, const SlabFrame& f, int u0, int v0, int nx, int jlo, int nr,
                                           int lane) {
  int lo[2] = {0, 0}, hi[2] = {-1, -1}, len[2] = {0, 0};
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int r = 2 * lane + e;
    if (r < nr) {
      slab_tile_span(f, u0, v0, nx, jlo + r, lo[e], hi[e]);
      len[e] = max(0, hi[e] - lo[e] + 1);
    }
  }
  int off = len[0] + len[1];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, off, o);
    if (lane >= o) off += v;
  }
  off -= len[0] + len[1];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int r = 2 * lane + e;
    // the capacity holds every tile of a rotation (slab_geom.h); a row that would pass it is cut
    if (r < nr) T.rows[r] = make_int4(off - lo[e], lo[e], min(hi[e], lo[e] + kSlabPix - 1 - off), 0);
    off += len[e];
  }
}

// 4, 8 or 16 bytes from global to shared memory, asynchronously
__device__ __forceinline__ void slab_copy(float2* dst, const float2* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void slab_copy(__nv_bfloat162* dst, const __nv_bfloat162* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void slab_copy(double2* dst, const double2* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ double2 slab_double2(float2 v) { return make_double2(v.x, v.y); }
__device__ __forceinline__ double2 slab_double2(double2 v) { return v; }
__device__ __forceinline__ float2 slab_float2(float2 v) { return v; }
__device__ __forceinline__ float2 slab_float2(__nv_bfloat162 v) { return make_float2(__low2float(v), __high2float(v)); }

// The spectrum values of the tile's pixels, by one warp, eight lanes per row:
// the stored pixel (I > 0, or I = 0 and J >= 0) or, for a mate, (-I, -J).
// Rows and spans stay within |I|, |J| < NX, so the reads are in range beyond
// the disc too.
template <class V>
__device__ __forceinline__ void slab_fetch(V* raw, const SlabTile& T, const V* spec, int nx, int jlo, int nr, int lane) {
  const int N = 2 * nx, rowlen = nx + 1;
  for (int r = lane >> 3; r < nr; r += 4) {
    const int4 row = T.rows[r];
    const int J = jlo + r;
    const V* up = spec + (J >= 0 ? J : N + J) * rowlen;
    const V* dn = spec + (J > 0 ? N - J : -J) * rowlen;
    for (int I = row.y + (lane & 7); I <= row.z; I += 8)
      slab_copy(raw + row.x + I, (I > 0 || (I == 0 && J >= 0)) ? up + I : dn - I);
  }
}

constexpr int kSlabMate = 1;   // not the canonical pixel of its pair
constexpr int kSlabRep = 2;    // the stored pixel of its pair

// Which residues of a window that starts at w lie in which bank.  Two banks:
// the sign of byte r says whether the window's voxel of residue r modulo 4
// lies in bank 0.  Three banks: bit 8 + 4 b + r.
template <int NB>
__device__ __forceinline__ int slab_masks(int w) {
  if (NB == 2) {   // residues r >= w mod 4 lie in bank (w / 4) mod 2, the others in the next
    const int m = (int)(0x80808080u << (8 * (w & 3)));
    return (w & 4 ? ~m : m) & (int)0x80808080u;
  }
  const unsigned m = 0xfu << slab_residue(w, NB);
  return (int)(((m | (m >> 12)) & 0xfffu) << 8);
}
// the sign of one byte of m over a word (PRMT's replicate mode, which __byte_perm masks out)
template <int SEL>
__device__ __forceinline__ int slab_sign(int m) {
  int r;
  asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(m), "n"(SEL));
  return r;
}
// Weights t by residue modulo 4 -> pairs (2 j, 2 j + 1) by residue modulo 4 NB
template <int NB>
__device__ __forceinline__ void slab_spread(const float4& t, int m, unsigned long long (&tt)[2 * NB]) {
  if (NB == 2) {
    const int x[4] = {__float_as_int(t.x), __float_as_int(t.y), __float_as_int(t.z), __float_as_int(t.w)};
    const int k[4] = {slab_sign<0x8888>(m), slab_sign<0x9999>(m), slab_sign<0xaaaa>(m), slab_sign<0xbbbb>(m)};
    tt[0] = slab_pack(__int_as_float(x[0] & k[0]), __int_as_float(x[1] & k[1]));
    tt[1] = slab_pack(__int_as_float(x[2] & k[2]), __int_as_float(x[3] & k[3]));
    tt[2] = slab_pack(__int_as_float(x[0] & ~k[0]), __int_as_float(x[1] & ~k[1]));
    tt[3] = slab_pack(__int_as_float(x[2] & ~k[2]), __int_as_float(x[3] & ~k[3]));
  } else {
#pragma unroll
    for (int k = 0; k < NB; ++k) {
      tt[2 * k] = slab_pack(m & (256 << (4 * k)) ? t.x : 0.0f, m & (512 << (4 * k)) ? t.y : 0.0f);
      tt[2 * k + 1] = slab_pack(m & (1024 << (4 * k)) ? t.z : 0.0f, m & (2048 << (4 * k)) ? t.w : 0.0f);
    }
  }
}

// The origin is its own mate: its reflected taps, x = -1 to x = 1, go out
// apart, once per slice.  b: its value.
template <class F>
__device__ __noinline__ void slab_origin(const float* tab, float fltb, void* G, int nx, double2 b) {
  const float w0 = tab[0], w1 = tab[slab_tab_index(0.0f, 1, fltb, kSlabTab - 1)];
  const int N = 2 * nx;
  for (int e = 0; e < 9; ++e) {
    const int y = e % 3 - 1, z = e / 3 - 1;
    const float wg = __fmul_rn(w1, __fmul_rn(y ? w1 : w0, z ? w1 : w0));
    const size_t i = ((size_t)(z < 0 ? N + z : z) * N + (y < 0 ? N + y : y)) * (size_t)(nx + 1) + 1;
    if (F::D) slab_red64(G, i, __dmul_rn(b.x, (double)wg), -__dmul_rn(b.y, (double)wg));
    else slab_red<F>(G, i, __fmul_rn((float)b.x, wg), -__fmul_rn((float)b.y, wg), wg);
  }
}

// The taps of a pixel whose value is not finite on the tile's columns, one by
// one: its products with zero weights, which slab_gather forms, would not be zero.
template <class F>
__device__ __noinline__ void slab_direct(const float* tab, const SlabTile& T, const SlabPix& p, double2 b) {
  const int nx = T.nx, N = 2 * nx;
  const int fu = slab_first(p.u), fv = slab_first(p.v), fw = slab_first(p.w);
  auto tap = [&](float c, int k) { return tab[slab_tab_index(c, k, T.fltb, kSlabTab - 1)]; };
  for (int e = 0; e < 64; ++e) {
    const int u = fu + (e & 3), v = fv + ((e >> 2) & 3), w = fw + (e >> 4);
    if (u < T.u0 || u >= T.u0 + kSlabTile || v < T.v0 || v >= T.v0 + kSlabTile) continue;
    const int x = T.f.d == 0 ? w : u, y = T.f.d == 0 ? u : T.f.d == 1 ? w : v, z = T.f.d == 2 ? w : v;
    if (x < 0 || (x == 0 && !p.canon)) continue;
    const float wg = __fmul_rn(tap(p.u, u), __fmul_rn(tap(p.v, v), tap(p.w, w)));
    if (wg == 0.0f) continue;
    const size_t i = ((size_t)(z < 0 ? N + z : z) * N + (y < 0 ? N + y : y)) * (size_t)(nx + 1) + x;
    if (F::D) slab_red64(T.g, i, __dmul_rn(b.x, (double)wg), __dmul_rn(b.y, (double)wg));
    else slab_red<F>(T.g, i, __fmul_rn((float)b.x, wg), __fmul_rn((float)b.y, wg), 0.0f);
  }
}

// The tile's pixels into the form that slab_gather reads: eight lanes per row
template <int NB, class F>
__device__ __forceinline__ void slab_stage(SlabSmem<F>& S, const SlabTile& T, const SlabFrame& f, int buf) {
  const int nx = T.nx, jlo = T.jlo, nr = T.nr, l8 = threadIdx.x & 7;
  const float fltb = T.fltb;
  for (int r = threadIdx.x >> 3; r < nr; r += kSlabThreads / 8) {
    const int4 row = T.rows[r];
    const int J = jlo + r;
#pragma unroll 1
    for (int I = row.y + l8; I <= row.z; I += 8) {
      const int q = row.x + I;
      const SlabPix p = slab_pixel(f, I, J);
      if (!slab_inside(f, p, I, J, nx)) {   // adds nothing
        if constexpr (F::D) {
          S.pix[q] = make_float2(p.u, p.v);
          S.raw[buf][q] = typename F::Raw{0, 0};
        } else {
          S.pix[q] = make_float4(p.u, p.v, 0.0f, 0.0f);
        }
        S.t[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        S.code[q] = 0;
        continue;
      }
      // SPIDER forward sign = conjugate of the cuFFT R2C output; conjugated again for a mate
      double2 val;
      bool fin;
      if constexpr (F::D) {
        const typename F::Raw sp = S.raw[buf][q];
        val = make_double2(sp.x, p.rep ? -sp.y : sp.y);
        fin = isfinite(sp.x) && isfinite(sp.y);
        S.pix[q] = make_float2(p.u, p.v);
        if (!fin) S.raw[buf][q] = typename F::Raw{0, 0};
      } else {
        const float2 sp = slab_float2(S.raw[buf][q]);
        const float bi = p.rep ? -sp.y : sp.y;
        val = make_double2(sp.x, bi);
        fin = isfinite(sp.x) && isfinite(bi);
        S.pix[q] = make_float4(p.u, p.v, fin ? sp.x : 0.0f, fin ? bi : 0.0f);
      }
      const int fw = slab_first(p.w);
      float tw[4];
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        tw[l] = S.tab[slab_nint(__fmul_rn(fabsf(__fsub_rn(p.w, (float)(fw + l))), fltb))];
        if (f.d == 0 && !p.canon && fw + l == 0) tw[l] = 0.0f;   // plane x = 0 takes the canonical pixels only
      }
      // residue r holds window position (r - fw) mod 4
      const bool s1 = fw & 1, s2 = fw & 2;
      const float a0 = s1 ? tw[3] : tw[0], a1 = s1 ? tw[0] : tw[1], a2 = s1 ? tw[1] : tw[2], a3 = s1 ? tw[2] : tw[3];
      S.t[q] = make_float4(s2 ? a2 : a0, s2 ? a3 : a1, s2 ? a0 : a2, s2 ? a1 : a3);
      S.code[q] = slab_masks<NB>(fw) | (p.canon ? 0 : kSlabMate) | (p.rep ? kSlabRep : 0);
      if (!fin) slab_direct<F>(S.tab, T, p, val);
      if (I == 0 && J == 0 && T.u0 <= 0 && T.u0 + kSlabTile > 0 && T.v0 <= 0 && T.v0 + kSlabTile > 0)
        slab_origin<F>(S.tab, fltb, T.g, nx, val);
    }
  }
}

// Voxels of one column by residue
struct SlabCol {
  int base, res, N;      // first voxel along w, its residue
  bool wx;               // w is x: no voxels below zero (the mate's taps)
  unsigned at0, step;    // voxel at w = 0 and the stride along w (grids hold < 2^32 voxels)
  template <int NB>
  __device__ __forceinline__ long long voxel(int j) const {   // of residue j; -1: none
    int off = j - res;
    if (off < 0) off += 4 * NB;
    int k = base + off;
    if (k < 0) {
      if (wx) return -1;
      k += N;
    }
    return (long long)(at0 + (unsigned)k * step);
  }
};
template <int NB>
__device__ __forceinline__ SlabCol slab_col(const SlabFrame& f, int nx, int U, int V) {
  SlabCol c;
  const unsigned rl = (unsigned)(nx + 1), N = 2u * (unsigned)nx;
  const unsigned iv = (unsigned)(V >= 0 ? V : (int)N + V);
  c.base = slab_col_base(f, (float)U, (float)V);
  c.res = slab_residue(c.base, NB);
  c.N = (int)N;
  c.wx = f.d == 0;
  if (f.d == 2) { c.at0 = iv * rl + (unsigned)U; c.step = N * rl; }
  else if (f.d == 1) { c.at0 = iv * N * rl + (unsigned)U; c.step = rl; }
  else { c.at0 = (iv * N + (unsigned)(U >= 0 ? U : (int)N + U)) * rl; c.step = 1u; }
  return c;
}

// Columns (U, V) .. (U, V + NC - 1): walk the pixels that reach them, keep the
// sums by residue in registers (pairs of residues 2 j, 2 j + 1 of Re X, Im X, W),
// and add them to the grid.
template <int NC, int NB, class F>
__device__ __forceinline__ void slab_gather(const SlabSmem<F>& S, const SlabTile& T, const SlabFrame& f, int U, int V) {
  const int nx = T.nx, jlo = T.jlo;
  const float fltb = T.fltb, u = (float)U, v = (float)V;
  constexpr int kSums = F::W ? 3 : 2;
  unsigned long long acc[NC][kSums][2 * NB];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int e = 0; e < kSums; ++e)
#pragma unroll
      for (int j = 0; j < 2 * NB; ++j) acc[c][e][j] = 0ull;
  const int mate = (f.d != 0 && U == 0) ? kSlabMate : 0;   // column x = 0 takes the canonical pixels only
  auto tap = [&](float p, float k) { return S.tab[slab_nint(__fmul_rn(fabsf(__fsub_rn(p, k)), fltb))]; };
  auto add = [&](const float4& b, const float4& t, int code, float wu, const float (&wv)[NC]) {
    unsigned long long tt[2 * NB];
    slab_spread<NB>(t, code, tt);
    if (code & mate) wu = 0.0f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const float w = __fmul_rn(wu, wv[c]), re = __fmul_rn(b.z, w), im = __fmul_rn(b.w, w);
      const unsigned long long w2 = slab_pack(w, w), re2 = slab_pack(re, re), im2 = slab_pack(im, im);
#pragma unroll
      for (int j = 0; j < 2 * NB; ++j) {
        slab_fma2(acc[c][0][j], re2, tt[j]);
        slab_fma2(acc[c][1][j], im2, tt[j]);
        if (F::W) slab_fma2(acc[c][kSums - 1][j], w2, tt[j]);
      }
    }
  };
  int r0, r1;
  slab_block_rows(f, u, v, 1, NC, jlo, T.nr, r0, r1);
  for (int r = r0; r <= r1; ++r) {
    const int4 row = T.rows[r];
    float fl, fh;
    slab_span(f, u, v + 0.5f * (NC - 1), kSlabR, kSlabR + 0.5f * (NC - 1), jlo + r, fl, fh);
    const int i0 = slab_ceil(fmaxf(fl, (float)row.y)), i1 = slab_floor(fminf(fh, (float)row.z));
    if (i0 > i1) continue;
    // the next pixel's reads and weights are under way while this one's products are added
    int q = row.x + i0;
    const int q1 = row.x + i1;
    float4 b = S.pix[q], t = S.t[q];
    int code = S.code[q];
    float wu = tap(b.x, u), wv[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) wv[c] = tap(b.y, v + (float)c);
    for (;;) {
      const int qn = min(q + 1, q1);
      const float4 bn = S.pix[qn], tn = S.t[qn];
      const int coden = S.code[qn];
      add(b, t, code, wu, wv);
      if (q >= q1) break;
      wu = tap(bn.x, u);
#pragma unroll
      for (int c = 0; c < NC; ++c) wv[c] = tap(bn.y, v + (float)c);
      b = bn; t = tn; code = coden; q = qn;
    }
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const SlabCol col = slab_col<NB>(f, nx, U, V + c);
#pragma unroll
    for (int j = 0; j < 2 * NB; ++j) {
      const float2 re = slab_unpack(acc[c][0][j]), im = slab_unpack(acc[c][1][j]), w = slab_unpack(acc[c][kSums - 1][j]);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float r = e ? re.y : re.x, i = e ? im.y : im.x, wg = e ? w.y : w.x;
        if (F::W ? wg == 0.0f : r == 0.0f && i == 0.0f) continue;
        const long long vx = col.voxel<NB>(2 * j + e);
        if (vx >= 0) slab_red<F>(T.g, (size_t)vx, r, i, wg);
      }
    }
  }
}

// The same with FP64 sums, one column: every tap's weight is the FP32 product
// TX * (TY * TZ) of the per-tap form, bit for bit, taken into FP64.
template <int NB, class F>
__device__ __forceinline__ void slab_gather64(const SlabSmem<F>& S, const SlabTile& T, const SlabFrame& f, int buf, int U,
                                              int V) {
  const int nx = T.nx, jlo = T.jlo;
  const float fltb = T.fltb, u = (float)U, v = (float)V;
  double re[4 * NB], im[4 * NB];
#pragma unroll
  for (int j = 0; j < 4 * NB; ++j) re[j] = im[j] = 0.0;
  const int mate = (f.d != 0 && U == 0) ? kSlabMate : 0;   // column x = 0 takes the canonical pixels only
  const bool wx = f.d == 0;                                // w is x: TX is the weight along w
  auto tap = [&](float p, float k) { return S.tab[slab_nint(__fmul_rn(fabsf(__fsub_rn(p, k)), fltb))]; };
  int r0, r1;
  slab_block_rows(f, u, v, 1, 1, jlo, T.nr, r0, r1);
  for (int r = r0; r <= r1; ++r) {
    const int4 row = T.rows[r];
    float fl, fh;
    slab_span(f, u, v, kSlabR, kSlabR, jlo + r, fl, fh);
    const int i0 = slab_ceil(fmaxf(fl, (float)row.y)), i1 = slab_floor(fminf(fh, (float)row.z));
    if (i0 > i1) continue;
    // the next pixel's reads and weights are under way while this one's products are added
    int q = row.x + i0;
    const int q1 = row.x + i1;
    float2 b = S.pix[q];
    float4 t = S.t[q];
    int code = S.code[q];
    double2 x = slab_double2(S.raw[buf][q]);
    float wu = tap(b.x, u), wv = tap(b.y, v);
    for (;;) {
      const int qn = min(q + 1, q1);
      const float2 bn = S.pix[qn];
      const float4 tn = S.t[qn];
      const int coden = S.code[qn];
      const double2 xn = slab_double2(S.raw[buf][qn]);
      if (code & mate) wu = 0.0f;
      const double xi = code & kSlabRep ? -x.y : x.y;
      const float tr[4] = {t.x, t.y, t.z, t.w};
      const float uv = __fmul_rn(wu, wv);
      int k[4];
      if (NB == 2) {
        k[0] = slab_sign<0x8888>(code); k[1] = slab_sign<0x9999>(code);
        k[2] = slab_sign<0xaaaa>(code); k[3] = slab_sign<0xbbbb>(code);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const double d = (double)(wx ? __fmul_rn(tr[e], uv) : __fmul_rn(wu, __fmul_rn(wv, tr[e])));
        if (NB == 2) {
          const int hi = __double2hiint(d), lo = __double2loint(d);
          const double d0 = __hiloint2double(hi & k[e], lo & k[e]), d1 = __hiloint2double(hi & ~k[e], lo & ~k[e]);
          re[e] = fma(x.x, d0, re[e]);
          im[e] = fma(xi, d0, im[e]);
          re[4 + e] = fma(x.x, d1, re[4 + e]);
          im[4 + e] = fma(xi, d1, im[4 + e]);
        } else {
#pragma unroll
          for (int n = 0; n < NB; ++n) {
            if (code & (256 << (4 * n + e))) {
              re[4 * n + e] = fma(x.x, d, re[4 * n + e]);
              im[4 * n + e] = fma(xi, d, im[4 * n + e]);
            }
          }
        }
      }
      if (q >= q1) break;
      wu = tap(bn.x, u);
      wv = tap(bn.y, v);
      b = bn; t = tn; code = coden; x = xn; q = qn;
    }
  }
  const SlabCol col = slab_col<NB>(f, nx, U, V);
#pragma unroll
  for (int j = 0; j < 4 * NB; ++j) {
    if (re[j] == 0.0 && im[j] == 0.0) continue;
    const long long vx = col.voxel<NB>(j);
    if (vx >= 0) slab_red64(T.g, (size_t)vx, re[j], im[j]);
  }
}

// One tile of one slice, by the consumer warps
template <int NB, class F>
__device__ __forceinline__ void slab_tile(SlabSmem<F>& S, const SlabTile& T, int buf) {
  const SlabFrame f = T.f;
  slab_stage<NB, F>(S, T, f, buf);
  slab_bar<2>(kSlabThreads);
  // Steep slices (three banks) and FP64 sums take a thread's two columns one after the
  // other: about as many operations as together, and their sums fit the registers.
  const int U = T.u0 + (threadIdx.x & 15), V = T.v0 + 2 * (threadIdx.x >> 4);
  if constexpr (F::D) {
#pragma unroll 1
    for (int c = 0; c < 2; ++c) slab_gather64<NB, F>(S, T, f, buf, U, V + c);
  } else if (NB == 2) {
    slab_gather<2, NB, F>(S, T, f, U, V);
  } else {
#pragma unroll 1
    for (int c = 0; c < 2; ++c) slab_gather<1, NB, F>(S, T, f, U, V + c);
  }
}

// A CTA is one producer warp and kSlabThreads consumers.  The producer takes
// work items (a slice's row of tiles along u, or every `parts`-th tile of it
// when a launch has few slices) in slice-major order and prepares tile k + 1
// -- its frame, rows and the copies of its slice values -- while the consumers
// stage and gather tile k.  The two meet once per tile.  `work`: a counter of
// the launch, zero at its start (a grid stride over the items instead left the
// SMs idle for a quarter of 240 slices at 128^3: rows differ in length).
template <class F>
__device__ __forceinline__ void slab_main(const SlabArgs& P, unsigned long long* __restrict__ work) {
  extern __shared__ __align__(16) unsigned char slab_raw[];
  SlabSmem<F>& S = *reinterpret_cast<SlabSmem<F>*>(slab_raw);
  const int tid = threadIdx.x;
  if (tid >= kSlabThreads) {
    const int lane = tid - kSlabThreads;
    using V = typename F::Raw;
    int buf = 0;
    unsigned long long next = 0;   // the item after the current one
    if (lane == 0) next = atomicAdd(work, 1ull);
    for (;;) {
      const long long item = (long long)__shfl_sync(0xffffffffu, next, 0);
      if (item >= P.nitems) break;
      if (lane == 0) next = atomicAdd(work, 1ull);
      int c = 0;
      while (c + 1 < P.ncls && P.cls[c + 1].item0 <= item) ++c;
      const SlabClass& C = P.cls[c];
      const int nx = C.nx, ntv = (2 * nx + kSlabTile - 1) / kSlabTile;
      const long long local = item - C.item0;
      const int per = ntv * C.parts;
      const int s = (int)(local / per), rem = (int)(local % per);
      const SliceDesc sd = C.slices[s];
      SlabFrame f;
      if (!slab_frame(sd.dm, f)) continue;
      const V* spec = static_cast<const V*>(C.spec) + (size_t)sd.img * (2 * nx) * (nx + 1);
      const int v0 = -nx + kSlabTile * (rem / C.parts);
      const int ub = f.d == 0 ? -nx : 0;
      const int ntu = (nx - ub + kSlabTile - 1) / kSlabTile;
      for (int tu = rem % C.parts; tu < ntu; tu += C.parts) {
        const int u0 = ub + kSlabTile * tu;
        if (!slab_tile_live(f, u0, v0, nx)) continue;
        SlabTile& T = S.tile[buf];
        int jlo, nr;
        slab_tile_rows(f, u0, v0, nx, jlo, nr);
        slab_setup(T, f, u0, v0, nx, jlo, nr, lane);
        if (lane == 0) {
          T.f = f;
          T.g = sd.grid ? C.g1 : C.g0;
          T.fltb = C.fltb;
          T.banks = slab_banks(f);
          T.u0 = u0; T.v0 = v0; T.jlo = jlo; T.nr = nr; T.nx = nx; T.cls = c;
        }
        __syncwarp();
        slab_fetch(S.raw[buf], T, spec, nx, jlo, nr, lane);
        asm volatile("cp.async.wait_all;" ::: "memory");
        slab_bar<1>(kSlabThreads + 32);   // hands tile k over; the consumers are done with tile k - 1
        buf ^= 1;
      }
    }
    if (lane == 0) S.tile[buf].banks = 0;
    slab_bar<1>(kSlabThreads + 32);
    return;
  }
  int have = -1;   // class whose table is in shared memory
  for (int buf = 0;; buf ^= 1) {
    slab_bar<1>(kSlabThreads + 32);
    const SlabTile& T = S.tile[buf];
    if (T.banks == 0) break;
    if (T.cls != have) {
      have = T.cls;
      for (int i = tid; i < kSlabTab; i += kSlabThreads) S.tab[i] = P.cls[have].tab[i];
      slab_bar<2>(kSlabThreads);
    }
    if (T.banks == 2) slab_tile<2, F>(S, T, buf);
    else slab_tile<3, F>(S, T, buf);
  }
}

// BP 3F / BP 32F
template <class F>
__global__ void __launch_bounds__(kSlabThreads + 32, kSlabBlocks) insert_x4_kernel(const __grid_constant__ SlabArgs P,
                                                                                unsigned long long* __restrict__ work) {
  slab_main<F>(P, work);
}

// Work items of the classes: a slice's row of tiles each, or its parts when
// all rows together would give the launch's `blocks` CTAs fewer than eight
// items (the tail of a launch is about half an item per CTA: 200 slices at
// 64^3 0.148 against 0.176 ms with whole rows).  Returns their number.
inline long long slab_items(long long blocks, SlabClass* cls, int ncls) {
  auto rows_of = [](const SlabClass& m) { return (long long)m.nslices * ((2 * m.nx + kSlabTile - 1) / kSlabTile); };
  long long rows = 0, items = 0;
  for (int k = 0; k < ncls; ++k) rows += rows_of(cls[k]);
  for (int k = 0; k < ncls; ++k) {
    const long long most = (cls[k].nx + kSlabTile - 1) / kSlabTile;
    const long long parts = rows > 0 ? (8 * blocks + rows - 1) / rows : 1;
    cls[k].parts = (int)(parts < 1 ? 1 : parts < most ? parts : most);
    cls[k].item0 = items;
    items += rows_of(cls[k]) * cls[k].parts;
  }
  return items;
}

}  // namespace spi
