// Column insertion of central slices (ONELINE, oneline.f:38-200) on sm_100a.
// Included by bp.cu after SliceDesc, load_spec and red_add_v4; the geometry
// is in slab_geom.h.
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

#include "slab_geom.h"

namespace spi {

constexpr int kSlabMaxClass = 16;
constexpr int kSlabThreads = kSlabTile * kSlabTile / 2;   // consumers: two columns each, neighbours along v
constexpr int kSlabBlocks = 4;                            // CTAs per SM (96 registers, 50 KB each)

struct SlabClass {
  const void* spec;            // spectra of the class's images in this launch
  const SliceDesc* slices;
  float4* g0;                  // grids the taps go to (half-set 1 and 2)
  float4* g1;
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
  float4* g;                   // grid of its slice
  float fltb;
  int banks;                   // 0: no tile is left
  int u0, v0, jlo, nr, nx, cls;
  int4 rows[kSlabRows];        // {first staged pixel - lo, lo, hi, 0}
};
template <bool BF16>
struct SlabSmem {
  float4 pix[kSlabPix];        // {u, v, Re, Im}
  float4 t[kSlabPix];          // weights along w by residue modulo 4
  int code[kSlabPix];          // slab_masks, kSlabMate
  SlabTile tile[2];
  typename std::conditional<BF16, __nv_bfloat162, float2>::type raw[2][kSlabPix];   // spectrum values
  float tab[kSlabTab];
};

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

// 8 (4) bytes from global to shared memory, asynchronously
__device__ __forceinline__ void slab_copy(float2* dst, const float2* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void slab_copy(__nv_bfloat162* dst, const __nv_bfloat162* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
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
// apart, once per slice.  br, bi: its value.
__device__ __noinline__ void slab_origin(const float* tab, float fltb, float4* __restrict__ G, int nx, float br, float bi) {
  const float w0 = tab[0], w1 = tab[slab_tab_index(0.0f, 1, fltb, kSlabTab - 1)];
  const int N = 2 * nx;
  for (int e = 0; e < 9; ++e) {
    const int y = e % 3 - 1, z = e / 3 - 1;
    const float wg = __fmul_rn(w1, __fmul_rn(y ? w1 : w0, z ? w1 : w0));
    red_add_v4(G + ((size_t)(z < 0 ? N + z : z) * N + (y < 0 ? N + y : y)) * (size_t)(nx + 1) + 1,
               make_float4(__fmul_rn(br, wg), -__fmul_rn(bi, wg), wg, 0.0f));
  }
}

// The taps of a pixel whose value is not finite on the tile's columns, one by
// one: its products with zero weights, which slab_gather forms, would not be zero.
__device__ __noinline__ void slab_direct(const float* tab, const SlabTile& T, const SlabPix& p, float br, float bi) {
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
    red_add_v4(T.g + ((size_t)(z < 0 ? N + z : z) * N + (y < 0 ? N + y : y)) * (size_t)(nx + 1) + x,
               make_float4(__fmul_rn(br, wg), __fmul_rn(bi, wg), 0.0f, 0.0f));
  }
}

// The tile's pixels into the form that slab_gather reads: eight lanes per row
template <int NB, bool BF16>
__device__ __forceinline__ void slab_stage(SlabSmem<BF16>& S, const SlabTile& T, const SlabFrame& f, int buf) {
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
        S.pix[q] = make_float4(p.u, p.v, 0.0f, 0.0f);
        S.t[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        S.code[q] = 0;
        continue;
      }
      // SPIDER forward sign = conjugate of the cuFFT R2C output; conjugated again for a mate
      const float2 sp = slab_float2(S.raw[buf][q]);
      const float bi = p.rep ? -sp.y : sp.y;
      const bool fin = isfinite(sp.x) && isfinite(bi);
      S.pix[q] = make_float4(p.u, p.v, fin ? sp.x : 0.0f, fin ? bi : 0.0f);
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
      S.code[q] = slab_masks<NB>(fw) | (p.canon ? 0 : kSlabMate);
      if (!fin) slab_direct(S.tab, T, p, sp.x, bi);
      if (I == 0 && J == 0 && T.u0 <= 0 && T.u0 + kSlabTile > 0 && T.v0 <= 0 && T.v0 + kSlabTile > 0)
        slab_origin(S.tab, fltb, T.g, nx, sp.x, bi);
    }
  }
}

// Columns (U, V) .. (U, V + NC - 1): walk the pixels that reach them, keep the
// sums by residue in registers (pairs of residues 2 j, 2 j + 1 of Re X, Im X, W),
// and add them to the grid.
template <int NC, int NB, bool BF16>
__device__ __forceinline__ void slab_gather(const SlabSmem<BF16>& S, const SlabTile& T, const SlabFrame& f, int U, int V) {
  const int nx = T.nx, jlo = T.jlo;
  const float fltb = T.fltb, u = (float)U, v = (float)V;
  unsigned long long acc[NC][3][2 * NB];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int e = 0; e < 3; ++e)
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
        slab_fma2(acc[c][2][j], w2, tt[j]);
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
  const int N = 2 * nx;
  const unsigned rl = (unsigned)(nx + 1);
  float4* G = T.g;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int Vc = V + c;
    const int base = slab_col_base(f, u, v + (float)c), res = slab_residue(base, NB);
    const unsigned iv = (unsigned)(Vc >= 0 ? Vc : N + Vc);
    unsigned col, step;   // voxel of the column at w = 0 and the stride along w (grids hold < 2^32 voxels)
    if (f.d == 2) { col = iv * rl + (unsigned)U; step = (unsigned)N * rl; }
    else if (f.d == 1) { col = iv * (unsigned)N * rl + (unsigned)U; step = rl; }
    else { col = (iv * (unsigned)N + (unsigned)(U >= 0 ? U : N + U)) * rl; step = 1u; }
#pragma unroll
    for (int j = 0; j < 2 * NB; ++j) {
      const float2 re = slab_unpack(acc[c][0][j]), im = slab_unpack(acc[c][1][j]), w = slab_unpack(acc[c][2][j]);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float wg = e ? w.y : w.x;
        if (wg == 0.0f) continue;
        int off = 2 * j + e - res;
        if (off < 0) off += 4 * NB;
        int k = base + off;
        if (k < 0) {
          if (f.d == 0) continue;   // x < 0: the mate's taps
          k += N;
        }
        red_add_v4(G + (size_t)(col + (unsigned)k * step), make_float4(e ? re.y : re.x, e ? im.y : im.x, wg, 0.0f));
      }
    }
  }
}

// One tile of one slice, by the consumer warps
template <int NB, bool BF16>
__device__ __forceinline__ void slab_tile(SlabSmem<BF16>& S, const SlabTile& T, int buf) {
  const SlabFrame f = T.f;
  slab_stage<NB, BF16>(S, T, f, buf);
  slab_bar<2>(kSlabThreads);
  // Steep slices (three banks) take a thread's two columns one after the other: as
  // many operations as together, and their sums fit the registers.
  const int U = T.u0 + (threadIdx.x & 15), V = T.v0 + 2 * (threadIdx.x >> 4);
  if (NB == 2) {
    slab_gather<2, NB, BF16>(S, T, f, U, V);
  } else {
#pragma unroll 1
    for (int c = 0; c < 2; ++c) slab_gather<1, NB, BF16>(S, T, f, U, V + c);
  }
}

// A CTA is one producer warp and kSlabThreads consumers.  The producer takes
// work items (a slice's row of tiles along u, or every `parts`-th tile of it
// when a launch has few slices) in slice-major order from one counter and
// prepares tile k + 1 -- its frame, rows and the copies of its spectrum values
// -- while the consumers stage and gather tile k.  The two meet once per tile.
template <bool BF16>
__global__ void __launch_bounds__(kSlabThreads + 32, kSlabBlocks) insert_x4_kernel(const __grid_constant__ SlabArgs P,
                                                                                  unsigned long long* __restrict__ work) {
  extern __shared__ __align__(16) unsigned char slab_raw[];
  SlabSmem<BF16>& S = *reinterpret_cast<SlabSmem<BF16>*>(slab_raw);
  const int tid = threadIdx.x;
  if (tid >= kSlabThreads) {
    const int lane = tid - kSlabThreads;
    using V = typename std::conditional<BF16, __nv_bfloat162, float2>::type;
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
    if (T.banks == 2) slab_tile<2, BF16>(S, T, buf);
    else slab_tile<3, BF16>(S, T, buf);
  }
}

}  // namespace spi
