// Geometry of the column insertion (slab.cuh), free of CUDA so that a CPU
// test can compile it.
//
// A central slice of radius NX through the 3D grid is a plane
// w = SU u + SV v over the two grid axes (u, v) other than the axis w its
// normal is longest along, so |SU|, |SV| <= 1.  The tap of pixel p on voxel k
// is nonzero only when |p - k| < 1.8 on all three axes (the table is zero
// from 1.8 on), so voxel column (u, v) meets the pixels of one parallelogram
// of the slice, all of its voxels lie in |w - (SU u + SV v)| < 1.8 (1 + |SU|
// + |SV|), and every voxel of the slice belongs to exactly one column.
//
// The slice is taken as the full disc of pixels (I, J): pixel -p is the
// Friedel mate of p (conjugate value).  ONELINE (oneline.f:38-200) inserts
// the one of the two with x >= 0 (the canonical one) and sends its taps with
// x < 0 to the reflected point with the conjugate value; that is the tap of
// the mate on the reflected voxel, with the same weight.  So a voxel with
// x > 0 takes the taps of every pixel of the disc, a voxel with x = 0 those
// of the canonical pixels, and only the origin, its own mate, needs its
// reflected taps added apart.
#pragma once

#ifdef __CUDACC__
#define SLAB_HD __host__ __device__ __forceinline__
#else
#define SLAB_HD inline
#endif

#include <cmath>
#include <cstring>

namespace spi {

// single-precision operations rounded one by one (the host compiles this
// with contraction off)
#ifdef __CUDA_ARCH__
SLAB_HD float sl_mul(float a, float b) { return __fmul_rn(a, b); }
SLAB_HD float sl_add(float a, float b) { return __fadd_rn(a, b); }
SLAB_HD float sl_sub(float a, float b) { return __fsub_rn(a, b); }
#else
SLAB_HD float sl_mul(float a, float b) { return a * b; }
SLAB_HD float sl_add(float a, float b) { return a + b; }
SLAB_HD float sl_sub(float a, float b) { return a - b; }
#endif
#ifdef __CUDA_ARCH__
SLAB_HD int sl_bits(float a) { return __float_as_int(a); }
#else
SLAB_HD int sl_bits(float a) { int i; memcpy(&i, &a, 4); return i; }
#endif
// Conversions by the addition of 2^23 (+ 2^22 for signed values), which
// leaves the integer in the low bits of the sum.  floor and ceil for |a| <
// 2^21, and Fortran's NINT (half away from zero) for 0 <= a < 2^22 as
// floor(a + 1/2) with both additions rounded down: a + 1/2 rounded down
// keeps its floor, which rounding to nearest would not (0.49999997).
#ifdef __CUDA_ARCH__
SLAB_HD float sl_add_down(float a, float b) { return __fadd_rd(a, b); }
#else
inline float sl_add_down(float a, float b) {
  const double x = a, y = b, s = x + y, z = s - x;
  const double rest = (x - (s - z)) + (y - z);   // a + b = s + rest exactly
  const float r = (float)s;
  return (double)r > s || ((double)r == s && rest < 0.0) ? nextafterf(r, -INFINITY) : r;
}
#endif
SLAB_HD int slab_floor(float a) { return sl_bits(sl_add_down(a, 12582912.0f)) - 0x4b400000; }
SLAB_HD int slab_ceil(float a) { return -slab_floor(-a); }
SLAB_HD int slab_nint(float a) { return sl_bits(sl_add_down(sl_add_down(a, 0.5f), 8388608.0f)) - 0x4b000000; }
SLAB_HD int sl_min(int a, int b) { return a < b ? a : b; }
SLAB_HD int sl_max(int a, int b) { return a > b ? a : b; }

constexpr int kSlabTile = 16;   // columns of a tile along u and along v
// Radius of the taps with a margin far above the coordinates' rounding
// (about 1e-4 at |p| = 512): candidates beyond 1.8 get weight zero.
constexpr float kSlabR = 1.81f;
// Rows and pixels of a tile: the tile grown by kSlabR is a square of side s =
// 15 + 2 * 1.81 = 18.62, its preimage a parallelogram of area s^2 / |n_w| <=
// s^2 sqrt(3) = 600.6 whose half perimeter is at most s sqrt(2) sqrt(1 +
// n_w^2) / |n_w| <= 52.7, so it holds at most 600.6 + 52.7 + 1 = 654 lattice
// points (a convex region holds at most area + perimeter / 2 + 1), on at most
// s sqrt(2) sqrt(3) + 1 = 47 rows.
constexpr int kSlabRows = 48, kSlabPix = 656;

// Entries of a table kept in shared memory: a table kb_window4_ok accepts is
// zero from floor(1.805 FLTB) = 3,007 on, which is also why columns within
// kSlabR of a pixel hold all of its taps.  Looking a pixel up for the columns
// of a block reaches distances of 1.81 + 1 and a rounding below 0.001, entry
// 4,685, so with zeros up to there no index needs a bound.
constexpr int kSlabTab = 4736;

struct SlabFrame {
  int d;                 // axis w: 0 x, 1 y, 2 z; (u, v) = (y, z), (x, z), (x, y)
  float au, av, aw;      // pixel (I, J) lies at u = I au + J bu, v = I av + J bv, w = I aw + J bw
  float bu, bv, bw;
  float idet;            // 1 / (au bv - av bu)
  float su, sv;          // w = su u + sv v
  float h;               // half height of a column: |w - (su u + sv v)| < h
  float iau, iav;        // 1 / au, 1 / av (or a huge number)
};

// Are DM(1:3) and DM(4:6) = dm the unit vectors of a rotation?  An angle that is
// not finite makes them NaN (CANG); such a slice has no taps, and its
// coordinates must not become indices.
SLAB_HD bool slab_rotation(const float* dm) {
  const float a = dm[0] * dm[0] + dm[1] * dm[1] + dm[2] * dm[2], b = dm[3] * dm[3] + dm[4] * dm[4] + dm[5] * dm[5];
  return a > 0.5f && a < 1.5f && b > 0.5f && b < 1.5f;   // false for NaN
}

// The frame of a slice with DM(1:6) = dm; false when they are not a rotation's,
// in which case the slice has no taps.
SLAB_HD bool slab_frame(const float* dm, SlabFrame& f) {
  if (!slab_rotation(dm)) return false;
  const float n0 = dm[1] * dm[5] - dm[2] * dm[4], n1 = dm[2] * dm[3] - dm[0] * dm[5], n2 = dm[0] * dm[4] - dm[1] * dm[3];
  const float m0 = fabsf(n0), m1 = fabsf(n1), m2 = fabsf(n2);
  f.d = (m2 >= m0 && m2 >= m1) ? 2 : (m1 >= m0 ? 1 : 0);
  const float nd = f.d == 2 ? n2 : f.d == 1 ? -n1 : n0;
  if (!(fabsf(nd) > 0.5f && fabsf(nd) < 1.5f)) return false;
  if (f.d == 2) { f.au = dm[0]; f.av = dm[1]; f.aw = dm[2]; f.bu = dm[3]; f.bv = dm[4]; f.bw = dm[5]; }
  else if (f.d == 1) { f.au = dm[0]; f.av = dm[2]; f.aw = dm[1]; f.bu = dm[3]; f.bv = dm[5]; f.bw = dm[4]; }
  else { f.au = dm[1]; f.av = dm[2]; f.aw = dm[0]; f.bu = dm[4]; f.bv = dm[5]; f.bw = dm[3]; }
  f.idet = 1.0f / nd;
  f.su = (f.bv * f.aw - f.av * f.bw) * f.idet;
  f.sv = (f.au * f.bw - f.bu * f.aw) * f.idet;
  f.h = kSlabR * (1.0f + fabsf(f.su) + fabsf(f.sv)) + 0.01f;
  f.iau = 1.0f / (fabsf(f.au) > 1e-9f ? f.au : 1e-9f);
  f.iav = 1.0f / (fabsf(f.av) > 1e-9f ? f.av : 1e-9f);
  return true;
}

// Banks of four voxels a column of this frame needs: its voxels are at most
// ceil(2 h) consecutive ones, so 8 (2 banks) while h <= 4, else 12 (h < 5.45).
SLAB_HD int slab_banks(const SlabFrame& f) { return f.h <= 4.0f ? 2 : 3; }

// Can columns (u0.., v0..) of a tile meet the disc of radius nx (and x >= 0)?
SLAB_HD bool slab_tile_live(const SlabFrame& f, int u0, int v0, int nx) {
  const float c = 0.5f * (kSlabTile - 1), e = c + kSlabR;
  const float uc = (float)u0 + c, vc = (float)v0 + c;
  const float ic = (uc * f.bv - vc * f.bu) * f.idet, jc = (vc * f.au - uc * f.av) * f.idet;
  const float ri = e * (fabsf(f.bu) + fabsf(f.bv)) * fabsf(f.idet), rj = e * (fabsf(f.au) + fabsf(f.av)) * fabsf(f.idet);
  // nearest point of the preimage's bounding box to the origin
  const float di = fmaxf(0.0f, fabsf(ic) - ri), dj = fmaxf(0.0f, fabsf(jc) - rj);
  if (di * di + dj * dj > (float)nx * (float)nx) return false;
  if (f.d == 0 && f.su * uc + f.sv * vc + e * (fabsf(f.su) + fabsf(f.sv)) < -2.0f) return false;
  return true;
}

// Pixel rows J = jlo .. jlo + nrows - 1 that reach the tile
SLAB_HD void slab_tile_rows(const SlabFrame& f, int u0, int v0, int nx, int& jlo, int& nrows) {
  const float c = 0.5f * (kSlabTile - 1), e = c + kSlabR;
  const float uc = (float)u0 + c, vc = (float)v0 + c;
  const float jc = (vc * f.au - uc * f.av) * f.idet, rj = e * (fabsf(f.au) + fabsf(f.av)) * fabsf(f.idet);
  jlo = sl_max(slab_ceil(jc - rj), -(nx - 1));
  nrows = sl_min(sl_min(slab_floor(jc + rj), nx - 1) - jlo + 1, kSlabRows);
  if (nrows < 0) nrows = 0;
}

// Pixels lo .. hi of row J (reals) that reach columns u in [uc - eu, uc + eu],
// v in [vc - ev, vc + ev]
SLAB_HD void slab_span(const SlabFrame& f, float uc, float vc, float eu, float ev, int J, float& lo, float& hi) {
  const float fj = (float)J;
  const float cu = (uc - fj * f.bu) * f.iau, cv = (vc - fj * f.bv) * f.iav;
  const float hu = eu * fabsf(f.iau), hv = ev * fabsf(f.iav);
  lo = fmaxf(cu - hu, cv - hv);
  hi = fminf(cu + hu, cv + hv);
}

// Pixels lo .. hi of row J that reach the tile; pixels beyond the disc among
// them are staged as reaching nothing
SLAB_HD void slab_tile_span(const SlabFrame& f, int u0, int v0, int nx, int J, int& lo, int& hi) {
  const float c = 0.5f * (kSlabTile - 1), e = c + kSlabR;
  float fl, fh;
  slab_span(f, (float)u0 + c, (float)v0 + c, e, e, J, fl, fh);
  lo = slab_ceil(fmaxf(fl, (float)(1 - nx)));
  hi = slab_floor(fminf(fh, (float)(nx - 1)));
}

// Rows r0 .. r1 of a tile (row r holds J = jlo + r, r < nrows) that reach
// the nu x nv block of columns from (u, v) on
SLAB_HD void slab_block_rows(const SlabFrame& f, float u, float v, int nu, int nv, int jlo, int nrows, int& r0, int& r1) {
  const float eu = kSlabR + 0.5f * (float)(nu - 1), uc = u + 0.5f * (float)(nu - 1);
  const float ev = kSlabR + 0.5f * (float)(nv - 1), vc = v + 0.5f * (float)(nv - 1);
  const float jc = (vc * f.au - uc * f.av) * f.idet, rj = (ev * fabsf(f.au) + eu * fabsf(f.av)) * fabsf(f.idet);
  r0 = sl_max(slab_ceil(jc - rj) - jlo, 0);
  r1 = sl_min(slab_floor(jc + rj) - jlo, nrows - 1);
}

// first voxel of column (u, v)
SLAB_HD int slab_col_base(const SlabFrame& f, float u, float v) { return slab_ceil(f.su * u + f.sv * v - f.h); }

// Pixel p = (I, J) of the full disc at (u, v, w), rounded as ONELINE rounds
// its mate's coordinates or its own (they differ by the sign alone).
struct SlabPix {
  float u, v, w;
  bool rep;     // the stored one of p, -p: I > 0, or I = 0 and J >= 0
  bool canon;   // the one that ONELINE inserts, with x >= 0
};
SLAB_HD SlabPix slab_pixel(const SlabFrame& f, int I, int J) {
  const float fi = (float)I, fj = (float)J;
  SlabPix p;
  p.u = sl_add(sl_mul(fi, f.au), sl_mul(fj, f.bu));
  p.v = sl_add(sl_mul(fi, f.av), sl_mul(fj, f.bv));
  p.w = sl_add(sl_mul(fi, f.aw), sl_mul(fj, f.bw));
  p.rep = I > 0 || (I == 0 && J >= 0);
  const float x = f.d == 0 ? p.w : p.u;
  p.canon = p.rep ? !(x < 0.0f) : x > 0.0f;   // ONELINE flips the stored one when its x is negative
  return p;
}
// Is p inside the disc and its canonical form within ONELINE's bounds on the
// nearest voxel?  Pixels 6 inside the edge always are.
SLAB_HD bool slab_inside(const SlabFrame& f, const SlabPix& p, int I, int J, int nx) {
  const int r2 = I * I + J * J;
  if (nx > 6 && r2 <= (nx - 6) * (nx - 6)) return true;
  if (r2 >= nx * nx) return false;
  const float fn = (float)(2 * nx), sg = p.canon ? 1.0f : -1.0f;
  const int iu = slab_floor(sl_add(sl_add(sg * p.u, 0.5f), fn)) - 2 * nx;   // IFIX of a positive value
  const int iv = slab_floor(sl_add(sl_add(sg * p.v, 0.5f), fn)) - 2 * nx;
  const int iw = slab_floor(sl_add(sl_add(sg * p.w, 0.5f), fn)) - 2 * nx;
  const int lo = -nx + 4, hi = nx - 3;
  return iu <= hi && iv <= hi && iw <= hi && iv >= lo && (f.d == 0 || iw >= lo) && (f.d != 0 || iu >= lo);
}

// Pixel (I, J), I >= 0, of a slice as the extraction takes it: at (x, y, z),
// flipped where its x was negative; false, and at the origin, when it is outside
// the disc or ONELINE's bounds on the nearest voxel.  (xj, yj, zj) = J DM(4:6).
// Pixels 6 inside the edge are inside without a look, so the slice has to be a
// rotation's (slab_rotation).
SLAB_HD bool slab_extract_pixel(const float* dm, float xj, float yj, float zj, int I, int J, int nx, float& x, float& y,
                                float& z, bool& flip) {
  const float fi = (float)I;
  x = sl_add(sl_mul(fi, dm[0]), xj);
  y = sl_add(sl_mul(fi, dm[1]), yj);
  z = sl_add(sl_mul(fi, dm[2]), zj);
  flip = x < 0.0f;
  if (flip) { x = -x; y = -y; z = -z; }
  const int r2 = I * I + J * J;
  bool ok = !(I == 0 && J < 0);
  if (nx <= 6 || r2 > (nx - 6) * (nx - 6)) {
    const int N = 2 * nx;
    const float fn = (float)N;
    const int ix = slab_floor(sl_add(sl_add(x, 0.5f), fn)) - N, iy = slab_floor(sl_add(sl_add(y, 0.5f), fn)) - N;
    const int iz = slab_floor(sl_add(sl_add(z, 0.5f), fn)) - N;
    ok = ok && r2 < nx * nx && ix <= nx - 3 && iy >= -nx + 4 && iy <= nx - 3 && iz >= -nx + 4 && iz <= nx - 3;
  }
  if (!ok) x = y = z = 0.0f;   // keeps look-ups in range
  return ok;
}

// first of the four voxels along an axis that hold every nonzero tap of
// coordinate c (those nearer than 2)
SLAB_HD int slab_first(float c) { return slab_floor(c) - 1; }

// table index of the tap of coordinate c on voxel k (Fortran NINT), cut at
// `last`, which like every later entry is zero
SLAB_HD int slab_tab_index(float c, int k, float fltb, int last) {
  return sl_min(slab_nint(sl_mul(fabsf(sl_sub(c, (float)k)), fltb)), last);
}

// residue of voxel w in a column of nb banks: w mod 4 nb
SLAB_HD int slab_residue(int w, int nb) {
  if (nb == 2) return w & 7;
  const int r = w % 12;
  return r < 0 ? r + 12 : r;
}

}  // namespace spi
