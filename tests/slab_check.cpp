// CPU check of the column insertion's and the extraction's geometry
// (spider_b200/csrc/slab_geom.h).
//
//   slab_check NX SEED COUNT   ->  two lines per rotation:
//   kind banks columns max_rows max_pixels taps_direct taps_columns bad
// compares, voxel by voxel, the taps that the columns of every tile find with
// ONELINE's own walk over the pixels (restated here from oneline.f:38-200).  The
// columns are walked in the blocks of slab_gather: `columns` = 2 (shallow slices in
// FP32) and 1 (steep slices, and all in FP64; both lines of a steep one).  `bad` counts taps that only one side has or whose three table
// entries differ, taps outside their column's voxel range, look-ups beyond the
// table in shared memory, and tiles over the capacity.
//
//   slab_check extract NX SEED COUNT   ->  bad
// counts look-ups and voxels of the extraction's pixels that are out of range, and
// matrices with an element or angle that is not finite which are taken for a
// rotation's.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <iterator>
#include <random>
#include <tuple>
#include <vector>

#include "../spider_b200/csrc/slab_geom.h"

using namespace spi;

static std::vector<float> g_tab;
static float g_fltb;
static const int kLast = kSlabTab - 1;

// the kernel's look-up, and ONELINE's with Fortran's NINT
static float tap(float c, int k) { return g_tab[slab_tab_index(c, k, g_fltb, kLast)]; }
static float tap_nint(float c, int k) {
  const float v = fabsf(c - (float)k) * g_fltb, f = floorf(v);
  return g_tab[(int)f + (v - f >= 0.5f ? 1 : 0)];
}

// a tap: voxel, pixel of the full disc, bits of its weights along x, y and z
typedef std::tuple<long long, int, uint32_t, uint32_t, uint32_t> Tap;

static long long vox(int x, int y, int z, int nx) {
  const int N = 2 * nx;
  const int iy = y >= 0 ? y : N + y, iz = z >= 0 ? z : N + z;
  return ((long long)iz * N + iy) * (nx + 1) + x;
}

static uint32_t bits(float w) {
  uint32_t b;
  memcpy(&b, &w, 4);
  return b;
}

// ONELINE over the half disc; pixel id of the canonical pixel and its mate
static void direct(const float* dm, int nx, std::vector<Tap>& t) {
  const int N = 2 * nx, W = 2 * nx + 1;
  for (int J = -nx + 1; J <= nx; ++J)
    for (int I = 0; I <= nx; ++I) {
      if (I * I + J * J >= nx * nx || (I == 0 && J < 0)) continue;
      float c[3];
      for (int a = 0; a < 3; ++a) {
        const float p = (float)I * dm[a], q = (float)J * dm[a + 3];
        c[a] = p + q;
      }
      int s = 1;
      if (c[0] < 0) { for (float& v : c) v = -v; s = -1; }
      int k[3];
      for (int a = 0; a < 3; ++a) { const float h = c[a] + 0.5f; k[a] = (int)(h + (float)N) - N; }
      if (!(k[0] <= nx - 3 && k[1] >= -nx + 4 && k[1] <= nx - 3 && k[2] >= -nx + 4 && k[2] <= nx - 3)) continue;
      for (int lz = -2; lz <= 2; ++lz)
        for (int ly = -2; ly <= 2; ++ly)
          for (int lx = -2; lx <= 2; ++lx) {
            const int x = k[0] + lx, y = k[1] + ly, z = k[2] + lz;
            const float wx = tap_nint(c[0], x), wy = tap_nint(c[1], y), wz = tap_nint(c[2], z);
            if (wx * (wy * wz) == 0.0f) continue;
            // pixel that lies where the tap lands: the canonical one, or its mate for a reflected tap
            const int sg = x < 0 ? -s : s;
            const int id = (sg * J + nx) * W + sg * I + nx;
            t.push_back({x < 0 ? vox(-x, -y, -z, nx) : vox(x, y, z, nx), id, bits(wx), bits(wy), bits(wz)});
          }
    }
}

// CANG in REAL (cang.f:44-81)
static void euler(float ps, float th, float ph, float* dm) {
  const float r = 3.14159265358979323846f / 180.0f;
  const float cp = std::cos(ps * r), sp = std::sin(ps * r), ct = std::cos(th * r), st = std::sin(th * r);
  const float cf = std::cos(ph * r), sf = std::sin(ph * r);
  const float m[6] = {cf * ct * cp - sf * sp, sf * ct * cp + cf * sp, -st * cp,
                      -cf * ct * sp - sf * cp, -sf * ct * sp + cf * cp, st * sp};
  memcpy(dm, m, sizeof(m));
}

// The extraction's windows (fs_extract.cuh): four lanes per pixel, 4 x 4 (y, z) voxels each
static int extract(int nx, unsigned seed, int count) {
  const int N = 2 * nx, kExTab = 3336;
  const long long rl = nx + 1, total = rl * N * N;
  const float fltb = 4999.0f / 3.0f, last = 1.8f * fltb;
  std::mt19937 rng(seed);
  std::uniform_real_distribution<float> U(0.0f, 1.0f);
  long long bad = 0;
  for (int q = 0; q < count; ++q) {
    const float d[3] = {q < 4 ? 90.0f * q : 360.0f * U(rng), q < 16 ? 45.0f * (q / 4) : 180.0f * U(rng), q < 8 ? 45.0f : 360.0f * U(rng)};
    float dm[6];
    euler(d[0], d[1], d[2], dm);
    SlabFrame f;
    if (!slab_rotation(dm) || !slab_frame(dm, f)) ++bad;
    for (float v : {NAN, INFINITY, -INFINITY})
      for (int e = 0; e < 9; ++e) {   // an angle, or an element of the matrix
        float b[6], a[3] = {d[0], d[1], d[2]};
        if (e < 3) { a[e] = v; euler(a[0], a[1], a[2], b); }
        else { memcpy(b, dm, sizeof(b)); b[e - 3] = v; }
        if (slab_rotation(b) || slab_frame(b, f)) ++bad;
      }
    for (int J = -nx + 1; J <= nx; ++J)
      for (int I0 = 0; slab_rotation(dm) && I0 <= nx && I0 * I0 + J * J < nx * nx; I0 += 8)
        for (int I = I0; I < I0 + 8; ++I) {
          float c[3];
          bool flip;
          const float fj = (float)J;
          const bool ok = slab_extract_pixel(dm, fj * dm[3], fj * dm[4], fj * dm[5], I, J, nx, c[0], c[1], c[2], flip);
          float t[3][4];
          int first[3];
          for (int a = 0; a < 3; ++a) {
            first[a] = slab_first(c[a]);
            for (int l = 0; l < 4; ++l) {
              const int i = slab_nint(fabsf(c[a] - (float)(first[a] + l)) * fltb);
              if (i < 0 || i >= kExTab) ++bad;
              t[a][l] = (float)i <= last ? 1.0f : 0.0f;
            }
          }
          for (int e = 0; ok && e < 64; ++e) {
            const int l = e & 3, m = (e >> 2) & 3, k = e >> 4, x = first[0] + l;
            if (t[0][l] * t[1][m] * t[2][k] == 0.0f) continue;
            const int y = x < 0 ? -(first[1] + m) : first[1] + m, z = x < 0 ? -(first[2] + k) : first[2] + k;
            const long long i = ((z < 0 ? N + z : z) * (long long)N + (y < 0 ? N + y : y)) * rl + (x < 0 ? -x : x);
            if (i < 0 || i >= total || y < -N || y >= N || (x < 0 ? -x : x) >= nx) ++bad;
          }
        }
  }
  printf("%lld\n", bad);
  return 0;
}

int main(int argc, char** argv) {
  if (argc == 5) return extract(atoi(argv[2]), atoi(argv[3]), atoi(argv[4]));
  const int nx = atoi(argv[1]), count = atoi(argv[3]);
  std::mt19937 rng(atoi(argv[2]));
  // a stand-in for FILLBESSIL's table with its support: nonzero up to 1.8, zero beyond
  g_fltb = 4999.0f / 3.0f;
  g_tab.assign(5000, 0.0f);
  for (int i = 0; i < 5000; ++i)
    if ((float)i / g_fltb <= 1.8f) g_tab[i] = 1.0f + (float)(5000 - i) * 1.37e-4f;
  std::uniform_real_distribution<float> U(0.0f, 1.0f);
  const float mag = 54.735610f;   // acos(1 / sqrt(3))
  for (int q = 0; q < count; ++q) {
    float d[3] = {360.0f * U(rng), 57.29578f * std::acos(1.0f - 2.0f * U(rng)), 360.0f * U(rng)};
    // the rotations where the geometry degenerates come first: axes, diagonals, planes of 45 degrees
    const float sp[12][3] = {{0, 0, 0}, {0, 90, 0}, {0, 90, 90}, {45, 0, 0}, {0, 45, 0}, {45, mag, 45}, {0, 180, 0},
                             {90, 90, 45}, {17.2f, 90, 45}, {180, mag, -45}, {0, mag, 45}, {63, 45, 90}};
    if (q < 12) memcpy(d, sp[q], sizeof(d));
    float dm[6];
    euler(d[0], d[1], d[2], dm);
    std::vector<Tap> A, B;
    direct(dm, nx, A);
    std::sort(A.begin(), A.end());
    SlabFrame f;
    if (!slab_frame(dm, f)) { printf("noframe\n"); continue; }
    const int banks = slab_banks(f), W = 2 * nx + 1;
    const int ntu = f.d == 0 ? (2 * nx + kSlabTile - 1) / kSlabTile : (nx + kSlabTile - 1) / kSlabTile;
    const int ntv = (2 * nx + kSlabTile - 1) / kSlabTile;
    for (int form = 0; form < 2; ++form) {
      const int nc = form == 0 && banks == 2 ? 2 : 1;   // columns along v of a thread's block
      long long bad = 0;
      int rows = 0, pixels = 0;
      B.clear();
      for (int tv = 0; tv < ntv; ++tv)
        for (int tu = 0; tu < ntu; ++tu) {
          const int u0 = (f.d == 0 ? -nx : 0) + kSlabTile * tu, v0 = -nx + kSlabTile * tv;
          if (!slab_tile_live(f, u0, v0, nx)) continue;
          int jlo, nr;
          slab_tile_rows(f, u0, v0, nx, jlo, nr);
          std::vector<int> lo(nr), hi(nr);
          int np = 0;
          for (int r = 0; r < nr; ++r) {
            slab_tile_span(f, u0, v0, nx, jlo + r, lo[r], hi[r]);
            np += hi[r] >= lo[r] ? hi[r] - lo[r] + 1 : 0;
          }
          if (nr > rows) rows = nr;
          if (np > pixels) pixels = np;
          if (nr >= kSlabRows || np > kSlabPix) ++bad;
          for (int du = 0; du < kSlabTile; ++du)
            for (int dv = 0; dv < kSlabTile; dv += nc) {
              int r0, r1;
              const float u = (float)(u0 + du), v = (float)(v0 + dv);
              slab_block_rows(f, u, v, 1, nc, jlo, nr, r0, r1);
              for (int r = r0; r <= r1; ++r) {
                float fl, fh;
                slab_span(f, u, v + 0.5f * (nc - 1), kSlabR, kSlabR + 0.5f * (nc - 1), jlo + r, fl, fh);
                const int i0 = slab_ceil(fmaxf(fl, (float)lo[r])), i1 = slab_floor(fminf(fh, (float)hi[r]));
                for (int I = i0; I <= i1; ++I) {
                  const SlabPix p = slab_pixel(f, I, jlo + r);
                  if (!slab_inside(f, p, I, jlo + r, nx)) continue;
                  const int au = f.d == 0 ? 1 : 0, av = f.d == 2 ? 1 : 2, aw = f.d;
                  float pos[3];
                  pos[au] = p.u;
                  pos[av] = p.v;
                  pos[aw] = p.w;
                  for (int c = 0; c < nc; ++c) {
                    int k[3];
                    k[au] = u0 + du;
                    k[av] = v0 + dv + c;
                    // the kernel's table has no bound on the index
                    if (slab_tab_index(p.u, k[au], g_fltb, 9999) >= kSlabTab || slab_tab_index(p.v, k[av], g_fltb, 9999) >= kSlabTab) ++bad;
                    const int base = slab_col_base(f, (float)k[au], (float)k[av]);
                    for (int l = 0; l < 4; ++l) {
                      k[aw] = slab_first(p.w) + l;
                      const float wx = tap(pos[0], k[0]), wy = tap(pos[1], k[1]), wz = tap(pos[2], k[2]);
                      if (wx * (wy * wz) == 0.0f) continue;
                      if (k[0] < 0 || (k[0] == 0 && !p.canon)) continue;
                      // the residue must give the voxel back
                      const int off = slab_residue(k[aw], banks) - slab_residue(base, banks);
                      if (base + (off < 0 ? off + 4 * banks : off) != k[aw]) ++bad;
                      B.push_back({vox(k[0], k[1], k[2], nx), (jlo + r + nx) * W + I + nx, bits(wx), bits(wy), bits(wz)});
                    }
                  }
                }
              }
            }
        }
      // the origin's reflected taps (it is its own mate)
      for (int y = -1; y <= 1; ++y)
        for (int z = -1; z <= 1; ++z) B.push_back({vox(1, -y, -z, nx), nx * W + nx, bits(tap(0, 1)), bits(tap(0, y)), bits(tap(0, z))});
      std::sort(B.begin(), B.end());
      std::vector<Tap> only;
      std::set_symmetric_difference(A.begin(), A.end(), B.begin(), B.end(), std::back_inserter(only));
      bad += (long long)only.size();
      printf("%d %d %d %d %d %zu %zu %lld\n", f.d, banks, nc, rows, pixels, A.size(), B.size(), bad);
    }
  }
  return 0;
}
