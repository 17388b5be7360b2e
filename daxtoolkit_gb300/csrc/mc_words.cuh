// Row-word helpers of the marching-cubes count passes: the eight corner
// windows of a word's cells, their case indices and the packed per-word
// counts (triangles << 16 | crossing edges).
#pragma once
#include <cstdint>

#include "common.cuh"
#include "mc_case.cuh"

namespace daxgb {

struct CornerWords {
  uint32_t a, a1, b, b1, c, c1, d, d1;
};

// Case index of cell q of the word; vertex order v0..v7 =
// (i,j,k) (i+1,j,k) (i+1,j+1,k) (i,j+1,k) and the same at k+1
// (dax/exec/internal/TopologyUniform.h:150-157); bit n = value[n] > iso.
__device__ __forceinline__ int case_of(const CornerWords& w, int q) {
  return (int)(((w.a >> q) & 1u) | (((w.a1 >> q) & 1u) << 1) | (((w.b1 >> q) & 1u) << 2) |
               (((w.b >> q) & 1u) << 3) | (((w.c >> q) & 1u) << 4) | (((w.c1 >> q) & 1u) << 5) |
               (((w.d1 >> q) & 1u) << 6) | (((w.d >> q) & 1u) << 7));
}

// Cells of the word that are neither all-inside nor all-outside.
__device__ __forceinline__ uint32_t active_cells(const CornerWords& w, uint32_t cell_mask) {
  const uint32_t all1 = w.a & w.a1 & w.b & w.b1 & w.c & w.c1 & w.d & w.d1;
  const uint32_t any1 = w.a | w.a1 | w.b | w.b1 | w.c | w.c1 | w.d | w.d1;
  return any1 & ~all1 & cell_mask;
}

// The eight corner words of word m of row r (a, a+x of rows (j..j+1,
// k..k+1)) and the masks that decide which of them are meaningful.
struct WordBits {
  CornerWords w;
  uint32_t pmask, xmask;
  bool hy, hz;
};

template <bool CG = false>
__device__ __forceinline__ WordBits load_word_bits(const Grid& g, const uint32_t* bits, unsigned r,
                                                   int m) {
  WordBits wb;
  int j, k;
  split_row(g, r, j, k);
  wb.hy = j < g.ny - 1;
  wb.hz = k < g.nz - 1;
  const long long dy = g.nx, dz = (long long)g.nx * g.ny;
  const long long pos = (long long)r * g.nx + 32ll * m;
  wb.pmask = low_mask(g.nx - 32 * m);
  wb.xmask = low_mask(g.nx - 1 - 32 * m);
  wb.w = CornerWords{};
  bits_at2<CG>(bits, pos, wb.w.a, wb.w.a1);
  if (wb.hy) bits_at2<CG>(bits, pos + dy, wb.w.b, wb.w.b1);
  if (wb.hz) bits_at2<CG>(bits, pos + dz, wb.w.c, wb.w.c1);
  if (wb.hy && wb.hz) bits_at2<CG>(bits, pos + dy + dz, wb.w.d, wb.w.d1);
  return wb;
}

// Triangles of the cells in `mask`, all 32 at once.  A row of the case table
// triangulates closed polygons on the cell's surface whose corners are its
// sign-change edges, and a polygon of n corners takes n - 2 triangles, so
//     NumFaces = (sign-change edges) - 2 (polygons).
// A cell that is neither all inside nor all outside has one polygon unless a
// face of it is ambiguous (its four edges all change sign) or two opposite
// corners are both cut off by their three edges; only those cells are looked
// up in the table.  (Both facts hold for all 256 rows:
// tests/test_count_words_cpu.py.)  The edges of the others are counted by
// bit-sliced carry-save additions of the twelve edge words.
__device__ __forceinline__ void add3(uint32_t a, uint32_t b, uint32_t c, uint32_t& s, uint32_t& k) {
  s = a ^ b ^ c;
  k = (a & b) | (c & (a | b));
}

__device__ __forceinline__ int word_tris(const CornerWords& w, uint32_t mask,
                                         const unsigned char* nf) {
  const uint32_t x0 = w.a ^ w.a1, x1 = w.b ^ w.b1, x2 = w.c ^ w.c1, x3 = w.d ^ w.d1;
  const uint32_t y0 = w.a ^ w.b, y1 = w.a1 ^ w.b1, y2 = w.c ^ w.d, y3 = w.c1 ^ w.d1;
  const uint32_t z0 = w.a ^ w.c, z1 = w.a1 ^ w.c1, z2 = w.b ^ w.d, z3 = w.b1 ^ w.d1;
  uint32_t odd = (x0 & y1 & x1) | (x2 & y3 & x3);                   // ambiguous z faces
  odd |= (x0 & z1 & x2) | (x1 & z3 & x3);                           // y faces
  odd |= (y0 & z2 & y2) | (y1 & z3 & y3);                           // x faces
  odd |= (x0 & y0 & z0) & (x3 & y3 & z3);                           // opposite corners
  odd |= (x0 & y1 & z1) & (x3 & y2 & z2);
  odd |= (x1 & y0 & z2) & (x2 & y3 & z1);
  odd |= (x1 & y1 & z3) & (x2 & y2 & z0);
  odd &= mask;
  const uint32_t one = active_cells(w, mask) & ~odd;
  uint32_t s0, s1, s2, s3, k0, k1, k2, k3, k4, t0, t1, t2, u0, u1, u2, e1, e2, e3;
  add3(x0, x1, x2, s0, k0);
  add3(x3, y0, y1, s1, k1);
  add3(y2, y3, z0, s2, k2);
  add3(z1, z2, z3, s3, k3);
  add3(s0, s1, s2, t0, k4);
  const uint32_t e0 = t0 ^ s3, k5 = t0 & s3;  // ones
  add3(k0, k1, k2, t1, u0);
  add3(k3, k4, k5, t2, u1);
  e1 = t1 ^ t2;                               // twos
  u2 = t1 & t2;
  add3(u0, u1, u2, e2, e3);                   // fours, eights
  int t = __popc(e0 & one) + 2 * (__popc(e1 & one) - __popc(one)) + 4 * __popc(e2 & one) +
          8 * __popc(e3 & one);
  for (uint32_t u = odd; u; u &= u - 1) t += nf[case_of(w, __ffs(u) - 1)];
  return t;
}

// Counts of one word from its eight corner words.
__device__ __forceinline__ uint32_t packed_counts(const CornerWords& w, bool hy, bool hz,
                                                  uint32_t pmask, uint32_t xmask,
                                                  const unsigned char* nf) {
  int v = __popc((w.a ^ w.a1) & xmask);
  if (hy) v += __popc((w.a ^ w.b) & pmask);
  if (hz) v += __popc((w.a ^ w.c) & pmask);
  int t = 0;
  if (hy && hz && active_cells(w, xmask)) t = word_tris(w, xmask, nf);
  return ((uint32_t)t << 16) | (uint32_t)v;
}

}  // namespace daxgb
