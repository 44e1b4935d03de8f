// higdon.cuh - the Higdon absorbing-boundary recurrence along one edge
// line (Boundary_3d, Boundary.f90:89-184,366-447) for the separate edge
// kernels (batch.cu).
#pragma once

#include <cstdint>

#include "batch.cuh"

namespace swave {

// One half line of the Higdon recurrence with all inputs loaded first:
// the 10 u2 and u1 values from 2 cells inside the innermost output to the
// outermost one, the two u3 values inside it and the 8 coefficients; then
// the 8 outputs in order in registers:
//   u3(i) = -(g1 u3(i+d) + g2 u3(i+2d) + g3 u2(i) + g4 u2(i+d) + g5 u2(i+2d)
//            + g6 u1(i) + g7 u1(i+d) + g8 u1(i+2d))
// summed left to right, d the step towards the interior.
// a and bq are the two u3 values inside the innermost output.
__device__ __forceinline__ void higdon_half(const float *__restrict__ gc, long long cs,
                                            const float *__restrict__ u1,
                                            const float *__restrict__ u2, float *u3,
                                            long long pstart, long long dst, float a, float bq) {
  float c[8], U2[10], U1[10];
#pragma unroll
  for (int q = 0; q < 8; ++q) c[q] = gc[q * cs];
#pragma unroll
  for (int m = 0; m < 10; ++m) {
    const long long pm = pstart - (long long)(m - 2) * dst;   // k = m - 2
    U2[m] = u2[pm];
    U1[m] = u1[pm];
  }
  float out[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    float r = c[0] * a;
    r = r + c[1] * bq;
    r = r + c[2] * U2[k + 2];
    r = r + c[3] * U2[k + 1];
    r = r + c[4] * U2[k];
    r = r + c[5] * U1[k + 2];
    r = r + c[6] * U1[k + 1];
    r = r + c[7] * U1[k];
    out[k] = -r;
    bq = a;
    a = out[k];
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) u3[pstart - (long long)k * dst] = out[k];
}
__device__ __forceinline__ void higdon_half(const float *__restrict__ gc, long long cs,
                                            const float *__restrict__ u1,
                                            const float *__restrict__ u2, float *u3,
                                            long long pstart, long long dst) {
  higdon_half(gc, cs, u1, u2, u3, pstart, dst, u3[pstart + dst], u3[pstart + 2 * dst]);
}

// Output m (0: the innermost) of a half line, from the same operations,
// without storing it.
__device__ __forceinline__ float higdon_val(const float *__restrict__ gc, long long cs,
                                            const float *__restrict__ u1,
                                            const float *__restrict__ u2, long long pstart,
                                            long long dst, float a, float bq, int m) {
  for (int k = 0; k <= m; ++k) {
    const long long p = pstart - (long long)k * dst;
    float r = gc[0] * a;
    r = r + gc[cs] * bq;
    r = r + gc[2 * cs] * u2[p];
    r = r + gc[3 * cs] * u2[p + dst];
    r = r + gc[4 * cs] * u2[p + 2 * dst];
    r = r + gc[5 * cs] * u1[p];
    r = r + gc[6 * cs] * u1[p + dst];
    r = r + gc[7 * cs] * u1[p + 2 * dst];
    bq = a;
    a = -r;
  }
  return a;
}

// One Higdon z half line (Boundary_3d, Boundary.f90:89-184) of column
// (j, k): the top (bottom = false) or bottom 8 cells of u3 from u2 and u1 of
// the column and the two u3 cells inside the edge.
__device__ __forceinline__ void higdon_zline(const ShotDev &S, int j, int k, bool bottom,
                                             const float *u1, const float *u2, float *u3) {
  const Geom &g = S.g;
  const int n2 = g.nmax2 - g.nmin2 + 1, n3 = g.nmax3 - g.nmin3 + 1;
  const long long cs = (long long)n2 * n3;
  const long long l = (long long)(j - g.nmin2) + (long long)n2 * (k - g.nmin3);
  if (bottom) {
    // Bottom half line: the last 10 cells of the padded column, in 8-byte
    // loads and stores when they start on an 8-byte boundary (n1p even).
    const long long pb = g.idx(g.nmax1 - 3, j, k) - 2;   // cell n1p - 10
    const float *gcb = S.gz + l + 8 * cs;
    if (((reinterpret_cast<uintptr_t>(u1 + pb) | reinterpret_cast<uintptr_t>(u2 + pb) |
          reinterpret_cast<uintptr_t>(u3 + pb)) & 7) != 0) {
      higdon_half(gcb, cs, u1, u2, u3, pb + 2, -1);
      return;
    }
    float c[8], col2[10], col1[10];
#pragma unroll
    for (int m = 0; m < 8; ++m) c[m] = gcb[m * cs];
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const float2 a2 = reinterpret_cast<const float2 *>(u2 + pb)[v];
      const float2 a1 = reinterpret_cast<const float2 *>(u1 + pb)[v];
      col2[2 * v] = a2.x; col2[2 * v + 1] = a2.y;
      col1[2 * v] = a1.x; col1[2 * v + 1] = a1.y;
    }
    const float2 t3 = reinterpret_cast<const float2 *>(u3 + pb)[0];   // cells pb, pb + 1
    float a = t3.y, bq = t3.x, out[8];
    // U(m) = cell pb + m, as in higdon_half with dst = -1 and pstart = pb + 2.
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
      float r = c[0] * a;
      r = r + c[1] * bq;
      r = r + c[2] * col2[kk + 2];
      r = r + c[3] * col2[kk + 1];
      r = r + c[4] * col2[kk];
      r = r + c[5] * col1[kk + 2];
      r = r + c[6] * col1[kk + 1];
      r = r + c[7] * col1[kk];
      out[kk] = -r;
      bq = a;
      a = out[kk];
    }
    // out[kk] belongs at cell pb + 2 + kk.
#pragma unroll
    for (int v = 0; v < 4; ++v)
      reinterpret_cast<float2 *>(u3 + pb + 2)[v] = make_float2(out[2 * v], out[2 * v + 1]);
    return;
  }
  // Top half line: its cells are the first 12 of the padded column (the
  // column starts on a 128-byte boundary: ld1 is a multiple of 32), so the
  // inputs come in 16-byte loads and the 8 outputs go out in two 16-byte
  // stores; the arithmetic is higdon_half's.
  const long long cb = g.idx(g.lo1, j, k);   // pstart = cb + 7
  const float *gc = S.gz + l;
  if (((reinterpret_cast<uintptr_t>(u1 + cb) | reinterpret_cast<uintptr_t>(u2 + cb) |
        reinterpret_cast<uintptr_t>(u3 + cb)) & 15) != 0) {
    higdon_half(gc, cs, u1, u2, u3, cb + 7, 1);
    return;
  }
  float c[8], col2[12], col1[12];
#pragma unroll
  for (int m = 0; m < 8; ++m) c[m] = gc[m * cs];
#pragma unroll
  for (int v = 0; v < 3; ++v) {
    const float4 a2 = reinterpret_cast<const float4 *>(u2 + cb)[v];
    const float4 a1 = reinterpret_cast<const float4 *>(u1 + cb)[v];
    col2[4 * v] = a2.x; col2[4 * v + 1] = a2.y; col2[4 * v + 2] = a2.z; col2[4 * v + 3] = a2.w;
    col1[4 * v] = a1.x; col1[4 * v + 1] = a1.y; col1[4 * v + 2] = a1.z; col1[4 * v + 3] = a1.w;
  }
  const float2 t3 = reinterpret_cast<const float2 *>(u3 + cb)[4];   // cells 8, 9
  float a = t3.x, bq = t3.y, out[8];
  // U(m) = column cell 9 - m (m = 0..9), as in higdon_half with dst = 1.
#pragma unroll
  for (int kk = 0; kk < 8; ++kk) {
    float r = c[0] * a;
    r = r + c[1] * bq;
    r = r + c[2] * col2[7 - kk];
    r = r + c[3] * col2[8 - kk];
    r = r + c[4] * col2[9 - kk];
    r = r + c[5] * col1[7 - kk];
    r = r + c[6] * col1[8 - kk];
    r = r + c[7] * col1[9 - kk];
    out[kk] = -r;
    bq = a;
    a = out[kk];
  }
  // out[kk] belongs at cell 7 - kk.
  reinterpret_cast<float4 *>(u3 + cb)[0] = make_float4(out[7], out[6], out[5], out[4]);
  reinterpret_cast<float4 *>(u3 + cb)[1] = make_float4(out[3], out[2], out[1], out[0]);
}

// One Higdon x half line of row i in plane k: the left (right = false) or
// right 8 cells.
__device__ __forceinline__ void higdon_xline(const ShotDev &S, int i, int k, bool right,
                                             const float *u1, const float *u2, float *u3) {
  const Geom &g = S.g;
  const int n1 = g.nmax1 - g.nmin1 + 1, n3 = g.nmax3 - g.nmin3 + 1;
  const long long cs = (long long)n1 * n3;
  const long long l = (long long)(i - g.nmin1) + (long long)n1 * (k - g.nmin3);
  const long long L = g.ld1;
  if (!right) higdon_half(S.gx + l, cs, u1, u2, u3, g.idx(i, g.nmin2 + 3, k), L);
  else higdon_half(S.gx + l + 8 * cs, cs, u1, u2, u3, g.idx(i, g.nmax2 - 3, k), -L);
}

// What the z lines, then the x lines leave in u3 at (i, j, k) (indices from
// 0 over the compute domain; k not among the 4 outer planes), computed from
// cells that no edge line writes: (i, j, k) itself, or up to two z lines and
// an x line over them.
__device__ __noinline__ float higdon_corner(const ShotDev &S, int i, int j, int k,
                                            const float *u1, const float *u2, const float *u3) {
  const Geom &g = S.g;
  const int n1 = g.nmax1 - g.nmin1 + 1, n2 = g.nmax2 - g.nmin2 + 1, n3 = g.nmax3 - g.nmin3 + 1;
  auto zed = [&](int jj) {
    if (i >= 4 && i < n1 - 4) return u3[g.idx(g.nmin1 + i, g.nmin2 + jj, g.nmin3 + k)];
    const bool bot = i >= 4;
    const long long cs = (long long)n2 * n3, dst = bot ? -1 : 1;
    const long long ps =
        g.idx(bot ? g.nmax1 - 3 : g.nmin1 + 3, g.nmin2 + jj, g.nmin3 + k);
    return higdon_val(S.gz + jj + (long long)n2 * k + (bot ? 8 * cs : 0), cs, u1, u2, ps, dst,
                      u3[ps + dst], u3[ps + 2 * dst], 3 - (bot ? n1 - 1 - i : i));
  };
  if (j >= 4 && j < n2 - 4) return zed(j);
  const bool right = j >= 4;
  const long long cs = (long long)n1 * n3, dst = right ? -(long long)g.ld1 : g.ld1;
  return higdon_val(S.gx + i + (long long)n1 * k + (right ? 8 * cs : 0), cs, u1, u2,
                    g.idx(g.nmin1 + i, right ? g.nmax2 - 3 : g.nmin2 + 3, g.nmin3 + k), dst,
                    zed(right ? n2 - 5 : 4), zed(right ? n2 - 6 : 5),
                    3 - (right ? n2 - 1 - j : j));
}

// The 3D edges of a step in one launch, a thread per half line.  The
// reference applies all z lines, then all x lines, then all y lines; a later
// line overwrites the earlier ones' cells in the 4 outer columns or planes
// and starts from two cells that an earlier one may have written.  So here a
// z line of the outer 4 columns or planes, and an x line of the outer
// planes, is left out (no later step reads the padding cells which only they
// wrote, and calls whose receivers or outputs do take the lines in order), and
// a line that starts in a corner forms those two cells itself
// (higdon_corner): the lines are independent.
__device__ __forceinline__ void edges3d(const ShotDev &S, int s, int q) {
  const Geom &g = S.g;
  const int n1 = g.nmax1 - g.nmin1 + 1, n2 = g.nmax2 - g.nmin2 + 1, n3 = g.nmax3 - g.nmin3 + 1;
  const float *u1 = S.f[(s + 2) % 5], *u2 = S.f[(s + 3) % 5];
  float *u3 = S.f[(s + 4) % 5];
  int part = 0, far = 0;
  for (;; ++part) {
    const int n = edge3d_part(g, part);
    if (q < 2 * n) {
      far = q >= n;
      q -= far ? n : 0;
      break;
    }
    q -= 2 * n;
  }
  if (part == 0) {
    const int j = q % (n2 - 8) + 4, k = q / (n2 - 8) + 4;
    if (k < n3 - 4) higdon_zline(S, g.nmin2 + j, g.nmin3 + k, far != 0, u1, u2, u3);
    return;
  }
  // Row and, along x lines, plane (along y lines, column) of the line.
  const int nr = part == 1 || part == 3 ? n1 - 8 : 8;
  const int row = q % nr, o = q / nr;
  const bool inner = part & 1;
  const int i = inner || row >= 4 ? (inner ? row + 4 : n1 - 8 + row) : row;
  if (part <= 2) {
    const int k = o + 4;
    if (k >= n3 - 4) return;
    const long long cs = (long long)n1 * n3, dst = far ? -(long long)g.ld1 : g.ld1;
    const long long ps = g.idx(g.nmin1 + i, far ? g.nmax2 - 3 : g.nmin2 + 3, g.nmin3 + k);
    const float *gc = S.gx + i + (long long)n1 * k + (far ? 8 * cs : 0);
    const float a = inner ? u3[ps + dst] : higdon_corner(S, i, far ? n2 - 5 : 4, k, u1, u2, u3);
    const float b =
        inner ? u3[ps + 2 * dst] : higdon_corner(S, i, far ? n2 - 6 : 5, k, u1, u2, u3);
    higdon_half(gc, cs, u1, u2, u3, ps, dst, a, b);
    return;
  }
  const int j = o;
  if (j >= n2) return;
  const long long P = g.plane();
  const long long cs = (long long)n1 * n2, dst = far ? -P : P;
  const long long ps = g.idx(g.nmin1 + i, g.nmin2 + j, far ? g.nmax3 - 3 : g.nmin3 + 3);
  const float *gc = S.gy + i + (long long)n1 * j + (far ? 8 * cs : 0);
  const bool plain = inner && j >= 4 && j < n2 - 4;
  const float a = plain ? u3[ps + dst] : higdon_corner(S, i, j, far ? n3 - 5 : 4, u1, u2, u3);
  const float b = plain ? u3[ps + 2 * dst] : higdon_corner(S, i, j, far ? n3 - 6 : 5, u1, u2, u3);
  higdon_half(gc, cs, u1, u2, u3, ps, dst, a, b);
}

}  // namespace swave
