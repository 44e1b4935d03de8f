// onchip2d.cuh - 2D propagation with the wavefields resident on the chip.
//
// A shot whose padded grid fits into the shared memory of (a share of) the
// device runs all its time steps in one cooperative launch.  The grid is cut
// into tiles, one CTA of 256 threads each; a CTA keeps its tile's four time
// levels in shared memory for the whole launch and only exchanges a 4-cell
// border with its (up to four) neighbours per step.  HBM sees the
// initial and final state, the saved snapshots, the injection terms and the
// receiver cells; no level is streamed per step.
//
// * Exchange: 16-byte packets of two {value, epoch} pairs, each 64-bit half
//   written and read as one relaxed access, into a two-deep inbox of the
//   neighbour: a value carries its own arrival flag, so no fence and no
//   separate flag trip.  A slot is rewritten two steps later, after the
//   neighbour's next packets have shown that it has read it.
// * Order of a step: the cells that border strips and edge lines need, then
//   the Higdon lines of edge tiles, then the packets, then the remaining
//   cells (which hide the packets' flight), the snapshot and receiver cells,
//   then the neighbours' packets.
// * The operations of a point are those of tile2d.cuh, in the same order.
//   The adjoint stencil acts on w = (v*v)*u, so adjoint tiles keep w (two
//   parities, with border) and exchange w instead of u.
// * Injection terms of a chunk of steps are formed before the launch
//   (k_oc_terms); receivers gather after it from the cells the launch saved
//   (k_oc_extract); imaging conditions run after it from the backward
//   snapshots (k_oc_image), reading and writing the image once per launch.
//
// Bound by the per-tile work (shared-memory loads of the stencil and FP32
// issue) for large tiles, by the packets' round trip through L2 for small
// ones.  Two CTAs per SM: one computes while the other waits; one CTA of 512
// threads took 3 % longer, three of 256 or two of 384 (80 registers) 15-25 %,
// 4 x 4 points per work item 9-15 %.  Time per step against the per-step
// kernels (one GB300): 201 x 401 modelling 12.4 -> 2.0 us, 301 x 901 RTM
// 9.2 -> 2.7 us (mean of both passes).  Forward steps of one, two, three and
// four 301 x 901 shots at a time take 2.5, 3.2, 4.1 and 4.9 us: 1.5 us of
// latency (packets, edge lines, barriers) and 0.85 per shot.
#pragma once

#include "batch.cuh"
#include "f32x2.cuh"

namespace swave {

constexpr int OC_THREADS = 256;
constexpr int OC_PER_SM = 2;   // resident CTAs
constexpr int NC = 2;          // columns of a work item
// Bounded wait: polls of one packet (about 0.7 us each) before giving up.
constexpr int OC_WAIT_LIMIT = 1 << 21;
// Smallest tile: 4 row groups and 6 column pairs, so that each edge line
// (10 cells) and each border strip lies in one tile.
constexpr int OC_MIN_GROUPS = 4, OC_MIN_PAIRS = 6;

struct OcShot {
  // Injection terms of the launch's steps, [step][m][column][row]: the m-th
  // term of each cell of the shot's box (its rows widened to whole groups of
  // 4 from padded row row0), -0 where a cell has fewer.
  const float *terms;
  int nent;             // terms per step: M * ncol * nrow
  int M, ncol, nrow, row0;
  float *tape;          // [step][ncell] receiver cells
  int ncell;
  const int *cells;     // per receiver cell: column << 16 | row within its tile
  float *bsnap;         // backward snapshots of the launch's imaging steps
};

struct OcArgs {
  const ShotDev *shots;
  const OcShot *oc;
  const OcTile *tiles;
  ulonglong2 *inbox;     // [cta][parity][side][cap]
  int cap;
  int s0, s1;            // steps of the launch (a shot stops at its own last step)
  unsigned epoch0;       // packets of step s carry epoch0 + (s - s0) + 1
  int rigid;
  int pad;               // see oc_strides
  int *err;
};

// Column strides: 16-byte aligned, an odd number of 16-byte units, so that
// neighbouring columns start in different banks.
__host__ __device__ inline int oc_stride(int rows) {
  const int q = (rows + 3) / 4;
  return 4 * (q | 1);
}
// Strides of the arrays with (hs) and without (cs) the border.  With pad
// they are the same modulo 4 units: the order of the work items that keeps
// the accesses of 8 lanes in different banks in one array then does so in
// the others.  Without room for it (2 or 4 units per column of some arrays)
// the bordered arrays alone are free of conflicts.
__host__ __device__ inline void oc_strides(int TZ, bool adj, bool pad, int *hs, int *cs) {
  *hs = oc_stride(TZ + 8);
  *cs = oc_stride(TZ);
  if (pad && adj) *hs = *cs + 16;
  if (pad && !adj) *cs = *hs;
}
// Dynamic shared memory of a tile: its levels (and velocity, vsm) and work items, and with them
// its injection terms (two parities) and edge lines (coefficients, velocity).
__host__ __device__ inline size_t oc_smem_bytes(const OcTile &t, bool adj, bool vsm, bool pad) {
  int hs, cs;
  oc_strides(t.TZ, adj, pad, &hs, &cs);
  const size_t h = (size_t)hs * (t.TX + 8), c = (size_t)cs * t.TX;
  const size_t items = (size_t)(t.TZ / 4) * (t.TX / 2);
  return 4 * ((adj ? 4 * c + 2 * h : 4 * h) + (vsm ? c : 0) + items) + 16 +
         8 * (size_t)t.nterm + (adj ? 64 : 32) * (size_t)t.nline;
}

__device__ __forceinline__ void oc_put(ulonglong2 *p, float a, float b, unsigned epoch) {
  const unsigned long long e = (unsigned long long)epoch << 32;
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p),
               "l"(e | __float_as_uint(a)), "l"(e | __float_as_uint(b))
               : "memory");
}
__device__ __forceinline__ ulonglong2 oc_get(const ulonglong2 *p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];"
               : "=l"(v.x), "=l"(v.y)
               : "l"(p)
               : "memory");
  return v;
}

// 16-byte asynchronous global -> shared copy.
__device__ __forceinline__ void oc_copy16(float *dst, const float *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ float4 oc_ld4(const float *p) {
  return *reinterpret_cast<const float4 *>(p);
}
__device__ __forceinline__ void oc_st4(float *p, P2 a, P2 b) {
  *reinterpret_cast<float4 *>(p) = make_float4(a.x, a.y, b.x, b.y);
}

// Higdon recurrence of one half line (Boundary_3d, Boundary.f90:89-184); the
// arguments are those of t2_higdon8 (tile2d.cuh).
__device__ __forceinline__ void oc_higdon8(const float c[8], const float U2[10],
                                           const float U1[10], float a, float bq, float out[8]) {
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
}

// Snapshot slot written at time sample it of a shot's phase: the forward
// snapshot (extract_wave), or the launch's buffer for the imaging that
// k_oc_image does; null when the step saves nothing.
__device__ __forceinline__ float *oc_save_slot(const ShotDev &S, const OcShot &O, int it, int s0,
                                               long long nphys) {
  if (it % S.snapi != 0) return nullptr;
  const int cnt = S.tstep > 0 ? it / S.snapi - (S.tcnt - 1) / S.snapi
                              : S.tcnt / S.snapi - (it - 1) / S.snapi;
  if (S.extract_wave) return cnt <= S.ntsnap ? S.wave + (long long)(cnt - 1) * nphys : nullptr;
  if (O.bsnap && S.ntsnap - cnt + 1 >= 1)
    return O.bsnap + (long long)((S.tmin - s0) / S.snapi - it / S.snapi) * nphys;
  return nullptr;
}

template <bool ADJ, bool VSM>
__global__ void __launch_bounds__(OC_THREADS, OC_PER_SM) k_onchip2d(OcArgs A) {
  extern __shared__ __align__(16) float oc_sm[];
  __shared__ int n_items[2], n_class[16], n_rank[16];
  __shared__ volatile int abort_flag;
  __shared__ ShotDev S;
  const OcTile T = A.tiles[blockIdx.x];
  const OcShot O = A.oc[T.shot];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // The shot's descriptor in shared memory: the packets' memory clobbers
  // would have it re-read from global memory every step.
  static_assert(sizeof(ShotDev) % 4 == 0, "descriptor words");
  for (int q = tid; q < (int)(sizeof(ShotDev) / 4); q += OC_THREADS)
    reinterpret_cast<int *>(&S)[q] = reinterpret_cast<const int *>(A.shots + T.shot)[q];
  __syncthreads();
  const int n1p = S.g.n1p, n2p = S.g.n2p, ld1 = S.g.ld1;
  const int TZ = T.TZ, TX = T.TX, r0 = T.r0, c0 = T.c0;
  int HS, CS;
  oc_strides(TZ, ADJ, A.pad != 0, &HS, &CS);
  const int hsz = HS * (TX + 8);
  // Levels: forward tiles keep them with the border (the stencil reads u2),
  // adjoint tiles without it (the stencil reads w).
  const int US = ADJ ? CS : HS, UO = ADJ ? 0 : 4 * HS + 4, usz = ADJ ? CS * TX : hsz;
  float *const lev0 = oc_sm;
  float *const w0 = oc_sm + 4 * usz;
  float *const V = w0 + (ADJ ? 2 * hsz : 0);   // its square, if there is room (VSM)
  int *const items = reinterpret_cast<int *>(V + (VSM ? CS * TX : 0));
  const bool hig = !A.rigid;
  const int se = min(A.s1, S.nsteps);   // this shot's steps: [s0, se)
  if (A.s0 >= se) return;               // uniform over the shot's CTAs
  const int NG = TZ / 4, NP = TX / NC;

  // ---- state into shared memory ----
  {
    const int ng = NG + 2;
    for (int q = tid; q < ng * (TX + 8); q += OC_THREADS) {
      const int c = q / ng - 4, g = q % ng - 1;   // column and row group, border included
      const int R = r0 + 4 * g, C = c0 + c;
      const bool in = R >= 0 && R < ld1 && C >= 0 && C < n2p;
      const bool core = g >= 0 && g < NG && c >= 0 && c < TX;
      const long long off = (long long)R + (long long)ld1 * C;
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      float4 v2 = zero;
      if (in && (ADJ || (VSM && core))) {
        const float4 v = oc_ld4(S.vel + off);
        v2 = make_float4(v.x * v.x, v.y * v.y, v.z * v.z, v.w * v.w);
        if (VSM && core) *reinterpret_cast<float4 *>(V + c * CS + 4 * g) = v2;
      }
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        const float4 u = in ? oc_ld4(S.f[(A.s0 + l) % 5] + off) : zero;
        if (!ADJ || core)
          *reinterpret_cast<float4 *>(lev0 + ((A.s0 + l) & 3) * usz + UO + c * US + 4 * g) = u;
        if (ADJ && l == 3) {
          float *w = w0 + (c + 4) * HS + 4 * g + 4;
          *reinterpret_cast<float4 *>(w + (A.s0 & 1) * hsz) =
              make_float4(v2.x * u.x, v2.y * u.y, v2.z * u.z, v2.w * u.w);
          // Cells no step writes (the padding of the rigid mode) stay zero.
          *reinterpret_cast<float4 *>(w + ((A.s0 + 1) & 1) * hsz) = zero;
        }
      }
    }
  }
  // ---- work items: 4 rows x NC columns, those that the border strips and
  // the edge lines need first ----
  // Rows and columns of the 8-cell Higdon zones are written by the edge
  // lines alone; of the x zones only the rows the z lines start from (two
  // beyond each z zone) are computed, in the first list.
  const int zlo = hig ? 8 : 4, zhi = hig ? n1p - 9 : n1p - 5;
  // Within a list they go round the 8 classes of (row group + column offset
  // in 16-byte units) modulo 8, so that a quarter warp's 16-byte accesses
  // meet 32 different banks whatever the stride and the holes of the lists.
  // In order of rows the items of a quarter warp took 2.6 passes of the
  // shared-memory pipe per access on average, which bound the step.
  if (warp == 0) {
    if (lane < 16) n_class[lane] = n_rank[lane] = 0;
    __syncwarp();
    int n0 = 0;
    for (int pass = 0; pass < 2; ++pass) {
      for (int q0 = 0; q0 < NG * NP; q0 += 32) {
        const int q = q0 + lane, p = q / NG, g = q % NG;
        const int R = r0 + 4 * g, C = c0 + NC * p;
        bool use = q < NG * NP && R + 3 >= zlo && R <= zhi;
        const bool zadj = hig && ((R <= 9 && R + 3 >= 8) || (R <= n1p - 9 && R + 3 >= n1p - 10));
        int f = 0;
#pragma unroll
        for (int h = 0; h < NC; ++h) {
          const int c = C + h;
          if (c >= 4 && c <= n2p - 5 && (!hig || zadj || (c >= 8 && c <= n2p - 9))) f |= 1 << h;
        }
        use = use && f != 0;
        const bool first = zadj || (g == 0 && T.nb[2] >= 0) || (g == NG - 1 && T.nb[3] >= 0) ||
                           (NC * p < 4 && T.nb[0] >= 0) ||
                           (NC * p >= TX - 4 && T.nb[1] >= 0) ||
                           (hig && ((C <= 9 && C + NC > 8) || (C <= n2p - 9 && C + NC > n2p - 10)));
        const int cls = (g + p * (NC * HS / 4)) & 7;
        const int key = use ? cls + (first ? 0 : 8) : -1;
        const unsigned m = __match_any_sync(0xffffffffu, key);
        const int before = __popc(m & ((1u << lane) - 1));
        int *const count = pass ? n_rank : n_class;
        if (pass && use) {
          // The items of the list that come earlier in the round.
          const int rank = n_rank[key] + before;
          int pos = first ? 0 : n0;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            pos += min(n_class[(key & 8) + k], rank + (k < cls ? 1 : 0));
          items[pos] = g | (p << 8) | (f << 16);
        }
        __syncwarp();
        if (use && before == 0) count[key] += __popc(m);
        __syncwarp();
      }
      if (pass == 0) {
        int n = 0;
        for (int k = 0; k < 16; ++k) {
          n += n_class[k];
          if (k == 7) n0 = n;
        }
        if (lane == 0) {
          n_items[0] = n0;
          n_items[1] = n;
        }
      }
    }
    if (lane == 0) abort_flag = 0;
  }
  __syncthreads();
  const int n_all = n_items[1];
  const int n_first = min(n_all, (n_items[0] + OC_THREADS - 1) / OC_THREADS * OC_THREADS);

  const float c0z = S.c.c0z, c1z = S.c.c1z, c2z = S.c.c2z, c3z = S.c.c3z, c4z = S.c.c4z;
  const float cx[5] = {S.c.c0x, S.c.c1x, S.c.c2x, S.c.c3x, S.c.c4x};
  const float k12 = S.k12;
  const P2 div11 = p2s(S.div11);
  const long long nphys = (long long)S.g.nz * S.g.nx;
  // Injection box: whole row groups, columns jb0..jb1.  The terms of the
  // tile's columns come from shared memory (nterm > 0: copied one step ahead,
  // two parities) or from global memory.
  const int jb0 = S.bj0 - S.g.lo2, jb1 = jb0 + O.ncol - 1;
  const bool inj_tile = S.inj_on && r0 < O.row0 + O.nrow && r0 + TZ > O.row0 && c0 <= jb1 &&
                        c0 + TX - 1 >= jb0;
  const bool inj_sm = inj_tile && T.nterm > 0;
  // First column and row, columns, rows (whole groups) and strides of the terms.
  const int joff = inj_sm ? max(c0, jb0) : jb0, ioff = inj_sm ? max(r0, O.row0) : O.row0;
  const int tcol = inj_sm ? min(c0 + TX - 1, jb1) - joff + 1 : O.ncol;
  const int trow = inj_sm ? min(r0 + TZ, O.row0 + O.nrow) - ioff : O.nrow;
  float *const sterm = reinterpret_cast<float *>(items + (NG * NP + 3) / 4 * 4);
  auto fetch_terms = [&](int s) {   // asynchronously, of step s
    float *dst = sterm + (s & 1) * T.nterm;
    const float *src = O.terms + (long long)(s - A.s0) * O.nent + (joff - jb0) * O.nrow +
                       (ioff - O.row0);
    const int ng = trow / 4, n = O.M * tcol * ng;
    for (int q = tid; q < n; q += OC_THREADS) {
      const int mc = q / ng, g = q - mc * ng, m = mc / tcol, c = mc - m * tcol;
      oc_copy16(dst + 4 * q, src + ((long long)m * O.ncol + c) * O.nrow + 4 * g);
    }
  };
  if (inj_sm) {
    fetch_terms(A.s0);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
  }
  const bool top = r0 == 0, bottom = r0 + TZ >= n1p, left = c0 == 0, right = c0 + TX >= n2p;
  const bool edge = hig && (top || bottom || left || right);
  // Edge lines: z lines first (one per column, top then bottom), then x lines
  // (one per row, left then right); [m][line] coefficients and, adjoint, v^2
  // of the 8 cells, innermost first.
  const int nzl = hig ? (top ? TX : 0) + (bottom ? TX : 0) : 0,
            nxl = hig ? (left ? TZ : 0) + (right ? TZ : 0) : 0, nline = nzl + nxl;
  float *const ecoef = sterm + 2 * T.nterm;
  float *const evel = ecoef + 8 * nline;
  for (int q = tid; q < nline; q += OC_THREADS) {
    const bool zl = q < nzl;
    const int k = zl ? q : q - nzl, len = zl ? TX : TZ, n1 = n1p - 8, n2 = n2p - 8;
    const bool far = zl ? !top || k >= TX : !left || k >= TZ;   // bottom, right
    const int x = far && (zl ? top : left) ? k - len : k;       // column or row of the tile
    const int G = (zl ? c0 : r0) + x;
    if (G < 4 || G > (zl ? n2p : n1p) - 5) continue;
    const int nl = zl ? n2 : n1, dir = far ? -1 : 1, p = far ? (zl ? n1p : n2p) - 8 : 7;
    const float *gc = (zl ? S.gz : S.gx) + (G - 4) + (far ? 8 * nl : 0);
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      ecoef[m * nline + q] = gc[m * nl];
      if (ADJ) {
        const int e = p - m * dir;
        const float v = S.vel[zl ? e + (long long)ld1 * G : G + (long long)ld1 * e];
        evel[m * nline + q] = v * v;
      }
    }
  }
  __syncthreads();
  const bool born = !ADJ && S.imaging == 4 && S.tstep > 0;   // ADJ: oc_eligible
  const bool saves = S.extract_wave || O.bsnap;
  const int tstep = S.tstep, snapi = S.snapi, nz = S.g.nz;
  const int nsave = min(3, snapi);   // steps a snapshot's saving is spread over
  int spart = 0;                     // parts of it saved so far
  // The tile's physical cells: first row and column, rows and columns.
  const int sra = max(0, 1 - S.g.lo1 - r0), snr = min(TZ, nz + 1 - S.g.lo1 - r0) - sra;
  const int sca = max(0, 1 - S.g.lo2 - c0), snc = min(TX, S.g.nx + 1 - S.g.lo2 - c0) - sca;
  const float *const vel0 = S.vel + (long long)ld1 * c0 + r0;
  float *sdst = nullptr;
  int it = S.tmin + A.s0 * tstep, itm = it % snapi;
  // Packets per side and in all; the first two of a thread are kept decoded
  // (offset within the operand, slot of the neighbour's or the own inbox).
  const int npx = 2 * TZ, npz = 2 * TX;
  const int pk1 = T.nb[0] >= 0 ? npx : 0, pk2 = pk1 + (T.nb[1] >= 0 ? npx : 0),
            pk3 = pk2 + (T.nb[2] >= 0 ? npz : 0), pk4 = pk3 + (T.nb[3] >= 0 ? npz : 0);

  auto sent = [&](int q, int &off, int &slot) {
    int side, k, r, c, to;   // side: of the receiver
    if (q < pk2) {
      side = q < pk1 ? 1 : 0;
      to = q < pk1 ? T.nb[0] : T.nb[1];
      k = q < pk1 ? q : q - pk1;
      r = 2 * (k >> 2);
      c = (side ? 0 : TX - 4) + (k & 3);
    } else {
      side = q < pk3 ? 3 : 2;
      to = q < pk3 ? T.nb[2] : T.nb[3];
      k = q < pk3 ? q - pk2 : q - pk3;
      r = (side == 3 ? 0 : TZ - 4) + 2 * (k & 1);
      c = k >> 1;
    }
    off = (c + 4) * HS + r + 4;
    slot = (to * 8 + side) * A.cap + k;
  };
  auto received = [&](int q, int &off, int &slot) {
    int side, k, r, c;
    if (q < pk2) {
      side = q < pk1 ? 0 : 1;
      k = q < pk1 ? q : q - pk1;
      r = 2 * (k >> 2);
      c = (side ? TX : -4) + (k & 3);
    } else {
      side = q < pk3 ? 2 : 3;
      k = q < pk3 ? q - pk2 : q - pk3;
      r = (side == 3 ? TZ : -4) + 2 * (k & 1);
      c = k >> 1;
    }
    off = (c + 4) * HS + r + 4;
    slot = ((int)blockIdx.x * 8 + side) * A.cap + k;
  };
  int so[2], ro[2], ss[2], rs[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    sent(min(tid + k * OC_THREADS, max(pk4 - 1, 0)), so[k], ss[k]);
    received(min(tid + k * OC_THREADS, max(pk4 - 1, 0)), ro[k], rs[k]);
  }

  for (int s = A.s0; s < se; ++s) {
    float *const u3 = lev0 + (s & 3) * usz + UO;          // u_1, then u3 in place
    const float *const u0 = lev0 + ((s + 1) & 3) * usz + UO;
    const float *const u1 = lev0 + ((s + 2) & 3) * usz + UO;
    const float *const u2 = lev0 + ((s + 3) & 3) * usz + UO;
    const float *const op = ADJ ? w0 + (s & 1) * hsz : lev0 + ((s + 3) & 3) * usz;
    float *const wn = ADJ ? w0 + ((s + 1) & 1) * hsz : nullptr;
    float *const out = ADJ ? wn : lev0 + (s & 3) * usz;   // next step's stencil operand
    const float *const gterm = O.terms + (long long)(s - A.s0) * O.nent;

    auto item = [&](int e) {
      const int rl = 4 * (e & 255), cl = NC * ((e >> 8) & 255);
      const float *col0 = op + (cl + 4) * HS + rl + 4;
      const int nrow = zhi - (r0 + rl) + 1;   // rows to store
      float4 vel[NC];   // the square of the velocity with VSM
#pragma unroll
      for (int cc = 0; cc < NC; ++cc)
        vel[cc] = VSM ? oc_ld4(V + (cl + cc) * CS + rl)
                      : oc_ld4(vel0 + ld1 * min(cl + cc, n2p - 1 - c0) + rl);
      // Columns cl-4 .. cl+NC+3, each loaded once.
      float4 N[NC + 8];
#pragma unroll
      for (int m = 0; m < NC + 8; ++m) N[m] = oc_ld4(col0 + (m - 4) * HS);
      P2 svc[NC][2], v2c[NC][2];
#pragma unroll
      for (int cc = 0; cc < NC; ++cc) {
        const float4 za = oc_ld4(col0 + cc * HS - 4), zc = oc_ld4(col0 + cc * HS + 4);
        const float4 zb = N[4 + cc];
        const P2 P[6] = {lo2(za), hi2(za), lo2(zb), hi2(zb), lo2(zc), hi2(zc)};
        // Pairs of rows at odd distances straddle the loaded pairs: scalar
        // sums there cost fewer instructions than the moves to form pairs.
        const float zr[12] = {za.x, za.y, za.z, za.w, zb.x, zb.y,
                              zb.z, zb.w, zc.x, zc.y, zc.z, zc.w};
        P2 tzz[2], txx[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int m = 4 + 2 * h;
          P2 a = s_mul(c0z, P[2 + h]);
          a = p_add(a, p2(__fmul_rn(c1z, zr[m + 1] + zr[m - 1]),
                          __fmul_rn(c1z, zr[m + 2] + zr[m])));
          a = p_add(a, s_mul(c2z, p_add(P[3 + h], P[1 + h])));
          a = p_add(a, p2(__fmul_rn(c3z, zr[m + 3] + zr[m - 3]),
                          __fmul_rn(c3z, zr[m + 4] + zr[m - 2])));
          a = p_add(a, s_mul(c4z, p_add(P[4 + h], P[h])));
          tzz[h] = a;
          txx[h] = s_mul(cx[0], P[2 + h]);
        }
#pragma unroll
        for (int l = 1; l <= 4; ++l) {
          const float4 rp = N[4 + cc + l], rm = N[4 + cc - l];
          txx[0] = p_add(txx[0], s_mul(cx[l], p_add(lo2(rp), lo2(rm))));
          txx[1] = p_add(txx[1], s_mul(cx[l], p_add(hi2(rp), hi2(rm))));
        }
        v2c[cc][0] = VSM ? lo2(vel[cc]) : p_mul(lo2(vel[cc]), lo2(vel[cc]));
        v2c[cc][1] = VSM ? hi2(vel[cc]) : p_mul(hi2(vel[cc]), hi2(vel[cc]));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          svc[cc][h] = p_add(txx[h], tzz[h]);
          if (!ADJ) svc[cc][h] = p_mul(v2c[cc][h], svc[cc][h]);
        }
      }
#pragma unroll
      for (int cc = 0; cc < NC; ++cc) {
        P2(&sv)[2] = svc[cc];
        // Injection (Injection.f90:151-456, 561-591): each cell's terms in
        // entry order (x + -0 = x for every x, so padding changes nothing).
        if (inj_tile) {
          const int ri = r0 + rl - ioff, j = c0 + cl + cc;
          if (ri >= 0 && ri < trow && j >= jb0 && j <= jb1) {
            const int tp = (j - joff) * trow + ri, ts = tcol * trow;
            float r[4] = {sv[0].x, sv[0].y, sv[1].x, sv[1].y};
            auto add = [&](float4 t) {
              r[0] = r[0] + t.x;
              r[1] = r[1] + t.y;
              r[2] = r[2] + t.z;
              r[3] = r[3] + t.w;
            };
            if (inj_sm) {
#pragma unroll 2
              for (int m = 0; m < O.M; ++m)
                add(oc_ld4(sterm + (s & 1) * T.nterm + tp + m * ts));
            } else {
#pragma unroll 4
              for (int m = 0; m < O.M; ++m) add(oc_ld4(gterm + tp + m * ts));
            }
            sv[0] = p2(r[0], r[1]);
            sv[1] = p2(r[2], r[3]);
          }
        }
        // Injection_Born (Imaging.f90:747-788).
        if (born && itm == 0) {
          const int cnt = it / snapi - (S.tcnt - 1) / snapi, j = c0 + cl + cc + S.g.lo2;
          if (cnt <= S.ntsnap && j >= 1 && j <= S.g.nx) {
            const float *ws = S.wave + (long long)(cnt - 1) * nphys;
            const float taper = S.taperx ? S.taperx[j - 1] * S.tapery[0] : 1.f;
            const float4 vq = VSM ? oc_ld4(vel0 + ld1 * (cl + cc) + rl) : vel[cc];
            const float vc[4] = {vq.x, vq.y, vq.z, vq.w};
            float r[4] = {sv[0].x, sv[0].y, sv[1].x, sv[1].y};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int i = r0 + rl + q + S.g.lo1;
              if (i < 1 || i > nz) continue;
              const long long pp = (long long)(i - 1) + (long long)nz * (j - 1);
              r[q] = r[q] + (((2.0f * taper) * S.ref[pp]) * ws[pp]) / vc[q];
            }
            sv[0] = p2(r[0], r[1]);
            sv[1] = p2(r[2], r[3]);
          }
        }
        // FD_2nd_time_derivative_grid (FDderivatives.f90:960-982).
        const int o = (cl + cc) * US + rl;
        const float4 uc = ADJ ? oc_ld4(u2 + o) : N[4 + cc];
        const float4 a1 = oc_ld4(u1 + o), a0 = oc_ld4(u0 + o), am = oc_ld4(u3 + o);
        P2 r[2], w[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          P2 a = s_mul(20.0f, h ? hi2(uc) : lo2(uc));
          a = p_sub(a, s_mul(6.0f, h ? hi2(a1) : lo2(a1)));
          a = p_sub(a, s_mul(4.0f, h ? hi2(a0) : lo2(a0)));
          a = p_add(a, h ? hi2(am) : lo2(am));
          a = p_add(a, s_mul(k12, sv[h]));
          r[h] = p_mul(a, div11);
          if (ADJ) w[h] = p_mul(v2c[cc][h], r[h]);
        }
        if (!(e & (1 << (16 + cc)))) continue;
        const int ow = (cl + cc + 4) * HS + rl + 4;
        if (nrow >= 4) {
          oc_st4(u3 + o, r[0], r[1]);
          if (ADJ) oc_st4(wn + ow, w[0], w[1]);
        } else {
          const float rv[4] = {r[0].x, r[0].y, r[1].x, r[1].y};
#pragma unroll
          for (int q = 0; q < 3; ++q)
            if (q < nrow) {
              u3[o + q] = rv[q];
              if (ADJ) wn[ow + q] = q == 0 ? w[0].x : q == 1 ? w[0].y : w[1].x;
            }
        }
      }
    };

    const unsigned epoch = A.epoch0 + (unsigned)(s - A.s0) + 1;
#pragma unroll 1
    for (int part = 0; part < 2; ++part) {
#pragma unroll 1
    for (int q = (part ? n_first : 0) + tid; q < (part ? n_all : n_first); q += OC_THREADS)
      item(items[q]);
    if (part) break;
    __syncthreads();
    if (edge) {
      // Higdon lines (Boundary.f90:17-184): z lines, then x lines.
      for (int q = tid; q < nzl; q += OC_THREADS) {
        const bool bot = !top || q >= TX;
        const int c = bot && top ? q - TX : q, C = c0 + c;
        if (C < 4 || C > n2p - 5) continue;
        const int dir = bot ? -1 : 1, p = (bot ? n1p - 8 : 7) - r0;
        float k[8], U2[10], U1[10], o8[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) k[m] = ecoef[m * nline + q];
#pragma unroll
        for (int m = 0; m < 10; ++m) {
          U2[m] = u2[c * US + p - (m - 2) * dir];
          U1[m] = u1[c * US + p - (m - 2) * dir];
        }
        oc_higdon8(k, U2, U1, u3[c * US + p + dir], u3[c * US + p + 2 * dir], o8);
#pragma unroll
        for (int m = 0; m < 8; ++m) {
          const int r = p - m * dir;
          u3[c * US + r] = o8[m];
          if (ADJ) wn[(c + 4) * HS + r + 4] = evel[m * nline + q] * o8[m];
        }
      }
      if (left || right) {
        __syncthreads();
        for (int q = tid; q < nxl; q += OC_THREADS) {
          const bool rgt = !left || q >= TZ;
          const int r = rgt && left ? q - TZ : q, R = r0 + r;
          if (R < 4 || R > n1p - 5) continue;
          const int dir = rgt ? -1 : 1, p = (rgt ? n2p - 8 : 7) - c0;
          float k[8], U2[10], U1[10], o8[8];
#pragma unroll
          for (int m = 0; m < 8; ++m) k[m] = ecoef[m * nline + nzl + q];
#pragma unroll
          for (int m = 0; m < 10; ++m) {
            U2[m] = u2[(p - (m - 2) * dir) * US + r];
            U1[m] = u1[(p - (m - 2) * dir) * US + r];
          }
          oc_higdon8(k, U2, U1, u3[(p + dir) * US + r], u3[(p + 2 * dir) * US + r], o8);
#pragma unroll
          for (int m = 0; m < 8; ++m) {
            const int c = p - m * dir;
            u3[c * US + r] = o8[m];
            if (ADJ) wn[(c + 4) * HS + r + 4] = evel[m * nline + nzl + q] * o8[m];
          }
        }
      }
      __syncthreads();
    }
    if (s + 1 < se) {
      // Border strips to the neighbours: 4 columns (rows) of the next
      // step's stencil operand, two rows of one column per packet.
      ulonglong2 *const box = A.inbox + (epoch & 1) * 4 * A.cap;
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (tid + k * OC_THREADS < pk4) {
          const float2 v = *reinterpret_cast<const float2 *>(out + so[k]);
          oc_put(box + ss[k], v.x, v.y, epoch);
        }
      for (int q = tid + 2 * OC_THREADS; q < pk4; q += OC_THREADS) {
        int off, slot;
        sent(q, off, slot);
        const float2 v = *reinterpret_cast<const float2 *>(out + off);
        oc_put(box + slot, v.x, v.y, epoch);
      }
      if (inj_sm) fetch_terms(s + 1);
    }
    }
    // Snapshot of u2 (Extraction.f90:562-601), spread over this step and the
    // next ones, in which the level is still there as u1 and u0.
    if (saves) {
      if (itm == 0) {
        sdst = oc_save_slot(S, O, it, A.s0, nphys);
        spart = 0;
      }
      if (sdst) {
        const float *u = (spart == 0 ? u2 : spart == 1 ? u1 : u0) + sca * US + sra;
        float *d = sdst + (long long)nz * (c0 + sca + S.g.lo2 - 1) + (r0 + sra + S.g.lo1 - 1);
        const int last = s + 1 == se ? nsave : spart + 1;   // the launch ends: all of it
        for (; spart < last; ++spart)
#pragma unroll 1
          for (int c = spart * (OC_THREADS / 32) + warp; c < snc; c += nsave * (OC_THREADS / 32)) {
            const float *uc = u + c * US;
            float *dc = d + c * nz;
#pragma unroll 1
            for (int r = lane; r < snr; r += 32) dc[r] = uc[r];
          }
        if (spart == nsave) sdst = nullptr;
      }
    }
    // Receiver cells of u2.
    if (T.ncell > 0) {
      float *tp = O.tape + (long long)(s - A.s0) * O.ncell + T.cell0;
      for (int q = tid; q < T.ncell; q += OC_THREADS) {
        const int e = O.cells[T.cell0 + q];
        tp[q] = u2[(e >> 16) * US + (e & 0xffff)];
      }
    }
    if (s + 1 < se) {
      const ulonglong2 *const box = A.inbox + (epoch & 1) * 4 * A.cap;
      auto take = [&](int off, int slot) {
        const ulonglong2 *p = box + slot;
        ulonglong2 v;
        bool ok = false;
        for (int w = 0; w < OC_WAIT_LIMIT; ++w) {
          v = oc_get(p);
          ok = (unsigned)(v.x >> 32) == epoch && (unsigned)(v.y >> 32) == epoch;
          if (ok || abort_flag) break;
          if ((w & 1023) == 1023 && *(volatile int *)A.err) break;
        }
        if (!ok) {
          atomicOr(A.err, 1);
          abort_flag = 1;
        }
        *reinterpret_cast<float2 *>(out + off) =
            make_float2(__uint_as_float((unsigned)v.x), __uint_as_float((unsigned)v.y));
      };
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (tid + k * OC_THREADS < pk4) take(ro[k], rs[k]);
      for (int q = tid + 2 * OC_THREADS; q < pk4; q += OC_THREADS) {
        int off, slot;
        received(q, off, slot);
        take(off, slot);
      }
      if (inj_sm) asm volatile("cp.async.wait_all;" ::: "memory");
    }
    it += tstep;
    itm += tstep;
    if (itm == snapi) itm = 0;
    if (itm < 0) itm = snapi - 1;
    __syncthreads();
    if (abort_flag) return;   // uniform: written before the barrier
  }

  // ---- state back to the level buffers ----
  for (int q = tid; q < NG * TX; q += OC_THREADS) {
    const int c = q / NG, g = q % NG, C = c0 + c;
    if (C >= n2p) continue;
    const long long off = (long long)(r0 + 4 * g) + (long long)ld1 * C;
#pragma unroll
    for (int l = 0; l < 4; ++l)
      *reinterpret_cast<float4 *>(S.f[(se + l) % 5] + off) =
          oc_ld4(lev0 + ((se + l) & 3) * usz + UO + c * US + 4 * g);
  }
}

// Injection terms (((v2r * trace(it)) * wz) * wx) * wy (Injection.f90:
// 151-456, 561-591) of steps [s0, s0 + ns) of one shot in the layout of
// OcShot::terms; ell[slot] is the slot's entry, -1 where there is none.
__global__ void k_oc_terms(const ShotDev *shots, int b, int s0, int ns, int nent,
                           const int *__restrict__ ell, float *terms) {
  const ShotDev &S = shots[b];
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nent) return;
  const int e = ell[q];
  const InjEntry E = e >= 0 ? S.inj_ent[e] : InjEntry{0, 0.f, 0.f, 0.f, 0.f};
  const float *tr = S.src_tr + (long long)E.tr * S.nt;
  const int k1 = min(ns, 8 * (int)(blockIdx.y + 1));
  for (int k = 8 * blockIdx.y; k < k1; ++k) {
    const int it = S.tmin + (s0 + k) * S.tstep;
    terms[(long long)k * nent + q] =
        e >= 0 ? (((E.v2r * tr[it - 1]) * E.wz) * E.wx) * E.wy : -0.f;
  }
}

// Receivers of steps [s0, s0 + ns) of one shot from its saved cells
// (Extraction.f90:71-135, 217-247, 511-560): a thread adds one receiver's
// products to one sample in the reference's loop order.  A block takes 32
// receivers x 32 steps: lanes run over receivers for the cells (neighbours
// in the tape), then over steps for the traces, through shared memory.
// idx: [tap][receiver] cell numbers, idxm those of the mirrored rows.
__global__ void __launch_bounds__(256) k_oc_extract(const ShotDev *shots, int b, int s0, int ns,
                                                    const float *__restrict__ tape, int ncell,
                                                    const int *__restrict__ idx,
                                                    const int *__restrict__ idxm) {
  __shared__ float sh[32][33];
  const ShotDev &S = shots[b];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int rb = 32 * blockIdx.x, kb = 32 * blockIdx.y;
  auto sample = [&](int r, int k) {
    return S.rec_tr + (long long)r * S.nt + (S.tmin + (s0 + k) * S.tstep - 1);
  };
  for (int q = w; q < 32; q += 8)
    if (rb + q < S.nrec && kb + lane < ns) sh[q][lane] = *sample(rb + q, kb + lane);
  __syncthreads();
  const int r = rb + lane, ls = 2 * S.ext_half + 1;
  if (r < S.nrec) {
    float v = S.vconst;
    if (S.ext_mode == 1) {
      const float vv = S.vel[S.g.idx(S.ric[3 * r], S.ric[3 * r + 1], 1)];
      v = vv * vv;
    }
    const float *wz = S.wz + (long long)r * ls, *wx = S.wx + (long long)r * ls;
    for (int k = w; k < 32 && kb + k < ns; k += 8) {
      const float *tp = tape + (long long)(kb + k) * ncell;
      float tr = sh[lane][k];
      if (S.ext_mode == 2) {   // Extraction_array_simple_afwi_noomp
        tr = tr + (S.ext_mirror ? tp[idx[r]] - tp[idxm[r]] : tp[idx[r]]);
      } else {
        for (int jj = 0, tap = 0; jj < ls; ++jj) {
          const float wxj = wx[jj];
          for (int ii = 0; ii < ls; ++ii, ++tap) {
            float u = tp[idx[tap * S.nrec + r]];
            if (S.ext_mirror) u = u - tp[idxm[tap * S.nrec + r]];
            tr = tr + ((v * u) * wz[ii]) * wxj;
          }
        }
      }
      sh[lane][k] = tr;
    }
  }
  __syncthreads();
  for (int q = w; q < 32; q += 8)
    if (rb + q < S.nrec && kb + lane < ns) *sample(rb + q, kb + lane) = sh[q][lane];
}

// RTM / LSRTM / AFWI imaging (Imaging.f90:228-422, 698-745) of one shot's
// backward steps [s0, s0 + ns): a thread adds the imaging steps of one
// physical point in time order, from the backward snapshots of the launch
// and the saved forward ones; image and illumination are read and written
// once.  Bound by HBM: 8 bytes per point and imaging step.
__global__ void __launch_bounds__(256) k_oc_image(const ShotDev *shots, int b, int s0, int ns,
                                                  const float *__restrict__ bsnap) {
  const ShotDev &S = shots[b];
  const int nz = S.g.nz;
  const long long nphys = (long long)nz * S.g.nx;
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nphys) return;
  const int j = (int)(q / nz) + 1, i = (int)(q % nz) + 1;
  const float taper = S.taperx ? S.taperx[j - 1] * S.tapery[0] : 1.f;
  const float v = S.imaging > 1 ? S.vel[S.g.idx(i, j, 1)] : 1.f;
  // Time samples it1, it1 - snapi, ... of the launch; index(it) counts down.
  const int itl = S.tmin - (s0 + ns - 1), m1 = (S.tmin - s0) / S.snapi;
  int n = m1 - (itl + S.snapi - 1) / S.snapi + 1;   // multiples of snapi in [itl, it1]
  const int index0 = S.ntsnap - (S.tcnt / S.snapi - (m1 * S.snapi - 1) / S.snapi) + 1;
  n = min(n, index0);                               // index >= 1
  if (n <= 0) return;
  const float *w = S.wave + (long long)(index0 - 1) * nphys + q;
  const float *u = bsnap + q;
  float im = S.image[q], il = S.illum[q];
  if (S.imaging == 3) {
    const float den = S.dt2snap * ((v * v) * v);
    float wp = S.wave[(long long)(min(index0 + 1, S.ntsnap) - 1) * nphys + q], wc = *w;
#pragma unroll 4
    for (int k = 0; k < n; ++k) {
      const int index = index0 - k;
      const float wm = index > 1 ? *(w - (long long)(k + 1) * nphys) : wc;
      const float tt = ((wm - 2.0f * wc) + wp) / den;
      im = im + (u[(long long)k * nphys] * tt) * taper;
      il = il + (wc * wc) * taper;
      wp = wc;
      wc = wm;
    }
  } else {
#pragma unroll 4
    for (int k = 0; k < n; ++k) {
      const float uc = u[(long long)k * nphys], wc = *(w - (long long)k * nphys);
      if (S.imaging == 1) im = im + (uc * wc) * taper;
      else im = im + (((2.0f * taper) * uc) * wc) / v;
      il = il + (wc * wc) * taper;
    }
  }
  S.image[q] = im;
  S.illum[q] = il;
}

}  // namespace swave
