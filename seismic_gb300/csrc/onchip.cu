// onchip.cu - plans and launches of the on-chip 2D propagation (onchip2d.cuh;
// compiled with --fmad=false).
#include <algorithm>
#include <cstring>
#include <vector>

#include "engine.h"
#include "onchip2d.cuh"

namespace swave {

namespace {

// Dynamic shared memory of one CTA (227 KB less the kernel's own variables).
constexpr size_t kSmemLimit = 228 * 1024 / OC_PER_SM - 2048;
// Smallest tile worth a CTA of its own: below it the border exchange costs
// more than the points.
constexpr long long kMinArea = 1024;
// Scratch of one launch: injection terms, receiver cells and backward
// snapshots of its steps; the launch covers as many steps as fit.
constexpr size_t kScratch = 512u << 20;
constexpr long long kMaxTerms = 1 << 20;   // injection terms of a shot and step, padding included
constexpr int kMinChunk = 32, kMaxChunk = 1 << 16;

struct Shape {
  std::vector<int> z, x;   // cuts: row groups and column pairs of the bands
  int TZ = 0, TX = 0;      // the largest tile
};

// Points that a tile's Higdon lines (per pair of opposite axes) and one
// injection term cost, so that edge tiles are cut smaller.
constexpr double kEdgePoints = 900.0, kTermPoints = 0.5;

// n units in k bands of at least `least`; the first and last take fewer by ef
// and el.
std::vector<int> cut(int n, int k, double ef, double el, int least) {
  std::vector<int> c(k + 1, n);
  c[0] = 0;
  if (k == 1) return c;
  const double t = (n + ef + el) / k;
  for (int q = 1; q < k; ++q) {
    const int v = (int)(q * t - ef + 0.5);
    c[q] = std::min(std::max(v, c[q - 1] + least), n - (k - q) * least);
  }
  return c;
}
int widest(const std::vector<int> &c) {
  int w = 0;
  for (size_t q = 1; q < c.size(); ++q) w = std::max(w, c[q] - c[q - 1]);
  return w;
}

// Tiles of a shot on at most ncta CTAs: the cut whose largest tile has the
// smallest area plus border.  tcol: injection terms per column of the box,
// in row group tgrp.
bool shape_for(const Geom &g, int ncta, bool adj, int tcol, int tgrp, Shape *out) {
  const int NG = (g.n1p + 3) / 4, NP = (g.n2p + 1) / 2;
  if (g.n1p < 24 || g.n2p < 24) return false;
  long long best = -1;
  for (int ntz = 1; ntz <= ncta; ++ntz) {
    if (ntz > 1 && NG / ntz < OC_MIN_GROUPS) break;
    const int ntx = std::max(1, std::min(ncta / ntz, NP / OC_MIN_PAIRS));
    // Even tiles first: an edge tile loses at most half its size.
    const double rows = 4.0 * NG / ntz, cols = 2.0 * NP / ntx;
    const double ez = std::min(kEdgePoints / cols, rows / 4) / 4,
                 ex = std::min(kEdgePoints / rows, cols / 4) / 2;
    const double ti = tgrp < NG / ntz ? std::min(kTermPoints * tcol, rows / 4) / 4 : 0.0;
    Shape s;
    s.z = cut(NG, ntz, ez + ti, ez, OC_MIN_GROUPS);
    s.x = cut(NP, ntx, ex, ex, OC_MIN_PAIRS);
    s.TZ = 4 * widest(s.z);
    s.TX = 2 * widest(s.x);
    if (s.TZ > 1020 || s.TX > 510) continue;
    // The first, widest and last band of each axis: tile and edge lines fit.
    bool fits = true;
    for (int a = 0; a < 3 && fits; ++a)
      for (int e = 0; e < 3 && fits; ++e) {
        OcTile t{};
        t.TZ = a == 1 ? s.TZ : 4 * (a == 0 ? s.z[1] : NG - s.z[ntz - 1]);
        t.TX = e == 1 ? s.TX : 2 * (e == 0 ? s.x[1] : NP - s.x[ntx - 1]);
        t.nline = t.TX * (ntz == 1 ? 2 : a != 1) + t.TZ * (ntx == 1 ? 2 : e != 1);
        fits = oc_smem_bytes(t, adj, false, false) <= kSmemLimit;
      }
    if (!fits) continue;
    const long long cost = (long long)s.TZ * s.TX + 8LL * (s.TZ + s.TX);
    if (best < 0 || cost < best) {
      best = cost;
      *out = s;
    }
  }
  return best >= 0;
}

int num_sms(int dev) {
  int n = 0;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n = 0;
  return n;
}

// What the kernel keeps in static shared memory beside a CTA's kSmemLimit (and
// the 1 KB that the system takes of each CTA's share).
static_assert(kSmemLimit + sizeof(ShotDev) + 40 * sizeof(int) + 1024 <= 228 * 1024 / OC_PER_SM,
              "OC_PER_SM CTAs of k_onchip2d no longer fit on an SM");

const void *kernel(bool adj, bool vsm) {
  return adj ? (vsm ? (const void *)k_onchip2d<true, true> : (const void *)k_onchip2d<true, false>)
             : (vsm ? (const void *)k_onchip2d<false, true> : (const void *)k_onchip2d<false, false>);
}

// CTAs of a form that are resident together on the context's device, asked
// once per context (with the shared-memory opt-in); 0 if it cannot be told.
int resident(sw_ctx *c, bool adj, bool vsm) {
  int &n = c->oc_resident[2 * adj + vsm];
  if (n < 0) {
    int per = 0;
    const void *k = kernel(adj, vsm);
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, OC_THREADS, kSmemLimit) !=
            cudaSuccess) {
      cudaGetLastError();
      per = 0;
    }
    n = per * num_sms(c->device);
  }
  return n;
}

bool clear_inbox(sw_ctx *c) {
  const DBuf &b = c->bufs["oc_inbox"];
  c->oc_epoch = 0;
  return c->oc_zeroed = cudaMemsetAsync(b.p, 0, b.cap, c->stream) == cudaSuccess;
}

}  // namespace

bool oc_eligible(const sw_ctx *c, const PhaseShot &p, const RunOpts &opt) {
  const sw_prop_desc &d = p.d;
  if (!d.g.twoD || p.io.rho_pad || d.g.surf_type != 0 || !opt.use_graph ||
      opt.tile.stream2d != 2 || !opt.onchip)
    return false;
  if (d.imaging < SW_IMG_NONE || d.imaging > SW_IMG_BORN) return false;
  // The adjoint form has no Born source (no driver runs it there).
  if (d.imaging == SW_IMG_BORN && d.fd_scheme == SW_FD_ADJOINT) return false;
  // A phase that both saves and images may read the slot it writes.
  if (d.extract_wave && d.imaging != SW_IMG_NONE) return false;
  const Geom g = make_geom(d.g);
  Shape sh;
  return g.total() < (1LL << 31) &&
         shape_for(g, OC_PER_SM * num_sms(c->device), d.fd_scheme == SW_FD_ADJOINT, 0, 0, &sh);
}

// Cuts the shots into launches and carves their plans; false (without an
// error) when the scratch does not fit or the CTAs of a launch would not all
// be resident, and the caller takes the per-step kernels.
bool oc_plan(sw_ctx *c, const std::vector<PhaseShot> &shots, const std::vector<Geom> &G,
             const std::vector<InjPlan> &inj, const std::vector<ExtPlan> &ext, OcRun &R) {
  const int nb = (int)shots.size(), nsm = OC_PER_SM * num_sms(c->device);
  const int nb1 = std::max(nb, 1);
  std::vector<int> order(nb), cmin(nb), nsteps(nb), adj(nb), tcol(nb, 0), tgrp(nb, 0);
  for (int b = 0; b < nb; ++b) {
    const sw_prop_desc &d = shots[b].d;
    order[b] = b;
    nsteps[b] = (d.tmax - d.tmin + d.tstep) / d.tstep;
    adj[b] = d.fd_scheme == SW_FD_ADJOINT;
    if (inj[b].on) {
      int M = 0;
      for (size_t q = 0; q + 1 < inj[b].off.size(); ++q)
        M = std::max(M, inj[b].off[q + 1] - inj[b].off[q]);
      const int a = (inj[b].bi0 - G[b].lo1) / 4, e = (inj[b].bi1 - G[b].lo1) / 4;
      // A single source loads one tile only; a line of receivers its band.
      if (inj[b].bj1 - inj[b].bj0 > G[b].n2p / 2) tcol[b] = M * 4 * (e - a + 1);
      tgrp[b] = a;
    }
    Shape sh;
    int lo = 1, hi = nsm;   // the fewest CTAs that hold the shot
    if (!shape_for(G[b], hi, adj[b], tcol[b], tgrp[b], &sh)) return false;
    while (lo < hi) {
      const int m = (lo + hi) / 2;
      if (shape_for(G[b], m, adj[b], tcol[b], tgrp[b], &sh)) hi = m;
      else lo = m + 1;
    }
    cmin[b] = lo;
  }
  // Shots of similar length share a launch; as few launches as hold them
  // all, evenly filled (a launch lasts as long as its longest shot, and a
  // shot gains less than proportionally from more CTAs).
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    return adj[a] != adj[b] ? adj[a] < adj[b] : nsteps[a] > nsteps[b];
  });
  auto pack = [&](int limit, std::vector<std::vector<int>> &out) {
    out.clear();
    int used = 0;
    for (int b : order) {
      const bool fresh = out.empty() || used + cmin[b] > nsm || (int)out.back().size() >= limit ||
                         adj[out.back()[0]] != adj[b];
      if (fresh) {
        out.push_back({});
        used = 0;
      }
      out.back().push_back(b);
      used += cmin[b];
    }
  };
  std::vector<std::vector<int>> grp, even;
  pack(nb1, grp);
  for (int lim = 1; lim <= nb1; ++lim) {
    pack(lim, even);
    if (even.size() <= grp.size()) {
      grp = even;
      break;
    }
  }
  R.groups.clear();
  R.tiles.clear();
  R.cells.clear();
  R.idx.clear();
  R.shot.assign(nb, OcShotPlan{});
  for (auto &m : grp) {
    OcGroup g;
    g.members = m;
    g.adj = adj[m[0]] != 0;
    g.tile0 = (int)R.tiles.size();
    size_t smem[4] = {0, 0, 0, 0};   // [vsm + 2 pad]
    std::vector<int> n(m.size());
    int used = 0;
    for (size_t q = 0; q < m.size(); ++q) used += n[q] = cmin[m[q]];
    // The CTAs left over, one by one to the shot with the largest tiles.
    while (used < nsm) {
      int pick = -1;
      double area = (double)kMinArea;
      for (size_t q = 0; q < m.size(); ++q) {
        const double a = (double)G[m[q]].n1p * G[m[q]].n2p / (n[q] + 1);
        if (a > area) {
          area = a;
          pick = (int)q;
        }
      }
      if (pick < 0) break;
      ++n[pick];
      ++used;
    }
    size_t per_step = 0;
    for (size_t q = 0; q < m.size(); ++q) {
      const int b = m[q];
      const Geom &gg = G[b];
      Shape sh;
      if (!shape_for(gg, n[q], adj[b], tcol[b], tgrp[b], &sh)) return false;
      g.cap = std::max(g.cap, 2 * std::max(sh.TZ, sh.TX));
      OcShotPlan &P = R.shot[b];
      // Receiver cells: the union of the footprints, numbered tile by tile.
      const int mode = ext[b].on ? ext[b].mode : 0;
      const int h = mode == SW_EXT_SIMPLE_AFWI ? 0 : shots[b].d.g.lsinc / 2, ls = 2 * h + 1;
      std::vector<int> id;
      if (mode) {
        id.assign((size_t)gg.n1p * gg.n2p, -1);
        for (int r = 0; r < ext[b].nrec; ++r) {
          const int i0 = ext[b].ic[3 * r] - gg.lo1, j0 = ext[b].ic[3 * r + 1] - gg.lo2;
          const int im = -ext[b].ic[3 * r] - gg.lo1;   // reflected row
          for (int jj = -h; jj <= h; ++jj)
            for (int ii = -h; ii <= h; ++ii) {
              id[(size_t)(j0 + jj) * gg.n1p + i0 + ii] = 0;
              if (ext[b].mirror) id[(size_t)(j0 + jj) * gg.n1p + im + ii] = 0;
            }
        }
      }
      if (inj[b].on) {
        // Terms by (m, column, row) over the box, its rows widened to whole
        // groups of 4; a shot whose cells differ too much in their number of
        // entries, or whose sources are far apart, is left to the per-step
        // kernels (their lists have no padding).
        const InjPlan &I = inj[b];
        const int nbi = I.bi1 - I.bi0 + 1;
        P.row0 = (I.bi0 - gg.lo1) & ~3;
        P.nrow = ((I.bi1 - gg.lo1) | 3) + 1 - P.row0;
        P.ncol = I.bj1 - I.bj0 + 1;
        for (size_t q = 0; q + 1 < I.off.size(); ++q) P.M = std::max(P.M, I.off[q + 1] - I.off[q]);
        const long long slots = (long long)P.M * P.ncol * P.nrow;
        if (slots > kMaxTerms) return false;
        P.nent = (int)slots;
        P.ell0 = R.idx.size();
        R.idx.resize(P.ell0 + P.nent, -1);
        int *ell = R.idx.data() + P.ell0;
        for (int j = 0; j < P.ncol; ++j)
          for (int i = 0; i < nbi; ++i) {
            const int cell = i + nbi * j, row = I.bi0 - gg.lo1 + i - P.row0;
            for (int e = I.off[cell]; e < I.off[cell + 1]; ++e)
              ell[((size_t)(e - I.off[cell]) * P.ncol + j) * P.nrow + row] = e;
          }
      }
      const int ntz = (int)sh.z.size() - 1, ntx = (int)sh.x.size() - 1;
      const int base = (int)R.tiles.size() - g.tile0;
      P.cell0 = (int)R.cells.size();
      for (int xi = 0; xi < ntx; ++xi)
        for (int zi = 0; zi < ntz; ++zi) {
          OcTile t;
          t.shot = b;
          t.r0 = 4 * sh.z[zi];
          t.TZ = 4 * (sh.z[zi + 1] - sh.z[zi]);
          t.c0 = 2 * sh.x[xi];
          t.TX = 2 * (sh.x[xi + 1] - sh.x[xi]);
          const int me = base + xi * ntz + zi;
          t.nb[0] = xi > 0 ? me - ntz : -1;
          t.nb[1] = xi + 1 < ntx ? me + ntz : -1;
          t.nb[2] = zi > 0 ? me - 1 : -1;
          t.nb[3] = zi + 1 < ntz ? me + 1 : -1;
          t.cell0 = (int)R.cells.size() - P.cell0;
          if (mode)
            for (int cc = t.c0; cc < std::min(t.c0 + t.TX, gg.n2p); ++cc)
              for (int rr = t.r0; rr < std::min(t.r0 + t.TZ, gg.n1p); ++rr) {
                int &v = id[(size_t)cc * gg.n1p + rr];
                if (v < 0) continue;
                v = (int)R.cells.size() - P.cell0;
                R.cells.push_back(((cc - t.c0) << 16) | (rr - t.r0));
              }
          t.ncell = (int)R.cells.size() - P.cell0 - t.cell0;
          // The tile's injection terms in shared memory if they fit.
          t.nterm = 0;
          t.nline = (t.r0 == 0 ? t.TX : 0) + (t.r0 + t.TZ >= gg.n1p ? t.TX : 0) +
                    (t.c0 == 0 ? t.TZ : 0) + (t.c0 + t.TX >= gg.n2p ? t.TZ : 0);
          const int ra = std::max(t.r0, P.row0), rb = std::min(t.r0 + t.TZ, P.row0 + P.nrow);
          const int ca = std::max(t.c0, inj[b].bj0 - gg.lo2),
                    cb = std::min(t.c0 + t.TX, inj[b].bj0 - gg.lo2 + P.ncol);
          if (P.nent && ra < rb && ca < cb) {
            t.nterm = P.M * (cb - ca) * (rb - ra);
            if (oc_smem_bytes(t, g.adj, false, false) > kSmemLimit) t.nterm = 0;
          }
          if (oc_smem_bytes(t, g.adj, false, false) > kSmemLimit) return false;
          for (int k = 0; k < 4; ++k)
            smem[k] = std::max(smem[k], oc_smem_bytes(t, g.adj, k & 1, k & 2));
          R.tiles.push_back(t);
        }
      P.ncell = (int)R.cells.size() - P.cell0;
      P.idx0 = R.idx.size();
      if (mode) {
        // [tap][receiver] cell numbers, z taps fastest; then the mirrored ones.
        for (int side = 0; side < (ext[b].mirror ? 2 : 1); ++side)
          for (int jj = -h; jj <= h; ++jj)
            for (int ii = -h; ii <= h; ++ii)
              for (int r = 0; r < ext[b].nrec; ++r) {
                const int i = ext[b].ic[3 * r];
                const int row = (side ? -ii - i : i + ii) - gg.lo1;
                R.idx.push_back(
                    id[(size_t)(ext[b].ic[3 * r + 1] + jj - gg.lo2) * gg.n1p + row]);
              }
        P.idxm0 = P.idx0 + (ext[b].mirror ? (size_t)ls * ls * ext[b].nrec : 0);
      }
      const sw_prop_desc &d = shots[b].d;
      const size_t nphys = (size_t)d.g.nz * d.g.nx;
      P.image = d.imaging >= 1 && d.imaging <= 3 && d.tstep < 0;
      per_step += 4 * ((size_t)P.nent + P.ncell) +
                  (P.image ? (4 * nphys + d.g.snapi - 1) / d.g.snapi : 0);
      g.steps = std::max(g.steps, nsteps[b]);
    }
    g.ncta = (int)R.tiles.size() - g.tile0;
    // The velocity on the chip before strides without bank conflicts.
    for (int k : {0, 2, 1, 3})
      if (smem[k] <= kSmemLimit) {
        g.smem = smem[k];
        g.vsm = k & 1;
        g.pad = k & 2;
      }
    if (g.ncta > resident(c, g.adj, g.vsm)) return false;
    size_t freeb = 0, totalb = 0;
    if (cudaMemGetInfo(&freeb, &totalb) != cudaSuccess) return false;
    size_t held = 0;
    auto it = c->bufs.find("oc_scratch");
    if (it != c->bufs.end()) held = it->second.cap;
    const size_t room = std::min<size_t>(kScratch, std::max(held, freeb / 4));
    // Imaging shots hold one more snapshot per launch than steps / snapi.
    size_t fixed = 4096;
    for (int b : m)
      fixed += 1024 + (R.shot[b].image ? 8 * (size_t)shots[b].d.g.nz * shots[b].d.g.nx : 0);
    if (fixed >= room) return false;
    const long long k = per_step ? (long long)((room - fixed) / per_step) : g.steps;
    g.chunk = (int)std::min<long long>({(long long)g.steps, k, (long long)kMaxChunk});
    if (g.chunk < std::min(g.steps, kMinChunk)) return false;
    R.scratch = std::max(R.scratch, fixed + per_step * (size_t)g.chunk);
    R.inbox = std::max(R.inbox, (size_t)g.ncta * 8 * g.cap * sizeof(ulonglong2));
    R.groups.push_back(g);
  }
  int st = SW_OK;
  const std::string keep = c->err;
  // Packets carry epochs that grow over the context's launches, so what an
  // earlier launch left in the inbox is never taken for a new packet; a new
  // buffer starts from zero, and so does a launch before which the epochs
  // would wrap (oc_run).
  const size_t had = c->bufs["oc_inbox"].cap;
  R.d_inbox = dbuf(c, "oc_inbox", R.inbox, &st);
  if (c->bufs["oc_inbox"].cap != had) c->oc_zeroed = false;
  if (R.d_inbox && !c->oc_zeroed && !clear_inbox(c)) return false;
  R.d_scratch = (char *)dbuf(c, "oc_scratch", R.scratch, &st);
  R.d_tiles = dbuf(c, "oc_tiles", R.tiles.size() * sizeof(OcTile), &st);
  R.d_cells = dbuf(c, "oc_cells", R.cells.size() * sizeof(int), &st);
  R.d_idx = dbuf(c, "oc_idx", R.idx.size() * sizeof(int), &st);
  R.d_oc = dbuf(c, "oc_shots", nb * sizeof(OcShot), &st);
  if (!R.d_scratch || !R.d_inbox || !R.d_tiles || !R.d_cells || !R.d_idx || !R.d_oc) {
    c->err = keep;
    return false;
  }
  return true;
}

// Runs the planned launches on the context's stream.  *refused: the device
// would not take the first of them (a share of it is held elsewhere) and
// nothing has run but the injection terms.
int oc_run(sw_ctx *c, const std::vector<ShotDev> &hs, const ShotDev *dshots, OcRun &R, bool rigid,
           int *derr, uint64_t *launches, bool *refused) {
  cudaStream_t s = c->stream;
  cudaError_t e;
  const int nb = (int)hs.size();
  SW_CK(cudaMemcpyAsync(R.d_tiles, R.tiles.data(), R.tiles.size() * sizeof(OcTile),
                        cudaMemcpyHostToDevice, s));
  if (!R.cells.empty())
    SW_CK(cudaMemcpyAsync(R.d_cells, R.cells.data(), R.cells.size() * sizeof(int),
                          cudaMemcpyHostToDevice, s));
  if (!R.idx.empty()) {
    SW_CK(cudaMemcpyAsync(R.d_idx, R.idx.data(), R.idx.size() * sizeof(int),
                          cudaMemcpyHostToDevice, s));
  }
  // Scratch of every shot (shots of different launches share it).
  std::vector<OcShot> ho(nb);
  std::vector<float *> terms(nb, nullptr);
  for (auto &g : R.groups) {
    char *cur = R.d_scratch;
    auto carve = [&](size_t n) {
      float *p = (float *)cur;
      cur += (n * sizeof(float) + 255) / 256 * 256;
      return p;
    };
    for (int b : g.members) {
      const OcShotPlan &P = R.shot[b];
      OcShot &O = ho[b];
      std::memset(&O, 0, sizeof(O));
      O.nent = P.nent;
      O.M = P.M;
      O.ncol = P.ncol;
      O.nrow = P.nrow;
      O.row0 = P.row0;
      O.ncell = P.ncell;
      if (P.nent) O.terms = terms[b] = carve((size_t)P.nent * g.chunk);
      if (P.ncell) O.tape = carve((size_t)P.ncell * g.chunk);
      O.cells = (const int *)R.d_cells + P.cell0;
      if (P.image)
        O.bsnap = carve((size_t)hs[b].g.nz * hs[b].g.nx * (g.chunk / hs[b].snapi + 1));
    }
    if ((size_t)(cur - R.d_scratch) > R.scratch) return fail(c, SW_CUDA_ERR, "on-chip scratch");
  }
  SW_CK(cudaMemcpyAsync(R.d_oc, ho.data(), nb * sizeof(OcShot), cudaMemcpyHostToDevice, s));
  cudaEvent_t ev[2] = {nullptr, nullptr};
  if (c->profiling) {
    SW_CK(cudaEventCreate(&ev[0]));
    SW_CK(cudaEventCreate(&ev[1]));
  }
  int st = SW_OK;
  bool ran = false;
  auto run = [&]() -> int {
    for (auto &g : R.groups) {
      OcArgs a;
      a.shots = dshots;
      a.oc = (const OcShot *)R.d_oc;
      a.tiles = (const OcTile *)R.d_tiles + g.tile0;
      a.inbox = (ulonglong2 *)R.d_inbox;
      a.cap = g.cap;
      a.rigid = rigid ? 1 : 0;
      a.pad = g.pad ? 1 : 0;
      a.err = derr;
      for (int s0 = 0; s0 < g.steps; s0 += g.chunk) {
        a.s0 = s0;
        a.s1 = std::min(s0 + g.chunk, g.steps);
        const unsigned used = (unsigned)(a.s1 - a.s0) + 1;
        if (c->oc_epoch > 0xffffffffu - used && !clear_inbox(c))
          return cuda_fail(c, cudaGetLastError(), "on-chip inbox");
        a.epoch0 = c->oc_epoch;
        c->oc_epoch += used;
        for (int b : g.members) {
          const int ns = std::min(a.s1, hs[b].nsteps) - s0;
          if (ns <= 0 || !R.shot[b].nent) continue;
          k_oc_terms<<<dim3((R.shot[b].nent + 255) / 256, (ns + 7) / 8), 256, 0, s>>>(
              dshots, b, s0, ns, R.shot[b].nent, (const int *)R.d_idx + R.shot[b].ell0, terms[b]);
          ++*launches;
        }
        if (c->profiling) SW_CK(cudaEventRecord(ev[0], s));
        // Cooperative: the CTAs wait for one another, so all must be resident.
        void *args[] = {&a};
        e = cudaLaunchCooperativeKernel(kernel(g.adj, g.vsm), dim3(g.ncta), dim3(OC_THREADS), args,
                                        g.smem, s);
        if (!ran && (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported)) {
          cudaGetLastError();
          *refused = true;
          return SW_OK;
        }
        if (e != cudaSuccess) return cuda_fail(c, e, "on-chip propagation");
        ran = true;
        ++*launches;
        if (c->profiling) {
          SW_CK(cudaEventRecord(ev[1], s));
          SW_CK(cudaEventSynchronize(ev[1]));
          float ms = 0.f;
          SW_CK(cudaEventElapsedTime(&ms, ev[0], ev[1]));
          c->stats.step_kernel_ms += ms;
        }
        for (int b : g.members) {
          const int ns = std::min(a.s1, hs[b].nsteps) - s0;
          const OcShotPlan &P = R.shot[b];
          if (ns <= 0) continue;
          if (P.ncell) {
            const int *ix = (const int *)R.d_idx + P.idx0;
            k_oc_extract<<<dim3((hs[b].nrec + 31) / 32, (ns + 31) / 32), 256, 0, s>>>(
                dshots, b, s0, ns, ho[b].tape, P.ncell, ix, (const int *)R.d_idx + P.idxm0);
            ++*launches;
          }
          if (P.image) {
            const long long np = (long long)hs[b].g.nz * hs[b].g.nx;
            k_oc_image<<<(unsigned)((np + 255) / 256), 256, 0, s>>>(dshots, b, s0, ns, ho[b].bsnap);
            ++*launches;
          }
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(c, e, "on-chip launches");
      }
    }
    return SW_OK;
  };
  st = run();
  for (auto &q : ev)
    if (q) cudaEventDestroy(q);
  return st;
}

}  // namespace swave
