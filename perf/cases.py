"""The work that this framework is measured by: one call (or one job) of the
public Python API per case, from the smallest modelling run to surveys that
fill the device, in 2D and 3D, forward and adjoint, plus the preconditioner
network and the trace band-pass.

Sizes are those of the repository's own configurations and tests: the
60 x 80 parity model, the 201 x 401 layered model, the 751 x 2301 batched RTM
survey, the 1201 x 3401 Born grid, the 301 x 901 FWI models, the
200 x 400 x 400 survey in 3D and its 100 x 200 x 200 training models.
Records are cut to a few hundred or thousand samples.

Velocities are layered, dipping models with correlated noise between 1500
and 4700 m/s; recorded data are sparse spikes convolved with the Ricker
wavelet.  Everything follows from the seed alone.
"""
import math

import numpy as np
import torch

import seismic_gb300 as sw

LSINC, SNAPI = 7, 4
CH = (2, 32, 32, 32, 1)
_CTX = []


def _ctx():
    """The program's one context."""
    if not _CTX:
        _CTX.append(sw.Context(0))
    return _CTX[0]


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # The smallest call: one shot on a test-sized model (launch latency).
        {"name": "shot2d_small", "op": "model", "nz": 60, "nx": 80, "ny": 1, "d": 10.0,
         "dt": 1.5e-3, "nt": 300, "ntaper": 10, "nrec": 80, "f0": 12.0, "vmax": 2600.0,
         "rho": False},
        # The plain 2D modelling configuration, whole record.
        {"name": "shot2d_layers", "op": "model", "nz": 201, "nx": 401, "ny": 1, "d": 10.0,
         "dt": 1e-3, "nt": 2000, "ntaper": 40, "nrec": 401, "f0": 15.0, "vmax": 2750.0,
         "rho": False},
        # Variable-density modelling on the survey-sized 2D grid.
        {"name": "shot2d_rho", "op": "model", "nz": 751, "nx": 2301, "ny": 1, "d": 4.0,
         "dt": 3.75e-4, "nt": 500, "ntaper": 20, "nrec": 767, "f0": 20.0, "rho": True},
        # RTM of one shot on a medium grid.
        {"name": "rtm2d_shot", "op": "rtm", "nz": 301, "nx": 901, "ny": 1, "d": 10.0,
         "dt": 9e-4, "nt": 1000, "ntaper": 20, "nrec": 451, "f0": 9.0},
        # The batched RTM survey: shots of uneven aperture and record length.
        {"name": "rtm2d_survey", "op": "job", "nz": 751, "nx": 2301, "ny": 1, "d": 4.0,
         "dt": 3.75e-4, "nt": 800, "ntaper": 20, "nshot": 16, "f0": 20.0},
        # Born modelling (the forward half of least-squares RTM) on the
        # largest 2D grid.
        {"name": "born2d", "op": "born", "nz": 1201, "nx": 3401, "ny": 1, "d": 6.25,
         "dt": 5e-4, "nt": 400, "ntaper": 20, "nrec": 1701, "f0": 15.0},
        # FWI misfit and gradient of a training-model survey.
        {"name": "fwi2d_gradient", "op": "fwi", "nz": 301, "nx": 901, "ny": 1, "d": 10.0,
         "dt": 9e-4, "nt": 1000, "ntaper": 20, "nshot": 20, "f0": 6.0},
        # One shot of modelling on the 3D survey grid.
        {"name": "shot3d", "op": "model", "nz": 200, "nx": 400, "ny": 400, "d": 12.5,
         "dt": 9e-4, "nt": 200, "ntaper": 20, "nrec": 2500, "f0": 15.0, "rho": False},
        # 3D RTM of one shot on a training-model grid.
        {"name": "rtm3d_shot", "op": "rtm", "nz": 100, "nx": 200, "ny": 200, "d": 12.5,
         "dt": 9e-4, "nt": 240, "ntaper": 20, "nrec": 625, "f0": 15.0},
        # Preconditioner inference on the FWI benchmark's image.
        {"name": "cnn_forward", "op": "cnn_forward", "nz": 601, "nx": 1801},
        # Preconditioner training gradient on a batch of training images.
        {"name": "cnn_gradient", "op": "cnn_gradient", "nz": 301, "nx": 901, "batch": 2},
        # FWI preprocessing: zero-phase high-cut of one shot gather.
        {"name": "bandpass", "op": "bandpass", "ntr": 901, "nt": 2223, "dt": 1.8e-3, "fhi": 20.0},
    ]


def _logu(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["model", "model", "rho", "rtm", "lsrtm", "born", "job", "fwi", "model3d",
                     "rtm3d", "cnn_forward", "cnn_gradient", "bandpass"])
    if op == "cnn_forward":
        return {"op": op, "nz": _logu(rng, 40, 601), "nx": _logu(rng, 60, 1801)}
    if op == "cnn_gradient":
        return {"op": op, "nz": _logu(rng, 40, 400), "nx": _logu(rng, 60, 901),
                "batch": rng.randint(1, 3)}
    if op == "bandpass":
        return {"op": op, "ntr": _logu(rng, 10, 1800), "nt": rng.randint(300, 3000),
                "dt": rng.choice([9e-4, 1e-3, 1.8e-3, 2e-3]), "fhi": rng.uniform(15.0, 30.0)}
    d = rng.choice([4.0, 6.25, 10.0, 12.5])
    dt, f0 = 9e-5 * d, rng.uniform(60.0, 100.0) / d
    taper = rng.choice([10, 16, 20, 40])
    if op in ("model3d", "rtm3d"):
        nz, nx, ny = (_logu(rng, 30, hi) for hi in (160, 260, 260))
        dt = 7e-5 * d
        c = {"op": op[:-2], "nz": nz, "nx": nx, "ny": ny, "d": d, "dt": dt,
             "nt": rng.randint(60, 160), "ntaper": min(taper, 20), "nrec": _logu(rng, 30, 1500),
             "f0": f0}
        return dict(c, rho=False) if op == "model3d" else c
    nz = _logu(rng, 50, 800)
    nx = _logu(rng, 60, 2300)
    c = {"op": op, "nz": nz, "nx": nx, "ny": 1, "d": d, "dt": dt, "nt": rng.randint(200, 900),
         "ntaper": taper, "f0": f0}
    if op in ("job", "fwi"):
        return dict(c, nx=max(nx, 120), nshot=rng.randint(2, 12))
    c["nrec"] = max(8, nx // rng.choice([1, 2, 3]))
    if op in ("model", "rho"):
        c.update(op="model", rho=op == "rho")
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _noise(gen, shape, cells):
    """Correlated noise of unit variance: white noise on a grid `cells`
    coarser, interpolated linearly."""
    coarse = [max(2, -(-n // cells) + 1) for n in shape]
    v = torch.randn([1, 1] + coarse, generator=gen, dtype=torch.float64).to(_dev())
    mode = "bilinear" if len(shape) == 2 else "trilinear"
    v = torch.nn.functional.interpolate(v, size=list(shape), mode=mode, align_corners=True)[0, 0]
    return v / v.std()


def _model(c, gen, lo=1500.0, nlayers=40):
    """Dipping layers with 3 % correlated noise, (ny, nx, nz) or (nx, nz)."""
    shape, hi = [c["ny"], c["nx"], c["nz"]], c.get("vmax", 4700.0)
    dev = _dev()
    z = torch.arange(c["nz"], dtype=torch.float64, device=dev) / c["nz"]
    x = torch.arange(c["nx"], dtype=torch.float64, device=dev) / c["nx"] - 0.5
    y = torch.arange(c["ny"], dtype=torch.float64, device=dev) / c["ny"] - 0.5
    dip = torch.rand(2, generator=gen, dtype=torch.float64).tolist()
    depths = torch.sort(torch.rand(nlayers, generator=gen, dtype=torch.float64))[0].to(dev)
    jit = torch.rand(nlayers + 1, generator=gen, dtype=torch.float64).to(dev)
    vl = lo + (hi - 300.0 - lo) * torch.arange(nlayers + 1, device=dev) / nlayers + 200.0 * jit
    depth = (z[None, None, :] + 0.2 * (dip[0] - 0.5) * x[None, :, None]
             + 0.2 * (dip[1] - 0.5) * y[:, None, None])
    v = vl[torch.bucketize(depth.contiguous(), depths)]
    if c["ny"] == 1:
        v = v[0] * (1.0 + 0.03 * _noise(gen, shape[1:], 5))
    else:
        v = v * (1.0 + 0.03 * _noise(gen, shape, 5))
    return v.clamp(lo, hi).float().cpu().numpy()


def _ricker(f0, dt, nt):
    t = np.arange(nt) * dt - 1.5 / f0
    a = (math.pi * f0 * t) ** 2
    return ((1.0 - 2.0 * a) * np.exp(-a)).astype(np.float32)


def _traces(gen, ntr, nt, w):
    """Sparse spikes (3 %) convolved with the wavelet: (ntr, nt) float32."""
    s = torch.randn((ntr, nt), generator=gen) * (torch.rand((ntr, nt), generator=gen) < 0.03)
    n = 2 * nt
    out = torch.fft.irfft(torch.fft.rfft(s.to(_dev()).double(), n=n)
                          * torch.fft.rfft(torch.as_tensor(w).to(_dev()).double(), n=n), n=n)
    return (0.1 * out[:, :nt]).float().cpu().numpy()


def _receivers(c, lo, hi, nrec):
    """nrec receivers at depth index 2 on columns lo..hi (2D), or on a
    regular patch over the whole model (3D)."""
    d = c["d"]
    if c["ny"] == 1:
        rec = np.zeros((nrec, 3), np.float32)
        rec[:, 1] = np.round(np.linspace(lo, hi, nrec)) * d
    else:
        k = max(1, int(math.sqrt(nrec)))
        gx = np.round(np.linspace(4, c["nx"] - 5, k)) * d
        gy = np.round(np.linspace(4, c["ny"] - 5, max(1, nrec // k))) * d
        X, Y = np.meshgrid(gx, gy, indexing="ij")
        rec = np.zeros((X.size, 3), np.float32)
        rec[:, 1], rec[:, 2] = X.ravel(), Y.ravel()
    rec[:, 0] = d
    return rec


def _inputs(c, seed):
    """Plain arrays of one case, from the seed alone."""
    gen = torch.Generator().manual_seed(1000003 * (seed % (1 << 31)) + 17)
    s = {"case": c}
    if c["op"].startswith("cnn"):
        nb = c.get("batch", 1)
        x = torch.stack([torch.stack([_noise(gen, (c["nx"], c["nz"]), k) for k in (6, 40)])
                         for _ in range(nb)])
        x[:, 1] = x[:, 1].abs()          # the source illumination
        t = torch.stack([0.5 * v[0] + 0.1 * _noise(gen, (c["nx"], c["nz"]), 12) for v in x])
        w = []
        for a, b in zip(CH[:-1], CH[1:]):
            w += [torch.randn(9 * a * b, generator=gen) * math.sqrt(2.0 / (9 * a)),
                  0.1 * torch.randn(b, generator=gen)]
        s.update(x=x.float().cpu().numpy(), t=t.float().cpu().numpy(), w=torch.cat(w).numpy())
        return s
    if c["op"] == "bandpass":
        s["traces"] = _traces(gen, c["ntr"], c["nt"], _ricker(12.0, c["dt"], c["nt"]))
        return s
    d, nz, nx, ny, nt = c["d"], c["nz"], c["nx"], c["ny"], c["nt"]
    s["vel"] = _model(c, gen)
    s["wavelet"] = w = _ricker(c["f0"], c["dt"], nt)
    if c["op"] in ("job", "fwi"):
        r = torch.rand((c["nshot"], 2), generator=gen).tolist()
        s["shots"] = []
        for q in range(c["nshot"]):
            sx = round((q + 0.5) * (nx - 1) / c["nshot"])
            if c["op"] == "job":        # own aperture and record length
                half = int((0.16 + 0.16 * r[q][0]) * nx)
                lo, hi, step = max(0, sx - half), min(nx - 1, sx + half), 3
                n = nt - int(0.25 * nt * r[q][1])
            else:
                lo, hi, step, n = 0, nx - 1, 2, nt
            rec = _receivers(c, lo, hi, max(4, (hi - lo) // step + 1))
            s["shots"].append({"sou": np.array([d, sx * d, 0.0], np.float32), "rec": rec,
                               "data": _traces(gen, len(rec), n, w[:n])})
        return s
    s["sou"] = np.array([2.3 * d, (nx // 2 + 0.31) * d, (ny // 2 - 0.2) * d if ny > 1 else 0.0],
                        np.float32)
    s["rec"] = _receivers(c, 0, nx - 1, c["nrec"])
    if c.get("rho"):
        s["rho"] = (0.31 * s["vel"].astype(np.float64) ** 0.25).astype(np.float32)   # Gardner
    if c["op"] in ("rtm", "lsrtm"):
        s["data"] = _traces(gen, len(s["rec"]), nt, w)
    if c["op"] == "born":
        spike = torch.rand(s["vel"].shape, generator=gen) < 0.01
        s["ref"] = (0.05 * torch.randn(s["vel"].shape, generator=gen) * spike).numpy()
    return s


def _genpar(c, nt=None):
    return sw.make_genpar(c["nz"], c["nx"], c["ny"], dz=c["d"], dx=c["d"], dy=c["d"], dt=c["dt"],
                          nt=nt or c["nt"], ntaper=c["ntaper"], lsinc=LSINC, snapi=SNAPI,
                          twoD=c["ny"] == 1)


def prepare(case, seed):
    s = _inputs(case, seed)
    ctx = _ctx()
    if case["op"].startswith("cnn"):
        s["net"] = sw.CNN(ctx, CH)
        s["net"].set_weights(s["w"])
        return s
    if case["op"] == "bandpass":
        return s
    s["g"] = _genpar(case)
    if case["op"] == "job":
        s["job"] = sw.RTMJob(ctx, s["g"], s["vel"], s["wavelet"], s["shots"])
    if case["op"] == "fwi":
        for shot in s["shots"]:
            shot["dobs"] = shot.pop("data")
        s["desc"] = _fwi_desc(s["g"])
    if case.get("rho"):
        p = sw.SwPropDesc()
        p.g = s["g"]
        p.tmin, p.tmax, p.tstep = 1, case["nt"], 1
        p.fd_scheme, p.injection, p.extraction = sw.FD_FORWARD, sw.INJ_SINC, sw.EXT_SINC
        s["desc"] = p
    return s


def _fwi_desc(g):
    p = sw.SwFwiDesc()
    p.g = g
    p.illu_pow = 1.0
    p.smooth_rect1, p.smooth_rect2, p.smooth_rect3 = 3, 5, 1
    p.smooth_doz = p.smooth_dox = 1
    return p


def run(state):
    c, ctx, s = state["case"], _ctx(), state
    op = c["op"]
    if op == "cnn_forward":
        return s["net"].forward(s["x"][0])
    if op == "cnn_gradient":
        return s["net"].gradient(s["x"], s["t"])
    if op == "bandpass":
        return ctx.bandpass(s["traces"], c["dt"], fhi=c["fhi"])
    if op == "job":
        s["job"].reset()
        s["job"].run()
        return s["job"].result()
    if op == "fwi":
        return ctx.fwi_fct_gdt(s["desc"], s["vel"], s["wavelet"], s["shots"])
    if op == "model" and c["rho"]:
        data = np.zeros((len(s["rec"]), c["nt"]), np.float32)
        ctx.propagate(s["desc"], s["vel"], sou_coord=s["sou"], sou_trace=s["wavelet"],
                      rec_coord=s["rec"], rec_trace=data, rho=s["rho"])
        return data
    if op == "model":      # the gather; in 2D the final wavefield too
        return ctx.modeling(s["g"], s["vel"], s["sou"], s["wavelet"], s["rec"],
                            final_u2=c["ny"] == 1)
    if op == "born":
        return ctx.born(s["g"], s["vel"], s["ref"], s["sou"], s["wavelet"], s["rec"])
    call = ctx.rtm if op == "rtm" else ctx.lsrtm
    return call(s["g"], s["vel"], s["sou"], s["wavelet"], s["rec"], s["data"])


def work(case):
    """Bytes and operations of one pass.  Propagation: per time step and
    compute-domain point four levels and the velocity read and one level
    written (24 B; 32 B with density), plus saved and read snapshots; the
    network: every layer's BF16 activations once in and once out."""
    c, op = case, case["op"]
    if op == "bandpass":
        n = c["ntr"] * c["nt"]
        return {"bytes": 8.0 * n, "flops": 2 * 4 * 9.0 * n}
    if op.startswith("cnn"):
        npix = c["nz"] * c["nx"] * c.get("batch", 1)
        act, mac = 0, 0
        for a, b in zip(CH[:-1], CH[1:]):
            act += 2 * (max(a, 16) + max(b, 16))
            mac += 9 * a * b
        k = 1 if op == "cnn_forward" else 3
        return {"bytes": float(k * npix * act), "flops": 2.0 * k * npix * mac}
    dims = 2 if c["ny"] == 1 else 3
    pad = 2 * c["ntaper"]

    def points(nx):
        return (c["nz"] + pad) * (nx + pad) * (1 if dims == 2 else c["ny"] + pad)

    per = 32 if c.get("rho") else 24
    flop = 60 if c.get("rho") else 17 + 13 * dims
    if op == "model":
        n = points(c["nx"]) * c["nt"]
        return {"bytes": float(per * n), "flops": float(flop * n)}
    phys, nxw, nshot = c["nz"] * c["nx"] * c["ny"], c["nx"], c.get("nshot", 1)
    nt = c["nt"]
    if op == "job":     # mean aperture (cut at the model's ends) and record
        nxw, nt = 0.45 * c["nx"], 0.875 * c["nt"]
        phys = c["nz"] * nxw
    n = 2 * points(nxw) * nt * nshot
    snaps = phys * (nt // SNAPI) * nshot
    return {"bytes": float(per * n + snaps * (12 if op == "born" else 24)),
            "flops": float(flop * n + 6 * snaps)}


# ---------------------------------------------------------------------------
# The same results in 64 bits, in plain torch
# ---------------------------------------------------------------------------
_C2 = (-205.0 / 72.0, 8.0 / 5.0, -1.0 / 5.0, 8.0 / 315.0, -1.0 / 560.0)
_C1 = (1225.0 / 1024.0, -1225.0 / (1024.0 * 15), 1225.0 / (1024.0 * 125), -1225.0 / (1024.0 * 1715))


def _sinc(n, shift):
    k = np.arange(1, n + 1)
    h = n // 2
    fact = np.where(k <= int(h + 1 + shift), (k - 1 - shift) / h, (n - k + shift) / h)
    fact = np.maximum(fact, 0.0)
    pos = math.pi * (k - (h + 1) - shift)
    safe = np.where(np.abs(pos) > 0.005, pos, 1.0)
    s = np.where(np.abs(pos) > 0.005, fact * np.sin(safe) / safe, fact * (1 - pos * pos / 6))
    return s / s.sum()


class _Wave:
    """The propagator on one padded grid, arrays [y][x][z] in 64 bits."""

    def __init__(self, c, vel, rho=None):
        self.c, self.dev = c, _dev()
        self.three = c["ny"] > 1
        self.pad = c["ntaper"] + 4
        p, q = self.pad, self.pad if self.three else 0
        v = torch.as_tensor(vel).to(self.dev).double().reshape(c["ny"], -1, c["nz"])
        self.phys = v
        self.nx = v.shape[1]
        # The three axes' ranges of the physical and of the compute domain.
        self.P = (slice(q, q + c["ny"]), slice(p, p + self.nx), slice(p, p + c["nz"]))
        self.v = self._edges(v, p, q)
        h = 4 if self.three else 0
        self.core = tuple(slice(b, n - b) for b, n in zip((h, 4, 4), self.v.shape))
        self.v2 = self.v * self.v
        self.lev = [torch.zeros_like(self.v) for _ in range(5)]
        self.axes = (2, 1, 0) if self.three else (2, 1)
        self.lines = {a: [self._line(a, o) for o in (False, True)] for a in self.axes}
        self.rho = None
        if rho is not None:
            self.rho_phys = torch.as_tensor(rho).to(self.dev).double().reshape(v.shape)
            self.rho = self._edges(self.rho_phys, p, q)
            r = self.rho
            for a in self.axes:
                k = torch.arange(r.shape[a], device=self.dev)
                r = sum(t * r.index_select(a, (k + l - 4).clamp(0, r.shape[a] - 1))
                        for l, t in enumerate(_sinc(9, 0.5)))
            self.delp = 1.0 / r

    @staticmethod
    def _edges(v, p, q):
        for a, n in ((2, p), (1, p), (0, q)):
            if n:
                k = torch.arange(-n, v.shape[a] + n, device=v.device).clamp(0, v.shape[a] - 1)
                v = v.index_select(a, k)
        return v

    def _line(self, a, far):
        """Higdon edge of one side of axis a as a matrix: 8 outputs from the
        two u3 values inside, 10 of u2 and 10 of u1, innermost first."""
        n = self.v.shape[a]
        pos = [n - 1 - k if far else k for k in range(9, -1, -1)]     # two inside .. outermost
        edge = [s for s in self.core]
        edge[a] = slice(n - 5, n - 4) if far else slice(4, 5)
        nu = (self.v[tuple(edge)] * self.c["dt"] / self.c["d"]).movedim(a, -1)
        w = 0.5

        def one(beta):
            f = (beta + nu) * (1 - w)
            return (w * (beta + nu) - nu) / f, (w * (beta + nu) - beta) / f, w / (w - 1.0)

        (qx, qt, qxt), (rx, rt, rxt) = one(1.0), one(0.7)
        k = [qx + rx, qx * rx, qt + rt, qx * rt + qt * rx + qxt + rxt, qx * rxt + rx * qxt,
             qt * rt, qt * rxt + rt * qxt, qxt * rxt * torch.ones_like(nu)]
        eye = torch.eye(22, dtype=torch.float64, device=self.dev)
        # pos[0], pos[1]: two and one inside; eye rows 0, 1: u3 there.
        a1, a2, rows = eye[1], eye[0], []
        for m in range(8):
            r = -(k[0] * a1 + k[1] * a2 + k[2] * eye[2 + m + 2] + k[3] * eye[2 + m + 1]
                  + k[4] * eye[2 + m] + k[5] * eye[12 + m + 2] + k[6] * eye[12 + m + 1]
                  + k[7] * eye[12 + m])
            rows.append(r)
            a2, a1 = a1, r
        ix = torch.tensor(pos, device=self.dev)
        return ix, torch.stack(rows, -2)

    def _lap(self, u):
        out = None
        for a in self.axes:
            sc = 1.0 / self.c["d"] ** 2
            for l, t in enumerate(_C2):
                for sgn in ((0,) if l == 0 else (1, -1)):
                    sl = list(self.core)
                    sl[a] = slice(sl[a].start + sgn * l, sl[a].stop + sgn * l)
                    if out is None:
                        out = u[tuple(sl)] * (t * sc)
                    else:
                        out.add_(u[tuple(sl)], alpha=t * sc)
        return out

    def _div_rho(self, u):
        """v^2 rho div(grad u / rho): differences at half cells, first order
        (with the face's 1/rho) in the three cells beyond each face, zero in
        the fourth."""
        total = None
        for a in self.axes:
            n, o = u.shape[a], 1.0 / self.c["d"]
            sl = list(self.core)
            sl[a] = slice(None)
            x, dp = u[tuple(sl)].movedim(a, -1), self.delp[tuple(sl)].movedim(a, -1)
            g = torch.zeros_like(x)
            g[..., 4:n - 4] = dp[..., 4:n - 4] * o * sum(
                t * (x[..., 5 + l:n - 3 + l] - x[..., 4 - l:n - 4 - l]) for l, t in enumerate(_C1))
            for r, f in ((slice(1, 4), 4), (slice(n - 4, n - 1), n - 5)):
                g[..., r] = o * (x[..., r.start + 1:r.stop + 1] - x[..., r]) * dp[..., f:f + 1]
            div = o * sum(t * (g[..., 4 + l:n - 4 + l] - g[..., 3 - l:n - 5 - l])
                          for l, t in enumerate(_C1))
            div = div.movedim(-1, a)
            total = div if total is None else total + div
        return total * self.v2[self.core] * self.rho[self.core]

    def nodes(self, coord, mode):
        """Flat indices into the padded array and weights (n, taps), and the
        nearest physical node of n points."""
        c, d = self.c, self.c["d"]
        co = np.asarray(coord, np.float64).reshape(-1, 3)
        n = np.floor(co / d + 0.5).astype(int)
        if not self.three:
            n[:, 2] = 0
        off = (co - n * d) / d
        h = LSINC // 2 if mode == "sinc" else 0
        k = np.arange(-h, h + 1)
        iz = n[:, 0, None] + k + self.P[2].start
        ix = n[:, 1, None] + k + self.P[1].start
        if mode == "sinc":
            wz = np.stack([_sinc(LSINC, o) for o in off[:, 0]])
            wx = np.stack([_sinc(LSINC, o) for o in off[:, 1]])
        else:
            wz = wx = np.ones((len(n), 1))
        iy, wy = ((n[:, 2, None] + k + self.P[0].start, wx) if self.three
                  else (np.zeros((len(n), 1), int), np.ones((len(n), 1))))
        sh = self.v.shape
        idx = (iy[:, :, None, None] * sh[1] + ix[:, None, :, None]) * sh[2] + iz[:, None, None, :]
        wgt = wy[:, :, None, None] * wx[:, None, :, None] * wz[:, None, None, :]
        t = lambda a: torch.as_tensor(a.reshape(len(n), -1)).to(self.dev)  # noqa: E731
        near = tuple(torch.as_tensor(n[:, a]).to(self.dev) for a in (2, 1, 0))
        return t(idx), t(wgt), near

    def run(self, nt, back=False, adjoint=False, inject=None, extract=None, on_step=None,
            source=None):
        """inject: (idx, weights (n, taps), traces (n, nt)); extract the same
        with the traces to fill; on_step(it, u2), source(it) -> addend on the
        physical domain."""
        k12 = 12.0 * self.c["dt"] ** 2
        um1, u0, u1, u2, u3 = self.lev
        rel = tuple(slice(p.start - q.start, p.stop - q.start) for p, q in zip(self.P, self.core))
        for it in (range(nt, 0, -1) if back else range(1, nt + 1)):
            if extract:
                extract[2][:, it - 1] += (u2.view(-1)[extract[0]] * extract[1]).sum(1)
            if on_step and it % SNAPI == 0:
                on_step(it, u2[self.P])
            if self.rho is not None:
                sv = self._div_rho(u2)
            elif adjoint:
                sv = self._lap(self.v2 * u2)
            else:
                sv = self._lap(u2) * self.v2[self.core]
            if inject:
                full = torch.zeros_like(u3)
                full.view(-1).index_add_(0, inject[0].reshape(-1),
                                         (inject[1] * inject[2][:, it - 1:it]).reshape(-1))
                sv += full[self.core]
            if source and it % SNAPI == 0:
                sv[rel] += source(it)
            k = self.core
            u3[k] = (20.0 * u2[k] - 6.0 * u1[k] - 4.0 * u0[k] + um1[k] + k12 * sv) / 11.0
            for a in self.axes:
                for ix, mat in self.lines[a]:
                    sl = list(self.core)
                    sl[a] = slice(None)
                    pick = lambda u, q: u[tuple(sl)].index_select(a, q).movedim(a, -1)  # noqa: E731,B023
                    vec = torch.cat([pick(u3, ix[:2]), pick(u2, ix), pick(u1, ix)], -1)
                    out = (mat * vec[..., None, :]).sum(-1)
                    u3[tuple(sl)] = u3[tuple(sl)].index_copy(a, ix[2:], out.movedim(-1, a))
            um1, u0, u1, u2, u3 = u0, u1, u2, u3, um1
        return u2


def _taper(nx, ny, dev):
    def one(n):
        m, t = min(n // 2, 10), np.ones(n)
        for i in range(1, min(m, n) + 1):
            t[i - 1] = math.sin(math.pi * (i - 1) / (2 * (m - 1))) ** 2
        i0 = max(1, n - m)
        for i in range(i0, n + 1):
            t[i - 1] = math.cos(math.pi * (i - i0) / (2 * m)) ** 2
        return t
    ty = one(ny) if ny > 1 else np.ones(1)
    return torch.as_tensor(ty[:, None, None] * one(nx)[None, :, None]).to(dev)


def _tr(a, dev):
    return torch.as_tensor(np.atleast_2d(a)).to(dev).double()


def _two_pass(c, op, vel, sou, w, rec, data, nt, ref=None):
    """Forward pass with snapshots, then the backward or Born pass."""
    f = _Wave(c, vel)
    dev, nx = f.dev, f.nx
    snaps = torch.zeros((max(1, nt // SNAPI),) + tuple(f.phys.shape), dtype=torch.float64, device=dev)

    def save(it, u):
        snaps[it // SNAPI - 1] = u

    i, k, n = f.nodes(sou, "sinc")
    res = torch.zeros((len(rec), nt), dtype=torch.float64, device=dev)
    ex = None
    if op == "fwi":
        ri, rk, _ = f.nodes(rec, "node")
        ex = (ri, rk, res)
    f.run(nt, inject=(i, k * f.phys[n][:, None] ** 2, _tr(w[:nt], dev)), on_step=save, extract=ex)
    tap = _taper(nx, c["ny"], dev)
    vol = c["d"] ** (3 if f.three else 2)
    f.lev = [torch.zeros_like(f.v) for _ in range(5)]
    ri, rk, n = f.nodes(rec, "node" if op == "fwi" else "sinc")
    if op == "born":
        r = torch.as_tensor(ref).to(dev).double().reshape(f.phys.shape)
        f.run(nt, extract=(ri, rk / vol, res),
              source=lambda it: 2.0 * tap * r * snaps[it // SNAPI - 1] / f.phys)
        return res
    image, illum = torch.zeros_like(f.phys), torch.zeros_like(f.phys)
    ns = nt // SNAPI
    dobs = _tr(data, dev)
    if op == "fwi":
        dobs = dobs - res
    d2 = (c["dt"] * SNAPI) ** 2

    def img(it, u):
        m = it // SNAPI - 1
        if m < 0 or m >= ns:
            return
        s = snaps[m]
        if op == "rtm":
            image.add_(u * s * tap)
        elif op == "lsrtm":
            image.add_(2.0 * tap * u * s / f.phys)
        else:
            second = snaps[max(m - 1, 0)] - 2.0 * s + snaps[min(m + 1, ns - 1)]
            image.add_(u * second / (d2 * f.phys ** 3) * tap)
        illum.add_(s * s * tap)

    wgt = rk / vol if op == "lsrtm" else rk * f.phys[n][:, None] ** 2
    f.run(nt, back=True, adjoint=op == "lsrtm" or (op == "rtm" and not f.three),
          inject=(ri, wgt, dobs), on_step=img)
    return image, illum, dobs


def _window(c, shot):
    cols = np.concatenate([shot["rec"][:, 1], shot["sou"][1:2]]) / c["d"]
    return int(round(cols.min())), int(round(cols.max())) + 1


def _shift(coord, c, lo):
    co = np.array(coord, np.float64).reshape(-1, 3)
    co[:, 1] -= lo * c["d"]
    return co


def _triangle(g, nr, axis):
    """triangle smoothing of radius nr along an axis with folded ends."""
    x = g.movedim(axis, 0)
    n = x.shape[0]
    k = torch.cat([torch.arange(1, nr + 1), torch.arange(nr - 1, 0, -1)]).double() / nr ** 2
    full = torch.zeros((n + 2 * nr - 2,) + tuple(x.shape[1:]), dtype=x.dtype, device=x.device)
    for j, w in enumerate(k.tolist()):
        full[j:j + n] += w * x
    out = full[nr - 1:nr - 1 + n].clone()
    for i in range(1, nr):
        out[i - 1] += full[nr - 1 - i]
        out[n - i] += full[n + nr - 2 + i]
    return out.movedim(0, axis)


def _norm(im, il):
    il = (il + il.max() / 10000.0) / torch.sqrt((il * il).mean())
    return im / il, il


def exact(case, seed):
    c, s, dev = case, _inputs(case, seed), _dev()
    op = c["op"]
    flat = lambda t: t.reshape(-1).cpu().numpy()  # noqa: E731
    if op.startswith("cnn"):
        return _exact_cnn(c, s)
    if op == "bandpass":
        return _exact_bandpass(c, s["traces"])
    if op == "model":
        f = _Wave(c, s["vel"], s.get("rho"))
        i, k, n = f.nodes(s["sou"], "sinc")
        v2 = f.phys[n][:, None] ** 2 * (f.rho_phys[n][:, None] if f.rho is not None else 1.0)
        ri, rk, n = f.nodes(s["rec"], "sinc")
        data = torch.zeros((len(s["rec"]), c["nt"]), dtype=torch.float64, device=dev)
        vr = f.phys[n][:, None]
        u = f.run(c["nt"], inject=(i, k * v2, _tr(s["wavelet"], dev)),
                  extract=(ri, rk * (vr if f.three else vr * vr), data))
        data = data.cpu().numpy()
        return data if c["rho"] or f.three else (data, u.cpu().numpy())
    if op == "born":
        return _two_pass(c, op, s["vel"], s["sou"], s["wavelet"], s["rec"], None, c["nt"],
                         s["ref"]).cpu().numpy()
    if op in ("rtm", "lsrtm"):
        a, b, _ = _two_pass(c, op, s["vel"], s["sou"], s["wavelet"], s["rec"], s["data"], c["nt"])
        return flat(a), flat(b)
    image = torch.zeros((c["nx"], c["nz"]), dtype=torch.float64, device=dev)
    illum, f, ntr = torch.zeros_like(image), 0.0, 0
    for shot in s["shots"]:
        lo, hi = _window(c, shot)
        nt = shot["data"].shape[1]
        a, b, r = _two_pass(c, "rtm" if op == "job" else op, s["vel"][lo:hi],
                            _shift(shot["sou"], c, lo), s["wavelet"], _shift(shot["rec"], c, lo),
                            shot["data"], nt)
        image[lo:hi] += a[0]
        illum[lo:hi] += b[0]
        f += float((r * r).sum()) / 2
        ntr += len(shot["rec"])
    if op == "job":
        return flat(image), flat(illum), flat(_norm(image, illum)[0])
    scale = 2.0 * c["nt"] * ntr
    g, il = _norm(2.0 * image / scale, illum)
    g = _triangle(_triangle(g, 5, 0), 3, 1)
    return f / scale, flat(g), flat(il)


def _exact_cnn(c, s):
    w = torch.as_tensor(s["w"]).to(_dev()).double()
    w.requires_grad_(c["op"] == "cnn_gradient")
    x = torch.as_tensor(s["x"]).to(_dev()).double()
    o, h = 0, x
    for l, (a, b) in enumerate(zip(CH[:-1], CH[1:])):
        k = w[o:o + 9 * a * b].reshape(b, 3, 3, a).permute(0, 3, 1, 2)
        o += 9 * a * b
        h = torch.nn.functional.conv2d(h, k, w[o:o + b], padding=1)
        o += b
        h = torch.relu(h) if l + 2 < len(CH) else h
    if c["op"] == "cnn_forward":
        return h[0, 0].cpu().numpy()
    loss = 0.5 * ((h[:, 0] - torch.as_tensor(s["t"]).to(_dev()).double()) ** 2).mean((1, 2)).mean()
    loss.backward()
    return w.grad.cpu().numpy(), float(loss)


def _exact_bandpass(c, traces):
    """Zero-phase Butterworth high-cut of 14 poles (7 each way), 10 samples
    of squared-sine ramps at both ends."""
    pad, a = 10, 2.0 * math.tan(math.pi * c["fhi"] * c["dt"])
    aa, sec = a * a, [(a / (a + 2), a / (a + 2), 0.0, (a - 2) / (a + 2), 0.0)]
    for j in range(1, 4):
        q = 4.0 * a * math.cos(j * math.pi / 7)
        b = aa / (aa + 4 + q)
        sec.append((b, 2 * b, b, (2 * aa - 8) / (aa + 4 + q), (aa + 4 - q) / (aa + 4 + q)))
    x = np.asarray(traces, np.float64).T
    k = np.arange(pad)
    ramp = np.sin(k * math.pi / (2 * (pad - 1)))[:, None] ** 2
    x = np.concatenate([x[:1] * ramp, x, x[-1:] * ramp[::-1]])
    for _ in range(2):
        for c0, c1, c2, c3, c4 in sec:
            y = np.zeros_like(x)
            for i in range(2, len(x)):
                y[i] = c0 * x[i] + c1 * x[i - 1] + c2 * x[i - 2] - c3 * y[i - 1] - c4 * y[i - 2]
            x = y
        x = np.concatenate([np.zeros((2, x.shape[1])), x[:1:-1]])
    return x[pad:pad + c["nt"]].T.copy()
