"""Timed cases of the tracer transport step: what a host model asks of it.

Five ways of calling it, each through ems_b200.gpu.TracerStep (a thin binding
of the C ABI in include/shoc_tr_gpu.h):

  hour    tracers resident on the GPU: `steps` steps on one flow field, the
          status read back, then the tracers handed over -- to another
          component on the same GPU as a device buffer (the halo entry point
          with every wet cell in its plan), or, for the compensated
          precision, which that entry point does not take, to the host
  tide    a short forecast from uploaded tracers with a new flow every step:
          velocities, diffusivity and surface uploaded, the transport-mode
          preamble on the device, one step; two flood and two ebb steps, the
          surface moving through a layer face on a part of the basin; then
          the hand-over of `hour`
  dropin  one step on host arrays, copies included: the call SHOC makes in
          place of its own advect_diffuse + vert_diffuse_3d
  batch   `hour` on several independent basins in one window, each with its
          own depth and number of tracers
  solve   the closures' tridiagonal solve on host arrays

A case's basin (ems_b200.synth) is the same for every seed, as a user's is;
the strength of the flow, the mixing and the tracer fields come from the seed.
Host arrays that cross the link every call are page-locked, as the library's users do.

exact() restates the step in plain torch, in 64 bits, from the window's maps
and the inputs alone.
"""
import copy
import functools
import math

import numpy as np
import torch

from ems_b200 import _abi, gpu, synth

PRECISION = {"fp64": gpu.FP64, "mixed": gpu.FP32_MIXED, "comp": gpu.FP32_COMP}
SCHEME = {"quickest": 0x20, "vanleer": 0x80, "order1": 0x2, "order2": 0x4, "order4": 0x10,
          "quickest_co": 0x40, "order2_uw": 0x2000}


def _case(name, call, precision, nx, ny, nz, ntr, steps=1, dt=60.0, scheme="quickest",
          ultimate=1, hdiff=0, layers="uniform", scale=0.0):
    return dict(name=name, call=call, precision=precision, nx=nx, ny=ny, nz=nz, ntr=ntr,
                steps=steps, dt=dt, scheme=scheme, ultimate=ultimate, hdiff=hdiff, layers=layers,
                scale=scale)


def listed():
    return [
        # a test basin stepped from the host model: latency of one call
        _case("small_dropin_fp64", "dropin", "fp64", 20, 14, 6, 3),
        # a teaching-size basin, one tracer: launches and gaps between them
        _case("basin64_fp64", "hour", "fp64", 64, 64, 20, 1, steps=10),
        # a coastal model in the reference's own precision
        _case("coast_fp64", "hour", "fp64", 384, 320, 40, 10, steps=4),
        # the same kind of model as a drop-in: the host link counts
        _case("coast_dropin_fp64", "dropin", "fp64", 256, 256, 40, 10),
        # a large shelf model with thin surface layers, the fast precision
        _case("shelf_mixed", "hour", "mixed", 1024, 512, 50, 24, steps=6, layers="stiff"),
        # the accurate FP32 precision on a long interval between outputs
        _case("shelf_comp", "hour", "comp", 448, 300, 50, 16, steps=30, layers="stiff"),
        # the other limiter, with horizontal diffusion, on an odd-sized strait
        _case("strait_vanleer_mixed", "hour", "mixed", 333, 217, 37, 5, steps=8,
              scheme="vanleer", hdiff=1),
        # an ensemble of small basins in one window
        _case("batch_mixed", "batch", "mixed", 0, 0, 60, 32, steps=6, scale=0.125),
        # a tidal estuary: a new flow each step, columns whose surface changes layer
        _case("tide_fp64", "tide", "fp64", 192, 160, 24, 6, steps=4, layers="stiff"),
        # a second-order upwind run
        _case("upwind_fp64", "hour", "fp64", 200, 180, 30, 6, steps=2, scheme="order2_uw"),
        # a long step that takes several sub-steps, called from the host model
        _case("substeps_dropin_mixed", "dropin", "mixed", 300, 257, 33, 8, dt=300.0),
        # a turbulence closure's solve
        _case("closure_solve", "solve", "fp64", 256, 256, 40, 1),
    ]


def draw(rng):
    def logi(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    call = rng.choices(["hour", "dropin", "tide", "batch", "solve"], [50, 22, 14, 7, 7])[0]
    nz = rng.randint(4, 60)
    if call == "batch":
        return pure(_case("", call, rng.choice(["fp64", "mixed", "comp"]), 0, 0, 60, 32,
                          steps=rng.randint(1, 4), scale=round(rng.uniform(0.03, 0.11), 4)))
    if call == "solve":
        return pure(_case("", call, "fp64", logi(16, 400), logi(16, 300), nz, 1))
    precision = rng.choice(["fp64", "mixed", "comp"])
    scheme = rng.choice(["quickest"] * 5 + ["vanleer"] * 2 + ["order1", "order2", "order4",
                                                              "quickest_co", "order2_uw"])
    fast = scheme in ("quickest", "vanleer")
    # values of all tracers of the window times steps: at most about 4e8 (1e7
    # where every column takes the general path or the host link counts)
    cap = {"hour": 2e8 if fast else 1e7, "dropin": 5e7 if fast else 1e7, "tide": 4e7}[call]
    while True:
        nx, ny, ntr = logi(16, 800), logi(16, 500), logi(1, 32)
        steps = rng.randint(1, 24) if call == "hour" else 4 if call == "tide" else 1
        if 4e3 <= nx * ny * nz * ntr * steps <= cap:
            break
    # the centred schemes are run with the limiter, and long steps (several
    # sub-steps) with the limited upwind ones: the others grow without bound
    ultimate = {"quickest": rng.choice([0, 1, 1, 1]), "vanleer": rng.randint(0, 1),
                "order1": 0, "order2_uw": rng.randint(0, 1)}.get(scheme, 1)
    return pure(_case("", call, precision, nx, ny, nz, ntr, steps=steps,
                      dt=rng.choice([30.0, 60.0, 90.0] + [200.0] * (fast and ultimate)),
                      scheme=scheme, ultimate=ultimate,
                      hdiff=rng.choice([0, 0, 1]) if call != "tide" else 0,
                      layers=rng.choice(["uniform", "stiff"]) if nz >= 20 else "uniform"))


def pure(c):
    return {k: v for k, v in c.items() if k != "name"}


# ---------------------------------------------------------------------------
# inputs


@functools.lru_cache(maxsize=2)
def _basin(key):
    """The window of a case with a base flow and base tracers (synth.Case)."""
    c = dict(key)
    if c["call"] == "batch":
        return synth.build_batch("batch", synth.BATCH8, seed=2048, scale=c["scale"], umax=1.0)
    nz, ntr = c["nz"], c["ntr"]
    depth = min(250.0, 5.0 * nz)
    tide = c["call"] == "tide"
    if c["layers"] == "stiff":
        z = synth.stiff_layers(nz, depth)
    else:
        z = synth.uniform_layers(nz, depth)
    z = z + (1.5 if tide else 0.0)  # the tide's range lies inside the thin layers
    case = synth.build_case(
        "case", c["nx"], c["ny"], z, seed=2048, ntr=ntr, dt=c["dt"],
        depth=(4.0 if tide else 2.0, depth - 2.0), land_frac=0.3,
        cell=(200.0, 900.0) if c["layers"] == "stiff" else (150.0, 150.0),
        curvilinear=c["layers"] == "stiff", umax=1.0, baroclinic=0.05,
        kz=("logu", 1e-6, 1e-1), tracers=("logn", 1e-2, 1e2), trasc=SCHEME[c["scheme"]],
        ultimate=c["ultimate"],
        hdiff=(20.0, [1] * ntr) if c["hdiff"] else None)
    return case


def _build(c, seed):
    """The inputs of a seed on the case's basin (synth.Case): the flow at 0.75
    to 1 of the base one, the diffusivity times one log-uniform factor per
    column, each tracer times a smooth field of its own."""
    base = _basin(tuple(sorted(dict(c, steps=1, precision="").items())))
    case, w = copy.copy(base), base.win
    r = np.random.default_rng(int(seed))
    n = min(w.sgsizS, len(w.s2i))
    x = (w.s2i[:n] + 0.5) / w.nx
    y = (w.s2j[:n] + 0.5) / w.ny
    m2d = torch.from_numpy(w.m2d.astype(np.int64)).clamp(0, w.sgsizS - 1)

    def per_column(f):
        """f [n] by 2D cell -> by cell [sgsiz]"""
        a = np.ones(w.sgsizS)
        a[:n] = f
        return torch.from_numpy(a)[m2d]

    q = r.uniform(0.75, 1.0)
    for name in ("u1", "u2", "u1flux3d", "u2flux3d", "w"):
        setattr(case, name, getattr(base, name) * q)
    case.Kz = (torch.from_numpy(base.Kz) * per_column(np.exp(r.uniform(-2.0, 1.0, n)))).numpy()
    tr = torch.empty((base.ntr, w.sgsiz), dtype=torch.float64)
    for i in range(base.ntr):
        kx, ky, p, a = r.uniform(1.0, 12.0), r.uniform(1.0, 12.0), r.uniform(0, 6.28), \
            r.uniform(0.2, 0.8)
        torch.mul(torch.from_numpy(base.tr[i]), per_column(1.0 + a * np.cos(kx * x + ky * y + p)),
                  out=tr[i])
    case.tr = tr.numpy()
    if c["call"] == "tide":
        # low water leaves 0.15 to 0.33 m in the surface layer (its faces at 0
        # and 0.5 m); high water adds 2 to 10 cm, and on one patch of the basin
        # enough to reach 0.15 m into the layer above
        p, q, x0, y0 = *r.uniform(0.0, 6.28, 2), *r.uniform(0.3, 0.7, 2)
        low = 0.24 + 0.09 * np.cos(3.0 * x + 2.0 * y + p)
        patch = (x - x0) ** 2 + (y - y0) ** 2 < 0.15 ** 2
        up = 0.06 + 0.04 * np.cos(2.0 * x - 3.0 * y + q)
        case.levels = [np.zeros(w.sgsizS) for _ in range(3)]
        for a, v in zip(case.levels, (low, np.where(patch, 0.4, low + 0.5 * up),
                                      np.where(patch, 0.65, low + up))):
            a[:n] = v
        case.flood, case.ebb = (case.u1, case.u2), (-case.u1, -case.u2)
        case.oldeta = case.eta = case.levels[0]
        case.sur_t, case.nsur_t = w.init_surface(case.eta)
    else:
        case.eta, case.oldeta = base.eta.copy(), base.oldeta.copy()
    return case


def _tide_steps(case):
    """Velocities, old and new surface of each step of a tide pass."""
    low, mid, high = case.levels
    return ((*case.flood, low, mid), (*case.flood, mid, high), (*case.ebb, high, mid),
            (*case.ebb, mid, low))


def _solve_inputs(c, seed):
    case = _build(c, seed)
    r = np.random.default_rng(int(seed) + 17)
    S = case.win.sgsiz
    lo, up = -r.uniform(0.01, 2.0, S), -r.uniform(0.01, 2.0, S)
    return case, dict(Cd=0.5 - lo - up, Cm1=lo, Cp1=up, rhs=r.uniform(-1.0, 5.0, S),
                      var=r.uniform(0.0, 1.0, S))


class State:
    """What the host program keeps between calls: the handle, its host arrays
    (page-locked) and the device buffer a pass hands over."""

    def __init__(self, c, seed):
        self.c = c
        self.pin = None
        arrays = []
        if c["call"] == "solve":
            self.case, self.a = _solve_inputs(c, seed)
            self.step = gpu.TracerStep(self.case, PRECISION[c["precision"]])
            self.step.set_flow(self.case.sur_t, self.case.nsur_t)
            self.step.sync()
            self.x = np.zeros(self.case.win.sgsiz)
            arrays = list(self.a.values()) + [self.x]
        else:
            self.case = case = _build(c, seed)
            self.step = gpu.TracerStep(case, PRECISION[c["precision"]])
            if c["call"] == "dropin":
                self.tr, self.sur, self.nsur = case.copy_state()
                arrays = [self.tr, case.u1, case.u2, case.w, case.u1flux3d, case.u2flux3d,
                          case.Kz, case.eta, case.oldeta]
                if c["hdiff"]:
                    case.dzu1, case.dzu2 = case.dzu1.copy(), case.dzu2.copy()
                    case.u1kh, case.u2kh = case.u1kh.copy(), case.u2kh.copy()
                    arrays += [case.dzu1, case.dzu2, case.u1kh, case.u2kh]
            else:
                self.step.start()
                self.step.sync()
                if c["call"] == "tide":
                    self.tr = case.tr
                    arrays = [self.tr, *case.flood, *case.ebb, case.Kz, *case.levels]
                if c["precision"] == "comp":
                    self.out = np.zeros((case.ntr, case.win.sgsiz))
                    arrays.append(self.out)
                else:
                    cells = np.ascontiguousarray(case.win.wet_cells(), np.int32)
                    self.step.halo_plan(cells, np.zeros(0, np.int32))
                    self.out = torch.empty(
                        (case.ntr, len(cells)), device="cuda",
                        dtype=torch.float64 if c["precision"] == "fp64" else torch.float32)
                    torch.cuda.synchronize()  # the handle writes it on its own stream
            case.tr = None  # the handle (or self.tr) has them
        self.pin = gpu.HostPinned(arrays)

    def __del__(self):
        if getattr(self, "step", None) is not None:
            self.step.close()
        if getattr(self, "pin", None) is not None:
            self.pin.close()


def prepare(case, seed):
    return State(case, seed)


# ---------------------------------------------------------------------------
# one pass


def _hand_over(s):
    s.step.sync()
    if s.c["precision"] == "comp":
        return s.step.download(s.out)
    s.step.halo_pack(s.out.data_ptr())
    return s.out


def run(state):
    s, call = state, state.c["call"]
    if call == "dropin":
        s.step.step(s.tr, s.sur, s.nsur)
        return {"tr": s.tr, "sur": s.sur, "nsur": s.nsur}
    if call == "solve":
        a = s.a
        np.copyto(s.x, a["var"])
        s.step.tridiag(a["Cd"], a["Cm1"], a["Cp1"], a["rhs"], s.x, 1e-6)
        return s.x
    if call == "tide":
        k = s.case
        s.step.upload(s.tr)
        for u1, u2, old, new in _tide_steps(k):
            k.u1, k.u2, k.oldeta, k.eta = u1, u2, old, new
            s.step.set_flow()
            s.step.set_preamble(True, (new - old) / k.dt)
            s.step.run(1)
        return _hand_over(s)
    s.step.run(s.c["steps"])
    return _hand_over(s)


# ---------------------------------------------------------------------------
# what a pass cannot do without


@functools.lru_cache(maxsize=None)
def _sizes(key):
    c = _build(dict(key), 1)
    return c.win.sgsiz, c.nwet, c.cell_tracers()


def work(case):
    """Bytes: every tracer value read and written once a step in the handle's
    precision (6 bytes a value with the compensation) and five per-cell fields
    read once a step; host calls move FP64 values.  Operations: about 30 per
    face and 25 for the column solve of each tracer cell and step."""
    c = pure(case)
    S, nwet, ct = _sizes(tuple(sorted(dict(c, steps=1, precision="fp64").items())))
    if c["call"] == "solve":
        return {"bytes": 6.0 * 8 * nwet, "flops": 9.0 * nwet}
    s = {"fp64": 8, "mixed": 4, "comp": 6}[c["precision"]]
    steps = c["steps"]
    if c["call"] == "dropin":
        nbytes = 2.0 * 8 * ct + 6.0 * 8 * nwet
    else:
        nbytes = steps * (2.0 * s * ct + 5.0 * s * nwet)
    return {"bytes": nbytes, "flops": 115.0 * ct * steps}


# ---------------------------------------------------------------------------
# the step in 64 bits


class _Exact:
    """The transport step (tracers.c's set_dz, advect_diffuse, surf_conc and
    implicit vertical diffusion) over whole arrays: horizontal terms on the
    wet cells, vertical ones on [layer, column]."""

    def __init__(self, c, case):
        self.c, self.case, win = c, case, case.win
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.dev = dev
        self.g = win.geom

        def ti(a):
            return torch.from_numpy(np.ascontiguousarray(a, np.int64)).to(dev)

        def td(a):
            return torch.from_numpy(np.ascontiguousarray(a, np.float64)).to(dev)

        self.ti, self.td = ti, td
        S, nz = win.sgsiz, win.nz
        self.S, self.nz = S, nz
        self.wet = ti(win.wet_cells())
        self.iswet = torch.zeros(S, dtype=torch.bool, device=dev)
        self.iswet[self.wet] = True
        self.xm1, self.xp1, self.ym1, self.yp1 = (ti(a) for a in (win.xm1, win.xp1, win.ym1,
                                                                 win.yp1))
        self.zm1, self.zp1, self.m2d = ti(win.zm1), ti(win.zp1), ti(win.m2d)
        self.e1 = torch.zeros(S, dtype=torch.bool, device=dev)
        self.e2 = torch.zeros(S, dtype=torch.bool, device=dev)
        g = self.g
        self.w3e1 = ti(np.ctypeslib.as_array(g.w3_e1, shape=(g.v3_e1 + 1,))[1:])
        self.w3e2 = ti(np.ctypeslib.as_array(g.w3_e2, shape=(g.v3_e2 + 1,))[1:])
        self.e1[self.w3e1] = True
        self.e2[self.w3e2] = True
        self.bpt, self.bin = ti(win.bpt[1:]), ti(win.bin[1:])
        self.h = {n: td(getattr(win, n)) for n in ("h1au1", "h2au2", "h1au2", "h2au1",
                                                   "h1acell", "h2acell", "cellarea", "botz")}
        self.gridz = td(win.gridz)
        top, bot = ti(win.w2_t[1:g.b2_t + 1]), ti(win.bot_t[1:g.b2_t + 1])
        self.top, self.bot, self.sed = top, bot, self.zm1[bot]
        self.kb = ti(win.s2k)[bot]
        cell, cur = [], bot
        for k in range(nz):
            on = k >= self.kb
            cell.append(torch.where(on, cur, torch.zeros_like(cur)))
            cur = torch.where(on, self.zp1[cur], cur)
        self.cell = torch.stack(cell)
        self.K = torch.arange(nz, device=dev)[:, None]
        self.on = self.K >= self.kb
        self.Z = self.gridz[self.cell]            # bottom of each layer
        self.area, self.botz = self.h["cellarea"][top], self.h["botz"][top]
        kof = ti(win.s2k)
        nsur = ti(case.nsur_t[1:g.b2_t + 1])
        self.kn = torch.where(nsur == self.sed, self.kb - 1, kof[nsur])
        self.dzu1, self.dzu2 = td(case.dzu1), td(case.dzu2)
        self.u1kh, self.u2kh = td(case.u1kh), td(case.u2kh)
        self.Kz = td(case.Kz)
        self.ntr2d = None if case.ntr2d is None else ti(case.ntr2d)[top]
        self.tr = td(case.tr)

    def flow(self, u1, u2, w, f1, f2, eta, oldeta):
        td = self.td
        self.u1, self.u2 = td(u1), td(u2)
        self.eta, self.oldeta = td(eta), td(oldeta)
        self.w, self.f1, self.f2 = (None if w is None else td(w)), td(f1), td(f2)

    # the transport-mode preamble: face fluxes from the surface, w from continuity
    def preamble(self, detadt):
        for u, lst, bm, hn, isin, name in (
                (self.u1, self.w3e1, self.xm1, "h2au1", self.e1, "f1"),
                (self.u2, self.w3e2, self.ym1, "h1au2", self.e2, "f2")):
            c2 = self.m2d[lst]
            nb = bm[c2]
            floor = torch.maximum(self.h["botz"][nb], self.h["botz"][c2])
            top = torch.maximum(torch.maximum(self.eta[c2], self.eta[nb]), floor)
            zp = self.zp1[lst]
            up = torch.where(zp == lst, torch.full_like(top, math.inf), self.gridz[zp])
            last = ~isin[self.zm1[lst]]
            lo = torch.where(last, floor, self.gridz[lst])
            d = torch.minimum(top, up) - lo
            dry = ~last & (self.gridz[lst] > top)
            f = torch.zeros_like(u)
            f[lst] = torch.where(dry, torch.zeros_like(d), u[lst] * d * self.h[hn][c2])
            setattr(self, name, f)
        det = self.td(detadt)[self.top]
        ko, kn = self.kn, self.new_surface()
        s = torch.minimum(ko, kn)
        wet = self.is_wet(s)
        w = torch.zeros(self.S, dtype=torch.float64, device=self.dev)
        fc = torch.zeros_like(det)
        for k in range(self.nz):
            c = self.cell[k]
            inside = wet & (k > self.kb) & (k <= ko)
            v = torch.where(inside, fc / self.area, torch.zeros_like(fc))
            v = torch.where((wet & (k > ko) & (k <= kn)) | (k > kn), det, v)
            w[c] = torch.where(self.on[k], v, torch.zeros_like(v))
            fc = fc + torch.where(self.on[k], self.f1[c] - self.f1[self.xp1[c]] + self.f2[c] -
                                  self.f2[self.yp1[c]], torch.zeros_like(fc))
        w[0] = 0.0
        self.w = w

    def new_surface(self):
        e = self.eta[self.top]
        below = self.on & (self.Z < e)
        return torch.where(below, self.K, (self.kb - 1)[None]).max(0).values

    def is_wet(self, s):
        tz = torch.minimum(self.eta[self.top], self.oldeta[self.top])
        return (tz > 0.05 * self.case.hmin + self.botz) & (s >= self.kb)

    def step(self):
        case, nz, K, kb = self.case, self.nz, self.K, self.kb
        dt, hmin = case.dt, case.hmin
        tr = self.tr
        tr[:, self.bpt] = tr[:, self.bin]
        ko, kn = self.kn, self.new_surface()
        ks = torch.minimum(ko, kn)
        wet = self.is_wet(ks)
        eta, oe = self.eta[self.top], self.oldeta[self.top]
        zero = torch.zeros_like(self.Z)
        # thicknesses (set_dz)
        up = torch.cat([self.Z[1:], self.Z[-1:]])
        lo = torch.where(K == kb, self.botz[None].expand_as(self.Z), self.Z)
        dz = torch.where(K == ko, oe - lo, up - lo)
        dz = torch.where(self.on & (K <= ko), dz, zero)
        dzo = dz.gather(0, ko.clamp(min=0)[None])[0]
        dz = torch.where(self.on & (K > ko), dzo[None].expand_as(dz), dz)
        below = torch.cat([zero[:1], dz[:-1]])
        w9 = torch.where(self.on, 0.5 * (dz + below), zero)
        w9m = torch.cat([zero[:1], w9[:-1]])
        w9p = torch.cat([w9[1:], w9[-1:]])
        w5 = below / (below + dz)
        # sub-step length
        u1, u2, w = self.u1, self.u2, self.w
        dmin = math.inf
        act = self.on & wet & (K <= ks)
        cc, c2 = self.cell, self.top[None]

        def speed(a):
            return torch.where(a.abs() < 1e-10, torch.full_like(a, 1e-10), a)

        if case.stab & _abi.SUB_STEP:
            d1 = 0.8 * (self.h["h1acell"][c2] / speed(0.5 * (u1[cc] + u1[self.xp1[cc]]))).abs()
            d2 = 0.8 * (self.h["h2acell"][c2] / speed(0.5 * (u2[cc] + u2[self.yp1[cc]]))).abs()
            d3 = 0.8 * (dz / speed(0.5 * (w[cc] + w[self.zp1[cc]]))).abs()
            for d, m in ((d1, act), (d2, act), (d3, act & (K != ks) & (d3 > 0))):
                v = d[m]
                if v.numel():
                    dmin = min(dmin, float(v.min()))
        dtm = min(dt, dmin)
        if dtm != dt:
            dtm = math.floor(dtm)
        # the implicit solve's rows
        solve = wet & (kn > kb) & (dz.gather(0, (kn - 1).clamp(min=0)[None])[0] != 0)
        row = self.on & solve & (K <= kn)
        cm1 = torch.where(row & (K > kb), -self.Kz[cc] / (0.5 * (dz + below)), zero)
        cp1 = torch.cat([cm1[1:], zero[:1]])
        trem, prev, first = dt, 0.0, True
        while trem > 0:
            dtu = min(dtm, trem)
            f = 1.0 + (dtu - trem) / dt
            sub = oe + f * (eta - oe)
            osub = oe if first else oe + prev * (eta - oe)
            last = trem - dtu <= 0
            for n in range(case.ntr):
                m = wet if self.ntr2d is None else wet & (n < self.ntr2d)
                self.tracer(tr[n], n, m, dtu, dz, w5, w9m, w9, w9p, ko, kn, ks, sub, osub)
                if last:
                    self.diffuse(tr[n], m & solve, dz, cm1, cp1, kn)
            prev, first, trem = f, False, trem - dtu
        self.kn = kn

    def limit(self, cr, F, tm2, tm1, t0, tp1):
        pos = cr > 0
        tc, tu, td = torch.where(pos, tm1, t0), torch.where(pos, tm2, tp1), torch.where(pos, t0,
                                                                                       tm1)
        diff = td - tu
        some = diff != 0
        d = torch.where(some, diff, torch.ones_like(diff))
        z = torch.zeros_like(d)
        nc, nu = torch.where(some, (tc - tu) / d, z), torch.where(some, (F - tu) / d, z)
        acr = torch.where(cr != 0, cr.abs(), torch.ones_like(cr))
        up = tu + nc * diff
        G = torch.where(nu > nc / acr, tu + nc * diff / acr, F)
        G = torch.where(nu < nc, up, G)
        G = torch.where(nu > 1.0, td, G)
        G = torch.where((nc >= 0) & (nc <= 1), G, up)
        return torch.where(cr == 0, F, G)

    def value(self, cr, vel, d, db, df, hm, h0, hp, tm2, tm1, t0, tp1):
        scheme = self.c["scheme"]
        z = torch.zeros_like(t0)
        if scheme in ("quickest", "quickest_co"):
            if scheme == "quickest":
                face = d * (t0 - tm1) + tm1
                cp, cn = (db * (hm * t0 + h0 * tm2) - 2.0 * tm1,
                          df * (h0 * tp1 + hp * tm1) - 2.0 * t0)
            else:
                face = 0.5 * (t0 + tm1)
                cp, cn = t0 - 2.0 * tm1 + tm2, tp1 - 2.0 * t0 + tm1
            curv = torch.where(cr > 0, cp, torch.where(cr < 0, cn, z))
            return face - 0.5 * cr * (t0 - tm1) - (1.0 - cr * cr) * curv / 6.0
        if scheme == "vanleer":
            p = (tm1 - tm2) * (t0 - tm1)
            q = (t0 - tm1) * (tp1 - t0)
            one = torch.ones_like(t0)
            p = torch.where(p > 0, 2.0 * p / torch.where(p > 0, t0 - tm2, one), z)
            q = torch.where(q > 0, 2.0 * q / torch.where(q > 0, tp1 - tm1, one), z)
            return torch.where(vel > 0, tm1 + 0.5 * (1.0 - cr) * p,
                               torch.where(vel < 0, t0 - 0.5 * (1.0 + cr) * q, z))
        if scheme == "order2":
            return d * (t0 - tm1) + tm1
        if scheme == "order4":
            return (7.0 * (tm1 + t0) - (tp1 + tm2)) / 12.0
        return torch.where(vel > 0, 0.5 * (3.0 - cr) * tm1 - 0.5 * (1.0 - cr) * tm2,
                           torch.where(vel < 0, 0.5 * (3.0 - cr) * t0 - 0.5 * (1.0 - cr) * tp1,
                                       z))

    def hflux(self, t, wc, m1, p1, e, u, f, hcell, hau, hdz, dzu, kh, dtu):
        """Flux through the backward face of every wet cell, on the flat array."""
        scheme, ult = self.c["scheme"], self.c["ultimate"]
        a, c2 = m1[wc], self.m2d[wc]
        b2, p2 = m1[c2], p1[c2]
        tm2, tm1, t0, tp1 = t[m1[a]], t[a], t[wc], t[p1[wc]]
        U = f[wc]
        if scheme == "order1":
            v = 0.5 * (U + U.abs()) * tm1 + 0.5 * (U - U.abs()) * t0
        else:
            H = self.h[hau]
            cr = u[wc] * dtu / H[c2]
            hc = self.h[hcell]
            v = self.value(cr, u[wc], hc[b2] / (hc[b2] + hc[c2]), 2.0 / (H[b2] + H[c2]),
                           2.0 / (H[c2] + H[p2]), H[b2], H[c2], H[p2], tm2, tm1, t0, tp1)
            if scheme not in ("quickest", "quickest_co"):
                v = torch.where(e[wc], v, torch.zeros_like(v))
            if ult:
                v = torch.where(e[wc], self.limit(cr, v, tm2, tm1, t0, tp1), v)
            v = v * U
        if self.c["hdiff"]:
            v = v - dzu[wc] * self.h[hdz][c2] * kh[wc] * (t0 - tm1) / self.h[hau][c2]
        out = torch.zeros(self.S, dtype=torch.float64, device=self.dev)
        out[wc] = v
        if scheme == "order1":  # its fluxes reach the ghost cells' faces too
            gh = p1[wc]
            gh = gh[~self.iswet[gh]]
            U = f[gh]
            out[gh] = 0.5 * (U + U.abs()) * t[m1[gh]] + 0.5 * (U - U.abs()) * t[gh]
        return out

    def tracer(self, t, n, m, dtu, dz, w5, w9m, w9, w9p, ko, kn, ks, sub, osub):
        scheme, ult = self.c["scheme"], self.c["ultimate"] and self.c["scheme"] != "order1"
        wc, cc, K, kb = self.wet, self.cell, self.K, self.kb
        fx = self.hflux(t, wc, self.xm1, self.xp1, self.e1, self.u1, self.f1, "h1acell",
                        "h1au1", "h2au1", self.dzu1, self.u1kh, dtu)
        fy = self.hflux(t, wc, self.ym1, self.yp1, self.e2, self.u2, self.f2, "h2acell",
                        "h2au2", "h1au2", self.dzu2, self.u2kh, dtu)
        dtr = (fx[self.xp1[cc]] - fx[cc] + fy[self.yp1[cc]] - fy[cc]) * dtu
        del fx, fy
        # vertical faces: the bottom of every layer
        t0 = t[cc]
        tb = t[self.bot]
        tm1 = torch.where(K > kb, torch.cat([t0[:1], t0[:-1]]), t0)
        tm2 = torch.where(K > kb, torch.cat([tm1[:1], tm1[:-1]]), t0)
        tp1 = torch.cat([t0[1:], t0[-1:]])
        w = self.w[cc]
        if scheme == "order1":
            fz = dtu * (0.5 * (w + w.abs()) * tm1 + 0.5 * (w - w.abs()) * t0)
        else:
            cz = torch.where(self.on, w * dtu / torch.where(self.on, w9, torch.ones_like(w9)),
                             torch.zeros_like(w9))
            v = self.value(cz, w, w5, 2.0 / (w9m + w9), 2.0 / (w9 + w9p), w9m, w9, w9p, tm2,
                           tm1, t0, tp1)
            if ult:
                v = self.limit(cz, v, tm2, tm1, t0, tp1)
            fz = v * (w * dtu)
        fzt = torch.cat([fz[1:], fz[-1:]])
        a = t0 - (dtr / self.area + (fzt - fz)) / dz
        new = torch.where(self.on & m & (K < ks), a, t0)
        # the surface cell's mass balance (surf_conc)
        kc = ks.clamp(min=0)[None]
        ts = t0.gather(0, kc)[0]
        st = fz.gather(0, kc)[0] * self.area
        wb = torch.where(ks == kb, self.botz, self.Z.gather(0, kc)[0])
        wbot = wb.clone()
        for k in range(self.nz):
            at = m & (k >= ks)
            lo = torch.where(k == kb, self.botz, self.Z[k])
            up = self.Z[min(k + 1, self.nz - 1)]
            add = torch.where(k < ko, t0[k] * self.area * (up - wbot) - dtr[k],
                              torch.where(k == ko, t0[k] * self.area * (osub - lo) - dtr[k],
                                          -dtr[k]))
            st = st + torch.where(at, add, torch.zeros_like(add))
            wbot = torch.where(at & (k < ko), up, wbot)
        dzs = sub - wb
        vol = dzs * self.area
        zero = torch.zeros_like(vol)
        dry = (vol == 0) | ((st < 0) & (dzs <= self.case.hmin))
        sv = torch.where(dry, zero, st / torch.where(vol == 0, torch.ones_like(vol), vol))
        keep = (self.botz > 0) & (dz.gather(0, kc)[0] < self.case.hmin)
        vs = torch.where(keep, ts, sv)
        new = torch.where(self.on & m & (K >= ks), vs[None].expand_as(new), new)
        t[cc[self.on]] = new[self.on]
        t[self.sed] = tb  # every column's sediment cell follows its bottom value

    def diffuse(self, t, m, dz, cm1, cp1, kn):
        """Implicit vertical diffusion: one tridiagonal system per column."""
        cc, kb, dt = self.cell, self.kb, self.case.dt
        a = t[cc]
        zero = torch.zeros_like(self.area)
        one = torch.ones_like(self.area)
        div, ud, sol = one, [], []
        s = zero
        for k in range(self.nz):
            row = m & (k >= kb) & (k <= kn)
            lo = torch.where(row, cm1[k], zero)
            hi = torch.where(row & (k < kn), cp1[k], zero)
            prev = torch.where(row & (k > kb), cp1[k - 1], zero) if k else zero
            u = prev / div
            r = dz[k] / dt
            div = torch.where(row, r - lo - hi - lo * u, one)
            s = torch.where(row, (r * a[k] - lo * s) / div, zero)
            ud.append(u)
            sol.append(s)
        x = zero
        up = zero
        for k in range(self.nz - 1, -1, -1):
            row = m & (k >= kb) & (k <= kn)
            x = torch.where(row, sol[k] - up * x, zero)
            up = torch.where(row, ud[k], zero)
            c = cc[k][row]
            t[c] = x[row]


def exact(case, seed):
    c = pure(case)
    if c["call"] == "solve":
        k, a = _solve_inputs(c, seed)
        return _exact_solve(k, a)
    k = _build(c, seed)
    e = _Exact(c, k)
    if c["call"] == "tide":
        for u1, u2, old, new in _tide_steps(k):
            e.flow(u1, u2, None, k.u1flux3d, k.u2flux3d, new, old)
            e.preamble((new - old) / k.dt)
            e.step()
    else:
        e.flow(k.u1, k.u2, k.w, k.u1flux3d, k.u2flux3d, k.eta, k.oldeta)
        for _ in range(c["steps"]):
            e.step()
    if c["call"] == "dropin":
        return {"tr": e.tr, "sur": None, "nsur": None}
    if c["precision"] == "comp":
        return e.tr
    return e.tr[:, e.wet]


def _exact_solve(case, a):
    """The closures' tridiagonal solve, every column from its bottom cell to
    its surface cell."""
    win = case.win
    kof, nb = win.s2k, win.geom.b2_t
    bot, sur = win.bot_t[1:nb + 1], case.nsur_t[1:nb + 1]
    kb, kn = kof[bot], kof[sur]
    x = a["var"].copy()
    on = win.zm1[sur] != sur
    n = win.nz
    sol, ud, cells = np.zeros((n, nb)), np.zeros((n, nb)), np.zeros((n, nb), np.int64)
    cur, div, s, up = bot.copy(), np.ones(nb), np.zeros(nb), np.zeros(nb)
    for k in range(n):
        row = on & (k >= kb) & (k <= kn)
        below = row & (k > kb)
        c = cur
        u = np.where(below, up / div, 0.0)
        lo = np.where(below, a["Cm1"][c], 0.0)
        div = np.where(row, a["Cd"][c] - lo * u, 1.0)
        s = np.where(row, (a["rhs"][c] - lo * s) / div, 0.0)
        sol[k], ud[k], cells[k] = s, u, c
        up = np.where(row, a["Cp1"][c], 0.0)
        cur = np.where(k >= kb, win.zp1[cur], cur)
    v, nxt = np.zeros(nb), np.zeros(nb)
    for k in range(n - 1, -1, -1):
        row = on & (k >= kb) & (k <= kn)
        v = np.where(row, sol[k] - nxt * v, 0.0)
        nxt = np.where(row, ud[k], 0.0)
        x[cells[k][row]] = np.maximum(v[row], 1e-6)
    return x
