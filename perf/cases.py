"""The work that a user of cress_b200 has it do, as measurable cases.

A case is one pass through the public entry points (cress_b200.Solver,
Ensemble, Mlp) as a host model drives them: the state lives on the device, a
pass advances it by an output interval and reads the new level back into
page-locked host arrays, or it is one call of the acoustic loop or of the
learned network's training arithmetic.

The named shapes are this repository's own: the dry warm bubble 64x64x40,
the moist supercell 256x256x64 and 512x512x64, the open-x squall line with
80 levels, ensembles of uneven domains 96-192 x 96-192 x 48, the
16-256-256-256-9 network at batches of 8192; the others are ragged sizes
between them.

exact() restates the dry step (HE-VI, HE-VE, forcing, filter) and the network
in 64 bits with plain torch.  The moist steps have none: the cold-rain scheme
over a whole domain and several steps takes plain array code far longer than
20 seconds.
"""
import functools
import math

import numpy as np
import torch

import cress_b200
from cress_b200 import cases as model

NOW, PAST, FORCING = cress_b200.NOW, cress_b200.PAST, cress_b200.FORCING
DRY = ["u", "v", "w", "pp", "ptp"]
MOIST = model.MOIST_NAMES
STAG = {"u": "u", "v": "v"}
VSPBAR = 0.005   # sponge coefficient above 0.6 of the model top, as bench.py sets it


def nsstp_of(dtbig, dtsml):
    """Acoustic substeps of one leapfrog step (SrcOrig/slvstep.f90:176)."""
    return 20 * int(1.e2 * (dtbig + .001)) // int(1.e3 * (dtsml + .0001))


def listed():
    return [
        # The repository's first configuration: a dry warm bubble on a grid that
        # does not fill the GPU; 30 s of model time between two outputs, replayed
        # from CUDA graphs.  Launches and their gaps count here.
        dict(name="bubble_64x64x40", kind="dry", nx=64, ny=64, nz=40, dx=500.0, dz=300.0, sthopt=0,
             dtbig=2.0, dtsml=0.25, steps=15, graphs=True, impopt=1, coropt=0, advopt=2, tile=0),
        # A single step of a small ragged dry domain with Coriolis and 4th-order
        # vertical advection, launched eagerly: the smallest call.
        dict(name="dry_step_75x51x37", kind="dry", nx=75, ny=51, nz=37, dx=500.0, dz=350.0, sthopt=1,
             dtbig=2.0, dtsml=0.25, steps=1, graphs=False, impopt=1, coropt=1, advopt=3, tile=0),
        # The explicit (HE-VE) small step at an ordinary size.
        dict(name="heve_192x160x48", kind="dry", nx=192, ny=160, nz=48, dx=500.0, dz=300.0, sthopt=1,
             dtbig=2.0, dtsml=0.25, steps=4, graphs=True, impopt=0, coropt=0, advopt=2, tile=0),
        # The acoustic loop alone (s_smalldrv on resident fields), ragged, with
        # the default tile.
        dict(name="acoustic_203x131x54", kind="acoustic", nx=203, ny=131, nz=54, dx=1000.0, dz=300.0,
             dts=1.0, nsstp=20, tile=0),
        # The dry step at the largest size, with the tile the autotuner picks there.
        dict(name="dry_512x512x64", kind="dry", nx=512, ny=512, nz=64, dx=1000.0, dz=281.0, sthopt=1,
             dtbig=5.0, dtsml=1.0, steps=6, graphs=True, impopt=1, coropt=0, advopt=2, tile=13),
        # The moist supercell: half a minute of model time between outputs.
        dict(name="supercell_256x256x64", kind="moist", nx=256, ny=256, nz=64, dx=1000.0, dtbig=5.0, dtsml=1.0,
             steps=6, graphs=True, tubopt=0, obc=0, advopt=2, tile=13, learned=False),
        # The largest: the headline workload.
        dict(name="supercell_512x512x64", kind="moist", nx=512, ny=512, nz=64, dx=1000.0, dtbig=5.0, dtsml=1.0,
             steps=6, graphs=True, tubopt=0, obc=0, advopt=2, tile=13, learned=False),
        # The TKE closure (the turbulence of every shipped configuration) on a
        # ragged domain, eager launches, the default tile.
        dict(name="tke_209x147x57", kind="moist", nx=209, ny=147, nz=57, dx=1000.0, dtbig=5.0, dtsml=1.0,
             steps=3, graphs=False, tubopt=2, obc=0, advopt=2, tile=0, learned=False),
        # The squall line: open radiation x boundaries, 80 levels.
        dict(name="squall_512x128x80", kind="moist", nx=512, ny=128, nz=80, dx=500.0, dtbig=3.0, dtsml=0.5,
             steps=6, graphs=True, tubopt=0, obc=4, advopt=2, tile=0, learned=False),
        # Learned microphysics in the supercell's step (weights seeded, envelope
        # wide enough that most cells take the network).
        dict(name="learned_256x192x64", kind="moist", nx=256, ny=192, nz=64, dx=1000.0, dtbig=5.0, dtsml=1.0,
             steps=4, graphs=True, tubopt=0, obc=0, advopt=2, tile=13, learned=True),
        # An ensemble of uneven domains stepped together.
        dict(name="ensemble_12", kind="ensemble", members=12, lo=96, hi=192, nz=48, dx=1000.0, dtbig=5.0,
             dtsml=1.0, steps=4, shapes=5),
        # The network's loss and gradient of one training batch, host arrays in
        # and out.
        dict(name="mlp_grad_8192", kind="mlp", n=8192),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dry", "dry", "acoustic", "acoustic", "moist", "moist", "moist", "moist", "ensemble", "mlp"])
    if kind == "mlp":
        return dict(kind="mlp", n=128 * _log(rng, 2, 128))
    if kind == "ensemble":
        return dict(kind="ensemble", members=rng.randint(2, 12), lo=rng.randint(40, 96), hi=rng.randint(100, 192),
                    nz=rng.randint(24, 64), dx=1000.0, dtbig=5.0, dtsml=1.0, steps=rng.randint(1, 4),
                    shapes=rng.randint(0, 1 << 20))
    nx, ny = _log(rng, 40, 512), _log(rng, 40, 512)
    tile = rng.choice([0, 0, 13])
    nz = rng.randint(24, 64 if tile == 13 else 80)
    while nx * ny * nz > 512 * 512 * 64:
        nx, ny = max(40, nx * 3 // 4), max(40, ny * 3 // 4)
    if kind == "acoustic":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, dx=1000.0, dz=round(18000.0 / nz, 1), dts=rng.choice([0.5, 1.0]),
                    nsstp=rng.randint(8, 24), tile=tile)
    steps = rng.randint(1, 5)
    if kind == "dry":
        impopt = rng.choice([0, 1, 1])
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, dx=500.0, dz=300.0, sthopt=rng.randint(0, 1), dtbig=2.0,
                    dtsml=0.25, steps=steps, graphs=rng.random() < .5, impopt=impopt,
                    coropt=rng.randint(0, 1), advopt=rng.choice([2, 2, 3]), tile=tile if impopt else 0)
    obc = rng.choice([0, 0, 0, 4, 5, 7])
    learned = not obc and rng.random() < .2
    nz = max(nz, 44)   # 18 km in layers of 100 to 500 m
    while nx * ny * nz > 512 * 512 * 64:
        nx, ny = max(40, nx * 3 // 4), max(40, ny * 3 // 4)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, dx=500.0 if obc else 1000.0, dtbig=3.0 if obc else 5.0,
                dtsml=0.5 if obc else 1.0, steps=steps, graphs=rng.random() < .6,
                tubopt=0 if obc or learned else rng.choice([0, 0, 1, 2]), obc=obc,
                advopt=2 if obc else rng.choice([2, 2, 3]), tile=tile, learned=learned)


# ---------------------------------------------------------------- inputs

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Random:
    """Seeded random numbers drawn on the GPU."""

    def __init__(self, *key):
        self.g = torch.Generator(device=_device())
        s = 1
        for k in key:
            s = (s * 6364136223846793005 + int(k) * 1442695040888963407 + 97) % (1 << 62)
        self.g.manual_seed(s)

    def uniform(self, shape, lo, hi):
        return torch.rand(shape, generator=self.g, device=_device()) * (hi - lo) + lo

    def normal(self, shape):
        return torch.randn(shape, generator=self.g, device=_device())

    def noise(self, shape, amp):
        """White noise smoothed over 3x3 points, largest value amp."""
        x = self.normal(shape)
        for ax in (1, 2):
            x = (x + torch.roll(x, 1, ax) + torch.roll(x, -1, ax)) / 3.0
        return x * (amp / (x.abs().max() + 1e-30))


def _wrap(a, stag="s"):
    """Both periodic ghost layers of an (nk, nj+2, ni+2) field."""
    nk, nj2, ni2 = a.shape
    sx = torch.from_numpy(model._wrap_index(ni2 - 2, stag == "u")).to(a.device)
    sy = torch.from_numpy(model._wrap_index(nj2 - 2, stag == "v")).to(a.device)
    return a.index_select(1, sy).index_select(2, sx).contiguous()


@functools.lru_cache(maxsize=2)
def _expanded(key, ni, nj, nk):
    """The horizontally uniform 3-D base arrays of one shape (the same for every seed)."""
    cols = _columns(key, nk)
    out = {}
    for n, c in cols.items():
        if n in model.BASE_NAMES + ["pbr", "qvbr", "ubr", "vbr", "rbct"]:
            out[n] = model.expand(c, ni, nj, nk)
    return out


@functools.lru_cache(maxsize=32)
def _columns(key, nk):
    """1-D base columns, winds and the sponge of one vertical grid."""
    kind, p1, p2 = key
    if kind == "dry":
        cols = model.base_columns(nk, p1, sthopt=p2, dthdz=0.003)
        jcb = np.asarray(cols["jcb"], np.float64)
        zph = np.zeros(nk + 1)
        for k in range(3, nk + 1):
            zph[k] = zph[k - 1] + jcb[k - 1] * p1
        zph[1] = -zph[3]
        cols["dz"] = p1
        cols["ubr"] = 5.0 + 10.0 * np.clip(cols["zs"] / zph[nk - 1], 0.0, 1.0)
        cols["vbr"] = np.zeros(nk + 1)
    else:
        cols = model.moist_columns(nk)
        zph, zs = cols["zph"], cols["zs"]
        if kind == "squall":
            cols["ubr"] = 20.0 * np.clip(zs / 2500.0, 0.0, 1.0)
            cols["vbr"] = np.zeros(nk + 1)
        else:   # quarter-circle hodograph, 30 m/s over 0-6 km
            th = 0.5 * np.pi * np.clip(zs / 2000.0, 0.0, 1.0)
            cols["ubr"] = np.where(zs < 2000.0, 7.0 * (1.0 - np.cos(th)),
                                   7.0 + 23.0 * np.clip((zs - 2000.0) / 4000.0, 0.0, 1.0))
            cols["vbr"] = 7.0 * np.sin(th)
    botbar, top = 0.6 * zph[nk - 1], zph[nk - 1]
    cols["zph"] = zph
    cols["ksp0"] = next((k - 1 for k in range(3, nk + 1) if zph[k] > botbar), 2)
    rbct = np.zeros(nk + 1, np.float32)   # SrcOrig/vspdmp.f90:269-292
    for k in range(2, nk):
        if zph[k] > botbar:
            rbct[k] = 0.5 * VSPBAR * (1.0 - math.cos(3.141592 * (zph[k] - botbar) / (top - botbar)))
    cols["rbct"] = rbct
    return cols


def _key(case):
    if case["kind"] in ("dry", "acoustic"):
        return ("dry", case["dz"], case.get("sthopt", 1))
    return ("squall" if case.get("obc") else "supercell", 0, 1)


def _bubble(case, cols, shape, rng, amp, rad_z=1400.0):
    nk, nj2, ni2 = shape
    d = _device()
    z = torch.as_tensor(cols["zs"][1:nk + 1], device=d, dtype=torch.float32)
    x = (torch.arange(ni2, device=d, dtype=torch.float32) - 0.5 * (ni2 - 1)) * case["dx"]
    y = (torch.arange(nj2, device=d, dtype=torch.float32) - 0.5 * (nj2 - 1)) * case["dx"]
    rad = min(10000.0, min(nj2, ni2) * case["dx"] / 5.0)
    ry = 0.0 if case.get("obc") else 1.0   # the squall line's thermal runs along y
    r = torch.sqrt((x[None, None, :] / rad) ** 2 + ry * (y[None, :, None] / rad) ** 2 +
                   ((z[:, None, None] - 1400.0) / rad_z) ** 2)
    pt = torch.where(r < 1.0, amp * torch.cos(0.5 * math.pi * r) ** 2, torch.zeros_like(r))
    return pt + rng.uniform(shape, -0.05, 0.05)


def _state(case, seed):
    """One time level's prognostic fields (GPU tensors, host layout)."""
    nk, nj2, ni2 = shape = (case["nz"] + 3, case["ny"] + 5, case["nx"] + 5)
    rng = _Random(seed, case["nx"], case["ny"], nk)
    cols = _columns(_key(case), nk)
    d = _device()
    col = lambda n: torch.as_tensor(np.asarray(cols[n], np.float32)[1:nk + 1], device=d)[:, None, None]
    f = {"u": col("ubr") + rng.noise(shape, 0.5), "v": col("vbr") + rng.noise(shape, 0.5),
         "w": torch.zeros(shape, device=d), "pp": torch.zeros(shape, device=d),
         "ptp": _bubble(case, cols, shape, rng, 2.0 if case["kind"] == "dry" else 3.0)}
    if case["kind"] != "dry":
        pbr = col("pbr")
        t = col("ptbr") * (pbr / 1.0e5) ** (model.RD / model.CP)
        z = torch.as_tensor(cols["zs"][1:nk + 1], device=d, dtype=torch.float32)[:, None, None]
        esw = 610.78 * torch.exp(17.269 * (t - 273.16) / (t - 35.86))
        qvs = 0.622 * esw / (pbr - esw)

        def blob(lo, hi, zlo, zhi, amp):
            return amp * ((rng.noise(shape, 1.0) - lo) / (hi - lo)).clamp(0.0, 1.0) * ((z > zlo) & (z < zhi))

        f["qv"] = ((0.8 + 0.3 * rng.noise(shape, 1.0)) * qvs).clamp(max=0.02)
        f["qc"] = blob(0.0, 0.6, 500.0, 9000.0, 1.5e-3)
        f["qr"] = blob(0.1, 0.8, 0.0, 6000.0, 2.0e-3)
        f["qi"] = blob(0.0, 0.7, 6000.0, 14000.0, 3.0e-4)
        f["qs"] = blob(0.0, 0.7, 4500.0, 12000.0, 1.0e-3)
        f["qg"] = blob(0.1, 0.8, 3000.0, 10000.0, 1.5e-3)
        f["ni"] = f["qi"] / 1.0e-11 * rng.uniform(shape, 0.5, 1.5)
        f["ns"] = f["qs"] / 5.0e-9 * rng.uniform(shape, 0.5, 1.5)
        f["ng"] = f["qg"] / 5.0e-8 * rng.uniform(shape, 0.5, 1.5)
        if case.get("tubopt") == 2:
            f["tke"] = rng.uniform(shape, 0.0, 2.0) * (z < 12000.0)
    return {n: _wrap(a, STAG.get(n, "s")) for n, a in f.items()}


def _acoustic_state(case, seed):
    """Past-level u, v, w, p' and the large step's forcings."""
    nk, nj2, ni2 = shape = (case["nz"] + 3, case["ny"] + 5, case["nx"] + 5)
    rng = _Random(seed, case["nx"], case["ny"], nk)
    rst = torch.as_tensor(np.asarray(_columns(_key(case), nk)["rst"], np.float32)[1:nk + 1],
                          device=_device())[:, None, None]
    w = rng.noise(shape, 1.5)
    w[1], w[nk - 2] = 0.0, 0.0
    st = {"u": rng.noise(shape, 6.0) + 8.0, "v": rng.noise(shape, 6.0) - 2.0, "w": w, "pp": rng.noise(shape, 40.0)}
    fr = {"u": rng.noise(shape, 2e-3) * rst, "v": rng.noise(shape, 2e-3) * rst, "w": rng.noise(shape, 4e-3) * rst,
          "pp": rng.noise(shape, 0.3)}
    return ({n: _wrap(a, STAG.get(n, "s")) for n, a in st.items()},
            {n: _wrap(a, STAG.get(n, "s")) for n, a in fr.items()})


def _mlp_params(rng):
    """Seeded weights in the library's layout (cress_mlp_get_params)."""
    w1 = rng.normal((256, 64)) * 0.25
    w1[:, 16:] = 0.0
    w4 = rng.normal((256, 64)) * 0.0625
    w4[:, 9:] = 0.0
    b4 = rng.normal((64,)) * 0.1
    b4[9:] = 0.0
    parts = [w1, rng.normal((256,)) * 0.1, rng.normal((256, 256)) * 0.09, rng.normal((256,)) * 0.1,
             rng.normal((256, 256)) * 0.09, rng.normal((256,)) * 0.1, w4, b4]
    return torch.cat([p.reshape(-1) for p in parts])


def _norm():
    """Means, scales and envelope of the network's inputs (temperature in
    Celsius, ln p, density, w, log10 contents and numbers, supersaturations)
    and outputs: most cells of the supercell lie inside."""
    xm = [-20, 10.8, 0.7, 0, -3, -6, -6, -7, -7, -7, 2, 1, 1, 0, 0, -5]
    xs = [30, 0.6, 0.3, 3, 1, 4, 4, 4, 4, 4, 3, 2, 2, 0.4, 0.4, 4]
    lo = [-62, 9.2, 0.0, -60, -12, -12, -12, -12, -12, -12, 0, 0, 0, -1, -1, -12]
    hi = [40, 12, 1.4, 60, 0, 0, 0, 0, 0, 0, 12, 12, 12, 1, 1, 0]
    return np.array(xm + xs + [0.0] * 9 + [1.0] * 9 + lo + hi, np.float32)


# ---------------------------------------------------------------- solver set-up

_program_stream = None


def _stream():
    """The one stream a program keeps its solvers on."""
    global _program_stream
    if _program_stream is None:
        _program_stream = torch.cuda.Stream()
    return _program_stream


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True).numpy()


def _put(solver, level_fields, levels):
    for n, a in level_fields.items():
        h = a.cpu().numpy()
        for lv in levels:
            solver.put_field(n, lv, h)


def _interior(name, a):
    """The physical points of one field (the ghost layers repeat them) on the
    levels the model defines: 1..nk of w, 1..nk-1 of the others."""
    return a[:a.shape[0] - (name != "w"), 2:-3, 2:-3]


class _Step:
    """A solver with its state on the device, its host output arrays and the
    size of an output interval."""

    def __init__(self, case, seed, own_stream=False):
        self.case = case
        ni, nj, nk = model.dims(case["nx"], case["ny"], case["nz"])
        key = _key(case)
        cols, b3 = _columns(key, nk), _expanded(key, ni, nj, nk)
        moist = case["kind"] != "dry"
        self.solver = s = cress_b200.Solver(
            ni, nj, nk, case["dx"], case["dx"], cols["dz"], sthopt=case.get("sthopt", 1), cphopt=3 if moist else 0,
            tile=case["tile"], impopt=case.get("impopt", 1), coropt=case.get("coropt", 0),
            fc=2.1e-5 if case.get("coropt") else 0.0, advopt=case["advopt"], tubopt=case.get("tubopt", 0),
            obc=case.get("obc", 0))
        if not own_stream:
            s.set_stream(_stream().cuda_stream)
        s.set_base3d(b3)
        s.set_base_large(b3["ubr"], b3["vbr"], b3["rbct"], cols["ksp0"])
        if moist:
            s.set_base_moist(b3["pbr"], b3["qvbr"])
        if case["graphs"]:
            s.set_graphs(True)
        fields = _state(case, seed)
        _put(s, fields, (PAST, NOW))
        self.names = list(fields)
        self.mlp = None
        if case.get("learned"):
            self.mlp = cress_b200.Mlp(seed=1)
            self.mlp.set_params(_mlp_params(_Random(seed, 5)).cpu().numpy())
            self.mlp.set_norm(_norm())
            s.set_learned_micro(self.mlp, 0, 1.0)
        self.out = [_pinned(s.shape) for _ in self.names]
        self.nsstp = nsstp_of(case["dtbig"], case["dtsml"])
        self.ctime = 0.0
        s.sync()

    def advance(self, steps):
        c = self.case
        for _ in range(steps):
            first = self.ctime == 0   # the leapfrog's first step is a half step without the filter
            h = 0.5 if first else 1.0
            self.solver.large_step(int(self.ctime), h * c["dtbig"], self.nsstp, h * c["dtsml"])
            self.ctime += 1000.0 * c["dtbig"]

    def read(self):
        self.solver.get_fields_async(NOW, self.names, self.out)
        return {n: _interior(n, a) for n, a in zip(self.names, self.out)}


class _Acoustic:
    def __init__(self, case, seed):
        self.case = case
        ni, nj, nk = model.dims(case["nx"], case["ny"], case["nz"])
        key = _key(case)
        self.solver = s = cress_b200.Solver(ni, nj, nk, case["dx"], case["dx"], case["dz"], sthopt=1,
                                            tile=case["tile"])
        s.set_stream(_stream().cuda_stream)
        s.set_base3d(_expanded(key, ni, nj, nk))
        st, fr = _acoustic_state(case, seed)
        _put(s, st, (PAST,))
        _put(s, fr, (FORCING,))
        self.names = list(st)
        self.out = [_pinned(s.shape) for _ in self.names]
        s.sync()

    def run(self):
        self.solver.small_steps(self.case["nsstp"], self.case["dts"])
        self.solver.get_fields_async(cress_b200.FUTURE, self.names, self.out)
        return {n: _interior(n, a) for n, a in zip(self.names, self.out)}


def _member_cases(case):
    """The members' uneven shapes: part of the case, not of the seed."""
    r = np.random.default_rng(case["shapes"])
    return [dict(kind="moist", nx=int(r.integers(case["lo"], case["hi"] + 1)),
                 ny=int(r.integers(case["lo"], case["hi"] + 1)), nz=max(44, case["nz"]), dx=case["dx"],
                 dtbig=case["dtbig"], dtsml=case["dtsml"], graphs=False, tubopt=0, obc=0, advopt=2, tile=13)
            for _ in range(case["members"])]


class _Ensemble:
    def __init__(self, case, seed):
        self.case = case
        self.members = [_Step(c, seed * 131 + m, own_stream=True) for m, c in enumerate(_member_cases(case))]
        self.ens = cress_b200.Ensemble([m.solver for m in self.members])
        self.ctime = 0.0

    def run(self):
        c = self.case
        nsstp = self.members[0].nsstp
        for _ in range(c["steps"]):
            h = 0.5 if self.ctime == 0 else 1.0
            self.ens.large_step(int(self.ctime), h * c["dtbig"], nsstp, h * c["dtsml"])
            self.ctime += 1000.0 * c["dtbig"]
        # the winds, theta', vapour and rain of every member go to the host
        keep = ["u", "w", "ptp", "qv", "qr"]
        got = []
        for m in self.members:
            outs = [m.out[m.names.index(n)] for n in keep]
            m.solver.get_fields_async(NOW, keep, outs)
            got.append([_interior(n, a) for n, a in zip(keep, outs)])
        return got

    def __del__(self):
        self.ens.close()


class _Mlp:
    def __init__(self, case, seed):
        rng = _Random(seed, case["n"])
        self.mlp = cress_b200.Mlp(seed=1)
        self.mlp.set_params(_mlp_params(rng).cpu().numpy())
        self.x = rng.normal((case["n"], 16)).cpu().numpy()
        self.t = rng.normal((case["n"], 9)).cpu().numpy()


def prepare(case, seed):
    """What a program has in hand before the call: the solver (or network)
    with its state on the device and the host arrays the outputs go to."""
    if case["kind"] == "acoustic":
        return _Acoustic(case, seed)
    if case["kind"] == "ensemble":
        return _Ensemble(case, seed)
    if case["kind"] == "mlp":
        return _Mlp(case, seed)
    return _Step(case, seed)


def run(state):
    if isinstance(state, _Step):
        state.advance(state.case["steps"])
        return state.read()
    if isinstance(state, _Mlp):
        loss, grad = state.mlp.loss_grad(state.x, state.t)
        return {"loss": np.array([loss], np.float32), "grad": grad}
    return state.run()


# ---------------------------------------------------------------- work and tolerance

def _step_work(c, cells):
    """Bytes and operations of one large step: each prognostic field's past
    and present level read and its present and future level written once
    (they exceed L2), and in each acoustic substep u, v, w, p' and their
    forcings read and u, v, w, p' written, once each per point."""
    nsstp = nsstp_of(c["dtbig"], c["dtsml"])
    nf = 5 if c["kind"] == "dry" else 14 + (c.get("tubopt") == 2)
    b = 16 * nf + 16 + 48 * nsstp
    f = 110 * nsstp + 110 * nf + (0 if c["kind"] == "dry" else 1200)
    if c.get("learned"):
        f += 2 * (16 * 256 + 2 * 256 * 256 + 256 * 9)
    return b * cells, f * cells


def work(case):
    if case["kind"] == "mlp":
        macs = 16 * 256 + 2 * 256 * 256 + 256 * 9
        p = 256 * 64 + 2 * 256 * 256 + 256 * 64 + 3 * 256 + 64
        return {"bytes": 4.0 * (case["n"] * 25 + 2 * p + 1), "flops": 6.0 * macs * case["n"]}
    if case["kind"] == "acoustic":
        cells = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": (48.0 * case["nsstp"] + 16) * cells, "flops": 110.0 * case["nsstp"] * cells}
    if case["kind"] == "ensemble":
        parts = [(c, c["nx"] * c["ny"] * c["nz"], 5) for c in _member_cases(case)]
    else:
        nf = 5 if case["kind"] == "dry" else 14 + (case["tubopt"] == 2)
        parts = [(case, case["nx"] * case["ny"] * case["nz"], nf)]
    b = f = 0.0
    for c, cells, nf in parts:
        sb, sf = _step_work(c, cells)
        b += case["steps"] * sb + 4 * nf * cells
        f += case["steps"] * sf
    return {"bytes": b, "flops": f}


def tolerance(case):
    """About four times what two correct FP32 forms of the path differ by
    (the HE-VI tiles against one another, and the dry step against exact())."""
    return TOLERANCE[case["kind"] if not case.get("learned") else "learned"]


TOLERANCE = {
    "acoustic": {"rel": 5e-6, "max": 4e-5},   # 1e-6 and 9e-6 between two tiles, 20 substeps
    "dry": {"rel": 1e-4, "max": 1e-3},        # 2.8e-5 and 2.1e-4 between two tiles, 12 steps; 1.6e-5 against exact()
    # thresholds of the microphysics take the other branch in a few cells:
    # 2.9e-4 and 0.12 between two tiles (graupel number, 12 steps)
    "moist": {"rel": 1e-3, "max": 0.5},
    "ensemble": {"rel": 1e-3, "max": 0.5},
    "learned": {"rel": 1e-3, "max": 0.5},
    "mlp": {"rel": 1.5e-2, "max": 0.5},       # 3.8e-3 against exact(): BF16 operands
}


# ---------------------------------------------------------------- the same in 64 bits

def _f32(x):
    return float(np.float32(x))


class _Dry64:
    """The dry step and the acoustic loop over the periodic interior (nx x ny
    columns, levels by index k = 0..nk) in float64: neighbours are rolls."""

    def __init__(self, case):
        self.c = case
        self.nk = nk = case["nz"] + 3
        d = _device()
        cols = _columns(_key(case), nk)
        self.b = {n: torch.as_tensor(np.asarray(cols[n], np.float32).astype(np.float64), device=d)[:, None, None]
                  for n in model.BASE_NAMES + ["ubr", "vbr", "rbct"]}
        self.ksp0 = cols["ksp0"]
        self.sth = case.get("sthopt", 1)
        self.dxi, self.dyi = 1.0 / _f32(case["dx"]), 1.0 / _f32(case["dx"])
        self.dz = _f32(cols["dz"])
        self.dzi = 1.0 / self.dz
        self.g, self.wei = 9.8, _f32(0.6)

    def load(self, a):
        """A host-layout field's physical points with a level 0."""
        x = a[:, 2:-3, 2:-3].double()
        return torch.cat([torch.zeros_like(x[:1]), x])

    def wc(self, w):
        r = torch.zeros_like(w)
        r[2:self.nk] = w[2:self.nk] / self.b["jcb8w"][2:self.nk] if self.sth else w[2:self.nk]
        return r

    def substeps(self, f, frc, nsstp, dts):
        nk, b, g, wei, dzi = self.nk, self.b, self.g, self.wei, self.dzi
        s, m = slice(2, nk - 1), slice(3, nk - 1)    # k = 2..nk-2 and 3..nk-2
        m1 = slice(2, nk - 2)
        u, v, w, p = (f[n].clone() for n in ("u", "v", "w", "pp"))
        wc = self.wc(w)
        e = lambda a: torch.roll(a, -1, 2)
        n_ = lambda a: torch.roll(a, -1, 1)
        implicit = self.c.get("impopt", 1) == 1
        dch = 0.05 / dts * _f32(self.c["dx"]) ** 2
        dcv = 0.05 / dts * self.dz ** 2
        if implicit:   # the w system's coefficients and elimination (s_stepwi, s_gaussel)
            t1 = 0.5 * g * b["rbr"] / b["rcsq"]
            t2 = dzi / b["jcb"]
            fw, wm = t1 + t2, t1 - t2
            a = (dts * wei) ** 2 * dzi / b["rst8w"][m]
            bb = 0.5 * g * (dts * wei) ** 2 / b["rst8w"][m]
            mm = bb * b["rst"][m1] - a * b["rcsq"][m1]
            nn = bb * b["rst"][m] + a * b["rcsq"][m]
            lower = (mm * fw[m1]).flatten().tolist()
            diag = (1.0 + (mm * wm[m1] + nn * fw[m])).flatten().tolist()
            upper = (nn * wm[m]).flatten().tolist()
        for _ in range(nsstp):
            U, V, W = b["rst8u"] * u, b["rst8v"] * v, b["rst8w"] * wc
            div = torch.zeros_like(p)
            div[1:nk] = (W[1:nk] - W[2:nk + 1]) * dzi + (U - e(U))[1:nk] * self.dxi + (V - n_(V))[1:nk] * self.dyi
            q = p + dcv * b["jcb"] * div
            wpg = torch.zeros_like(p)
            wpg[2:nk] = (q[1:nk - 1] - q[2:nk]) * dzi
            q = b["jcb"] * p + dch * div
            u[s] += dts * (frc["u"] + (torch.roll(q, 1, 2) - q) * self.dxi)[s] / b["rst8u"][s]
            v[s] += dts * (frc["v"] + (torch.roll(q, 1, 1) - q) * self.dyi)[s] / b["rst8v"][s]
            for a_ in (u, v):
                a_[1], a_[nk - 1] = a_[2], a_[nk - 2]
            U, V = b["jcb8u"] * u, b["jcb8v"] * v
            hdiv = ((U - e(U)) * self.dxi + (V - n_(V)) * self.dyi)
            if implicit:
                fp = torch.zeros_like(p)
                up = lambda w_: g * 0.5 * (w_[2:nk - 1] + w_[3:nk]) * b["rst"][s] + \
                    b["rcsq"][s] * (w_[2:nk - 1] - w_[3:nk]) * dzi
                fp[s] = frc["pp"][s] + b["rcsq"][s] * hdiv[s] + (1.0 - wei) * up(w)
                r = torch.zeros_like(p)
                fj = fp / torch.where(b["jcb"] == 0, torch.ones_like(b["jcb"]), b["jcb"])
                wb = torch.zeros_like(p)
                wb[s] = (p[s] * b["rst"][s] + fp[s] * b["rbr"][s] * dts * wei) / b["rcsq"][s] * (-0.5 * g)
                r[m] = frc["w"][m] + wpg[m] + (fj[m1] - fj[m]) * dts * dzi * wei + (wb[m1] + wb[m])
                y = w[m] + dts * r[m] / b["rst8w"][m]
                ss, n = [], y.shape[0]
                for k in range(n):
                    aa = 1.0 / (diag[k] - (lower[k] * ss[k - 1] if k else 0.0))
                    ss.append(upper[k] * aa)
                    y[k] = (y[k] - lower[k] * y[k - 1]) * aa if k else y[k] * aa
                for k in range(n - 2, -1, -1):
                    y[k] -= ss[k] * y[k + 1]
                w = w.clone()
                w[m] = y
            else:
                r = torch.zeros_like(p)
                r[2:nk] = frc["w"][2:nk] + wpg[2:nk]
                wb = torch.zeros_like(p)
                wb[s] = p[s] * b["rst"][s] / b["rcsq"][s] * (-0.5 * g)
                r[m] += wb[m1] + wb[m]
                w = w.clone()
                w[2:nk] += dts * r[2:nk] / b["rst8w"][2:nk]
            wc = self.wc(w)
            w[1], w[nk] = -b["jcb8w"][3] * wc[3], -b["jcb8w"][nk - 2] * wc[nk - 2]
            w[2], w[nk - 1] = 0.0, 0.0
            if implicit:
                fp[s] += wei * up(w)
            else:
                J = b["jcb8w"] * wc
                fp = torch.zeros_like(p)
                fp[s] = frc["pp"][s] + g * 0.5 * (w[2:nk - 1] + w[3:nk]) * b["rst"][s] + \
                    b["rcsq"][s] * ((J[2:nk - 1] - J[3:nk]) * dzi + hdiv[s])
            p = p.clone()
            p[s] += dts * fp[s] / b["jcb"][s]
            p[1], p[nk - 1] = 2.0 * p[2] - p[3], p[nk - 2]
        return {"u": u, "v": v, "w": w, "pp": p}

    def smooth(self, a, klo, khi):
        """4th-order smoothing of a over levels klo..khi (smhcoe 0.001, smvcoe 0.0004)."""
        t1 = torch.roll(a, -1, 2) + torch.roll(a, 1, 2) - 2.0 * a
        t2 = torch.roll(a, -1, 1) + torch.roll(a, 1, 1) - 2.0 * a
        t3 = torch.zeros_like(a)
        t3[klo:khi + 1] = a[klo + 1:khi + 2] + a[klo - 1:khi] - 2.0 * a[klo:khi + 1]
        t3[klo - 1], t3[khi + 1] = t3[klo], t3[khi]
        r = torch.zeros_like(a)
        k = slice(klo, khi + 1)
        h = (2.0 * t1 - torch.roll(t1, -1, 2) - torch.roll(t1, 1, 2) +
             2.0 * t2 - torch.roll(t2, -1, 1) - torch.roll(t2, 1, 1))
        r[k] = _f32(0.001) * h[k] + _f32(0.0004) * (2.0 * t3[k] - t3[klo + 1:khi + 2] - t3[klo - 1:khi])
        return r

    def advect(self, fx, fy, fz, a, wpoint=False, qx=None, qy=None, qz=None):
        """4th-order horizontal, 2nd- or 4th-order vertical advection of a.
        fx, fy, fz: fluxes at the west, south and lower faces of a's point;
        qx, qy, qz: the flux sums of the 2-delta differences where they are
        not the sum of the two faces (a wind along its own direction)."""
        nk = self.nk
        E, N, W, S = (lambda x: torch.roll(x, -1, 2)), (lambda x: torch.roll(x, -1, 1)), \
            (lambda x: torch.roll(x, 1, 2)), (lambda x: torch.roll(x, 1, 1))
        t1 = fx * (a - W(a)) * (-0.5 * self.dxi)
        t2 = fy * (a - S(a)) * (-0.5 * self.dyi)
        q1 = (fx + E(fx) if qx is None else qx) * (E(a) - W(a)) * (self.dxi / 24.0)
        q2 = (fy + N(fy) if qy is None else qy) * (N(a) - S(a)) * (self.dyi / 24.0)
        h = 4.0 / 3.0 * (t1 + E(t1) + t2 + N(t2)) + W(q1) + E(q1) + S(q2) + N(q2)
        z = torch.zeros_like(a)
        t3 = torch.zeros_like(a)
        hi = nk if wpoint else nk - 1
        t3[2:hi + 1] = fz[2:hi + 1] * (a[2:hi + 1] - a[1:hi]) * (-0.5 * self.dzi)
        z[2:hi] = t3[2:hi] + t3[3:hi + 1]
        if self.c.get("advopt", 2) == 3:
            q = torch.zeros_like(a)
            fs = fz[2:hi] + fz[3:hi + 1] if qz is None else qz[2:hi]
            q[2:hi] = fs * (a[3:hi + 1] - a[1:hi - 1]) * (self.dzi / 24.0)
            k = slice(3, hi - 1)
            z[k] = 4.0 / 3.0 * z[k] + q[2:hi - 2] + q[4:hi]
        return h + z

    def step(self, past, now, dtb, nsstp, dts, filt):
        nk, b = self.nk, self.b
        up = lambda x: torch.cat([x[:1] * 0, x[:-1]])          # x[k-1]
        dn = lambda x: torch.cat([x[1:], x[-1:] * 0])          # x[k+1]
        W, S, E, N = (lambda x: torch.roll(x, 1, 2)), (lambda x: torch.roll(x, 1, 1)), \
            (lambda x: torch.roll(x, -1, 2)), (lambda x: torch.roll(x, -1, 1))
        one = torch.ones_like(b["jcb"])
        inv = lambda x: torch.where(x == 0, 0 * one, 1.0 / torch.where(x == 0, one, x))
        u, v, w, pp, pt = (now[n] for n in DRY)
        wc = self.wc(w)
        X, Y, Z = b["rst8u"] * u, b["rst8v"] * v, b["rst8w"] * wc
        frc = {}
        frc["u"] = self.smooth(b["rst8u"] * (past["u"] - b["ubr"]) * inv(b["jcb8u"]), 2, nk - 2)
        frc["v"] = self.smooth(b["rst8v"] * (past["v"] - b["vbr"]) * inv(b["jcb8v"]), 2, nk - 2)
        frc["w"] = self.smooth(b["rst8w"] * past["w"] * inv(b["jcb8w"]), 2, nk - 1)
        ks = slice(self.ksp0 - 1, nk - 1)
        kw = slice(self.ksp0, nk)
        r8 = 0.5 * (b["rbct"] + dn(b["rbct"]))
        frc["u"][ks] -= (b["rst8u"] * r8 * (past["u"] - b["ubr"]))[ks]
        frc["v"][ks] -= (b["rst8v"] * r8 * (past["v"] - b["vbr"]))[ks]
        frc["w"][kw] -= (b["rbct"] * b["rst8w"] * past["w"])[kw]
        if self.c.get("coropt"):
            fc = _f32(2.1e-5)
            t = fc * b["rst"] * (v + N(v))
            frc["u"] += W(t) + t
            t = -fc * b["rst"] * (u + E(u))
            frc["v"] += S(t) + t
        wb = 0.5 * self.g * b["rst"] * pt * inv(b["ptbr"])
        m = slice(3, nk - 1)
        frc["w"][m] += (up(wb) + wb)[m]
        frc["u"] += self.advect(0.5 * (W(X) + X), 0.5 * (W(Y) + Y), 0.5 * (W(Z) + Z), u, qx=W(X) + E(X))
        frc["v"] += self.advect(0.5 * (S(X) + X), 0.5 * (S(Y) + Y), 0.5 * (S(Z) + Z), v, qy=S(Y) + N(Y))
        frc["w"] += self.advect(0.5 * (up(X) + X), 0.5 * (up(Y) + Y), 0.5 * (up(Z) + Z), w, True, qz=up(Z) + dn(Z))
        frc["pp"] = self.advect(b["jcb8u"] * u, b["jcb8v"] * v, b["jcb8w"] * wc, pp) + \
            self.smooth(past["pp"], 2, nk - 2)
        ft = self.advect(X, Y, Z, pt) + self.smooth(b["rbr"] * past["ptp"], 2, nk - 2)
        ft[ks] -= (0.5 * (b["rbct"] + dn(b["rbct"])) * b["rst"] * past["ptp"])[ks]
        t = torch.zeros_like(w)
        t[2:nk] = ((up(b["rbr"]) + b["rbr"]) * w * (up(b["ptbr"]) - b["ptbr"]))[2:nk] * (0.25 * self.dzi)
        ft += t + dn(t)
        fut = self.substeps(past, frc, nsstp, dts)
        f = past["ptp"].clone()
        f[2:nk - 1] += 2.0 * dtb * (ft * inv(b["rst"]))[2:nk - 1]
        f[1], f[nk - 1] = f[2], f[nk - 2]
        fut["ptp"] = f
        if filt:
            fc = _f32(0.1)
            now = {n: (1.0 - 2.0 * fc) * now[n] + fc * (fut[n] + past[n]) for n in DRY}
        return now, fut


def _defined(name, x, nk):
    """The levels _interior() keeps."""
    return x[1:nk + (name == "w")]


def exact(case, seed):
    if case["kind"] == "mlp":
        return _mlp_exact(case, seed)
    if case["kind"] == "acoustic":
        d = _Dry64(case)
        st, fr = _acoustic_state(case, seed)
        f = {n: d.load(a) for n, a in st.items()}
        r = d.substeps(f, {n: d.load(a) for n, a in fr.items()}, case["nsstp"], float(np.float32(case["dts"])))
        return {n: _defined(n, a, d.nk) for n, a in r.items()}
    if case["kind"] == "dry":
        d = _Dry64(case)
        past = {n: d.load(a) for n, a in _state(case, seed).items()}
        now = {n: a.clone() for n, a in past.items()}
        nsstp = nsstp_of(case["dtbig"], case["dtsml"])
        for k in range(case["steps"]):
            h = 0.5 if k == 0 else 1.0
            past, now = d.step(past, now, h * case["dtbig"], nsstp, h * case["dtsml"], k > 0)
        return {n: _defined(n, now[n], d.nk) for n in DRY}
    return None


def _mlp_exact(case, seed):
    rng = _Random(seed, case["n"])
    p = _mlp_params(rng).double().requires_grad_(True)
    x, t = rng.normal((case["n"], 16)).double(), rng.normal((case["n"], 9)).double()
    o, parts = 0, []
    for shape in ((256, 64), (256,), (256, 256), (256,), (256, 256), (256,), (256, 64), (64,)):
        n = math.prod(shape)
        parts.append(p[o:o + n].reshape(shape))
        o += n
    w1, b1, w2, b2, w3, b3, w4, b4 = parts
    a = torch.nn.functional.pad(x, (0, 48))
    for w, b in ((w1, b1), (w2, b2), (w3, b3)):
        a = torch.nn.functional.silu(a @ w.T + b)
    y = (a @ w4 + b4)[:, :9]
    loss = ((y - t) ** 2).mean()
    loss.backward()
    return {"loss": loss.detach().reshape(1), "grad": p.grad}
