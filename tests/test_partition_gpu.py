"""A small periodic domain, repeated in x and y, is the same model state on a
larger grid.  How the kernels cut the work depends on the grid: strips of one row
or of many, the column whole or in level chunks, tiles at the domain's edge or
inside.  None of it may show: every copy equals the small run bit for bit, at
both time levels, after three large steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DRY = ["u", "v", "w", "pp", "ptp"]
MOIST = DRY + ["qv", "qc", "qr", "qi", "qs", "qg", "ni", "ns", "ng"]
NX, NY = 40, 24


def widen(core, rx, ry):
    """The physical points (nk, NY, NX) repeated, in the host layout with both
    ghost layers."""
    nj, ni = NY * ry + 3, NX * rx + 3
    j, i = (np.arange(nj + 2) - 2) % NY, (np.arange(ni + 2) - 2) % NX
    return np.ascontiguousarray(core[:, j][:, :, i])


def run(cress, oracle_lib, case, init, rx, ry, impopt, tubopt, advopt, dx, dtbig, dtsml):
    from cress_b200 import cases
    nk = case["dims"][2]
    ni, nj = NX * rx + 3, NY * ry + 3
    moist = len(init) > 6
    names = list(init)
    zph = case["zph"]
    rbct, ksp0 = oracle_lib.vspdmp(nk, zph, 0.005, 0.6 * zph[nk - 1])
    base = {n: np.broadcast_to(a[:, :1, :1], (nk, nj + 2, ni + 2)) for n, a in case["base"].items()}
    s = cress.Solver(ni, nj, nk, dx, dx, case["dz"], sthopt=1, cphopt=3 if moist else 0, impopt=impopt,
                     tubopt=tubopt, advopt=advopt)
    s.set_base3d(base)
    s.set_base_large(base["ubr"], base["vbr"], cases.expand(rbct, ni, nj, nk), ksp0)
    if moist:
        s.set_base_moist(base["pbr"], base["qvbr"])
    for n, a in init.items():
        full = widen(a, rx, ry)
        s.put_field(n, cress.PAST, full)
        s.put_field(n, cress.NOW, full)
    nsstp = 20 * int(1.e2 * (dtbig + .001)) // int(1.e3 * (dtsml + .0001))
    for step in range(3):
        h = 0.5 if step == 0 else 1.0
        s.large_step(round(step * dtbig * 1000), h * dtbig, nsstp, h * dtsml)
    out = {(n, l): s.get_field(n, l)[:nk - (n != "w"), 2:nj - 1, 2:ni - 1] for n in names
           for l in (cress.PAST, cress.NOW)}
    s.close()
    return out


@pytest.mark.parametrize("kind,nz,rx,ry,impopt,tubopt,advopt", [
    ("dry", 24, 11, 13, 1, 0, 3),
    ("dry", 7, 11, 13, 1, 0, 2),      # several blocks per SM
    ("dry", 37, 11, 13, 1, 1, 2),
    ("dry", 30, 11, 13, 0, 1, 2),
    ("dry", 78, 7, 13, 1, 0, 2),
    ("moist", 48, 11, 13, 1, 0, 2),
    ("moist", 54, 11, 13, 1, 2, 2),
    ("moist", 26, 23, 15, 1, 1, 3),
])
def test_copies_of_a_periodic_domain(cress, oracle_lib, kind, nz, rx, ry, impopt, tubopt, advopt):
    from cress_b200 import cases
    if kind == "dry":
        dx, dtbig, dtsml = 500.0, 2.0, 0.25
        case = cases.dry_case(NX, NY, nz, dx, 300.0, sthopt=1, seed=nz, vspbar=0.005, dthdz=0.0, noise=0.5)
        case["dz"] = 300.0
        init = dict(zip(DRY, case["level"]))
    else:
        dx, dtbig, dtsml = 1000.0, 5.0, 1.0
        case = cases.supercell_case(NX, NY, nz, dx, ztop=10000.0, seed=nz, cloud=True, rad=(5000.0, 5000.0, 1400.0))
        init = dict(zip(MOIST, list(case["level"]) + [case["moist"][n] for n in MOIST[5:]]))
    if tubopt == 2:
        rng = np.random.default_rng(nz)
        init["tke"] = rng.uniform(0.0, 1.0, init["u"].shape).astype(np.float32)
    init = {n: a[:, 2:NY + 2, 2:NX + 2].copy() for n, a in init.items()}
    args = (impopt, tubopt, advopt, dx, dtbig, dtsml)
    small = run(cress, oracle_lib, case, init, 1, 1, *args)
    large = run(cress, oracle_lib, case, init, rx, ry, *args)
    for key, a in small.items():
        assert np.isfinite(a).all(), key
        assert np.array_equal(np.tile(a, (1, ry, rx)), large[key]), key
