"""The moist scalars' kernel, the sedimentation's sweeps and the microphysics'
per-level table at their edges, against the CPU oracle with the criteria of the moist large steps
(every case here is two steps of the same state at another size): blocks with
one column pair or one row beyond a tile, and columns of a few levels, where
the vertical stencils are clamped at both ends and a block's chunk is cut
short, for each form of the kernel (with and without turbulence, 2nd- and
4th-order vertical advection)."""
import numpy as np
import pytest

from test_micro_gpu import MICRO, compare, setup_solver
from test_moist_gpu import NAMES, check, run_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,tubopt,advopt", [
    (33, 9, 7, 1, 3), (32, 8, 6, 0, 2), (65, 17, 8, 0, 3), (31, 10, 9, 1, 2), (34, 8, 11, 1, 3)])
def test_moist_scalars_edges(cress, oracle_lib, monkeypatch, nx, ny, nz, tubopt, advopt):
    # a lower model top, which the few layers reach
    from cress_b200 import cases
    whole = cases.supercell_case
    monkeypatch.setattr(cases, "supercell_case", lambda *a, **kw: whole(*a, **dict(kw, ztop=300.0 * nz)))
    dims, ref, got = run_case(cress, oracle_lib, nx, ny, nz, 2, seed=nx + nz, tubopt=tubopt, advopt=advopt,
                              dtbig=2.0)
    check(dims, ref, got)


@pytest.mark.parametrize("nz,dz,dtb,npstp", [
    (6, 300.0, 2.0, 1), (6, 300.0, 10.0, 2), (6, 300.0, 20.0, 3), (12, 900.0, 90.0, 4), (6, 300.0, 40.0, 5),
    (17, 700.0, 120.0, 6), (20, 600.0, 120.0, 7), (6, 300.0, 70.0, 9)])
def test_sedimentation_sweeps(cress, oracle_lib, nz, dz, dtb, npstp):
    # one to four sub-steps per sweep and more than one sweep, in columns shorter
    # and longer than a batch of loads; criteria of test_micro_gpu
    from cress_b200 import cases
    dims, base, past, fut, _ = cases.micro_case(34, 33, nz, dz, seed=nz)
    ni, nj, nk = dims
    ref = {k: v.copy() for k, v in fut.items()}
    prec_ref = np.zeros((5, 2, nj + 2, ni + 2), np.float32)
    assert oracle_lib.cloudphy(dims, base, past, ref, prec_ref, dtb, dz) == npstp
    s = setup_solver(cress, dims, base, dz)
    for k in MICRO:
        s.put_field(k, cress.PAST, past[k])
        s.put_field(k, cress.FUTURE, fut[k])
    s.put_field("pp", cress.PAST, past["pp"])
    s.cloudphy(dtb)
    got = {k: s.get_field(k, cress.FUTURE) for k in MICRO}
    prec = s.get_precip()
    s.close()
    sl = (slice(0, nk - 1), slice(2, nj - 1), slice(2, ni - 1))
    for k in MICRO:
        compare(k, got[k][sl], ref[k][sl])
    psl = (slice(None), slice(None), slice(2, nj - 1), slice(2, ni - 1))
    assert float(np.abs(prec[psl] - prec_ref[psl]).max()) <= 1e-3 * float(np.abs(prec_ref[psl]).max()) + 1e-30


def test_base_state_set_again(cress):
    # the microphysics' level table follows the base state: another one set
    # before, and used, leaves no trace
    from cress_b200 import cases
    case = cases.supercell_case(34, 12, 10, 1000.0, ztop=3000.0, seed=4, cloud=True, rad=(6000.0, 6000.0, 1400.0))
    ni, nj, nk = case["dims"]
    base = case["base"]
    other = dict(base, pbr=base["pbr"] * np.float32(.97), rbr=base["rbr"] * np.float32(.9),
                 rst=base["rst"] * np.float32(.9))
    init = dict(zip(NAMES, list(case["level"]) + [case["moist"][n] for n in NAMES[5:]]))
    out = []
    for bases in ((base,), (other, base)):
        s = cress.Solver(ni, nj, nk, 1000.0, 1000.0, case["dz"], sthopt=1, cphopt=3, thresq=1e-12)
        for b in bases:
            s.set_base3d(b)
            s.set_base_moist(b["pbr"], b["qvbr"])
            for n in NAMES[3:]:
                s.put_field(n, cress.PAST, init[n])
                s.put_field(n, cress.FUTURE, init[n])
            s.cloudphy(10.0)
        out.append({n: s.get_field(n, cress.FUTURE) for n in NAMES[4:]})
        s.close()
    changed = 0
    for n in out[0]:
        assert np.array_equal(out[0][n], out[1][n]), n
        changed += int((out[0][n] != init[n]).sum())
    assert changed
