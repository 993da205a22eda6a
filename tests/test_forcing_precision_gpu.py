"""The smoothing in the forcing of u against 64 bits where a strong base wind
carries small departures.  u varies along y and z alone and v = w = 0, so that
advection vanishes exactly and the forcing is the 4th-order smoothing of
rst8u (u - ubr) / jcb8u (smoo4uvw.f90).

Bar: u, the departures' differences and the per-level constants carry one FP32
rounding each, and the horizontal part adds eight differences, weighted 4 and 1,
of the departures' own size: a 2-norm error of at most sixteen half-ulps of the
result, 16 * 2^-24 = 1e-6.  Rounded with the whole wind it is 80 times the
wind's own ulp over the departure, 1e-5 at 60 m/s."""
import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wind", [0.0, 40.0, -60.0])
def test_smoothing_of_departures_from_a_strong_wind(cress, wind):
    nx, ny, nz, dz = 40, 37, 30, 300.0
    ni, nj, nk = H.dims(nx, ny, nz)
    base = H.base3d(ni, nj, nk, dz, 1)
    rng = np.random.default_rng(5)
    ubr = (wind * (1.0 + 0.02 * np.arange(nk))).astype(np.float32)
    u = np.empty((nk, nj + 2, ni + 2), np.float32)
    u[:] = (ubr[:, None] + 0.5 * rng.standard_normal((nk, nj + 2)).astype(np.float32))[:, :, None]
    H.bcycle(u, "u")
    zero = np.zeros_like(u)
    s = cress.Solver(ni, nj, nk, 1000.0, 1000.0, dz, sthopt=1)
    s.set_base3d(base)
    s.set_base_large(H.expand(np.concatenate([[0], ubr]).astype(np.float32), ni, nj, nk), zero, zero, nk)
    for n, a in (("u", u), ("v", zero), ("w", zero), ("pp", zero), ("ptp", zero)):
        s.put_field(n, cress.PAST, a)
        s.put_field(n, cress.NOW, a)
    s.large_step(0, 1.0, 1, 1.0)
    got = s.get_field("u", cress.FORCING)[1:nk - 2, 2:nj - 1, 4].astype(np.float64)   # levels 2..nk-2
    s.close()

    a = (base["rst8u"][:, 2:nj - 1, 4].astype(np.float64) * (u[:, 2:nj - 1, 4].astype(np.float64) - ubr[:, None]) /
         base["jcb8u"][:, 2:nj - 1, 4])
    t2 = np.roll(a, -1, 1) + np.roll(a, 1, 1) - 2 * a
    h = 2 * t2 - np.roll(t2, -1, 1) - np.roll(t2, 1, 1)
    t3 = np.zeros_like(a)
    t3[1:nk - 2] = a[2:nk - 1] + a[:nk - 3] - 2 * a[1:nk - 2]
    t3[0], t3[nk - 2] = t3[1], t3[nk - 3]
    k = slice(1, nk - 2)
    want = float(np.float32(0.001)) * h[k] + float(np.float32(0.0004)) * (2 * t3[k] - t3[2:nk - 1] - t3[:nk - 3])
    got, want = got[:, 1:-1], want[:, 1:-1]   # the outermost rows read a second ghost row, which is not set here
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert err <= 1e-6, err
