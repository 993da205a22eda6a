"""The row-marching HE-VI kernel (tiles 0 and 13) where its partition can go
wrong: widths around its 60-column tiles, column heights around its chunk
lengths (2, 3, 4 and 5 levels per warp) and a partial top chunk, strips of one
row, and several substeps, so that the second and later ones read the rows
whose periodic images are not written in between.  Against the FP32 oracle with
the small step's tolerance (test_small_gpu.py)."""
import numpy as np
import pytest

import helpers as H

from test_ensemble_gpu import NAMES, member
from test_small_gpu import check, run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [
    (5, 5, 5),       # the smallest grid cress_create takes
    (59, 7, 32),     # one tile with an odd last column; 16 chunks of 2
    (60, 9, 33),     # a full tile; chunks of 3
    (61, 6, 48),     # a second tile of one column
    (120, 13, 49),   # two full tiles; chunks of 4
    (181, 5, 65),    # a last tile of one column; chunks of 5, the last one full
    (62, 21, 78),    # a partial top chunk
])
def test_partition_edges(cress, oracle_lib, nx, ny, nz):
    ni, nj, nk, ref, out = run_pair(cress, oracle_lib, nx, ny, nz, 3, sthopt=1, seed=nx + nz, tile=0)
    check(ni, nj, nk, ref, out, 3)


@pytest.mark.parametrize("divopt,sthopt", [(0, 1), (1, 0), (2, 0)])
def test_options(cress, oracle_lib, divopt, sthopt):
    ni, nj, nk, ref, out = run_pair(cress, oracle_lib, 70, 34, 27, 4, sthopt=sthopt, divopt=divopt, seed=4, tile=0)
    check(ni, nj, nk, ref, out, 4)


@pytest.mark.parametrize("nx,ny,nz", [
    (250, 118, 20),   # chunks of 2, strips of 5 rows, the last of 3
    (130, 259, 37),   # chunks of 3, strips of 6 rows, the last of 1
    (190, 203, 54),   # chunks of 4, strips of 6 rows, the last of 5
    (190, 151, 80),   # 16 full chunks of 5, strips of 5 rows, the last of 1
])
def test_strips_of_several_rows(cress, oracle_lib, nx, ny, nz):
    # what a solved row leaves for the next: parked values, the exchange
    # buffers used again, the copies' parity over many rows; tiles without edge
    ni, nj, nk, ref, out = run_pair(cress, oracle_lib, nx, ny, nz, 3, sthopt=1, seed=nx + nz, tile=0)
    check(ni, nj, nk, ref, out, 3)


def test_levels_beyond_the_chunks_run_the_ring_kernel(cress, oracle_lib):
    ni, nj, nk, ref, out = run_pair(cress, oracle_lib, 40, 12, 82, 2, sthopt=1, seed=8, tile=0, dz=150.0)
    check(ni, nj, nk, ref, out, 2)


def test_tile_13_is_tile_0_up_to_its_height(cress, oracle_lib):
    """Tiles 0 and 13 are one kernel up to nk = 68, which the autotuner times
    once; above, tile 13 stays refused."""
    for nz in (65, 66):
        ni, nj, nk = H.dims(24, 12, nz)
        base = H.base3d(ni, nj, nk, 200.0, 1)
        st, frc = H.small_state(ni, nj, nk, 2, base)
        out = []
        for tile in (0, 13):
            s = cress.Solver(ni, nj, nk, 1000.0, 1000.0, 200.0, sthopt=1, tile=tile)
            s.set_base3d(base)
            if tile == 13 and nk > 68:
                with pytest.raises(cress.CressError) as e:
                    s.smalldrv(2, 0.5, *st, *frc)
                assert e.value.code == 2             # CRESS_E_UNSUPPORTED
            else:
                out.append(s.smalldrv(2, 0.5, *st, *frc))
                best, ms = s.autotune(2, 0.5, reps=2)
                assert ms[0] > 0 and best != 13
                assert ms[13] == (ms[0] if nk <= 68 else -1)
            s.close()
        for a in out[1:]:
            for x, y in zip(out[0], a):
                assert np.array_equal(x, y)


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("sizes", [
    [(40, 33, 22, 1), (64, 20, 36, 2), (29, 45, 22, 3)],
    [(190, 41, 22, 1), (131, 70, 22, 2), (64, 20, 22, 3)],   # members with tiles inside the edges, strips of two rows
    # one launch for heights of equal chunk length (22 and 30: 11 and 15 warps), four in all
    [(40, 33, 22, 1), (64, 20, 30, 2), (29, 45, 40, 3), (24, 18, 54, 4), (31, 25, 60, 5), (24, 20, 69, 6)],
])
def test_ensemble_of_different_heights_matches_members(cress, oracle_lib, sizes, graphs):
    """Members of different heights share a launch where their chunks are
    equally long; each equals the member stepped alone, bit for bit."""
    out = []
    for together in (False, True):
        sols = [member(cress, oracle_lib, *sz) for sz in sizes]
        ens = cress.Ensemble(sols, graphs=graphs) if together else None
        for step in range(9 if graphs else 2):
            h = 0.5 if step == 0 else 1.0
            for s in [ens] if together else sols:
                s.large_step(step * 5000, 5.0 * h, 10, h)
        out.append([s.get_field(n, cress.NOW) for s in sols for n in NAMES])
        if ens:
            ens.close()
        for s in sols:
            s.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("nx,ny,nz", [
    (61, 9, 26),     # 13 chunks of 2, the last one full
    (61, 9, 33),     # 11 full chunks of 3
    (61, 9, 40),     # 14 chunks of 3, one level in the last: it holds nk-1 and nk as well
    (61, 9, 41),     # two levels in the last: nk-1
    (61, 9, 49),     # 13 chunks of 4, one level in the last
    (61, 9, 64),     # 16 full chunks of 4
    (61, 9, 72),     # 15 chunks of 5, two levels in the last
    (61, 9, 80),     # 16 full chunks of 5: the tallest column and the most shared memory
])
def test_levels_the_operator_does_not_read_may_hold_anything(cress, oracle_lib, nx, ny, nz):
    """NaN in every level that s_hevi does not read: the forcings below level 2
    and above nk-2, that of w at level 2 too, and u, v, p', w below the first and
    above the last level they are used at.  The oracle's interior does not
    change by a bit, and the kernel's is the same as without them."""
    ni, nj, nk = H.dims(nx, ny, nz)
    dz = 18000.0 / nz
    base = H.base3d(ni, nj, nk, dz, 1)
    st, frc = H.small_state(ni, nj, nk, nz, base)
    nst, nfrc = [a.copy() for a in st], [a.copy() for a in frc]
    for n, a in enumerate(nst):       # index k-1; w is used at nk-1, the others up to nk-2
        a[0] = np.nan
        a[nk - 1 if n == 2 else nk - 2:] = np.nan
    for a in nfrc:
        a[0] = a[nk - 2:] = np.nan
    nfrc[2][1] = np.nan
    cfg = dict(ni=ni, nj=nj, nk=nk, dx=1000.0, dy=1000.0, dz=dz, sthopt=1, divopt=2, buyopt=1, weicoe=0.6)
    inner = (slice(1, nk - 2), slice(1, nj), slice(1, ni))
    want = [oracle_lib.small_steps(cfg, base, f, [a.copy() for a in s], 3, 0.5, prec=32, fp64_solve=1)
            for s, f in ((st, frc), (nst, nfrc))]
    out = []
    for s_, f in ((st, frc), (nst, nfrc)):
        s = cress.Solver(ni, nj, nk, 1000.0, 1000.0, dz, sthopt=1)
        s.set_base3d(base)
        out.append(s.smalldrv(3, 0.5, *s_, *f))
        s.close()
    for name, a, b, c, d in zip(("u", "v", "w", "pp"), *want, *out):
        assert np.array_equal(a[inner], b[inner]), name
        assert np.isfinite(d[inner]).all(), name
        assert np.array_equal(c[inner], d[inner]), name
    check(ni, nj, nk, want[0], out[0], 3)
