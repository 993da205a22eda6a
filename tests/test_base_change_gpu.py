"""Another base state set on a context that has already stepped: every table
formed from the old one (elimination factors, level and microphysics
tables), and every captured step, must follow.  The steps after the change equal, bit for
bit, those of a fresh context that was given the second base state and the
fields at the change; eagerly and from CUDA graphs, alone and in an ensemble."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ["u", "v", "w", "pp", "ptp", "qv", "qc", "qr", "qi", "qs", "qg", "ni", "ns", "ng"]
SIZE = (36, 28, 20)


def case_of(nx, ny, nz, seed):
    from cress_b200 import cases
    return cases.supercell_case(nx, ny, nz, 1000.0, ztop=7000.0, seed=seed, cloud=True, rad=(5000.0, 5000.0, 1200.0))


def solver(cress, case, base, damp):
    ni, nj, nk = case["dims"]
    s = cress.Solver(ni, nj, nk, 1000.0, 1000.0, case["dz"], sthopt=1, cphopt=3)
    set_base(s, case, base, damp, "all")
    return s


def set_base(s, case, base, damp, what):
    from cress_b200 import cases
    ni, nj, nk = case["dims"]
    if what in ("3d", "all"):
        s.set_base3d(base)
    if what in ("large", "all"):
        rbct, ksp0 = damp
        s.set_base_large(base["ubr"], base["vbr"], cases.expand(rbct, ni, nj, nk), ksp0)
    if what in ("moist", "all"):
        s.set_base_moist(base["pbr"], base["qvbr"])


def other(base, what):
    """base with the arrays of one call changed."""
    f = np.float32
    b = dict(base)
    if what in ("3d", "all"):
        for n in ("rbr", "rst", "rst8u", "rst8v", "rst8w"):
            b[n] = b[n] * f(.98)
        b["rcsq"] = b["rcsq"] * f(.99)
    if what in ("large", "all"):
        b["ubr"] = b["ubr"] * f(.9)
    if what in ("moist", "all"):
        b["pbr"] = b["pbr"] * f(.995)
    return b


def damping(oracle_lib, case, what):
    zph, nk = case["zph"], case["dims"][2]
    one = oracle_lib.vspdmp(nk, zph, 0.005, 0.6 * zph[nk - 1])
    two = oracle_lib.vspdmp(nk, zph, 0.004, 0.5 * zph[nk - 1])
    return one, (two if what in ("large", "all") else one)


def put(s, cress, case):
    for n, a in zip(NAMES, list(case["level"]) + [case["moist"][n] for n in NAMES[5:]]):
        s.put_field(n, cress.PAST, a)
        s.put_field(n, cress.NOW, a)


def steps(s, first, n):
    for k in range(first, first + n):
        s.large_step(k * 5000, 2.5 if k == 0 else 5.0, 10, 0.5 if k == 0 else 1.0)


def levels(s, cress):
    return [[s.get_field(n, l) for n in NAMES] for l in (cress.PAST, cress.NOW)]


def same(a, b):
    for x, y in zip(a, b):
        for n, p, q in zip(NAMES, x, y):
            assert np.isfinite(q).all(), n
            assert np.array_equal(p, q), n


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("what", ["3d", "large", "moist"])
def test_context_follows(cress, oracle_lib, what, graphs):
    case = case_of(*SIZE, 6)
    d1, d2 = damping(oracle_lib, case, what)
    s = solver(cress, case, case["base"], d1)
    put(s, cress, case)
    s.set_graphs(graphs)
    steps(s, 0, 9)
    at = levels(s, cress)
    two = other(case["base"], what)
    set_base(s, case, two, d2, what)
    steps(s, 9, 9)
    got = levels(s, cress)
    s.close()
    f = solver(cress, case, two, d2)
    f.set_graphs(graphs)
    for l, a in zip((cress.PAST, cress.NOW), at):
        for n, x in zip(NAMES, a):
            f.put_field(n, l, x)
    steps(f, 9, 9)
    want = levels(f, cress)
    f.close()
    same(want, got)


def test_ensemble_follows(cress, oracle_lib):
    sizes = [SIZE, (40, 33, 22)]
    all_cases = [case_of(*sz, 3 + n) for n, sz in enumerate(sizes)]
    damp = [damping(oracle_lib, c, "all") for c in all_cases]
    twos = [other(c["base"], "all") for c in all_cases]
    sols = [solver(cress, c, c["base"], d[0]) for c, d in zip(all_cases, damp)]
    for s, c in zip(sols, all_cases):
        put(s, cress, c)
    ens = cress.Ensemble(sols)
    steps(ens, 0, 9)
    at = [levels(s, cress) for s in sols]
    for s, c, b, d in zip(sols, all_cases, twos, damp):
        set_base(s, c, b, d[1], "all")
    steps(ens, 9, 9)
    got = [levels(s, cress) for s in sols]
    ens.close()
    for s in sols:
        s.close()
    for c, b, d, a, g in zip(all_cases, twos, damp, at, got):
        f = solver(cress, c, b, d[1])
        for l, x in zip((cress.PAST, cress.NOW), a):
            for n, y in zip(NAMES, x):
                f.put_field(n, l, y)
        steps(f, 9, 9)
        same(levels(f, cress), g)
        f.close()


@pytest.mark.parametrize("what", ["3d", "large", "moist"])
def test_refused_base_changes_nothing(cress, oracle_lib, what):
    """A base state with one value out of line in its last array is refused,
    and a host that goes on gets the one in use: also for step lengths it
    uses for the first time, whose tables are formed after the refusal."""
    case = case_of(*SIZE, 8)
    damp, _ = damping(oracle_lib, case, what)
    bad = other(case["base"], what)
    last = {"3d": "rcsq", "large": "vbr", "moist": "qvbr"}[what]
    bad[last] = bad[last].copy()
    at = (SIZE[2] - 2, 9, 11)
    bad[last][at] += np.float32(.01) * abs(bad[last][at]) + np.float32(1e-3)
    out = []
    for refuse in (False, True):
        s = solver(cress, case, case["base"], damp)
        put(s, cress, case)
        steps(s, 0, 1)
        if refuse:
            with pytest.raises(cress.CressError) as e:
                set_base(s, case, bad, damp, what)
            assert e.value.code == 4                 # CRESS_E_NONUNIFORM
        steps(s, 1, 2)
        out.append(levels(s, cress))
        s.cloudphy(7.0)
        out[-1].append([s.get_field(n, cress.FUTURE) for n in NAMES])
        s.close()
    same(*out)
