"""The barriers of the fused inference kernel (cress_b200/csrc/mlp_fused.cuh) in
every order its roles can run: warps 0-3 (features), warps 4-7 (application)
and the MMA thread step through their arrivals and parity waits, and every
interleaving over several tiles is visited.  A wait by parity that can be overtaken
by two phases shows as a state in which nobody can go on.  With one barrier for the
features of all tiles there is such a state; with one for the even and one for
the odd tiles, as the kernel has them, there is none.  CPU only."""
import pytest


def roles(tiles, nx):
    """Each role's program: ("arrive", barrier) and ("wait", barrier, parity)."""
    x = lambda n: ("x", n % nx)
    ph = lambda n: n // nx % 2
    feat, app, mma = [("arrive", x(0))], [], []
    acc = hs = 0                       # phases of acc_full and h_full so far
    for n in range(tiles):
        mma.append(("wait", x(n), ph(n)))
        app.append(("wait", x(n), ph(n)))
        for l in range(4):
            if l > 0 or n > 0:
                mma.append(("wait", "h", hs % 2))
                hs += 1
            mma.append(("arrive", "acc"))
            for r in (feat, app):
                r.append(("wait", "acc", acc % 2))
                r.append(("arrive", "h"))
            acc += 1
            if l == 0 and n + 1 < tiles:
                feat.append(("arrive", x(n + 1)))
    return {"feat": feat, "app": app, "mma": mma}


def stuck_states(tiles, nx):
    prog = roles(tiles, nx)
    names = sorted(prog)
    need = {"h": {"feat", "app"}, "acc": {"mma"}}
    for n in range(nx):
        need[("x", n)] = {"feat"}
    bars = sorted(need, key=str)
    start = (tuple(0 for _ in names), tuple((0, frozenset()) for _ in bars))   # positions; completed phases, arrived
    seen, todo, stuck = {start}, [start], 0
    while todo:
        pos, state = todo.pop()
        moved = False
        for i, r in enumerate(names):
            if pos[i] == len(prog[r]):
                continue
            op = prog[r][pos[i]]
            b = bars.index(op[1])
            done, got = state[b]
            new = list(state)
            if op[0] == "wait":
                if done % 2 == op[2]:          # the phase of this parity is the one under way
                    continue
            else:
                assert r not in got, (r, op)   # an arrival in a phase that already has it
                got = got | {r}
                new[b] = (done + 1, frozenset()) if got == need[op[1]] else (done, got)
            moved = True
            nxt = (pos[:i] + (pos[i] + 1,) + pos[i + 1:], tuple(new))
            if nxt not in seen:
                seen.add(nxt)
                todo.append(nxt)
        if not moved and any(pos[i] < len(prog[r]) for i, r in enumerate(names)):
            stuck += 1
    return stuck


@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 7])
def test_every_order_finishes(tiles):
    assert stuck_states(tiles, 2) == 0


def test_one_barrier_for_all_tiles_can_be_overtaken():
    assert stuck_states(4, 1) > 0
