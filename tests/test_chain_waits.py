"""The waits of the one-launch momentum chain (mom_chain_kernel, k_momentum.cu), replayed
on the CPU.

A line's visits receive their neighbours' values as asynchronous stores into the line's
mailboxes; the stores complete on the line's mbarrier (arrival count one), whose phase the
visiting warp arms with the bytes the visit waits for.  Restated here: the order in which a
warp runs the visits of its (one or two) lines, whom a visit waits for and whom it pushes
to, and the barrier's counts; stores land late and in any order.  Checked, with waits
that run out at any time:

* a phase is armed only when the one before it is over (an arrival on a barrier with no
  arrival pending is undefined);
* every store lands in the phase of the visit it is for;
* no store is under way when a CTA leaves.

The form that went on without waiting once a wait had run out breaks the first, so it is
checked that the replay notices that.  The GPU test at the end lets the waits run out.
"""
import random

import numpy as np
import pytest

T, B, N, S = range(4)
BACK = (B, T, S, N)
DJ, DK = (0, 0, 1, -1), (1, -1, 0, 0)


class Broken(Exception):
    pass


class Barrier:
    """An mbarrier of arrival count one."""

    def __init__(self):
        self.phase, self.pending, self.tx = 0, 1, 0

    def _check(self):
        if self.pending == 0 and self.tx == 0:
            self.phase, self.pending = self.phase + 1, 1

    def arrive_expect(self, n):
        if self.pending == 0:
            raise Broken("armed while the phase before is open")
        self.pending, self.tx = 0, self.tx + n
        self._check()

    def complete(self, n):
        self.tx -= n
        self._check()


def waits(exact, v, c, near):
    """Directions visit v of a line of colour c waits for, of the in-box ones `near`."""
    if exact:
        want = {S} | ({N} if v >= 1 else set()) | ({T} if v % 2 == 0 else set()) | ({B} if v == 2 else set())
        return near & want
    return set() if c == 0 and v == 0 else near


def pushes(exact, v, c, near):
    if exact:
        want = {N} | ({S} if v < 3 else set()) | ({B} if v % 2 else set()) | ({T} if v == 1 else set())
        return near & want
    return set() if c == 1 and v == 3 else near


def fed_visit(exact, d, v):
    """The neighbour's visit that a push of visit v in direction d is for: the first one
    past what it has used that waits for this direction's value."""
    if not exact:
        return None  # by colour, below
    if d == N:
        return v
    if d == S:
        return v + 1
    if d == B:
        return v - 1
    return 2  # d == T, v == 1


def replay(J, K, nc, nw, exact, rng, rule, runout=0.0, dies=0.0):
    """One launch: four equations of four visits a line.  rule "wait": a wait that runs out
    records that and goes on; "go on": visits go on without waiting.  dies: chance that a
    waiting warp gives up for good.  Returns (waits that ran out, warps that gave up)."""
    half = (J + 1) // 2
    nl = J * K if exact else 2 * half * K
    lpc = -(-nl // nc)

    def slot_line(l):
        if l >= nl:
            return None
        if exact:
            return l % J, l // J
        q = l >> 1
        k, r = divmod(q, half)
        j = ((l & 1) - k) % 2 + 2 * r
        return (j, k) if j < J else None

    owner, lines = {}, {}
    for cta in range(nc):
        for loc in range(lpc):
            jk = slot_line(cta * lpc + loc)
            if jk and cta * lpc + loc < nl:
                near = {d for d in range(4) if 0 <= jk[0] + DJ[d] < J and 0 <= jk[1] + DK[d] < K}
                lines[jk] = {"bar": Barrier(), "near": near, "c": sum(jk) & 1, "used": []}
                owner.setdefault((cta, loc % nw), []).append(jk)
    assert len(lines) == J * K and all(len(w) <= 2 for w in owner.values())

    def order(jk, v):
        if not exact:
            return 2 * v + lines[jk]["c"]
        m = (v >> 1) * K + K - 1 - jk[1]
        return (3 * m + jk[0] + 2 * (v & 1)) * 1024 + m

    def program(eq, w):
        """The visits of warp w in an equation, in its order."""
        v = {jk: 0 for jk in owner[w]}
        while any(q < 4 for q in v.values()):
            jk = min((a for a in owner[w] if v[a] < 4), key=lambda a: (order(a, v[a]), owner[w].index(a)))
            yield jk, v[jk]
            v[jk] += 1

    flying = []  # (target line, equation, its visit, bytes)
    ok = {w: True for w in owner}
    out = gone = 0

    def land(some):
        rng.shuffle(flying)
        for _ in range(min(some, len(flying))):
            jk, eq, v = flying.pop()
            if rule == "wait" and not dies and lines[jk]["bar"].phase != lines[jk]["want"][eq, v]:
                raise Broken("a store landed in another visit's phase")
            lines[jk]["bar"].complete(1)

    for jk, ln in lines.items():  # the phase each visit's stores belong to
        ln["want"], p = {}, 0
        for eq in range(4):
            for v in range(4):
                ln["want"][eq, v] = p
                p += bool(waits(exact, v, ln["c"], ln["near"]))
    for eq in range(4):
        progs = {w: program(eq, w) for w in owner}
        at = {w: next(p, None) for w, p in progs.items()}
        armed = set()
        phase0 = {}
        while any(a is not None for a in at.values()):
            moved = False
            for w in rng.sample(sorted(at), len(at)):
                if at[w] is None or (flying and rng.random() < 0.3):
                    continue
                jk, v = at[w]
                ln = lines[jk]
                need = waits(exact, v, ln["c"], ln["near"])
                if need and (ok[w] or rule == "go on") and w not in armed:
                    phase0[w] = ln["bar"].phase
                    ln["bar"].arrive_expect(len(need))
                    armed.add(w)
                if need and ok[w] and ln["bar"].phase == phase0[w]:
                    if rng.random() < runout:
                        out += 1
                        if rule == "go on":
                            ok[w] = False
                    if rng.random() < dies:
                        ok[w], gone = False, gone + 1
                    if ok[w]:
                        continue
                armed.discard(w)
                if ok[w] or rule == "go on":
                    for d in pushes(exact, v, ln["c"], ln["near"]):
                        to = (jk[0] + DJ[d], jk[1] + DK[d])
                        tv = fed_visit(exact, d, v) if exact else (v if ln["c"] == 0 else v + 1)
                        assert BACK[d] in waits(exact, tv, lines[to]["c"], lines[to]["near"])
                        flying.append((to, eq, tv))
                at[w] = next(progs[w], None)
                moved = True
            before = len(flying)
            land(rng.randint(0, 4) if moved else len(flying))
            if not moved and before == 0:  # nothing on its way: the waits that are left end for good
                for w in at:
                    if at[w] is not None and w in armed and rng.random() < 0.5:
                        if not dies:
                            raise Broken("stuck")
                        ok[w], gone = False, gone + 1
                        armed.discard(w)
                        at[w] = next(progs[w], None)
    if not all(ok.values()) and rule == "wait":
        land(len(flying))  # the wait before the last cluster barrier
    if flying:
        raise Broken("a CTA leaves with stores under way to it")
    return out, gone


SHAPES = [(1, 1, 1, 2), (1, 4, 2, 2), (5, 1, 2, 2), (3, 3, 3, 2), (4, 5, 4, 3), (5, 4, 6, 2), (6, 5, 16, 1), (7, 4, 4, 4)]


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("J,K,nc,nw", SHAPES)
def test_waits_that_run_out_keep_the_phases(J, K, nc, nw, exact):
    rng = random.Random(1)
    total = 0
    for _ in range(12):
        total += replay(J, K, nc, nw, exact, rng, "wait", runout=rng.choice([0.0, 0.1, 1.0]))[0]
    assert total > 0 or J * K == 1


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("J,K,nc,nw", SHAPES)
def test_warps_that_give_up_for_good(J, K, nc, nw, exact):
    rng = random.Random(2)
    total = 0
    for _ in range(12):
        total += replay(J, K, nc, nw, exact, rng, "wait", runout=0.3, dies=0.05)[1]
    assert total > 0 or J * K == 1


@pytest.mark.parametrize("exact", [False, True])
def test_replay_notices_a_phase_armed_twice(exact):
    rng = random.Random(3)
    broken = 0
    for _ in range(20):
        try:
            replay(4, 5, 4, 3, exact, rng, "go on", runout=0.2)
        except Broken:
            broken += 1
    assert broken > 0


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("graphs", [0, 1])
def test_chain_wait_budget_runs_out_with_timeout(prec, graphs, tmp_path):
    """With a launch per pass the energy solve has no waits, and after a step with the beam
    off (no box) every iteration takes the chain: its waits may poll once and run out, and
    the step fails with AMCFD_E_TIMEOUT.  A fresh solver in the same process is as good
    as ever."""
    import amcfd
    import amcfd_decks as D
    dk = D.small("wait", nx=40, ny=22, nz=12, steps=4, power=350.0)
    x, y, ztop = 0.3 * 40 * 30e-6, 0.5 * 22 * 30e-6, 0.3e-3
    dk.single_track = None
    dk.toolpath = [(0.0, x, y, ztop, 0, 1), (2.5 * dk.dt, x, y, ztop, 0, 1), (1e-3, x + 0.3e-3, y, ztop, 1, 1)]
    d = amcfd.Deck(dk.write(str(tmp_path)))
    kw = dict(order=amcfd.ORDER_REDBLACK, precision=prec, use_graphs=graphs, pass_launch=1)
    s = amcfd.Solver(d, wait_polls=1, **kw)
    for _ in range(2):
        assert s.step()["momentum_cells"] == 0
    with pytest.raises(amcfd.AmcfdError) as e:
        for _ in range(4):
            s.step()
    assert e.value.code == -6, str(e.value)
    assert "device wait gave up (code -6, line -6)" in str(e.value)
    with pytest.raises(amcfd.AmcfdError) as e:
        s.step()
    assert e.value.code == -6
    s.close()
    a, b = amcfd.Solver(d, **kw), amcfd.Solver(d, serial_launch=1, small_box=0, **dict(kw, use_graphs=0))
    for _ in range(4):
        ra, rb = a.step(), b.step()
    assert ra["momentum_cells"] == rb["momentum_cells"] > 0
    for f in ("temp", "uvel", "vvel", "wvel", "pressure"):
        assert np.array_equal(a.get(f), b.get(f)), f
    a.close()
    b.close()
