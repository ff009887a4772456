"""A model of the stage hand-over of the integer tensor-core products (csrc/rsvd_tc.cu), run
under random schedules: two groups of 8 unpack warps arrive on a stage's named barrier, the
MMA warp joins it, and a barrier completes on any 9 arrivals. The waits that may run out
(for loads; for the MMAs of a stage's previous fill) do so at random. With the guard on
`joined` every run ends with every generation made of its own 9 warps; without it
some runs hang, which is why the kernel has it."""
import random

GROUPS, WARPS, KSTEPS = 2, 8, 4


class Named:
    def __init__(self):
        self.generation, self.here = 0, []

    def arrive(self, who):
        self.here.append(who)
        if len(self.here) == WARPS + 1:
            self.generation, self.here = self.generation + 1, []


def run(seed, blocks, nstage, p_out, guard):
    """True when every warp came to its end; AssertionError for a mixed generation."""
    rnd = random.Random(seed)
    bar, done = [Named() for _ in range(nstage)], [0] * nstage
    state = {"abort": False, "joined": 0, "loaded": 0}
    mmas = []   # issued, not finished

    def wait(ready):   # the bounded wait
        while not ready():
            if state["abort"]:
                return False
            if rnd.random() < p_out:
                state["abort"] = True
                return False
            yield
        return True

    def mma():
        for n in range(blocks * KSTEPS):
            if n % KSTEPS == 0:
                yield from wait(lambda: state["loaded"] > n // KSTEPS)
            s = n % nstage
            mine = bar[s].generation
            bar[s].arrive("mma")
            while bar[s].generation == mine:
                yield True   # blocked: nothing but an arrival helps
            mmas.append(s)
            state["joined"] = n + 1

    def unpack(group, warp):
        for n in range(blocks * KSTEPS):
            if n % KSTEPS == 0:
                yield from wait(lambda: state["loaded"] > n // KSTEPS)
            if n % GROUPS != group:
                continue
            s, fill = n % nstage, n // nstage
            if fill:
                ok = yield from wait(lambda: done[s] >= fill)
                while guard and not ok and state["joined"] < n - nstage + 1:
                    yield True
            if guard:
                assert (group, warp) not in bar[s].here and bar[s].generation == fill
            yield
            bar[s].arrive((group, warp))

    live = [mma()] + [unpack(g, w) for g in range(GROUPS) for w in range(WARPS)]
    idle = 0
    while live and idle < 4000:   # idle: steps in which every warp met was blocked
        idle += 1
        if rnd.random() < 0.05 and state["loaded"] < blocks:
            state["loaded"] += 1
        if mmas and rnd.random() < 0.2:
            done[mmas.pop(0)] += 1
        w = rnd.choice(live)
        try:
            if next(w) is None:
                idle = 0
        except StopIteration:
            live.remove(w)
            idle = 0
    return not live


def test_every_run_ends_with_the_guard():
    assert all(run(s, 1 + s % 7, 2 + s % 3, 0.0, True) for s in range(40))
    assert all(run(s, 1 + s % 7, 2 + s % 3, 10.0 ** -(1 + s % 4), True) for s in range(400))
    assert all(run(s, 1 + s % 7, 2 + s % 3, 1.0, True) for s in range(40))


def test_without_the_guard_some_runs_hang():
    assert not all(run(s, 3, 3, 10.0 ** -(1 + s % 4), False) for s in range(100))
