"""The hand-off protocol of the tensor-core sweep, simulated: producers, the ring of slabs, MMAs that
finish when they like, TMEM slots and the ring of row exponents, with roles of any relative speed."""
import os
import random
import re

import pytest

SRC = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                        'boast-lig_gb300', 'csrc', 'tc_kernel.cuh')).read()


def constant(name):
    return int(re.search(r'constexpr \w+ (?:\w+ = \w+, )*' + name + r' = (\d+)', SRC).group(1))


SLOTS, TSLOTS, EXP_RING = constant('kSlots'), constant('kTmemSlots'), constant('kExpRing')


class Overwritten(AssertionError):
    pass


class Barrier:
    """mbarrier: `done` phases are complete; a wait names a phase by its parity only."""

    def __init__(self, count):
        self.count, self.pending, self.done = count, count, 0

    def arrive(self, n=1):
        self.pending -= n
        assert self.pending >= 0
        if self.pending == 0:
            self.pending, self.done = self.count, self.done + 1

    def passes(self, phase):
        """Whether a wait for `phase` returns; the phase must not be two ahead of the waiter."""
        assert self.done <= phase + 2, 'a phase ran two ahead of its waiter'
        assert self.done != phase + 2, 'a waiter would sleep through its phase'
        return (self.done - 1) % 2 == phase % 2


def simulate(strips, W, rng, speed, ring=EXP_RING, nprod=2):
    """Runs a CTA over `strips` (blocks of each); speed(role) weighs the scheduler's choice."""
    full, empty = [Barrier(nprod) for _ in range(SLOTS)], [Barrier(W) for _ in range(SLOTS)]
    tfull, drained = [Barrier(2) for _ in range(TSLOTS)], [Barrier(4) for _ in range(TSLOTS)]
    slab = [[None] * SLOTS for _ in range(nprod)]        # what each producer warp's rows hold
    tmem, exps = [None] * TSLOTS, [[None] * ring for _ in range(nprod)]
    queues, drains = {}, []

    def producer(w):
        n = 0
        for si, nb in enumerate(strips):
            exps[w][si % ring] = si
            for k in range(nb + W - 1):
                while not empty[n % SLOTS].passes(n // SLOTS - 1):
                    yield
                slab[w][n % SLOTS] = (si, k)
                yield
                full[n % SLOTS].arrive()
                n += 1
                yield

    class Issue:                                         # the warp's view of the next block to issue
        def __init__(self):
            self.strip, self.j, self.blk, self.slab = 0, 0, 0, 0

        def step(self):
            self.blk += 1
            self.slab += 1
            self.j += 1
            if self.j == strips[self.strip]:
                self.slab += W - 1
                self.j = 0
                self.strip += 1

        def left(self):
            return self.strip < len(strips)

    def issue_next(name, lq, I):
        if not I.left():
            return
        if lq == (I.blk >> 1) & 3:
            ts, last = I.blk % TSLOTS, I.slab + W - 1
            if I.blk >= TSLOTS:
                while not drained[ts].passes(I.blk // TSLOTS - 1):
                    yield
            while not full[last % SLOTS].passes(last // SLOTS):
                yield
            arrivals = []
            for w in range(W):
                k = I.j + w
                first = max(0, k - W + 1)
                readers = min(k, strips[I.strip] - 1) - first + 1
                s = (I.slab + w) % SLOTS
                arrivals.append(s)
                if first == I.j and readers < W:
                    empty[s].arrive(W - readers)
            queues[name].append((I.strip, I.j, I.blk, I.slab, arrivals))
            tfull[ts].arrive()
            yield
        I.step()
        if I.left():
            I.step()

    def epilogue(name, hf, lq):
        I = Issue()
        if hf and I.left():
            I.step()
        yield from issue_next(name, lq, I)
        blk0 = 0
        for si, nb in enumerate(strips):
            for j in range((blk0 ^ hf) & 1, nb, 2):
                blk = blk0 + j
                while not tfull[blk % TSLOTS].passes(blk // TSLOTS):
                    yield
                yield
                if j < 2 and any(e[si % ring] != si for e in exps):      # read once, at the first block
                    raise Overwritten((si, [e[si % ring] for e in exps]))
                yield from issue_next(name, lq, I)
                yield
                assert tmem[blk % TSLOTS] == (si, j)
                drains.append((blk, name))
                drained[blk % TSLOTS].arrive()
                yield
            blk0 += nb

    def tensor(name):                                    # the MMAs one warp issued, in its order
        q = queues[name]
        while len(drains) < 4 * sum(strips):
            if q:
                si, j, blk, n, arrivals = q[0]
                for w in range(W):                       # operands are read until the end
                    assert all(s[(n + w) % SLOTS] == (si, j + w) for s in slab)
                yield
                assert all(s[(n + w) % SLOTS] == (si, j + w) for s in slab for w in range(W))
                tmem[blk % TSLOTS] = (si, j)
                q.pop(0)
                tfull[blk % TSLOTS].arrive()
                for s in arrivals:
                    empty[s].arrive()
            yield

    roles = {('prod', w): producer(w) for w in range(nprod)}
    for hf in range(2):
        for lq in range(4):
            queues[hf, lq] = []
            roles['epi', hf, lq] = epilogue((hf, lq), hf, lq)
            roles['mma', hf, lq] = tensor((hf, lq))
    names = list(roles)
    weights = [speed(n) for n in names]
    for _ in range(3000000):
        if not names:
            break
        i = rng.choices(range(len(names)), weights)[0]
        try:
            next(roles[names[i]])
        except StopIteration:
            del names[i], weights[i]
    assert not names, 'deadlock'
    assert sorted(drains) == sorted((b, (h, q)) for b in range(sum(strips)) for h in [b & 1] for q in range(4))


def speeds(kind, rng):
    slow = ('epi', rng.randrange(2), rng.randrange(4))
    return {'even': lambda n: 1.0,
            'slow epilogue warp': lambda n: 0.03 if n == slow else 1.0,
            'slow producers': lambda n: 0.05 if n[0] == 'prod' else 1.0,
            'slow tensor core': lambda n: 0.05 if n[0] == 'mma' else 1.0,
            'one slow producer': lambda n: 0.05 if n == ('prod', 0) else 1.0}[kind]


KINDS = ['even', 'slow epilogue warp', 'slow producers', 'slow tensor core', 'one slow producer']


@pytest.mark.parametrize('kind', KINDS)
@pytest.mark.parametrize('W', [2, 3])
@pytest.mark.parametrize('most', [1, 2, 7])
def test_protocol(W, most, kind):
    """Every operand is intact while its MMAs run, every block is drained by its group, exponents are
    those of the strip, no phase runs two ahead: strips of one block, of one or two, and longer."""
    for seed in range(3):
        rng = random.Random(1000 * seed + 10 * most + W)
        simulate([rng.randint(1, most) for _ in range(14)], W, rng, speeds(kind, rng))


def test_exponent_ring_is_as_long_as_it_must_be():
    """One entry less than the kernel's bound (kSlots, W = 2, TMEM slots) is overwritten in use when
    an epilogue warp is slow: the simulation sees what the bound excludes."""
    need = (SLOTS + 2) // 2 + TSLOTS
    assert EXP_RING >= need
    lost = 0
    for seed in range(20):
        rng = random.Random(seed)
        try:
            simulate([1] * 30, 2, rng, speeds('slow epilogue warp', rng), ring=need - 1)
        except Overwritten:
            lost += 1
    assert lost
