"""The barriers between the final stage's warps (csrc/final_tc.cu, split float16), modelled on the host: two loaders that
alternate, twelve producer warps that share a subaperture's items in turn, two issuers and the epilogue, each with random
durations and now and then a long delay. An mbarrier's wait names a phase by its parity only, so a wait is sound only where
its barrier cannot be two phases away."""
import heapq
import random

import pytest

NPW, LS, NLD = 12, 8, 2


class Barrier:
    def __init__(self, count):
        self.count = self.left = count
        self.phase = 0
        self.waiting = []

    def passed(self, parity):                     # the phase of this parity has completed, as far as one bit tells
        return (self.phase & 1) != parity


class Violation(Exception):
    pass


def simulate(nwi, Pf, units, S, seg, every, seed):
    """One run of a block; every: all producers wait and arrive in every subaperture (else only with an item)."""
    rng = random.Random(seed)
    nis = 2 if Pf >= 2 else 1
    rs, ntot, nsg = S // nis, units * Pf, -(-Pf // seg)
    count = NPW if every else nwi
    full, empty = [Barrier(count) for _ in range(S)], [Barrier(1) for _ in range(S)]
    lfull, lempty = [Barrier(1) for _ in range(LS)], [Barrier(count) for _ in range(LS)]
    accf, acce = [Barrier(nis) for _ in range(2)], [Barrier(1) for _ in range(2)]
    slot, stage, built = [None] * LS, [None] * S, [0] * S     # subaperture held, being built or read, items built
    queue, now, tick = [], [0.0], [0]
    slow = rng.choice([0.0, 0.01, 0.05])

    def at(dt, fn):
        tick[0] += 1
        heapq.heappush(queue, (now[0] + dt, tick[0], fn))

    def arrive(b):
        b.left -= 1
        if b.left < 0:
            raise Violation('an arrival too many')
        if b.left == 0:
            b.phase, b.left = b.phase + 1, b.count
            for wake in b.waiting:
                at(rng.uniform(0.01, 0.1), wake)
            b.waiting = []

    def work(t):                                  # a duration, rarely a long delay
        return t * rng.uniform(0.7, 1.3) + (rng.uniform(2, 8) if rng.random() < slow else 0.0)

    alive = [0]

    def start(gen):
        alive[0] += 1

        def step():
            try:
                kind, arg = next(gen)
            except StopIteration:
                alive[0] -= 1
                return
            if kind == 'work':
                at(work(arg), step)
            else:
                poll(*arg)

        def poll(b, parity):
            if b.passed(parity):
                at(0.01, step)
            else:
                b.waiting.append(lambda: poll(b, parity))
        at(0.0, step)

    def loader(k):
        landed = [0.0]
        for it in range(k, ntot, NLD):
            ls = it % LS
            if it >= LS:
                yield 'wait', (lempty[ls], (it // LS - 1) & 1)
            slot[ls] = None
            yield 'work', 0.5

            def land(ls=ls, it=it):
                slot[ls] = it
                arrive(lfull[ls])
            landed[0] = max(landed[0], now[0] + work(1.0))
            at(landed[0] - now[0], land)

    def producer(pw):
        ps, pp, p, first, turn = [0, 0], [0, 0], 0, pw, (nwi + 1) % NPW
        for it in range(ntot):
            ls, kq = it % LS, p & 1 if nis == 2 else 0
            stg = kq + nis * ps[kq]
            mine = range(first, nwi, NPW)
            if every or mine:
                yield 'wait', (lfull[ls], (it // LS) & 1)
                yield 'wait', (empty[stg], pp[kq] ^ 1)
            for _ in mine:
                if stage[stg] not in (None, it):
                    raise Violation(f'stage {stg} still holds {stage[stg]}, built for {it}')
                stage[stg] = it
                for _half in range(2):
                    if slot[ls] != it:
                        raise Violation(f'slot {ls} holds {slot[ls]}, read for {it}')
                    yield 'work', 0.4
                built[stg] += 1
                if not every:
                    arrive(full[stg])
                    arrive(lempty[ls])
            if every:
                arrive(full[stg])
                arrive(lempty[ls])
            first = (first - turn) % NPW
            ps[kq] += 1
            if ps[kq] == rs:
                ps[kq], pp[kq] = 0, pp[kq] ^ 1
            p = (p + 1) % Pf

    def issuer(k):
        slotn, par, done, sg = 0, 0, [0.0], 0
        for j in range(units * nsg):
            yield 'wait', (acce[j & 1], ((j >> 1) & 1) ^ 1)
            for p in range(sg * seg + k, min(Pf, (sg + 1) * seg), nis):
                stg, it = k + nis * slotn, j // nsg * Pf + p
                yield 'wait', (full[stg], par)
                if stage[stg] != it or built[stg] != nwi:
                    raise Violation(f'stage {stg} holds {stage[stg]} ({built[stg]} of {nwi} items), multiplied for {it}')

                def consumed(stg=stg):
                    stage[stg], built[stg] = None, 0
                    arrive(empty[stg])
                done[0] = max(done[0], now[0]) + work(0.2)
                at(done[0] - now[0], consumed)
                slotn += 1
                if slotn == rs:
                    slotn, par = 0, par ^ 1
            done[0] = max(done[0], now[0]) + 0.01
            at(done[0] - now[0], lambda ab=j & 1: arrive(accf[ab]))
            sg = (sg + 1) % nsg

    def epilogue():
        for j in range(units * nsg):
            yield 'wait', (accf[j & 1], (j >> 1) & 1)
            yield 'work', 2.0
            arrive(acce[j & 1])

    for k in range(NLD):
        start(loader(k))
    for pw in range(NPW):
        start(producer(pw))
    for k in range(nis):
        start(issuer(k))
    start(epilogue())
    while queue:
        now[0], _, fn = heapq.heappop(queue)
        fn()
    if alive[0]:
        raise Violation('warps that wait for ever')


def _runs(every):
    for nwi in (2, 4, 6, 8, 10, 12, 14, 24):                 # even counts: an A and a B item per group of samples
        for Pf, S, seg in ((1, 6, 1), (3, 6, 2), (9, 6, 48), (10, 6, 48), (33, 6, 24), (40, 4, 16)):
            for seed in range(3):
                yield nwi, Pf, S, seg, seed


def test_every_warp_waits_and_arrives():
    """The kernel's protocol: no slot read before its load, no stage overwritten or multiplied early, an end to each run."""
    for nwi, Pf, S, seg, seed in _runs(True):
        simulate(nwi, Pf, max(2, 150 // Pf), S, seg, True, seed)


@pytest.mark.parametrize('nwi', [2, 4, 6])
def test_model_finds_skipped_waits(nwi):
    """The model sees the fault it is made for: producers that wait only where they have an item read slots too early,
    overwrite stages or end in waits that nothing completes."""
    found = 0
    for n, Pf, S, seg, seed in _runs(False):
        if n == nwi:
            try:
                simulate(nwi, Pf, max(2, 150 // Pf), S, seg, False, seed)
            except Violation:
                found += 1
    assert found > 0
