"""The barriers of the GEMM kernels that run on pairs of CTAs (fp8_linear_tc_kernel, kexp_tc_kernel), as a model on the CPU: both CTAs copy
into their rings, the first one's issuer multiplies for both and commits to both, both read the accumulators out. Roles run in random
order, copies and arrivals come late, those at the other CTA in any order. A stage may not be filled while it is read, an accumulator
not be overwritten before both have read it, and nothing may be on its way to a CTA that has left."""
import os
import random
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cwick_b200", "csrc")


class Fault(Exception):
    pass


class Bar:
    def __init__(self, count):
        self.count, self.pending, self.done = count, count, 0

    def arrive(self):
        self.pending -= 1
        if self.pending == 0:
            self.done += 1
            self.pending = self.count

    def passes(self, parity):                                # a wait sees the parity only
        return self.done & 1 != parity


def model(steps, seed, stages, per_tile, tail):
    """per_tile: steps that one accumulator takes. tail: the producers wait for the last uses of their stages before they end."""
    rnd = random.Random(seed)
    empty = [[Bar(1) for _ in range(stages)] for _ in range(2)]                     # [cta][stage]
    full = [Bar(2) for _ in range(stages)]                                          # in the first CTA: both CTAs' copies
    ready, read = [[Bar(1), Bar(1)] for _ in range(2)], [Bar(2), Bar(2)]            # [cta][accumulator]; in the first CTA
    stage, acc = [[None] * stages for _ in range(2)], [[None, None] for _ in range(2)]
    left = [False, False]
    local, sent = [], []                                     # under way: (in order) in the first CTA, (in none) between the two
    tiles = steps // per_tile

    def wait(bar, parity):
        while not bar.passes(parity):
            yield

    def deliver(cta, f):
        def g():
            if left[cta]:
                raise Fault("an arrival at a CTA that has left")
            f()
        return g

    def producer(cta):
        for c in range(steps):
            s = c % stages
            yield from wait(empty[cta][s], (c // stages & 1) ^ 1)
            if stage[cta][s] is not None:
                raise Fault("a stage filled before it was read")

            def land(s=s, c=c):
                stage[cta][s] = c
                full[s].arrive()
            sent.append(deliver(0, land))
            yield
        if tail:
            for c in range(max(0, steps - stages), steps):
                yield from wait(empty[cta][c % stages], c // stages & 1)

    def issuer():
        for c in range(steps):
            s, t, d = c % stages, c // per_tile, c // per_tile & 1
            if c % per_tile == 0:
                yield from wait(read[d], (t >> 1 & 1) ^ 1)
                if acc[0][d] is not None or acc[1][d] is not None:
                    raise Fault("an accumulator overwritten before it was read")
            yield from wait(full[s], c // stages & 1)

            def end(s=s, c=c, t=t, d=d):
                if stage[0][s] != c or stage[1][s] != c:
                    raise Fault("step %d with the stages of %s" % (c, (stage[0][s], stage[1][s])))
                stage[0][s] = stage[1][s] = None
                if c % per_tile == per_tile - 1:
                    acc[0][d] = acc[1][d] = t
                for cta in range(2):
                    some = [empty[cta][s].arrive] + ([ready[cta][d].arrive] if c % per_tile == per_tile - 1 else [])
                    for f in some:
                        sent.append(deliver(cta, f)) if cta else f()
            local.append(end)
            yield

    def epilogue(cta):
        for t in range(tiles):
            d = t & 1
            yield from wait(ready[cta][d], t >> 1 & 1)
            if acc[cta][d] != t:
                raise Fault("the accumulator of tile %s for tile %d" % (acc[cta][d], t))
            acc[cta][d] = None
            sent.append(read[d].arrive) if cta else read[d].arrive()      # (a thread's arrival: before the cluster's closing barrier)
            yield

    roles = [(0, producer(0)), (1, producer(1)), (0, issuer()), (0, epilogue(0)), (1, epilogue(1))]
    slow = rnd.random() < 0.5
    idle = 0
    while roles:
        if sent and (idle > 60 if slow else rnd.random() < 0.2):
            sent.pop(rnd.randrange(len(sent)))()
            idle = 0
            continue
        if local and rnd.random() < 0.3:
            local.pop(0)()
            idle = 0
            continue
        i = rnd.randrange(len(roles))
        idle += 1
        try:
            next(roles[i][1])
        except StopIteration:
            roles.pop(i)
        if idle > 3000:
            raise Fault("stuck")
    # the closing barrier of the cluster: what the threads did is ordered before it (their arrivals), committed MMAs' arrivals are not
    left[:] = [True, True]
    for f in sent:
        f()


def kernel(name):
    """Stages, steps per accumulator and whether the producers wait for the last uses of their stages, as the kernel has them."""
    if name == "fp8_linear_tc_kernel":
        text = open(os.path.join(CSRC, "fp8_linear_tc.cu")).read()
        stages, per_tile, empty = re.search(r"\bSTAGES = (\d+)", text)[1], 1, r"GB_EMPTY \+ s % STAGES"
    else:
        text = open(os.path.join(CSRC, "mla_prefill_attn.cu")).read()
        stages, per_tile, empty = re.search(r"\bKX_ST = (\d+)", text)[1], 4, r"KB_AEMPTY \+ c % KX_ST"
    body = text[text.index(name + "("):]
    body = body[:body.index("\n}\n")]
    tail = re.search(r"for \(int (\w) = max\(0, \w+ - (?:STAGES|KX_ST)\); [^\n]*\n?\s*ok = mbar_wait\(bar\(%s\), \(uint32_t\)\(\(\1 / \w+\) & 1\)" % empty, body)
    return int(stages), per_tile, tail is not None


@pytest.mark.parametrize("name", ["fp8_linear_tc_kernel", "kexp_tc_kernel"])
def test_the_pairs_ring(name):
    stages, per_tile, tail = kernel(name)
    for steps in (per_tile, 2 * per_tile, 12, 40):
        for seed in range(20):
            model(steps, seed, stages, per_tile, tail)


def test_the_model_finds_arrivals_at_a_cta_that_has_left():
    with pytest.raises(Fault, match="has left"):
        for seed in range(20):
            model(40, seed, 4, 1, False)
