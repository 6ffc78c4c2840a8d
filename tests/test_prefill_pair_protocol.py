"""The barriers of the MLA prompt attention's pair of CTAs (prefill_pair_kernel), as a model on the CPU: the roles of both CTAs as
coroutines in random order, MMAs and copies that complete late, waits that see a barrier's parity only. What one CTA sends to the other
(copies, arrivals of committed MMAs) arrives in any order. Every P and row sum
must be the tile's or item's own when it is read, no buffer may be written while something still reads it, no barrier may complete twice in a
phase's stead, everybody must come to the end, and by then nothing may be on its way to the other CTA, which leaves."""
import os
import random
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cwick_b200", "csrc", "mla_prefill_attn.cu")


class Fault(Exception):
    pass


class Bar:
    """An mbarrier: `count` arrivals and all announced bytes end a phase; a wait knows the parity only."""

    def __init__(self, count):
        self.count, self.pending, self.tx, self.done = count, count, 0, 0

    def arrive(self, tx=0):
        if self.pending == 0:
            raise Fault("an arrival that no phase expects")
        self.pending -= 1
        self.tx += tx
        self.turn()

    def bytes(self, n):
        self.tx -= n
        self.turn()

    def turn(self):
        if self.pending == 0 and self.tx == 0:
            self.done += 1
            self.pending = self.count

    def passes(self, parity):
        return self.done & 1 != parity


class Cta:
    def __init__(self, rank, kst, cst, pbars, arrivals):
        b = Bar
        self.rank = rank
        self.kfull, self.kempty = [b(1) for _ in range(kst)], [b(1) for _ in range(kst)]
        self.cfull, self.cempty = [b(1) for _ in range(cst)], [b(1) for _ in range(cst)]
        self.sfull, self.sempty = [b(1), b(1)], [b(1), b(1)]
        self.pfull, self.pempty = [b(1) for _ in range(4)], [b(arrivals) for _ in range(pbars)]
        self.odone, self.qempty, self.qfull, self.ofree, self.xm, self.xl = b(1), b(1), b(2), b(2), b(2), b(2)
        self.peer = [b(1), b(1)]
        self.k, self.c, self.s, self.p, self.readers = [None] * kst, [None] * cst, [None, None], [None] * 4, [0] * 4
        self.sum, self.item_m, self.q = [None, None], None, None


def model(items, seed, kst, cst, pbars, told, arrivals=2):
    """told(T, rank): the CTAs, as bits, that CTA `rank` tells of the end of its value products with tile T."""
    rnd = random.Random(seed)
    ctas = [Cta(0, kst, cst, pbars, arrivals), Cta(1, kst, cst, pbars, arrivals)]
    late = []                                                # completions under way in a CTA: a list per source, in order within it
    sent = []                                                # under way from one CTA to the other, in no order

    def wait(bar, parity):
        while not bar.passes(parity):
            yield

    def scored(rank, T, tiles):
        return [0] + [d for d in range(1, tiles) if (T + d) & 1 == rank]

    def chain():
        q = []
        late.append(q)
        return q

    def keys(c):
        kc, T = 0, 0
        tma = [chain() for _ in range(kst)]
        for k, tiles in enumerate(items):
            for d in scored(c.rank, T, tiles):
                ks = kc % kst
                yield from wait(c.kempty[ks], (kc // kst & 1) ^ 1)
                c.kfull[ks].arrive(1)

                def land(ks=ks, tag=T + d):
                    c.k[ks] = tag
                    c.kfull[ks].bytes(1)
                tma[ks].append(land)
                kc += 1
            T += tiles

    def latents(c):                                          # announces the peer's P with the tile's latents
        tma = [chain() for _ in range(cst)]
        for T in range(sum(items)):
            cs = T % cst
            yield from wait(c.cempty[cs], (T // cst & 1) ^ 1)
            if T & 1 != c.rank:
                c.pfull[T & 3].arrive(1)
            c.cfull[cs].arrive(1)

            def land(cs=cs, T=T):
                c.c[cs] = T
                c.cfull[cs].bytes(1)
            tma[cs].append(land)
            yield

    def scores(c):
        kc, T, mma = 0, 0, chain()
        for k, tiles in enumerate(items):
            yield from wait(c.qfull, k & 1)
            for d in scored(c.rank, T, tiles):
                ks, sb = kc % kst, kc & 1
                yield from wait(c.kfull[ks], kc // kst & 1)
                yield from wait(c.sempty[sb], (kc >> 1 & 1) ^ 1)
                if c.k[ks] != T + d:
                    raise Fault("scores of tile %d from the keys of %s" % (T + d, c.k[ks]))
                if c.q != k:
                    raise Fault("scores against another item's query")

                def end(ks=ks, sb=sb, tag=T + d):
                    c.kempty[ks].arrive()
                    c.s[sb] = tag
                    c.sfull[sb].arrive()
                mma.append(end)
                kc += 1
            mma.append(c.qempty.arrive)
            T += tiles
            yield

    def values(c):
        T, mma = 0, chain()
        for k, tiles in enumerate(items):
            if k:
                yield from wait(c.ofree, k - 1 & 1)
            for _ in range(tiles):
                pb, cs = T & 3, T % cst
                yield from wait(c.cfull[cs], T // cst & 1)
                yield from wait(c.pfull[pb], T >> 2 & 1)
                if c.p[pb] != T or c.c[cs] != T:
                    raise Fault("values of tile %d with the P of %s and the latents of %s" % (T, c.p[pb], c.c[cs]))
                c.readers[pb] += 1

                def end(pb=pb, cs=cs, T=T):
                    c.readers[pb] -= 1
                    c.cempty[cs].arrive()
                    for x in ctas:
                        if told(T, c.rank) >> x.rank & 1:
                            if x is c:
                                x.pempty[T % pbars].arrive()
                            else:
                                sent.append(x.pempty[T % pbars].arrive)
                mma.append(end)
                T += 1
            mma.append(c.odone.arrive)
            yield

    def sender(c):
        other = ctas[1 - c.rank]
        for T in range(c.rank, sum(items), 2):
            pb = T & 3
            yield from wait(c.pfull[pb], T >> 2 & 1)
            if c.p[pb] != T:
                raise Fault("tile %d sent with the P of %s" % (T, c.p[pb]))
            c.readers[pb] += 1

            def arrive_there(pb=pb, T=T):
                c.readers[pb] -= 1
                if other.readers[pb]:
                    raise Fault("P of tile %d sent into a buffer in use" % T)
                other.p[pb] = T
                other.pfull[pb].bytes(1)
            sent.append(arrive_there)
            yield

    def free(c, T):
        if T >= 4:
            yield from wait(c.pempty[(T - 4) % pbars], (T - 4) // pbars & 1)

    def softmax(c, which):                                   # one of the two sets
        kc, T, other = 0, 0, ctas[1 - c.rank]
        state = c.__dict__.setdefault("soft", {"q": 0})

        def query(k):                                        # both sets copy a part; the tile is whole with the second arrival
            state["q"] += 1
            if state["q"] % 2 == 0:
                c.q = k
            c.qfull.arrive()
        query(0)
        for k, tiles in enumerate(items):
            todo = scored(c.rank, T, tiles)
            if kc & 1 != which:
                c.xm.arrive()
                yield from wait(c.xm, k & 1)
            for e in range((kc ^ which) & 1, len(todo), 2):
                sb, t = kc + e & 1, T + todo[e]
                yield from wait(c.sfull[sb], kc + e >> 1 & 1)
                if c.s[sb] != t:
                    raise Fault("softmax of tile %d from the scores of %s" % (t, c.s[sb]))
                c.sempty[sb].arrive()
                if e == 0:
                    c.xm.arrive()
                    yield from wait(c.xm, k & 1)
                    if T & 1 != c.rank:
                        continue
                yield
                yield from free(c, t)
                if c.readers[t & 3]:
                    raise Fault("P of tile %d written into a buffer in use" % t)
                c.p[t & 3] = t
                c.pfull[t & 3].arrive()
                yield
            kc += len(todo)
            T += tiles
            if k + 1 < len(items):
                yield from wait(c.qempty, k & 1)
                query(k + 1)
            c.xl.arrive()
            yield from wait(c.xl, k & 1)
            if which == 0:
                c.peer[k & 1].arrive(1)

                def arrive_there(k=k):
                    other.sum[k & 1] = k
                    other.peer[k & 1].bytes(1)
                sent.append(arrive_there)
            yield from wait(c.peer[k & 1], k >> 1 & 1)
            yield from wait(c.odone, k & 1)
            own = T if T & 1 == c.rank else T + 1
            yield from free(c, own)
            yield from free(c, own + 2)
            if c.readers[own & 3] or c.readers[own + 2 & 3]:
                raise Fault("staging of item %d in a buffer in use" % k)
            if c.sum[k & 1] != k:
                raise Fault("item %d with the row sums of %s" % (k, c.sum[k & 1]))
            c.ofree.arrive()
            yield

    roles = [r for c in ctas for r in (keys(c), latents(c), scores(c), values(c), sender(c), softmax(c, 0), softmax(c, 1))]
    weight = [rnd.choice((1, 1, 4, 20)) for _ in roles]      # some roles are slow
    slow = rnd.random() < 0.5                                # the way between the CTAs: nothing arrives until all wait for it
    idle = 0
    while roles:
        ready = [q for q in late if q]
        if sent and (idle > 100 if slow else rnd.random() < 0.15):
            sent.pop(rnd.randrange(len(sent)))()
            idle = 0
            continue
        if ready and rnd.random() < 0.3:
            rnd.choice(ready).pop(0)()
            idle = 0
            continue
        i = rnd.choices(range(len(roles)), [1.0 / w for w in weight])[0]
        before = sum(x.done + x.pending for c in ctas for v in c.__dict__.values() for x in (v if isinstance(v, list) else [v]) if isinstance(x, Bar))
        try:
            next(roles[i])
        except StopIteration:
            roles.pop(i)
            weight.pop(i)
            idle = 0
            continue
        after = sum(x.done + x.pending for c in ctas for v in c.__dict__.values() for x in (v if isinstance(v, list) else [v]) if isinstance(x, Bar))
        idle = 0 if after != before or ready else idle + 1
        if idle > 5000:
            raise Fault("stuck")
    if sent:
        raise Fault("%d arrivals at a CTA that has left" % len(sent))


ITEMS = [[1], [2], [3], [1, 1, 1, 1, 1, 1, 1, 1, 1], [2, 1, 2, 1, 3, 1], [5, 4, 3, 2, 1], [7, 1, 6, 2, 9], [12, 11], [1, 8, 1, 1, 8, 3, 3]]


def source():
    """Key and latent slots, barriers of the P buffers and who is told of the end of a tile's value products, as the kernel has them."""
    text = open(SRC).read()
    kst, cst = map(int, re.search(r"struct PrCfg \{\s*static constexpr int KST = (\d+), CST = (\d+)", text).groups())
    pbars = int(re.search(r"PR_ODONE = PR_PEMPTY \+ (\d+)", text)[1])
    told = eval("lambda T, rank: " + re.search(r"umma_commit_to\(bar\(PR_PEMPTY \+ \(T & 7\)\), ([^;]+)\);", text)[1])
    return kst, cst, pbars, told


@pytest.mark.parametrize("items", ITEMS, ids=str)
def test_the_pairs_protocol(items):
    kst, cst, pbars, told = source()
    for seed in range(12):
        model(items, seed, kst, cst, pbars, told)


def test_the_model_finds_buffers_freed_too_early():
    with pytest.raises(Fault):
        for seed in range(100):
            model([7, 1, 6, 2, 9], seed, 2, 3, 8, lambda T, rank: 1 << rank, arrivals=1)


def test_the_model_finds_arrivals_that_nobody_waits_for():
    with pytest.raises(Fault, match="has left"):
        for seed in range(100):
            model([7, 1, 6, 2, 9], seed, 2, 3, 8, lambda T, rank: 3)
