"""A CPU model of the pipeline of the tensor-core kNN filter (k_knn_tc in
gpu-sg-sne_b200/csrc/sgt_knn.cu) with the places of sgt_knn_rules.h compiled
from that file, under random delays.

One thread issues the copies of a block's query image and of the candidate
stages, one the MMAs, and the scanning warps empty the two accumulators; the
places run on over query blocks, which end in a block barrier.  Checked:

- an MMA reads the stage and the image that its step means, after their copies;
- a copy goes to a stage whose MMAs are complete, an image likewise;
- an MMA goes to an accumulator that has been scanned, a scan reads its tile;
- nobody waits for good;
- a block that gives up ends with no copy and no MMA in flight.

The model starts at any number of steps, as after hours of a search.  The same
model with places taken from 32-bit counts fails where they wrap.
"""
import ctypes
import os
import random
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "gpu-sg-sne_b200", "csrc")


class CRing(ctypes.Structure):
    _fields_ = [("at", ctypes.c_int), ("flying", ctypes.c_int), ("phase", ctypes.c_uint)]


@pytest.fixture(scope="module")
def ring(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring")
    src = d / "r.cpp"
    src.write_text('#include "sgt_knn_rules.h"\n'
                   'extern "C" void next(SgtRing *r, int n) { r->next(n); }\n'
                   'extern "C" int back(SgtRing *r, int n) { return r->back(n); }\n')
    so = d / "r.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(src), "-o",
                    str(so)], check=True)
    lib = ctypes.CDLL(str(so))

    class Ring:
        def __init__(self, n, count):
            self.n, self.r = n, CRing(count % n, 0, (count // n) & 1)

        at = property(lambda self: self.r.at)
        phase = property(lambda self: self.r.phase)
        before = property(lambda self: self.r.phase ^ 1)

        def next(self):
            lib.next(ctypes.byref(self.r), self.n)

        def back(self):
            return bool(lib.back(ctypes.byref(self.r), self.n))

    return Ring


class Counted:
    """Places by a 32-bit count of all uses; `before` is None in the first round."""

    def __init__(self, n, count):
        self.n, self.c = n, count

    at = property(lambda self: (self.c & 0xFFFFFFFF) % self.n)
    phase = property(lambda self: ((self.c & 0xFFFFFFFF) // self.n) & 1)

    @property
    def before(self):
        turn = (self.c & 0xFFFFFFFF) // self.n
        return None if turn == 0 else (turn - 1) & 1

    def next(self):
        self.c += 1


class Barrier:
    def __init__(self, done):
        self.done = done  # phases completed

    def passes(self, parity):
        return parity is None or (self.done & 1) != parity


def run(Ring, nst, nch, ntile, nblk, resident, rng, steps0=0, tiles0=0, give_up=None,
        wait_image=True):
    """Runs the model; raises AssertionError where it goes wrong.  give_up: the
    number of events after which the block gives up."""
    used = lambda count, n, k: (count + n - 1 - k) // n  # uses of buffer k before `count`
    full = [Barrier(used(steps0, nst, k)) for k in range(nst)]
    free = [Barrier(used(steps0, nst, k)) for k in range(nst)]
    accb = [Barrier(used(tiles0, 2, k)) for k in range(2)]
    scan = [Barrier(used(tiles0, 2, k)) for k in range(2)]
    image = Barrier(0)
    s = dict(stage={}, reading={}, acc={}, image=None)
    rings = {}
    late, mmas = [], []  # copies in flight; MMAs and commits, in order

    def copier():
        load, step = Ring(nst, steps0), steps0
        rings["load"] = load
        for blk in range(nblk):
            if resident:
                assert not mmas, "the image is read"
                s["image"] = None
                rings["block"] = blk
                late.append(("image", blk))
            for g in range(ntile * nch):
                yield free[load.at], load.before
                k = load.at
                assert s["reading"].get(k) is None, "copy into a stage that is read"
                s["stage"][k], s["reading"][k] = None, step
                late.append(("stage", k, step))
                step += 1
                load.next()
            yield "block"

    def issuer():
        at, acc, step, tile = Ring(nst, steps0), Ring(2, tiles0), steps0, tiles0
        rings["step"], rings["acc"] = at, acc
        for blk in range(nblk):
            if resident:
                yield image, blk & 1
            for g in range(ntile * nch):
                if g % nch == 0:
                    yield scan[acc.at], acc.before
                    assert s["acc"].get(acc.at) is None, "MMA into an accumulator not scanned"
                yield full[at.at], at.phase
                assert s["stage"].get(at.at) == step, "MMA of a stage not filled"
                assert not resident or s["image"] == blk
                mmas.append(("free", at.at, step))
                if g % nch == nch - 1:
                    s["acc"][acc.at] = ("busy", tile)
                    mmas.append(("acc", acc.at, tile))
                    tile += 1
                    acc.next()
                step += 1
                at.next()
            yield "block"

    def scanner():
        acc, tile = Ring(2, tiles0), tiles0
        for blk in range(nblk):
            for _ in range(ntile):
                yield accb[acc.at], acc.phase
                assert s["acc"].get(acc.at) == ("full", tile), "scan of another tile"
                yield None
                s["acc"][acc.at] = None
                scan[acc.at].done += 1
                tile += 1
                acc.next()
            yield "block"

    def complete(what, i):
        if what == "copy":
            c = late.pop(i)
            if c[0] == "image":
                s["image"] = c[1]
                image.done += 1
            else:
                s["stage"][c[1]] = c[2]
                full[c[1]].done += 1
        else:
            kind, k, num = mmas.pop(0)
            if kind == "free":
                assert s["reading"][k] == num
                s["reading"][k] = None
                free[k].done += 1
            else:
                s["acc"][k] = ("full", num)
                accb[k].done += 1

    def flights():
        return [("copy", i) for i in range(len(late))] + [("mma", 0)] * bool(mmas)

    agents = [copier(), issuer(), scanner()]
    want = [next(a) for a in agents]
    events = 0
    while any(a is not None for a in agents):
        if events == give_up:
            waits = [(image, rings["block"] & 1)] if resident and wait_image else []
            while rings["load"].back():
                waits.append((full[rings["load"].at], rings["load"].phase))
            if rings["step"].back():
                waits.append((free[rings["step"].at], rings["step"].phase))
            if rings["acc"].back():
                waits.append((accb[rings["acc"].at], rings["acc"].phase))
            while not all(bar.passes(parity) for bar, parity in waits):
                assert flights(), "the end waits for good"
                complete(*rng.choice(flights()))
            assert not late, "a copy in flight at the end"
            assert not mmas, "an MMA in flight at the end"
            return
        events += 1
        can = [("agent", i) for i, w in enumerate(want) if agents[i] is not None and w != "block" and
               (w is None or w[0].passes(w[1]))] + flights()
        if all(agents[i] is None or want[i] == "block" for i in range(3)) and not mmas:
            can = [("agent", i) for i in range(3) if agents[i] is not None]
            for _, i in can:
                want[i] = next(agents[i], "end")
                if want[i] == "end":
                    agents[i] = None
            continue
        assert can, "everyone waits"
        what, i = rng.choice(can)
        if what == "agent":
            want[i] = next(agents[i], "end")
            if want[i] == "end":
                agents[i] = None
        else:
            complete(what, i)


@pytest.mark.parametrize("nst,nch,resident", [(5, 1, True), (5, 2, True), (3, 3, False),
                                              (8, 1, True), (2, 13, False)])
@pytest.mark.parametrize("steps0,tiles0", [(0, 0), (7, 3), (2 ** 32 - 6, 2 ** 32 - 3),
                                           (2 ** 33 + 1, 2 ** 32)])
def test_places(ring, nst, nch, resident, steps0, tiles0):
    rng = random.Random(nst * 100 + nch)
    for _ in range(8):
        run(ring, nst, nch, rng.choice([1, 2, 7]), 3, resident, rng, steps0, tiles0)


def test_counts_of_32_bits_go_wrong_where_they_wrap(ring):
    rng = random.Random(1)
    run(Counted, 5, 1, 7, 3, True, rng)
    with pytest.raises(AssertionError):
        for _ in range(20):
            run(Counted, 5, 1, 7, 3, True, rng, 2 ** 32 - 6, 2 ** 32 - 3)


def test_back_goes_over_the_uses_in_flight(ring):
    for n in (1, 2, 5):
        for uses in range(2 * n + 2):
            r, places = ring(n, 0), []
            for _ in range(uses):
                places.append((r.at, r.phase))
                r.next()
            got = []
            while r.back():
                got.append((r.at, r.phase))
            assert got == places[::-1][:n]


@pytest.mark.parametrize("nst,nch,resident", [(5, 1, True), (5, 2, True), (3, 3, False)])
def test_nothing_is_in_flight_after_giving_up(ring, nst, nch, resident):
    rng = random.Random(nst)
    for events in range(120):
        run(ring, nst, nch, 7, 3, resident, rng, give_up=events)


def test_the_query_image_is_one_of_the_copies_to_wait_for(ring):
    rng = random.Random(2)
    with pytest.raises(AssertionError, match="a copy in flight"):
        for events in range(40):
            run(ring, 5, 1, 7, 3, True, rng, give_up=events, wait_image=False)
