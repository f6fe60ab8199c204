"""The barrier rings of conv_stem_kernel, on a model of its warps: a wait by parity is only sound while the barrier cannot have gone
a phase further, and a packed row may only be overwritten once no tile reads it.  One warp is stopped ahead of each of its waits in turn,
the others run as far as they get."""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "armnn_b200", "csrc", "conv_tc.cu")
K = {name: int(value) for name, value in re.findall(r"^constexpr int (ST_\w+) = (\d+);", open(SOURCE).read(), re.M)}


class Rings:
    """The waits and signals of a CTA that walks `tiles` output rows from the `first` on.  Barriers are counters of completed phases."""

    def __init__(self, kh, stride, oh, first, tiles, accumulators):
        self.count, self.mma, self.written, self.fault = {}, [False] * tiles, {}, None
        step = min(kh, stride)                                      # (packed rows are the rows that some tile reads)
        hp = (oh - 1) * step + kh
        rows = [t // oh * hp + t % oh * step for t in range(first, first + tiles)]
        self.lo, self.kh = [r - rows[0] for r in rows], kh
        self.new, top = [], 0                                       # the packed rows that each tile is the first to need
        for lo in self.lo:
            self.new.append(list(range(max(lo, top), lo + kh)))
            top = max(top, lo + kh)
        self.tiles, self.acc = tiles, accumulators
        self.lookahead = 2 if kh > 8 and oh < 3 else K["ST_LOOKAHEAD"]
        warps = [self.issuer(i) for i in range(K["ST_ISSUERS"])] + [self.loader(), self.epilogue()]
        self.warps = warps + [self.expander(e) for e in range(K["ST_EXPANDERS"])]
        self.waiting = [next(w, None) for w in self.warps]          # (barrier, phase) that has to be complete

    def signal(self, barrier):
        self.count[barrier] = self.count.get(barrier, 0) + 1

    def issuer(self, me):
        waited = 0
        for i in range(me, self.tiles, K["ST_ISSUERS"]):
            for rv in range(max(self.lo[i], waited), self.lo[i] + self.kh):
                yield ("row", rv % K["ST_SLOTS"]), rv // K["ST_SLOTS"]
            waited = self.lo[i] + self.kh
            yield ("acc_empty", i % self.acc), i // self.acc - 1
            self.mma[i] = True
            self.signal(("acc_full", i % self.acc))
            self.signal(("done", i % K["ST_DONE"]))

    def loader(self):
        for n in range(sum(map(len, self.new))):                    # (no padding rows: more rows on their way than with them)
            yield ("raw_empty", n % K["ST_RAW"]), n // K["ST_RAW"] - 1
            self.signal(("raw", n % K["ST_RAW"]))

    def expander(self, me):
        n = 0
        for i in range(self.tiles):
            if i >= self.lookahead:
                j = i - self.lookahead
                yield ("done", j % K["ST_DONE"]), j // K["ST_DONE"]
            for rv in self.new[i]:
                if rv % K["ST_EXPANDERS"] == me:
                    yield ("raw", n % K["ST_RAW"]), n // K["ST_RAW"]
                    old = self.written.get(rv % K["ST_SLOTS"])
                    if old is not None and any(not self.mma[t] and self.lo[t] <= old < self.lo[t] + self.kh for t in range(self.tiles)):
                        self.fault = "row %d written over row %d, which a tile still needs" % (rv, old)
                    self.written[rv % K["ST_SLOTS"]] = rv
                    self.signal(("raw_empty", n % K["ST_RAW"]))
                    self.signal(("row", rv % K["ST_SLOTS"]))
                n += 1

    def epilogue(self):
        for i in range(self.tiles):
            yield ("acc_full", i % self.acc), i // self.acc
            self.signal(("acc_empty", i % self.acc))

    def ready(self, w):
        barrier, phase = self.waiting[w]
        return self.count.get(barrier, 0) > phase

    def run(self, stopped=None, waits=None):
        """Until nothing moves, warp `stopped` for that many waits only.  Whether it has a wait left."""
        moved = True
        while moved:
            moved = False
            for w in range(len(self.warps)):
                while self.waiting[w] is not None and self.ready(w) and not (w == stopped and waits == 0):
                    if w == stopped:
                        waits -= 1
                    self.waiting[w] = next(self.warps[w], None)
                    moved = True
        return stopped is None or self.waiting[stopped] is not None


def check(kh, stride, oh, first, tiles=44, accumulators=4):
    """None, or what goes wrong."""
    free = Rings(kh, stride, oh, first, tiles, accumulators)
    free.run()
    if any(w is not None for w in free.waiting):
        return "no end: %s" % free.waiting
    for w in range(len(free.warps)):
        for n in range(10 ** 6):
            r = Rings(kh, stride, oh, first, tiles, accumulators)
            if not r.run(w, n):
                break
            barrier, phase = r.waiting[w]
            if r.count.get(barrier, 0) > phase + 1:
                return "warp %d ahead of %s: phase %d, the barrier is %d phases on" % (w, barrier, phase, r.count[barrier])
            if r.fault:
                return r.fault
    return None


# filter rows, stride, output rows per image, first output row
@pytest.mark.parametrize("kh,stride,oh,first", [(1, 1, 50, 0), (2, 1, 7, 3), (3, 1, 50, 0), (3, 1, 5, 2), (5, 1, 50, 0), (7, 1, 9, 8), (3, 2, 50, 0), (7, 2, 50, 0),
                                                (7, 2, 3, 1), (11, 4, 50, 0), (11, 4, 3, 2), (11, 1, 4, 0), (4, 4, 6, 0), (3, 3, 50, 0), (1, 2, 8, 0), (1, 4, 5, 3), (2, 3, 8, 1), (3, 4, 7, 0),
                                                (8, 1, 1, 0), (9, 1, 1, 0), (11, 4, 1, 0), (8, 4, 2, 1), (9, 4, 2, 0), (10, 2, 2, 1), (11, 1, 2, 1), (11, 4, 2, 0)])
@pytest.mark.parametrize("accumulators", [2, 4])
def test_no_wait_is_overtaken(kh, stride, oh, first, accumulators):
    assert check(kh, stride, oh, first, accumulators=accumulators) is None
