"""CPU: barrier model (tests/barrier_model.py) of the decode kernel, dadgpt_b200/csrc/decode.cu, with persistent
CTAs: the producer with its ring of row tiles and of items, two of the consumer warps."""
import random

import pytest

from tests.barrier_model import Aborted, Model, survives

WARPS = (0, 1)


class Decode(Model):
    """Items are numbers of row tiles; an item may have none (its only row comes with the token)."""
    STAGES, RING = 3, 2
    need = {"empty": 2, "item_free": 2}

    def __init__(self, items, rng, agreed=True, abort=False):
        super().__init__(rng, abort)
        self.items, self.agreed = items, agreed

    def producer(self):
        g = 0
        for n, tiles in enumerate(self.items):
            for _ in range(tiles):
                s, lap = g % self.STAGES, g // self.STAGES
                if lap > 0:
                    yield ("wait", f"empty[{s}]", lap - 1)
                yield ("tma", f"full[{s}]", [(("rows", s), g)])
                g += 1
            if n >= self.RING:
                yield ("wait", f"item_free[{n % self.RING}]", n // self.RING - 1)
            yield ("write", ("item", n % self.RING), n + 1)
            yield ("arrive", f"item_ready[{n % self.RING}]")

    def consumer(self, w):
        ok, g, n, have = True, 0, 0, True
        while have:
            for _ in range(self.items[n]):
                if ok:
                    try:
                        yield ("wait", f"full[{g % self.STAGES}]", g // self.STAGES)
                        yield ("read", ("rows", g % self.STAGES), g)
                        yield ("arrive", f"empty[{g % self.STAGES}]")
                    except Aborted:
                        ok = False
                g += 1
            have = False
            if ok:
                try:
                    yield ("wait", f"item_ready[{n % self.RING}]", n // self.RING)
                    yield ("read", ("item", n % self.RING), n + 1)
                    yield ("arrive", f"item_free[{n % self.RING}]")
                    have = n + 1 < len(self.items)
                except Aborted:
                    ok = False
            yield ("write", ("acc", w), n)
            yield ("sync", "merge", 2)
            for v in WARPS:
                yield ("read", ("acc", v), n)
            if self.agreed:
                if (yield ("any", "merged", 2, not ok)):
                    have = False
            else:
                yield ("sync", "merged", 2)
            n += 1

    def agents(self):
        return {"producer": self.producing(self.producer()), **{f"consumer{w}": self.consumer(w) for w in WARPS}}


ITEMS = [[9, 3, 0, 1], [0, 0, 0, 0], [1, 1, 1, 1, 1], [5], [2, 7, 2]]


@pytest.mark.parametrize("abort", [False, True], ids=["runs", "gives_up"])
def test_every_schedule_ends(abort):
    for items in ITEMS:
        assert survives(lambda s: Decode(items, random.Random(s), abort=abort), range(150)) is None, items


def test_consumers_have_to_agree_on_whether_they_go_on():
    found = survives(lambda s: Decode([2, 2, 2, 2], random.Random(s), agreed=False, abort=True), range(500))
    assert found is not None and "stuck" in found[1]


def test_the_model_catches_rows_on_their_way_when_the_block_retires():
    class Leaves(Decode):
        def producing(self, body):
            return body

    found = survives(lambda s: Leaves([4, 4, 4], random.Random(s), abort=True), range(500))
    assert found is not None and "at work" in found[1]
