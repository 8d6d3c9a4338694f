"""CPU: barrier model (tests/barrier_model.py) of the head-size-128 forward with two query tiles per CTA,
dadgpt_b200/csrc/flash_fwd128_sm100.cu. An item is (key tiles of group A, of group B, ring tile of B's first); a
softmax group is two agents, each with its rows. The request for another block is a load whose answer names the item."""
import random

import pytest

from tests.barrier_model import Aborted, Model, survives

PARTS = (0, 1)


class Forward(Model):
    SLOTS, RING = 5, 4
    need = {"slot_empty": 2, "item_free": 7, "p_full0": 2, "p_full1": 2, "q_empty": 2}

    def __init__(self, items, rng, abort=False):
        super().__init__(rng, abort)
        self.items = [*items, (0, 0, 0)]

    def tiles(self, i):   # through the ring
        a, b, first_b = self.items[i]
        return max(a, b + first_b)

    def fetch(self, i):
        yield ("wait", f"item_ready[{i % self.RING}]", i // self.RING)
        yield ("read", ("item", i % self.RING), i)
        yield ("arrive", f"item_free[{i % self.RING}]")

    def scheduler(self):
        def publish(i):
            if i >= self.RING:
                yield ("wait", f"item_free[{i % self.RING}]", i // self.RING - 1)
            yield ("write", ("item", i % self.RING), i)
            yield ("arrive", f"item_ready[{i % self.RING}]")

        yield from publish(0)
        at = 0
        for i in range(len(self.items) - 1):
            yield ("tma", "stolen", [("answer", i + 1)])
            for _ in range(2 * self.tiles(i)):
                s, use = at % self.SLOTS, at // self.SLOTS
                if use > 0:
                    yield ("wait", f"slot_empty[{s}]", use - 1)
                yield ("tma", f"slot_full[{s}]", [(("kv", s), at)])
                at += 1
            yield ("wait", "stolen", i)
            yield ("read", "answer", i + 1)
            yield from publish(i + 1)

    def q_producer(self):
        n = [0, 0]
        for i, item in enumerate(self.items):
            yield from self.fetch(i)
            for x in PARTS:
                if item[x]:
                    if n[x] > 0:
                        yield ("wait", f"q_empty[{x}]", n[x] - 1)
                    yield ("tma", f"q_full[{x}]", [(("q", x, a), ("Q", i)) for a in PARTS])
                    n[x] += 1

    def issuer(self, x):
        at = g = u = 0

        def full():
            return ("wait", f"slot_full[{at % self.SLOTS}]", at // self.SLOTS)

        for i, item in enumerate(self.items):
            yield from self.fetch(i)
            n, before = item[x], item[2] if x and item[x] else 0
            if not n:
                before = self.tiles(i)
            for _ in range(2 * before):
                yield full()
                yield ("arrive", f"slot_empty[{at % self.SLOTS}]")
                at += 1
            if not n:
                continue
            yield ("wait", f"q_full[{x}]", u)
            for j in range(n + 1):
                if j > 0:
                    yield full()
                    for c in PARTS:
                        yield ("wait", f"p_full{c}[{x}]", g)
                        so_far = [(("o", x), (i, j - 2 + c / 2))] if j > 1 or c else []
                        yield ("mma", [(("s", c, x, a), ("p", i, j - 1)) for a in PARTS] + [(("kv", at % self.SLOTS), at)] + so_far,
                               [(("o", x), (i, j - 1.5 + c / 2))])
                    yield ("commit", f"slot_empty[{at % self.SLOTS}]")
                    at += 1
                    g += 1
                if j < n:
                    yield full()
                    yield ("mma", [(("q", x, a), ("Q", i)) for a in PARTS] + [(("kv", at % self.SLOTS), at)],
                           [(("s", c, x, a), ("s", i, j)) for c in PARTS for a in PARTS])
                    yield ("commit", f"slot_empty[{at % self.SLOTS}]")
                    yield ("commit", f"s_full[{x}]")
                    at += 1
            yield ("commit", f"o_done[{x}]")
            u += 1
            for _ in range(2 * (self.tiles(i) - before - n)):
                yield full()
                yield ("arrive", f"slot_empty[{at % self.SLOTS}]")
                at += 1

    def softmax(self, x, a):
        g = u = 0
        for i, item in enumerate(self.items):
            yield from self.fetch(i)
            if not item[x]:
                continue
            for j in range(item[x]):
                yield ("wait", f"s_full[{x}]", g)
                for c in PARTS:
                    yield ("read", ("s", c, x, a), ("s", i, j))
                if j > 0 and self.rng.random() < 0.3:   # the rescale
                    yield ("read", ("o", x), (i, j - 1))
                for c in PARTS:   # the keys' halves
                    yield ("write", ("s", c, x, a), ("p", i, j))
                    yield ("arrive", f"p_full{c}[{x}]")
                g += 1
            yield ("wait", f"o_done[{x}]", u)
            yield ("read", ("o", x), (i, item[x] - 1))
            yield ("write", ("q", x, a), ("out", i))   # (its store has read them when it goes on)
            yield ("read", ("q", x, a), ("out", i))
            yield ("arrive", f"q_empty[{x}]")
            u += 1

    def loading(self, body, mine):
        """As Model.producing, with the loads of one of the two producers."""
        try:
            yield from body
        except Aborted:
            pass
        for bar, n in sorted(self.loads.items()):
            if bar.split("[")[0] in mine:
                yield ("settle", bar, n - 1)

    def agents(self):
        return {"scheduler": self.loading(self.scheduler(), ("slot_full", "stolen")),
                "q producer": self.loading(self.q_producer(), ("q_full",)),
                **{f"issuer{x}": self.issuing(self.issuer(x), f"settled[{x}]") for x in PARTS},
                **{f"softmax{x}{a}": self.softmax(x, a) for x in PARTS for a in PARTS}}


# long and short items, an odd number of tiles (nothing for B), one-tile sequences of two units and of one
WORK = ([(1, 2, 0)], [(5, 6, 0), (3, 4, 0), (1, 2, 0)], [(3, 0, 0), (1, 2, 0), (3, 0, 0), (1, 2, 0)],
        [(1, 1, 1)] * 6 + [(1, 0, 0)], [(7, 0, 0)], [(1, 2, 0)] * 7, [(3, 0, 0)] * 5, [(1, 0, 0)] * 20)


@pytest.mark.parametrize("abort", [False, True], ids=["runs", "gives_up"])
@pytest.mark.parametrize("items", WORK)
def test_every_schedule(items, abort):
    assert survives(lambda s: Forward(items, random.Random(s), abort), range(80)) is None


@pytest.mark.parametrize("role,gone", [("scheduler", "slot_empty"), ("q_producer", "q_empty"),
                                       ("issuer", "q_full"), ("issuer", "p_full0"), ("issuer", "p_full1"),
                                       ("softmax", "s_full"), ("softmax", "o_done"), ("scheduler", "stolen")])
def test_the_model_misses_no_wait_that_is_left_out(role, gone):
    class Faulty(Forward):
        pass

    def faulty(self, *args):
        for op in getattr(Forward, role)(self, *args):
            if not (op[0] == "wait" and op[1].split("[")[0] == gone):
                yield op
    setattr(Faulty, role, faulty)
    assert any(survives(lambda s: Faulty(items, random.Random(s)), range(200)) for items in WORK)
