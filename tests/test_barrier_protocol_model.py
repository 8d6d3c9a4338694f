"""CPU: barrier model (tests/barrier_model.py) of the head-size-64 forward, dadgpt_b200/csrc/flash_fwd64_sm100.cu:
TMA producer, one product issuer per softmax group, each group as two agents (the halves of a row, which never
synchronise inside an item). Every K/V tile is two sub-steps with two score buffers per group."""
import random

import pytest

from tests.barrier_model import Model, survives

KV_STAGES = 4
HALVES = (0, 1)


class FwdSim(Model):
    """Work items are (tiles of group A, tiles of group B): B has one tile more than A, or none when the pair's
    second tile lies beyond the sequence. `one`: sequences of one tile, whose items are two units of one tile
    each, (1, 1), or a last one alone, (1, 0): ring tile 0 is group A's, ring tile 1 group B's."""
    need = {"kv_empty": 2, "q_empty": 2, "p_full": 2, "o_free": 2, "stat_full": 2}
    stat_buffers = 2   # of the (max, sum) pairs that the halves exchange

    def __init__(self, items, rng, one=False, abort=False, rescale_prob=0.3):
        super().__init__(rng, abort)
        self.items, self.one, self.rescale_prob = items, one, rescale_prob

    def n_kv(self, item):
        return item[0] + item[1] if self.one else item[1] or item[0]

    def span(self, item, X):
        """The group takes part in the item's ring tiles begin .. end - 1."""
        if self.one and X and item[1]:
            return item[0], item[0] + item[1]
        return 0, item[X]

    def producer(self):
        g = 0
        for k, item in enumerate(self.items):
            qb = k & 1
            if k >= 2:
                yield ("wait", f"q_empty[{qb}]", (k >> 1) - 1)
            yield ("tma", f"q_full[{qb}]", [(("q", qb), k)])
            for _ in range(self.n_kv(item)):
                s, use = g % KV_STAGES, g // KV_STAGES
                if use > 0:
                    yield ("wait", f"kv_empty[{s}]", use - 1)
                yield ("tma", f"k_full[{s}]", [(("k", s), g)])
                yield ("tma", f"v_full[{s}]", [(("v", s), g)])
                g += 1

    def issuer_x(self, X):
        items = self.items
        n_s = 0   # sub-steps of this group whose scores have been issued

        def scores(k, g, c):
            nonlocal n_s
            t = n_s
            n_s += 1
            yield ("mma", [(("q", k & 1), k), (("k", g % KV_STAGES), g)], [(("scores", X, c, h), ("s", t)) for h in HALVES])
            yield ("commit", f"s_full[{X}][{c}]")

        yield ("wait", "q_full[0]", 0)
        yield ("wait", "k_full[0]", 0)
        begin, end = self.span(items[0], X)
        if end > 0 and begin == 0:
            yield from scores(0, 0, 0)
            yield from scores(0, 0, 1)
            if end == 1:
                yield ("commit", "q_empty[0]")
        if end == 0:
            yield ("arrive", "q_empty[0]")
        g = n_pv = n_done = 0
        for k, item in enumerate(items):
            qb, n_kv = k & 1, self.n_kv(item)
            j0, j1 = self.span(item, X)
            for j in range(n_kv):
                s, last = g % KV_STAGES, j + 1 == n_kv
                have_next = not last or k + 1 < len(items)
                ni = items[k + 1] if last and have_next else item
                nj, nqb = (0, qb ^ 1) if last else (j + 1, qb)
                b, e = self.span(ni, X)
                yield ("wait", f"v_full[{s}]", g // KV_STAGES)
                s_next = have_next and e > 0 and b <= nj < e
                issued = next_ready = False
                for c in (0, 1):
                    if j0 <= j < j1:
                        first = j == j0 and c == 0
                        if first and n_done > 0:
                            yield ("wait", f"o_free[{X}]", n_done - 1)
                        yield ("wait", f"p_full[{X}][{c}]", n_pv >> 1)
                        for h in HALVES:
                            yield ("mma", [(("scores", X, c, h), ("p", n_pv)), (("v", s), g)] + ([] if first else [(("out", X, h), n_pv - 1)]),
                                   [(("out", X, h), n_pv)])
                        yield ("commit", f"o_done[{X}][{n_pv & 1}]")
                        n_pv += 1
                        issued = True
                    if s_next:
                        if not next_ready:
                            if nj == b:
                                yield ("wait", f"q_full[{nqb}]", (k + 1 if last else k) >> 1)
                            yield ("wait", f"k_full[{(g + 1) % KV_STAGES}]", (g + 1) // KV_STAGES)
                            next_ready = True
                        yield from scores(k + 1 if last else k, g + 1, c)
                        issued = True
                        if c == 1 and nj + 1 == e:
                            yield ("commit", f"q_empty[{nqb}]")
                if have_next and e == 0 and nj == 0:
                    if last:
                        yield ("wait", f"q_full[{nqb}]", (k + 1) >> 1)
                    yield ("arrive", f"q_empty[{nqb}]")
                yield ("commit", f"kv_empty[{s}]") if issued else ("arrive", f"kv_empty[{s}]")
                g += 1
            if j1 > j0:
                n_done += 1

    def softmax(self, X, h):
        t = n_item = 0
        for item in self.items:
            if item[X] == 0:
                continue
            for v in range(2 * item[X]):
                c = v & 1
                yield ("wait", f"s_full[{X}][{c}]", t >> 1)
                yield ("read", ("scores", X, c, h), ("s", t))
                if v > 0 and self.rng.random() < self.rescale_prob:   # the lazy rescale looks at O
                    yield ("wait", f"o_done[{X}][{(t - 1) & 1}]", (t - 1) >> 1)
                    yield ("read", ("out", X, h), t - 1)
                    yield ("write", ("out", X, h), t - 1)
                yield ("write", ("scores", X, c, h), ("p", t))
                yield ("arrive", f"p_full[{X}][{c}]")
                t += 1
            at = n_item % self.stat_buffers
            yield ("write", ("stat", X, at, h), n_item)
            yield ("arrive", f"stat_full[{X}]")
            yield ("wait", f"stat_full[{X}]", n_item)
            yield ("wait", f"o_done[{X}][{(t - 1) & 1}]", (t - 1) >> 1)
            for other in HALVES:
                yield ("read", ("stat", X, at, other), n_item)
                yield ("read", ("out", X, other), t - 1)
            yield ("arrive", f"o_free[{X}]")
            n_item += 1

    def agents(self):
        return {"producer": self.producing(self.producer()),
                **{f"issuer {'AB'[X]}": self.issuing(self.issuer_x(X), f"settled[{X}]") for X in (0, 1)},
                **{f"softmax {'AB'[X]}{h}": self.softmax(X, h) for X in (0, 1) for h in HALVES}}


FWD_ITEM_LISTS = [
    [(7, 8), (5, 6), (3, 4), (1, 2)],             # the GPT-2 shape's pairs, heaviest first
    [(1, 2)] * 7,
    [(1, 0)] * 9,                                 # lone tiles: group B and its issuer idle throughout
    [(9, 0), (7, 8), (1, 0), (3, 4)],             # odd tile count: a lone last tile longer than the ring
    [(5, 0), (1, 2), (5, 0)],
    [(1, 2), (1, 0), (1, 2), (1, 0), (3, 4)],
]


@pytest.mark.parametrize("abort", [False, True], ids=["runs", "gives_up"])
def test_forward_protocol_survives_every_schedule(abort):
    for items in FWD_ITEM_LISTS:
        assert survives(lambda s: FwdSim(items, random.Random(s), abort=abort), range(60)) is None, items


def test_forward_model_catches_an_ungated_idle_issuer():
    """The rule the idle issuer follows (wait for the stage's data before releasing it) is what
    keeps it from arriving twice within one phase of kv_empty; a model without that wait must
    trip the audit, or the model is not looking."""
    class Ungated(FwdSim):
        def issuer_x(self, X):
            for op in super().issuer_x(X):
                if X == 1 and op[0] == "wait" and op[1].startswith("v_full"):
                    continue
                yield op

    assert survives(lambda s: Ungated([(9, 0), (9, 0), (9, 0)], random.Random(s)), range(200)) is not None


@pytest.mark.parametrize("role,gone", [("issuer_x", "p_full"), ("issuer_x", "q_full"), ("softmax", "o_done"), ("softmax", "stat_full"),
                                       ("producer", "kv_empty")])
def test_forward_model_misses_no_wait_that_is_left_out(role, gone):
    """(o_free is not among them: the probabilities that a product of the next item needs come after the epilogue.)"""
    class Faulty(FwdSim):
        pass

    def faulty(self, *args):
        for op in getattr(FwdSim, role)(self, *args):
            if not (op[0] == "wait" and op[1].split("[")[0] == gone):
                yield op
    setattr(Faulty, role, faulty)
    assert survives(lambda s: Faulty([(3, 4), (1, 2), (1, 2)], random.Random(s)), range(300)) is not None


@pytest.mark.parametrize("items,one", [([(3, 4), (1, 2), (1, 2), (1, 2)], False), ([(1, 1)] * 6, True)])
def test_the_statistics_need_two_buffers(items, one):
    """The scores of an item of one tile are formed without waiting for the epilogue of the item before: a half can be
    at its next statistics while the other has not read the last ones."""
    class Single(FwdSim):
        stat_buffers = 1

    found = survives(lambda s: Single(items, random.Random(s), one), range(200))
    assert found is not None and "stat" in found[1]
    assert survives(lambda s: FwdSim(items, random.Random(s), one), range(200)) is None
