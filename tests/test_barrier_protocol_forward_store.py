"""CPU: the head-size-64 forward's results leave through the item's Q buffer (dadgpt_b200/csrc/flash_fwd64_sm100.cu):
each half stages its part over the group's Q tile and gives the buffer back once the store has read it, one sub-step
into the next item; a group without work gives its share back once the buffer is loaded. The rest of the protocol is
test_barrier_protocol_model's."""
import random

import pytest

from tests.barrier_model import survives
from tests.test_barrier_protocol_model import FWD_ITEM_LISTS, HALVES, FwdSim


class StoreSim(FwdSim):
    need = {**FwdSim.need, "q_empty": 4}   # every half of both groups

    def __init__(self, *args, **kw):
        super().__init__(*args, **kw)
        self.mine = {}   # an agent's last store

    def issue(self, who, op):
        if op[0] == "bulk":
            self.mine[who] = len(self.bulk)
        if op[0] == "bulk_wait":   # of its own stores only
            return ("bulk_wait", self.mine.get(who))
        return super().issue(who, op)

    def ready(self, op):
        if op[0] == "bulk_wait":
            return op[1] is None or self.bulk[op[1]] is None
        return super().ready(op)

    def producer(self):
        for op in super().producer():
            if op[0] == "tma" and op[1].startswith("q_full"):
                (cell, k), = op[2]
                op = (op[0], op[1], [((*cell, X, h), k) for X in (0, 1) for h in HALVES])
            yield op

    def issuer_x(self, X):
        # (without its releases of the Q buffers, and the wait ahead of the one where the group has no work)
        for op in super().issuer_x(X):
            if op[1] == "q_empty[0]" or op[1] == "q_empty[1]":
                continue
            if op[0] == "mma" and op[1][0][0][0] == "q":
                (cell, k), *rest = op[1]
                op = (op[0], [((*cell, X, h), k) for h in HALVES] + rest, op[2])
            yield op

    def softmax(self, X, h):
        t = n_item = 0
        owed = None
        for k, item in enumerate(self.items):
            if item[X] == 0:
                if owed is not None:
                    yield ("bulk_wait", 0)
                    yield ("arrive", f"q_empty[{owed}]")
                    owed = None
                yield ("wait", f"q_full[{k & 1}]", k >> 1)
                yield ("arrive", f"q_empty[{k & 1}]")
                continue
            for v in range(2 * item[X]):
                c = v & 1
                if v == 1 and owed is not None:
                    yield ("bulk_wait", 0)
                    yield ("arrive", f"q_empty[{owed}]")
                    owed = None
                yield ("wait", f"s_full[{X}][{c}]", t >> 1)
                yield ("read", ("scores", X, c, h), ("s", t))
                if v > 0 and self.rng.random() < self.rescale_prob:
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
            yield ("write", ("q", k & 1, X, h), ("staged", k))
            yield ("bulk", [(("q", k & 1, X, h), ("staged", k))])
            owed = k & 1
            n_item += 1
        yield ("bulk_wait", 0)


CASES = [(items, False) for items in FWD_ITEM_LISTS] + [([(1, 1)] * 5 + [(1, 0)], True)]


@pytest.mark.parametrize("abort", [False, True], ids=["runs", "gives_up"])
def test_results_leave_through_the_q_buffers(abort):
    for items, one in CASES:
        assert survives(lambda s: StoreSim(items, random.Random(s), one, abort=abort), range(60)) is None, items


@pytest.mark.parametrize("role,gone", [("softmax", "bulk_wait"), ("softmax", "q_full"), ("producer", "q_empty")])
def test_no_wait_of_it_can_be_left_out(role, gone):
    class Faulty(StoreSim):
        pass

    def faulty(self, *args):
        for op in getattr(StoreSim, role)(self, *args):
            if not (op[0] == gone or op[0] == "wait" and op[1].split("[")[0] == gone):
                yield op
    setattr(Faulty, role, faulty)
    assert survives(lambda s: Faulty([(3, 4), (1, 0), (1, 0), (1, 0), (1, 2), (1, 0), (1, 2)], random.Random(s)), range(300)) is not None
