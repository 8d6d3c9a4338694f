"""CPU: barrier models (tests/barrier_model.py) of the exact fp32 kernels on the tensor cores,
dadgpt_b200/csrc/flash_f32_tc_fwd_sm100.cu and flash_f32_tc_bwd_sm100.cu: loaders and compute warps as two agents
each, one issuer. `many`: persistent CTAs with several items, else one item whose results leave through the rings."""
import random

import pytest

from tests.barrier_model import Aborted, Model, Violation, survives

PARTS = (0, 1)   # the two agents of the loaders, and of the compute warps


class Forward(Model):
    """Items are numbers of 64-key steps."""
    STAGES = 3
    need = {"q_full": 2, "p_full": 2, "k_full": 2, "v_full": 2}

    def __init__(self, items, rng, many=True, joins=True, abort=False):
        super().__init__(rng, abort)
        self.items, self.many, self.joins = items, many, joins

    def loader(self, t):
        g = 0
        for n_it in self.items:
            for _ in range(n_it):
                s, lap = g % self.STAGES, g // self.STAGES
                for m in "kv":
                    if lap > 0:
                        yield ("wait", f"{m}_empty[{s}]", lap - 1)
                    yield ("write", (m, s, t), g)
                    yield ("arrive", f"{m}_full[{s}]")
                g += 1

    def issuer(self):
        def x(g, n):
            s = g % self.STAGES
            yield ("wait", f"k_full[{s}]", g // self.STAGES)
            yield ("mma", [(("k", s, t), g) for t in PARTS] + [(("q", a), n) for a in PARTS],
                   [(("scores", g & 1, a), ("s", g)) for a in PARTS])
            yield ("commit", f"x_full[{g & 1}]")
            yield ("commit", f"k_empty[{s}]")

        g = 0
        for n, n_it in enumerate(self.items):
            yield ("wait", "q_full", n)
            yield from x(g, n)
            if n_it >= 2:
                yield from x(g + 1, n)
            for i in range(n_it):
                s = (g + i) % self.STAGES
                yield ("wait", f"v_full[{s}]", (g + i) // self.STAGES)
                yield ("wait", "p_full", g + i)
                yield ("mma", [(("v", s, t), g + i) for t in PARTS] + [(("scores", (g + i) & 1, a), ("p", g + i)) for a in PARTS]
                       + [(("third", a), g + i) for a in PARTS], [("sum", g + i)])
                yield ("commit", f"v_empty[{s}]")
                yield ("commit", "acc_done")
                if i + 2 < n_it:
                    yield from x(g + i + 2, n)
            g += n_it

    def compute(self, a):
        turn = 0      # barriers of the row's warps joined so far
        staged = False
        try:
            step = 0
            for n in range(len(self.items) + 1):
                if n < len(self.items):
                    yield ("write", ("q", a), n)
                    yield ("arrive", "q_full")
                if n > 0:
                    yield ("wait", "acc_done", step - 1)
                    yield ("read", "sum", step - 1)
                    yield ("write", ("part", turn & 1, a), turn)
                    yield ("sync", "rows", 2)
                    turn += 1
                    for b in PARTS:
                        yield ("read", ("part", (turn - 1) & 1, b), turn - 1)
                    if not self.many:
                        yield ("write", ("k", 0, a), "results")
                        yield ("sync", "compute", 2)
                        staged = True
                        for b in PARTS:
                            yield ("read", ("k", 0, b), "results")
                if n == len(self.items):
                    return
                for i in range(self.items[n]):
                    yield ("wait", f"x_full[{step & 1}]", step >> 1)
                    yield ("read", ("scores", step & 1, a), ("s", step))
                    yield ("write", ("part", turn & 1, a), turn)
                    yield ("sync", "rows", 2)
                    turn += 1
                    for b in PARTS:
                        yield ("read", ("part", (turn - 1) & 1, b), turn - 1)
                    if i > 0:
                        yield ("wait", "acc_done", step - 1)
                        yield ("read", "sum", step - 1)
                    yield ("write", ("scores", step & 1, a), ("p", step))
                    yield ("write", ("third", a), step)
                    yield ("arrive", "p_full")
                    step += 1
        except Aborted:
            if not self.joins:
                raise
            while turn < sum(self.items) + len(self.items):
                yield ("sync", "rows", 2)
                turn += 1
            if not self.many and not staged:
                yield ("sync", "compute", 2)

    def agents(self):
        return {"issuer": self.issuing(self.issuer()), **{f"loader{t}": self.loader(t) for t in PARTS},
                **{f"compute{a}": self.compute(a) for a in PARTS}}


class Backward(Model):
    """Items are (is_q, number of 64-row steps); is_q: queries resident, dQ."""
    need = {"a_full": 2, "p_full": 2, "b1_full": 2, "b2_full": 2}

    def __init__(self, items, rng, many=True, delta_given=False, joins=True, abort=False):
        super().__init__(rng, abort)
        self.items, self.many, self.delta_given, self.joins = items, many, delta_given, joins

    def loader(self, t):
        g = 0
        for _, n_it in self.items:
            for _ in range(n_it):
                if g >= 3:
                    yield ("wait", f"b2_empty[{g % 3}]", g // 3 - 1)
                yield ("write", ("b2", g % 3, t), g)
                yield ("write", ("vec", g % 3, t), g)
                yield ("arrive", f"b2_full[{g % 3}]")
                if g >= 2:
                    yield ("wait", f"b1_empty[{g & 1}]", (g >> 1) - 1)
                yield ("write", ("b1", g & 1, t), g)
                yield ("arrive", f"b1_full[{g & 1}]")
                g += 1

    def issuer(self):
        def x(g, n):
            for m, s, use in (("2", g % 3, g // 3), ("1", g & 1, g >> 1)):
                yield ("wait", f"b{m}_full[{s}]", use)
                yield ("mma", [(("b" + m, s, t), g) for t in PARTS] + [(("a" + m, a), n) for a in PARTS],
                       [(("x" + m, g & 1, a), ("s", g)) for a in PARTS])
            yield ("commit", f"x_full[{g & 1}]")

        g = 0
        for n, (is_q, n_it) in enumerate(self.items):
            yield ("wait", "a_full", n)
            yield from x(g, n)
            if n_it >= 2:
                yield from x(g + 1, n)
            for i in range(n_it):
                h = g + i
                yield ("wait", "p_full", h)
                if not is_q:
                    yield ("mma", [(("b2", h % 3, t), h) for t in PARTS] + [((x_, h & 1, a), ("p", h)) for x_ in ("x1", "x2") for a in PARTS],
                           [("sum1", h)])
                yield ("commit", f"b2_empty[{h % 3}]")
                yield ("mma", [(("b1", h & 1, t), h) for t in PARTS] + [(("x2", h & 1, a), ("p", h)) for a in PARTS]
                       + [(("extra", a), h) for a in PARTS], [("sum2", h)])
                yield ("commit", f"b1_empty[{h & 1}]")
                yield ("commit", "acc_done")
                if i + 2 < n_it:
                    yield from x(h + 2, n)
            g += n_it

    def barriers(self, first=0):
        """Barriers of all compute warps from item `first` on."""
        return sum(is_q and not self.delta_given for is_q, _ in self.items[first:]) + (not self.many)

    def compute(self, a):
        turn = 0   # barriers joined so far
        try:
            step = 0
            for n in range(len(self.items) + 1):
                if n < len(self.items):
                    yield ("write", ("a1", a), n)
                    yield ("write", ("a2", a), n)
                    if self.items[n][0] and not self.delta_given:
                        yield ("write", ("own", n & 1, a), n)
                    yield ("arrive", "a_full")
                if n > 0:
                    yield ("wait", "acc_done", step - 1)
                    if not self.items[n - 1][0]:
                        yield ("read", "sum1", step - 1)
                    yield ("read", "sum2", step - 1)
                    if not self.many:
                        yield ("write", ("b1", 0, a), "results")
                        yield ("sync", "compute", 2)
                        turn += 1
                        for b in PARTS:
                            yield ("read", ("b1", 0, b), "results")
                if n == len(self.items):
                    return
                is_q, n_it = self.items[n]
                if is_q and not self.delta_given:
                    yield ("sync", "compute", 2)
                    turn += 1
                    for b in PARTS:
                        yield ("read", ("own", n & 1, b), n)
                for i in range(n_it):
                    yield ("wait", f"x_full[{step & 1}]", step >> 1)
                    if not is_q:
                        yield ("wait", f"b2_full[{step % 3}]", step // 3)
                    for x in ("x1", "x2"):
                        yield ("read", (x, step & 1, a), ("s", step))
                    if not is_q:
                        for t in PARTS:
                            yield ("read", ("vec", step % 3, t), step)
                    if i > 0:
                        yield ("wait", "acc_done", step - 1)
                        if not is_q:
                            yield ("read", "sum1", step - 1)
                        yield ("read", "sum2", step - 1)
                    for x in ("x1", "x2") if not is_q else ("x2",):
                        yield ("write", (x, step & 1, a), ("p", step))
                    yield ("write", ("extra", a), step)
                    yield ("arrive", "p_full")
                    step += 1
        except Aborted:
            if not self.joins:
                raise
            while turn < self.barriers():
                yield ("sync", "compute", 2)
                turn += 1

    def agents(self):
        return {"issuer": self.issuing(self.issuer()), **{f"loader{t}": self.loader(t) for t in PARTS},
                **{f"compute{a}": self.compute(a) for a in PARTS}}


FORWARD_ITEMS = [[16, 14, 1, 1], [1, 1, 1, 1, 1], [2, 1, 2, 3], [5, 4], [1, 7, 1]]
BACKWARD_ITEMS = [[(False, 8), (True, 8), (True, 1), (False, 1)], [(True, 1)] * 5, [(False, 1), (True, 2), (False, 3), (True, 4)],
                  [(False, 1)] * 4, [(True, 5), (False, 2), (False, 1), (True, 1)]]


@pytest.mark.parametrize("abort", [False, True], ids=["runs", "gives_up"])
def test_forward(abort):
    for items in FORWARD_ITEMS:
        assert survives(lambda s: Forward(items, random.Random(s), abort=abort), range(100)) is None, items
    for n_it in (1, 2, 3, 9):
        assert survives(lambda s: Forward([n_it], random.Random(s), many=False, abort=abort), range(100)) is None, n_it


@pytest.mark.parametrize("delta_given", [False, True])
@pytest.mark.parametrize("abort", [False, True], ids=["runs", "gives_up"])
def test_backward(abort, delta_given):
    for items in BACKWARD_ITEMS:
        assert survives(lambda s: Backward(items, random.Random(s), True, delta_given, abort=abort), range(100)) is None, items
    for item in ((True, 1), (True, 4), (False, 1), (False, 3)):
        assert survives(lambda s: Backward([item], random.Random(s), False, delta_given, abort=abort), range(100)) is None, item


@pytest.mark.parametrize("make", [lambda s: Forward([5, 3, 2], random.Random(s), joins=False, abort=True),
                                  lambda s: Forward([2], random.Random(s), many=False, joins=False, abort=True),
                                  lambda s: Backward([(True, 2), (True, 2), (True, 1)], random.Random(s), joins=False, abort=True),
                                  lambda s: Backward([(False, 2)], random.Random(s), many=False, joins=False, abort=True)])
def test_warps_that_give_up_have_to_join_the_barriers_that_are_left(make):
    found = survives(make, range(500))
    assert found is not None and "stuck" in found[1]


def test_the_model_catches_planes_stored_ahead_of_the_last_sums():
    class Early(Forward):
        def compute(self, a):
            for op in super().compute(a):
                if op[:2] != ("wait", "acc_done"):
                    yield op

    assert survives(lambda s: Early([6], random.Random(s)), range(100)) is not None


def test_the_model_catches_one_buffer_for_the_row_maxima():
    class OneBuffer(Forward):
        def compute(self, a):
            for op in super().compute(a):
                yield (op[0], ("part", 0, op[1][2]), op[2]) if op[0] in ("read", "write") and op[1][0] == "part" else op

    assert survives(lambda s: OneBuffer([6], random.Random(s)), range(100)) is not None


def test_the_model_catches_two_stages_released_as_three():
    class Short(Backward):
        def loader(self, t):
            for op in super().loader(t):
                yield ("wait", op[1], op[2] - 1) if op[0] == "wait" and op[1].startswith("b2") and op[2] > 0 else op

    with pytest.raises(Violation):
        for seed in range(200):
            Short([(False, 9)], random.Random(seed)).run()


def test_the_model_catches_products_at_work_when_the_block_retires():
    class Leaves(Forward):
        def issuing(self, body, bar="settled"):
            return body

    found = survives(lambda s: Leaves([3, 3], random.Random(s), abort=True), range(500))
    assert found is not None and "at work" in found[1]
