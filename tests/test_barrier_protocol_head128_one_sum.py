"""CPU: barrier model (tests/barrier_model.py) of the head-size-128 forward with one query tile per CTA, in its form with
one maximum and one accumulator per row (ONE_SUM of dadgpt_b200/csrc/flash_bf16_sm100.cu): a row's halves tell each other
their maxima of every tile, and look at the other's behind some of their own exponentials."""
import random

import pytest

from tests.barrier_model import survives
from tests.test_barrier_protocol_head128 import LENGTHS, PARTS, Forward, _without


class ForwardOneSum(Forward):
    def __init__(self, n, rng, abort=False, max_buffers=2, max_full=2):
        super().__init__(n, rng, abort)
        self.max_buffers, self.max_full = max_buffers, max_full
        self.grows = [j > 0 and rng.random() < 0.3 for j in range(n)]   # (both see the same two maxima)

    def issuer(self):
        for op in super().issuer():
            if op[0] == "mma" and any(c[0] == "out" for c, _ in op[2]):   # both halves' products write all of O
                i = op[2][0][1]
                first = op[2][0][0][1] == 0
                before = [(("out", h), i - 1 if first else ("half", i)) for h in PARTS] if i or not first else []
                op = ("mma", [r for r in op[1] if r[0][0] != "out"] + before, [(("out", h), ("half", i) if first else i) for h in PARTS])
            yield op

    def softmax(self, h):
        for j in range(self.n):
            b, f = j % self.max_buffers, j % self.max_full
            yield ("wait", f"s_full[{j & 1}]", j >> 1)
            yield ("read", ("scores", j & 1, h), ("s", j))
            yield ("write", ("max", b, h), j)
            yield ("arrive", f"max_full[{f}, {h}]")
            yield ("wait", f"max_full[{f}, {1 - h}]", j // self.max_full)
            yield ("read", ("max", b, 1 - h), j)
            if self.grows[j]:
                yield ("wait", f"o_done[{(j - 1) & 1}]", (j - 1) >> 1)
                yield ("read", ("out", h), j - 1)
                yield ("write", ("out", h), j - 1)
            yield ("write", ("scores", j & 1, h), ("p", j))
            yield ("arrive", self.wait_p(j)[0])
        yield ("write", "q", "stat")
        yield ("write", ("stat", h), True)
        yield ("arrive", "stat_full")
        yield ("wait", "stat_full", 0)
        yield ("wait", f"o_done[{(self.n - 1) & 1}]", (self.n - 1) >> 1)
        for other in PARTS:
            yield ("read", ("stat", other), True)
            yield ("read", ("out", other), self.n - 1)


@pytest.mark.parametrize("abort", [False, True], ids=["runs", "gives_up"])
def test_every_schedule(abort):
    for n in LENGTHS:
        assert survives(lambda s: ForwardOneSum(n, random.Random(s), abort), range(80)) is None, n


@pytest.mark.parametrize("missing", [{"max_buffers": 1}, {"max_full": 1}])
def test_the_agreed_maximum_needs_two_buffers_with_a_barrier_each(missing):
    assert survives(lambda s: ForwardOneSum(9, random.Random(s), **missing), range(300)) is not None


@pytest.mark.parametrize("role,gone", [("softmax", "o_done"), ("softmax", "max_full"), ("producer", "v_empty")])
def test_the_model_misses_no_wait_that_is_left_out(role, gone):
    assert survives(lambda s: _without(ForwardOneSum, role, gone)(9, random.Random(s)), range(300)) is not None
