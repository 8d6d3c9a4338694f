"""CPU: barrier models (tests/barrier_model.py) of the bf16 kernels of head size 128, the forward of
dadgpt_b200/csrc/flash_bf16_sm100.cu and the single-pass backward of flash_bwd_fused128_sm100.cu, and of the
two-kernel backward of flash_bwd_bf16_sm100.cu (both head sizes). Softmax, compute and drain warps are two agents."""
import random

import pytest

from tests.barrier_model import Model, survives

PARTS = (0, 1)


class Forward(Model):
    """n key tiles. The agents of the softmax are the two halves of a row."""
    STAGES = 2
    need = {"p_full": 2, "stat_full": 2}

    def __init__(self, n, rng, abort=False, p_full=2):
        super().__init__(rng, abort)
        self.n, self.p_full = n, p_full   # p_full: barriers for "the probabilities are there"

    def wait_p(self, i):
        return f"p_full[{i % self.p_full}]", i // self.p_full

    def producer(self):
        yield ("tma", "q_full", [("q", "Q")])
        for j in range(self.n):
            s, use = j % self.STAGES, j // self.STAGES
            for m in "kv":
                if use > 0:
                    yield ("wait", f"{m}_empty[{s}]", use - 1)
                yield ("tma", f"{m}_full[{s}]", [((m, s), j)])

    def issuer(self):
        def pv(i):
            s = i % self.STAGES
            yield ("wait", f"v_full[{s}]", i // self.STAGES)
            yield ("wait", *self.wait_p(i))
            for h in PARTS:
                yield ("mma", [(("scores", i & 1, h), ("p", i)), (("v", s), i)] + ([(("out", h), i - 1)] if i else []), [(("out", h), i)])
            yield ("commit", f"v_empty[{s}]")
            yield ("commit", f"o_done[{i & 1}]")

        yield ("wait", "q_full", 0)
        for j in range(self.n):
            s = j % self.STAGES
            yield ("wait", f"k_full[{s}]", j // self.STAGES)
            yield ("mma", [("q", "Q"), (("k", s), j)], [(("scores", j & 1, h), ("s", j)) for h in PARTS])
            yield ("commit", f"k_empty[{s}]")
            yield ("commit", f"s_full[{j & 1}]")
            if j > 0:
                yield from pv(j - 1)
        yield from pv(self.n - 1)

    def softmax(self, h):
        for j in range(self.n):
            yield ("wait", f"s_full[{j & 1}]", j >> 1)
            yield ("read", ("scores", j & 1, h), ("s", j))
            if j > 0 and self.rng.random() < 0.3:   # the lazy rescale
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

    def agents(self):
        return {"producer": self.producing(self.producer()), "issuer": self.issuing(self.issuer()),
                **{f"softmax{h}": self.softmax(h) for h in PARTS}}


class Backward(Model):
    """n steps of 64 queries."""
    STAGES = 4
    need = {"x_full": 2, "x_free": 2, "w_full": 2, "dq_drained": 2}

    def __init__(self, n, rng, abort=False):
        super().__init__(rng, abort)
        self.n = n

    def producer(self):
        yield ("tma", "kv_full", [("kv", True)])
        for i in range(self.n):
            s, use = i % self.STAGES, i // self.STAGES
            if use > 0:
                yield ("wait", f"qdo_empty[{s}]", use - 1)
            yield ("tma", f"qdo_full[{s}]", [(("qdo", s), i)])

    def issuer(self):
        def x(i):
            s = i % self.STAGES
            yield ("wait", f"qdo_full[{s}]", i // self.STAGES)
            yield ("mma", [("kv", True), (("qdo", s), i)], [((c, a), i) for c in ("scores", "dp") for a in PARTS])
            yield ("commit", f"x_full[{i & 1}]")

        yield ("wait", "kv_full", 0)
        yield from x(0)
        for i in range(self.n):
            s = i % self.STAGES
            if i + 1 < self.n:
                yield ("wait", "x_free", i)
                yield from x(i + 1)
            yield ("wait", "w_full", i)
            yield ("mma", [((c, a), i) for c in ("p", "ds_t") for a in PARTS] + [(("qdo", s), i)] + ([("dkv", i - 1)] if i else []),
                   [("dkv", i)])
            yield ("commit", f"qdo_empty[{s}]")
            if i > 0:
                yield ("wait", "dq_drained", i - 1)
            yield ("mma", [("kv", True)] + [(("ds", a), i) for a in PARTS], [("dq", i)])
            yield ("commit", "acc_done")

    def scalars(self):
        for i in range(self.n):
            if i >= 2:
                yield ("wait", f"qdo_empty[{(i - 2) % self.STAGES}]", (i - 2) // self.STAGES)
            yield ("write", ("scalars", i & 1), i)
            yield ("arrive", f"x_full[{i & 1}]")

    def drain(self, d):
        for i in range(self.n):
            yield ("wait", "acc_done", i)
            yield ("read", "dq", i)
            yield ("arrive", "dq_drained")

    def compute(self, a):
        for i in range(self.n):
            yield ("wait", f"x_full[{i & 1}]", i >> 1)
            yield ("read", ("scores", a), i)
            yield ("read", ("dp", a), i)
            yield ("arrive", "x_free")
            yield ("read", ("scalars", i & 1), i)
            if i > 0:
                yield ("wait", "acc_done", i - 1)
            for c in ("p", "ds_t", "ds"):
                yield ("write", (c, a), i)
            yield ("arrive", "w_full")
        yield ("wait", "acc_done", self.n - 1)
        yield ("read", "dkv", self.n - 1)

    def agents(self):
        return {"producer": self.producing(self.producer()), "issuer": self.issuing(self.issuer()), "scalars": self.scalars(),
                **{f"compute{a}": self.compute(a) for a in PARTS}, **{f"drain{d}": self.drain(d) for d in PARTS}}


class TwoKernel(Model):
    """n steps; `bufs` score buffers (1 at head size 64, 2 at 128); kv: the kernel with row scalars per step."""
    STAGES = 3
    need = {"x_free": 2, "w_full": 2, "vec_full": 2}

    def __init__(self, n, rng, bufs, kv, abort=False):
        super().__init__(rng, abort)
        self.n, self.bufs, self.kv = n, bufs, kv

    def producer(self):
        yield ("tma", "r_full", [("r", True)])
        for i in range(self.n):
            s, use = i % self.STAGES, i // self.STAGES
            if use > 0:
                yield ("wait", f"c_empty[{s}]", use - 1)
            for m in "12":
                yield ("tma", f"c{m}_full[{s}]", [(("c" + m, s), i)])

    def issuer(self):
        def x(i):
            s = i % self.STAGES
            for m in "12":
                yield ("wait", f"c{m}_full[{s}]", i // self.STAGES)
                yield ("mma", [("r", True), (("c" + m, s), i)], [(("x" + m, i % self.bufs, a), i) for a in PARTS])
            yield ("commit", f"x_full[{i % self.bufs}]")

        yield ("wait", "r_full", 0)
        for i in range(min(self.bufs, self.n)):
            yield from x(i)
        for i in range(self.n):
            if i + self.bufs < self.n:
                yield ("wait", f"x_free[{i % self.bufs}]", i // self.bufs)
                yield from x(i + self.bufs)
            s = i % self.STAGES
            yield ("wait", "w_full", i)
            yield ("mma", [(("w", a), i) for a in PARTS] + [(("c" + m, s), i) for m in "12"], [("acc", i)])
            yield ("commit", f"c_empty[{s}]")
            yield ("commit", "acc_done")

    def compute(self, a):
        for i in range(self.n):
            if self.kv:
                if i > 0:
                    yield ("wait", "w_full", i - 1)
                yield ("write", ("vec", a), i)
                yield ("arrive", "vec_full")
                yield ("wait", "vec_full", i)
            yield ("wait", f"x_full[{i % self.bufs}]", i // self.bufs)
            for m in "12":
                yield ("read", ("x" + m, i % self.bufs, a), i)
            yield ("arrive", f"x_free[{i % self.bufs}]")
            if self.kv:
                for b in PARTS:
                    yield ("read", ("vec", b), i)
            if i > 0:
                yield ("wait", "acc_done", i - 1)
            yield ("write", ("w", a), i)
            yield ("arrive", "w_full")
        yield ("wait", "acc_done", self.n - 1)
        yield ("read", "acc", self.n - 1)

    def agents(self):
        return {"producer": self.producing(self.producer()), "issuer": self.issuing(self.issuer()),
                **{f"compute{a}": self.compute(a) for a in PARTS}}


LENGTHS = (1, 2, 3, 5, 17)


@pytest.mark.parametrize("abort", [False, True], ids=["runs", "gives_up"])
@pytest.mark.parametrize("make", [Forward, Backward, *(lambda n, rng, abort, b=b, kv=kv: TwoKernel(n, rng, b, kv, abort)
                                                       for b in (1, 2) for kv in (False, True))])
def test_every_schedule(make, abort):
    for n in LENGTHS:
        assert survives(lambda s: make(n, random.Random(s), abort), range(80)) is None, n


def test_the_forward_needs_a_probability_barrier_per_score_buffer():
    """With one for both, a warp a tile ahead stood in for another's arrival, and products ran on scores."""
    found = survives(lambda s: Forward(8, random.Random(s), p_full=1), range(300))
    assert found is not None and ("scores" in found[1] or "p_full" in found[1])


def _without(base, role, gone):
    class Model_(base):
        pass

    def faulty(self, *args):
        for op in getattr(base, role)(self, *args):
            if not (op[0] == "wait" and op[1].split("[")[0] == gone):
                yield op
    setattr(Model_, role, faulty)
    return Model_


@pytest.mark.parametrize("base,role,gone", [(Forward, "producer", "k_empty"), (Forward, "producer", "v_empty"), (Forward, "softmax", "o_done"),
                                            (Forward, "softmax", "stat_full"), (Backward, "issuer", "x_free"), (Backward, "issuer", "dq_drained"),
                                            (Backward, "compute", "acc_done"), (Backward, "scalars", "qdo_empty"), (Backward, "producer", "qdo_empty")])
def test_the_models_miss_no_wait_that_is_left_out(base, role, gone):
    assert survives(lambda s: _without(base, role, gone)(9, random.Random(s)), range(300)) is not None
