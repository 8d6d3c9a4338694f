"""CPU: barrier model (tests/barrier_model.py) of the single-pass backward of head size 64,
dadgpt_b200/csrc/flash_bwd_fused_sm100.cu: three Q / dO stages, scores and dP^T with barriers of their own, a warp
that delivers the row scalars, the ring of work items with its seven readers, dQ, dV and dK through two staging
panels in turns (one turn for dV and dK of an item with bf16 results, two with fp32 results). Compute and drain
warps are two agents each."""
import random

import pytest

from tests.barrier_model import Model, survives

STAGES, RING = 3, 4
PARTS = (0, 1)

# query tiles of a CTA's items, in the order they come
ITEM_LISTS = [
    [3, 1, 1, 2],
    [8, 7, 1, 1, 1, 4, 1],
    [1, 1, 1, 1, 1, 1, 1],
    [2, 2, 2, 2],
    [5],
    [1, 6, 1, 6, 1],
]


class Fused64(Model):
    # compute and drain warps, row scalars, issuer and reducer read an item
    need = {"s_full": 2, "p_full": 2, "w_full": 2, "staged": 2, "dq_drained": 2, "dkv_drained": 2, "item_free": 7}

    def __init__(self, items, rng, f32=False, abort=False):
        super().__init__(rng, abort)
        self.items, self.f32 = items, f32

    def producer(self):
        def publish(n):
            if n >= RING:
                yield ("wait", f"item_free[{n % RING}]", n // RING - 1)
            yield ("write", ("item", n % RING), n)
            yield ("arrive", f"item_ready[{n % RING}]")

        yield from publish(0)
        g = 0
        for j, n_it in enumerate(self.items):
            if j >= 2:
                yield ("wait", f"kv_empty[{j & 1}]", (j >> 1) - 1)
            yield ("tma", f"kv_full[{j & 1}]", [(("kv", j & 1), j)])
            yield from publish(j + 1)   # (the end mark behind the last item)
            for _ in range(n_it):
                if g >= STAGES:
                    yield ("wait", f"qdo_empty[{g % STAGES}]", g // STAGES - 1)
                yield ("tma", f"qdo_full[{g % STAGES}]", [(("qdo", g % STAGES), g)])
                g += 1

    def fetch(self, n):
        yield ("wait", f"item_ready[{n % RING}]", n // RING)
        yield ("read", ("item", n % RING), n)
        yield ("arrive", f"item_free[{n % RING}]")

    def scalars(self):
        yield from self.fetch(0)
        yield from self.fetch(1)
        g = 0
        for j, n_it in enumerate(self.items):
            for _ in range(n_it):
                if g >= 2:
                    yield ("wait", f"qdo_empty[{(g - 2) % STAGES}]", (g - 2) // STAGES)
                yield ("write", ("scalars", g & 1), g)
                yield ("arrive", f"s_full[{g & 1}]")
                g += 1
            if j + 1 < len(self.items):
                yield from self.fetch(j + 2)

    def issuer(self):
        def scores(g, j):
            yield ("mma", [(("kv", j & 1), j), (("qdo", g % STAGES), g)], [(("scores", a), g) for a in PARTS])
            yield ("commit", f"s_full[{g & 1}]")

        def dp(g, j):
            yield ("mma", [(("kv", j & 1), j), (("qdo", g % STAGES), g)], [(("dp", a), ("dP", g)) for a in PARTS])
            yield ("commit", "dp_full")

        yield from self.fetch(0)
        yield ("wait", "kv_full[0]", 0)
        yield ("wait", "qdo_full[0]", 0)
        yield from scores(0, 0)
        yield from dp(0, 0)
        g = 0
        for j, n_it in enumerate(self.items):
            for i in range(n_it):
                last = i + 1 == n_it
                if last:
                    yield from self.fetch(j + 1)
                more = not last or j + 1 < len(self.items)
                jn = j + 1 if last else j
                stage = (("qdo", g % STAGES), g)
                yield ("wait", "p_full", g)
                if more:
                    if last:
                        yield ("wait", f"kv_full[{jn & 1}]", jn >> 1)
                    yield ("wait", f"qdo_full[{(g + 1) % STAGES}]", (g + 1) // STAGES)
                    yield from scores(g + 1, jn)
                if i == 0 and j > 0:
                    yield ("wait", "dkv_drained", j - 1)
                yield ("mma", [(("p", a), g) for a in PARTS] + [stage] + ([("dv", g - 1)] if i else []), [("dv", g)])
                yield ("wait", "w_full", g)
                yield ("mma", [(("dp", a), ("dS", g)) for a in PARTS] + [stage] + ([("dk", g - 1)] if i else []), [("dk", g)])
                if more:
                    yield from dp(g + 1, jn)
                yield ("commit", f"qdo_empty[{g % STAGES}]")
                if g > 0:
                    yield ("wait", "dq_drained", g - 1)
                yield ("mma", [(("ds", a), g) for a in PARTS] + [(("kv", j & 1), j)], [("dq", g)])
                yield ("commit", "acc_done")
                if last:
                    yield ("commit", f"kv_empty[{j & 1}]")
                g += 1

    def compute(self, a):
        g = 0
        for j, n_it in enumerate(self.items):
            yield from self.fetch(j)
            for _ in range(n_it):
                yield ("wait", f"s_full[{g & 1}]", g >> 1)
                yield ("read", ("scores", a), g)
                yield ("read", ("scalars", g & 1), g)
                yield ("wait", "dp_full", g)
                yield ("write", ("p", a), g)
                yield ("arrive", "p_full")
                yield ("read", ("dp", a), ("dP", g))
                yield ("read", ("scalars", g & 1), g)
                if g > 0:
                    yield ("wait", "acc_done", g - 1)
                yield ("write", ("dp", a), ("dS", g))
                yield ("write", ("ds", a), g)
                yield ("arrive", "w_full")
                g += 1
        yield from self.fetch(len(self.items))

    def drain(self, d):
        g = turn = 0

        def one_turn(sources, drained):
            """`sources`: what goes to each of the two panels."""
            for p in (0, 1):
                yield ("read", sources[p], g)
                if p == 1 and drained:
                    yield ("arrive", drained)
                if turn > 0:
                    yield ("wait", f"sent[{p}]", turn - 1)
                yield ("write", ("panel", p, d), turn)
                yield ("arrive", f"staged[{p}]")

        for j, n_it in enumerate(self.items):
            yield from self.fetch(j)
            for i in range(n_it):
                yield ("wait", "acc_done", g)
                if i + 1 == n_it:
                    if self.f32:
                        yield from one_turn(("dv", "dv"), None)
                        turn += 1
                        yield from one_turn(("dk", "dk"), "dkv_drained")
                    else:
                        yield from one_turn(("dv", "dk"), "dkv_drained")
                    turn += 1
                yield from one_turn(("dq", "dq"), "dq_drained")
                turn += 1
                g += 1
        yield from self.fetch(len(self.items))

    def reducer(self):
        turn = 0
        for j, n_it in enumerate(self.items):
            yield from self.fetch(j)
            for i in range(n_it):
                for _ in range((3 if self.f32 else 2) if i + 1 == n_it else 1):
                    for p in (0, 1):
                        yield ("wait", f"staged[{p}]", turn)
                        yield ("bulk", [(("panel", p, d), turn) for d in PARTS])
                    for p in (0, 1):
                        yield ("bulk_wait", 1 - p)
                        yield ("arrive", f"sent[{p}]")
                    turn += 1
        yield from self.fetch(len(self.items))
        yield ("bulk_wait", 0)

    def agents(self):
        return {"producer": self.producing(self.producer()), "issuer": self.issuing(self.issuer()), "scalars": self.scalars(),
                "reducer": self.reducer(), **{f"compute{a}": self.compute(a) for a in PARTS},
                **{f"drain{d}": self.drain(d) for d in PARTS}}


@pytest.mark.parametrize("abort", [False, True], ids=["runs", "gives_up"])
@pytest.mark.parametrize("f32", [False, True])
def test_every_schedule(f32, abort):
    for items in ITEM_LISTS:
        assert survives(lambda s: Fused64(items, random.Random(s), f32, abort), range(60)) is None, items


def _without(role, gone):
    """The kernel with a role's waits for one barrier left out."""
    class Model_(Fused64):
        pass

    def faulty(self, *args):
        for op in getattr(Fused64, role)(self, *args):
            if not (op[0] == "wait" and op[1].split("[")[0] == gone):
                yield op
    setattr(Model_, role, faulty)
    return Model_


@pytest.mark.parametrize("role,gone", [("issuer", "dq_drained"), ("issuer", "dkv_drained"), ("issuer", "p_full"), ("issuer", "w_full"),
                                       ("compute", "acc_done"), ("compute", "dp_full"), ("drain", "sent"), ("producer", "kv_empty"),
                                       ("producer", "qdo_empty"), ("scalars", "qdo_empty")])
def test_the_model_misses_no_wait_that_is_left_out(role, gone):
    """(The producer's wait for a free place of the item ring is not among them: the K / V buffers hold it back first.)"""
    items = [2, 1, 3, 1, 1, 1, 1, 2]
    assert survives(lambda s: _without(role, gone)(items, random.Random(s)), range(300)) is not None


def test_the_model_catches_row_scalars_that_follow_the_arithmetic():
    """Waiting for the arithmetic's own barrier would not do: it runs two phases ahead of this warp."""
    class Late(Fused64):
        def scalars(self):
            for op in super().scalars():
                if op[0] == "wait" and op[1].startswith("qdo_empty"):
                    s = int(op[1].split("[")[1][:-1])
                    op = ("wait", "w_full", op[2] * STAGES + s)
                yield op

    assert survives(lambda s: Late([5, 1, 2], random.Random(s)), range(300)) is not None
