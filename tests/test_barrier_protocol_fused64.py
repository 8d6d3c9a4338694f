"""CPU: the host-only barrier model of test_barrier_protocol_model.py for the single-pass backward of
head size 64 as it stands in flash_bwd_fused_sm100.cu: three Q / dO stages, scores and dP^T with barriers
of their own, a warp that delivers the row scalars, dQ, dV and dK through two staging panels in turns (one
turn for dV and dK of an item with bf16 results, two with fp32 results)."""
import random

import pytest

from tests.test_barrier_protocol_model import ITEM_LISTS, Sim, Violation

STAGES = 3


class FusedSim(Sim):
    def __init__(self, items, rng, f32=False):
        super().__init__(items, True, rng)
        self.f32 = f32
        self.need = {"s_full": 2}   # the product and the row scalars

    def producer(self):
        g = 0
        for j, n_it in enumerate(self.items):
            if j >= 2:
                yield ("wait", f"kv_empty[{j & 1}]", (j >> 1) - 1)
            yield ("tma", f"kv_full[{j & 1}]")
            for _ in range(n_it):
                if g >= STAGES:
                    yield ("wait", f"qdo_empty[{g % STAGES}]", g // STAGES - 1)
                yield ("tma", f"qdo_full[{g % STAGES}]")
                g += 1

    def scalars(self):
        for g in range(sum(self.items)):
            if g >= 2:
                yield ("wait", f"qdo_empty[{(g - 2) % STAGES}]", (g - 2) // STAGES)
            yield ("arrive", f"s_full[{g & 1}]")

    def issuer(self):
        yield ("wait", "kv_full[0]", 0)
        yield ("wait", "qdo_full[0]", 0)
        yield ("commit", "s_full[0]")
        yield ("commit", "dp_full")
        g, n = 0, sum(self.items)
        for j, n_it in enumerate(self.items):
            for i in range(n_it):
                yield ("wait", "p_full", g)
                if g + 1 < n:
                    if i + 1 == n_it:
                        yield ("wait", f"kv_full[{(j + 1) & 1}]", (j + 1) >> 1)
                    yield ("wait", f"qdo_full[{(g + 1) % STAGES}]", (g + 1) // STAGES)
                    yield ("commit", f"s_full[{(g + 1) & 1}]")
                if i == 0 and j > 0:
                    yield ("wait", "dkv_drained", j - 1)
                yield ("wait", "w_full", g)
                if g + 1 < n:
                    yield ("commit", "dp_full")
                yield ("commit", f"qdo_empty[{g % STAGES}]")
                if g > 0:
                    yield ("wait", "dq_drained", g - 1)
                yield ("commit", "acc_done")
                if i + 1 == n_it:
                    yield ("commit", f"kv_empty[{j & 1}]")
                g += 1

    def compute(self):
        for g in range(sum(self.items)):
            yield ("wait", f"s_full[{g & 1}]", g >> 1)
            yield ("wait", "dp_full", g)
            yield ("arrive", "p_full")
            if g > 0:
                yield ("wait", "acc_done", g - 1)
            yield ("arrive", "w_full")

    def drain(self):
        g = turn = 0

        def one_turn(read):
            for p in (0, 1):
                if p == 1 and read:
                    yield ("arrive", read)
                if turn > 0:
                    yield ("wait", f"sent[{p}]", turn - 1)
                yield ("arrive", f"staged[{p}]")

        for n_it in self.items:
            for i in range(n_it):
                yield ("wait", "acc_done", g)
                if i + 1 == n_it:
                    if self.f32:
                        yield from one_turn(None)
                        turn += 1
                    yield from one_turn("dkv_drained")
                    turn += 1
                yield from one_turn("dq_drained")
                turn += 1
                g += 1

    def reducer(self):
        turn = 0
        for n_it in self.items:
            for i in range(n_it):
                for _ in range((3 if self.f32 else 2) if i + 1 == n_it else 1):
                    for p in (0, 1):
                        yield ("wait", f"staged[{p}]", turn)
                    for p in (0, 1):
                        yield ("arrive", f"sent[{p}]")
                    turn += 1

    def roles(self):
        return {**super().roles(), "scalars": self.scalars()}


@pytest.mark.parametrize("f32", [False, True])
def test_no_schedule_breaks_a_parity_wait(f32):
    for items in ITEM_LISTS:
        for seed in range(200):
            FusedSim(items, random.Random(seed), f32).run()


def test_the_model_catches_row_scalars_that_follow_the_arithmetic():
    """Waiting for the arithmetic's own barrier would not do: it runs two phases ahead of this warp."""
    class Late(FusedSim):
        def scalars(self):
            for g in range(sum(self.items)):
                if g >= 2:
                    yield ("wait", "w_full", g - 2)
                yield ("arrive", f"s_full[{g & 1}]")

    with pytest.raises(Violation):
        for seed in range(300):
            Late([5, 1, 2], random.Random(seed)).run()
