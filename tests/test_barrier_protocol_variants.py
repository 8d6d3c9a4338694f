"""CPU: the barrier model of test_barrier_protocol_model.py for the head-size-64 forward on sequences of one tile
(flash_fwd64_kernel<.., true>, dadgpt_b200/csrc/flash_fwd64_sm100.cu)."""
import random

import pytest

from tests.barrier_model import survives
from tests.test_barrier_protocol_model import FwdSim

ONE_TILE_LISTS = [[(1, 1)] * 9, [(1, 1), (1, 1), (1, 0)], [(1, 0)], [(1, 1)], [(1, 1)] * 4 + [(1, 0)]]


@pytest.mark.parametrize("abort", [False, True], ids=["runs", "gives_up"])
def test_one_tile_forward_survives_every_schedule(abort):
    for items in ONE_TILE_LISTS:
        assert survives(lambda s: FwdSim(items, random.Random(s), True, abort), range(100)) is None, items


def test_the_model_catches_a_q_buffer_loaded_without_its_release():
    class Unreleased(FwdSim):
        def producer(self):
            return (op for op in super(Unreleased, self).producer() if not op[1].startswith("q_empty"))

    assert survives(lambda s: Unreleased([(1, 1)] * 9, random.Random(s), True), range(300)) is not None


def test_the_tile_spans_cover_the_ring():
    for items in ONE_TILE_LISTS:
        model = FwdSim(items, random.Random(0), True)
        for item in items:
            spans = [model.span(item, X) for X in (0, 1)]
            assert sorted(t for b, e in spans for t in range(b, e)) == list(range(model.n_kv(item)))
