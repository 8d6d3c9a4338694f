"""CPU: the host-only barrier models of test_barrier_protocol_model.py for two more layouts: the gradient
kernel that writes fp32 results (flash_bwd_fused_kernel<0, true>, flash_bwd_fused_sm100.cu) and the
head-size-64 forward on sequences of one tile (flash_fwd64_kernel<.., true>, flash_fwd64_sm100.cu)."""
import random

import pytest

from tests.test_barrier_protocol_model import ITEM_LISTS, KV_STAGES, FwdSim, Sim, Violation


class F32Sim(Sim):
    """dV of an item leaves through the dQ staging buffer ahead of its last tile's dQ: one more use of
    that buffer per item. dK leaves through the item's K and V buffers."""

    def __init__(self, items, rng, wait_between=True):
        super().__init__(items, True, rng)
        self.wait_between = wait_between

    def drain(self):
        g = used = 0
        for j, n_it in enumerate(self.items):
            for i in range(n_it):
                if used > 0:
                    yield ("wait", "dq_sent", used - 1)
                yield ("wait", "acc_done", g)
                if i + 1 == n_it:
                    yield ("arrive", "dq_staged")             # dV
                    used += 1
                    yield ("arrive", "dkv_drained")
                    yield ("arrive", self.dkv(j)[0])          # dK
                    if self.wait_between:
                        yield ("wait", "dq_sent", used - 1)
                yield ("arrive", "dq_drained")
                yield ("arrive", "dq_staged")
                g += 1
                used += 1

    def reducer(self):
        g = 0   # uses of the staging buffer
        for j, n_it in enumerate(self.items):
            for i in range(n_it):
                if i + 1 == n_it:
                    yield ("wait", "dq_staged", g)
                    yield ("arrive", "dq_sent")
                    g += 1
                yield ("wait", "dq_staged", g)
                if i + 1 == n_it:
                    yield ("wait", *self.dkv(j))
                yield ("arrive", "dq_sent")
                if i + 1 == n_it:
                    yield ("arrive", f"dkv_sent[{j & 1}]")
                g += 1


def test_fp32_results_survive_every_schedule():
    for items in ITEM_LISTS:
        for seed in range(300):
            F32Sim(items, random.Random(seed)).run()


def test_the_model_catches_a_staging_buffer_used_twice_at_once():
    with pytest.raises(Violation):
        for seed in range(300):
            F32Sim([3, 1, 1, 2], random.Random(seed), wait_between=False).run()


class OneTileSim(FwdSim):
    """Items are two units of one tile each, (1, 1), or a last one alone, (1, 0). Ring tile 0 is group
    A's, ring tile 1 group B's: each group takes part in the tiles begin .. end - 1."""

    @staticmethod
    def n_kv(item):
        return item[0] + item[1]

    @staticmethod
    def span(item, X):
        return (item[0], item[0] + item[1]) if X and item[1] else (0, item[X])

    def issuer_x(self, X):
        q, items = f"tensor_{'AB'[X]}", self.items
        yield ("wait", "q_full[0]", 0)
        yield ("wait", "k_full[0]", 0)
        begin, end = self.span(items[0], X)
        if end > 0 and begin == 0:
            yield ("commit", f"s_full[{X}][0]", q)
            yield ("commit", f"s_full[{X}][1]", q)
            if end == 1:
                yield ("commit", "q_empty[0]", q)
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
                        if j == j0 and c == 0 and n_done > 0:
                            yield ("wait", f"o_free[{X}]", n_done - 1)
                        yield ("wait", f"p_full[{X}][{c}]", n_pv >> 1)
                        yield ("commit", f"o_done[{X}][{n_pv & 1}]", q)
                        n_pv += 1
                        issued = True
                    if s_next:
                        if not next_ready:
                            if nj == b:
                                yield ("wait", f"q_full[{nqb}]", (k + 1 if last else k) >> 1)
                            yield ("wait", f"k_full[{(g + 1) % KV_STAGES}]", (g + 1) // KV_STAGES)
                            next_ready = True
                        yield ("commit", f"s_full[{X}][{c}]", q)
                        issued = True
                        if c == 1 and nj + 1 == e:
                            yield ("commit", f"q_empty[{nqb}]", q)
                if have_next and e == 0 and nj == 0:
                    if last:
                        yield ("wait", f"q_full[{nqb}]", (k + 1) >> 1)
                    yield ("arrive", f"q_empty[{nqb}]")
                yield ("commit", f"kv_empty[{s}]", q) if issued else ("arrive", f"kv_empty[{s}]")
                g += 1
            if j1 > j0:
                n_done += 1


ONE_TILE_LISTS = [[(1, 1)] * 9, [(1, 1), (1, 1), (1, 0)], [(1, 0)], [(1, 1)], [(1, 1)] * 4 + [(1, 0)]]


def test_one_tile_forward_survives_every_schedule():
    for items in ONE_TILE_LISTS:
        for seed in range(200):
            OneTileSim(items, random.Random(seed)).run()


def test_the_model_catches_a_q_buffer_loaded_without_its_release():
    class Unreleased(OneTileSim):
        def producer(self):
            return (op for op in super(Unreleased, self).producer() if not op[1].startswith("q_empty"))

    with pytest.raises(Violation):
        for seed in range(300):
            Unreleased([(1, 1)] * 9, random.Random(seed)).run()


def test_the_tile_spans_cover_the_ring():
    for items in ONE_TILE_LISTS:
        for item in items:
            spans = [OneTileSim.span(item, X) for X in (0, 1)]
            assert sorted(t for b, e in spans for t in range(b, e)) == list(range(OneTileSim.n_kv(item)))
