"""CPU: a host-only model of the decode kernel's item counter (dadgpt_b200/csrc/decode.cu). CTA c of G starts
with item c, further items come from a counter in the workspace, and whoever makes the last claim of a
call returns it to zero. A CTA in which a bounded wait ran out stops working; the next call on the
workspace must find the counter at zero all the same."""
import random

import pytest


def run_call(counter, n_items, n_ctas, rng, abort_prob, claims_after_abort):
    """One call, the CTAs' steps in random order. Returns (counter afterwards, items taken up)."""
    taken = []

    def cta(c):
        nonlocal counter

        def claim():
            nonlocal counter
            at = counter
            counter = 0 if at == n_items - 1 else at + 1
            return min(at + n_ctas, n_items)

        item, ok = c, True
        while ok:
            taken.append(item)
            yield
            ok = rng.random() >= abort_prob          # a wait of the item's rows
            if ok:
                item = claim()
                yield
                ok = rng.random() >= abort_prob      # the wait for a slot of the item ring
            if ok and item >= n_items:
                return
        while claims_after_abort and item < n_items:
            item = claim()
            yield

    running = [cta(c) for c in range(n_ctas)]
    while running:
        c = rng.choice(running)
        if next(c, "end") == "end":
            running.remove(c)
    return counter, taken


@pytest.mark.parametrize("n_items,n_ctas", [(2, 1), (7, 3), (40, 8), (41, 40)])
def test_the_counter_is_zero_after_every_call(n_items, n_ctas):
    rng = random.Random(n_items)
    for call in range(300):
        abort_prob = 0.0 if call % 2 == 0 else 0.2
        counter, taken = run_call(0, n_items, n_ctas, rng, abort_prob, claims_after_abort=True)
        assert counter == 0
        if abort_prob == 0.0:
            assert sorted(taken) == list(range(n_items))


def test_the_model_shows_the_counter_left_behind_by_a_cta_that_only_stops():
    rng = random.Random(1)
    left = [run_call(0, 40, 8, rng, 0.2, claims_after_abort=False)[0] for _ in range(50)]
    assert any(left)
    counter = next(x for x in left if x)
    _, taken = run_call(counter, 40, 8, rng, 0.0, claims_after_abort=True)
    assert len(set(taken)) < 40   # items of the next call that nobody took up
