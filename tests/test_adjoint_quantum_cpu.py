"""The block-wide maximum of the adjoint kernels, whose slots are shared by
batches that only one barrier separates, and the quantum that follows it: the code
of the kernels' header, run on the host."""
import itertools

import numpy as np
import pytest

from device_math_build import load


@pytest.fixture(scope="module")
def dm(tmp_path_factory):
    return load(str(tmp_path_factory.mktemp("device_math")))


def maxima(slots, slot, cleared, order, values):
    """What the threads read as each batch's maximum when, between two barriers,
    the reads of a batch, thread 0's clear and the next batch's collection take
    place in the given order (a reader may come last of all)."""
    mem, got = [0] * slots, []
    mem[slot(0)] = max(mem[slot(0)], values[0])  # collected before the first barrier
    for it in range(len(values)):
        for what in order:
            if what == "read":
                got.append(mem[slot(it)])
            elif what == "clear":
                mem[cleared(it)] = 0
            elif it + 1 < len(values):
                mem[slot(it + 1)] = max(mem[slot(it + 1)], values[it + 1])
    return got


VALUES = [5, 3, 9, 1, 4, 4, 8, 2]


@pytest.mark.parametrize("order", list(itertools.permutations(("read", "clear", "collect"))))
def test_every_order_between_two_barriers_gives_each_batch_its_maximum(dm, order):
    assert maxima(dm.dm_max_slots(), dm.dm_max_slot, dm.dm_max_cleared, order, VALUES) == VALUES


def test_two_slots_lose_a_maximum():
    """the check finds the fault that two slots have: cleared after the barrier by
    thread 0, while another warp already collects the next batch there"""
    got = maxima(2, lambda it: it & 1, lambda it: (it & 1) ^ 1, ("read", "collect", "clear"), VALUES)
    assert got != VALUES


@pytest.mark.parametrize("form,bits,coarsest,least", [("plain", 50, 44, -900), ("mixed", 30, 22, -93)])
def test_quantum_holds_a_batch_and_rounds_it_no_coarser(dm, form, bits, coarsest, least):
    """Over batches whose largest value jumps by any power of two: every contribution
    is below 2^bits quanta, and the quantum is at most 2^-coarsest of the power of two
    above the batch's largest (except below the least quantum)."""
    rng = np.random.default_rng(3)
    plain = form == "plain"
    quantum = dm.dm_quantum_plain if plain else dm.dm_quantum_mixed
    lo, hi = (-1000, 1000) if plain else (-126, 126)
    E = dm.dm_no_quantum()
    for e in np.concatenate([rng.integers(lo, hi, 2000), np.cumsum(rng.integers(-4, 5, 2000)).clip(lo, hi), [hi, lo, hi]]):
        v = rng.uniform(1.0, 2.0) * 2.0 ** float(e)
        word = int(np.float64(v).view(np.uint64) >> np.uint64(32)) if plain else int(np.float32(v).view(np.uint32))
        E = quantum(E, word)
        top = int(e) + 1  # v < 2^top
        assert top <= E and E >= least
        assert E - bits <= top - coarsest or E == least
        assert quantum(E, word) == E
