"""The count by which the cluster kernels' publisher knows that a step's output tile is whole
(csrc/rnn_cluster.cu), on a model of that count alone, with a warp held up as long as the kernel's waits
allow: why one count for all steps is not enough and one for each parity is.  The kernel itself is
compared bit for bit with the level launches on a device (test_gpu_dilated_flow.py, clusters; the grid's
in test_gpu_parity.py); an order of its warps that fails only rarely cannot be forced there."""
import random

import pytest

WARPS = 16


def _early_stores(counters, seed, steps=40):
    """Walks random interleavings of WARPS epilogue warps and the publisher.  A warp may stage step i once the
    publisher has stored step i - 2, whatever the other warps have done (a layer whose step needs the state
    two or more steps back).  Returns the steps stored while a warp's part of them was missing."""
    rng = random.Random(seed)
    done = [0] * WARPS         # steps staged by each warp
    count = [0] * counters
    stored, early = 0, []
    while stored < steps:
        if rng.random() < 0.5:
            # a few fast warps run, the others are held up
            w = rng.choice([0, 0, 0, 0, 1, 1, 2]) if rng.random() < 0.7 else rng.randrange(WARPS)
            i = done[w]
            if i < steps and stored >= i - 1:
                done[w] += 1
                count[i % counters] += 1
        elif count[stored % counters] >= WARPS * (stored // counters + 1):
            if min(done) <= stored:
                early.append(stored)
            stored += 1
    return early


@pytest.mark.parametrize("seed", range(20))
def test_a_count_for_each_parity_is_enough(seed):
    assert _early_stores(2, seed) == []


def test_one_count_is_not():
    assert any(_early_stores(1, seed) for seed in range(20))


def test_kernel_counts_by_parity():
    """That the source keeps the count the model is of (nothing more)."""
    import os
    import fractaltensor_b200.build as b
    src = open(os.path.join(b.CSRC, "rnn_cluster.cu")).read()
    assert "atomicAdd(&out_issued[i & 1], 1)" in src and "kEpiWarps * ((i >> 1) + 1)" in src
