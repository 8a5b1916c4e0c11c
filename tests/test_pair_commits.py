"""What the CTAs of a pair tell each other.  Commits that signal the other CTA of a pair (tcgen05.commit with a multicast arrive): a CTA may leave only when every one
that is addressed to it has arrived.  A model of who waits for which, with commits that arrive late and in any order: why the
barriers that hand on data are not enough, and waiting for the last slots of each ring (ring_drain, csrc/ptx.cuh) is."""
import os
import random

import pytest

import fractaltensor_b200.build as b


def _late_arrivals(rings, steps, drain, seed):
    """A step gives back one slot of each ring (name: its number of slots) and completes one accumulator, which the CTA's
    epilogue waits for.  Its producers wait for a slot before they fill it again and, with `drain`, for all slots at the end.
    Returns the commits that arrive after the CTA has left."""
    rng = random.Random(seed)
    arrives = {}
    for t in range(steps):
        for name in list(rings) + ["acc"]:
            arrives[name, t] = t + rng.choice([0.1, 0.1, 0.2, 3.0])
    waited = [arrives["acc", t] for t in range(steps)]
    for name, slots in rings.items():
        waited += [arrives[name, t] for t in range(steps if drain else steps - slots)]
    left = max(waited)
    return [k for k, at in arrives.items() if at > left]


KERNELS = {
    "lstm_flow.cuh": ({"in": 1, "ring": 4, "swept": 1}, 3),
    "flash_pair.cu": ({"k_empty": 4, "pv_done": 4, "q_empty": 2}, 3),
    "project.cu": ({"b": 6}, 1),
    "cell_gemm.cu": ({"stage": 6}, 1),
    "lstm_static.cu": ({"stage": 6}, 1),
}


@pytest.mark.parametrize("name", KERNELS)
def test_waiting_for_the_last_slots_is_enough(name):
    assert not any(_late_arrivals(KERNELS[name][0], 40, True, seed) for seed in range(50))


@pytest.mark.parametrize("name", KERNELS)
def test_waiting_for_the_accumulators_is_not(name):
    assert any(_late_arrivals(KERNELS[name][0], 40, False, seed) for seed in range(50))


@pytest.mark.parametrize("name", KERNELS)
def test_kernels_wait_for_each_ring(name):
    """That the source has the waits that the model is of (nothing more)."""
    src = open(os.path.join(b.CSRC, name)).read()
    rings = src.count("ring_drain(") + src.count("mbar_wait(&swept, ")
    if name == "flash_pair.cu":  # all rings at once, behind the last barrier
        teardown = src[src.rindex("tc_fence_before();"):src.rindex("cluster_sync_all();")]
        rings = sum("ctl.%s + i" % ring in teardown for ring in KERNELS[name][0])
    assert "umma_commit_pair" in src and rings == KERNELS[name][1]


def test_scopes_of_a_state_s_hand_over_include_each_other():
    """The state of a pair's other CTA is released at the cluster's scope; the wait in front of the MMAs that read it has that
    scope too (on a device the bits come out right either way: the scopes are a matter of the text)."""
    flow, ptx = (open(os.path.join(b.CSRC, f)).read() for f in ("lstm_flow.cuh", "ptx.cuh"))
    assert "mbar_arrive_peer_smem(map_to_cta(smem_u32(&st_full), 0))" in flow and "mbar_wait_cluster(&st_full, " in flow
    release = ptx[ptx.index("void mbar_arrive_peer_smem"):].split("\n}")[0]
    acquire = ptx[ptx.index("bool mbar_wait_cluster"):].split("\n}")[0]
    assert "fence.release" in release and "cta.cluster;" in release and "try_wait.parity.acquire.cluster" in acquire
