"""Horizon gradients linearise at the states that were admitted.

A state recomputed from a checkpoint is bit for bit the one of the forward
sweep, whichever schedule the checkpoints follow: the stored cotangents are
scaled by powers of two, so FP32 gradients of schedules that step the
cotangent alike are equal to the last bit.
"""
import numpy as np
import pytest

from implexity_b200 import LbmSolver, workloads

pytestmark = pytest.mark.gpu

T = 12
W = np.array([0.3, 0.1, 0.0, 1e3, 1e3, 0.0, 1.0, 1e6])


def problem(shape, lattice, storage, reconstruction=None):
    solid = np.zeros(shape, bool)
    solid[shape[0] // 2, : shape[1] // 2, 1:3] = True
    p = workloads.channel_problem(shape=shape, steps=T, lattice=lattice, storage=storage, solid=solid)
    if reconstruction:
        p["ports"][1]["reconstruction"] = reconstruction
        p["design_region"][-2] = False
    return p


CASES = {
    "14x9x8": problem((14, 9, 8), "D3Q19", "float32"),
    "23x17x13_q27": problem((23, 17, 13), "D3Q27", "float32"),
    "23x17x13_f16": problem((23, 17, 13), "D3Q19", "float16"),
    # steps launch by launch
    "extrapolating": problem((14, 9, 8), "D3Q19", "float32", "non_equilibrium_extrapolation"),
}


@pytest.mark.parametrize("name", CASES)
def test_recomputed_states_are_the_admitted_ones(gpu_lib, name):
    """Spans of 2 to 12 states, the kept records, and two levels of spans."""
    prob = CASES[name]
    with LbmSolver(prob) as s:
        s.set_design(workloads.uniform_design(tuple(prob["shape"]), 3))
        kept, _ = s.gradient(W)
        for K in (2, 3, 4, 6, 12):
            g, rep = s.gradient(W, checkpoint_every=K)
            assert rep.forward_recomputed > 0
            assert np.array_equal(g, kept), K
        record = int(np.prod(prob["shape"])) * 16
        two, rep = s.gradient(W, checkpoint_every=12, record_budget_bytes=2 * record + (8 << 10))
        assert rep.forward_recomputed > T
        assert np.array_equal(two, kept)


@pytest.mark.parametrize("name", CASES)
def test_binomial_states_are_the_admitted_ones(gpu_lib, name):
    """Both schedules take one transposed step at a time."""
    prob = CASES[name]
    with LbmSolver(prob) as s:
        s.set_design(workloads.uniform_design(tuple(prob["shape"]), 3))
        one, _ = s.gradient(W, checkpoint_every=1)
        for snapshots in (2, 5):
            g, _ = s.gradient(W, checkpointing="binomial", snapshots=snapshots)
            assert np.array_equal(g, one), snapshots


def test_kept_sixteen_bit_cotangents_over_several_spans(gpu_lib):
    """Spans of 7 states, each rescaled, kept and recomputed alike."""
    prob = workloads.channel_problem(shape=(23, 17, 13), steps=40)
    with LbmSolver(prob) as s:
        s.set_design(workloads.uniform_design((23, 17, 13), 3))
        for storage in ("float16", "bfloat16"):
            kept, a = s.gradient(W, lambda_storage=storage)
            g, b = s.gradient(W, lambda_storage=storage, record_budget_bytes=1 << 30)
            assert a.forward_recomputed == 0 and b.forward_recomputed > 0
            assert np.array_equal(g, kept), storage


def test_kept_float32_cotangents_over_several_spans(gpu_lib):
    """Kept FP32 records are rescaled every 256 steps, recomputed ones every 25."""
    prob = workloads.channel_problem(shape=(9, 7, 6), steps=600)
    with LbmSolver(prob) as s:
        s.set_design(workloads.uniform_design((9, 7, 6), 3))
        kept, _ = s.gradient(W)
        g, rep = s.gradient(W, record_budget_bytes=1 << 30)
    assert rep.forward_recomputed > 0
    assert np.array_equal(g, kept)
