"""The scale of the stored cotangent over the range of FP32."""
import numpy as np
import pytest

from implexity_b200 import LbmSolver, normalize, workloads
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

STEPS = 20


@pytest.mark.parametrize("storage", ["float32", "float16", "bfloat16"])
def test_gradient_is_linear_in_tiny_weights(gpu_lib, storage):
    """Weights that put the seeds' root mean square near 2^-124.5, above FP32's
    smallest normal value: stored at a scale of one, a 16-bit cotangent would
    be zero.  What a step adds to the gradient is formed in true units, where
    FP32's spacing is 2^-149: STEPS of those, beside the roundings that the
    gradient has anyway (2e-6 in FP32; 16-bit cotangents are stored as the same
    numbers but where a seed's last bit tips the rounding, 4 units of the
    format at most)."""
    shape = (14, 9, 8)
    prob = workloads.channel_problem(shape=shape, steps=STEPS)
    w = np.zeros(8)
    w[6] = 1.0  # the pressure drop: seeds of one size in the 84 port cells
    port = prob["density_kg_m3"] * (prob["spacing_m"] / prob["step_s"]) ** 2 / 3.0 / 42.0
    k = round(-124.5 - np.log2(port * np.sqrt(84 / np.prod(shape))))
    with LbmSolver(prob) as s:
        s.set_design(workloads.uniform_design(shape, 3))
        g, _ = s.gradient(w, lambda_storage=storage, checkpoint_every=5)
        tiny, _ = s.gradient(w * 2.0**k, lambda_storage=storage, checkpoint_every=5)
    err = np.linalg.norm(tiny * 2.0**-k - g) / np.linalg.norm(g)
    floor = STEPS * 2.0**-149 * np.sqrt(np.prod(shape)) / (np.linalg.norm(g) * 2.0**k)
    assert err < floor + {"float32": 2e-6, "float16": 2.0**-9, "bfloat16": 2.0**-6}[storage], (err, floor)


@pytest.mark.parametrize("lattice,collision,tau,every,bound",
                         [("D3Q19", "mrt", 1.0, 40, 2.0e-4), ("D3Q27", "trt", 0.8, 0, 1.8e-4)])
def test_half_precision_gradient_error(gpu_lib, lattice, collision, tau, every, bound):
    """A horizon of 300 steps, state and cotangent in FP16, against FP64.  The
    cotangents of a pressure objective are nearly one value; scaled to a root
    mean square of one they left 1.07e-4 to 1.44e-4 (MRT) and 1.32e-4 to 1.68e-4
    (D3Q27) over six designs.  Scaled by a power of two, 0.7 to 1.4, they left
    3.3e-4 and 1.9e-4 at least."""
    shape = (40, 24, 20)
    prob = workloads.channel_problem(shape=shape, steps=300, tau=tau, collision=collision, lattice=lattice,
                                     storage="float16", mrt_bulk_rate=1.2 if collision == "mrt" else None)
    norm = normalize(prob)
    w = workloads.objective_weights()
    raw = workloads.uniform_design(shape, 2)
    g_ref, _, _, st = Oracle(norm).gradient(raw, w, mode="horizon", K=18)
    assert st == 0
    with LbmSolver(norm) as s:
        s.set_design(raw)
        g, _ = s.gradient(w, lambda_storage="float16", checkpoint_every=every)
    err = np.linalg.norm(g.ravel() - g_ref) / np.linalg.norm(g_ref)
    assert err < bound, err
