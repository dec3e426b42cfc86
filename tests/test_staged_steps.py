"""The staged kernels (one launch per step) on small grids, and runs of steps
on grids where a thread owns several cells.

Grids below a million cells step in runs; what reaches the staged kernels on
them is a forward call of one step, one transposed step per segment
(checkpoint_every=1), an extrapolating port and the general MRT collision.

Bounds.  FP32: those of the parity tests (1e-5 of the largest population,
gradients 1e-4 relative L2 against FP64, 2e-5 between two FP32 orders of
operations).  16-bit storage of a state or a cotangent rounds every value once
a step, by u = 2^-10 (FP16, either way) or 2^-7 (BF16) of it; the roundings of
cells and steps are independent, so T steps leave sqrt(T) u, twice that as the
bound: of the deviations (f - w)/w direction by direction, of the gradient in
relative L2.  A direction lost or swapped, or a wall link taken from the wrong
slot, is off by the whole of it.
"""
import numpy as np
import pytest

from implexity_b200 import LbmSolver, normalize, workloads
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

U = {"float32": 0.0, "float16": 2.0**-10, "bfloat16": 2.0**-7}
W = np.array([0.3, 0.1, 0.0, 1e3, 1e3, 0.0, 1.0, 1e6])


def rel_l2(a, b):
    a, b = np.asarray(a, float).ravel(), np.asarray(b, float).ravel()
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def solids(shape):
    """Obstacles that stand on both z walls and in a corner."""
    nx, ny, nz = shape
    solid = np.zeros(shape, bool)
    solid[nx // 2, : ny // 2, :1] = True
    solid[nx // 3, ny // 3 : ny // 2, nz - 1 :] = True
    solid[2 * nx // 3, ny - 2 :, nz // 2 :] = True
    return solid


def channel(shape, steps, lattice="D3Q19", collision="trt", storage="float32", even_rate=None):
    p = workloads.channel_problem(shape=shape, steps=steps, lattice=lattice, collision=collision, storage=storage,
                                  mrt_bulk_rate=1.2 if collision == "mrt" else None, solid=solids(shape))
    if even_rate:
        p["solver_options"]["collision"]["even_rate"] = even_rate
    return p


def box(shape, steps, lattice="D3Q19", periodic=(True, False, True), storage="float32"):
    p = workloads.channel_problem(shape=shape, steps=steps, lattice=lattice, ports=False, storage=storage,
                                  solid=solids(shape))
    p["periodic_axes"] = list(periodic)
    p["acceleration_m_s2"] = [2e-5, -1e-6, 1e-6]
    return p


def pulsatile(shape, steps, lattice="D3Q19"):
    p = workloads.pulsatile_problem(shape=shape, steps=steps, lattice=lattice, period_steps=9)
    p["solid_mask"] = solids(shape)
    p["design_region"] &= ~p["solid_mask"]
    return p


T = 13
ADJOINT = {
    "closed_odd_nz": lambda q: channel((11, 7, 5), T, q),
    "closed_even_nz": lambda q: channel((14, 9, 8), T, q),
    "closed_nz_2": lambda q: box((12, 9, 2), T, q, (True, False, False)),
    "periodic_z": lambda q: box((12, 9, 7), T, q, (False, False, True)),
    "mrt_bulk": lambda q: channel((13, 8, 7), T, q, "mrt"),
    "mrt_general": lambda q: channel((13, 8, 7), T, q, "mrt", even_rate=1.4),
    "stage": lambda q: pulsatile((13, 8, 7), T, q),
    # more tiles than resident blocks: a block walks over several z residues
    "several_tiles": lambda q: channel((61, 47, 43), 5, q),
}


@pytest.mark.parametrize("storage", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("lattice", ["D3Q19", "D3Q27"])
@pytest.mark.parametrize("name", ADJOINT)
def test_single_transposed_steps_match_oracle(gpu_lib, name, lattice, storage):
    prob = ADJOINT[name](lattice)
    steps, shape = prob["step_count"], tuple(prob["shape"])
    norm = normalize(prob)
    raw = workloads.uniform_design(shape, 3)
    stage = name == "stage"
    g_ref, _, _, st = Oracle(norm).gradient(raw, W, mode="time_average" if stage else "horizon", K=steps)
    assert st == 0
    with LbmSolver(norm) as s:
        s.set_design(raw)
        g, rep = s.gradient(W, lambda_storage=storage, checkpoint_every=1,
                            objective="time_average" if stage else "final")
    assert rep.iterations == steps
    assert rel_l2(g, g_ref) < max(1e-4, 2.0 * np.sqrt(steps) * U[storage]), rel_l2(g, g_ref)


FORWARD = {
    "closed_odd_nz": lambda q, s: channel((11, 7, 5), T, q, storage=s),
    "mrt_bulk": lambda q, s: channel((13, 8, 7), T, q, "mrt", storage=s),
    "mrt_general": lambda q, s: channel((13, 8, 7), T, q, "mrt", storage=s, even_rate=1.4),
    "box": lambda q, s: box((12, 9, 7), T, q, storage=s),
    "closed_nz_2": lambda q, s: box((12, 9, 2), T, q, (True, False, False), storage=s),
    "several_tiles": lambda q, s: channel((61, 47, 43), 5, q, storage=s),
}


def deviations(f, rest):
    """(f - w)/w of fluid cells, [cells, q]."""
    return f / rest - 1.0


def per_direction(a, b):
    """Largest root-mean-square difference of a direction, of the whole's root mean square."""
    return float(np.sqrt(np.max(np.mean((a - b) ** 2, axis=0)) / np.mean(b**2)))


@pytest.mark.parametrize("storage", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("lattice", ["D3Q19", "D3Q27"])
@pytest.mark.parametrize("name", FORWARD)
def test_single_forward_steps_match_oracle(gpu_lib, name, lattice, storage):
    prob = FORWARD[name](lattice, storage)
    steps, shape = prob["step_count"], tuple(prob["shape"])
    norm = normalize(prob)
    raw = workloads.uniform_design(shape, 3)
    fluid = ~np.asarray(prob["solid_mask"]).ravel()
    o = Oracle(norm)
    _, alpha = o.design(raw)
    f_ref, _ = o.history(alpha, steps)
    rest = o.initial().reshape(f_ref.shape)[fluid]
    f_ref = f_ref[fluid]
    with LbmSolver(norm) as s:
        s.set_design(raw)
        s.forward(1)
        for _ in range(steps - 1):
            s.advance(1)
        f = s.populations()[fluid]
    assert np.max(np.abs(f - f_ref)) < max(1e-5, 2.0 * np.sqrt(steps) * U[storage]) * np.max(np.abs(f_ref))
    got, want = deviations(f, rest), deviations(f_ref, rest)
    assert per_direction(got, want) < max(1e-4, 2.0 * np.sqrt(steps) * U[storage])


# ------------------------------------------------------------------ runs, several cells per thread
RUNS = {  # 75 776 threads are resident at two blocks per SM
    "q27": lambda s: channel((67, 45, 43), T, "D3Q27", storage=s),
    "q19_mrt": lambda s: channel((61, 47, 45), T, "D3Q19", "mrt", storage=s),
    "box_q19": lambda s: box((53, 47, 45), T, storage=s),
    "box_q27": lambda s: box((47, 45, 43), T, "D3Q27", (True, True, True), storage=s),
}


@pytest.mark.parametrize("storage", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("name", RUNS)
def test_run_of_several_cells_per_thread_matches_single_steps(gpu_lib, name, storage):
    prob = RUNS[name](storage)
    fluid = ~np.asarray(prob["solid_mask"]).ravel()
    norm = normalize(prob)
    rest = Oracle(norm).initial().reshape(fluid.size, -1)[fluid]
    with LbmSolver(norm) as s:
        s.set_design(workloads.uniform_design(tuple(prob["shape"]), 3))
        s.forward(1)
        for _ in range(T - 1):
            s.advance(1)
        one = deviations(s.populations()[fluid], rest)
        s.forward()
        run = deviations(s.populations()[fluid], rest)
    # FP32: two roundings of 2^-24 of a population a step, of deviations near 0.1
    assert per_direction(run, one) < max(2e-5, 2.0 * np.sqrt(T) * U[storage])


@pytest.mark.parametrize("storage", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("name", ["q27", "q19_mrt", "box_q19", "box_q27", "stage_q19", "stage_q27"])
def test_transposed_run_of_several_cells_per_thread_matches_single_steps(gpu_lib, name, storage):
    if name.startswith("stage"):
        prob = pulsatile((47, 45, 43), T, "D3Q" + name[7:])
    else:
        prob = RUNS[name]("float32")
    objective = "time_average" if name.startswith("stage") else "final"
    with LbmSolver(prob) as s:
        s.set_design(workloads.uniform_design(tuple(prob["shape"]), 3))
        one, _ = s.gradient(W, lambda_storage=storage, checkpoint_every=1, objective=objective)
        run, _ = s.gradient(W, lambda_storage=storage, checkpoint_every=T, objective=objective)
    assert rel_l2(run, one) < max(2e-5, 2.0 * np.sqrt(T) * U[storage]), rel_l2(run, one)
