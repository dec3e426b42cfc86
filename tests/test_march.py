"""Runs of steps in one launch against one launch per step.

Grids below the march limit step a whole run per launch; a run of one step
takes the staged kernels.  Both perform the same FP32 operations per cell, up
to the compiler's choice of fused multiply-adds, so FP32 states agree to a few
roundings per step: 2e-6 of the largest population after the 13 steps here
(13 steps x 2 roundings x 6e-8), gradients to 2e-5 (their cancellation is the
~10x that the oracle comparisons show).  16-bit states may round a last digit
the other way: one unit of the storage format (2^-11, 2^-8) of (f - w)/w.
"""
import numpy as np
import pytest

from implexity_b200 import ContractError, LbmSolver, workloads

pytestmark = pytest.mark.gpu

T = 13


def rel_l2(a, b):
    a, b = np.asarray(a, float).ravel(), np.asarray(b, float).ravel()
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def channel(shape, lattice, collision, storage, **kw):
    solid = np.zeros(shape, bool)
    solid[shape[0] // 2, : shape[1] // 2, 1:3] = True
    return workloads.channel_problem(shape=shape, steps=T, lattice=lattice, collision=collision, storage=storage,
                                     mrt_bulk_rate=1.2 if collision == "mrt" else None, solid=solid, **kw)


def box(shape, lattice, periodic):
    p = channel(shape, lattice, "trt", "float32", ports=False)
    p["periodic_axes"] = list(periodic)
    p["acceleration_m_s2"] = [2e-5, -1e-6, 1e-6]
    return p


def regularized(shape):
    p = channel(shape, "D3Q19", "trt", "float32")
    for port in p["ports"]:
        port["reconstruction"] = "regularized_known_stress"
    return p


CASES = {
    # one block; several blocks of 128; one cell per thread over 256-thread blocks, two and three per SM;
    # several cells per thread
    "8x6x5": channel((8, 6, 5), "D3Q19", "bgk", "float32"),
    "23x17x13_mrt": channel((23, 17, 13), "D3Q19", "mrt", "float32"),
    "41x31x29_q27": channel((41, 31, 29), "D3Q27", "trt", "float32"),
    "53x45x43": channel((53, 45, 43), "D3Q19", "trt", "float32"),
    "67x45x43": channel((67, 45, 43), "D3Q19", "trt", "float32"),
    "67x45x43_f16": channel((67, 45, 43), "D3Q19", "trt", "float16"),
    "19x11x9_bf16": channel((19, 11, 9), "D3Q27", "mrt", "bfloat16"),
    "box_xyz": box((9, 7, 8), "D3Q27", (True, True, True)),
    "box_y": box((9, 7, 2), "D3Q19", (False, True, False)),
    "regularized": regularized((14, 9, 8)),
}
TOL = {"float32": 2e-6, "float16": 2.0**-11, "bfloat16": 2.0**-8}


@pytest.mark.parametrize("name", CASES)
def test_run_matches_single_steps(gpu_lib, name):
    prob = CASES[name]
    shape, storage = tuple(prob["shape"]), prob["solver_options"]["population_storage"]
    raw = workloads.uniform_design(shape, 3)
    with LbmSolver(prob) as s:
        s.set_design(raw)
        f0 = s.forward(1) and s.populations()
        s.set_populations(f0)
        one = {"mass": [], "min_population": [], "max_speed": []}
        for _ in range(T):
            s.advance(1)
            tr = s.trajectory()
            for k in one:
                one[k].append(tr[k][0])
        f_one = s.populations()
        s.set_populations(f0)
        d = s.advance(T)
        tr = s.trajectory()
        f_run = s.populations()
    assert d.steps == T
    assert np.max(np.abs(f_run - f_one)) <= TOL[storage] * np.max(np.abs(f_one))
    if storage == "float32":  # (single 16-bit steps restart the rounding's step count)
        for k in one:
            assert np.allclose(tr[k][:T], one[k], rtol=2e-6, atol=0.0), k


@pytest.mark.parametrize("name", [k for k in CASES if "16" not in k])
def test_adjoint_run_matches_single_steps(gpu_lib, name):
    """checkpoint_every=1 and check_every=1 take one transposed step per launch."""
    prob = CASES[name]
    w = np.array([0.3, 0.1, 0.0, 1e3, 1e3, 0.0, 1.0, 1e6])
    with LbmSolver(prob) as s:
        s.set_design(workloads.uniform_design(tuple(prob["shape"]), 3))
        g_one, a = s.gradient(w, mode="horizon", checkpoint_every=1)
        g_run, b = s.gradient(w, mode="horizon", checkpoint_every=T)
        assert a.iterations == b.iterations == T
        assert rel_l2(g_run, g_one) <= 2e-5
        if not prob["ports"]:  # a closed box conserves mass: its steady series does not converge
            return
        s.forward()
        g_steady, rep = s.gradient(w, mode="steady", tolerance=1e6, check_every=T)
        assert rep.iterations == T
        g_single, rep1 = s.gradient(w, mode="steady", tolerance=1e-3 * rep.residual, check_every=1,
                                    max_iterations=100000)
        g_again, rep2 = s.gradient(w, mode="steady", tolerance=1e-3 * rep.residual, check_every=rep1.iterations)
        assert rep2.iterations == rep1.iterations
        assert abs(rep2.residual - rep1.residual) <= 1e-3 * rep1.residual
        assert rel_l2(g_again, g_single) <= 2e-5


def test_pulsatile_run_matches_single_steps(gpu_lib):
    """Port maps, stage seeds and response sums that change from state to state."""
    prob = workloads.pulsatile_problem(shape=(17, 9, 8), steps=T, lattice="D3Q27", period_steps=9)
    w = np.array([0.3, 0.0, 0.0, 1e3, 1e3, 0.0, 1.0, 1e6])
    with LbmSolver(prob) as s:
        s.set_design(workloads.uniform_design((17, 9, 8), 3))
        s.forward()
        mean = s.time_average()
        g_one, _ = s.gradient(w, mode="horizon", checkpoint_every=1, objective="time_average")
        g_run, _ = s.gradient(w, mode="horizon", checkpoint_every=5, objective="time_average")
        g_bin, _ = s.gradient(w, mode="horizon", checkpointing="binomial", snapshots=3, objective="time_average")
        acc = np.zeros(8)
        for t in range(1, T + 1):
            s.forward(t)
            acc += s.responses() / T
    assert rel_l2(g_run, g_one) <= 2e-5
    assert rel_l2(g_bin, g_one) <= 2e-5
    # per-state sums in FP32 per cell against FP64 per cell
    assert np.allclose(mean[[0, 3, 4, 5, 6, 7]], acc[[0, 3, 4, 5, 6, 7]], rtol=1e-5)


@pytest.mark.parametrize("objective", ["final", "time_average"])
def test_kept_records_match_recomputed_ones(gpu_lib, objective):
    """checkpoint_every=0 keeps every state's record where they fit; a record
    budget makes it checkpoint.  The same records either way, on a grid whose
    odd cell count leaves a record's end unaligned."""
    prob = workloads.pulsatile_problem(shape=(9, 7, 5), steps=T, lattice="D3Q19", period_steps=9)
    w = np.array([0.3, 0.0, 0.0, 1e3, 1e3, 0.0, 1.0, 1e6])
    with LbmSolver(prob) as s:
        s.set_design(workloads.uniform_design((9, 7, 5), 3))
        g, kept = s.gradient(w, mode="horizon", objective=objective)
        g_ck, ck = s.gradient(w, mode="horizon", objective=objective, record_budget_bytes=1 << 30)
        g_one, _ = s.gradient(w, mode="horizon", objective=objective, checkpoint_every=1)
    assert kept.forward_recomputed == 0 and ck.forward_recomputed > 0
    assert kept.iterations == ck.iterations == T
    assert rel_l2(g, g_ck) <= 1e-6
    assert rel_l2(g, g_one) <= 2e-5


def test_staged_sums_across_chunks(gpu_lib):
    """Staged steps combine the partials of sixteen steps at a time: response
    sums and admission records of every state of a longer run, against the
    responses of each state (FP32 per cell against FP64) and single steps."""
    steps = 21
    prob = workloads.pulsatile_problem(shape=(11, 8, 7), steps=steps, lattice="D3Q19", period_steps=9)
    prob["ports"][1]["reconstruction"] = "non_equilibrium_extrapolation"  # a run of steps does not take it
    prob["design_region"][-2] = False
    with LbmSolver(prob) as s:
        s.set_design(workloads.uniform_design((11, 8, 7), 3))
        s.forward()
        mean, tr = s.time_average(), s.trajectory()
        acc = np.zeros(8)
        for t in range(1, steps + 1):
            s.forward(t)
            acc += s.responses() / steps
            one = s.trajectory()
            for k in ("mass", "min_population", "max_speed", "exchange"):
                assert one[k][t] == tr[k][t], (k, t)
    assert np.allclose(mean[[0, 3, 4, 5, 6, 7]], acc[[0, 3, 4, 5, 6, 7]], rtol=1e-5)


@pytest.mark.parametrize("shape", [(9, 8, 7), (40, 26, 24)])
def test_refused_design_keeps_the_last_map(gpu_lib, shape):
    """Checked on the host (504 cells) and on the device (24 960 cells)."""
    prob = workloads.channel_problem(shape=shape, steps=3)
    good = workloads.uniform_design(shape, 2)
    with LbmSolver(prob) as s:
        s.set_design(good)
        phi, alpha = s.design()
        for bad_value in (np.nan, 1.0 + 1e-9, -1e-300, np.inf):
            bad = workloads.uniform_design(shape, 5)
            bad[-1, -1, -1] = bad_value
            with pytest.raises(ContractError):
                s.set_design(bad)
        phi2, alpha2 = s.design()
        s.set_design(good)
        phi3, _ = s.design()
    assert np.array_equal(phi, phi2) and np.array_equal(alpha, alpha2) and np.array_equal(phi, phi3)


@pytest.mark.parametrize("lattice,shape", [("D3Q19", (5, 4, 3)), ("D3Q27", (17, 16, 15)), ("D3Q19", (96, 80, 64))])
def test_population_round_trip(gpu_lib, lattice, shape):
    """Less than a block, a partial last block, and more cells than one piece
    of the staging holds (441 505); g = f - w is kept in FP32, 2^-24 of 0.02."""
    q, n = int(lattice[3:]), int(np.prod(shape))
    prob = workloads.channel_problem(shape=shape, steps=1, lattice=lattice, ports=False)
    f = 0.05 + 0.02 * np.random.default_rng(0).uniform(-1.0, 1.0, (n, q))
    with LbmSolver(prob) as s:
        s.set_populations(f)
        back = s.populations()
    assert np.max(np.abs(back - f)) <= 2.0**-24
