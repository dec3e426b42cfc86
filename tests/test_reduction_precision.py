"""The admission sums are compensated: terms that cancel leave the small ones."""
import pytest

from implexity_b200 import ContractError, LbmSolver, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 4])
def test_mass_keeps_small_terms_beside_cancelling_large_ones(gpu_lib, steps):
    """rho - 1 of three cells: 2^40, 2^-24, -2^40.  Plain FP64 drops 2^-24
    beside 2^40 (2^-24 < 2^-53 2^40); two-sum keeps it, whichever cells share a
    warp.  One step is a launch of its own, four are a run.  (Such a state is
    not admitted; its record is there all the same.)"""
    shape = (9, 8, 7)
    prob = workloads.channel_problem(shape=shape, steps=steps, ports=False)
    with LbmSolver(prob) as s:
        s.set_design(workloads.uniform_design(shape, 1))
        s.forward(1)
        rest = s.populations()  # f = w: no port drives the fluid
        for large, small, minus in ((40, 41, 42), (3, 200, 450), (31, 32, 33)):
            masses = []
            for term in (0.0, 2.0**-24):
                f = rest.copy()
                f[large, 0] += 2.0**40
                f[small, 0] += term
                f[minus, 0] -= 2.0**40
                s.set_populations(f)
                with pytest.raises(ContractError):
                    s.advance(steps)
                masses.append(s.trajectory()["mass"][0])
            assert masses[1] - masses[0] == 2.0**-24, (large, small, minus, masses)
