"""The one-launch block PCG of the reduced system at the sizes where its launch changes (one CTA, 8 /
16 / 32 block rows per CTA, more rows than the chip has warps), with an initial guess, an iteration
limit, single precision and every precision mode, and after a failed factorisation.

Tolerances are those of the other solve tests: 1e-6 (FP64) and 1e-4 (FP32) relative against the
oracle, which solves to 1e-10."""
import numpy as np
import pytest
import torch

from gpu_util import dev, host
from plamatrix_b200 import schur as SC
from plamatrix_b200 import workloads as W

pytestmark = pytest.mark.gpu

SMS = 148


def _equations(prob, dtype=np.float64):
    ne = SC.DeviceNormalEquations(prob["P"], prob["L"], 6, 3, dtype)
    ne.accumulate_observations(dev(prob["obs_primary"]), dev(prob["obs_eliminated"]), dev(prob["jp"].astype(dtype)),
                               dev(prob["jl"].astype(dtype)), dev(prob["residual"].astype(dtype)), prob["huber_delta"])
    return ne


def _problem(P, seed=3):
    # two CTAs' worth of structure is enough: 15 points per camera, four views from a window of ten
    return W.bundle_problem(P, max(60, 15 * P), per_eliminated=min(4, P), window=min(P, 10), seed=seed)


@pytest.mark.parametrize("P", [1, 2, 7, 32, 33, 8 * SMS, 8 * SMS + 1, 16 * SMS + 1, 32 * SMS, 32 * SMS + 1])
def test_block_row_counts(checkers, P):
    prob = _problem(P)
    orc = checkers.normal_equations_from_observations(prob)
    dp_ref, dl_ref, rep_ref = orc.solve(1e-3, relative_tolerance=1e-10, max_iterations=300)
    ne = _equations(prob)
    for precision in ("native", "mixed", "mixed_fp32_assembly"):
        opts = SC.SchurComplementSolverOptions(max_iterations=300, relative_tolerance=1e-10, precision=precision)
        dp, dl, rep = SC.solve_damped_schur_complement(ne, 1e-3, opts)
        assert rep["converged"] and rep_ref["converged"], rep["message"]
        assert rep["true_relative_residual"] <= 1.5e-10
        if precision == "native":
            assert abs(rep["iterations"] - rep_ref["iterations"]) <= 1
        assert np.linalg.norm(host(dp) - dp_ref) <= 1e-6 * np.linalg.norm(dp_ref)
        assert np.linalg.norm(host(dl) - dl_ref) <= 1e-6 * np.linalg.norm(dl_ref)


@pytest.mark.parametrize("P", [20, 700])
def test_single_precision(checkers, P):
    prob = _problem(P, seed=5)
    orc = checkers.normal_equations_from_observations(prob)
    dp_ref, dl_ref, _ = orc.solve(1e-3, relative_tolerance=1e-10, max_iterations=300)
    opts = SC.SchurComplementSolverOptions(max_iterations=300, relative_tolerance=1e-6)
    dp, dl, rep = SC.solve_damped_schur_complement(_equations(prob, np.float32), 1e-3, opts)
    assert rep["converged"] and rep["true_relative_residual"] == -1.0
    assert np.linalg.norm(host(dp) - dp_ref) <= 1e-4 * np.linalg.norm(dp_ref)
    assert np.linalg.norm(host(dl) - dl_ref) <= 1e-4 * np.linalg.norm(dl_ref)


@pytest.mark.parametrize("P", [20, 700])
def test_initial_guess_and_iteration_limit(P):
    """k iterations and then the rest from there reach the same step; a solve cut short keeps its
    iterate, reports the limit and leaves the eliminated step zero."""
    ne = _equations(_problem(P, seed=7))
    full = SC.SchurComplementSolverOptions(max_iterations=300, relative_tolerance=1e-10)
    dp_ref, dl_ref, _ = SC.solve_damped_schur_complement(ne, 1e-3, full)
    dp = torch.zeros(6 * P, dtype=torch.float64, device="cuda")
    short = SC.SchurComplementSolverOptions(max_iterations=2, relative_tolerance=1e-10)
    _, dl, rep = SC.solve_damped_schur_complement(ne, 1e-3, short, primary_step=dp)
    assert not rep["converged"] and rep["iterations"] == 2 and rep["message"] == "PCG iteration limit reached"
    assert dp.any() and not dl.any() and rep["true_relative_residual"] == -1.0
    again = SC.SchurComplementSolverOptions(max_iterations=300, relative_tolerance=0.0, use_initial_guess=True,
                                            absolute_tolerance=1e-10 * rep["initial_residual_norm"])
    _, dl, rep = SC.solve_damped_schur_complement(ne, 1e-3, again, primary_step=dp)
    assert rep["converged"] and rep["true_relative_residual"] <= 1.5e-10
    assert torch.linalg.norm(dp - dp_ref) <= 1e-8 * torch.linalg.norm(dp_ref)
    assert torch.linalg.norm(dl - dl_ref) <= 1e-8 * torch.linalg.norm(dl_ref)
    # the exact guess takes no iteration and stays as it is
    kept = dp.clone()
    _, _, rep = SC.solve_damped_schur_complement(ne, 1e-3, again, primary_step=dp)
    assert rep["converged"] and rep["iterations"] == 0 and torch.equal(dp, kept)


def test_failed_factorisation_leaves_the_steps_zero():
    """Nothing is solved behind an eliminated block that is not positive definite."""
    prob = _problem(40, seed=9)
    ne = _equations(prob)
    state = ne.download()
    state["eliminated_diagonal"][17] = -np.eye(3)
    bad = SC.DeviceNormalEquations(prob["P"], prob["L"], 6, 3)
    bad.upload(state)
    dp, dl, rep = SC.solve_damped_schur_complement(bad, 1e-3)
    assert not rep["converged"] and rep["message"] == "eliminated block is not positive definite"
    assert not dp.any() and not dl.any()
