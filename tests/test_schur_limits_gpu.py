"""Schur solves at the limits of the problem's shape."""
import numpy as np
import pytest
import torch

from gpu_util import dev, host
from plamatrix_b200 import schur as SC
from plamatrix_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [1, 32, 70])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_no_primary_blocks(L, dtype):
    """P = 0: every eliminated block is moved by its own damped gradient, and the empty primary step is
    neither read nor written.  The 3x3 systems have condition numbers below 100: 1e-12 (FP64) and 1e-4
    (FP32) relative are far above their rounding."""
    rng = np.random.default_rng(L)
    a = rng.standard_normal((L, 3, 3))
    hessian = (a @ a.transpose(0, 2, 1) + 3.0 * np.eye(3)).astype(dtype)
    gradient = rng.standard_normal((L, 3)).astype(dtype)
    ne = SC.DeviceNormalEquations(0, L, 6, 3, dtype)
    ne.upload({"primary_diagonal": np.zeros((0, 6, 6)), "eliminated_diagonal": hessian,
               "primary_gradient": np.zeros((0, 6)), "eliminated_gradient": gradient,
               "adjacency_offsets": np.zeros(L + 1, np.int64), "cross_primary": np.zeros(0, np.int64),
               "cross_values": np.zeros((0, 6, 3)), "primary_cross_row": np.zeros(0, np.int64),
               "primary_cross_col": np.zeros(0, np.int64), "primary_cross_values": np.zeros((0, 6, 6))})
    step = torch.empty(0, dtype=ne.tdtype, device="cuda")
    dp, dl, rep = SC.solve_damped_schur_complement(ne, 1e-3, primary_step=step)
    assert rep["converged"] and rep["iterations"] == 0 and dp.numel() == 0
    damped = hessian.astype(np.float64).copy()
    damped[:, range(3), range(3)] *= 1.0 + 1e-3
    want = np.linalg.solve(damped, -gradient.astype(np.float64)[:, :, None])[:, :, 0]
    tolerance = 1e-12 if dtype == np.float64 else 1e-4
    error = np.linalg.norm(host(dl).reshape(-1, 3) - want, axis=1)
    assert np.all(error <= tolerance * np.linalg.norm(want, axis=1))


@pytest.mark.parametrize("P", [9 * 148, 16 * 148, 17 * 148 + 3, 24 * 148, 24 * 148 + 1])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_block_rows_per_cta(checkers, P, dtype):
    """Rows of more than 32 blocks, 9 to 25 of them in each CTA of the one-launch PCG.  Tolerances of the other
    solve tests: 1e-6 (FP64) and 1e-4 (FP32) relative against the oracle, which solves to 1e-10."""
    prob = W.bundle_problem(P, 20 * P, per_eliminated=4, window=24, seed=P)
    ne = SC.DeviceNormalEquations(P, prob["L"], 6, 3, dtype)
    ne.accumulate_observations(dev(prob["obs_primary"]), dev(prob["obs_eliminated"]), dev(prob["jp"].astype(dtype)),
                               dev(prob["jl"].astype(dtype)), dev(prob["residual"].astype(dtype)), prob["huber_delta"])
    want_p, want_l, _ = checkers.normal_equations_from_observations(prob).solve(
        1e-3, relative_tolerance=1e-10, max_iterations=300)
    ws = SC.SchurComplementSolverWorkspace()
    tolerance = 1e-6 if dtype == np.float64 else 1e-4
    options = SC.SchurComplementSolverOptions(max_iterations=300,
                                              relative_tolerance=1e-10 if dtype == np.float64 else 1e-6)
    dp, dl, rep = SC.solve_damped_schur_complement(ne, 1e-3, options, ws)
    assert rep["converged"] and ws.dims()[2] > 32 * P
    assert np.linalg.norm(host(dp) - want_p) <= tolerance * np.linalg.norm(want_p)
    assert np.linalg.norm(host(dl) - want_l) <= tolerance * np.linalg.norm(want_l)


@pytest.mark.parametrize("P, L, k", [(30, 1500, 4), (120, 3000, 4), (120, 40000, 6), (420, 30000, 4), (420, 250000, 12)])
@pytest.mark.parametrize("precision", ["native", "mixed_fp32_assembly"])
def test_reported_shape_gives_the_bits(P, L, k, precision):
    """Few and many blocks, few and many pairs in each: the shape that a workspace reports after a solve, set in
    another one, assembles the same values."""
    prob = W.bundle_problem_device(P, L, per_eliminated=k, seed=P)
    ne = SC.DeviceNormalEquations(P, L, 6, 3)
    ne.accumulate_observations(*(prob[key] for key in ("obs_primary", "obs_eliminated", "jp", "jl", "residual")), 1.0)
    options = SC.SchurComplementSolverOptions(max_iterations=300, relative_tolerance=1e-8, precision=precision)
    free, pinned = SC.SchurComplementSolverWorkspace(), SC.SchurComplementSolverWorkspace()
    SC.solve_damped_schur_complement(ne, 1e-3, options, free)
    pinned.assembly_shape = free.assembly_shape
    SC.solve_damped_schur_complement(ne, 1e-3, options, pinned)
    assert torch.equal(free.export()["values"], pinned.export()["values"])
    # a shape that is chosen stays, whatever the rule says
    pinned.assembly_shape = 6
    SC.solve_damped_schur_complement(ne, 1e-3, options, pinned)
    assert pinned.assembly_shape == 6


@pytest.mark.parametrize("P", [40, 5000])
def test_closed_workspace_on_another_stream(P):
    """close() gives every buffer back: the workspace then serves another stream, with the bits of a fresh one.
    Both PCG forms (up to 4,736 block rows in one launch)."""
    prob = W.bundle_problem_device(P, 20 * P, per_eliminated=4, window=10, seed=P)
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    shared, steps = SC.SchurComplementSolverWorkspace(), []
    for stream in streams + [streams[0]]:
        with torch.cuda.stream(stream):
            ne = SC.DeviceNormalEquations(P, 20 * P, 6, 3)
            ne.accumulate_observations(*(prob[k] for k in ("obs_primary", "obs_eliminated", "jp", "jl", "residual")), 1.0)
            dp, dl, rep = SC.solve_damped_schur_complement(ne, 1e-3, None, shared)
            assert rep["converged"]
            steps.append((dp.clone(), dl.clone()))
        stream.synchronize()
        shared.close()
    assert all(torch.equal(a, b) for step in steps[1:] for a, b in zip(step, steps[0]))
