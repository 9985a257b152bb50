"""The FP64 back-substitution and matrix-free product where their 32-block runs end: block counts
around a warp, blocks without and with many crosses, a step vector off a 16-byte boundary; the
default assembly shapes on both sides of their rule; and the block-Jacobi inverses.

Tolerances: the steps as in the other solve tests (1e-6 relative against the oracle, solved to 1e-10);
reduced systems of different shapes within 1e-12 of the largest entry; inverses of the FP64 diagonal
blocks within 1e-10 relative (condition numbers below 1e5)."""
import numpy as np
import pytest
import torch

from gpu_util import dev, host
from plamatrix_b200 import schur as SC
from plamatrix_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _problem(P, counts, seed):
    """Eliminated block l seen by counts[l] distinct primaries."""
    rng = np.random.default_rng(seed)
    obs_l = np.repeat(np.arange(len(counts)), counts)
    obs_p = np.concatenate([rng.permutation(P)[:k] for k in counts]) if len(obs_l) else np.zeros(0, np.int64)
    n = len(obs_l)
    order = rng.permutation(n)
    return {"P": P, "L": len(counts), "bp": 6, "bl": 3, "m": 2, "huber_delta": 1.0,
            "obs_primary": np.ascontiguousarray(obs_p[order].astype(np.int64)),
            "obs_eliminated": np.ascontiguousarray(obs_l[order].astype(np.int64)),
            "jp": rng.standard_normal((n, 2, 6)), "jl": rng.standard_normal((n, 2, 3)),
            "residual": rng.standard_normal((n, 2))}


def _equations(prob):
    ne = SC.DeviceNormalEquations(prob["P"], prob["L"], 6, 3)
    ne.accumulate_observations(dev(prob["obs_primary"]), dev(prob["obs_eliminated"]), dev(prob["jp"]), dev(prob["jl"]),
                               dev(prob["residual"]), prob["huber_delta"])
    return ne


@pytest.mark.parametrize("L", [31, 32, 33, 127, 129, 500])
@pytest.mark.parametrize("kind", ["even", "uneven"])
@pytest.mark.parametrize("offset", [0, 1])
def test_runs_of_eliminated_blocks(checkers, L, kind, offset):
    P = 80
    rng = np.random.default_rng(L)
    counts = np.full(L, 16) if kind == "even" else rng.integers(3, 30, L)
    if kind == "uneven":
        counts[[0, L // 2, L - 1]] = [70, 64, 65]  # longer than one step of 32
    prob = _problem(P, counts, L)
    orc = checkers.normal_equations_from_observations(prob)
    dp_ref, dl_ref, _ = orc.solve(1e-3, relative_tolerance=1e-10, max_iterations=400)
    ne = _equations(prob)
    for precision in ("native", "mixed_fp32_assembly"):
        opts = SC.SchurComplementSolverOptions(max_iterations=400, relative_tolerance=1e-10, precision=precision)
        step = torch.zeros(6 * P + offset, dtype=torch.float64, device="cuda")[offset:]
        dp, dl, rep = SC.solve_damped_schur_complement(ne, 1e-3, opts, primary_step=step)
        assert rep["converged"], rep["message"]
        assert np.linalg.norm(host(dp) - dp_ref) <= 1e-6 * np.linalg.norm(dp_ref)
        assert np.linalg.norm(host(dl) - dl_ref) <= 1e-6 * np.linalg.norm(dl_ref)


def test_blocks_without_crosses():
    """An unobserved eliminated block in the uploaded state: only its own gradient moves it."""
    prob = _problem(40, np.full(200, 12), 5)
    state = _equations(prob).download()
    offs = state["adjacency_offsets"]
    gone = [0, 31, 32, 100, 199]
    keep = np.ones(len(state["cross_primary"]), bool)
    for l in gone:
        keep[offs[l]:offs[l + 1]] = False
    counts = np.diff(offs)
    counts[gone] = 0
    state["adjacency_offsets"] = np.concatenate([[0], np.cumsum(counts)])
    state["cross_primary"], state["cross_values"] = state["cross_primary"][keep], state["cross_values"][keep]
    ne = SC.DeviceNormalEquations(40, 200, 6, 3)
    ne.upload(state)
    opts = SC.SchurComplementSolverOptions(max_iterations=400, relative_tolerance=1e-10)
    _, dl, rep = SC.solve_damped_schur_complement(ne, 1e-3, opts)
    assert rep["converged"], rep["message"]
    for l in gone:
        H = state["eliminated_diagonal"][l].copy()
        H[np.diag_indices(3)] *= 1.0 + 1e-3
        want = np.linalg.solve(H, -state["eliminated_gradient"][l])
        assert np.allclose(host(dl).reshape(-1, 3)[l], want, rtol=1e-10, atol=0)


@pytest.mark.parametrize("P, L, k", [(30, 1500, 4), (120, 3000, 4), (120, 40000, 6), (400, 30000, 4), (420, 250000, 12)])
@pytest.mark.parametrize("precision", ["native", "mixed_fp32_assembly"])
def test_default_shape_and_inverses(P, L, k, precision):
    """Few and many pairs per block, few and many blocks: the default's reduced system is that of a
    pinned shape, and the preconditioner holds the inverses of its diagonal blocks."""
    prob = W.bundle_problem_device(P, L, per_eliminated=k, seed=P)
    ne = SC.DeviceNormalEquations(P, L, 6, 3)
    ne.accumulate_observations(*(prob[key] for key in ("obs_primary", "obs_eliminated", "jp", "jl", "residual")), 1.0)
    opts = SC.SchurComplementSolverOptions(max_iterations=300, relative_tolerance=1e-8, precision=precision)
    systems = []
    for pinned in (None, 1):
        ws = SC.SchurComplementSolverWorkspace()
        assert ws.assembly_shape == 0
        if pinned is not None:
            ws.assembly_shape = pinned
        _, _, rep = SC.solve_damped_schur_complement(ne, 1e-3, opts, ws)
        assert rep["converged"], rep["message"]
        systems.append(ws.export())
    a, b = (s["values"] for s in systems)
    assert (a - b).abs().max() <= (1e-12 if precision == "native" else 1e-6) * b.abs().max()
    if precision == "native":
        s = systems[0]
        dense = torch.sparse_csr_tensor(s["row_offsets"], s["col_indices"], s["values"], (6 * P, 6 * P)).to_dense()
        blocks = torch.stack([dense[6 * p:6 * p + 6, 6 * p:6 * p + 6] for p in range(P)])
        inverse = torch.linalg.inv(blocks)
        got = s["preconditioner"].view(P, 6, 6)
        assert ((got - inverse).flatten(1).norm(dim=1) <= 1e-10 * inverse.flatten(1).norm(dim=1)).all()


def test_batched_graph_follows_the_batch():
    """One workspace over batches of other sizes, options and step vectors: its kept iteration graph
    gives the bits of a fresh workspace every time."""
    batches = [[(12, 700), (30, 900)], [(40, 2000), (9, 500), (25, 800)], [(12, 700), (30, 900)]]
    shared = SC.SchurComplementSolverWorkspace()
    for k, sizes in enumerate(batches):
        probs = [W.bundle_problem(P, L, per_eliminated=4, seed=10 * k + i) for i, (P, L) in enumerate(sizes)]
        union = SC.pack_observation_systems(probs)
        ne = _equations(union)
        for precision, tol in (("native", 1e-8), ("native", 1e-6), ("mixed", 1e-8), ("native", 1e-8)):
            opts = SC.SchurComplementSolverOptions(max_iterations=200, relative_tolerance=tol, precision=precision)
            hold = torch.empty(6 * union["P"] + 64, dtype=torch.float64, device="cuda")  # moves the next step vector
            got = SC.solve_batched_schur_complement(ne, 1e-3, union["primary_offsets"], opts, shared)
            want = SC.solve_batched_schur_complement(ne, 1e-3, union["primary_offsets"], opts)
            assert got[2]["converged"] and want[2]["converged"]
            assert [s["iterations"] for s in got[3]] == [s["iterations"] for s in want[3]]
            assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
            del hold
