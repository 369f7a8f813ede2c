"""The solver's lambda is a warm start with the library's choice of PCG kernel (pcg_cluster_size 0): one that meets the
tolerance is returned as it came, after no iteration; from any other the multipliers are the system's solution."""
import importlib

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("schur_fp64,graph,mode", [(1, 0, 0), (1, 1, 0), (0, 1, 0), (1, 1, 1)])
@pytest.mark.parametrize("Ns", [[2], [32], [64, 5, 33], [300], [20] * 150])
def test_the_given_lambda_is_where_the_solve_starts(problem_mod, Ns, schur_fp64, graph, mode):
    """One SQP iteration from the multipliers of a first one.  A float32 lambda leaves a residual of up to 6e-8 |S| |lambda| /
    |gamma|, far above usable tolerances, so the start that has to be kept is given a tolerance above it (1e3), and in
    another run no iteration at all.  A start off by the size of the solution leads to the solution from 0 within the
    bound of the kernel's tests, 1e-6 of the largest component (the same rows, so FP32 ones too), and so does one that
    is off at a single knot only; one that is not finite ends the solve."""
    import torch
    gpt = importlib.import_module("gpu-pcg-tracking_b200")
    B = len(Ns)
    p = problem_mod.make_batch(Ns, seed0=7)
    dev = lambda k: torch.as_tensor(p[k], device="cuda")  # noqa: E731
    goal = dev("goal")

    def solve(lam, tol, most):
        xu = dev("xu")
        sv = gpt.Solver(max_knot_points=max(Ns), max_batch=B, sqp_max_iter=1, pcg_max_iter=most, pcg_exit_tol=tol,
                        pcg_exit_mode=mode, schur_fp64=schur_fp64, sqp_graph=graph, timestep=0.01, integrator=1, qd_cost=1e-2, r_cost=1e-4)
        lam = torch.as_tensor(lam, device="cuda", dtype=torch.float32).clone()
        _, stats = sv.sqp_solve_batched(Ns, goal, lam, xu, [1e-3] * B)
        sv.close()
        return lam.cpu().numpy(), [s["pcg_iters_total"] for s in stats]

    first, its = solve(np.zeros(14 * sum(Ns)), 1e-6, 20)
    assert min(its) >= 1
    kept, its = solve(first, 1e3, 20)
    assert its == [0] * B and np.array_equal(kept, first)
    kept, its = solve(first, 1e-6, 0)
    assert its == [0] * B and np.array_equal(kept, first)
    rng = np.random.default_rng(len(Ns))
    off = np.concatenate([[0], np.cumsum(Ns)]) * 14
    starts = [(first + rng.normal(0, np.abs(first).max(), first.shape), 1e-9)]
    if mode == 0:
        last = first.copy()
        for e in off[1:]:
            last[e - 14:e] *= 1e9
        starts.append((last, 1e3))
    for start, tol in starts:
        other, its = solve(start, tol, 20)
        assert min(its) >= 1
        for b in range(B):
            want = first[off[b]:off[b + 1]]
            assert np.abs(other[off[b]:off[b + 1]] - want).max() <= 1e-6 * np.abs(want).max(), b
    first[-1] = np.nan
    with pytest.raises(gpt.GptError):
        solve(first, 1e-6, 20)


@pytest.mark.gpu
@pytest.mark.parametrize("N", [5, 33, 129, 300])
@pytest.mark.parametrize("at", [0.3, 0.5, 0.99])
def test_a_system_that_is_not_finite_leaves_the_start(N, at):
    """gpt_pcg reports a NaN in S, wherever it is, and returns the lambda that it was given."""
    import torch
    gpt = importlib.import_module("gpu-pcg-tracking_b200")
    S = torch.zeros(N, 3, 14, 14, device="cuda")
    S[:, 1] = -2.0 * torch.eye(14, device="cuda")
    S[int(at * N), 1] = float("nan")
    gam, lam = torch.ones(14 * N, device="cuda"), torch.arange(14.0 * N, device="cuda")
    lam64 = torch.zeros(14 * N, device="cuda", dtype=torch.float64)
    want = lam.clone()
    sv = gpt.Solver(max_knot_points=N, timestep=0.01, integrator=1, qd_cost=1e-2, r_cost=1e-4)
    with pytest.raises(gpt.GptError):
        sv.pcg(N, S.reshape(-1), torch.zeros_like(S).reshape(-1), gam, lam, 20, 1e-6, 0, lam64=lam64)
    assert torch.equal(lam, want) and torch.equal(lam64, want.double())
    sv.close()
