"""KKT formation with one knot per lane, which batches of 9216 knots and more take (horizons up to 128), against the
half-warp form of the single-trajectory entry point, through the FP64 solution of each one's system.

Tolerance: the two forms differ by FP32 rounding, a few ulp of the largest entry of each block.  The reference system's
blocks are therefore perturbed at random by 5e-7 (8 ulp) of that, three times, and the multipliers may differ by 4 times
the largest change this makes."""
import importlib

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("pattern,integrator,ref_terminal,short", [
    ([2, 3, 31, 32, 33, 128], 1, 1, 0), ([127, 5, 64, 17], 0, 1, 0), ([128, 2, 65], 1, 0, 0), ([30, 97], 0, 0, 0),
    ([48], 1, 1, 0), ([2, 3, 31, 32, 33, 128], 1, 1, 1)])
def test_lane_form_gives_the_step(problem_mod, pattern, integrator, ref_terminal, short):
    """One SQP iteration of a batch just above 9216 knots (short: just below, the half-warp form) against the FP64
    solution of each horizon's system; parts of the batch (graph branches) give the same bits."""
    import torch
    gpt = importlib.import_module("gpu-pcg-tracking_b200")
    check = importlib.import_module("gpu-pcg-tracking_b200.fp64check")
    cfg = dict(timestep=0.01, integrator=integrator, qd_cost=1e-2, r_cost=1e-4, ref_terminal=ref_terminal)
    Ns = []
    while sum(Ns) < 9216:
        Ns.append(pattern[len(Ns) % len(pattern)])
    if short:
        Ns.pop()
    B = len(Ns)
    probs = [problem_mod.make_problem(n, 500 + i, dt=0.01) for i, n in enumerate(pattern)]
    pad = np.zeros(7, np.float32)
    dev = lambda key, tail: torch.as_tensor(  # noqa: E731
        np.concatenate([np.concatenate([probs[i % len(pattern)][key], tail]) for i in range(B)]), device="cuda")
    goal, off = dev("goal", pad[:0]), np.concatenate([[0], np.cumsum(Ns)])
    got = []
    for branches in (1, 3):
        sv = gpt.Solver(max_knot_points=max(Ns), max_batch=B, sqp_max_iter=1, pcg_max_iter=20, pcg_exit_tol=1e-9,
                        sqp_graph=branches, **cfg)
        lam, xu = dev("lam", pad[:0]), dev("xu", pad)
        sv.sqp_solve_batched(Ns, goal, lam, xu, [1e-3] * B)
        got.append((lam.cpu().numpy(), xu.cpu().numpy()))
        if branches == 1:
            lam1, xu1 = dev("lam", pad[:0]), dev("xu", pad)
            _, _, tr = sv.sqp_solve_batched_trace(Ns, goal, lam1, xu1, [1e-3] * B, 1)
            lam_step = tr["lam"][0].cpu().numpy()
        sv.close()
    assert all(np.array_equal(a, b) for a, b in zip(*got))
    rng = np.random.default_rng(len(pattern))
    one = gpt.Solver(max_knot_points=max(Ns), **cfg)
    for i, n in enumerate(pattern):
        z = lambda m: torch.zeros(m, device="cuda")  # noqa: E731
        G, Cm, g, c = z(245 * n - 49), z(294 * (n - 1)), z(21 * n - 7), z(14 * n)
        d = {k: torch.as_tensor(v, device="cuda") for k, v in probs[i].items()}
        one.form_kkt(n, d["xu"], d["goal"], d["xs"], G, Cm, g, c)
        G, Cm, g, c = (t.cpu().numpy().astype(np.float64) for t in (G, Cm, g, c))
        want, _ = check.solve_step(n, 1e-3, G, Cm, g, c)
        # (c = x - f is a difference: its rounding is that of x)
        x = max(1.0, np.abs(probs[i]["xu"]).max())
        ulp = lambda a, m: a + 5e-7 * m * rng.uniform(-1, 1, a.shape)  # noqa: E731
        tol = 4 * max(check.rel_err(check.solve_step(n, 1e-3, G, ulp(Cm, np.abs(Cm).max()), ulp(g, np.abs(g).max()),
                                                     ulp(c, x))[0], want) for _ in range(3))
        for b in {i, len(pattern) * ((B - 1 - i) // len(pattern)) + i}:  # its first and last instance
            assert check.rel_err(lam_step[14 * off[b]:14 * off[b + 1]], want) <= tol, (n, b, tol)
    one.close()
