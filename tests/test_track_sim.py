"""The plant simulation of a control update, after the solve (fewer than three whole plant steps) or beside it: the state
after one update is gpt_simulate's over the trajectory's controls, bit for bit (the same steps)."""
import importlib

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("period_us", [100.0, 400.0, 500.0, 600.0, 2000.0])
@pytest.mark.parametrize("graph", [0, 1])
def test_one_updates_plant_state(problem_mod, period_us, graph):
    import torch
    gpt = importlib.import_module("gpu-pcg-tracking_b200")
    Ns, S = [8, 5, 8], 12
    cfg = dict(timestep=0.01, integrator=1, qd_cost=1e-2, r_cost=1e-4)
    rng = np.random.default_rng(3)
    rows = rng.normal(0, 0.5, (3, S, 21)).astype(np.float32)
    goal = rng.normal(0, 0.5, (3, S, 6)).astype(np.float32)
    xs0 = rng.normal(0, 0.5, (3, 14)).astype(np.float32)
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a).reshape(-1), device="cuda")  # noqa: E731
    sv = gpt.Solver(max_knot_points=8, max_batch=3, sqp_max_iter=2, sqp_graph=graph, **cfg)
    xs = dev(xs0)
    sv.track_batched(Ns, [S] * 3, dev(goal), dev(rows), xs,
                     gpt.default_track_config(sim_period_us=period_us, max_control_updates=1))
    got = xs.cpu().numpy().reshape(3, 14)
    for b, n in enumerate(Ns):
        want = dev(xs0[b])
        sv.simulate(n, want, dev(rows[b].reshape(-1)[:21 * n - 7]), 0.0, period_us)
        assert np.array_equal(got[b], want.cpu().numpy()), b
    assert not np.array_equal(got, xs0)
    sv.close()
