"""The tuner does not choose a grid for the KKT kernel that takes one knot per lane, which ignores it."""
import importlib

import pytest


@pytest.mark.gpu
def test_tuner_leaves_the_lane_forms_grid(problem_mod):
    import torch
    gpt = importlib.import_module("gpu-pcg-tracking_b200")
    Ns = [128] * 73  # 9344 knots: one knot per lane
    p = problem_mod.make_batch(Ns, seed0=11)
    sv = gpt.Solver(max_knot_points=128, max_batch=73, sqp_max_iter=2, timestep=0.01, integrator=1, qd_cost=1e-2,
                    r_cost=1e-4)
    sched = {}
    sv.autotune(Ns, *(torch.as_tensor(p[k], device="cuda") for k in ("goal", "lam", "xu")), [1e-3] * 73, schedule=sched)
    sv.close()
    assert sched["kkt"] == 16
