"""The KKT formation with one knot per lane by itself: every entry that a live instance owns is written, whatever its
neighbours in the block do, and agrees with the FP64 oracle.

Tolerances, as multiples of FP32 rounding (2^-24 = 6e-8): the blocks of C within 1e-4 of their largest entry (the bound of
the same dynamics tangents in test_grid); the position gradient J^T (p - goal) within 1e-5 (a product of at most 1.3 m of
lever and 3 terms of at most 2 m, each off by the kinematics' rounding of seven rotations, some 30 roundings, 2e-6); the
velocity and control gradients, one rounded product each, within 2e-7 of their value; the defects, differences of the state
and the dynamics' step, within 1e-6 of the largest state plus 1e-5 of the step's acceleration (test_grid's bound)."""
import ctypes
import importlib

import numpy as np
import pytest

from harness import build


@pytest.fixture(scope="module")
def stages(tmp_path_factory):
    return build(tmp_path_factory.mktemp("stages"))


def problems(problem_mod, pattern, seed):
    """One problem per horizon of the pattern, off the path and with controls."""
    out = []
    rng = np.random.default_rng(seed)
    for i, n in enumerate(pattern):
        p = problem_mod.make_problem(n, seed + i, dt=0.01)
        x = p["xu"]
        x += rng.normal(0, 0.02, x.shape).astype(np.float32)
        for k in range(n - 1):
            x[21 * k + 14:21 * k + 21] = rng.normal(0, 3, 7)
        p["xs"] = p["xs"] + np.float32(0.01)
        out.append(p)
    return out


def form(stages, Ns, active, b0, B, lane, cfg, xu, goal, xs):
    import torch
    K = sum(Ns)
    off = (ctypes.c_int * (len(Ns) + 1))(*np.concatenate([[0], np.cumsum(Ns)]).tolist())
    on = (ctypes.c_ubyte * len(Ns))(*active)
    C, g, c = (torch.full((n * K,), float("nan"), device="cuda") for n in (294, 21, 14))
    f, p = ctypes.c_float, lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    torch.cuda.synchronize()
    rc = stages.stage_kkt(len(Ns), off, on, b0, B, lane, f(cfg["dt"]), cfg["integrator"], f(cfg["qd_cost"]),
                          f(cfg["r_cost"]), cfg["ref_terminal"], p(xu), p(goal), p(xs), p(C), p(g), p(c))
    assert rc == 0
    return tuple(t.cpu().numpy().astype(np.float64) for t in (C, g, c))


# (horizons of the pattern, its repetitions, activity of the pattern or None for a random one, part of the batch)
CASES = [([97], 97, (1,), None),                                # 9409 = 147 x 64 + 1 knots: a last knot alone in a block
         ([97], 194, (1,), (97, 97)),                           # a part batch of that size
         ([65, 20, 43], 75, (1, 0, 0), None),                   # a last knot opens a block, the others have stopped
         ([65, 20, 43], 75, None, (1, 223)),
         ([2, 3, 31, 128, 33, 64], 40, None, None)]


@pytest.mark.gpu
@pytest.mark.parametrize("pattern,times,activity,part", CASES)
@pytest.mark.parametrize("integrator,ref_terminal", [(0, 0), (1, 0), (1, 1)])
def test_every_live_knot_is_formed(oracle, problem_mod, stages, pattern, times, activity, part, integrator, ref_terminal):
    import torch
    cfg = dict(dt=0.01, integrator=integrator, qd_cost=1e-2, r_cost=1e-4, ref_terminal=ref_terminal)
    par = oracle.make_params(**cfg)
    Ns = pattern * times
    rng = np.random.default_rng(times)
    active = list(activity) * times if activity else rng.integers(0, 2, len(Ns)).tolist()
    b0, B = part or (0, len(Ns))
    probs = problems(problem_mod, pattern, 900)
    pad = np.zeros(7, np.float32)
    dev = lambda key, tail: torch.as_tensor(  # noqa: E731
        np.concatenate([np.concatenate([p[key], tail]) for p in probs] * times), device="cuda")
    C, g, c = form(stages, Ns, active, b0, B, 1, cfg, dev("xu", pad), dev("goal", pad[:0]), dev("xs", pad[:0]))
    off = np.concatenate([[0], np.cumsum(Ns)])
    want = []
    for n, p in zip(pattern, probs):
        _, wC, wg, wc = oracle.form_kkt(par, n, p["xu"].astype(np.float64), p["goal"].astype(np.float64),
                                        p["xs"].astype(np.float64))
        x = np.append(p["xu"], pad).reshape(n, 21).astype(np.float64)
        qdd = np.abs([oracle.fd(r[:7], r[7:14], r[14:]) for r in x[:n - 1]]).max()
        want.append((wC.reshape(n - 1, 294), wg, wc,
                     1e-6 * max(1.0, np.abs(x).max()) + 1e-5 * cfg["dt"] * max(1.0, qdd)))
    for b, n in enumerate(Ns):
        k0, k1 = off[b], off[b + 1]
        gb, cb, Cb = g[21 * k0:21 * k1], c[14 * k0:14 * k1], C[294 * k0:294 * k1].reshape(n, 294)
        if not (active[b] and b0 <= b < b0 + B):
            assert np.isnan(gb).all() and np.isnan(cb).all() and np.isnan(Cb).all(), b
            continue
        wC, wg, wc, tol_c = want[b % len(pattern)]
        for blk in (slice(0, 98), slice(98, 196), slice(196, 294)):
            err = np.abs(Cb[:n - 1, blk] - wC[:, blk]).max(1)
            assert (err <= 1e-4 * np.abs(wC[:, blk]).max(1)).all(), (b, err.max())
        got, ref = np.append(gb[:21 * n - 7], np.zeros(7)).reshape(n, 21), np.append(wg, np.zeros(7)).reshape(n, 21)
        assert np.abs(got[:, :7] - ref[:, :7]).max() <= 1e-5, b
        assert (np.abs(got[:, 7:] - ref[:, 7:]) <= 2e-7 * np.abs(ref[:, 7:])).all(), b
        assert np.abs(cb - wc).max() <= tol_c, b


@pytest.mark.gpu
def test_batches_whose_last_knot_stands_alone(problem_mod):
    """97 instances of 97 knots with ref_terminal 0 on a handle whose workspace another solve has filled: the last one's
    multipliers are the FP64 solution of its system (tolerance as in test_kkt_lane: four times what 8 ulp of the blocks
    move it); two such batches as the branches of one give the bits of the whole."""
    import torch
    gpt = importlib.import_module("gpu-pcg-tracking_b200")
    check = importlib.import_module("gpu-pcg-tracking_b200.fp64check")
    n, cfg = 97, dict(timestep=0.01, integrator=1, qd_cost=1e-2, r_cost=1e-4, ref_terminal=0)
    probs, other = (problem_mod.make_batch([n] * 8, seed0=s) for s in (40, 80))
    tile = lambda p, B: {k: torch.as_tensor(  # noqa: E731
        np.resize(p[k], B * n * (len(p[k]) // (8 * n))), device="cuda") for k in ("xu", "goal", "lam")}

    def step(B, branches):
        sv = gpt.Solver(max_knot_points=n, max_batch=B, sqp_max_iter=1, pcg_max_iter=20, pcg_exit_tol=1e-9,
                        sqp_graph=branches, **cfg)
        o = tile(other, B)
        sv.sqp_solve_batched([n] * B, o["goal"], o["lam"], o["xu"], [1e-3] * B)
        p = tile(probs, B)
        sv.sqp_solve_batched([n] * B, p["goal"], p["lam"], p["xu"], [1e-3] * B)
        sv.close()
        return p["lam"].cpu().numpy(), p["xu"].cpu().numpy()

    lam, _ = step(97, 1)
    one = gpt.Solver(max_knot_points=n, **cfg)
    z = lambda m: torch.zeros(m, device="cuda")  # noqa: E731
    G, Cm, g, c = z(245 * n - 49), z(294 * (n - 1)), z(21 * n - 7), z(14 * n)
    xu, goal = (torch.as_tensor(probs[k][:w * n], device="cuda") for k, w in (("xu", 21), ("goal", 6)))
    one.form_kkt(n, xu, goal, xu[:14].clone(), G, Cm, g, c)
    one.close()
    G, Cm, g, c = (t.cpu().numpy().astype(np.float64) for t in (G, Cm, g, c))
    want, _ = check.solve_step(n, 1e-3, G, Cm, g, c)
    rng = np.random.default_rng(n)
    ulp = lambda a, m: a + 5e-7 * m * rng.uniform(-1, 1, a.shape)  # noqa: E731
    tol = 4 * max(check.rel_err(check.solve_step(n, 1e-3, G, ulp(Cm, np.abs(Cm).max()), ulp(g, np.abs(g).max()),
                                                 ulp(c, max(1.0, np.abs(probs["xu"]).max())))[0], want) for _ in range(3))
    for b in (0, 96):  # both hold problem 0
        assert check.rel_err(lam[14 * n * b:14 * n * (b + 1)], want) <= tol, (b, tol)
    assert all(np.array_equal(a, b) for a, b in zip(step(194, 1), step(194, 2)))
