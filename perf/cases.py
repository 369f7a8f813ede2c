"""The work this framework is used for, as cases that can be timed and compared.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) the inputs, on the GPU, and the handle a program keeps
    run(state)          one pass through the public entry points, and its outputs
    work(case)          the bytes and operations a pass cannot do without
    exact(case, seed)   the outputs in 64 bits, by plain torch (None where there is no such value)

A case's "do" names the entry point:

    solve    sqp_solve (one instance) or sqp_solve_batched: SQP iterations from a spline guess, as a
             controller or a trajectory optimiser calls it once per control step or per plan
    adjoint  sqp_adjoint: the backward pass of a solve (goal and cost-weight gradients)
    track    track_batched: a few control updates of the receding-horizon loop, or with "grad"
             track_batched_adjoint: the same with the weight gradients of every update accumulated
    stages   form_kkt, form_schur, pcg, compute_dz and ls_compute_merit, each on inputs of its own:
             a program that drives the linear algebra of one instance itself
    rows     forward_dynamics, forward_dynamics_gradient and end_effector_positions over many rows,
             as for the goals of a data set of trajectories and for a plant model

Horizons of a batch lie between "short" and "long" knots (equal: every instance has that length).
The problems are joint-space splines through random waypoints with the end-effector path of the spline
as the goal, started a little off the path: the distribution of this repository's benchmark.  "euler"
takes the reference's settings (explicit Euler, dt 1/64, cost weights 1e-4) instead of the benchmark's
(semi-implicit Euler, dt 0.01, weights 1e-2 and 1e-4).  "pcg" is pcg_cluster_size (0: the library's
choice; 64: the partitioned kernel, which the autotuner picks on this GPU) and "branches" is sqp_graph.
"""
import importlib
import math

import torch

NX, NS, NU = 21, 14, 7
BENCH = dict(timestep=0.01, integrator=1, qd_cost=1e-2, r_cost=1e-4)
EULER = dict(timestep=1.0 / 64.0, integrator=0, qd_cost=1e-4, r_cost=1e-4)
RHO = 1e-3


def listed():
    return [
        # one control step of one arm: the smallest call, all latency (horizon of the reference's sweep)
        dict(name="solve_1x32", do="solve", batch=1, short=32, long=32, iters=4, pcg=0, branches=1, tol=1e-5,
             euler=True),
        # the plain path of the benchmark: one arm, its headline horizon, the tuned kernel
        dict(name="solve_1x128", do="solve", batch=1, short=128, long=128, iters=4, pcg=64, branches=1, tol=1e-5,
             euler=False),
        # the longest horizon of the plain path, one knot short of the limit
        dict(name="solve_1x511", do="solve", batch=1, short=511, long=511, iters=2, pcg=64, branches=1, tol=1e-5,
             euler=False),
        # a handful of arms or of restarts planned together, ragged, nothing tuned
        dict(name="solve_11_ragged", do="solve", batch=11, short=20, long=77, iters=3, pcg=0, branches=1, tol=1e-4,
             euler=False),
        # the benchmark's mixed-horizon batch, a quarter of its size
        dict(name="solve_128_mixed", do="solve", batch=128, short=32, long=256, iters=3, pcg=64, branches=4, tol=1e-5,
             euler=False),
        # the headline batch at the iteration count of a control step
        dict(name="solve_512x128", do="solve", batch=512, short=128, long=128, iters=4, pcg=64, branches=4, tol=1e-5,
             euler=False),
        # training through the solver: the backward pass of the headline batch, and of a small ragged one
        dict(name="adjoint_512x128", do="adjoint", batch=512, short=128, long=128, pcg=0, branches=1, tol=1e-5,
             euler=False),
        dict(name="adjoint_24_ragged", do="adjoint", batch=24, short=30, long=70, pcg=64, branches=1, tol=1e-6,
             euler=False),
        # closed-loop evaluation of 64 arms; and tuning the cost weights over such runs
        dict(name="track_64x64", do="track", batch=64, short=64, long=64, rows=96, updates=4, iters=2, pcg=64,
             branches=1, tol=1e-5, grad=False, euler=False),
        dict(name="track_grad_33_ragged", do="track", batch=33, short=24, long=96, rows=120, updates=3, iters=2, pcg=64,
             branches=1, tol=1e-5, grad=True, euler=False),
        # the reference's kernels one by one
        dict(name="stages_100", do="stages", knots=100, tol=1e-5, pcg=0, euler=False),
        # rigid-body quantities of a data set of trajectories, an odd number of rows
        dict(name="rows_200003", do="rows", rows=200003),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    do = rng.choice(["solve", "solve", "solve", "adjoint", "track", "stages", "rows"])
    tol = rng.choice([1e-4, 1e-5, 1e-6])
    if do == "rows":
        return dict(do=do, rows=log_int(1, 300000))
    euler = rng.random() < 0.25
    if do == "stages":
        return dict(do=do, knots=log_int(2, 128), tol=tol, pcg=rng.choice([0, 32, 64]), euler=euler)
    batch = log_int(1, 512)
    long = min(512, max(2, log_int(8, 512)))
    while batch * long > 65536:
        long = max(8, long // 2 + rng.randrange(8))
        batch = min(batch, 65536 // long)
    short = long if rng.random() < 0.5 else max(2, long - rng.randrange(long))
    case = dict(do=do, batch=batch, short=short, long=long, pcg=rng.choice([0, 64, 64]), branches=rng.choice([1, 1, 4]),
                tol=tol, euler=euler)
    if do == "solve":
        case["iters"] = rng.choice([1, 2, 3])
    elif do == "track":
        case.update(rows=long + rng.randrange(60), updates=rng.choice([1, 2, 3]), iters=rng.choice([1, 2]),
                    grad=rng.random() < 0.5)
    # without a chosen kernel a long horizon is spread over CTAs that iterate, to the tolerance only; the
    # reference's weights at its longer time step are too badly conditioned for float32 data past this
    most = min(128 if case["pcg"] == 0 else 512, 96 if euler else 512)
    case["long"] = min(case["long"], most)
    case["short"] = min(case["short"], case["long"])
    if "rows" in case:
        case["rows"] = max(case["long"], min(case["rows"], case["long"] + 59))
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def horizons(case):
    lo, hi = case["short"], case["long"]
    return [hi if i == 0 else lo + (i * 7919 + 13) % (hi - lo + 1) for i in range(case["batch"])]


def settings(case):
    return EULER if case["euler"] else BENCH


LIMITS = [math.radians(d) for d in (170.0, 120.0, 170.0, 120.0, 170.0, 120.0, 175.0)]


def splines(count, steps, dt, gen, dev):
    """q, qd [count, steps, 7] of natural cubic splines through 5 waypoints over 2 s (held after it)."""
    f = dict(dtype=torch.float64, device=dev)
    W = (torch.rand(count, 5, 7, generator=gen, **f) - 0.5) * torch.tensor(LIMITS, **f)
    h = 0.5
    A = torch.eye(5, **f)
    for i in (1, 2, 3):
        A[i, i - 1], A[i, i], A[i, i + 1] = 1.0, 4.0, 1.0
    rhs = torch.zeros_like(W)
    rhs[:, 1:4] = 6.0 / h ** 2 * (W[:, 2:] - 2.0 * W[:, 1:4] + W[:, :3])
    M = torch.linalg.solve(A, rhs)  # second derivatives at the waypoints
    raw = torch.arange(steps, **f) * dt
    t = raw.clamp(max=2.0)
    i = (t / h).long().clamp(max=3)
    a, b = ((i + 1) * h - t)[None, :, None], (t - i * h)[None, :, None]
    M0, M1, W0, W1 = M[:, i], M[:, i + 1], W[:, i], W[:, i + 1]
    q = (M0 * a ** 3 + M1 * b ** 3) / (6 * h) + (W0 / h - M0 * h / 6) * a + (W1 / h - M1 * h / 6) * b
    qd = (M1 * b ** 2 - M0 * a ** 2) / (2 * h) + (W1 - W0) / h - (M1 - M0) * h / 6
    return q, qd * (raw <= 2.0).to(torch.float64)[None, :, None]


def generator(seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    return g, dev


def problems(case, seed, steps=None):
    """Padded problems: Ns, xu [B, L, 21] (initial guess), goal [B, L, 6], as the float32 values a call gets."""
    gen, dev = generator(seed)
    Ns = horizons(case) if "batch" in case else [case["knots"]]
    L = steps or max(Ns)
    q, qd = splines(len(Ns), L, settings(case)["timestep"], gen, dev)
    xu = torch.cat([q, qd, torch.zeros_like(q)], 2)
    xu[:, 0, :7] += 0.01 * torch.randn(len(Ns), 7, generator=gen, dtype=torch.float64, device=dev)
    xu[:, 0, 7:14] = 0.0
    return Ns, xu.float(), ee_pose(q).float(), gen, dev


def pack(v, Ns):
    """Rows of a padded batch as the knot-by-knot layout of the entry points."""
    return torch.cat([v[b, :n].reshape(-1) for b, n in enumerate(Ns)])


def stage_inputs(case, seed):
    """Inputs of each stage: the values in 64 bits of the stage before, rounded to what the stage takes."""
    Ns, xu, goal, gen, dev = problems(case, seed)
    N, cfg = Ns[0], settings(case)
    xs = xu[:, 0, :14] + 0.01 * torch.randn(1, 14, generator=gen, dtype=torch.float64, device=dev).float()
    xu[:, :, 14:] = 2.0 * torch.randn(1, N, 7, generator=gen, dtype=torch.float64, device=dev).float()
    xu[:, :, :14] += 0.003 * torch.randn(1, N, 14, generator=gen, dtype=torch.float64, device=dev).float()
    i = dict(xu=xu, goal=goal, xs=xs)
    k = kkt64(xu.double(), goal.double(), xs.double(), torch.tensor([N], device=dev), cfg, weights(cfg, 1, dev))
    i.update({n: k[n].float() for n in ("Q", "q", "r", "A", "B", "c")}, R=cfg["r_cost"])
    s = schur64(k32(i, N, dev), RHO)
    i.update({n: s[n].float() for n in ("left", "diag", "gamma")})
    i["pinv"] = (-torch.linalg.inv(-s["diag"])).float()
    i.update(Qi=s["Qi"], Ri=s["Ri"])
    i["lam"] = solve64(i["left"].double(), i["diag"].double(), i["gamma"].double())
    i["dz"] = dz64(k32(i, N, dev), s["Qi"], s["Ri"], i["lam"]).float()
    return N, cfg, i, dev


def k32(i, N, dev):
    """The float32 KKT blocks of the stages as doubles."""
    k = {n: i[n].double() for n in ("Q", "q", "r", "A", "B", "c")}
    k["R"] = torch.eye(7, dtype=torch.float64, device=dev).expand(1, N, 7, 7) * float(torch.tensor(i["R"]).float())
    return k


def flat(parts, N, last):
    """Knot-interleaved column-major blocks of one instance, the last knot's trailing `last` values dropped."""
    rows = torch.cat([p[0].transpose(-1, -2).reshape(N, -1) if p.dim() == 4 else p[0] for p in parts], 1).reshape(-1)
    return rows[:rows.numel() - last].contiguous()


def three(left, diag):
    """Block rows (left, diagonal, right = the next row's left transposed), column-major."""
    right = torch.zeros_like(left)
    right[:, :-1] = left[:, 1:].transpose(-1, -2)
    return torch.stack([left, diag, right], 2)[0].transpose(-1, -2).reshape(-1).contiguous()


def prepare(case, seed):
    gpt = importlib.import_module("gpu-pcg-tracking_b200")
    if case["do"] == "rows":
        gen, dev = generator(seed)
        n = case["rows"]
        lim = torch.tensor(LIMITS, device=dev)
        x = torch.cat([(torch.rand(n, 7, generator=gen, device=dev) * 2 - 1) * lim,
                       torch.randn(n, 7, generator=gen, device=dev), 10 * torch.randn(n, 7, generator=gen, device=dev)], 1)
        return dict(case=case, gpt=gpt, x=x.contiguous())
    if case["do"] == "stages":
        N, cfg, i, dev = stage_inputs(case, seed)
        sv = gpt.Solver(max_knot_points=N, pcg_max_iter=1000, pcg_exit_tol=case["tol"], pcg_cluster_size=case["pcg"],
                        **cfg)
        R = torch.eye(7, device=dev).expand(1, N, 7, 7) * i["R"]
        f = lambda n, t=torch.float32: torch.zeros(n, dtype=t, device=dev)  # noqa: E731
        zero = torch.zeros(1, N, 14, 14, device=dev)
        s = dict(case=case, sv=sv, N=N, xu=pack(i["xu"], [N])[:21 * N - 7].contiguous(), goal=pack(i["goal"], [N]),
                 xs=i["xs"][0].contiguous(), G=flat([i["Q"], R], N, 49), C=flat([i["A"], i["B"]], N, 294),
                 g=flat([i["q"], i["r"]], N, 7), c=pack(i["c"], [N]), S=three(i["left"], i["diag"]),
                 P=three(zero, i["pinv"]), gamma=pack(i["gamma"], [N]), Gi=flat([i["Qi"], i["Ri"]], N, 49).float(),
                 Gi64=flat([i["Qi"], i["Ri"]], N, 49), lam32=pack(i["lam"], [N]).float(), lam64=pack(i["lam"], [N]),
                 dz=pack(i["dz"], [N])[:21 * N - 7].contiguous())
        s["out"] = dict(G=f(245 * N - 49), C=f(294 * (N - 1)), g=f(21 * N - 7), c=f(14 * N), S=f(588 * N), Pinv=f(588 * N),
                        gamma=f(14 * N), Ginv=f(245 * N - 49), lam=f(14 * N), lam64=f(14 * N, torch.float64),
                        dz=f(21 * N - 7), merits=f(8))
        return s
    cfg = settings(case)
    track = case["do"] == "track"
    if track:
        Ns, xu, goal, gen, dev = problems(case, seed, case["rows"])
        rows = [case["rows"]] * len(Ns)
    else:
        Ns, xu, goal, gen, dev = problems(case, seed)
        rows = Ns
    sv = gpt.Solver(max_knot_points=max(Ns), max_batch=len(Ns), sqp_max_iter=case.get("iters", 1), pcg_max_iter=1000,
                    pcg_exit_tol=case["tol"], pcg_cluster_size=case["pcg"], sqp_graph=case["branches"], **cfg)
    xs = xu[:, 0, :14].contiguous()
    s = dict(case=case, sv=sv, Ns=Ns, rows=rows, goal=pack(goal, rows), xu0=pack(xu, rows), xs0=xs.reshape(-1))
    if track:
        s["tc"] = gpt.default_track_config(sim_period_us=1e6 * cfg["timestep"], max_control_updates=case["updates"])
        s["xs"] = torch.empty_like(s["xs0"])
        s["errors"] = torch.zeros(sum(rows), device=dev)
        return s
    T = sum(Ns)
    s["rho"] = [RHO] * len(Ns)
    if case["do"] == "adjoint":
        s["grad"] = adjoint_loss(T, gen, dev)
        s["xun"] = torch.zeros(21 * T, device=dev)
    else:
        s["lam0"] = torch.zeros(14 * T, device=dev)
        s["xu"], s["lam"] = torch.empty_like(s["xu0"]), torch.empty_like(s["lam0"])
    return s


def adjoint_loss(T, gen, dev):
    return torch.randn(21 * T, generator=gen, dtype=torch.float64, device=dev).float()


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(s):
    case = s["case"]
    do = case["do"]
    if do == "rows":
        gpt, x = s["gpt"], s["x"]
        qdd, df = gpt.forward_dynamics_gradient(x)
        return dict(pose=gpt.end_effector_positions(x, 21), fd=gpt.forward_dynamics(x), qdd=qdd, df=df)
    sv = s["sv"]
    if do == "stages":
        N, o = s["N"], s["out"]
        sv.form_kkt(N, s["xu"], s["goal"], s["xs"], o["G"], o["C"], o["g"], o["c"])
        sv.form_schur(N, RHO, s["G"], s["C"], s["g"], s["c"], o["S"], o["Pinv"], o["gamma"], o["Ginv"])
        o["lam"].zero_()
        sv.pcg(N, s["S"], s["P"], s["gamma"], o["lam"], 1000, case["tol"], 0, o["lam64"])
        sv.compute_dz(N, s["Gi"], s["C"], s["g"], s["lam32"], o["dz"], s["lam64"], s["Gi64"])
        sv.ls_compute_merit(N, s["xs"], s["xu"], s["goal"], s["dz"], o["merits"])
        return o
    if do == "adjoint":
        out = sv.sqp_adjoint(s["Ns"], s["goal"], s["xs0"], s["xu0"], s["rho"], s["grad"], s["xun"])
        return dict(out, xu_next=s["xun"])
    if do == "track":
        s["xs"].copy_(s["xs0"])
        call = sv.track_batched_adjoint if case["grad"] else sv.track_batched
        got = call(s["Ns"], s["rows"], s["goal"], s["xu0"], s["xs"], s["tc"], s["errors"])
        out = dict(errors=got[0], xs=s["xs"])
        if case["grad"]:
            out.update(weight_grad=got[2], loss=got[3])
        return out
    s["xu"].copy_(s["xu0"])
    s["lam"].copy_(s["lam0"])
    if case["batch"] == 1:
        r = sv.sqp_solve(s["Ns"][0], s["goal"], s["lam"], s["xu"], RHO)
        rho = [r.rho]
    else:
        rho, _ = sv.sqp_solve_batched(s["Ns"], s["goal"], s["lam"], s["xu"], s["rho"])
    return dict(xu=s["xu"], lam=s["lam"], rho=torch.tensor(rho))


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

# operations of one knot: its dynamics with their gradient (inverse dynamics of 7 + 1 columns, 14 tangents,
# the 7 x 7 inverse), its row of the Schur complement (four products of 14 x 14 blocks), the elimination of
# its block (a Cholesky factor, a triangular product and a symmetric update), the step and 8 line-search merits
KKT_FLOPS, FD_FLOPS, SCHUR_FLOPS, ELIM_FLOPS, DZ_FLOPS, ROW_FLOPS = 2.5e4, 5e3, 1.7e4, 7e3, 1.5e3, 1.2e3


def work(case):
    do = case["do"]
    if do == "rows":
        n = case["rows"]
        return dict(bytes=4.0 * n * (21 + 6 + 7 + 7 + 147), flops=n * (KKT_FLOPS + FD_FLOPS + 500))
    if do == "stages":
        N = case["knots"]
        floats = (21 + 6 + 574) + (574 + 588 * 2 + 14 + 245) + (588 + 14 * 4) + (245 * 2 + 294 + 21 + 28 + 21) + (48 + 8)
        return dict(bytes=4.0 * N * floats,
                    flops=N * (KKT_FLOPS + SCHUR_FLOPS + ELIM_FLOPS + ROW_FLOPS + DZ_FLOPS + 8 * FD_FLOPS))
    T = sum(horizons(case))
    step = KKT_FLOPS + SCHUR_FLOPS + ELIM_FLOPS + 2 * ROW_FLOPS + DZ_FLOPS
    if do == "adjoint":
        return dict(bytes=4.0 * T * (21 + 6 + 21 + 21 + 6), flops=T * (step + 2 * ROW_FLOPS + DZ_FLOPS + 1000))
    solve = T * case["iters"] * (step + 8 * FD_FLOPS)
    if do == "solve":
        return dict(bytes=4.0 * T * (21 * 2 + 6 + 14 * 2), flops=solve)
    grad = T * (step + 2 * ROW_FLOPS + DZ_FLOPS + 1000) if case["grad"] else 0
    rows = case["rows"] * case["batch"]
    return dict(bytes=4.0 * rows * 28, flops=case["updates"] * (solve + grad))


# ---------------------------------------------------------------------------
# the same in 64 bits, by plain torch
# ---------------------------------------------------------------------------

# the iiwa14: joint origins, fixed rotations (0 identity, 1 rpy(pi/2, 0, pi), 2 rpy(pi/2, 0, 0)), link
# masses, centres of mass and inertias about them (xx yy zz xy xz yz)
ORIGIN = [[0, 0, 0.1575], [0, 0, 0.2025], [0, 0.2045, 0], [0, 0, 0.2155], [0, 0.1845, 0], [0, 0, 0.2155], [0, 0.081, 0]]
KIND = [0, 1, 1, 2, 1, 2, 1]
FIXED = [[[1, 0, 0], [0, 1, 0], [0, 0, 1]], [[-1, 0, 0], [0, 0, 1], [0, 1, 0]], [[1, 0, 0], [0, 0, -1], [0, 1, 0]]]
MASS = [5.76, 6.35, 3.5, 3.5, 3.5, 1.8, 1.2]
COM = [[0, -0.03, 0.12], [0.0003, 0.059, 0.042], [0, 0.03, 0.13], [0, 0.067, 0.034], [0.0001, 0.021, 0.076],
       [0, 0.0006, 0.0004], [0, 0, 0.02]]
INERTIA = [[0.121, 0.116, 0.0175, 0, 0, -0.021], [0.0638, 0.0416, 0.0331, 0.0001, 0.00008, 0.0157],
           [0.0873, 0.083, 0.0108, 0, 0, 0.014], [0.0368, 0.02045, 0.02171, 0, 0, 0.008],
           [0.0318, 0.028916, 0.006, 0.000007, 0.000027, 0.005586], [0.0049, 0.0047, 0.0036, 0, 0, 0],
           [0.0055, 0.0055, 0.005, 0, 0, 0]]


def joints(q):
    """Per joint the rotation child -> parent [..., 3, 3] and the origin in the parent [3]."""
    f = dict(dtype=q.dtype, device=q.device)
    out = []
    for j in range(7):
        c, s, z, o = torch.cos(q[..., j]), torch.sin(q[..., j]), torch.zeros_like(q[..., j]), torch.ones_like(q[..., j])
        Rz = torch.stack([c, -s, z, s, c, z, z, z, o], -1).reshape(q.shape[:-1] + (3, 3))
        out.append((torch.tensor(FIXED[KIND[j]], **f) @ Rz, torch.tensor(ORIGIN[j], **f)))
    return out


def frames(q):
    R, p, out = None, None, []
    for W, o in joints(q):
        p = o.expand(q.shape[:-1] + (3,)) if R is None else p + (R @ o)
        R = W if R is None else R @ W
        out.append((R, p))
    return out


def ee_pose(q):
    R, p = frames(q)[-1]
    return torch.cat([p, torch.stack([torch.atan2(R[..., 2, 1], R[..., 2, 2]),
                                      -torch.atan2(R[..., 2, 0], torch.sqrt(R[..., 2, 1] ** 2 + R[..., 2, 2] ** 2)),
                                      torch.atan2(R[..., 1, 0], R[..., 0, 0])], -1)], -1)


def ee_jac(q):
    """Position [..., 3] and its Jacobian [..., 3, 7]."""
    F = frames(q)
    p = F[-1][1]
    return p, torch.stack([torch.linalg.cross(R[..., :, 2], p - o) for R, o in F], -1)


def inverse_dynamics(q, qd, qdd):
    """Recursive Newton-Euler without gravity."""
    f = dict(dtype=q.dtype, device=q.device)
    J, cross = joints(q), torch.linalg.cross
    ez = torch.tensor([0.0, 0.0, 1.0], **f)
    mv = lambda M, v: (M @ v.unsqueeze(-1)).squeeze(-1)  # noqa: E731
    shape = torch.broadcast_shapes(q.shape[:-1], qdd.shape[:-1]) + (3,)
    w = v = dw = dv = torch.zeros(shape, **f)
    F, Nn = [], []
    for j in range(7):
        E, p = J[j][0].transpose(-1, -2), J[j][1].expand(shape)
        v, dv = mv(E, v + cross(w, p)), mv(E, dv + cross(dw, p))
        w, dw = mv(E, w), mv(E, dw)
        s = ez * qd[..., j:j + 1]
        w = w + s
        dw = dw + cross(w, s) + ez * qdd[..., j:j + 1]
        dv = dv + cross(v, s)
        c, m = torch.tensor(COM[j], **f).expand(w.shape), MASS[j]
        xx, yy, zz, xy, xz, yz = INERTIA[j]
        Ic = torch.tensor([[xx, xy, xz], [xy, yy, yz], [xz, yz, zz]], **f)
        mom = lambda a, b: (mv(Ic, a) + m * cross(c, b + cross(a, c)), m * (b + cross(a, c)))  # noqa: E731
        (n1, f1), (nv, fv) = mom(dw, dv), mom(w, v)
        Nn.append(n1 + cross(w, nv) + cross(v, fv))
        F.append(f1 + cross(w, fv))
    tau = [None] * 7
    for j in range(6, -1, -1):
        tau[j] = Nn[j][..., 2]
        if j:
            W, p = J[j][0], J[j][1].expand(shape)
            f0 = mv(W, F[j])
            F[j - 1] = F[j - 1] + f0
            Nn[j - 1] = Nn[j - 1] + mv(W, Nn[j]) + cross(p, f0)
    return torch.stack(tau, -1)


def fd(z):
    """Forward dynamics of rows [q, qd, u]."""
    q, qd, u = z[..., :7], z[..., 7:14], z[..., 14:21]
    zero, e = torch.zeros_like(q), torch.eye(7, dtype=z.dtype, device=z.device)
    M = inverse_dynamics(q.unsqueeze(-2), zero.unsqueeze(-2), e.expand(q.shape[:-1] + (7, 7)))
    return torch.linalg.solve(M, u - inverse_dynamics(q, qd, zero))


def fd_jac(z):
    """Forward dynamics and its Jacobian [..., 7, 21]."""
    z, shape = z.reshape(-1, 21), z.shape[:-1]
    parts = []
    for y in z.split(16384):
        e = torch.eye(21, dtype=z.dtype, device=z.device)
        parts.append(torch.func.vmap(lambda d: torch.func.jvp(fd, (y,), (d.expand_as(y),))[1], out_dims=-1)(e))
    return fd(z).reshape(shape + (7,)), torch.cat(parts).reshape(shape + (7, 21))


def step_of(z, qdd, cfg):
    dt = float(torch.tensor(cfg["timestep"]).float())
    qd = z[..., 7:14] + dt * qdd
    return torch.cat([z[..., :7] + dt * (qd if cfg["integrator"] else z[..., 7:14]), qd], -1)


def weights(cfg, B, dev):
    f = lambda v: float(torch.tensor(v).float())  # noqa: E731
    w = lambda v, *s: torch.full(s, v, dtype=torch.float64, device=dev)  # noqa: E731
    return dict(qd=w(f(cfg["qd_cost"]), B, 7), r=w(f(cfg["r_cost"]), B, 7), ee=w(1.0, B))


def cost_blocks(z, goal, N, w):
    """Q, q, r of every knot.  The terminal knot's are taken at the knot before it, with the first
    three entries of that knot's Q as the target (what the reference's kernel computes)."""
    p, J = ee_jac(z[..., :7])
    ee, B = w["ee"][:, None, None], z.shape[0]
    vq = ee * (J.transpose(-1, -2) @ (p - goal[..., :3]).unsqueeze(-1)).squeeze(-1)
    b, at = torch.arange(B, device=z.device), N - 2
    tgt = vq[b, at, :1] * vq[b, at, :3]
    vt = w["ee"][:, None] * (J[b, at].transpose(-1, -2) @ (p[b, at] - tgt).unsqueeze(-1)).squeeze(-1)
    last = (torch.arange(z.shape[1], device=z.device)[None] == (N - 1)[:, None])[..., None]
    vq = torch.where(last, vt[:, None], vq)
    qd = torch.where(last, z[b, at, 7:14][:, None], z[..., 7:14])
    q = torch.cat([vq, w["qd"][:, None] * qd], -1)
    Q = torch.zeros(z.shape[:2] + (14, 14), dtype=z.dtype, device=z.device)
    Q[..., :7, :7] = vq.unsqueeze(-1) * vq.unsqueeze(-2)
    Q[..., 7:, 7:] = torch.diag_embed(w["qd"])[:, None]
    return Q, q, w["r"][:, None] * z[..., 14:21]


def kkt64(z, goal, xs, N, cfg, w):
    """The KKT blocks of a padded batch: Q, R, q, r, A = -df/dx, B = -df/du, defects c."""
    Q, q, r = cost_blocks(z, goal, N, w)
    dt = float(torch.tensor(cfg["timestep"]).float())
    qdd, D = fd_jac(z)
    f = dict(dtype=z.dtype, device=z.device)
    Av = torch.zeros(z.shape[:2] + (14, 21), **f)
    Av[..., 7:, :] = dt * D
    Av[..., 7:, 7:14] += torch.eye(7, **f)
    Av[..., :7, :7] = torch.eye(7, **f)
    if cfg["integrator"]:
        Av[..., :7, :] += dt * Av[..., 7:, :]
    else:
        Av[..., :7, 7:14] = dt * torch.eye(7, **f)
    c = torch.empty(z.shape[:2] + (14,), **f)
    c[:, 0] = z[:, 0, :14] - xs
    c[:, 1:] = z[:, 1:, :14] - step_of(z, qdd, cfg)[:, :-1]
    return dict(Q=Q, R=torch.diag_embed(w["r"])[:, None].expand(z.shape[:2] + (7, 7)), q=q, r=r, A=-Av[..., :14],
                B=-Av[..., 14:], c=c)


def schur64(k, rho):
    """S (left and diagonal blocks), gamma and the inverses; rho a number or one per instance."""
    f = dict(dtype=torch.float64, device=k["Q"].device)
    rho = torch.as_tensor(rho, **f).reshape(-1, 1, 1, 1)
    Qi = torch.linalg.inv(k["Q"] + rho * torch.eye(14, **f))
    Ri = torch.linalg.inv(k["R"] + rho * torch.eye(7, **f))
    mv = lambda M, v: (M @ v.unsqueeze(-1)).squeeze(-1)  # noqa: E731
    phi, br = k["A"] @ Qi, k["B"] @ Ri
    left, diag, gam = torch.zeros_like(k["Q"]), -Qi.clone(), k["c"] - mv(Qi, k["q"])
    left[:, 1:] = -phi[:, :-1]
    diag[:, 1:] -= (phi @ k["A"].transpose(-1, -2) + br @ k["B"].transpose(-1, -2))[:, :-1]
    gam[:, 0] -= k["c"][:, 0]
    gam[:, 1:] -= (mv(phi, k["q"]) + mv(br, k["r"]))[:, :-1]
    return dict(left=left, diag=diag, gamma=gam, Qi=Qi, Ri=Ri)


def solve64(left, diag, gam):
    """Block-tridiagonal solve along the knots.  A knot past an instance's end has its left block zeroed
    by the caller, so it does not touch the knots before it."""
    L = diag.shape[1]
    mv = lambda M, v: (M @ v.unsqueeze(-1)).squeeze(-1)  # noqa: E731
    inv, y = [], []
    for k in range(L):
        D, g = diag[:, k], gam[:, k]
        if k:
            T = left[:, k] @ inv[-1]
            D, g = D - T @ left[:, k].transpose(-1, -2), g - mv(T, y[-1])
        inv.append(torch.linalg.inv(D))
        y.append(g)
    x = [mv(inv[-1], y[-1])]
    for k in range(L - 2, -1, -1):
        x.append(mv(inv[k], y[k] - mv(left[:, k + 1].transpose(-1, -2), x[-1])))
    return torch.stack(x[::-1], 1)


def dz64(k, Qi, Ri, lam):
    mv = lambda M, v: (M @ v.unsqueeze(-1)).squeeze(-1)  # noqa: E731
    nxt = torch.zeros_like(lam)
    nxt[:, :-1] = lam[:, 1:]
    dx = mv(Qi, k["q"] - lam - mv(k["A"].transpose(-1, -2), nxt))
    du = mv(Ri, k["r"] - mv(k["B"].transpose(-1, -2), nxt))
    return torch.cat([dx, du], -1)


def kkt_step(k, rho, N, q=None, r=None, c=None):
    """(dz, lambda) of the KKT system for its own right-hand side or the given one."""
    k = dict(k, q=k["q"] if q is None else q, r=k["r"] if r is None else r, c=k["c"] if c is None else c)
    s = schur64(k, rho)
    live = torch.arange(k["q"].shape[1], device=N.device)[None] < N[:, None]
    left, gam = s["left"] * live[..., None, None], s["gamma"] * live[..., None]
    lam = solve64(left, s["diag"], gam) * live[..., None]
    A = k["A"] * (torch.arange(k["q"].shape[1], device=N.device)[None] < (N - 1)[:, None])[..., None, None]
    return dz64(dict(k, A=A), s["Qi"], s["Ri"], lam) * live[..., None], lam


def merit64(z, dz, alpha, goal, xs, N, cfg, w, line_search):
    y = z if dz is None else z + alpha * dz
    B, L = y.shape[:2]
    k = torch.arange(L, device=z.device)[None]
    live, run = (k < N[:, None]), (k < (N - 1)[:, None])
    p, _ = ee_jac(y[..., :7])
    cost = 0.5 * ((w["qd"][:, None] * y[..., 7:14] ** 2).sum(-1) + w["ee"][:, None] * ((p - goal[..., :3]) ** 2).sum(-1))
    cost = cost * live + 0.5 * (w["r"][:, None] * y[..., 14:21] ** 2).sum(-1) * run
    d = torch.zeros_like(cost)
    d[:, :-1] = (y[:, 1:, :14] - step_of(y, fd(y), cfg)[:, :-1]).abs().sum(-1)
    m = (cost + 10.0 * d * run).sum(1)
    return m + 10.0 * (y[:, 0, :14] - xs).abs().sum(-1) if line_search else m


def solve_exact(z, goal, Ns, cfg, iters):
    """The SQP iterations (factors of the step size and of rho as in the solver's defaults)."""
    dev, B = z.device, len(Ns)
    N, w, xs = torch.tensor(Ns, device=dev), weights(cfg, B, dev), z[:, 0, :14].clone()
    rho, drho = torch.full((B,), RHO, dtype=torch.float64, device=dev), torch.ones(B, dtype=torch.float64, device=dev)
    lam = None
    m0 = merit64(z, None, 0.0, goal, xs, N, cfg, w, False)
    for _ in range(iters):
        dz, lam = kkt_step(kkt64(z, goal, xs, N, cfg, w), rho, N)
        ms = torch.stack([merit64(z, dz, -(2.0 ** -p), goal, xs, N, cfg, w, True) for p in range(8)], 1)
        best, at = ms.min(1)
        ok = best < m0
        drho = torch.where(ok, torch.clamp(drho / 1.2, max=1 / 1.2), torch.clamp(drho * 1.2, min=1.2))
        rho = torch.clamp(rho * drho, min=RHO)
        z = z - (ok * 0.5 ** at.double())[:, None, None] * dz
        m0 = torch.where(ok, best, m0)
    return z, lam, rho


def exact(case, seed):
    do = case["do"]
    if do == "rows":
        x = prepare_rows(case, seed)
        qdd, D = fd_jac(x)
        return dict(pose=ee_pose(x[:, :7]), fd=qdd, qdd=qdd, df=D.transpose(-1, -2).reshape(x.shape[0], -1))
    if do == "stages":
        N, cfg, i, dev = stage_inputs(case, seed)
        n, w = torch.tensor([N], device=dev), weights(cfg, 1, dev)
        xu, goal, xs = i["xu"].double(), i["goal"].double(), i["xs"].double()
        k = kkt64(xu, goal, xs, n, cfg, w)
        s = schur64(k32(i, N, dev), RHO)
        zero = torch.zeros_like(s["left"])
        lam = pack(i["lam"], [N])
        dz = dz64(k32(i, N, dev), i["Qi"], i["Ri"], i["lam"])
        merits = torch.cat([merit64(xu, i["dz"].double(), -(2.0 ** -p), goal, xs, n, cfg, w, True) for p in range(8)])
        return dict(G=flat([k["Q"], k["R"]], N, 49), C=flat([k["A"], k["B"]], N, 294), g=flat([k["q"], k["r"]], N, 7),
                    c=pack(k["c"], [N]), S=three(s["left"], s["diag"]), Pinv=three(zero, -torch.linalg.inv(-s["diag"])),
                    gamma=pack(s["gamma"], [N]), Ginv=flat([s["Qi"], s["Ri"]], N, 49), lam=lam, lam64=lam,
                    dz=pack(dz, [N])[:21 * N - 7], merits=merits)
    if do == "track":
        return None  # rounding travels through the closed loop: every update starts from the one before
    cfg = settings(case)
    Ns, xu, goal, gen, dev = problems(case, seed)
    z, goal, T = xu.double(), goal.double(), sum(Ns)
    if do == "solve":
        z, lam, rho = solve_exact(z, goal, Ns, cfg, case["iters"])
        return dict(xu=pack(keep_tail(z, xu, Ns), Ns), lam=pack(lam, Ns), rho=rho)
    N, w = torch.tensor(Ns, device=dev), weights(cfg, len(Ns), dev)
    grad = torch.zeros_like(z)
    flatg, at = adjoint_loss(T, gen, dev).double().reshape(T, 21), 0
    for b, n in enumerate(Ns):
        grad[b, :n] = flatg[at:at + n]
        grad[b, n - 1, 14:] = 0.0
        at += n
    k = kkt64(z, goal, z[:, 0, :14], N, cfg, w)
    dz, _ = kkt_step(k, RHO, N)
    mu, _ = kkt_step(k, RHO, N, -grad[..., :14], -grad[..., 14:], torch.zeros_like(k["c"]))
    live = (torch.arange(z.shape[1], device=dev)[None] < N[:, None])[..., None]
    run = (torch.arange(z.shape[1], device=dev)[None] < (N - 1)[:, None])[..., None]
    th = dict(w, goal=goal)
    th = {n: v.clone().requires_grad_(True) for n, v in th.items()}
    Q, q, r = cost_blocks(z, th["goal"], N, th)
    val = (mu[..., :14] * (q - (Q @ dz[..., :14].unsqueeze(-1)).squeeze(-1)) * live).sum()
    val = val + (mu[..., 14:] * (r - th["r"][:, None] * dz[..., 14:]) * run).sum()
    gr = torch.autograd.grad(val, [th["goal"], th["qd"], th["r"], th["ee"]])
    return dict(goal=pack(gr[0], Ns), qd=gr[1], r=gr[2], q_ee=gr[3], xu_next=next_state(z, dz, Ns))


def prepare_rows(case, seed):
    gen, dev = generator(seed)
    n = case["rows"]
    lim = torch.tensor(LIMITS, device=dev)
    return torch.cat([(torch.rand(n, 7, generator=gen, device=dev) * 2 - 1) * lim,
                      torch.randn(n, 7, generator=gen, device=dev),
                      10 * torch.randn(n, 7, generator=gen, device=dev)], 1).double()


def keep_tail(z, xu0, Ns):
    """The unused control slot after an instance's last knot keeps what the call was given."""
    z = z.clone()
    for b, n in enumerate(Ns):
        z[b, n - 1, 14:] = xu0[b, n - 1, 14:].double()
    return z


def next_state(z, dz, Ns):
    v = pack(keep_tail(z - dz, z.float(), Ns), Ns)
    v[-7:] = 0.0  # past the batch's last state: not written
    return v
