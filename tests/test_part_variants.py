"""The partitioned PCG's variants (2 to 32 parts per instance on 1 to 8 CTAs, chosen by the batch size and the longest
horizon) at the edges of their ranges, and their part layouts.

Tolerance: the multipliers are the FP64 solution of a system of condition up to about 2e7 (2.2e-16 x 2e7 x
a growth factor of 100 = 5e-7), so 1e-6 of the largest component."""
import importlib
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SPEC_CFG = dict(timestep=0.01, integrator=1, qd_cost=1e-2, r_cost=1e-4)

PROGRAM = r"""
#include "gpt_layout.h"
template <int NW> int check(int edge)
{
    for (int n = 2; n <= 512; ++n) {
        const gpt::PartLayout<NW> L = gpt::part_layout<NW>(n, edge);
        int pos = 0;
        if (L.P < 1 || L.P > NW) return 1;
        for (int p = 0; p < L.P; ++p) {
            if (L.a[p] != pos || L.b[p] < pos - 1) return 2;
            pos = L.b[p] + 1;
            if (p < L.P - 1 && L.s[p] != pos++) return 3;
            // equally spaced separators: the kernel keeps the first one and the spacing
            if (NW > 2 && p < L.P - 1 && L.s[p] != L.s[0] + p * (L.s[NW > 2 ? 1 : 0] - L.s[0])) return 4;
        }
        if (pos != n) return 5;
    }
    return 0;
}
int main()
{
    for (int edge = 13; edge <= 15; edge += 2)
        if (check<2>(edge) || check<4>(edge) || check<8>(edge) || check<16>(edge) || check<32>(edge)) return 1;
    return 0;
}
"""


def test_part_layouts(tmp_path):
    (tmp_path / "l.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "gpu-pcg-tracking_b200", "csrc"),
                    str(tmp_path / "l.cpp"), "-o", str(tmp_path / "l")], check=True)
    assert subprocess.run([str(tmp_path / "l")]).returncode == 0


# (instances in SM counts, more instances, horizons that are repeated over the batch)
SIZES = [(0, 1, [64]), (0, 5, [2, 3, 4, 15, 63]), (0, 9, [2, 3, 5, 7, 15, 16, 17, 18, 64]), (1, 0, [70, 9, 33]),
         (1, 1, [2, 3, 4, 5, 6, 7, 8, 9, 31]), (2, 0, [2, 7, 8, 65]), (2, 1, [2, 3, 4, 5, 6, 17, 40]),
         # one instance at the edges of 4, 8, 16 and 32 parts; batches on clusters of 8, 4 and 2 CTAs, and just above
         (0, 1, [23]), (0, 1, [24]), (0, 1, [47]), (0, 1, [48]), (0, 1, [255]), (0, 1, [256]), (0, 1, [511]),
         (0, 12, [300, 2, 3, 31, 62, 63, 64, 65, 17, 5]), (0, 13, [256, 9, 2]), (0, 32, [48, 2, 3, 15, 30, 31, 32, 33]),
         (0, 33, [48, 2, 3, 14, 15, 16, 17]), (0, 74, [50, 2, 5, 15, 16, 29]), (0, 75, [50, 2, 5, 15, 16, 29])]


@pytest.mark.gpu
@pytest.mark.parametrize("sms,more,pattern", SIZES)
@pytest.mark.parametrize("tol,mode,schur_fp64", [(1e-5, 0, 1), (1e-13, 0, 1), (1e-6, 1, 1), (1e-5, 0, 0)])
def test_part_variants_solve_the_system(problem_mod, sms, more, pattern, tol, mode, schur_fp64):
    """One SQP iteration's multipliers against an FP64 host solve of the same KKT system: the first
    preconditioner application is exact (tolerance 1e-5), and the iteration goes on correctly (a tolerance
    below the rounding of the residual, and the exit test on r . z, which needs a second application).  With
    FP32 Schur rows (schur_fp64 0) the system itself is rounded: the bound there is the FP32 rounding times
    the condition, so only the residual's convergence is checked, by the iteration count."""
    import torch
    gpt = importlib.import_module("gpu-pcg-tracking_b200")
    check = importlib.import_module("gpu-pcg-tracking_b200.fp64check")
    B = sms * torch.cuda.get_device_properties(0).multi_processor_count + more
    Ns = [pattern[i % len(pattern)] for i in range(B)]
    probs = [problem_mod.make_problem(n, 300 + i, dt=0.01) for i, n in enumerate(pattern)]
    pad = np.zeros(7, np.float32)
    dev = lambda key, tail: torch.as_tensor(  # noqa: E731
        np.concatenate([np.concatenate([probs[i % len(pattern)][key], tail]) for i in range(B)]), device="cuda")
    xu, goal, lam = dev("xu", pad), dev("goal", pad[:0]), dev("lam", pad[:0])
    sv = gpt.Solver(max_knot_points=max(Ns), max_batch=B, sqp_max_iter=1, pcg_max_iter=6, pcg_exit_tol=tol,
                    pcg_exit_mode=mode, pcg_cluster_size=gpt.PCG_WARP_QUAD, schur_fp64=schur_fp64, **SPEC_CFG)
    _, stats, tr = sv.sqp_solve_batched_trace(Ns, goal, lam, xu, [1e-3] * B, 1)
    got, off = tr["lam"][0].cpu().numpy(), np.concatenate([[0], np.cumsum(Ns)])
    its = [s["pcg_iters_total"] for s in stats]
    if mode == 0 and tol == 1e-5:
        assert max(its) <= 2
    for i, n in enumerate(pattern):
        if not schur_fp64 or i >= B:
            break
        z = lambda m: torch.zeros(m, device="cuda")  # noqa: E731
        G, Cm, g, c = z(245 * n - 49), z(294 * (n - 1)), z(21 * n - 7), z(14 * n)
        d = {k: torch.as_tensor(v, device="cuda") for k, v in probs[i].items()}
        sv.form_kkt(n, d["xu"], d["goal"], d["xs"], G, Cm, g, c)
        want, _ = check.solve_step(n, 1e-3, *(t.cpu().numpy() for t in (G, Cm, g, c)))
        for b in {i, len(pattern) * ((B - 1 - i) // len(pattern)) + i}:  # the first and last instance of this horizon
            assert check.rel_err(got[14 * off[b]:14 * off[b + 1]], want) <= 1e-6, (n, b)
    sv.close()


@pytest.mark.gpu
@pytest.mark.parametrize("N", [2, 3, 33, 64, 129])
def test_pcg_entry_point_starts_from_the_given_lambda(oracle, problem_mod, N):
    """gpt_pcg with the library's choice of kernel: from any start it reaches the FP64 Cholesky solution, and from a
    solution it takes no iteration and returns it unchanged (the solution rounded to float32 keeps a residual of
    about 6e-8 x |S| |lambda| / |gamma|, far above any tolerance a user sets, so that start is checked with a
    tolerance above it)."""
    import torch
    gpt = importlib.import_module("gpu-pcg-tracking_b200")
    p = problem_mod.make_problem(N, 70 + N, dt=0.01)
    par = oracle.make_params(dt=0.01, integrator=1, qd_cost=1e-2, r_cost=1e-4)
    S, Pv, gam, _ = oracle.form_schur(N, 1e-2, *(np.asarray(x, np.float32) for x in oracle.form_kkt(
        par, N, p["xu"], p["goal"], p["xs"])))
    S, Pv, gam = (np.asarray(x, np.float32) for x in (S, Pv, gam))
    ref = oracle.banded_cholesky(N, S.astype(np.float64), gam.astype(np.float64))
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a, np.float32), device="cuda")  # noqa: E731
    sv = gpt.Solver(max_knot_points=N, **SPEC_CFG)
    rng = np.random.default_rng(N)
    for start in (np.zeros(14 * N), rng.normal(0, np.abs(ref).max(), 14 * N), ref):
        lam, lam64 = dev(start), torch.zeros(14 * N, device="cuda", dtype=torch.float64)
        it, maxed = sv.pcg(N, dev(S), dev(Pv), dev(gam), lam, 50, 1e-9, 0, lam64=lam64)
        assert not maxed and it <= 3
        assert np.abs(lam64.cpu().numpy() - ref).max() <= 1e-6 * np.abs(ref).max()
    lam, lam64 = dev(ref), torch.zeros(14 * N, device="cuda", dtype=torch.float64)
    it, maxed = sv.pcg(N, dev(S), dev(Pv), dev(gam), lam, 50, 1e3, 0, lam64=lam64)
    assert it == 0 and not maxed
    assert np.array_equal(lam.cpu().numpy(), ref.astype(np.float32))
    sv.close()
