"""Rigid-body library kernels and trajectory files: gpt_end_effector_positions against the
reference's own FK file (testfiles/0_0_eepos.traj: end_effector_positions_kernel on every row of
0_0_traj.csv, generateeepos.cu:101-107), gpt_forward_dynamics against the reference's explicit-Euler
trajectories (testfiles/*_traj.csv, dt = 1/64, gravity 0) and the oracle, and gpt_read_csv (the
readCSVToVecVec of runme.cu:18-44) on files written from those rows."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


# ---------------------------------------------------------------------------
# CPU: the trajectory reader
# ---------------------------------------------------------------------------

def test_read_csv_round_trips_reference_rows(gpt, golden, tmp_path):
    tr = golden["traj_0_1"]
    f = tmp_path / "0_1_traj.csv"
    f.write_text("\n".join(",".join(f"{v:.9g}" for v in row) for row in tr) + "\n")
    got = gpt.read_csv(str(f))
    assert got.shape == tr.shape
    np.testing.assert_array_equal(got, tr.astype(np.float32))


def test_read_csv_edge_cases(gpt, tmp_path):
    f = tmp_path / "a.csv"
    f.write_text("1,2,3,\r\n4,5e-3,-6\n\n")  # trailing comma (no empty field), CRLF, blank line
    np.testing.assert_array_equal(gpt.read_csv(str(f)), np.array([[1, 2, 3], [4, 5e-3, -6]], np.float32))
    g = tmp_path / "ragged.csv"
    g.write_text("1,2,3\n4,5\n")
    with pytest.raises(gpt.GptError):
        gpt.read_csv(str(g))
    with pytest.raises(gpt.GptError):
        gpt.read_csv(str(tmp_path / "missing.csv"))


# ---------------------------------------------------------------------------
# GPU
# ---------------------------------------------------------------------------

def dev(a):
    return torch.as_tensor(np.ascontiguousarray(a, np.float32), device="cuda")


@pytest.mark.gpu
def test_end_effector_positions_match_reference_file(gpt, oracle, golden):
    """All 666 rows of 0_0_traj.csv in one launch (row stride 21): within 3e-5 of the reference's
    printed FK (6 significant digits), the FP32 oracle's bound; a stride-14 state batch gives the
    same values."""
    tr, ee = golden["traj_0_0"], golden["eepos_0_0"]
    got = gpt.end_effector_positions(dev(tr), 21).cpu().numpy()
    assert got.shape == ee.shape
    assert np.abs(got - ee).max() < 3e-5, np.abs(got - ee).max()
    want = np.stack([oracle.fk(r[:7].astype(np.float64)) for r in tr[:50]])
    assert np.abs(got[:50] - want).max() < 3e-5
    got14 = gpt.end_effector_positions(dev(tr[:, :14]), 14).cpu().numpy()
    np.testing.assert_array_equal(got14, got)


@pytest.mark.gpu
def test_forward_dynamics_reproduces_reference_trajectories(gpt, oracle, golden):
    """qd_{k+1} = qd_k + dt FD(x_k, u_k) on the reference's explicit-Euler rollouts (the bound the
    oracle meets, 2e-5), and FD within 1e-5 relative of the FP64 oracle row by row."""
    dt = 1.0 / 64
    for name in ("traj_0_1", "traj_1_2", "traj_2_3", "traj_3_4", "traj_4_0"):
        tr = golden[name]
        qdd = gpt.forward_dynamics(dev(tr), 21).cpu().numpy().astype(np.float64)
        x = tr.astype(np.float64)
        res = np.abs(x[2:, 7:14] - (x[1:-1, 7:14] + dt * qdd[1:-1])).max()
        assert res < 2e-5, (name, res)
        for k in range(0, len(tr), 17):
            want = oracle.fd(x[k, :7], x[k, 7:14], x[k, 14:21])
            assert np.abs(qdd[k] - want).max() <= 1e-5 * max(1.0, np.abs(want).max()), (name, k)


@pytest.mark.gpu
def test_library_kernels_reject_bad_strides(gpt):
    x = torch.zeros(21 * 4, device="cuda")
    with pytest.raises(gpt.GptError):
        gpt.forward_dynamics(x, 14)
    with pytest.raises(gpt.GptError):
        gpt.end_effector_positions(x, 3)


@pytest.mark.gpu
def test_forward_dynamics_gradient_matches_oracle(gpt, oracle, golden):
    """gpt_forward_dynamics_gradient (forwardDynamicsAndGradient) on rows of the reference's
    trajectories against the FP64 oracle's fd_grad: qdd within 1e-5 and each 7 x 7 block of df/du
    within 1e-4 of its largest entry (FP32 tangent inverse dynamics); qdd also agrees with
    gpt_forward_dynamics."""
    tr = np.concatenate([golden["traj_0_1"][::5], golden["traj_3_4"][::5]])
    qdd, df = (t.cpu().numpy().astype(np.float64) for t in gpt.forward_dynamics_gradient(dev(tr), 21))
    qdd_fd = gpt.forward_dynamics(dev(tr), 21).cpu().numpy().astype(np.float64)
    assert np.abs(qdd - qdd_fd).max() <= 1e-5 * max(1.0, np.abs(qdd_fd).max())
    for k, row in enumerate(tr.astype(np.float64)):
        wq, wdf = oracle.fd_grad(row[:7], row[7:14], row[14:21])
        assert np.abs(qdd[k] - wq).max() <= 1e-5 * max(1.0, np.abs(wq).max()), k
        for b in range(3):
            blk = slice(49 * b, 49 * (b + 1))
            assert np.abs(df[k, blk] - wdf[blk]).max() <= 1e-4 * max(1e-3, np.abs(wdf[blk]).max()), (k, b)


@pytest.mark.gpu
@pytest.mark.parametrize("n,stride", [(8191, 21), (8192, 21), (8193, 22), (8192 + 63, 24), (18944 + 65, 21), (40001, 21)])
def test_forward_dynamics_gradient_by_row_count(gpt, oracle, golden, n, stride):
    """Both forms of the gradient (a half-warp per row below 8192 rows, a lane per row from there on) against the FP64
    oracle at the edges of their ranges, with the tolerances of the test above; a row of NaN stays alone, and nothing is
    written past the last row."""
    tr = np.concatenate([golden["traj_0_1"], golden["traj_3_4"]])
    rng = np.random.default_rng(n)
    rows = tr[rng.integers(0, len(tr), n), :21] + rng.uniform(-0.1, 0.1, (n, 21)).astype(np.float32)
    bad = n // 2
    x = np.zeros((n, stride), np.float32)
    x[:, :21] = rows
    x[bad, 3] = np.nan
    xu = dev(x)
    qdd_t, df_t = (torch.full((n + 3, w), 7.0, device="cuda") for w in (7, 147))
    gpt._check(gpt.lib().gpt_forward_dynamics_gradient(n, gpt._ptr(xu), stride, gpt._ptr(qdd_t), gpt._ptr(df_t),
                                                       gpt._stream(None)))
    torch.cuda.synchronize()
    qdd, df = qdd_t.cpu().numpy(), df_t.cpu().numpy()
    assert (qdd[n:] == 7.0).all() and (df[n:] == 7.0).all()
    ok = np.arange(n) != bad
    assert np.isfinite(qdd[:n][ok]).all() and np.isfinite(df[:n][ok]).all() and np.isnan(qdd[bad]).all()
    check = np.unique(np.concatenate([np.arange(3), np.arange(n - 40, n), [bad - 1, bad + 1], rng.integers(0, n, 40)]))
    for k in check[check != bad]:
        row = x[k].astype(np.float64)
        wq, wdf = oracle.fd_grad(row[:7], row[7:14], row[14:21])
        assert np.abs(qdd[k] - wq).max() <= 1e-5 * max(1.0, np.abs(wq).max()), k
        for b in range(3):
            blk = slice(49 * b, 49 * (b + 1))
            assert np.abs(df[k, blk] - wdf[blk]).max() <= 1e-4 * max(1e-3, np.abs(wdf[blk]).max()), (k, b)


@pytest.mark.gpu
@pytest.mark.parametrize("n,stride", [(4095, 21), (4096, 21), (4097, 22), (4096 + 63, 24), (37888 + 33, 21)])
def test_forward_dynamics_by_row_count(gpt, oracle, golden, n, stride):
    """Both forms of the forward dynamics (eight lanes per row below 4096 rows, a lane per row from there on) against the
    FP64 oracle with the tolerance used for the gradient's qdd; a row of NaN stays alone, and nothing is written past the
    last row."""
    tr = np.concatenate([golden["traj_0_1"], golden["traj_3_4"]])
    rng = np.random.default_rng(n)
    x = np.zeros((n, stride), np.float32)
    x[:, :21] = tr[rng.integers(0, len(tr), n), :21] + rng.uniform(-0.1, 0.1, (n, 21)).astype(np.float32)
    bad = n // 2
    x[bad, 3] = np.nan
    xu, out = dev(x), torch.full((n + 3, 7), 7.0, device="cuda")
    gpt._check(gpt.lib().gpt_forward_dynamics(n, gpt._ptr(xu), stride, gpt._ptr(out), gpt._stream(None)))
    torch.cuda.synchronize()
    qdd = out.cpu().numpy()
    assert (qdd[n:] == 7.0).all() and np.isnan(qdd[bad]).all()
    assert np.isfinite(qdd[:n][np.arange(n) != bad]).all()
    check = np.unique(np.concatenate([np.arange(3), np.arange(n - 40, n), [bad - 1, bad + 1], rng.integers(0, n, 40)]))
    for k in check[check != bad]:
        row = x[k].astype(np.float64)
        wq, _ = oracle.fd_grad(row[:7], row[7:14], row[14:21])
        assert np.abs(qdd[k] - wq).max() <= 1e-5 * max(1.0, np.abs(wq).max()), k
