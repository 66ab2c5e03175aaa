"""The 3-D update with its FP64 island on badly scaled and strongly correlated covariances, where
the residual's z column, which the double form leaves out, is largest.  One layer at the tracks' own z
and no covariance with z: the propagation changes nothing, and the update alone is compared
with the full Joseph form in 80-bit arithmetic."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# track covariance scale and correlation, hit sigma scales (x, y, z) and correlation
CASES = {"ordinary": (1, 0.4, (1, 1, 1), 0.3), "large_track": (1e8, 0.4, (1, 1, 1), 0.3),
         "correlated_track": (1e4, 30, (1, 1, 1), 0.3), "correlated_hit": (1, 0.4, (1, 1, 1), 100),
         "both": (1e4, 30, (1, 1, 1), 100), "coarse_z": (1, 0.4, (1, 1, 1e4), 30), "fine_z": (1, 0.4, (1, 1, 1e-6), 30),
         "fine_xy": (1, 0.4, (1e-4, 1e-4, 1), 30)}
LIVE = [0, 1, 3, 4, 5]


def _spd(r, n, d, rho):
    low = np.tril(r.uniform(-1, 1, (n, d, d)) * rho)
    i = np.arange(d)
    low[:, i, i] = 1
    a = low @ low.transpose(0, 2, 1)
    s = np.sqrt(a[:, i, i])
    return a / s[:, :, None] / s[:, None, :]


def _joseph(C, V):
    """(I - K H) C (I - K H)^T + K V K^T for the live rows, x and y measured and z with no covariance."""
    C, V = C.astype(np.longdouble), V.astype(np.longdouble)
    R = V.copy()
    R[:, :2, :2] += C[:, :2, :2]
    A = np.empty_like(R)
    for i in range(3):
        for j in range(3):
            a, b, c, d = ((i + 1) % 3, (j + 1) % 3, (i + 2) % 3, (j + 2) % 3)
            A[:, i, j] = R[:, a, b] * R[:, c, d] - R[:, a, d] * R[:, c, b]
    det = (R[:, 0] * A[:, 0]).sum(1)
    CH = np.zeros((len(C), 5, 3), dtype=np.longdouble)
    CH[:, :, :2] = C[:, :, :2]
    mul = lambda x, y: (x[:, :, :, None] * y[:, None, :, :]).sum(2)  # noqa: E731 (matmul has no long double)
    K = mul(CH, A / det[:, None, None])
    M = np.broadcast_to(np.eye(5, dtype=np.longdouble), C.shape).copy()
    M[:, :, :2] -= K[:, :, :2]
    return (mul(mul(M, C), M.transpose(0, 2, 1)) + mul(mul(K, V), K.transpose(0, 2, 1))).astype(np.float64)


@pytest.mark.parametrize("name", list(CASES))
def test_update_alone(p2z, ctx, name):
    scale, rho_c, sv, rho_v = CASES[name]
    r = np.random.default_rng(17)
    n = 4096
    cfg = p2z.make_config(bsize=32, nevts=1, ntrks=n, nlayer=1, update="3x3_f64")
    trk, hit = p2z.generate_physics(cfg)
    sigma = np.exp(r.uniform(np.log(0.3), np.log(3), (n, 5))) * [0.1, 0.1, 0.01, 1e-3, 1e-3] * np.sqrt(scale)
    C = (_spd(r, n, 5, rho_c) * sigma[:, :, None] * sigma[:, None, :]).astype(np.float32)
    s = np.array([3e-3, 3e-3, 1e-4]) * sv
    V = (_spd(r, n, 3, rho_v) * s[:, None] * s[None, :]).astype(np.float32)
    C, V = (np.tril(a) + np.tril(a, -1).transpose(0, 2, 1) for a in (C, V))
    lanes = lambda a: a.reshape(n // 32, 32).astype(np.float32)  # noqa: E731
    trk[:, 6:27] = 0
    at = {(i, j): i * (i + 1) // 2 + j for i in range(6) for j in range(i + 1)}
    for a, i in enumerate(LIVE):
        for b, j in enumerate(LIVE[:a + 1]):
            trk[:, 6 + at[i, j]] = lanes(C[:, a, b])
    for i in range(3):
        for j in range(i + 1):
            hit[:, 0, 3 + at[i, j]] = lanes(V[:, i, j])
    hit[:, 0, 2] = trk[:, 2]
    out = np.empty_like(trk)
    ctx.run(cfg, trk, hit, out)
    ok = np.linalg.eigvalsh(V.astype(np.float64))[:, 0] > 0  # (rounded to float it may no longer be a covariance)
    assert ok.mean() > 0.9
    ref = _joseph(C, V)
    for a, i in enumerate(LIVE):
        for b, j in enumerate(LIVE[:a + 1]):
            got = out[:, 6 + at[i, j]].reshape(-1).astype(np.float64)
            # the float's own rounding, and a quarter of one of the diagonal's scale: evaluated in double, either
            # form is within 6e-10 of that scale on such inputs
            bound = 2.0 ** -24 * np.abs(ref[:, a, b]) + 2.0 ** -26 * np.sqrt(ref[:, a, a] * ref[:, b, b])
            assert (np.abs(got - ref[:, a, b]) <= bound)[ok].all(), (i, j)
