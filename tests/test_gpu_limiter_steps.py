"""GPU: the limiter's bounds and three steps against a numpy restatement (PositiveLimiter.h:57-258), for every rule it
has, at cell counts that leave a warp's last cells and a block's last warps empty, with states that reach each step, with
NaN and infinite cells, and on rows that start on an odd double."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from fve_dg_b200 import ExplicitConvection, box_mesh, problems
from fve_dg_b200 import _lib as L

pytestmark = pytest.mark.gpu

TOL = 1e-12  # relative L2, the FP64 parity bar
RULES = [(1, 0), (1, 2), (2, 1), (2, 2), (3, 3), (3, 4), (4, 5), (4, 6)]


def rmax(a, b):  # std::max and std::min: a NaN on the right is skipped
    return np.where(a < b, b, a)


def rmin(a, b):
    return np.where(b < a, b, a)


def pressure(S, gamma=1.4):
    rho = S[..., 0]
    ke = (S[..., 1] ** 2 + S[..., 2] ** 2 + S[..., 3] ** 2) / (2.0 * rho)
    return np.where(rho <= 1e-16, -1.0, (gamma - 1.0) * (S[..., 4] - ke))


def reference(m, U, Uprev, P, qv, only_avg):
    phi, _ = problems.basis(P, problems.quad_rule(0, qv)[0])
    points = lambda W: np.einsum("gb,ebk->egk", phi, W.reshape(m.ncell, -1, 5))
    prev = Uprev.reshape(m.ncell, -1, 5)
    if only_avg:
        hi, lo = prev[:, 0].copy(), prev[:, 0].copy()
    else:
        V = points(Uprev)
        hi, lo = np.full((m.ncell, 5), -np.finfo(float).max), V[:, -1].copy()
        for g in range(V.shape[1]):
            hi = rmax(hi, V[:, g])
    nbr = np.arange(m.ncell)[:, None].repeat(4, 1)
    for f in range(m.nface):
        a, b = m.face_cells[f]
        if b >= 0:
            nbr[a, np.flatnonzero(m.cell_faces[a] == f)] = b
            nbr[b, np.flatnonzero(m.cell_faces[b] == f)] = a
    bmax, bmin = hi.copy(), lo.copy()
    for q in range(4):
        bmax, bmin = rmax(bmax, hi[nbr[:, q]]), rmin(bmin, lo[nbr[:, q]])
    C = U.reshape(m.ncell, -1, 5).copy()
    avg, v = C[:, 0].copy(), points(U)
    reached = [0, 0, 0]
    for k in range(5):
        out = ((v[..., k] < bmin[:, None, k]) | (v[..., k] > bmax[:, None, k])).any(1)
        vmin, vmax = np.nanmin(v[..., k], 1), np.nanmax(v[..., k], 1)
        tmin = np.where(avg[:, k] != vmin, (avg[:, k] - bmin[:, k]) / (avg[:, k] - vmin + 1e-32), 0.0)
        tmax = np.where(avg[:, k] != vmax, (bmax[:, k] - avg[:, k]) / (vmax - avg[:, k] + 1e-32), 0.0)
        theta = np.where(out, rmin(rmin(tmin, tmax), 1.0), 1.0)
        reached[0] += out.sum()
        C[out, 1:, k] *= theta[out, None]
        v[out, :, k] = avg[out, None, k] + theta[out, None] * (v[out, :, k] - avg[out, None, k])
    low = (v[..., 0] < 1e-16).any(1)
    eff = rmax(avg[:, 0], 1e-16)
    den = eff - v[..., 0].min(1)
    theta = np.where(den < 1e-32, 0.0, rmin(1.0, (eff - 1e-16) / den))
    C[low, 1:, 0] *= theta[low, None]
    v[low, :, 0] = avg[low, None, 0] + theta[low, None] * (v[low, :, 0] - avg[low, None, 0])
    reached[1] = low.sum()
    neg = pressure(v) < 0
    a = np.zeros(neg.shape)
    b = np.ones(neg.shape)
    for _ in range(100):
        mid = 0.5 * (a + b)
        bad = pressure((1.0 - mid[..., None]) * avg[:, None] + mid[..., None] * v) < 0
        a, b = np.where(bad, a, mid), np.where(bad, mid, b)
    tp = np.where(neg, mid, 1.0).min(1)
    C[:, 1:] *= np.where(neg.any(1), tp, 1.0)[:, None, None]
    reached[2] = neg.any(1).sum()
    return C.reshape(U.shape), reached


def states(m, P, A, noise, seed):
    rng = np.random.default_rng(seed)
    Uprev = problems.project(m, P, problems.density_wave(A=A))
    hi = np.arange(Uprev.shape[1]) >= 5
    U = Uprev + noise * rng.standard_normal(Uprev.shape) * hi * np.abs(Uprev[:, :5]).max()
    U[:, :5] += 0.01 * rng.standard_normal((U.shape[0], 5))
    return U, Uprev


@pytest.mark.parametrize("only_avg", [False, True])
@pytest.mark.parametrize("n", [1, 3])  # 6 and 162 cells
@pytest.mark.parametrize("P,qv", RULES)
def test_limiter_matches_numpy(P, qv, n, only_avg):
    m = box_mesh(n, jitter=0.1 if n > 1 else 0.0, seed=5, periodic=(0, 0, 0), bc="Dirichlet")
    c = ExplicitConvection(m, order=P, quad_vol=qv, quad_face=2 if P < 4 else 3)
    steps = np.zeros(3, int)
    for A, noise, seed in ((0.2, 0.05, 1), (0.97, 0.3, 2)):
        U, Uprev = states(m, P, A, noise, 100 * P + seed)
        want, reached = reference(m, U, Uprev, P, qv, only_avg)
        got = c.limit(U, Uprev, only_neighbor_avg=only_avg)
        assert np.array_equal(got[:, :5], U[:, :5])
        assert rel_l2(got, want) < TOL
        steps += reached
    assert steps[0] > 0 and (n == 1 or only_avg or steps[2] > 0)  # bounds from means alone leave no negative pressure
    # a NaN and an infinite cell in the previous state: skipped by their neighbours' bounds, kept in their own
    U, Uprev = states(m, P, 0.2, 0.05, 9)
    Uprev[1, 5 * 0 + 4] = np.nan
    Uprev[m.ncell - 2, 0] = np.inf
    with np.errstate(all="ignore"):
        want, _ = reference(m, U, Uprev, P, qv, only_avg)
    got = c.limit(U, Uprev, only_neighbor_avg=only_avg)
    ok = np.isfinite(want).all(1)
    assert ok.sum() > m.ncell // 2 and rel_l2(got[ok], want[ok]) < TOL
    # device rows on an odd double give the same bits
    U, Uprev = states(m, P, 0.97, 0.3, 3)
    got = c.limit(U, Uprev, only_neighbor_avg=only_avg)
    for shift in (0, 1):
        d = torch.zeros(U.size + 1, dtype=torch.float64, device="cuda")
        d[shift:shift + U.size] = torch.from_numpy(U.ravel())
        prev = torch.from_numpy(Uprev).cuda()
        torch.cuda.synchronize()
        L.check(L.lib().dg_limit_device(c._ctx, d.data_ptr() + 8 * shift, prev.data_ptr(), int(only_avg), None), "dg_limit_device")
        torch.cuda.synchronize()
        assert np.array_equal(d[shift:shift + U.size].cpu().numpy().reshape(U.shape), got)
