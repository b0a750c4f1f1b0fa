"""GPU: conservation sums, wave speed and non-physical point count against numpy, at element counts that leave a last
group of eight partial, for every order and volume rule."""
import numpy as np
import pytest

from fve_dg_b200 import ExplicitConvection, box_mesh, problems
from fve_dg_b200 import _lib as L

pytestmark = pytest.mark.gpu

RULES = [(0, 0), (0, 2), (1, 0), (1, 2), (2, 1), (2, 2), (3, 3), (3, 4), (4, 5), (4, 6), (5, 7), (2, 5)]


def values(m, U, P, qv):
    x, w = problems.quad_rule(0, qv)
    phi, _ = problems.basis(P, x)  # [g][b]
    return np.einsum("gb,ebk->egk", phi, U.reshape(m.ncell, -1, 5)), w


@pytest.mark.parametrize("n", [1, 3])  # 6 cells (one partial group), 162 (20 groups and two cells)
@pytest.mark.parametrize("P,qv", RULES)
def test_reductions(P, qv, n):
    m = box_mesh(n, jitter=0.1 if n > 1 else 0.0, seed=4, periodic=(0, 0, 0), bc="Dirichlet")
    U = problems.project(m, P, problems.density_wave(A=0.3))
    U += 1e-2 * np.random.default_rng(P).standard_normal(U.shape)
    c = ExplicitConvection(m, order=P, quad_vol=qv, quad_face=2 if P < 4 else 4)
    c.set_state(U)
    V, w = values(m, U, P, qv)
    d = m.points[m.cells]
    dj = np.abs(np.linalg.det(d[:, 1:] - d[:, :1]))
    rho, mom2 = V[..., 0], (V[..., 1:4] ** 2).sum(-1)
    want = np.append((U.reshape(m.ncell, -1, 5)[:, 0] * dj[:, None] / 6).sum(0), (w * dj[:, None] * 0.5 * mom2 / rho).sum())
    # sums of positive and negative terms: the rounding of each term, a few times over
    scale = np.append((np.abs(U.reshape(m.ncell, -1, 5)[:, 0]) * dj[:, None] / 6).sum(0), abs(want[5]))
    assert np.all(np.abs(c.conservation() - want) <= 1e-13 * scale)
    p = 0.4 * (V[..., 4] - 0.5 * mom2 / rho)
    assert p.min() > 0
    lam = (np.sqrt(mom2) / rho + np.sqrt(1.4 * p / rho)).max()
    assert abs(c.max_wave_speed() - lam) <= 1e-13 * lam
    assert c.check_state() == 0
    # cells with a negative pressure at every point, a NaN, an infinity: each counts its points; the wave speed leaves
    # them out
    Ub = U.reshape(m.ncell, -1, 5).copy()
    Ub[0, 0, 4] = -50.0
    Ub[2, 0, 2] = np.nan
    Ub[m.ncell - 1, 0, 0] = np.inf
    c.set_state(Ub.reshape(U.shape))
    bad = c.check_state()
    assert bad == 3 * V.shape[1]
    keep = np.ones(m.ncell, bool)
    keep[[0, 2, m.ncell - 1]] = False
    lam = (np.sqrt(mom2) / rho + np.sqrt(1.4 * p / rho))[keep].max()
    assert abs(c.max_wave_speed() - lam) <= 1e-13 * lam
