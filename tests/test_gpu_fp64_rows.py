"""GPU: the FP64 kernels for rows of eight (meshes of about 6,000 cells and more; orders 0 and 5 always) against
the oracle: residual parts with every boundary treatment, partial groups, buffers on 8-byte boundaries, stepping."""
import numpy as np
import pytest

from conftest import CASES, rel_l2
from fve_dg_b200 import Ensemble, ExplicitConvection, box_mesh, problems
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu

TOL = 1e-12  # relative L2, the FP64 parity bar
ROWS_CASES = [(0, 2, 2)] + CASES + [(5, 7, 4)]


def mesh(P, walls="", seed=5):
    n = 4 if P in (0, 5) else 11  # 7,986 cells: rows of eight, and no class a multiple of eight
    return box_mesh(n, jitter=0.1, seed=seed, periodic={"": (1, 1, 1), "z": (1, 1, 0), "box": (0, 0, 0)}[walls],
                    bc="Dirichlet" if walls == "box" else "Pseudo3DZ")


def state(m, P, seed=0):
    U = problems.project(m, P, problems.density_wave())
    return U + 1e-3 * np.random.default_rng(seed + P).standard_normal(U.shape)


@pytest.mark.parametrize("walls", ["", "z"])
@pytest.mark.parametrize("P,qv,qf", ROWS_CASES)
def test_residual_parts_match_oracle(P, qv, qf, walls):
    m = mesh(P, walls)
    U, o = state(m, P), Oracle.from_mesh(m)
    for flux in ("LF", "Roe"):
        c = ExplicitConvection(m, order=P, flux=flux, quad_vol=qv, quad_face=qf)
        for part in range(4):
            want, got = o.residual(U, P, qv, qf, flux=flux, part=part), c._eval(U, 0.0, part)
            assert np.linalg.norm(got - want) <= TOL * np.linalg.norm(want), (flux, part)
        c.close()


@pytest.mark.parametrize("P,qv,qf", ROWS_CASES)
def test_dirichlet_faces_match_static_kernels(P, qv, qf):
    """Against the scalar FP64 kernels (dg_residual_device_static), which read the same boundary data."""
    import torch
    from fve_dg_b200 import _lib as L
    m = box_mesh(4 if P in (0, 5) else 10, jitter=0.1, seed=6, periodic=(0, 0, 0), bc="Dirichlet")
    U = state(m, P)
    c = ExplicitConvection(m, order=P, flux="Roe", quad_vol=qv, quad_face=qf)
    uv, _ = problems.quad_rule(1, qf)
    lam = np.concatenate([1.0 - uv.sum(1, keepdims=True), uv], axis=1)
    c.set_dirichlet(problems.density_wave()(np.einsum("ga,fad->fgd", lam, m.points[m.faces])))
    u = torch.from_numpy(U).cuda()
    for part in range(4):
        want = torch.zeros_like(u)
        assert L.lib().dg_residual_device_static(c._ctx, u.data_ptr(), want.data_ptr(), part, None) == 0
        torch.cuda.synchronize()
        assert rel_l2(c._eval(U, 0.0, part), want.cpu().numpy()) < TOL, part


@pytest.mark.parametrize("P,qv,qf", ROWS_CASES)
def test_device_buffers_on_odd_boundaries(P, qv, qf):
    import torch
    m = mesh(P, seed=7)
    U = state(m, P)
    c = ExplicitConvection(m, order=P, quad_vol=qv, quad_face=qf)
    want = c.eval(U)
    for i, o in ((0, 1), (1, 0), (1, 1)):
        a = torch.zeros(U.size + 2, dtype=torch.float64, device="cuda")
        b = torch.full((U.size + 2,), 7.0, dtype=torch.float64, device="cuda")
        a[i:i + U.size] = torch.from_numpy(U.ravel())
        c.eval_device(a.data_ptr() + 8 * i, b.data_ptr() + 8 * o, stream=torch.cuda.current_stream().cuda_stream)
        got = b.cpu().numpy()
        assert np.array_equal(got[o:o + U.size].reshape(U.shape), want)
        assert np.all(got[:o] == 7.0) and np.all(got[o + U.size:] == 7.0)


@pytest.mark.parametrize("P,qv,qf", [(0, 2, 2), (1, 0, 1), (2, 2, 3), (3, 3, 3), (4, 5, 3), (5, 7, 4)])
def test_stepping_matches_oracle(P, qv, qf):
    m = mesh(P)
    U, dt = state(m, P), 2e-4
    c = ExplicitConvection(m, order=P, quad_vol=qv, quad_face=qf)
    c.set_state(U)
    before = c.conservation()
    c.ssprk3(dt, 1)
    c.ssprk3(dt, 1, graph=True)
    got, after = c.get_state(), c.conservation()
    want = Oracle.from_mesh(m).ssprk3(U, P, qv, qf, dt, 2)
    assert rel_l2(got, want) < TOL
    assert rel_l2(got - U, want - U) < 1e-10
    assert np.all(np.abs(after[:5] - before[:5]) <= 1e-12 * np.maximum(1.0, np.abs(before[:5])))


def test_ensemble_uses_its_time_steps():
    ms = [box_mesh(n, jitter=0.05, seed=n) for n in (8, 9)]
    U = [state(m, 2, i) for i, m in enumerate(ms)]
    dts = np.array([1e-3, 5e-4])
    e = Ensemble(ms, order=2, quad_vol=1, quad_face=2)
    e.set_state(np.concatenate(U))
    e.ssprk3(dts, 2, graph=True)
    for got, m, u, dt in zip(e.split(e.get_state()), ms, U, dts):
        assert rel_l2(got, Oracle.from_mesh(m).ssprk3(u, 2, 1, 2, dt, 2)) < TOL
