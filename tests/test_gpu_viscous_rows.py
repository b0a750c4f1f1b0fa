"""GPU: the viscous operator in rows of eight (meshes of about 1,200 cells and more) against the kernels with one
warp per item, which smaller meshes run: a whole mesh against its eighths (998 cells), whose owned elements have the
same viscous residual. And the fused Navier-Stokes stage against a loop built from the two residuals."""
import numpy as np
import pytest

from conftest import CASES, rel_l2
from fve_dg_b200 import ExplicitConvection, box_mesh, problems
from fve_dg_b200.partition import LocalMesh, partition_elements

pytestmark = pytest.mark.gpu

TOL = 1e-12  # relative L2, the FP64 parity bar


def mesh(walls):
    return box_mesh(11, jitter=0.1, seed=5, periodic={"": (1, 1, 1), "z": (1, 1, 0), "box": (0, 0, 0)}[walls],
                    bc="Dirichlet" if walls == "box" else "Pseudo3DZ")


def state(m, P, seed=0):
    U = problems.project(m, P, problems.density_wave(A=0.3))
    return U + 1e-2 * np.random.default_rng(seed + P).standard_normal(U.shape)


def boundary(m, qf):
    uv, _ = problems.quad_rule(1, qf)
    lam = np.concatenate([1.0 - uv.sum(1, keepdims=True), uv], axis=1)
    return problems.density_wave()(np.einsum("ga,fad->fgd", lam, m.points[m.faces]))


@pytest.mark.parametrize("walls", ["", "z", "box"])
@pytest.mark.parametrize("P,qv,qf", CASES)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_whole_mesh_matches_its_eighths(P, qv, qf, walls, precision):
    if precision == "mixed" and (walls != "" or (P, qv) not in ((2, 1), (4, 5))):
        pytest.skip("the operator is the same in a mixed context: two cases")
    m = mesh(walls)
    U = state(m, P)
    kw = dict(order=P, quad_vol=qv, quad_face=qf, precision=precision)
    whole = ExplicitConvection(m, **kw)
    if walls == "box":
        whole.set_dirichlet(boundary(m, qf))
    R = whole.viscous_eval(U, mu=0.7, prandtl=0.72)
    owner = partition_elements(m, 8)
    for r in range(8):
        p = LocalMesh(m, owner, r)
        c = ExplicitConvection(p.mesh, **kw)
        if walls == "box":
            c.set_dirichlet(boundary(p.mesh, qf))
        got = c.viscous_eval(U[p.l2g], mu=0.7, prandtl=0.72)[:p.n_owned]
        assert p.n_owned < 1184 and np.abs(got).max() > 0
        assert rel_l2(R[p.l2g[:p.n_owned]], got) < TOL
        c.close()


@pytest.mark.parametrize("P,qv,qf,flux,walls", [(1, 0, 1, "LF", ""), (2, 1, 2, "Roe", "z"), (3, 3, 3, "Roe", ""), (4, 5, 3, "LF", "box")])
def test_fused_stage_matches_residuals(P, qv, qf, flux, walls):
    m = mesh(walls)
    U, dt, mu = state(m, P), 1e-5, 0.05
    kw = dict(order=P, flux=flux, quad_vol=qv, quad_face=qf)
    c = ExplicitConvection(m, mu=mu, prandtl=0.72, **kw)
    e = ExplicitConvection(m, **kw)
    for x in (c, e):
        if walls == "box":
            x.set_dirichlet(boundary(m, qf))
    b = e.mass()

    def L(V):
        return (e.viscous_eval(V, mu=mu, prandtl=0.72) - e.eval(V)) / b

    V1 = U + dt * L(U)
    V2 = 0.75 * U + 0.25 * (V1 + dt * L(V1))
    V = U / 3 + 2.0 / 3 * (V2 + dt * L(V2))
    c.set_state(U)
    before = c.conservation()
    for graph in (False, True):
        c.set_state(U)
        c.ssprk3(dt, 1, graph=graph)
        got = c.get_state()
        assert rel_l2(got, V) < TOL and rel_l2(got - U, V - U) < 1e-10
    if walls == "":
        after = c.conservation()
        assert np.all(np.abs(after[:5] - before[:5]) <= 1e-12 * np.maximum(1.0, np.abs(before[:5])))
