"""GPU: what the mixed form is off from FP64 after many steps, where errors that are the same in every step add up.
The bounds are what the kernels for groups of three gave on the same runs (to the digits they were recorded with)."""
import pytest

from fve_dg_b200 import ExplicitConvection, box_mesh, problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,jitter,flux,steps,rho,energy", [
    (32, 0.1, "LF", 200, 8.15e-8, 4.55e-8),  # density wave, P2, 196,608 tets
])
def test_density_wave_after_many_steps(n, jitter, flux, steps, rho, energy):
    m = box_mesh(n, jitter=jitter)
    U0 = problems.project(m, 2, problems.density_wave())
    dt = None
    state = {}
    for prec in ("fp64", "mixed"):
        c = ExplicitConvection(m, order=2, flux=flux, quad_vol=1, quad_face=2, precision=prec)
        c.set_state(U0)
        if dt is None:
            dt = problems.cfl_dt(0.3, 1.0 / n, 2, c.max_wave_speed())
        c.ssprk3(dt, steps, graph=True)
        state[prec] = c.get_state()
        c.close()
    err = problems.l2_errors(m, 2, state["mixed"], Uref=state["fp64"])
    assert err[0] <= rho and err[4] <= energy, err
