"""GPU: which kernels a context takes, and those that no other test reaches: groups of sixteen at P4, the mixed
Navier-Stokes update in groups of sixteen, and meshes whose node orders leave too few items with equal face maps."""
import numpy as np
import pytest

from conftest import rel_l2
from fve_dg_b200 import ExplicitConvection, Mesh, box_mesh, problems
from fve_dg_b200 import _lib as L
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu

RES_TOL = 1e-4  # the mixed form's residual: about 16 bits on the deviations, FP32 fluxes


def state(m, P, seed=0):
    U = problems.project(m, P, problems.density_wave())
    return U + 1e-3 * np.random.default_rng(seed + P).standard_normal(U.shape)


def any_order(m, seed=0):
    """The mesh with the nodes of every cell and face in an arbitrary order, as another program may list them."""
    r = np.random.default_rng(seed)
    cells = r.permuted(m.cells, axis=1)
    order = r.permuted(np.tile(np.arange(3), (m.nface, 1)), axis=1)
    turned = [np.take_along_axis(f, order, axis=1) for f in (m.faces, m.face_nodes1)]
    return Mesh(points=m.points, cells=cells, faces=turned[0], face_cells=m.face_cells, face_nodes1=turned[1],
                periodic=m.periodic, bc=m.bc)


@pytest.mark.parametrize("P,n,precision,group", [
    (0, 2, "fp64", 8), (5, 2, "fp64", 8),                              # no tensor-core kernels but these
    (1, 9, "fp64", 3), (1, 10, "fp64", 8), (2, 8, "fp64", 3), (2, 9, "fp64", 8), (4, 8, "fp64", 3), (4, 9, "fp64", 8),
    (4, 12, "fp64", 3),                                                # a second round of groups that is nearly empty
    (1, 15, "mixed", 3), (1, 16, "mixed", 16), (3, 15, "mixed", 3), (3, 16, "mixed", 16),
    (4, 10, "mixed", 3), (4, 11, "mixed", 16), (4, 12, "mixed", 3), (4, 13, "mixed", 16),
])
def test_group_of_a_context(P, n, precision, group):
    """Sizes either side of the lines, for 148 SMs."""
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the sizes are for 148 SMs")
    qv, qf = {0: (-1, -1), 1: (0, 1), 2: (1, 2), 3: (3, 3), 4: (5, 3), 5: (-1, -1)}[P]
    c = ExplicitConvection(box_mesh(n), order=P, quad_vol=qv, quad_face=qf, precision=precision)
    assert c.kernel_group() == group and c.kernel_group(viscous=True) == 0
    c.close()


@pytest.mark.parametrize("walls", ["", "z", "box"])
@pytest.mark.parametrize("qv,qf", [(5, 3), (6, 3)])
def test_p4_groups_of_sixteen(qv, qf, walls):
    """As test_gpu_mixed16.py, whose P4 mesh (10,368 cells) lies between the lines."""
    m = box_mesh(11, jitter=0.1, seed=5, periodic={"": (1, 1, 1), "z": (1, 1, 0), "box": (0, 0, 0)}[walls],
                 bc="Dirichlet" if walls == "box" else "Pseudo3DZ")
    U = state(m, 4)
    for flux in ("LF", "Roe"):
        out = {}
        for prec in ("fp64", "mixed"):
            c = ExplicitConvection(m, order=4, flux=flux, quad_vol=qv, quad_face=qf, precision=prec)
            assert c.kernel_group() == (16 if prec == "mixed" else 8)
            if walls == "box":
                uv, _ = problems.quad_rule(1, qf)
                lam = np.concatenate([1.0 - uv.sum(1, keepdims=True), uv], axis=1)
                c.set_dirichlet(problems.density_wave()(np.einsum("ga,fad->fgd", lam, m.points[m.faces])))
            out[prec] = [c._eval(U, 0.0, part) for part in range(4)]
            c.close()
        for part, (a, b) in enumerate(zip(out["mixed"], out["fp64"])):
            if part == 3 and walls == "":
                assert not a.any()
            else:
                assert rel_l2(a, b) < RES_TOL, (flux, part, rel_l2(a, b))


@pytest.mark.parametrize("qv", [5, 6])
def test_p4_schedules_and_odd_boundaries(qv):
    import torch
    m = box_mesh(11, jitter=0.1, seed=7)
    U = state(m, 4)
    out = []
    for schedule in ("two-launch", "persistent"):
        c = ExplicitConvection(m, order=4, flux="Roe", quad_vol=qv, quad_face=3, precision="mixed", schedule=schedule)
        assert c.kernel_group() == 16
        want = c.eval(U)
        for i, o in ((0, 1), (1, 0), (1, 1)):
            a = torch.zeros(U.size + 2, dtype=torch.float64, device="cuda")
            b = torch.full((U.size + 2,), 7.0, dtype=torch.float64, device="cuda")
            a[i:i + U.size] = torch.from_numpy(U.ravel())
            c.eval_device(a.data_ptr() + 8 * i, b.data_ptr() + 8 * o, stream=torch.cuda.current_stream().cuda_stream)
            got = b.cpu().numpy()
            assert np.array_equal(got[o:o + U.size].reshape(U.shape), want)
            assert np.all(got[:o] == 7.0) and np.all(got[o + U.size:] == 7.0)
        c.set_state(U)
        before = c.conservation()
        c.ssprk3(1e-4, 2)
        c.ssprk3(1e-4, 2, graph=True)
        after = c.conservation()
        assert np.all(np.abs(after[:5] - before[:5]) <= 1e-12 * np.maximum(1.0, np.abs(before[:5])))
        out.append(c.get_state())
        c.close()
    assert np.array_equal(out[0], out[1])
    ref = ExplicitConvection(m, order=4, flux="Roe", quad_vol=qv, quad_face=3)
    ref.set_state(U)
    ref.ssprk3(1e-4, 4)
    assert rel_l2(out[0], ref.get_state()) < 1e-6


@pytest.mark.parametrize("P,n,schedule", [(1, 16, "two-launch"), (3, 16, "persistent"), (4, 11, "two-launch")])
def test_mixed_navier_stokes_in_groups_of_sixteen(P, n, schedule):
    """The viscous residual in the mixed update (Rv): the first stage with viscosity less the one without is
    dt R_visc / b, but for the rounding of the two stages: 2 units of 2^-53 of the state, under 1e-10 of this."""
    import torch
    m = box_mesh(n, jitter=0.1, seed=32)
    U, dt, mu = state(m, P), 1e-4, 0.05
    stage = []
    for visc in (mu, 0.0):
        c = ExplicitConvection(m, order=P, mu=visc, prandtl=0.72, precision="mixed", schedule=schedule)
        assert c.kernel_group() == 16
        c.set_state(U)
        L.check(L.lib().dg_ssprk3_stage(c._ctx, dt, 0), "dg_ssprk3_stage")
        torch.cuda.synchronize()

        class Stage:
            __cuda_array_interface__ = {"shape": c.shape, "typestr": "<f8", "version": 3,
                                        "data": (L.lib().dg_state_device(c._ctx, 1), False)}
        stage.append(torch.as_tensor(Stage(), device="cuda").cpu().numpy())
        want = dt * c.viscous_eval(U, mu=mu, prandtl=0.72) / c.mass()
        assert c.kernel_group(viscous=True) == 8
        c.close()
    got = stage[0] - stage[1]
    assert np.linalg.norm(want) > 1e-5 * np.linalg.norm(U)
    assert rel_l2(got, want) < 1e-10


@pytest.mark.parametrize("P,qv,qf,group", [(0, 2, 2, 1), (2, 1, 2, 3), (3, 3, 3, 3), (5, 7, 4, 1)])
def test_many_classes_of_face_maps(P, qv, qf, group):
    """Too few items of a kind to fill groups of eight: the kernels for few items, and the same operator."""
    m = any_order(box_mesh(4 if P in (0, 5) else 9, jitter=0.1, seed=3))
    U = state(m, P)
    o = Oracle.from_mesh(m)
    c = ExplicitConvection(m, order=P, flux="Roe", quad_vol=qv, quad_face=qf)
    assert c.kernel_group() == group
    for part in range(3):
        want, got = o.residual(U, P, qv, qf, flux="Roe", part=part), c._eval(U, 0.0, part)
        assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want), part
    if 1 <= P <= 4:
        c.viscous_eval(U)
        assert c.kernel_group(viscous=True) == 1
    c.close()


def test_many_classes_of_face_maps_mixed():
    m = any_order(box_mesh(17, jitter=0.1, seed=3))  # 29,478 cells
    U = state(m, 2)
    out = []
    for prec, group in (("fp64", 3), ("mixed", 3)):
        c = ExplicitConvection(m, order=2, quad_vol=1, quad_face=2, precision=prec)
        assert c.kernel_group() == group
        out.append(c.eval(U))
        c.close()
    assert rel_l2(out[1], out[0]) < RES_TOL


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_viscous_operator_between_the_convective_lines(precision):
    """P4 with the 44-point rule at 10,368 cells: the convective kernels' line there is not the viscous ones'."""
    m = box_mesh(12, jitter=0.1, seed=5)
    U = state(m, 4)
    out = []
    for mu in (0.0, 0.3):  # mu > 0 in FP64: the fused kernels' groups, at any size
        c = ExplicitConvection(m, order=4, quad_vol=5, quad_face=3, precision=precision, mu=mu)
        out.append(c.viscous_eval(U, mu=0.3, prandtl=0.72))
        assert c.kernel_group() == 3 and c.kernel_group(viscous=True) == 8
        c.close()
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("P,n,group", [(2, 17, 16), (2, 8, 3)])
def test_autotune_reports_the_tiles_that_ran(P, n, group):
    m = box_mesh(n, jitter=0.1, seed=5)
    c = ExplicitConvection(m, order=P, quad_vol=1, quad_face=2, precision="mixed", schedule="persistent")
    assert c.kernel_group() == group
    U = state(m, P)
    c.set_state(U)
    rec = c.autotune(1e-4)
    tiles = {(x["tile_f"], x["tile_e"]) for x in rec["candidates"]}
    # asked for in groups of three; groups of sixteen: three eighths as many, of faces and elements alike
    asked = {(32, 16), (16, 8), (64, 32), (128, 64)}
    assert rec["items_per_group"] == group
    assert tiles == (asked if group == 3 else {(f * 3 // 8, f * 3 // 8) for f, _ in asked})
    assert (rec["chosen"]["tile_f"], rec["chosen"]["tile_e"]) in tiles
    assert np.array_equal(c.get_state(), U)
    c.close()
    # the shape of the two-launch element kernel: one in groups of sixteen, pinned or not
    c = ExplicitConvection(m, order=P, quad_vol=1, quad_face=2, precision="mixed")
    assert len(c.set_state(U) or c.autotune(1e-4)["candidates"]) == (1 if group == 16 else 3)
    out = []
    for staged in (False, True):
        c.set_element_shape(staged, 1)
        c.set_state(U)
        c.ssprk3(1e-4, 1)
        out.append(c.get_state())
    assert np.array_equal(out[0], out[1])
