"""GPU: the mixed form's kernels for groups of sixteen (meshes of about 24,000 cells and more, P4 from
about 7,000): residual parts against the FP64 form on ragged meshes with every boundary treatment, device
buffers on 8-byte boundaries, both schedules, a split mesh and an ensemble."""
import numpy as np
import pytest

from conftest import CASES, rel_l2
from fve_dg_b200 import Ensemble, ExplicitConvection, box_mesh, problems

pytestmark = pytest.mark.gpu

# As for the groups of three: about 16 bits on the deviations through each contraction, FP32 fluxes.
RES_TOL = 1e-4
N = {1: 17, 2: 17, 3: 17, 4: 12}  # cubes per side: no multiple of sixteen in a class, so partial groups too


def state(m, P, seed=0):
    U = problems.project(m, P, problems.density_wave())
    return U + 1e-3 * np.random.default_rng(seed + P).standard_normal(U.shape)


@pytest.mark.parametrize("walls", ["", "z", "box"])
@pytest.mark.parametrize("P,qv,qf", CASES)
def test_residual_parts_close_to_fp64(P, qv, qf, walls):
    m = box_mesh(N[P], jitter=0.1, seed=5, periodic={"": (1, 1, 1), "z": (1, 1, 0), "box": (0, 0, 0)}[walls],
                 bc="Dirichlet" if walls == "box" else "Pseudo3DZ")
    U = state(m, P)
    for flux in ("LF", "Roe"):
        out = {}
        for prec in ("fp64", "mixed"):
            c = ExplicitConvection(m, order=P, flux=flux, quad_vol=qv, quad_face=qf, precision=prec)
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


@pytest.mark.parametrize("P,qv,qf", [(1, 0, 1), (2, 1, 2), (3, 3, 3), (4, 5, 3)])
def test_device_buffers_on_odd_boundaries(P, qv, qf):
    """Rows that start 8 bytes past a 16-byte boundary, in the input, the output or both."""
    import torch
    m = box_mesh(N[P], jitter=0.1, seed=6)
    U = state(m, P)
    c = ExplicitConvection(m, order=P, quad_vol=qv, quad_face=qf, precision="mixed")
    want = c.eval(U)
    for i, o in ((0, 1), (1, 0), (1, 1)):
        a = torch.zeros(U.size + 2, dtype=torch.float64, device="cuda")
        b = torch.full((U.size + 2,), 7.0, dtype=torch.float64, device="cuda")
        a[i:i + U.size] = torch.from_numpy(U.ravel())
        c.eval_device(a.data_ptr() + 8 * i, b.data_ptr() + 8 * o, stream=torch.cuda.current_stream().cuda_stream)
        got = b.cpu().numpy()
        assert np.array_equal(got[o:o + U.size].reshape(U.shape), want)
        assert np.all(got[:o] == 7.0) and np.all(got[o + U.size:] == 7.0)


@pytest.mark.parametrize("P,qv,qf", [(1, 0, 1), (2, 1, 2), (3, 3, 3), (3, 4, 3), (4, 5, 3), (4, 6, 3)])
def test_persistent_schedule_is_bit_identical(P, qv, qf):
    m = box_mesh(N[P], jitter=0.1, seed=7)
    U = state(m, P)
    out = []
    for schedule in ("two-launch", "persistent"):
        c = ExplicitConvection(m, order=P, flux="Roe", quad_vol=qv, quad_face=qf, precision="mixed", schedule=schedule)
        c.set_state(U)
        before = c.conservation()
        c.ssprk3(1e-4, 2)
        c.ssprk3(1e-4, 2, graph=True)
        after = c.conservation()
        assert np.all(np.abs(after[:5] - before[:5]) <= 1e-12 * np.maximum(1.0, np.abs(before[:5])))
        out.append(c.get_state())
        c.close()
    assert np.array_equal(out[0], out[1])
    ref = ExplicitConvection(m, order=P, flux="Roe", quad_vol=qv, quad_face=qf)
    ref.set_state(U)
    ref.ssprk3(1e-4, 4)
    assert rel_l2(out[0], ref.get_state()) < 1e-6


def test_split_mesh_matches_whole():
    """Two parts of 24,000 owned cells, stepped stage by stage with their ghost rows exchanged on the host,
    in one go and in two phases."""
    import ctypes
    from fve_dg_b200 import _lib as L
    from fve_dg_b200.partition import LocalMesh, partition_elements
    import torch
    P, qv, qf, dt = 2, 1, 2, 1e-3
    m = box_mesh(20, jitter=0.1, seed=8)
    U = state(m, P)
    whole = ExplicitConvection(m, order=P, quad_vol=qv, quad_face=qf, precision="mixed")
    whole.set_state(U)
    whole.ssprk3(dt, 2)
    want = whole.get_state()
    owner = partition_elements(m, 2)
    parts = [LocalMesh(m, owner, r) for r in range(2)]
    for phased in (False, True):
        ctx = [ExplicitConvection(p.mesh, order=P, quad_vol=qv, quad_face=qf, precision="mixed") for p in parts]
        for c, p in zip(ctx, parts):
            c.set_state(U[p.l2g])

        def buffer(c, which):
            class B:
                __cuda_array_interface__ = {"shape": c.shape, "typestr": "<f8", "version": 3,
                                            "data": (L.lib().dg_state_device(c._ctx, which), False)}
            return torch.as_tensor(B(), device="cuda")
        for step in range(2):
            for stage in range(3):
                if phased:
                    for c in ctx:
                        assert L.lib().dg_ssprk3_stage_phase(c._ctx, dt, stage, 0) == 0
                torch.cuda.synchronize()
                full = torch.empty((m.ncell, ctx[0].shape[1]), dtype=torch.float64, device="cuda")
                for c, p in zip(ctx, parts):
                    full[torch.as_tensor(p.l2g[:p.n_owned], device="cuda")] = buffer(c, stage)[:p.n_owned]
                for c, p in zip(ctx, parts):
                    buffer(c, stage)[p.n_owned:] = full[torch.as_tensor(p.l2g[p.n_owned:], device="cuda")]
                torch.cuda.synchronize()
                for c in ctx:
                    if phased:
                        assert L.lib().dg_ssprk3_stage_phase(c._ctx, dt, stage, 1) == 0
                    else:
                        assert L.lib().dg_ssprk3_stage(c._ctx, dt, stage) == 0
        for c, p in zip(ctx, parts):
            c.ssprk3(dt, 0)
            assert rel_l2(c.get_state()[:p.n_owned], want[p.l2g[:p.n_owned]]) < 1e-13
            c.close()


def test_ensemble_matches_its_schedules():
    ms = [box_mesh(n, jitter=0.05, seed=n) for n in (12, 13, 11)]
    U = np.concatenate([state(m, 2, i) for i, m in enumerate(ms)])
    dts = np.array([1e-3, 5e-4, 2e-3])
    out = []
    for schedule in ("two-launch", "persistent"):
        e = Ensemble(ms, order=2, quad_vol=1, quad_face=2, precision="mixed", schedule=schedule)
        e.set_state(U)
        e.ssprk3(dts, 3, graph=schedule == "persistent")
        out.append(e.get_state())
        e.close()
    assert np.array_equal(out[0], out[1])
    ref = Ensemble(ms, order=2, quad_vol=1, quad_face=2)
    ref.set_state(U)
    ref.ssprk3(dts, 3)
    assert rel_l2(out[0], ref.get_state()) < 1e-6
