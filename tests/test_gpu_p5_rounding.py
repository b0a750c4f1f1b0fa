"""GPU: rounding of the P5 kernels for rows of eight against extended precision: no further off than the scalar FP64
kernels (dg_residual_device_static), which sum a mode's points one by one."""
import math

import numpy as np
import pytest

from fve_dg_b200 import ExplicitConvection, box_mesh, problems
from fve_dg_b200 import _lib as L

pytestmark = pytest.mark.gpu

LD = np.longdouble
G1 = LD(1.4) - 1
P, QV, QF = 5, 7, 4


def basis(x, y, z):
    """Values of the modal basis at points; complex arguments give derivatives by a complex step."""
    def jac(n, a, y, s):
        return sum(math.comb(n + a, n - m) * math.comb(n, m) * (y - s) ** m * y ** (n - m) for m in range(n + 1))
    one = np.ones_like(x)
    return np.stack([jac(d - q - r, 2 * (q + r) + 2, x, one) * jac(q, 2 * r + 1, y, 1 - x) * jac(r, 0, z, 1 - x - y)
                     for d in range(P + 1) for r in range(d + 1) for q in range(d - r + 1)], 1)


def flux(U):
    u = U[..., 1:4] / U[..., :1]
    p = G1 * (U[..., 4] - (U[..., 1:4] * u).sum(-1) / 2)
    F = U[..., :, None] * u[..., None, :]
    for i in range(3):
        F[..., 1 + i, i] += p
    F[..., 4, :] += p[..., None] * u
    return F, np.sqrt((u * u).sum(-1)) + np.sqrt(LD(1.4) * p / U[..., 0])


def residual(m, U):
    """(volume term, whole residual) of the Lax-Friedrichs operator, periodic mesh."""
    (pts, wv), (uv, wf) = ([np.asarray(a).astype(LD) for a in problems.quad_rule(*q)] for q in ((0, QV), (1, QF)))
    C, X = U.astype(LD).reshape(U.shape[0], -1, 5), m.points.astype(LD)
    x = [pts[:, i].astype(np.clongdouble) for i in range(3)]
    phi = basis(*x).real
    dphi = np.stack([basis(*[c + 1e-25j * (j == i) for j, c in enumerate(x)]).imag / LD(1e-25) for i in range(3)], 2)
    E = X[m.cells][:, 1:] - X[m.cells][:, :1]
    cof = np.stack([np.cross(E[:, (i + 1) % 3], E[:, (i + 2) % 3]) for i in range(3)], 2)  # det E times its inverse
    det = np.einsum("ei,ei->e", E[:, 0], cof[:, :, 0])
    F = np.einsum("egkm,emd->egkd", flux(np.einsum("gb,ebk->egk", phi, C))[0], cof * np.sign(det)[:, None, None])
    V = -np.einsum("gbd,g,egkd->ebk", dphi, wv, F)
    T, (c0, c1) = X[m.faces], m.face_cells.T
    n = np.cross(T[:, 1] - T[:, 0], T[:, 2] - T[:, 0])
    n *= np.sign((n * (T.mean(1) - X[m.cells][c0].mean(1))).sum(-1))[:, None]
    area = np.sqrt((n * n).sum(-1))
    lam = np.concatenate([1 - uv.sum(1, keepdims=True), uv], 1)
    corner = np.concatenate([np.zeros((1, 3), LD), np.eye(3, dtype=LD)])
    trace, maps = [], []
    for cell, nodes in ((c0, m.faces), (c1, m.face_nodes1)):
        slot = (m.cells[cell][:, None, :] == nodes[:, :, None]).argmax(-1)
        v, mp = np.zeros((len(cell), len(wf), 5), LD), []
        for s in np.unique(slot, axis=0):
            at = np.nonzero((slot == s).all(1))[0]
            ph = basis(*(lam @ corner[s]).T)
            v[at] = np.einsum("gb,fbk->fgk", ph, C[cell[at]])
            mp.append((at, cell[at], ph))
        trace.append(v)
        maps.append(mp)
    (FL, sL), (FR, sR) = flux(trace[0]), flux(trace[1])
    Fn = (((FL + FR) * n[:, None, None, :]).sum(-1)
          + (np.maximum(sL, sR) * area[:, None])[..., None] * (trace[0] - trace[1])) * wf[:, None] / 2
    R = V.copy()
    for sign, mp in zip((1, -1), maps):
        for at, cell, ph in mp:
            np.add.at(R, cell, sign * np.einsum("gb,fgk->fbk", ph, Fn[at]))
    return V.reshape(U.shape), R.reshape(U.shape)


@pytest.mark.parametrize("n,jitter,seed", [(3, 0.1, 1), (2, 0.0, 2)])
def test_no_further_off_than_the_scalar_kernels(n, jitter, seed):
    import torch
    m = box_mesh(n, jitter=jitter, seed=seed)
    U = problems.project(m, P, problems.density_wave())
    U = U + 1e-3 * np.random.default_rng(seed).standard_normal(U.shape) / (1 + np.arange(U.shape[1]))
    V, R = residual(m, U)
    c = ExplicitConvection(m, order=P, flux="LF", quad_vol=QV, quad_face=QF)
    a = torch.from_numpy(U).cuda()
    b = torch.empty_like(a)
    for part, exact in ((1, V), (0, R)):
        L.check(L.lib().dg_residual_device_static(c._ctx, a.data_ptr(), b.data_ptr(), part, 0), "static")
        torch.cuda.synchronize()
        off = [float(np.sqrt(((r - exact) ** 2).sum())) for r in (c._eval(U, 0.0, part), b.cpu().numpy())]
        assert 0 < off[0] <= off[1], (part, off)
