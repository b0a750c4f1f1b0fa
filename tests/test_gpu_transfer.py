"""GPU: host arrays of 4 MB and more, copied in parts by several threads, against the same operator on device buffers:
rows packed and apart, parts that don't fill their chunks, pinned arrays, several contexts and threads at once."""
import threading

import numpy as np
import pytest
import torch

from fve_dg_b200 import ExplicitConvection, box_mesh, problems
from fve_dg_b200 import _lib as L

pytestmark = pytest.mark.gpu


def on_device(c, U):
    d = torch.from_numpy(U).cuda()
    r = torch.zeros_like(d)
    torch.cuda.synchronize()
    L.check(L.lib().dg_residual_device(c._ctx, d.data_ptr(), r.data_ptr(), 0.0, 0, None), "dg_residual_device")
    torch.cuda.synchronize()
    return r.cpu().numpy()


@pytest.mark.parametrize("P,n", [(1, 17), (2, 13), (2, 14), (4, 11)])  # 4.7, 5.3, 6.6, 11.2 MB
def test_host_arrays(P, n):
    m = box_mesh(n, jitter=0.1, seed=2)
    c = ExplicitConvection(m, order=P)
    U = problems.project(m, P, problems.density_wave()) + 1e-3 * np.random.default_rng(n).standard_normal((m.ncell, 5 * problems.num_basis(P)))
    assert U.nbytes >= 4 << 20
    want = on_device(c, U)
    for _ in range(3):
        assert np.array_equal(c.eval(U), want)
    pinned, out = torch.from_numpy(U).pin_memory().numpy(), torch.zeros(U.shape, dtype=torch.float64).pin_memory().numpy()
    L.check(L.lib().dg_residual(c._ctx, L.dptr(pinned), L.dptr(out), 0, 0.0, 0), "dg_residual")
    assert np.array_equal(out, want)
    apart, out = np.full((m.ncell, U.shape[1] + 3), np.nan), np.full((m.ncell, U.shape[1] + 3), 7.0)
    apart[:, :U.shape[1]] = U
    L.check(L.lib().dg_residual(c._ctx, L.dptr(apart), L.dptr(out), apart.strides[0], 0.0, 0), "dg_residual")
    assert np.array_equal(out[:, :U.shape[1]], want) and np.all(out[:, U.shape[1]:] == 7.0)
    c.set_state(U)
    assert np.array_equal(c.get_state(), U)


def test_threads():
    m = box_mesh(13, jitter=0.1, seed=2)
    U = [problems.project(m, 2, problems.density_wave(A=0.1 * (i + 1))) for i in range(3)]
    ctx = [ExplicitConvection(m, order=2) for _ in U]
    want = [on_device(c, u) for c, u in zip(ctx, U)]
    bad = []

    def work(i):
        for _ in range(8):
            if not np.array_equal(ctx[i].eval(U[i]), want[i]):
                bad.append(i)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
    for c in ctx:
        c.close()
    c = ExplicitConvection(m, order=2)  # after the staging memory went with the last context
    assert np.array_equal(c.eval(U[0]), want[0])
