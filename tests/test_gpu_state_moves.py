"""State transfers in CTAs of 128 cells and step scalars written by the last CTA: at cell counts
around the tile, at sub-arrays that start on 8 bytes, with one array or wider strides (which take
the general kernel), and over several reported steps.  Copies and repeated steps are exact."""
import ctypes

import numpy as np
import pytest
import torch

from cases import GAMMA_43
from radrhd_solver_b200 import _lib as L
from radrhd_solver_b200 import mesh as Mm
from radrhd_solver_b200 import rhllc

pytestmark = pytest.mark.gpu
SIZES = [(1, 1, 1), (3, 7, 1), (2, 11, 1), (4, 4, 4), (5, 13, 1), (7, 7, 7)]  # 6 cells to 2058, 126, 132, 384, 390


def make(shape):
    m = Mm.kuhn_box(*shape, lo=(0, 0, 0), hi=(1, 1, 1), jitter=0.1, seed=5)
    g = rhllc.Grid(m, eos=1, gamma=GAMMA_43)
    rng = np.random.default_rng(m.n_cells)
    W = np.concatenate([rng.uniform(0.5, 2, (m.n_cells, 1)), rng.uniform(-0.3, 0.3, (m.n_cells, 3)),
                        rng.uniform(0.1, 1, (m.n_cells, 1))], 1)
    return m, g, W, rng.uniform(1, 2, W.shape)


@pytest.mark.parametrize("shape", SIZES)
def test_moves(shape):
    m, g, W, U = make(shape)
    n = m.n_cells
    g.set_state(W, U)
    for a, b in zip(g.get_state(), (W, U)):
        assert np.array_equal(a, b)
    # device arrays that start 8 bytes past an aligned address
    pad = torch.zeros(2, 5 * n + 1, dtype=torch.float64, device="cuda")
    dW, dU = pad[0][1:], pad[1][1:]
    dW.copy_(torch.tensor(W[::-1].copy()).reshape(-1))
    dU.copy_(torch.tensor(U[::-1].copy()).reshape(-1))
    torch.cuda.synchronize()
    L.check(L.lib.rrhd_set_state(g.handle, dW.data_ptr(), dU.data_ptr(), 5, L.RRHD_DEVICE))
    for a, b in zip(g.get_state(), (W[::-1], U[::-1])):
        assert np.array_equal(a, b)
    out = torch.zeros(2, 5 * n + 1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    L.check(L.lib.rrhd_get_state(g.handle, out[0][1:].data_ptr(), out[1][1:].data_ptr(), 5, L.RRHD_DEVICE))
    g.sync()
    assert torch.equal(out[:, 1:], pad[:, 1:]) and not out[:, 0].any()
    # one array, and rows of 8
    g.set_state(W=W)
    wide = torch.full((n, 8), -1.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    L.check(L.lib.rrhd_get_state(g.handle, wide.data_ptr(), None, 8, L.RRHD_DEVICE))
    g.sync()
    assert np.array_equal(wide.cpu().numpy()[:, :5], W) and torch.all(wide[:, 5:] == -1)
    assert np.array_equal(g.get_state()[1], U[::-1])
    g.close()


@pytest.mark.parametrize("shape", SIZES)
def test_reported_steps(shape):
    m, g, W, _ = make(shape)
    tau = 0.1 * m.h_min
    g.set_state_prim(W)
    seen = [rhllc.Hllc3dStab(tau, g) for _ in range(3)]
    state = g.get_state()
    for reported in range(3):  # only one of the steps is reported
        g.set_state_prim(W)
        for k in range(3):
            s = L.StepStats() if k == reported else None
            L.check(L.lib.rrhd_hydro_step(g.handle, tau, ctypes.byref(s) if s is not None else None))
            if s is not None:
                assert (s.max_speed, s.n_fallback, s.n_failed) == (
                    seen[k].max_speed, seen[k].n_fallback, seen[k].n_failed)
        for a, b in zip(g.get_state(), state):
            assert np.array_equal(a, b)
    assert 0 < seen[0].max_speed <= 1
    g.close()
