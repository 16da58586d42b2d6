"""The sweep kernel at the edges of its layout rules, against the FP64 oracle: directions per SM (one or
two CTAs), group counts with and without a compile-time kernel, slots in shared memory, beyond it and
beyond 16 bits, the sweep without its geometry stream, and the arrays of the coupled step (through the
sweep's own layout, or read in place).  Tolerances: 1e-12 relative in double, 1e-7 (one float rounding
of S and of I) in mixed precision, the bars of test_gpu_sweep.py."""
import numpy as np
import pytest
import torch

import oracle
from cases import GAMMA_43
from radrhd_solver_b200 import illum, rad_rhd, rhllc
from radrhd_solver_b200.mesh import Directions, fibonacci_directions, kuhn_box

pytestmark = pytest.mark.gpu


def _inputs(m, M, G, seed):
    rng = np.random.default_rng(seed)
    alpha = 10 ** rng.uniform(-1, 1.5, m.n_cells)
    return (alpha, 0.5 * alpha, 10 ** rng.uniform(-2, 0, (m.n_cells, G)),
            10 ** rng.uniform(-3, -1, (m.n_cells * G, M)))


def _sweep(m, d, G, inputs, bc=0.0):
    grid = rhllc.Grid(m, gamma=GAMMA_43)
    dg = illum.DirectionGrid(d)
    sw = illum.TransportSweep(grid, dg, groups=G, precision="fp64", boundary_value=bc)
    t = [torch.tensor(a, dtype=torch.float64, device="cuda").contiguous() for a in inputs]
    I = torch.full_like(t[3], float("nan"))
    torch.cuda.synchronize()
    illum.CalculateIllum(sw, *t, I)
    grid.sync()
    out = I.cpu().numpy()
    grid.close()
    dg.close()
    return out


def _check(m, d, G, seed, bc=0.0):
    inputs = _inputs(m, d.size, G, seed)
    want, missing = oracle.port_sweep(m, d.dirs, *inputs, bc=bc)
    assert missing == 0
    got = _sweep(m, d, G, inputs, bc)
    assert np.max(np.abs(got - want) / np.abs(want)) <= 1e-12


@pytest.mark.parametrize("shape,M,G,bc", [
    ((1, 1, 1), 1, 1, 0.0),      # six cells, one direction
    ((1, 1, 3), 33, 1, 0.5),     # levels of a few cells
    ((5, 4, 6), 148, 2, 0.25),   # one CTA per SM
    ((5, 4, 6), 149, 2, 0.25),   # two CTAs per SM
    ((4, 5, 3), 40, 3, 0.1),     # group loop
    ((9, 8, 7), 8, 4, 0.0),
    ((12, 11, 12), 6, 64, 0.3),  # 64 groups: slots beyond a CTA's shared memory (452 of them)
])
def test_sweep_layouts(shape, M, G, bc):
    m = kuhn_box(*shape, lo=(-1, -1, -1), hi=(1, 1, 1), seed=31)
    _check(m, fibonacci_directions(M), G, 32, bc)


def test_sweep_slots_beyond_16_bits():
    """A plate one hex thick swept through its thickness: the front is the whole plate."""
    m = kuhn_box(210, 210, 1, lo=(-1, -1, 0), hi=(1, 1, 0.01), jitter=0.1, seed=33)
    w = np.array([[0.02, 0.01, 1.0], [0.01, -0.03, -1.0]])
    w /= np.linalg.norm(w, axis=1, keepdims=True)
    _check(m, Directions(w, np.full(2, 2 * np.pi), 4 * np.pi), 1, 34)


def test_sweep_without_geometry_stream():
    """With little memory free the plan keeps no geometry stream; the sweep forms the same values itself."""
    m = kuhn_box(12, 12, 12, lo=(-1, -1, -1), hi=(1, 1, 1), seed=35)
    d, G = fibonacci_directions(24), 64
    inputs = _inputs(m, d.size, G, 36)
    full = _sweep(m, d, G, inputs)
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    # the stream (10 MB) and three arrays of the intensity's size (127 MB each) must not fit, the rest must
    fill = torch.empty(free - 127 * 2**20 - 360 * 2**20, dtype=torch.uint8, device="cuda")
    lean = _sweep(m, d, G, inputs)
    del fill
    torch.cuda.empty_cache()
    assert np.array_equal(lean, full)


@pytest.mark.parametrize("precision,G", [("fp64", 1), ("fp64", 2), ("fp64", 4), ("fp64", 8), ("mixed", 1),
                                         ("mixed", 2), ("mixed", 4)])
def test_coupled_sweep_layouts(precision, G):
    """The intensity of one coupled step with a given scattering integral and no emission (so no source
    term: the state after the step is the state the opacities were taken from)."""
    m = kuhn_box(6, 5, 4, lo=(-1, -1, -1), hi=(1, 1, 1), seed=37)
    d = fibonacci_directions(64)
    rng = np.random.default_rng(38)
    W = np.zeros((m.n_cells, 5))
    W[:, 0] = 10 ** rng.uniform(-1, 1, m.n_cells)
    W[:, 4] = 0.1
    S = 10 ** rng.uniform(-3, -1, (m.n_cells * G, d.size))
    if precision == "mixed":
        S = S.astype(np.float32).astype(np.float64)
    grid = rhllc.Grid(m, gamma=GAMMA_43)
    grid.set_state_prim(W)
    dg = illum.DirectionGrid(d)
    sw = illum.TransportSweep(grid, dg, groups=G, precision=precision)
    step = rad_rhd.RadRHDStep(sw, em=rad_rhd.emission(1.0, 0.0), scatter="fp64" if precision == "fp64" else "f16x3")
    step.set("S", S)
    step(1e-3 * m.h_min)
    grid.sync()
    rho = grid.get_state()[0][:, 0]
    want, missing = oracle.port_sweep(m, d.dirs, rho, 0.5 * rho, np.zeros((m.n_cells, G)), S)
    assert missing == 0
    got = step.get("I")
    grid.close()
    dg.close()
    # opacities are compared through a state that went through con2prim once more: 1e-11 of the pressure scale
    assert np.max(np.abs(got - want) / np.abs(want)) <= (1e-10 if precision == "fp64" else 1e-7)
