"""The sweep and the coupled step with little device memory left: an allocation that does not fit is an error
that leaves the context as it was, and memory the sweep can do without is given back before one is reported.
A mesh of 24,576 cells and 256 directions in double: an array of the intensity's size is 50 MB a group.
Same values are asked for bit for bit: neither the scratch nor the geometry stream changes an operation."""
import ctypes as C

import numpy as np
import pytest
import torch

from cases import GAMMA_43
from radrhd_solver_b200 import _lib as L
from radrhd_solver_b200 import illum, rad_rhd, rhllc
from radrhd_solver_b200.mesh import fibonacci_directions, kuhn_box

pytestmark = pytest.mark.gpu
M = 256
MB = 2 ** 20


def leave(megabytes):
    """Holds all but this much of the device's free memory."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(free - megabytes * MB, dtype=torch.uint8, device="cuda")


@pytest.fixture(scope="module")
def mesh():
    return kuhn_box(16, 16, 16, lo=(-1, -1, -1), hi=(1, 1, 1), seed=51)


class Context:
    def __init__(self, m, G, precision="fp64"):
        W = np.zeros((m.n_cells, 5))
        W[:, 0] = 10 ** np.random.default_rng(52).uniform(-1, 1, m.n_cells)
        W[:, 4] = 0.1
        self.m = m
        self.grid = rhllc.Grid(m, gamma=GAMMA_43)
        self.grid.set_state_prim(W)
        self.dg = illum.DirectionGrid(fibonacci_directions(M))
        self.sw = illum.TransportSweep(self.grid, self.dg, groups=G, precision=precision)
        self.step = rad_rhd.RadRHDStep(self.sw, em=rad_rhd.emission(1.0, 10.0),
                                       scatter="fp64" if precision == "fp64" else "f16x3")

    def steps(self):
        for _ in range(2):
            self.step(1e-2 * self.m.h_min)
        self.grid.sync()

    def close(self):
        self.grid.close()
        self.dg.close()


def test_coupled_arrays_all_or_none(mesh):
    """8 groups: arrays of 402 MB.  The intensity is there (the sweep's scratch), the scattering integral does
    not fit, not even with the stream's 277 MB given back; the next calls find nothing that this one left behind
    (the intensity fits, then)."""
    c = Context(mesh, 8)
    S = 10 ** np.random.default_rng(53).uniform(-3, -1, (mesh.n_cells * 8, M))
    held = leave(100)
    for _ in range(2):
        assert L.lib.rrhd_rad_set(c.grid.handle, L.RRHD_RAD_S, L.ptr(S)) == L.RRHD_ERR_OOM
        assert L.lib.rrhd_rad_get(c.grid.handle, L.RRHD_RAD_S, L.ptr(np.empty_like(S))) == L.RRHD_ERR_STATE
        assert L.lib.rrhd_coupled_step(c.grid.handle, 1e-3, C.byref(c.step.opts), None, None) == L.RRHD_ERR_OOM
    del held
    torch.cuda.empty_cache()
    c.step.set("S", S)
    assert np.array_equal(c.step.get("S"), S)
    c.close()


@pytest.mark.parametrize("megabytes", [60, 320])
def test_coupled_step_takes_the_sweeps_memory(mesh, megabytes):
    """4 groups: a sweep has made its scratch of 201 MB, and what is free holds less than the coupled step's
    two arrays: with the scratch (320 MB free) or the scratch and the stream (60 MB) given back it does."""
    want = Context(mesh, 4)
    want.steps()
    c = Context(mesh, 4)
    rows, n = mesh.n_cells * 4, mesh.n_cells
    one = [torch.ones(n, dtype=torch.float64, device="cuda") for _ in range(2)]
    q, S = (torch.ones(x, dtype=torch.float64, device="cuda") for x in ((n, 4), (rows, M)))
    torch.cuda.synchronize()
    illum.CalculateIllum(c.sw, *one, q, S)
    c.grid.sync()
    del one, q, S
    held = leave(megabytes)
    c.steps()
    del held
    torch.cuda.empty_cache()
    for what in ("I", "S", "G4", "MOM"):
        assert np.array_equal(c.step.get(what), want.step.get(what))
    for a, b in zip(c.grid.get_state(), want.grid.get_state()):
        assert np.array_equal(a, b)
    c.close()
    want.close()


@pytest.mark.parametrize("precision,G", [("fp64", 4), ("mixed", 3)])
def test_transfers_in_pieces(mesh, precision, G):
    """I and S to and from the host with less free than one of them takes (201 and 151 MB of doubles)."""
    c = Context(mesh, G, precision)
    rng = np.random.default_rng(54)
    values = [rng.uniform(0, 1, (mesh.n_cells * G, M)).astype(np.float32).astype(np.float64) for _ in range(2)]
    c.step.set("I", values[0])
    held = leave(20)
    assert np.array_equal(c.step.get("I"), values[0])
    c.step.set("S", values[1])
    assert np.array_equal(c.step.get("S"), values[1])
    assert np.array_equal(c.step.get("I"), values[0])
    del held
    torch.cuda.empty_cache()
    assert np.array_equal(c.step.get("S"), values[1])
    c.close()


@pytest.mark.parametrize("G,megabytes,dirs", [(4, 60, M), (8, 20, M // 2)])
def test_scratch_takes_the_streams_memory(mesh, G, megabytes, dirs):
    """A sweep after a coupled step, which has taken the scratch: it is made again from the stream's memory, of
    all directions (4 groups: 201 MB against 60 free and 151 of weights) or of half of them (8 groups: 402 MB,
    20 free, 277 of weights and stream)."""
    rows, n = mesh.n_cells * G, mesh.n_cells
    gen = torch.Generator("cuda").manual_seed(55)
    rand = lambda *s: torch.rand(*s, generator=gen, device="cuda", dtype=torch.float64)
    x = [rand(n) + 0.1, rand(n), rand(n, G), rand(rows, M)]
    torch.cuda.synchronize()
    fresh = Context(mesh, G)
    want = illum.CalculateIllum(fresh.sw, *x)
    fresh.grid.sync()
    fresh.close()
    c = Context(mesh, G)
    c.steps()
    assert c.sw.plan_form()["scratch_dirs"] == 0 and c.sw.plan_form()["stream"] == 2
    I = torch.empty_like(x[3])
    held = leave(megabytes)
    illum.CalculateIllum(c.sw, *x, I)
    c.grid.sync()
    assert c.sw.plan_form()["scratch_dirs"] == dirs and c.sw.plan_form()["stream"] < 2
    del held
    torch.cuda.empty_cache()
    assert torch.equal(I, want)
    c.close()
