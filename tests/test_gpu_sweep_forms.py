"""Every form the sweep takes, asked for and seen to be the one that ran (rrhd_rad_plan_form): values beyond a
CTA's shared memory with one CTA an SM, with two and with slots beyond 16 bits, several CTAs a direction, all of
the geometry stream, its first part and none, scratch of all directions, of some and of one, and plans built in
several passes.  Against the FP64 oracle (1e-12 relative, the bar of test_gpu_sweep.py), or bit for bit where two
forms of the same sweep are compared: neither memory nor the order of directions changes an operation."""
import numpy as np
import pytest
import torch

import oracle
from cases import GAMMA_43
from radrhd_solver_b200 import illum, rhllc
from radrhd_solver_b200.mesh import Directions, fibonacci_directions, kuhn_box

pytestmark = pytest.mark.gpu


def box(*shape):
    return kuhn_box(*shape, lo=(-1, -1, -1), hi=(1, 1, 1), seed=31)


def inputs_of(m, M, G, precision, seed=32):
    rng = np.random.default_rng(seed)
    real = np.float64 if precision == "fp64" else np.float32
    alpha = 10 ** rng.uniform(-1, 1.5, m.n_cells)
    return [np.ascontiguousarray(x.astype(real)) for x in (alpha, 0.5 * alpha, 10 ** rng.uniform(-2, 0, (m.n_cells, G)),
                                                          10 ** rng.uniform(-3, -1, (m.n_cells * G, M)))]


def sweep(m, d, G, precision, inputs, bc=0.0, memory=-1, levels=False):
    """Two sweeps of a context that may keep `memory` bytes beyond its plan -> I, the form, plan levels."""
    grid = rhllc.Grid(m, gamma=GAMMA_43)
    illum.limit_sweep_memory(grid, memory)
    dg = illum.DirectionGrid(d)
    sw = illum.TransportSweep(grid, dg, groups=G, precision=precision, boundary_value=bc)
    t = [torch.tensor(x, device="cuda") for x in inputs]
    I = torch.full_like(t[3], float("nan"))
    torch.cuda.synchronize()
    for _ in range(2):
        illum.CalculateIllum(sw, *t, I)
    grid.sync()
    form, lv = sw.plan_form(), sw.plan_levels() if levels else None
    grid.close()
    dg.close()
    return I.cpu().numpy(), form, lv


def bytes_of(m, M, G, precision):
    """A direction's scratch and the stream's first part."""
    return (8 if precision == "fp64" else 4) * m.n_cells * G, (12 if precision == "fp32" else 20) * m.n_cells * M


@pytest.mark.parametrize("shape,M,two", [((12, 11, 12), 75, False), ((8, 8, 8), 149, True), ((7, 7, 7), 149, True)])
def test_slots_in_both_memories(shape, M, two):
    """64 groups: 452 slots fit a CTA's shared memory, 226 that of one of two."""
    m, d, G = box(*shape), fibonacci_directions(M), 64
    inputs = inputs_of(m, M, G, "fp64")
    got, form, _ = sweep(m, d, G, "fp64", inputs, bc=0.3)
    assert form["cluster"] == 1 and form["ctas_per_sm"] == (2 if two else 1) and not form["wide_slots"]
    assert form["slots_shared"] == (226 if two else 452) and form["slots_global"] > 40
    want, missing = oracle.port_sweep(m, d.dirs, *inputs, bc=0.3)
    assert missing == 0
    assert np.max(np.abs(got - want) / np.abs(want)) <= 1e-12


def test_wide_slots_with_and_without_a_cluster():
    """A plate one hex thick swept through its thickness: the front is the whole plate."""
    m = kuhn_box(210, 210, 1, lo=(-1, -1, 0), hi=(1, 1, 0.01), jitter=0.1, seed=33)
    w = np.array([[0.02, 0.01, 1.0], [0.01, -0.03, -1.0]] * 38)[:75]
    w /= np.linalg.norm(w, axis=1, keepdims=True)
    d = Directions(w, np.full(75, 4 * np.pi / 75), 4 * np.pi)
    inputs = inputs_of(m, 75, 1, "fp64")
    many, form, _ = sweep(m, d, 1, "fp64", inputs)
    assert form["wide_slots"] and form["cluster"] == 1 and form["slots_shared"] > 20000 and form["slots_global"] > 20000
    few, form, _ = sweep(m, d.subset(0, 2), 1, "fp64", inputs[:3] + [np.ascontiguousarray(inputs[3][:, :2])])
    assert form["wide_slots"] and form["cluster"] > 1
    assert np.array_equal(many[:, :2], few)
    want, missing = oracle.port_sweep(m, d.dirs[:2], *inputs[:3], inputs[3][:, :2])
    assert missing == 0
    assert np.max(np.abs(few - want) / np.abs(want)) <= 1e-12


@pytest.mark.parametrize("shape,M,G,precision,cluster", [((10, 9, 10), 8, 64, "fp64", 2), ((90, 90, 1), 2, 2, "fp64", 2),
                                                         ((210, 210, 1), 2, 1, "fp64", 8)])
def test_clusters_of_every_size(shape, M, G, precision, cluster):
    m = box(*shape) if shape[2] > 1 else kuhn_box(*shape, lo=(-1, -1, 0), hi=(1, 1, 0.01), jitter=0.1, seed=33)
    d = fibonacci_directions(M)
    if shape[2] == 1:
        w = np.array([[0.02, 0.01, 1.0], [0.01, -0.03, -1.0]])
        d = Directions(w / np.linalg.norm(w, axis=1, keepdims=True), np.full(2, 2 * np.pi), 4 * np.pi)
    inputs = inputs_of(m, M, G, precision)
    got, form, _ = sweep(m, d, G, precision, inputs, bc=0.2)
    assert form["cluster"] == cluster
    want, missing = oracle.port_sweep(m, d.dirs, *inputs, bc=0.2)
    assert missing == 0
    assert np.max(np.abs(got - want) / np.abs(want)) <= 1e-12


def test_cluster_of_four():
    """Against one CTA a direction: the first directions of a larger set give the same bits alone."""
    m, d = box(64, 64, 64), fibonacci_directions(75)
    inputs = inputs_of(m, 75, 1, "fp64")
    many, form, _ = sweep(m, d, 1, "fp64", inputs)
    assert form["cluster"] == 1
    few, form, _ = sweep(m, d.subset(0, 8), 1, "fp64", inputs[:3] + [np.ascontiguousarray(inputs[3][:, :8])])
    assert form["cluster"] == 4
    assert np.array_equal(many[:, :8], few)


SPILLED = ((11, 11, 11), 75, 64)   # beyond one CTA's shared memory
SHARED_SM = ((7, 7, 7), 149, 64)   # ... of two CTAs an SM
CLUSTER = ((10, 9, 10), 8, 64)     # several CTAs a direction


@pytest.mark.parametrize("shape,M,G,precision", [
    ((9, 8, 7), 33, 1, "fp64"), ((9, 8, 7), 33, 2, "fp64"), ((9, 8, 7), 33, 4, "fp64"), ((9, 8, 7), 33, 3, "fp64"),
    ((9, 8, 7), 33, 1, "mixed"), ((9, 8, 7), 33, 2, "mixed"), ((9, 8, 7), 33, 4, "mixed"), ((9, 8, 7), 33, 5, "mixed"),
    ((9, 8, 7), 33, 1, "fp32"), ((9, 8, 7), 33, 2, "fp32"), ((9, 8, 7), 33, 4, "fp32"), ((9, 8, 7), 33, 3, "fp32"),
    SPILLED + ("fp64",), SHARED_SM + ("fp64",), CLUSTER + ("fp64",), CLUSTER + ("mixed",),
    ((15, 14, 15), 8, 64, "fp32")])
def test_geometry_kept_or_formed_again(shape, M, G, precision):
    m, d = box(*shape), fibonacci_directions(M)
    inputs = inputs_of(m, M, G, precision)
    x, geo = bytes_of(m, M, G, precision)
    want, full, _ = sweep(m, d, G, precision, inputs, bc=0.25)
    assert full["stream"] == 2 and full["scratch_dirs"] == M
    if (shape, M, G) in (SPILLED, SHARED_SM):
        assert full["slots_global"] > 0 and full["cluster"] == 1
    if M == 8:
        assert full["cluster"] > 1
    if precision == "fp64":
        ref, missing = oracle.port_sweep(m, d.dirs, *inputs, bc=0.25)
        assert missing == 0
        assert np.max(np.abs(want - ref) / np.abs(ref)) <= 1e-12
    some, form, _ = sweep(m, d, G, precision, inputs, bc=0.25, memory=x * M + geo)
    assert form["stream"] == (2 if precision == "fp32" else 1) and form["scratch_dirs"] == M
    assert np.array_equal(some, want)
    none, form, _ = sweep(m, d, G, precision, inputs, bc=0.25, memory=x * M)
    assert form["stream"] == 0 and form["scratch_dirs"] == M and form["ctas_per_sm"] == 1
    assert np.array_equal(none, want)


@pytest.mark.parametrize("G,precision", [(1, "fp64"), (4, "mixed"), (3, "fp32")])
def test_scratch_and_build_of_some_directions(G, precision):
    M = 160
    m, d = box(6, 5, 7), fibonacci_directions(M)
    inputs = inputs_of(m, M, G, precision)
    x, geo = bytes_of(m, M, G, precision)
    want, full, levels = sweep(m, d, G, precision, inputs, levels=True)
    assert full["scratch_dirs"] == M and full["build_dirs"] == M
    run = 148 * full["ctas_per_sm"] if full["ctas_per_sm"] == 1 else M
    for memory, dirs, stream in ((x * run + geo, run, None), (x * 40, 40, 0), (28 * m.n_cells * 7, None, 0), (0, 1, 0)):
        got, form, lv = sweep(m, d, G, precision, inputs, memory=memory, levels=True)
        assert dirs is None or form["scratch_dirs"] == dirs
        assert stream is None or form["stream"] == stream
        assert form["build_dirs"] == max(1, min(M, memory // (28 * m.n_cells)))
        assert np.array_equal(got, want) and np.array_equal(lv, levels)


def test_memory_given_back_and_taken_again():
    M, G = 64, 2
    m, d = box(6, 6, 6), fibonacci_directions(M)
    inputs = inputs_of(m, M, G, "fp64")
    x, geo = bytes_of(m, M, G, "fp64")
    grid = rhllc.Grid(m, gamma=GAMMA_43)
    dg = illum.DirectionGrid(d)
    sw = illum.TransportSweep(grid, dg, groups=G)
    t = [torch.tensor(a, device="cuda") for a in inputs]
    torch.cuda.synchronize()
    want = illum.CalculateIllum(sw, *t)
    seen = []
    for memory in (x * M + geo, geo, x * 3, 0, -1):
        illum.limit_sweep_memory(grid, memory)
        I = illum.CalculateIllum(sw, *t)
        grid.sync()
        assert torch.equal(I, want)
        f = sw.plan_form()
        seen.append((f["stream"], f["scratch_dirs"]))
    assert seen[0][0] <= 1 and seen[3] == (0, 1) and seen[4] == (2, M)
    assert all(s[1] >= 1 for s in seen)
    grid.close()
    dg.close()
