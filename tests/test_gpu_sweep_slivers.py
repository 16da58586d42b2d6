"""The sweep on tetrahedra whose out-face is a small part of their surface, against the FP64 oracle.

A needle with its base up, seen from below, has three in-faces and one out-face of some 1e-6 of the
surface; where nothing enters, the cell's value is that face's alone, and its weight has to hold all
its digits: one minus the others' would be off by 2^-53 / 1e-6 = 1e-10.  Among the cells: base triangles of
all shapes, local face orders of all kinds, and flat ones, whose out-face is the largest.  Bars: 1e-12 relative in double, 1e-7 (one float rounding of I) in mixed
precision and 1e-5 in float, as in test_gpu_sweep.py."""
import numpy as np
import pytest
import torch

import oracle
from cases import GAMMA_43
from radrhd_solver_b200 import illum, rhllc
from radrhd_solver_b200.mesh import Directions, Mesh

pytestmark = pytest.mark.gpu


def single_cells(corners):
    """A mesh of tetrahedra without neighbours: corners [N, 4, 3], face j opposite corner j."""
    n = len(corners)
    normal, area = np.zeros((n, 4, 3)), np.zeros((n, 4))
    for j in range(4):
        a, b, c = (corners[:, (j + k) % 4] for k in (1, 2, 3))
        x = np.cross(b - a, c - a)
        area[:, j] = 0.5 * np.linalg.norm(x, axis=1)
        x /= np.linalg.norm(x, axis=1, keepdims=True)
        outward = np.einsum("ij,ij->i", x, a - corners[:, j]) > 0
        normal[:, j] = np.where(outward[:, None], x, -x)
    volume = np.abs(np.einsum("ij,ij->i", corners[:, 1] - corners[:, 0],
                              np.cross(corners[:, 2] - corners[:, 0], corners[:, 3] - corners[:, 0]))) / 6
    return Mesh(np.repeat(np.arange(n, dtype=np.int32), 4), np.full(4 * n, -1, np.int32),
                np.ascontiguousarray(normal.reshape(-1, 3)), area.reshape(-1),
                np.arange(4 * n, dtype=np.int32).reshape(n, 4), np.full(n, 15, np.uint8), volume,
                np.ascontiguousarray(corners.mean(1)), h_min=1e-9)


def needles(n, width, height, seed):
    """Base triangles of the given width around (0, 0, height) over a tip at the origin (cells without
    neighbours may lie in one another)."""
    rng = np.random.default_rng(seed)
    phi = 2 * np.pi * (np.array([0, 1, 2]) / 3 + rng.uniform(-0.12, 0.12, (n, 3)))
    r = width * rng.uniform(0.3, 1.0, (n, 3))
    base = np.stack([r * np.cos(phi), r * np.sin(phi), np.full((n, 3), height)], -1)
    corners = np.concatenate([base, np.zeros((n, 1, 3))], 1)
    return np.stack([q[rng.permutation(4)] for q in corners])


def directions(tilt):
    w = np.array([[0, 0, 1.0], [tilt, 0, 1.0], [-tilt, 2 * tilt, 1.0], [0, 0, -1.0]])
    w /= np.linalg.norm(w, axis=1, keepdims=True)
    return Directions(np.ascontiguousarray(w), np.full(len(w), 4 * np.pi / len(w)), 4 * np.pi)


def slim(n, width, seed):
    """Tetrahedra over a tip below the middle of a base with one short side: the third in-face is small."""
    rng = np.random.default_rng(seed)
    a, b = rng.uniform(0.5, 1, (n, 2)), -rng.uniform(0.5, 1, (n, 2))
    c = b + width * rng.uniform(-1, 1, (n, 2))
    mid = (a + b + c) / 3
    z = np.ones((n, 1))
    corners = np.stack([np.hstack([x, y * z]) for x, y in ((a, 1), (b, 1), (c, 1), (mid, 0))], 1)
    return np.stack([q[rng.permutation(4)] for q in corners])


@pytest.mark.parametrize("bc", [0.0, 0.25])
@pytest.mark.parametrize("precision,width,bar", [("fp64", 1e-6, 1e-12), ("mixed", 1e-6, 1e-7), ("fp32", 1e-3, 1e-5)])
def test_small_out_faces(precision, width, bar, bc):
    corners = needles(240, width, 1.0, 61)
    corners[::4] = needles(240, 1.0, 0.2, 62)[::4]  # flat cells: the out-face is the largest
    check(corners, directions(0.02 * width), precision, bar, bc)


@pytest.mark.parametrize("bc", [0.0, 0.25])
@pytest.mark.parametrize("precision,bar", [("fp64", 1e-12), ("mixed", 1e-7), ("fp32", 1e-5)])
def test_small_third_in_face(precision, bar, bc):
    """Weights of 0.001 to 0.3 among the in-faces."""
    corners = np.concatenate([slim(120, 0.05, 64), slim(120, 0.5, 65)])
    check(corners, directions(0.01), precision, bar, bc)


def check(corners, d, precision, bar, bc):
    n, G = len(corners), 2
    m = single_cells(corners)
    real = np.float64 if precision == "fp64" else np.float32
    rng = np.random.default_rng(63)
    alpha = 10 ** rng.uniform(0.5, 1.5, n)  # no thin cells: 1 - exp(-k t) has its digits as well
    inputs = [np.ascontiguousarray(x.astype(real)) for x in
              (alpha, 0.5 * alpha, 10 ** rng.uniform(-2, 0, (n, G)), 10 ** rng.uniform(-3, -1, (n * G, d.size)))]
    want, missing = oracle.port_sweep(m, d.dirs, *(x.astype(np.float64) for x in inputs), bc=bc)
    assert missing == 0
    grid = rhllc.Grid(m, gamma=GAMMA_43)
    dg = illum.DirectionGrid(d)
    sw = illum.TransportSweep(grid, dg, groups=G, precision=precision, boundary_value=bc)
    t = [torch.tensor(x, device="cuda") for x in inputs]
    torch.cuda.synchronize()
    got = illum.CalculateIllum(sw, *t)
    grid.sync()
    got = got.double().cpu().numpy()
    grid.close()
    dg.close()
    assert np.max(np.abs(got - want) / np.abs(want)) <= bar
