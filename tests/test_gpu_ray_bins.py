"""The binned image-plane trace at the edges of its split: bins a thread tests and bins a warp
takes up, an every-ray list shorter and longer than one shared-memory stage, frames that end
inside a block, surfaces whose bins are dealt to warps one triangle or several at a time.  Every
code is the oracle's; a curve over any number of pixels is the sum in double precision within
1e-13 (a sum of non-negative terms in a fixed order)."""
import os

import numpy as np
import pytest
import torch

import oracle
from cases import ray_surface
from radrhd_solver_b200 import ray_tracing as RT

pytestmark = pytest.mark.gpu


def check(ids, abc, rays, modes=(RT.SURFACE, RT.ROCHE, RT.INNER)):
    rt = RT.RayTracer(RT.face_cells(ids, abc))
    d_rays = torch.tensor(rays, device="cuda")
    for mode in modes:
        want = oracle.port_ray_trace(mode, rays, ids, abc, nthreads=os.cpu_count() or 1)
        assert np.array_equal(rt.trace(d_rays, mode).cpu().numpy(), want)
    rt.close()


def fan(rays, count, seed):
    """count small triangles around one ray of the frame, at random depths, the last two alike."""
    rng = np.random.default_rng(seed)
    o, d = rays[len(rays) // 2 + 150, :3], rays[0, 3:]
    u = np.cross(d, [0.3, 0.5, 0.8])
    u /= np.linalg.norm(u)
    v = np.cross(d, u)
    angle = rng.uniform(0, 2 * np.pi, (count, 1)) + np.array([0, 2.1, 4.2])
    r = rng.uniform(0.001, 0.004, (count, 3))
    depth = rng.uniform(1.0, 3.0, (count, 1)) + rng.uniform(-0.003, 0.003, (count, 3))
    p = o + depth[..., None] * d + (r * np.cos(angle))[..., None] * u + (r * np.sin(angle))[..., None] * v
    p[-1] = p[-2]
    return p.reshape(count, 9)


@pytest.mark.parametrize("count", [2, 31, 32, 33, 64, 65, 129, 1000])
def test_long_bins(count):
    rays = RT.MakeRays(7)
    ids, abc = ray_surface(4, 6)
    abc = np.concatenate([abc, fan(rays, count, count)])
    ids = np.concatenate([ids, 4 * len(abc) + np.arange(count)]).astype(np.int32)
    check(ids, abc, rays)


@pytest.mark.parametrize("count", [63, 64, 65, 130])
def test_every_ray_list(count):
    """Slivers, which every ray tests."""
    rays = RT.MakeRays(7)
    rng = np.random.default_rng(count)
    a = rng.uniform([0.5, -0.3, -0.2], [1.3, 0.3, 0.2], (count, 3))
    e = rng.normal(size=(count, 3)) * 0.3
    abc = np.concatenate([a, a + e, a + e * 1.01 + rng.normal(size=(count, 3)) * 1e-5], 1)
    check(np.arange(count, dtype=np.int32), abc, rays, (RT.SURFACE,))


@pytest.mark.parametrize("M", [1, 31, 127, 128, 129, 8191, 8192, 8193, 65537])
def test_ragged_frames_and_curves(M):
    rays = RT.MakeRays(7)[:: 180000 // M][:M].copy()
    ids, abc = ray_surface(6, 8)
    check(ids, abc, rays)
    rng = np.random.default_rng(M)
    codes = torch.tensor(rng.integers(-4, 400, M).astype(np.int32), device="cuda")
    values = rng.uniform(0.5, 2.0, 100)
    image, curve = RT.RayTracer.image(codes, torch.tensor(values, device="cuda"))
    c = codes.cpu().numpy()
    want = np.select([c == -1, c == -4, c == -2, c == -3], [0.0, 1e-5, 5.0, 10.0], default=values[np.maximum(c, 0) // 4])
    assert np.array_equal(image.cpu().numpy(), want)
    assert curve == pytest.approx(np.sum(want * RT.PIXEL_AREA), rel=1e-13, abs=0)


@pytest.mark.parametrize("n", [1, 31, 33, 8191, 8193])
def test_surface_sizes(n):
    rays = RT.MakeRays(11)[::7].copy()
    ids, abc = ray_surface(32, 32)
    pick = np.random.default_rng(n).permutation(len(abc))[:n]
    check(np.ascontiguousarray(ids[pick]), np.ascontiguousarray(abc[pick]), rays, (RT.SURFACE,))
