"""FP64 scattering and moments at the edges of their tiles (rows and directions around multiples of the
tile sizes, every row-tile size, all group counts of the cell-direction-group layout, unaligned arrays).
Reference rounding: bit for bit against the oracle.  One FMA per term: 1e-13 relative, the bar of
test_gpu_radiation.py."""
import numpy as np
import pytest
import torch

import oracle
from cases import intensity
from radrhd_solver_b200 import _lib as L
from radrhd_solver_b200 import illum
from radrhd_solver_b200.mesh import fibonacci_directions

pytestmark = pytest.mark.gpu


def _want(I, d):
    return (oracle.port_scatter(I, d.dirs, d.areas, d.full_area, nthreads=8),
            *oracle.port_moments(I, d.dirs, d.areas, d.full_area, nthreads=8))


@pytest.mark.parametrize("rows,M", [(1, 1), (15, 16), (17, 17), (127, 33), (129, 64), (250, 65), (3000, 31),
                                    (19_000, 96), (19_001, 26), (40_003, 15), (152_000, 7)])
def test_rows_layout(rows, M):
    d = fibonacci_directions(M)
    dg = illum.DirectionGrid(d)
    I = intensity(rows, M, seed=rows)
    S, E, F, T = _want(I, d)
    # one double past a 16-byte boundary: the arrays need no more than their own alignment
    Id = torch.empty(rows * M + 1, dtype=torch.float64, device="cuda")[1:].view(rows, M)
    Id.copy_(torch.tensor(I))
    out = torch.empty(rows * M + 1, dtype=torch.float64, device="cuda")[1:].view(rows, M)
    assert np.array_equal(illum.CalculateIntScattering(dg, Id, out).cpu().numpy(), S)
    fma = illum.CalculateIntScattering(dg, Id, out, exact=False).cpu().numpy()
    assert np.all(np.abs(fma - S) <= 1e-13 * np.abs(S))
    for got, want in zip(illum.CalculateAllParam(dg, Id), (E, F, T)):
        assert np.array_equal(got.cpu().numpy(), want)
    dg.close()


@pytest.mark.parametrize("cells,G,M", [(1, 1, 5), (70, 2, 64), (33, 4, 100), (19, 8, 33), (9, 16, 17), (5, 32, 40),
                                       (3, 64, 66), (2400, 8, 30), (700, 64, 20)])
def test_cell_direction_group_layout(cells, G, M):
    d = fibonacci_directions(M)
    dg = illum.DirectionGrid(d)
    rows = cells * G
    I = intensity(rows, M, seed=cells)
    S, E, F, T = _want(I, d)
    cdg = lambda a: np.ascontiguousarray(a.reshape(cells, G, M).transpose(0, 2, 1))  # noqa: E731
    Id = torch.tensor(cdg(I), device="cuda")
    out = torch.empty_like(Id)
    st = torch.cuda.current_stream().cuda_stream
    L.check(L.lib.rrhd_scatter_fp64_cdg(dg.handle, L.ptr(Id), L.ptr(out), cells, G, 1, st))
    assert np.array_equal(out.cpu().numpy(), cdg(S))
    L.check(L.lib.rrhd_scatter_fp64_cdg(dg.handle, L.ptr(Id), L.ptr(out), cells, G, 0, st))
    assert np.all(np.abs(out.cpu().numpy() - cdg(S)) <= 1e-13 * np.abs(cdg(S)))
    mom = [torch.empty(rows, k, dtype=torch.float64, device="cuda") for k in (1, 3, 9)]
    L.check(L.lib.rrhd_moments_fp64_cdg(dg.handle, L.ptr(Id), *(L.ptr(t) for t in mom), cells, G, st))
    for got, want in zip(mom, (E, F, T)):
        assert np.array_equal(got.cpu().numpy().reshape(want.shape), want)
    dg.close()
