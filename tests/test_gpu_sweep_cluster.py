"""The sweep with several CTAs to a direction (few directions whose slots one cannot hold) against one CTA to each:
the directions of a sweep do not touch one another, so the first ones of a larger set give the same
bits alone, whatever number of CTAs has them."""
import pytest
import torch

from cases import GAMMA_43
from radrhd_solver_b200 import illum, rhllc
from radrhd_solver_b200.mesh import fibonacci_directions, kuhn_box

pytestmark = pytest.mark.gpu


def sweep(m, d, G, precision, bc, arrays, S):
    grid = rhllc.Grid(m, gamma=GAMMA_43)
    dg = illum.DirectionGrid(d)
    sw = illum.TransportSweep(grid, dg, groups=G, precision=precision, boundary_value=bc)
    I = torch.full_like(S, float("nan"))
    torch.cuda.synchronize()
    for _ in range(2):
        illum.CalculateIllum(sw, *arrays, S, I)
    grid.sync()
    grid.close()
    dg.close()
    return I


@pytest.mark.parametrize("G,precision,bc", [(4, "fp64", 0.25), (4, "mixed", 0.0), (7, "fp32", 0.5)])
def test_directions_alone(G, precision, bc):
    m = kuhn_box(48, 47, 49, lo=(-1, -1, -1), hi=(1, 1, 1), seed=41)
    d = fibonacci_directions(75)  # two CTAs for each would be more than there are SMs
    real = torch.float64 if precision == "fp64" else torch.float32
    gen = torch.Generator("cuda").manual_seed(5)
    rand = lambda *n: torch.rand(*n, generator=gen, device="cuda", dtype=torch.float64)
    alpha = 10 ** (2.5 * rand(m.n_cells) - 1)
    arrays = [x.to(real).contiguous() for x in (alpha, 0.5 * alpha, 10 ** (2 * rand(m.n_cells, G) - 2))]
    S = (10 ** (2 * rand(m.n_cells * G, 75) - 3)).to(real).contiguous()
    want = sweep(m, d, G, precision, bc, arrays, S)
    assert torch.isfinite(want).all()
    for n in (1, 9, 19, 37, 74):  # clusters of 8, 8, 4, 4 and 2
        assert torch.equal(sweep(m, d.subset(0, n), G, precision, bc, arrays, S[:, :n].contiguous()), want[:, :n])
