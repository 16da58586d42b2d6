"""Row pre-pass of the scaled tensor-core forms (FP64 matrix instruction) and the drain's stores, at the
edges of their layout rules: few rows (four warps a task) and many (a warp a task, more than the grid), rows
that fill no task, every direction count and group count, arrays 16 but not 32 bytes aligned, negative and
zero intensities.  Moments: an FP64 sum stored as FP32, so half an ulp of FP32 (2^-24) relative to the sum of
the terms' sizes, and of the FP64 sums (M 2^-53) less.  S: 1e-6 relative, the bar of test_gpu_scatter_tc.py."""
import numpy as np
import pytest
import torch

from radrhd_solver_b200 import _lib as L
from radrhd_solver_b200 import illum
from radrhd_solver_b200.mesh import fibonacci_directions

pytestmark = pytest.mark.gpu


def _basis(d):
    w, a = d.dirs, d.areas / d.full_area
    x, y, z = w.T
    return a[:, None] * np.stack([np.ones_like(x), x, y, z, x * x, x * y, x * z, y * y, y * z, z * z], 1)


def _run(dg, form, I, groups, moments=True):
    """I: float32 [rows, M] numpy -> S [rows, M], moments, through the layout of `groups`, off a 32-byte boundary."""
    rows, M = I.shape
    cdg = np.ascontiguousarray(I.reshape(rows // groups, groups, M).transpose(0, 2, 1))
    Id = torch.empty(I.size + 4, dtype=torch.float32, device="cuda")[4:]
    Sd = torch.full((I.size + 4,), float("nan"), dtype=torch.float32, device="cuda")[4:]
    Id.copy_(torch.tensor(cdg).reshape(-1))
    mom = torch.full((rows, 16), float("nan"), dtype=torch.float32, device="cuda") if moments else None
    tc = illum.ScatterTC(dg, form)
    st = torch.cuda.current_stream().cuda_stream
    if groups == 1:
        L.check(L.lib.rrhd_scatter_tc_run(tc._h, Id.data_ptr(), Sd.data_ptr(), L.ptr(mom), rows, st))
    else:
        L.check(L.lib.rrhd_scatter_tc_run_cdg(tc._h, Id.data_ptr(), Sd.data_ptr(), L.ptr(mom), rows // groups, groups, st))
    tc.check()
    S = Sd.cpu().numpy().reshape(cdg.shape).transpose(0, 2, 1).reshape(rows, M)
    return S, mom.cpu().numpy() if moments else None


@pytest.mark.parametrize("rows,M,groups", [(1, 64, 1), (31, 128, 1), (33, 256, 1), (600, 512, 1), (129, 1024, 1),
                                           (2, 128, 2), (66, 256, 2), (4, 256, 4), (132, 64, 4), (1004, 512, 4),
                                           (40_001, 64, 1), (90_002, 128, 2), (80_004, 64, 4)])
@pytest.mark.parametrize("form", ["f16x3", "bf16x3"])
def test_prepass_and_stores(rows, M, groups, form):
    d = fibonacci_directions(M)
    dg = illum.DirectionGrid(d)
    rng = np.random.default_rng(rows + M)
    I = np.exp(rng.normal(0, 1, (rows, M))).astype(np.float32)
    I[0] = 0.0
    if rows > 5:
        I[5] *= np.float32(1e-20)
    S, mom = _run(dg, form, I, groups)
    mu = d.dirs @ d.dirs.T
    K = (d.areas / d.full_area)[:, None] * 0.75 * (1 + mu * mu)
    pick = np.unique(np.concatenate([np.arange(min(rows, 200)), np.arange(max(0, rows - 200), rows)]))
    I64 = I[pick].astype(np.float64)
    want = I64 @ K
    tol = 1e-6 if form == "f16x3" else 2e-5  # the split-bf16 form's own bar is 1e-5 over its cases
    assert np.all(np.abs(S[pick] - want) <= tol * np.abs(want))
    B = _basis(d)
    size = np.abs(I64) @ np.abs(B)
    if form == "f16x3":
        assert np.all(np.abs(mom[pick, :10] - I64 @ B) <= (2.0 ** -24 + M * 2.0 ** -53) * size)
    assert np.all(mom[:, 10:] == 0)
    S2, _ = _run(dg, form, I, groups, moments=False)
    assert np.array_equal(S2, S) if form == "f16x3" else np.all(np.abs(S2[pick] - want) <= tol * np.abs(want))
    dg.close()


def test_prepass_signed_and_non_finite():
    """A negative intensity is summed as it is; an infinite one leaves no finite value in its row and changes no other."""
    M = 128
    d = fibonacci_directions(M)
    dg = illum.DirectionGrid(d)
    rng = np.random.default_rng(9)
    I = rng.normal(0, 1, (300, M)).astype(np.float32)
    I[7, 3] = np.inf
    S, mom = _run(dg, "f16x3", I, 1)
    fine = np.arange(300) != 7
    B = _basis(d)
    I64 = I[fine].astype(np.float64)
    assert np.all(np.abs(mom[fine, :10] - I64 @ B) <= (2.0 ** -24 + M * 2.0 ** -53) * (np.abs(I64) @ np.abs(B)))
    mu = d.dirs @ d.dirs.T
    K = (d.areas / d.full_area)[:, None] * 0.75 * (1 + mu * mu)
    assert np.all(np.abs(S[fine] - I64 @ K) <= 1e-6 * (np.abs(I64) @ K))
    assert not np.any(np.isfinite(S[7]))
    dg.close()
