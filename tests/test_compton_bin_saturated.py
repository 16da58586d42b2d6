"""The bin estimate of the full-spectrum Compton kernel in the form it computes
(radrhd_solver_b200/csrc/compton.cu, frq_slot): (t / 100.4)^2 by one saturating FMA, 100 - rint(t)
read from the low bits of t 100.4 + 1.5 2^23.  The same operations in FP32 on the CPU, log2 off by
its error bound either way, give the exact count of edges below x or one less; anything that is
not a positive number still gives a slot of the padded row."""
import numpy as np
import pytest

import oracle

T = 100.4
kBLn2 = np.float32(350.0 * 0.69314718055994530942 / (T * T))
kBLnF0 = np.float32(350.0 * 55.262042231857095 / (T * T))
EDGES = np.array([np.nextafter(0.5 * (oracle.port_compton_frq(1) + oracle.port_compton_frq(0)), -np.inf)] +
                 [oracle.port_compton_frq(j) for j in range(1, 100)] + [np.inf])


def slot(x, dlg):
    hi = (x.view(np.uint64) >> np.uint64(32)).astype(np.uint32)
    with np.errstate(over="ignore", invalid="ignore", divide="ignore"):
        xf = (hi * np.uint32(8) - np.uint32(0xC0000000)).view(np.float32)
        lg = (np.log2(xf.astype(np.float64)) + dlg).astype(np.float32)
        t2 = (np.float64(-kBLn2) * lg.astype(np.float64) + np.float64(kBLnF0)).astype(np.float32)
        t2 = np.where(np.isnan(t2), np.float32(0), np.clip(t2, np.float32(0), np.float32(1)))
        t = np.sqrt(t2.astype(np.float64)).astype(np.float32)
        magic = (t.astype(np.float64) * np.float64(np.float32(T)) + 12582912.0).astype(np.float32)
    c = (magic.view(np.uint32) * np.uint32(0xFFFFFFF8) + np.uint32((0x4B400000 + 100) * 8 % 2 ** 32)).view(np.int32)
    assert np.all(c % 8 == 0)
    c = c // 8
    assert c.min() >= 0 and c.max() <= 100
    return c, c + (x.view(np.int64) > EDGES.view(np.int64)[c])


@pytest.mark.parametrize("dlg", [-2.0 ** -21, 0.0, 2.0 ** -21])
def test_slot_is_exact(dlg):
    rng = np.random.default_rng(4)
    e = EDGES[:100]
    xs = np.concatenate([10 ** rng.uniform(3, 28, 400000),
                         np.concatenate([v * (1 + rng.uniform(-1e-6, 1e-6, 200)) for v in e]),
                         np.nextafter(e, -np.inf), e, np.nextafter(e, np.inf), [1e24, 2e24]])
    true = np.searchsorted(e, xs, side="left")
    c, fixed = slot(xs, dlg)
    assert np.all((c == true) | (c == true - 1))
    assert np.array_equal(fixed, true)


def test_invalid_frequencies_stay_in_the_row():
    xs = np.array([0.0, -0.0, -1.0, -1e24, np.inf, -np.inf, np.nan, -np.nan, 5e-324, 1e-300, 1e300, 1.7e308])
    _, s = slot(xs, 0.0)
    assert np.all((s >= 0) & (s <= 101))
