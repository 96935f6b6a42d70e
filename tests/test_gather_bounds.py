"""The staged and few-view gathers' candidate bounds, restated in FP32 with quick divisions
that are off by their two units in the last place, against FP64: on the largest detectors that
those gathers take, rows stay within their margin of 0.002 and detector columns within 0.01.
Larger detectors are left to the gathers that divide exactly."""
import os
import re

import numpy as np
import pytest

from conftest import ROOT

F = np.float32


def _fma(a, b, c):
    """FP32 fmaf of FP32 values: the product is exact in FP64."""
    return (np.float64(a) * np.float64(b) + np.float64(c)).astype(F)


def _quick_div(a, b, ulps):
    q = (np.float64(a) / np.float64(b)).astype(F)
    return (np.float64(q) + ulps * np.spacing(np.abs(q)).astype(np.float64)).astype(F)


def _limits():
    src = open(os.path.join(ROOT, "recon_b200", "csrc", "gather_staged.cu")).read()
    m = re.search(r"staged_bounds_hold\(const Plan& P\) \{ return P\.eg\.Nv <= (\d+) && P\.eg\.Nu <= (\d+); \}", src)
    return int(m.group(1)), int(m.group(2))


@pytest.mark.parametrize("ulps", [-2, 0, 2])
def test_rows(ulps):
    nv = _limits()[0]
    rng = np.random.default_rng(7)
    for _ in range(40):
        Z = int(rng.integers(64, 4096)) // 2 * 2
        ry, rf = rng.uniform(300, 1500, 2)
        rad = rf * rng.uniform(0.02, 0.8)
        # rows that just cover the volume's lower half from the nearest depth
        vz = F(rng.uniform(0.05, 1.0))
        dv = F(0.5 * Z * float(vz) * ry / (rf - rad) / (nv / 2))
        ez, oz = F(ry / float(dv)), F((nv - 1) / 2)
        P0, RF = F(-0.5 * Z * float(vz)), F(rf)
        k = rng.integers(0, Z // 2, 4000)
        lane, slot = k % 32, k // 32
        A = rng.uniform(-rad, rad, k.size).astype(F)
        d = (A + RF).astype(F)
        c = _quick_div(np.full(k.size, ez, F), d, ulps)
        z = _fma(lane.astype(F), vz, P0)
        step = (F(32) * vz * c).astype(F)
        f = _fma(slot.astype(F), step, _fma(z, c, np.full(k.size, oz, F)))
        exact = (np.float64(P0) + k * np.float64(vz)) * np.float64(ez) / (np.float64(A) + np.float64(RF)) + np.float64(oz)
        on = (exact > -1) & (exact < nv)
        assert on.any()
        assert np.abs(np.float64(f) - exact)[on].max() < 0.002


@pytest.mark.parametrize("ulps", [-2, 0, 2])
def test_columns(ulps):
    nu = _limits()[1]
    rng = np.random.default_rng(8)
    for _ in range(40):
        ry, rf = rng.uniform(300, 1500, 2)
        rad = rf * rng.uniform(0.02, 0.85)
        eu = F(nu / 2 / (rad / np.sqrt(rf * rf - rad * rad)))  # the shadow just fills the detector
        ou, RF = F((nu - 1) / 2), F(rf)
        t, r = rng.uniform(0, 2 * np.pi, 4000), rad * np.sqrt(rng.uniform(0, 1, 4000))
        X, Y = (r * np.cos(t)).astype(F), (r * np.sin(t)).astype(F)
        th = rng.uniform(0, 2 * np.pi, 4000)
        cs, sn = np.cos(th), np.sin(th)
        c, s = cs.astype(F), sn.astype(F)
        a = _fma(X, c, -(Y * s).astype(F))
        b = _fma(X, s, (Y * c).astype(F))
        u = _fma(_quick_div(a, (b + RF).astype(F), ulps), eu, np.full(a.size, ou, F))
        X, Y = np.float64(X), np.float64(Y)
        exact = (X * cs - Y * sn) / (X * sn + Y * cs + np.float64(RF)) * np.float64(eu) + np.float64(ou)
        on = (exact > -1) & (exact < nu)
        assert on.any()
        assert np.abs(np.float64(u) - exact)[on].max() < 0.01
