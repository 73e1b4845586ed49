"""The integer walk of the grid kernel (fixed_walk.cuh) against exact rational
arithmetic, on the host build of the functions the kernel runs.

Each segment is redone exactly from the integers it started at.  It may lose,
in units of the position (2^-kx nm): two in the product of the displacement,
half for the rounded velocity, and for an exit time ten ticks (two of the
product, eight of the 58-bit reciprocal) or for a flight's length two (its
64-bit mantissa and the shift to ticks, or 2^-61 of a longer one) at less than
half a unit per tick: 8 in all.  A line reached within a unit counts
as a unit away, which a slow crossing stretches by the ratio of the speeds.
Every time bin holds exactly its ticks."""
from fractions import Fraction as F

import numpy as np
import pytest

import btegpu

# extent, cells, bin width: an ordinary grid, short bins, bins many times the
# flight across the domain (walked in parts), a tiny and a large domain
GRIDS = [(1000.0, 50, 10.0), (2000.0, 100, 0.01), (40.0, 2, 500.0), (0.7, 3, 1.0), (3.0e5, 7, 50.0)]


def _flights(rng, n, ext):
    v = 12.0 * np.exp(rng.uniform(np.log(1e-9), 0.0, (n, 2))) * rng.choice([-1.0, 1.0], (n, 2))
    v[rng.random((n, 2)) < 0.2] = 0.0
    tau = np.exp(rng.uniform(np.log(0.01), np.log(ext), n))
    e = (-np.log(rng.integers(0, 2 ** 23, n).astype(np.float32) + np.float32(0.5)) + np.float32(23 * np.log(2)))
    return np.maximum(e, np.float32(6e-8)).astype(np.float32), tau, v


@pytest.mark.parametrize("ext,cells,step", GRIDS)
def test_walk_against_exact_arithmetic(ext, cells, step):
    rng = np.random.default_rng(int(ext * 10) + cells)
    gx = np.linspace(-20.0, ext, cells + 1)
    gy = np.array([0.0, 0.3 * ext, 0.31 * ext, ext])
    worst = 0.0
    for trial in range(20):
        e, tau, v = _flights(rng, 60, ext)
        p = (float(rng.uniform(gx[0], gx[-1])), float(rng.uniform(gy[0], gy[-1])))
        rows, (kx, kt, sub) = btegpu.debug_fixwalk(gx, gy, 12.0, step, 400, p, e, tau, v[:, 0], v[:, 1])
        ux, ut = F(2) ** kx, F(2) ** kt
        assert len(rows) and (gx[-1] - gx[0]) * 2.0 ** kx >= 2.0 ** 55
        x, y = round((F(p[0]) - F(gx[0])) * ux), round((F(p[1]) - F(gy[0])) * ux)
        part, t_bin, left, last = round(F(step) * F(2) ** (kt - sub)), 0, 0, -1
        for m, (k, kind, qx, qy, ticks) in enumerate(rows):
            qx, qy, ticks = int(qx), int(qy), int(ticks)
            if k != last:  # the flight, in ticks
                left, last = int(F(float(e[k])) * F(float(tau[k])) * ut), k
                tol = 2 + (left >> 61)
            vx, vy = (F(float(c)) * ux / ut for c in v[k])  # units per tick
            vx, vy = (c if abs(c) * 2 ** 64 >= 2 else F(0) for c in (vx, vy))
            slack = F(8)
            if kind & 1:
                seg = F(qx - x) / vx
                slack += abs(vy / vx)
            elif kind & 2:
                seg = F(qy - y) / vy
                slack += abs(vx / vy)
            elif kind & 4:
                seg = F(left)
            else:
                seg = F(part - t_bin)
            if not kind & 3:
                assert abs(ticks - seg) <= (tol if kind & 4 else 0), (trial, m)
            err = max(abs(x + seg * vx - qx), abs(y + seg * vy - qy))
            assert err <= slack, (trial, m, int(kind), float(err), float(slack))
            worst = max(worst, float(err))
            x, y, left, t_bin = qx, qy, left - ticks, t_bin + ticks
            assert left >= 0 and t_bin <= part and (left <= tol or not kind & 4)
            assert (kind & 8 != 0) == (t_bin == part)
            if kind & 8:
                t_bin = 0
    assert worst > 0.0  # the walk moved
