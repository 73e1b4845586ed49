"""The integer walk of the grid kernel (fixed_walk.cuh) beside the same walk in
doubles, whole particles at a time: what each leaves in its (cell, time bin)
entries, time and displacement, against the same sums in exact rational
arithmetic.  The integers replaced doubles, so over the shapes and bins of
ordinary runs their errors may be no larger: the root mean square over the
entries, of a displacement as a part of the domain along its axis and of a time
as a part of the time bin."""
import math
from collections import defaultdict
from fractions import Fraction as F

import numpy as np
import pytest

import btegpu
VMAX, BINS, FLIGHTS, PARTICLES = 12.0, 40, 20, 300

# length, width, columns, rows, bin width: ribbons from the ordinary to the
# longest and narrowest with short and long bins, the porous rectangle from
# its smallest to its largest, a stack of ribbons as one geometry
SHAPES = [(1000.0, 100.0, 50, 1, 10.0), (1500.0, 20.0, 60, 1, 5.0), (1500.0, 20.0, 3, 1, 20.0), (100.0, 400.0, 60, 1, 5.0),
          (2000.0, 500.0, 100, 25, 50.0), (300.0, 160.0, 15, 8, 50.0), (1000.0, 16000.0, 50, 64, 10.0)]


def _flights(rng, n, ext):
    v = VMAX * np.exp(rng.uniform(np.log(1e-3), 0.0, (n, 2))) * rng.choice([-1.0, 1.0], (n, 2))
    tau = np.exp(rng.uniform(np.log(0.01), np.log(ext), n))
    e = -np.log((rng.integers(0, 2 ** 23, n) + 0.5) / 2.0 ** 23)
    return np.maximum(e, 6e-8).astype(np.float32), tau, v


def _cell(g, x):
    return min(max(int(np.searchsorted(g, x, side="right")) - 1, 0), len(g) - 2)


def _exact(gx, gy, step, p, e, tau, v):
    """The entries of the straight flights, crossings from each flight's start."""
    out = defaultdict(lambda: [F(0)] * 3)
    X, Y, T, step = F(p[0]), F(p[1]), F(0), F(step)
    i, j = _cell(gx, p[0]), _cell(gy, p[1])
    bin_ = 0
    for k in range(len(e)):
        vx, vy = F(float(v[k, 0])), F(float(v[k, 1]))
        d, t = F(float(e[k])) * F(float(tau[k])), F(0)
        while True:
            tx = (F(float(gx[i + (vx > 0)])) - X) / vx if vx else None
            ty = (F(float(gy[j + (vy > 0)])) - Y) / vy if vy else None
            stops = [(d, 0), ((bin_ + 1) * step - T, 3)] + [(s, q) for s, q in ((tx, 1), (ty, 2)) if s is not None]
            s, what = min(stops)
            a = out[i, j, bin_]
            for q, c in enumerate((F(1), vx, vy)):
                a[q] += c * (s - t)
            t = s
            if what == 1:
                i += 1 if vx > 0 else -1
            elif what == 2:
                j += 1 if vy > 0 else -1
            elif what == 3:
                bin_ += 1
            if what == 0 or bin_ == BINS or not (0 <= i < len(gx) - 1 and 0 <= j < len(gy) - 1):
                break
        if what:
            return out
        X, Y, T = X + vx * d, Y + vy * d, T + d
    return out


def _fma(a, b, c):
    return float(F(a) * F(b) + F(c))


def _doubles(gx, gy, step, p, e, tau, v):
    """The walk as an FP64 kernel does it: one exit time per axis, positions by
    FMA, an entry's sums the differences since it was opened."""
    out = defaultdict(lambda: [0.0] * 3)
    x, y, rb = p[0], p[1], step
    i, j, bin_ = _cell(gx, x), _cell(gy, y), 0
    r0, x0, y0 = rb, x, y
    for k in range(len(e)):
        vx, vy = (float(c) for c in v[k])
        dt = float(e[k]) * float(tau[k])
        while True:
            ux, uy = vx >= 0, vy >= 0
            xw, yw = float(gx[i + ux]), float(gy[j + uy])
            tx = (xw - x) * (1.0 / vx) if vx else math.inf
            ty = (yw - y) * (1.0 / vy) if vy else math.inf
            te = max(min(tx, ty), 0.0)
            lim = min(te, rb)
            kind = 4 if dt <= lim else (1 if tx <= ty else 2) if te <= rb else 8
            seg = dt if kind == 4 else lim
            x, y = xw if kind == 1 else _fma(seg, vx, x), yw if kind == 2 else _fma(seg, vy, y)
            rb = 0.0 if kind == 8 else rb - seg
            dt -= seg
            if kind == 4:
                break
            a = out[i, j, bin_]
            for q, c in enumerate((r0 - rb, x - x0, y - y0)):
                a[q] += c
            if kind == 1:
                i += 1 if ux else -1
            elif kind == 2:
                j += 1 if uy else -1
            else:
                bin_, rb = bin_ + 1, step
            if bin_ == BINS or not (0 <= i < len(gx) - 1 and 0 <= j < len(gy) - 1):
                return out
            r0, x0, y0 = rb, x, y
    a = out[i, j, bin_]
    for q, c in enumerate((r0 - rb, x - x0, y - y0)):
        a[q] += c
    return out


def _integers(gx, gy, step, p, e, tau, v):
    rows, (kx, kt, sub) = btegpu.debug_fixwalk(gx, gy, VMAX, step, BINS, p, e, tau, v[:, 0], v[:, 1])
    out = defaultdict(lambda: [0.0] * 3)
    pend = [0, 0, 0]
    i, j, part = _cell(gx, p[0]), _cell(gy, p[1]), 0
    x, y = (round((F(c) - F(float(g[0]))) * F(2) ** kx) for c, g in zip(p, (gx, gy)))

    def flush():
        a = out[i, j, part >> sub]
        for q, c in enumerate(pend):
            a[q] += float(c) * 2.0 ** -(kt if q == 0 else kx)
        pend[:] = 0, 0, 0

    for k, kind, qx, qy, ticks in (map(int, r) for r in rows):
        pend = [pend[0] + ticks, pend[1] + qx - x, pend[2] + qy - y]
        x, y = qx, qy
        if kind != 4:
            flush()
        if kind == 1:
            i += 1 if v[k, 0] >= 0 else -1
        elif kind == 2:
            j += 1 if v[k, 1] >= 0 else -1
        elif kind == 8:
            part += 1
    if any(pend):
        flush()
    return out


@pytest.mark.parametrize("lx,ly,nx,ny,step", SHAPES)
def test_errors_are_no_larger_than_in_doubles(built, lx, ly, nx, ny, step):
    rng = np.random.default_rng(int(lx + 10 * ly + nx + step))
    gx, gy = np.linspace(0.0, lx, nx + 1), np.linspace(0.0, ly, ny + 1)
    err = {"integers": [], "doubles": []}
    for trial in range(PARTICLES):
        e, tau, v = _flights(rng, FLIGHTS, max(lx, ly))
        p = (float(rng.uniform(0.0, lx)), float(rng.uniform(0.0, ly)))
        want = _exact(gx, gy, step, p, e, tau, v)
        for name, walk in (("integers", _integers), ("doubles", _doubles)):
            got = walk(gx, gy, step, p, e, tau, v)
            for key in set(want) | set(got):
                err[name].append([float(F(g) - w) for g, w in zip(got[key], want[key])])
    rms = {}
    for name in err:
        a = np.array(err[name]) / (step, lx, ly)
        rms[name] = np.sqrt(np.mean(a ** 2, axis=0))
        print(f"{lx} x {ly} nm, {step} ps, {name}: {len(a)} entries, time {rms[name][0]:.2e} of the bin, "
              f"displacement {rms[name][1]:.2e} {rms[name][2]:.2e} of the domain")
    assert len(err["integers"]) > 1000
    assert np.all(rms["integers"] <= rms["doubles"])
