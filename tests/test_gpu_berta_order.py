"""Order of the sources within one beRTA step, against the CPU restatement.

A step of the reference (src/beyondRTA_MC2d.cpp:2138-2425) advects the
particles, makes and advects the gradient source's and the isothermal walls'
particles, and only then re-emits from the adiabatic walls what all of these
left on them; what the re-emitted particles leave on the walls waits for the
next step.  In a ribbon 10 nm wide a step of 4 ps takes most new particles to a
wall, so after one step a re-emission that missed them would change the
energy and the number of particles by tens of percent.  Replicas are
independent; the bars are those of parity_stats."""
import numpy as np
import pytest

import pyoracle
import synth
from parity_stats import check

pytestmark = pytest.mark.gpu

R = 24
STEPS = 2


def _geometry(source):
    hot, cold = (301.0, 299.0) if source == "walls" else (300.0, 300.0)
    return synth.ribbon_geometry(100.0, 10.0, 4, T_hot=hot, T_cold=cold)


def _obs(r):
    # per step: the cells' energy densities and the particles alive
    s = slice(1, STEPS + 1)
    return np.concatenate([r["ed"][s, :4].ravel(), r["nparticles"][s].astype(float)])


@pytest.mark.parametrize("rta", [False, True])
@pytest.mark.parametrize("source", ["walls", "gradient"])
def test_new_particles_on_adiabatic_walls_leave_within_the_step(engine, source, rta):
    m = synth.mode_table(8, 3, 3, 300.0, config=100)
    g, P = _geometry(source), synth.propagator(m)
    engine.load_modes(m)
    engine.load_geometry(g)
    engine.load_propagator(P)
    # across the ribbon: its two long walls absorb opposite signs
    kw = dict(dt=4.0, maxtime=4.0 * (STEPS - 1), Eeff=1e-24, rta=rta,
              gradient=(0.0, 0.02) if source == "gradient" else None)
    gpu = np.array([_obs(engine.berta_run(seed=10 + i, **kw)) for i in range(R)])
    cpu = np.array([_obs(pyoracle.berta_run(m, g, P, seed=500 + i, **kw)) for i in range(R)])
    assert cpu[:, -1].mean() > 1000
    names = [f"ed_{s}_{b}" for s in range(1, STEPS + 1) for b in range(4)] + [f"n_{s}" for s in range(1, STEPS + 1)]
    check(gpu, cpu, names, f"beRTA source order {source} rta={rta}")
