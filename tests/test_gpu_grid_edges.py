"""The grid kernel at the edges of its dispatch.

- A run that cannot fill the GPU spreads its particles over a few lanes of
  each warp (one lane up to 16 particles per SM, all 32 from 8 warps of them
  per SM).  Every particle draws its own stream, so the counters are those of
  a launch of fixed shape exactly, and the tallies, sums of the same flushes
  in another order, agree to M 2^-53 of the sum of their magnitudes: with
  fewer than 2^20 flushes per entry and sums of one sign per wall, 2^-33 of
  the largest entry; 1e-9 leaves a factor of ten for cancellation.
- The linked-cell and the replay kernel spread a small run in the same way:
  the counters of a run are the sums over the parts of its particle range,
  whose sizes lie on both sides of each border of the rule.
- A time bin much longer than a flight across the domain is walked in equal
  parts.  Its means must be those of the replay mode, which knows no parts:
  five standard errors over independent seeds."""
import numpy as np
import pytest

import btegpu
import synth

pytestmark = pytest.mark.gpu

KEYS = ("events", "wall_hits", "crossings", "absorbed", "specular_hits", "tally_updates")


@pytest.mark.parametrize("N", [2, 33, 16 * 152, 16 * 152 + 1, 17 * 152 + 1, 8 * 31 * 152, 8 * 31 * 152 + 1, 8 * 32 * 152 + 1])
def test_lanes_of_a_small_run(engine, N):
    engine.load_modes(synth.mode_table(8, 3, 3, 300.0, config=100))
    engine.load_geometry(synth.ribbon_geometry(100.0, 50.0, 5))
    args = dict(T0=300.0, dt=10.0, maxtime=100.0, N=N, seed=5, source=btegpu.SOURCE_WALLS, specularity=0.3)
    small = engine.rta_run(**args)
    try:
        engine.set_tuning(block_threads=256, blocks_per_sm=3, smem_tally=0)
        full = engine.rta_run(**args)
    finally:
        engine.set_tuning(block_threads=0, blocks_per_sm=0, smem_tally=0)
    for k in KEYS:
        assert small[k] == full[k], k
    for k in ("gz", "gz_jx", "gz_jy"):
        assert np.abs(small[k] - full[k]).max() <= 1e-9 * np.abs(full[k]).max(), k


@pytest.mark.parametrize("mode", [btegpu.MODE_PRODUCTION, btegpu.MODE_REPLAY])
@pytest.mark.parametrize("part", [1, 16 * 152, 16 * 152 + 1, 8 * 31 * 152 + 1])
def test_parts_of_a_run_add_up(engine, mode, part):
    engine.load_modes(synth.mode_table(8, 3, 3, 300.0, config=100))
    engine.load_geometry(synth.periodic_bar_geometry())
    N = part + 8 * 32 * 152 + 1
    args = dict(T0=300.0, dt=10.0, maxtime=50.0, N=N, seed=9, source=btegpu.SOURCE_WALLS, mode=mode)
    whole = engine.rta_run(**args)
    parts = [engine.rta_run(begin=0, end=part, **args), engine.rta_run(begin=part, end=N, **args)]
    for k in KEYS:
        assert whole[k] == sum(p[k] for p in parts), k
    for k in ("gz", "gz_jx", "gz_jy"):
        assert np.abs(whole[k] - sum(p[k] for p in parts)).max() <= 1e-9 * np.abs(whole[k]).max(), k


@pytest.mark.parametrize("dt", [200.0, 4000.0])
def test_long_bins_repeat_the_replay_means(engine, dt):
    engine.load_modes(synth.mode_table(8, 3, 3, 300.0, config=100))
    engine.load_geometry(synth.ribbon_geometry(20.0, 20.0, 4))
    seeds = range(24)
    both = []
    for mode in (btegpu.MODE_PRODUCTION, btegpu.MODE_REPLAY):
        v = [engine.rta_run(300.0, dt, 2 * dt, 5000, seed=1000 * mode + s, source=btegpu.SOURCE_WALLS,
                            mode=mode)["gz"][:, 0] for s in seeds]
        both.append(np.array(v).reshape(len(v), -1))
    mean = [b.mean(axis=0) for b in both]
    err = np.sqrt(sum(b.var(axis=0, ddof=1) / len(b) for b in both))
    assert np.all(np.abs(mean[0] - mean[1]) <= 5 * err)
