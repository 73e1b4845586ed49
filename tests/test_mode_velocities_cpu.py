"""A mode table with a velocity in the plane that is not finite is refused like one with
such a rate: the integer walk would cut its time bins into 2^24 parts."""
import numpy as np
import pytest

import btegpu
import synth


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("axis", [0, 1])
def test_velocities_must_be_finite(built, bad, axis):
    m = synth.mode_table(8, 3, 3, 300.0, config=100)
    g = synth.ribbon_geometry(200.0, 50.0, 5)
    assert btegpu.debug_lambert(m, g)[0] > 0
    vg = np.array(m["vg"], dtype=float).reshape(-1, 3)
    vg[7, axis] = bad
    assert btegpu.debug_lambert(dict(m, vg=vg), g)[0] <= 0
