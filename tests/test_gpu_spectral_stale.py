"""bte_get_spectral forms the last run's outputs from a tally on the device,
with the tables it was made with: once other modes, crystals, boxes or
materials are loaded, or the last run failed, there is nothing to form."""
import numpy as np
import pytest

import btegpu
import synth

pytestmark = pytest.mark.gpu


@pytest.fixture()
def run(engine):
    case = synth.small_case(n_particles=2000)
    bins = int(round(case["maxtime"] / case["dt"]))

    def go(**kw):
        engine.load_modes(case["modes"])
        engine.load_geometry(case["geom"])
        engine.set_spectral([1, 3], nomega=50)
        engine.rta_run(case["T0"], case["dt"], case["maxtime"], case["N"], seed=4, **kw)
        return engine.get_spectral(bins)

    yield case, bins, go
    engine.load_modes(case["modes"])
    engine.load_geometry(case["geom"])
    engine.set_spectral([])


LOADS = {
    "larger mode table": lambda e, c: e.load_modes(synth.mode_table(32, 3, 3, 300.0, config=100)),
    "smaller mode table": lambda e, c: e.load_modes(synth.mode_table(5, 3, 3, 300.0, config=100)),
    "crystals": lambda e, c: e.load_mode_tables([c["modes"], c["modes"]]),
    "geometry": lambda e, c: e.load_geometry(synth.ribbon_geometry(100.0, 50.0, 2)),
    "materials": lambda e, c: e.load_materials([c["modes"]["w"]] * 2, [c["T0"], c["T0"] + 10.0]),
}


@pytest.mark.parametrize("what", sorted(LOADS))
def test_other_tables_end_the_spectral_outputs(engine, run, what):
    case, bins, go = run
    first = go()
    LOADS[what](engine, case)
    with pytest.raises(btegpu.BteError) as ex:
        engine.get_spectral(bins)
    assert ex.value.code == btegpu.BTE_ERR_STATE
    again = go()
    assert again["raw"].shape == first["raw"].shape
    assert np.allclose(again["raw"], first["raw"], rtol=1e-9, atol=1e-12 * np.abs(first["raw"]).max())


def test_a_load_that_fails_leaves_the_spectral_outputs(engine, run):
    case, bins, go = run
    first = go()
    bad = dict(case["modes"], w=-np.asarray(case["modes"]["w"]))
    with pytest.raises(btegpu.BteError):
        engine.load_modes(bad)
    with pytest.raises(btegpu.BteError):
        engine.load_materials([bad["w"]], [case["T0"]])
    assert np.array_equal(engine.get_spectral(bins)["raw"], first["raw"])


@pytest.mark.parametrize("steady", [False, True])
def test_locations_beyond_a_smaller_geometry_are_refused(engine, run, steady):
    """Location 7 of eight boxes, then a geometry of five: no run starts."""
    case, bins, go = run
    engine.load_modes(case["modes"])
    engine.load_geometry(synth.periodic_cell_geometry(40.0, 40.0, 2, 2))
    engine.set_spectral([7], nomega=50)
    engine.load_geometry(synth.periodic_cell_geometry(40.0, 40.0, 1, 1))
    with pytest.raises(btegpu.BteError) as ex:
        if steady:
            engine.steady_run(300.0, (0.01, 0.0), 1000)
        else:
            engine.load_geometry(synth.ribbon_geometry(100.0, 50.0, 3))
            engine.rta_run(300.0, 10.0, 100.0, 1000)
    assert ex.value.code == btegpu.BTE_ERR_INPUT and "spectral" in str(ex.value)
    go()


@pytest.mark.parametrize("mode", [btegpu.MODE_PRODUCTION, btegpu.MODE_REPLAY])
def test_a_failed_run_leaves_no_spectral_outputs(engine, run, mode):
    case, bins, go = run
    go()
    with pytest.raises(btegpu.BteError) as ex:
        go(mode=mode, flight_cap=3)
    assert ex.value.code == btegpu.BTE_ERR_LIMIT
    with pytest.raises(btegpu.BteError) as ex:
        engine.get_spectral(bins)
    assert ex.value.code == btegpu.BTE_ERR_STATE
