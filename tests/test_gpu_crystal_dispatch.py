"""Crystals on a grid take the linked-cell kernel: what only the grid kernel
does is refused for them, replica groups among it."""
import ctypes as C

import numpy as np
import pytest

import btegpu
import synth

pytestmark = pytest.mark.gpu


def test_groups_are_refused_with_crystals(engine):
    A, B = (synth.mode_table(8, 3, 3, 300.0, config=c) for c in (100, 101))
    g = synth.ribbon_geometry(200.0, 50.0, 10)
    engine.load_mode_tables([A, B])
    engine.load_geometry(dict(g, material=np.array([0] * 5 + [1] * 5 + [0, 1], dtype=np.int32)))
    run = dict(T0=300.0, dt=10.0, maxtime=100.0, N=4000, seed=3)
    engine.set_groups(4)
    try:
        with pytest.raises(btegpu.BteError) as ex:
            engine.rta_run(**run)
        assert ex.value.code == btegpu.BTE_ERR_INPUT
        with pytest.raises(btegpu.BteError) as ex:
            engine.group_result(0, (12, 10))
        assert ex.value.code == btegpu.BTE_ERR_STATE
        # the groups of one mode table on that grid add up to the run
        engine.load_modes(A)
        engine.load_geometry(g)
        whole = engine.rta_run(**run)["gz"]
        parts = [engine.group_result(k, whole.shape, raw=True)["gz"] for k in range(4)]
        assert all(np.abs(p).max() > 0 for p in parts)
        assert np.abs(np.mean(parts, axis=0) - whole).max() <= 1e-9 * np.abs(whole).max()
    finally:
        engine.set_groups(0)


def test_allocation_free_run_refuses_interfaces(engine):
    import torch
    A, B = (synth.mode_table(8, 3, 3, 300.0, config=c) for c in (100, 101))
    g = synth.ribbon_geometry(200.0, 50.0, 10)
    engine.load_mode_tables([A, B])
    params = btegpu.params_struct(300.0, 10.0, 100.0, 4000, 3)
    dev = torch.zeros((12, 10, 3), dtype=torch.float64, device="cuda:0")
    # the crystals in one ribbon, and each in a ribbon of its own (no interface)
    apart = synth.sweep_union_geometry([{"T": T, "width": 50.0, "budget": 1} for T in (300.0, 300.0)], length=200.0, ncells=4)
    for geom, want in ((dict(g, material=np.array([0] * 5 + [1] * 5 + [0, 1], dtype=np.int32)), btegpu.BTE_ERR_INPUT),
                       (apart, btegpu.BTE_OK)):
        engine.load_geometry(geom)
        engine.rta_run(300.0, 10.0, 100.0, 4000, seed=3)
        r = btegpu.RtaResult()
        assert engine.lib.bte_rta_run_noalloc(engine.ctx, C.byref(params), C.c_void_p(dev.data_ptr()), C.byref(r)) == want
