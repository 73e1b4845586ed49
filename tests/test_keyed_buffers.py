"""Device buffers that are kept while what determines them stays: a fill that
fails must not leave the buffer marked as filled, for the key it held before
or for the one it was given."""
import ctypes as C

import numpy as np
import pytest

import btegpu
import synth


@pytest.mark.parametrize("keys,fails,filled,valid", [
    ([0, 0, 1, 1, 0], [0, 0, 0, 0, 0], [1, 0, 1, 0, 1], 1),
    ([7, 8, 7, 7], [0, 1, 0, 0], [1, 1, 1, 0], 1),   # back to the key before the failure
    ([7, 8, 8, 8], [0, 1, 0, 0], [1, 1, 1, 0], 1),   # the failed key again
    ([7, 7], [1, 0], [1, 1], 1),
    ([7, 8], [0, 1], [1, 1], 0),
])
def test_a_failed_fill_leaves_no_key(built, keys, fails, filled, valid):
    k, f = (np.array(a, dtype=np.int32) for a in (keys, fails))
    got = np.full(len(keys), -1, dtype=np.int32)
    ip = C.POINTER(C.c_int)
    r = btegpu.load_library().btegpu_debug_keyed(k.ctypes.data_as(ip), f.ctypes.data_as(ip), len(keys), got.ctypes.data_as(ip))
    assert list(got) == filled and r == valid


@pytest.mark.gpu
def test_particle_buffers_after_a_capacity_that_cannot_be_had(engine):
    """8 TB of particles fail to allocate; the next run, of a capacity that the
    buffers had before, allocates them again."""
    engine.load_modes(synth.mode_table(8, 3, 3, 300.0, config=100))
    engine.load_geometry(synth.ribbon_geometry(200.0, 50.0, 5))
    run = dict(dt=1.0, maxtime=5.0, Eeff=2e-23, rta=True, seed=3)
    before = engine.berta_run(capacity=1 << 20, **run)
    with pytest.raises(btegpu.BteError) as ex:
        engine.berta_run(capacity=1 << 40, **run)
    assert ex.value.code == btegpu.BTE_ERR_CUDA
    after = engine.berta_run(capacity=1 << 20, **run)
    assert after["nsteps"] == before["nsteps"]
    assert abs(after["nparticles"][-1] - before["nparticles"][-1]) < 0.1 * before["nparticles"][-1]


@pytest.mark.gpu
def test_a_source_that_cannot_be_built_leaves_the_present_one(engine):
    """A ribbon at one temperature has no initial deviation: asking for one
    fails, and the walls' generators of the run before it still serve the
    allocation-free run, which builds nothing."""
    import torch
    engine.load_modes(synth.mode_table(8, 3, 3, 300.0, config=100))
    engine.load_geometry(synth.ribbon_geometry(200.0, 50.0, 5))
    walls = engine.rta_run(300.0, 10.0, 100.0, 2000, seed=3, source=btegpu.SOURCE_WALLS)
    with pytest.raises(btegpu.BteError):
        engine.rta_run(300.0, 10.0, 100.0, 2000, seed=3, source=btegpu.SOURCE_INITIAL)
    dev = torch.zeros((7, 10, 3), dtype=torch.float64, device="cuda:0")
    params = btegpu.params_struct(300.0, 10.0, 100.0, 2000, 3)
    r = btegpu.RtaResult()
    st = engine.lib.bte_rta_run_noalloc(engine.ctx, C.byref(params), C.c_void_p(dev.data_ptr()), C.byref(r))
    assert st == btegpu.BTE_OK and r.events == walls["events"]
