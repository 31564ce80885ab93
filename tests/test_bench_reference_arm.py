"""The reference arm of bench.py runs the scene's steps on the oracle through
the same loop as the device."""
import numpy as np


def test_scene_steps_run_on_the_oracle(oracle_mod):
    import bench
    from dropfluid import abi, scenes
    sc = scenes.box48()
    sc.config.mg_cycles = 1
    sims = oracle_mod.OracleSim(sc.config), oracle_mod.OracleSim(sc.config)
    assert bench.run_scene_steps(sc, sims[0], 0, 2, timed=False) == 0.0
    for d in sc.releases_at(0):
        sc.release(sims[1], d)
    sims[1].step(2)
    for f in (abi.FIELD_VEL_V, abi.FIELD_CONC):
        a, b = (e.get_field(f) for e in sims)
        assert np.abs(a).max() > 0
        np.testing.assert_array_equal(a, b)
