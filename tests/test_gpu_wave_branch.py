"""Steps of one call with the wave solver (DOB_PHYS_WAVE): the next step's wave
substep runs beside this step's parcels and dye, from a uniform block copied
ahead.  The same bits as one call per step, captured or launched kernel by
kernel, are required in every field: a wave run twice, skipped, with another
step's block, or beside something that it must wait for shows in them.  Every
block differs (time, dt, the drops, spawning), one drop drains and makes waves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = (40, 48, 32)


def _block(k):
    from dropfluid import uniforms as U
    snap = U.DropSnapshot(sim_time=0.4 + 0.01 * k, active_count=2)
    snap.slots[0] = U.DropSlot(active=True, center=(0.03, 0.285 - 0.001 * k, -0.02), radius=0.05, vel_y=-0.3,
                               oscillation=0.01, vol_drain_rate=0.42 - 0.01 * k, seed=1.5)
    snap.slots[1] = U.DropSlot(active=True, center=(-0.12, 0.31 - 0.004 * k, 0.09), radius=0.03, vel_y=-0.5,
                               oscillation=0.0, vol_drain_rate=0.05, seed=2.7)
    return U.SimUniformPacker().pack(drops=snap, dt=(1 / 60, 1 / 90, 1 / 45)[k % 3], global_seed=1.5,
                                     spawn_cursor=256 * k, spawn_count=256).copy()


def _sim(light=False):
    from dropfluid import DropFluid, abi
    c = abi.config_reference()
    c.nx, c.ny, c.nz = DIMS
    c.mg_levels, c.parcel_capacity = 3, 16384
    c.physics_flags = abi.DOB_PHYS_REFERENCE_ALL | abi.DOB_PHYS_WAVE | (abi.DOB_PHYS_LIGHTING if light else 0)
    e = DropFluid(c)
    e.set_uniforms(_block(0))
    e.reset()
    shape, _ = e.field_shape(abi.FIELD_CONC)
    z, y, x = np.meshgrid(*[np.linspace(-1, 1, n) for n in shape[:3]], indexing="ij")
    dye = np.zeros(shape, np.float32)
    dye[..., 1] = np.clip(0.6 - x * x - (y - 0.5) ** 2 - z * z, 0, 1)
    e.set_field(abi.FIELD_CONC, dye)
    return e


def _state(e, light=False):
    from dropfluid import abi
    names = ["WAVE", "VEL_U", "VEL_V", "VEL_W", "PRESSURE", "CONC", "CONC_PRED"] + (["LIGHT", "BRICKS"] if light else [])
    out = {n: e.get_field(getattr(abi, "FIELD_" + n)) for n in names}
    out["parcels"] = e.get_parcels()
    return out


def _same(a, b):
    assert np.abs(a["WAVE"]).max() > 0
    for n in a:
        np.testing.assert_array_equal(a[n].view(np.uint32), b[n].view(np.uint32), err_msg=n)


@pytest.mark.parametrize("steps", [1, 2, 3, 7])
@pytest.mark.parametrize("light", [False, True])
def test_blocks_of_one_call(gpu_lib, steps, light):
    a, b, c = _sim(light), _sim(light), _sim(light)
    at = 0
    for _ in range(2):  # the second call begins where the first has ended
        blocks = [_block(at + k) for k in range(steps)]
        a.step_uniforms(np.stack(blocks))
        for blk in blocks:
            b.set_uniforms(blk)
            b.step(1)
            c.set_uniforms(blk)
            c.step(1, graph=False)
        at += steps
        _same(_state(a, light), _state(b, light))
        _same(_state(a), _state(c))


def test_steps_of_one_call(gpu_lib):
    a, b = _sim(), _sim()
    for k in range(3):
        for e in (a, b):
            e.set_uniforms(_block(k))
        a.step(k + 2)
        for _ in range(k + 2):
            b.step(1)
        _same(_state(a), _state(b))
    a.time_steps(4)
    for _ in range(4):
        b.step(1)
    _same(_state(a), _state(b))


def test_statistics_call(gpu_lib):
    a, b = _sim(), _sim()
    blocks = np.stack([_block(k) for k in range(5)])
    a.step_uniforms(blocks, stats=True)
    for blk in blocks:
        b.set_uniforms(blk)
        sb = b.step(1, stats=True)
    _same(_state(a), _state(b))
    for e in (a, b):
        e.set_uniforms(_block(5))
    sa, sb = a.step(2, stats=True), [b.step(1, stats=True) for _ in range(2)][-1]
    assert sa["max_div"] == sb["max_div"] and sa["parcels_alive"] == sb["parcels_alive"]
    _same(_state(a), _state(b))


@pytest.mark.parametrize("word", [5, 38])
def test_refused_block(gpu_lib, word):
    """The call fails at the block, with everything as after the one before it."""
    a, b = _sim(), _sim()
    blocks = np.stack([_block(k) for k in range(5)])
    bad = blocks.copy()
    bad[3, word] = np.nan
    with pytest.raises(Exception):
        a.step_uniforms(bad)
    for blk in blocks[:3]:
        b.set_uniforms(blk)
        b.step(1)
    _same(_state(a), _state(b))
    for e in (a, b):  # and goes on from there
        e.step_uniforms(blocks[3:])
    _same(_state(a), _state(b))
