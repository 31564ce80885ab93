"""Steps that skip clear water (flags per 8x8x8 dye brick: what a skipped voxel
holds already is not stored again, and dye, bracket and splats are read only
where there may be any) against the same steps with every flag set: a field
written from outside marks every brick.  The same bits are required: a
skipped value is a +0 either way, and splat sums are integers.  Grids with
remainders in the bricks, below and above a million voxels (from where the
stages work on a list of bricks); between steps the dye is replaced, single stages run and a snapshot is
restored, so flags and arrays are seen in every order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fields(abi, ref):
    f = [abi.FIELD_VEL_U, abi.FIELD_VEL_V, abi.FIELD_VEL_W, abi.FIELD_PRESSURE, abi.FIELD_CONC]
    return f + ([abi.FIELD_CONC_PRED] if ref else [])


def _drop(shape, centre, radius, value):
    g = np.stack(np.meshgrid(*[(np.arange(n) + 0.5) / n for n in shape], indexing="ij"), -1)
    return np.where(((g - centre) ** 2).sum(-1) < radius ** 2, value, 0.0).astype(np.float32)


def _run(sims, abi, ref, act, steps):
    """act on both, then `steps` steps, the second with all flags set before each"""
    a, b = sims
    for e in sims:
        act(e)
    for _ in range(steps):
        a.step(1)
        b.set_field(abi.FIELD_CONC, b.get_field(abi.FIELD_CONC))
        b.step(1)
    for f in _fields(abi, ref):
        x, y = a.get_field(f), b.get_field(f)
        np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32), err_msg=f"field {f}")
    np.testing.assert_array_equal(a.get_parcels(), b.get_parcels())


@pytest.mark.parametrize("dims", [(16, 16, 16), (40, 56, 24), (72, 104, 56), (136, 92, 104)])
@pytest.mark.parametrize("mixed", [False, True])
def test_closed_box(dims, mixed):
    from dropfluid import DropFluid, abi
    cfg = abi.config_closed_box(*dims)
    cfg.precision_mode = abi.DOB_PREC_MIXED if mixed else abi.DOB_PREC_FP32
    cfg.parcel_capacity = 64
    sims = DropFluid(cfg), DropFluid(cfg)
    shape = dims[::-1]
    z, y, x = np.meshgrid(*[np.linspace(0, 2 * np.pi, n) for n in shape], indexing="ij")

    def begin(e):
        e.set_field(abi.FIELD_VEL_U, (3 * np.sin(x) * np.cos(y)).astype(np.float32))
        e.set_field(abi.FIELD_VEL_V, (-3 * np.cos(x) * np.sin(y)).astype(np.float32))
        e.set_field(abi.FIELD_CONC, _drop(shape, (0.3, 0.6, 0.4), 0.12, 0.7))
        e.run_stage(abi.STAGE_MAC_TO_CENTER)
        e.save_state(0)

    def other_place(e):
        e.set_field(abi.FIELD_CONC, _drop(shape, (0.8, 0.2, 0.7), 0.15, 0.5))

    def stages(e):
        e.run_stage(abi.STAGE_CONC_PREDICT)
        e.run_stage(abi.STAGE_CONC_RESOLVE)

    _run(sims, abi, False, begin, 4)
    _run(sims, abi, False, other_place, 3)
    _run(sims, abi, False, stages, 2)
    _run(sims, abi, False, lambda e: e.load_state(0), 3)


@pytest.mark.parametrize("dims", [(24, 32, 24), (48, 64, 48), (72, 40, 56)])
@pytest.mark.parametrize("half", [False, True])
def test_reference_mode(dims, half):
    from dropfluid import DropFluid, abi
    from dropfluid.sequencer import SubstepSequencer
    cfg = abi.config_reference()
    cfg.nx, cfg.ny, cfg.nz = dims
    cfg.mg_levels = 3
    cfg.precision_mode = abi.DOB_PREC_REFERENCE_FP16 if half else abi.DOB_PREC_FP32
    cfg.physics_flags = abi.DOB_PHYS_REFERENCE_ALL
    cfg.parcel_capacity = 49152
    sims = DropFluid(cfg), DropFluid(cfg)
    seq = SubstepSequencer(parcel_capacity=cfg.parcel_capacity, seed=3.0)
    first = seq.reset_simulation(3.0, (0.05, -0.02))
    blocks = [seq.advance_substep()[0] for _ in range(96)]
    for e in sims:
        e.set_uniforms(first)
        e.reset()
        e.step_uniforms(np.stack(blocks[:90]))
        e.save_state(0)
    assert np.count_nonzero(sims[0].get_field(abi.FIELD_CONC)) > 0

    def uniforms(k):
        def act(e):
            e.set_uniforms(blocks[k])
        return act

    def pred(e):
        shape = e.get_field(abi.FIELD_CONC_PRED).shape
        e.set_field(abi.FIELD_CONC_PRED, _drop(shape, (0.5, 0.3, 0.4), 0.2, 0.3))

    def dye(e):
        c = e.get_field(abi.FIELD_CONC)
        c[..., 1] += _drop(c.shape[:3], (0.6, 0.5, 0.4), 0.1, 0.2)
        e.set_field(abi.FIELD_CONC, c)

    def stages(e):
        e.run_stage(abi.STAGE_CONC_PREDICT)
        e.run_stage(abi.STAGE_CONC_RESOLVE)

    _run(sims, abi, True, uniforms(90), 3)
    _run(sims, abi, True, pred, 2)
    _run(sims, abi, True, dye, 3)
    _run(sims, abi, True, stages, 2)
    _run(sims, abi, True, lambda e: e.load_state(0), 3)


@pytest.mark.parametrize("dims", [(24, 32, 24), (72, 40, 56)])
def test_light_volume(dims):
    from dropfluid import DropFluid, abi
    from dropfluid.sequencer import SubstepSequencer
    cfg = abi.config_reference()
    cfg.nx, cfg.ny, cfg.nz = dims
    cfg.mg_levels = 3
    cfg.physics_flags = abi.DOB_PHYS_REFERENCE_ALL | abi.DOB_PHYS_LIGHTING
    cfg.parcel_capacity = 49152
    e = DropFluid(cfg)
    seq = SubstepSequencer(parcel_capacity=cfg.parcel_capacity, seed=3.0)
    e.set_uniforms(seq.reset_simulation(3.0, (0.05, -0.02)))
    e.reset()
    e.step_uniforms(np.stack([seq.advance_substep()[0] for _ in range(90)]))
    got = []
    for _ in range(2):  # the second with all flags set
        e.bench_kernel(2, 1)  # the lighting passes on their own
        got.append((e.get_field(abi.FIELD_LIGHT), e.get_field(abi.FIELD_BRICKS)))
        e.set_field(abi.FIELD_CONC, e.get_field(abi.FIELD_CONC))
    assert got[0][1].max() > 0
    for x, y in zip(*got):
        np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32))
