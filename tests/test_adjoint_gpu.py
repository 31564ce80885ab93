"""The CUDA discrete adjoint (k_adjoint.cu, dob_tape.cu) through the C ABI.

Per stage, the adjoint of the same forward state and cotangents is compared
with the FP64 oracle's; the linear stages also pass the dot-product test on
the device.  A recorded drop trajectory (checkpointed forward, segment
recomputation, reverse pass) gives the drop-impulse gradient within 1e-3 of
the FP64 oracle's and of central differences of the loss on the device,
independently of the checkpoint interval.
"""
import numpy as np
import pytest

import adjoint_cases as AC
from dropfluid import abi
from helpers import rel_l2

pytestmark = pytest.mark.gpu

# FP32 device adjoint vs FP64 oracle adjoint at the same (float32) state.  The
# centre-velocity
# adjoints of the dye stages see a few departure points that FP32 rounds onto
# a grid node (a sub-ulp displacement) where FP64 does not; the two then take
# different one-sided / mean slopes of the interpolation at that node.
STAGE_TOL = 1e-5
NODE_TOL = 1e-3


@pytest.fixture(scope="module")
def pair(gpu_lib, oracle_mod):
    from dropfluid import DropFluid
    cfg = AC.box_config((16, 24, 16))
    g = DropFluid(cfg)
    o = oracle_mod.OracleSim(cfg, fp64=True)
    yield cfg, g, o, AC.stage_state(cfg, seed=3)
    g.close()


@pytest.mark.parametrize("stage", sorted(AC.STAGES))
def test_stage_adjoint_matches_fp64_oracle(pair, stage):
    cfg, g, o, st = pair
    ins, outs, _, _ = AC.STAGES[stage]
    ys = AC.seeded_cotangents(g, outs, 100 + stage)
    rg = AC.run_stage_adjoint(g, st, stage, ys)
    ro = AC.run_stage_adjoint(o, st, stage, ys)
    for f in ins:
        if stage == abi.STAGE_PRESSURE_SOLVE and f == abi.FIELD_PRESSURE:
            # the warm-start adjoint is what survives the contracting
            # V-cycles: compare its error with the incoming cotangent's size
            err = np.linalg.norm((rg[f] - ro[f]).ravel()) / np.linalg.norm(ys[f].ravel())
            assert err < STAGE_TOL, (abi.STAGE_NAMES[stage], f, err)
            continue
        tol = NODE_TOL if f == abi.FIELD_VEL_CENTER else STAGE_TOL
        assert rel_l2(rg[f], ro[f]) < tol, (abi.STAGE_NAMES[stage], f, rel_l2(rg[f], ro[f]))


@pytest.mark.parametrize("dims,levels", [((20, 24, 16), 2), ((40, 32, 48), 3), ((48, 32, 48), 4)])
def test_pressure_adjoint_other_grids(gpu_lib, oracle_mod, dims, levels):
    """Levels whose rows take the scalar smoother (nx not a multiple of 8),
    and deeper hierarchies."""
    from dropfluid import DropFluid
    cfg = AC.box_config(dims, levels=levels)
    st = AC.stage_state(cfg, seed=5)
    stage = abi.STAGE_PRESSURE_SOLVE
    with DropFluid(cfg) as g:
        o = oracle_mod.OracleSim(cfg, fp64=True)
        ys = AC.seeded_cotangents(g, [abi.FIELD_PRESSURE], 7)
        rg = AC.run_stage_adjoint(g, st, stage, ys)
        ro = AC.run_stage_adjoint(o, st, stage, ys)
        assert rel_l2(rg[abi.FIELD_RHS], ro[abi.FIELD_RHS]) < 1e-4
        dp = rg[abi.FIELD_PRESSURE] - ro[abi.FIELD_PRESSURE]
        assert np.linalg.norm(dp.ravel()) / np.linalg.norm(ys[abi.FIELD_PRESSURE].ravel()) < 1e-5


@pytest.mark.parametrize("stage", AC.LINEAR)
def test_linear_stage_dot_product_on_device(pair, stage):
    cfg, g, o, st = pair
    ins, outs, _, _ = AC.STAGES[stage]
    xs = AC.seeded_cotangents(g, ins, 10 + stage)
    ys = AC.seeded_cotangents(g, outs, 20 + stage)
    AC.load(g, st)
    for f, a in xs.items():
        g.set_field(f, a)
    g.run_stage(stage)
    lhs = sum(float(np.sum(g.get_field(f).astype(np.float64) * ys[f])) for f in outs)
    adj = AC.run_stage_adjoint(g, st, stage, ys)
    rhs = sum(float(np.sum(xs[f].astype(np.float64) * adj[f])) for f in ins)
    assert abs(lhs - rhs) <= 1e-4 * abs(lhs), (lhs, rhs)


def test_trajectory_gradient(gpu_lib, oracle_mod):
    from dropfluid import DropFluid
    cfg, center, r = AC.drop_scene((24, 32, 24))
    g = DropFluid(cfg)
    o = oracle_mod.OracleSim(cfg, fp64=True)
    steps = 8
    AC.init_drop(o, center, r, 1.1)
    o.tape_forward(steps)
    target = o.get_field(abi.FIELD_CONC).astype(np.float64)

    def run(e, imp, k):
        AC.init_drop(e, center, r, imp)
        e.tape_forward(steps, k)
        d = e.get_field(abi.FIELD_CONC).astype(np.float64) - target
        return float(np.sum(d * d)), d

    grads = {}
    for name, e, k in (("gpu3", g, 3), ("gpu8", g, 8), ("orc", o, None)):
        _, d = run(e, 1.0, k)
        e.tape_backward((2 * d).astype(np.float32))
        grads[name] = (e.gradients(), e.sphere_impulse(center, r, [0.0, -2.0, 0.0]))
    gi, oi = grads["gpu3"][1], grads["orc"][1]
    assert abs(gi - oi) <= 1e-3 * abs(oi), (gi, oi)
    # checkpoint interval 3 (three segments, the last one partial) vs 8
    assert rel_l2(grads["gpu3"][0]["u"], grads["gpu8"][0]["u"]) < 1e-5
    assert abs(grads["gpu3"][1] - grads["gpu8"][1]) <= 1e-5 * abs(oi)
    # field gradients: FP32 vs FP64 trajectories take different limiter
    # branches at a few cells, which the per-cell gradient sees
    for k in ("u", "v", "w"):
        assert rel_l2(grads["gpu3"][0][k], grads["orc"][0][k]) < 5e-2, k
    # central differences of the device loss in the impulse
    h = 1e-2
    fd = (run(g, 1.0 + h, 8)[0] - run(g, 1.0 - h, 8)[0]) / (2 * h)
    assert abs(fd - gi) <= 1e-3 * abs(fd), (fd, gi)
    g.close()


def test_adjoint_rejects_other_modes(gpu_lib):
    from dropfluid import DropFluid, DropFluidError
    cfg = abi.config_reference()
    cfg.nx, cfg.ny, cfg.nz = 32, 32, 32
    cfg.mg_levels = 3
    cfg.parcel_capacity = 1024
    with DropFluid(cfg) as sim:
        with pytest.raises(DropFluidError):
            sim.adjoint_stage(abi.STAGE_PROJECT)
        with pytest.raises(DropFluidError):
            sim.tape_forward(2, 1)
    cfg = AC.box_config((16, 24, 16))
    with DropFluid(cfg) as sim:
        with pytest.raises(DropFluidError):
            sim.tape_backward(np.zeros((16, 24, 16), np.float32))  # nothing recorded
        with pytest.raises(DropFluidError):
            sim.adjoint_stage(abi.STAGE_CLEAR_SPLATS)


def test_soft_injection_bit_exact(gpu_lib, oracle_mod):
    """dob_inject_sphere_soft (compiled without FMA contraction) adds the
    same bits as the FP32 oracle's restatement, also on top of a drop that
    is already there."""
    from dropfluid import DropFluid
    cfg, center, r = AC.drop_scene((24, 32, 24))
    g = DropFluid(cfg)
    o = oracle_mod.OracleSim(cfg, fp64=False)
    for e in (g, o):
        AC.init_soft_drop(e, center, r, 1.0)
        e.inject_sphere_soft([center[0] + 1.3, center[1], center[2] - 0.7], 3.0, 1.5, 0.5, [0.5, -1.0, 0.25], 0.1, 3)
    for f in (abi.FIELD_VEL_U, abi.FIELD_VEL_V, abi.FIELD_VEL_W, abi.FIELD_CONC):
        a, b = g.get_field(f), o.get_field(f)
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), f
    assert np.count_nonzero(g.get_field(abi.FIELD_CONC)) > 0
    g.close()


def test_soft_drop_gradient(gpu_lib, oracle_mod):
    """Impulse and centre gradient of a soft drop's trajectory: the device
    against the FP64 oracle (1e-3), and against central differences of the
    device loss (impulse 1e-3; centre, whose FP32 differences need a 0.05-cell
    step, 1e-2 of the gradient's norm)."""
    from dropfluid import DropFluid
    cfg, center, r = AC.drop_scene((24, 32, 24))
    g = DropFluid(cfg)
    o = oracle_mod.OracleSim(cfg, fp64=True)
    steps = 8
    shifted = [center[0] + 0.3, center[1] - 0.2, center[2] + 0.25]
    AC.init_soft_drop(o, shifted, r, 1.1)
    o.tape_forward(steps)
    target = o.get_field64(abi.FIELD_CONC)

    def run(e, c, imp, k=None):
        AC.init_soft_drop(e, c, r, imp)
        e.tape_forward(steps, k or steps)
        d = np.asarray(e.get_field(abi.FIELD_CONC), np.float64) - target
        return float(np.sum(d * d)), d

    grads = {}
    for name, e, k in (("gpu", g, 4), ("orc", o, None)):
        _, d = run(e, center, 1.0, k)
        e.tape_backward((2 * d).astype(np.float32))
        grads[name] = AC.soft_drop_grad(e, center, r)
    (gi, gp), (oi, op) = grads["gpu"], grads["orc"]
    assert abs(gi - oi) <= 1e-3 * abs(oi), (gi, oi)
    assert np.linalg.norm(gp - op) <= 1e-3 * np.linalg.norm(op), (gp, op)
    h = 1e-2
    fd = (run(g, center, 1.0 + h, 4)[0] - run(g, center, 1.0 - h, 4)[0]) / (2 * h)
    assert abs(fd - gi) <= 1e-3 * abs(fd), (fd, gi)
    eps = 5e-2
    for k in range(3):
        cp, cm = list(center), list(center)
        cp[k] = float(np.float32(center[k] + eps))
        cm[k] = float(np.float32(center[k] - eps))
        fdk = (run(g, cp, 1.0, 4)[0] - run(g, cm, 1.0, 4)[0]) / (cp[k] - cm[k])
        assert abs(fdk - gp[k]) <= 1e-2 * np.linalg.norm(gp), (k, fdk, gp)
    g.close()


def test_recorded_forward_matches_steps_and_repeats(gpu_lib):
    """dob_tape_forward computes its last segment with the recording kernels
    (the backward then does not recompute it): the context ends in the same
    bits as plain steps from the same state, parcels included, and a second
    backward without a new forward, which recomputes that segment from its
    checkpoint, gives the same gradients."""
    from dropfluid import DropFluid, scenes
    cfg, center, r = AC.drop_scene((24, 32, 24))
    cfg.parcel_capacity = 512
    cfg.mg_cycles_injected = 0  # recorded steps run mg_cycles V-cycles
    a, b = DropFluid(cfg), DropFluid(cfg)
    p = scenes.parcels_in_sphere(center, r, 512, 5)
    for e in (a, b):
        AC.init_drop(e, center, r, 1.0)
        e.set_parcels(p)
    steps, k = 7, 3  # three segments, the last one partial
    a.tape_forward(steps, k)
    b.run_stage(abi.STAGE_MAC_TO_CENTER)
    b.step(steps)
    for f in (abi.FIELD_VEL_U, abi.FIELD_VEL_V, abi.FIELD_VEL_W, abi.FIELD_VEL_CENTER, abi.FIELD_PRESSURE,
              abi.FIELD_CONC):
        x, y = a.get_field(f), b.get_field(f)
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), f
    x, y = a.get_parcels(), b.get_parcels()
    assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
    gd = (1e-3 * a.get_field(abi.FIELD_CONC)).astype(np.float32)
    a.tape_backward(gd)
    g1 = {c: v.copy() for c, v in a.gradients().items()}
    a.tape_backward(gd)
    g2 = a.gradients()
    for c in ("u", "v", "w", "dye"):
        assert rel_l2(g2[c], g1[c]) < 1e-6, c
    a.close()
    b.close()


def test_gradient_directions_against_fp64_differences(gpu_lib, oracle_mod):
    """Directional derivatives of the trajectory loss along seeded random
    directions of the initial MAC velocity: the device gradient (the adjoint
    of the FP32 trajectory) and the FP64 oracle's adjoint against central
    differences of the FP64 oracle's loss (step 1e-6, below every limiter
    and clamp branch of the FP64 trajectory), each within 1e-3 per
    direction, and the device's field gradients within 1e-3 (relative L2)
    of the FP64 adjoint's.  The scene is the benchmark's drop (-1.5
    cells/step with N(0, 0.05) face noise) on the 48x64x48 box, 8 steps."""
    from dropfluid import DropFluid, scenes
    sc = scenes.box48()
    sc.drops[0].n_parcels = 0
    sc.drops[0].w_cells_per_step = -1.5
    sc.drops[0].noise_cells_per_step = 0.05
    cfg = sc.config
    cfg.mg_cycles_injected = 0  # recorded steps run mg_cycles
    steps = 8
    g = DropFluid(cfg)
    o = oracle_mod.OracleSim(cfg, fp64=True)

    def init(e, scale=1.0, pert=None):
        e.reset()
        w0 = sc.drops[0].w_cells_per_step
        sc.drops[0].w_cells_per_step = w0 * scale
        sc.release(e, 0)
        sc.drops[0].w_cells_per_step = w0
        for f, a in (pert or {}).items():
            e.set_field64(f, e.get_field64(f) + a)

    init(o, 1.1)
    o.tape_forward(steps)
    target = o.get_field64(abi.FIELD_CONC)
    grads = {}
    for name, e in (("gpu", g), ("orc", o)):
        init(e)
        if name == "gpu":
            e.tape_forward(steps, 4)
            dye = np.asarray(e.get_field(abi.FIELD_CONC), np.float64)
        else:
            e.tape_forward(steps)
            dye = e.get_field64(abi.FIELD_CONC)
        e.tape_backward((2 * (dye - target)).astype(np.float32))
        grads[name] = {k: np.asarray(v, np.float64) for k, v in e.gradients().items()}
    vel = (abi.FIELD_VEL_U, abi.FIELD_VEL_V, abi.FIELD_VEL_W)

    def loss64(pert):
        init(o, 1.0, pert)
        o.tape_forward(steps)
        dd = o.get_field64(abi.FIELD_CONC) - target
        return float(np.sum(dd * dd))

    rng = np.random.default_rng(2)
    eps = 1e-6
    shape = grads["gpu"]["u"].shape
    dev_err, orc_err = [], []
    for _ in range(6):
        dirs = {f: rng.standard_normal(shape) for f in vel}
        fd = (loss64({f: eps * a for f, a in dirs.items()}) - loss64({f: -eps * a for f, a in dirs.items()})) / (2 * eps)
        for name, errs in (("gpu", dev_err), ("orc", orc_err)):
            ad = sum(float(np.sum(grads[name][k] * dirs[f])) for k, f in zip("uvw", vel))
            errs.append(abs(ad - fd) / abs(fd))
    print("directional rel err, device:", ["%.1e" % x for x in dev_err])
    print("directional rel err, FP64 adjoint:", ["%.1e" % x for x in orc_err])
    for k in "uvw":
        print(f"field gradient {k}: device vs FP64 adjoint rel L2 {rel_l2(grads['gpu'][k], grads['orc'][k]):.2e}")
    # measured: FP64 adjoint 1.3e-4, device 2.1e-4 at worst; field gradients 1.5e-4
    assert max(orc_err) < 1e-3, orc_err
    assert max(dev_err) < 1e-3, dev_err
    for k in "uvw":
        assert rel_l2(grads["gpu"][k], grads["orc"][k]) < 1e-3, k
    g.close()


def _mixed_drop_scene():
    """box48's drop (-1.5 cells/step, N(0, 0.05) face noise), no parcels, in
    the mixed mode: binary16 dye, the pressure pair solved to ||b - A p|| <=
    1e-8 ||b|| and max |div| dt/dx <= 1e-5 on every step."""
    from dropfluid import scenes
    sc = scenes.box48()
    sc.drops[0].n_parcels = 0
    sc.drops[0].w_cells_per_step = -1.5
    sc.drops[0].noise_cells_per_step = 0.05
    cfg = sc.config
    cfg.precision_mode = abi.DOB_PREC_MIXED
    cfg.mg_rel_tol = 1e-8
    cfg.mg_div_tol = 1e-5
    cfg.mg_max_outer = 8
    cfg.mg_cycles = 0
    cfg.mg_cycles_injected = 0
    return sc


def test_mixed_recorded_forward_matches_steps(gpu_lib):
    """The mixed mode's recorded forward (binary16 dye and the pressure pair
    on the tape, each recording step a captured graph) ends where plain
    steps from the same state end, and a second backward (which recomputes
    the last segment from its checkpoint) repeats the first one's
    gradients.  The solve stops on FP64 reductions whose summation order
    may differ between runs, so the comparison is to 1e-6, not bits."""
    from dropfluid import DropFluid
    sc = _mixed_drop_scene()
    a, b = DropFluid(sc.config), DropFluid(sc.config)
    for e in (a, b):
        e.reset()
        sc.release(e, 0)
    steps, k = 7, 3
    a.tape_forward(steps, k)
    b.run_stage(abi.STAGE_MAC_TO_CENTER)
    b.step(steps)
    for f in (abi.FIELD_VEL_U, abi.FIELD_VEL_V, abi.FIELD_VEL_W, abi.FIELD_PRESSURE, abi.FIELD_CONC):
        assert rel_l2(a.get_field(f), b.get_field(f)) < 1e-6, f
    gd = (1e-3 * a.get_field(abi.FIELD_CONC)).astype(np.float32)
    a.tape_backward(gd)
    g1 = {c: v.copy() for c, v in a.gradients().items()}
    a.tape_backward(gd)
    g2 = a.gradients()
    for c in ("u", "v", "w", "dye"):
        assert rel_l2(g2[c], g1[c]) < 1e-6, c
    a.close()
    b.close()


def test_mixed_gradient_directions_against_fp64_differences(gpu_lib, oracle_mod):
    """The adjoint of the mixed-precision trajectory (binary16 dye read at
    its stored values; the pressure solve's adjoint is the same mixed solve
    on the adjoint right-hand side, to 1e-6) against central differences of
    an FP64 oracle run whose pressure is converged (16 V-cycles per step),
    along seeded random directions of the initial MAC velocity, and its
    field gradients against that run's FP64 adjoint."""
    from dropfluid import DropFluid
    sc = _mixed_drop_scene()
    steps = 8
    g = DropFluid(sc.config)
    ocfg = _mixed_drop_scene().config
    ocfg.precision_mode = abi.DOB_PREC_FP32
    ocfg.mg_cycles = 16
    o = oracle_mod.OracleSim(ocfg, fp64=True)

    def init(e, scale=1.0, pert=None):
        e.reset()
        w0 = sc.drops[0].w_cells_per_step
        sc.drops[0].w_cells_per_step = w0 * scale
        sc.release(e, 0)
        sc.drops[0].w_cells_per_step = w0
        for f, a in (pert or {}).items():
            e.set_field64(f, e.get_field64(f) + a)

    init(o, 1.1)
    o.tape_forward(steps)
    target = o.get_field64(abi.FIELD_CONC)
    grads = {}
    for name, e in (("gpu", g), ("orc", o)):
        init(e)
        if name == "gpu":
            e.tape_forward(steps, 4)
            dye = np.asarray(e.get_field(abi.FIELD_CONC), np.float64)
        else:
            e.tape_forward(steps)
            dye = e.get_field64(abi.FIELD_CONC)
        e.tape_backward((2 * (dye - target)).astype(np.float32))
        grads[name] = {k: np.asarray(v, np.float64) for k, v in e.gradients().items()}
    vel = (abi.FIELD_VEL_U, abi.FIELD_VEL_V, abi.FIELD_VEL_W)

    def loss64(pert):
        init(o, 1.0, pert)
        o.tape_forward(steps)
        dd = o.get_field64(abi.FIELD_CONC) - target
        return float(np.sum(dd * dd))

    rng = np.random.default_rng(2)
    eps = 1e-6
    shape = grads["gpu"]["u"].shape
    dev_err, orc_err = [], []
    for _ in range(6):
        dirs = {f: rng.standard_normal(shape) for f in vel}
        fd = (loss64({f: eps * a for f, a in dirs.items()}) - loss64({f: -eps * a for f, a in dirs.items()})) / (2 * eps)
        for name, errs in (("gpu", dev_err), ("orc", orc_err)):
            ad = sum(float(np.sum(grads[name][k] * dirs[f])) for k, f in zip("uvw", vel))
            errs.append(abs(ad - fd) / abs(fd))
    print("mixed: directional rel err, device:", ["%.1e" % x for x in dev_err])
    print("mixed: directional rel err, FP64 adjoint:", ["%.1e" % x for x in orc_err])
    for k in "uvw":
        print(f"mixed: field gradient {k}: device vs FP64 adjoint rel L2 {rel_l2(grads['gpu'][k], grads['orc'][k]):.2e}")
    # measured: device 3.7e-4 at worst against the differences; the field
    # gradients sit at 0.6-1.5e-3 of the FP64 adjoint's, linearised at dye
    # values rounded to binary16 (2^-11 relative per store) where the FP64
    # run keeps them exact
    assert max(orc_err) < 1e-3, orc_err
    assert max(dev_err) < 1e-3, dev_err
    for k in "uvw":
        assert rel_l2(grads["gpu"][k], grads["orc"][k]) < 3e-3, k
    g.close()



@pytest.mark.parametrize("dims", [(16, 16, 16), (24, 32, 16)])
def test_first_pressure_gradient_has_no_constant(gpu_lib, dims):
    """The closed box's solve passes a constant through and removes the mean, so
    d loss / d (first pressure) sums to zero over the black cells, which carry
    it (the first half-sweep overwrites the red ones).  Bound: the mean is taken
    out in FP32, one rounding of 2^-24 of each value."""
    from dropfluid import DropFluid, abi
    from dropfluid.adjoint import DropTrajectory
    c = abi.config_closed_box(*dims)
    c.parcel_capacity = 64
    sim = DropFluid(c)
    shape = dims[::-1]
    z, y, x = np.meshgrid(*[np.linspace(0, 2 * np.pi, n) for n in shape], indexing="ij")
    sim.set_field(abi.FIELD_VEL_U, np.sin(x + y).astype(np.float32))
    sim.set_field(abi.FIELD_CONC, (0.5 + 0.4 * np.cos(y) * np.sin(z)).astype(np.float32))
    sim.run_stage(abi.STAGE_MAC_TO_CENTER)
    traj = DropTrajectory(sim, 2)
    traj.forward(3)
    g = np.asarray(traj.backward(np.cos(x + 2 * z).astype(np.float32))["p"], np.float64)
    black = g[(np.indices(shape).sum(0) & 1) == 1]
    assert np.abs(black).max() > 0
    assert abs(black.sum()) <= 2.0 ** -24 * np.abs(black).sum()
