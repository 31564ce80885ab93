"""The pressure solve on small levels: legs of the V-cycle in one launch
(dob_mgleg.cuh), all sweeps of the coarsest grid in one CTA or one cluster,
and the exact coarsest solve with the inverse held in registers, against the
oracle's in-place sweeps.  Grids at the edges of the blocks' tiles (8 and 24
cells wide for 2 sweeps, 12 and 28 for 1), one block to many, both boundary
modes, every sweep count the legs cover and one they do not.

Tolerance: the stage bar of the parity tests, 2e-5 relative L2 (FP32 with and
without multiply-add contraction)."""
import numpy as np
import pytest

from helpers import rel_l2, smooth_field

pytestmark = pytest.mark.gpu


def _solve(cfg, oracle_mod, seed):
    from dropfluid import DropFluid, abi
    shape = (cfg.nz, cfg.ny, cfg.nx)
    b = smooth_field(shape, seed, 1.0).astype(np.float64)
    if cfg.bc_mode == abi.DOB_BC_CLOSED_BOX:
        b -= b.mean()
    p0 = smooth_field(shape, seed + 1, 2.0)
    out = []
    for e in (DropFluid(cfg), oracle_mod.OracleSim(cfg)):
        e.set_field(abi.FIELD_RHS, b.astype(np.float32))
        e.set_field(abi.FIELD_PRESSURE, p0)
        e.run_stage(abi.STAGE_PRESSURE_SOLVE)
        out.append(e.get_field(abi.FIELD_PRESSURE))
        e.close()
    return out


def _config(mode, dims, levels, pre, post, coarse):
    from dropfluid import abi
    c = abi.config_closed_box(*dims) if mode == "box" else abi.config_reference()
    c.nx, c.ny, c.nz = dims
    c.mg_levels, c.mg_pre, c.mg_post, c.mg_coarse_sweeps = levels, pre, post, coarse
    c.mg_cycles = 2
    c.parcel_capacity = 64
    return c


@pytest.mark.parametrize("mode", ["box", "ref"])
@pytest.mark.parametrize("dims,levels,pre,post,coarse", [
    ((8, 8, 8), 2, 2, 2, 6),          # one block, most of its region outside the grid
    ((8, 16, 24), 3, 2, 2, -1),
    ((24, 8, 16), 2, 1, 1, 6),        # one tile wide
    ((28, 12, 12), 2, 1, 2, -1),      # tiles of the one-sweep legs
    ((52, 28, 36), 2, 2, 1, 6),       # remainders in every direction
    ((40, 56, 24), 3, 2, 2, -1),
    ((40, 56, 24), 3, 3, 3, 6),       # sweep counts without one-launch legs
    ((48, 64, 48), 2, 2, 2, 4),       # coarsest grid of 18432 cells: a cluster of 8
    ((52, 60, 28), 2, 2, 2, 3),       # a cluster whose slabs differ (14 planes)
    ((96, 72, 72), 4, 2, 2, 6),       # close to the largest level with one-launch legs
    ((32, 32, 32), 2, 2, 2, -1),      # 4096 cells solved exactly (inverse read from memory)
])
def test_small_levels_match_oracle(gpu_lib, oracle_mod, mode, dims, levels, pre, post, coarse):
    if any(n % (1 << levels) for n in dims):
        levels = max(L for L in range(1, levels + 1) if all(n % (1 << L) == 0 for n in dims))
    cfg = _config(mode, dims, levels, pre, post, coarse)
    dev, ref = _solve(cfg, oracle_mod, 7 + levels)
    assert rel_l2(dev, ref) < 2e-5


def test_small_levels_mixed(gpu_lib):
    """Levels 2-3 in BF16 (legs from FP32 into BF16 and within BF16): every
    step of the mixed mode meets its targets, as the box48 scene's do."""
    from dropfluid import DropFluid, abi
    cfg = abi.config_closed_box(64, 96, 64)
    assert cfg.mg_levels == 4
    cfg.precision_mode = abi.DOB_PREC_MIXED
    cfg.mg_cycles = 1
    cfg.mg_rel_tol, cfg.mg_div_tol, cfg.mg_max_outer = 1e-8, 1e-5, 30
    cfg.parcel_capacity = 64
    g = DropFluid(cfg)
    g.inject_sphere((30.0, 80.0, 33.0), 6.0, 1.0, (0.0, -100.0, 0.0), 2.5, 1)
    for k in range(6):
        st = g.step(1, stats=True)
        assert st["residual_l2"] <= 1.05e-8 * st["rhs_l2"], (k, st)
        assert st["max_div"] <= 1e-5, (k, st)
    g.close()
