"""The transposed V-cycle's launch chain: transposed prolongation, injection,
residual passes and the colour-exchanged half-sweeps.  Levels of up to half a
million cells with one or two sweeps each way run as legs in one launch, so the
chain takes other sweep counts (0 and 3) on small grids, and larger grids, on
rows that are (vectors of four) and are not (scalars) multiples of 8."""
import numpy as np
import pytest

import adjoint_cases as AC
from dropfluid import abi
from helpers import rel_l2

pytestmark = pytest.mark.gpu


def _config(dims, levels, pre, post, coarse):
    cfg = AC.box_config(dims, levels=levels)
    cfg.mg_pre, cfg.mg_post, cfg.mg_coarse_sweeps, cfg.mg_cycles = pre, post, coarse, 2
    return cfg


@pytest.mark.parametrize("coarse", [-1, 4])
@pytest.mark.parametrize("pre,post", [(3, 3), (0, 2), (2, 0), (3, 1), (0, 0)])
@pytest.mark.parametrize("dims,levels", [((20, 24, 16), 2), ((40, 32, 48), 3)])
def test_sweep_counts_without_legs(gpu_lib, oracle_mod, dims, levels, pre, post, coarse):
    """Against the FP64 oracle, at the bounds of the other grids' test (1e-4 of
    the right-hand side's adjoint; 1e-5 of the cotangent, or of the warm start's
    adjoint where few sweeps leave it larger)."""
    from dropfluid import DropFluid
    cfg = _config(dims, levels, pre, post, coarse)
    st = AC.stage_state(cfg, seed=5)
    stage = abi.STAGE_PRESSURE_SOLVE
    with DropFluid(cfg) as g:
        o = oracle_mod.OracleSim(cfg, fp64=True)
        ys = AC.seeded_cotangents(g, [abi.FIELD_PRESSURE], 7)
        rg = AC.run_stage_adjoint(g, st, stage, ys)
        ro = AC.run_stage_adjoint(o, st, stage, ys)
    assert rel_l2(rg[abi.FIELD_RHS], ro[abi.FIELD_RHS]) < 1e-4
    dp = np.linalg.norm((rg[abi.FIELD_PRESSURE] - ro[abi.FIELD_PRESSURE]).ravel())
    size = max(np.linalg.norm(a.ravel()) for a in (ys[abi.FIELD_PRESSURE], ro[abi.FIELD_PRESSURE]))
    assert dp / size < 1e-5


@pytest.mark.parametrize("dims,levels", [((88, 80, 80), 3), ((84, 84, 80), 2), ((104, 96, 64), 1), ((96, 128, 96), 2)])
def test_large_levels(gpu_lib, dims, levels):
    """<A x, y> = <x, A^T y> on the device, at the bound of the stages' test.
    The last grid's coarsest level sweeps half by half and divides."""
    from dropfluid import DropFluid
    cfg = _config(dims, levels, 2, 2, 5)
    stage = abi.STAGE_PRESSURE_SOLVE
    ins, outs, _, _ = AC.STAGES[stage]
    with DropFluid(cfg) as g:
        xs, ys = AC.seeded_cotangents(g, ins, 10), AC.seeded_cotangents(g, outs, 20)
        st = AC.stage_state(cfg, seed=5)
        AC.load(g, st)
        for f, a in xs.items():
            g.set_field(f, a)
        g.run_stage(stage)
        lhs = sum(float(np.sum(g.get_field(f).astype(np.float64) * ys[f])) for f in outs)
        adj = AC.run_stage_adjoint(g, st, stage, ys)
        rhs = sum(float(np.sum(xs[f].astype(np.float64) * adj[f])) for f in ins)
    scale = sum(float(np.linalg.norm(xs[f]) * np.linalg.norm(adj[f])) for f in ins)
    assert abs(lhs - rhs) <= 1e-4 * max(abs(lhs), 1e-3 * scale), (lhs, rhs)


# |device - FP64 oracle| over the black cells, the mean taken out, relative to
# the warm start's adjoint there, as the half-sweeps transposed one by one
# (which update the adjoint in every launch) had it: smooth and white cotangent
TRANSPOSED_ONE_BY_ONE = [
    ((40, 56, 24), 2, 2, 2, 6, 3.47e-6, 6.94e-7),
    ((72, 104, 56), 3, 2, 2, 6, 9.51e-6, 2.95e-6),
    ((52, 60, 28), 2, 2, 2, 6, 2.22e-6, 6.19e-7),
    ((40, 56, 24), 3, 2, 0, 6, 2.05e-6, 3.04e-6),
    ((84, 84, 80), 2, 2, 2, 6, 8.38e-7, 7.44e-7),  # the finest grid on the launch chain
    ((24, 24, 16), 1, 2, 2, 6, 1.31e-7, 1.29e-7),
]


@pytest.mark.parametrize("dims,levels,pre,post,coarse,smooth,white", TRANSPOSED_ONE_BY_ONE)
def test_warm_start_adjoint_keeps_its_precision(gpu_lib, oracle_mod, dims, levels, pre, post, coarse, smooth, white):
    """What the cycles leave of the warm start's adjoint is small against what
    they take out of it; its error may be no larger than before the transposed
    cycle ran as a V-cycle (a quarter for other summation orders), and the red
    cells, which the first half-sweep overwrites, are zeros."""
    from dropfluid import DropFluid
    cfg = _config(dims, levels, pre, post, coarse)
    cfg.mg_cycles = 3 if (pre, post) == (2, 0) or levels == 1 else 4
    st = AC.stage_state(cfg, seed=5)
    shape = dims[::-1]
    black = (np.indices(shape).sum(0) & 1) == 1
    o = oracle_mod.OracleSim(cfg, fp64=True)
    with DropFluid(cfg) as g:
        for y, before in ((AC.sines(shape, 9, 1.0), smooth), (np.random.default_rng(7).standard_normal(shape), white)):
            ys = {abi.FIELD_PRESSURE: y.astype(np.float32)}
            d, e = (AC.run_stage_adjoint(s, st, abi.STAGE_PRESSURE_SOLVE, ys)[abi.FIELD_PRESSURE].astype(np.float64)
                    for s in (g, o))
            assert not d[~black].any()
            off, ref = (d - e)[black], e[black]
            assert np.linalg.norm(off - off.mean()) <= 1.25 * before * np.linalg.norm(ref - ref.mean())
