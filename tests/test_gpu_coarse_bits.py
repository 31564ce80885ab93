"""The sweeps of the coarsest grid, restated operation by operation in FP32:
grids of up to 25600 cells for each of 8, 4 or 2 slabs of whole planes divide by
the diagonal everywhere, in one launch or half by half, larger ones multiply by
1/6 where it is 6 (on rows that are not multiples of 8: in the interior).  Every
value has to be the same.  Grids on both sides of the limits of one CTA, of a
cluster of eight and of the slabs, whose number the planes decide.

A cycle without smoothing on the finer grid hands the averaged right-hand side
down and the interpolated result up: the right-hand side is constant on 2x2x2
blocks and short enough for exact sums, and the pressure starts at zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
F = np.float32


def _neighbours(e):
    p = np.pad(e, 1)
    return (p[1:-1, 1:-1, :-2], p[1:-1, 1:-1, 2:], p[1:-1, :-2, 1:-1], p[1:-1, 2:, 1:-1], p[:-2, 1:-1, 1:-1],
            p[2:, 1:-1, 1:-1])


def _sweeps(b, n, divides):
    """n red-black sweeps from zero with h^2 = 4, Dirichlet top"""
    e = np.zeros_like(b)
    diag = sum((s != 0).astype(F) for s in _neighbours(np.ones_like(b)))
    diag[:, -1, :] += F(1)
    colour = np.indices(b.shape).sum(0) & 1
    inner = diag == 6 if b.shape[2] % 8 == 0 else sum(s != 0 for s in _neighbours(np.ones_like(b))) == 6
    sixth = np.zeros_like(inner) if divides else inner
    for _ in range(n):
        for c in (0, 1):
            xm, xp, ym, yp, zm, zp = _neighbours(e)
            t = ((((xm + xp) + ym) + yp) + zm) + zp - F(4) * b
            e = np.where(colour == c, np.where(sixth, t * (F(1) / F(6)), t / diag), e)
    return e


def _up(e, axis, top, second):
    """Linear interpolation along an axis; the fused product is b t or a (1 - t)."""
    nc = e.shape[axis]
    x = np.arange(2 * nc)
    c = (((x + 0.5).astype(F) / F(2 * nc)).astype(np.float64) * nc - 0.5).astype(F)
    t = (c - np.floor(c)).astype(F)
    i = (x + 1) // 2 - 1
    tap = [np.take(e, np.clip(i + k, 0, nc - 1), axis) for k in (0, 1)]
    sh = [1, 1, 1]
    sh[axis] = -1
    if top:
        tap[1] = np.where((i + 1 >= nc).reshape(sh), F(0), tap[1])
    t = t.reshape(sh)
    s = F(1) - t
    if second:
        return (tap[1].astype(np.float64) * t + (tap[0] * s).astype(np.float64)).astype(F)
    return (tap[0].astype(np.float64) * s + (tap[1] * t).astype(np.float64)).astype(F)


@pytest.mark.parametrize("coarse,divides", [
    ((16, 24, 20), True),     # one CTA
    ((32, 32, 8), True),      # its limit of 4096 cells of a colour
    ((32, 34, 8), True),      # a cluster of eight
    ((64, 64, 16), True),     # its limit
    ((64, 66, 16), True),     # eight slabs of two planes, half by half
    ((48, 64, 48), True),     # of six planes
    ((50, 66, 48), True),     # rows that are not multiples of 8
    ((80, 80, 4), True),      # four slabs
    ((96, 64, 4), True),
    ((60, 62, 6), True),      # two slabs
    ((64, 62, 14), False),    # cells for a cluster of eight, but no slabs that hold them
    ((80, 80, 32), True),     # 204800 cells
    ((82, 80, 32), False),
    ((88, 80, 32), False),
])
def test_coarsest_sweeps(gpu_lib, coarse, divides):
    from dropfluid import DropFluid, abi
    c = abi.config_reference()
    c.nx, c.ny, c.nz = (2 * n for n in coarse)
    c.mg_levels, c.mg_pre, c.mg_post, c.mg_coarse_sweeps, c.mg_cycles, c.reference_schedule = 2, 0, 0, 3, 1, 0
    c.parcel_capacity = 64
    b = np.random.default_rng(sum(coarse)).integers(-999, 1000, coarse[::-1]).astype(F) / F(1024)
    sim = DropFluid(c)
    sim.set_field(abi.FIELD_RHS, np.kron(b, np.ones((2, 2, 2), F)))
    sim.set_field(abi.FIELD_PRESSURE, np.zeros([2 * n for n in b.shape], F))
    sim.run_stage(abi.STAGE_PRESSURE_SOLVE)
    got = sim.get_field(abi.FIELD_PRESSURE)
    sim.close()
    e = _sweeps(b, 3, divides)
    want = [_up(_up(_up(e, 2, False, s), 1, True, s), 0, False, s) for s in (True, False)]
    assert any(np.array_equal(got, w) for w in want), [np.abs(got - w).max() for w in want]
