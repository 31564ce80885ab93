"""A level's legs in one launch (dob_mgleg.cuh) against the launch chain they
stand for: the same bits.

With mg_coarse_sweeps = 0 the coarsest grid's correction is zero, and a level
above it smooths pre + post sweeps.  The legs cover one or two sweeps each way;
(pre + post, 0) runs the same sweeps on the chain, and so does a single grid of
the level's size.  Rows that are and are not multiples of 8 (the half-sweep
kernels k_rbgs_v4 and k_rbgs_split), both boundary modes: below a Dirichlet top
the two multiply by 1/6 and divide by 6."""
import numpy as np
import pytest

from helpers import smooth_field

pytestmark = pytest.mark.gpu


def _pressure(mode, dims, levels, pre, post, schedule):
    from dropfluid import DropFluid, abi
    c = abi.config_closed_box(*dims) if mode == "box" else abi.config_reference()
    c.nx, c.ny, c.nz = dims
    c.mg_levels, c.mg_pre, c.mg_post, c.mg_coarse_sweeps, c.mg_cycles = levels, pre, post, 0, 2
    c.reference_schedule = schedule
    c.parcel_capacity = 64
    shape = dims[::-1]
    rng = np.random.default_rng(sum(dims))
    b = smooth_field(shape, 3, 1.0) + 0.2 * rng.normal(size=shape)
    e = DropFluid(c)
    e.set_field(abi.FIELD_RHS, (b - b.mean()).astype(np.float32))
    e.set_field(abi.FIELD_PRESSURE, (smooth_field(shape, 4, 2.0) + rng.normal(size=shape)).astype(np.float32))
    e.run_stage(abi.STAGE_PRESSURE_SOLVE)
    out = e.get_field(abi.FIELD_PRESSURE)
    e.close()
    return out


SWEEPS = [(2, 2), (1, 2), (2, 1), (1, 1)]


@pytest.mark.parametrize("pre,post", SWEEPS)
@pytest.mark.parametrize("mode", ["box", "ref"])
@pytest.mark.parametrize("dims", [(28, 36, 20), (20, 24, 28), (52, 60, 28), (24, 40, 40), (48, 64, 48)])
def test_finest_grid(gpu_lib, mode, dims, pre, post):
    legs = _pressure(mode, dims, 2, pre, post, 0)
    chain = _pressure(mode, dims, 1, pre, post, 0)
    np.testing.assert_array_equal(legs, chain)


@pytest.mark.parametrize("pre,post", [(2, 2), (2, 1), (1, 2)])
@pytest.mark.parametrize("mode", ["box", "ref"])
@pytest.mark.parametrize("dims", [(24, 40, 40), (56, 80, 72), (40, 56, 24), (64, 80, 64)])
def test_second_grid(gpu_lib, mode, dims, pre, post):
    """Level 1, from zero; the finest grid runs its one sweep each way
    (reference_schedule) in legs on both sides."""
    legs = _pressure(mode, dims, 3, pre, post, 1)
    chain = _pressure(mode, dims, 3, pre + post, 0, 1)
    np.testing.assert_array_equal(legs, chain)
