"""Field readback: what is not FP32 in natural order goes through a device
buffer of 2^21 values, and the pages of a large host buffer are populated
first.  Every value has to come back as it was stored, on both sides of the
buffer's edge and of the 8 MB from which pages are populated."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(16, 16, 16), (128, 128, 128), (136, 128, 128), (72, 344, 88)])
@pytest.mark.parametrize("mixed", [False, True])
def test_fields_come_back_as_stored(dims, mixed):
    from dropfluid import DropFluid, abi
    cfg = abi.config_closed_box(*dims)
    cfg.precision_mode = abi.DOB_PREC_MIXED if mixed else abi.DOB_PREC_FP32
    sim = DropFluid(cfg)
    rng = np.random.default_rng(sum(dims))
    shape = dims[::-1]
    p = rng.normal(size=shape).astype(np.float32)
    dye = rng.normal(size=shape).astype(np.float32) * 1e-3
    dye.flat[-1], dye.flat[0] = np.inf, 6e-8  # a subnormal binary16, and no number at the end
    sim.set_field(abi.FIELD_PRESSURE, p)
    sim.set_field(abi.FIELD_CONC, dye)
    np.testing.assert_array_equal(sim.get_field(abi.FIELD_PRESSURE), p)
    stored = dye.astype(np.float16).astype(np.float32) if mixed else dye
    np.testing.assert_array_equal(sim.get_field(abi.FIELD_CONC), stored)
