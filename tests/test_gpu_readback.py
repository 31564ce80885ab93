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


def test_reading_into_a_used_buffer_costs_the_copy(gpu_lib):
    """A buffer that has its pages is not populated again: one call over 256 MB
    takes no longer than forty calls over its pieces of less than 8 MB, which
    are never populated."""
    import ctypes
    import time
    from dropfluid import DropFluid, abi
    cfg = abi.config_closed_box(16, 16, 16)
    n, pieces = 8000000, 40
    cfg.parcel_capacity = n
    sim = DropFluid(cfg)
    out = np.zeros((n, abi.PARCEL_FLOATS), np.float32)
    out += 1.0  # backed with memory

    def read(first, count):
        p = out[first:].ctypes.data_as(ctypes.POINTER(ctypes.c_float))
        assert gpu_lib.dob_get_parcels(sim._h, p, count, first) == 0

    def whole():
        read(0, n)

    def parts():
        for k in range(pieces):
            read(k * (n // pieces), n // pieces)

    def best(f):
        times = []
        for _ in range(20):
            t = time.perf_counter()
            f()
            times.append(time.perf_counter() - t)
        return min(times)

    best(parts)
    assert best(whole) <= best(parts)
    sim.close()
