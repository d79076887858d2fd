"""Marker lists of changing length on one handle, against a fresh handle per list.

The kept buffers (both marker buffers, schedule, cells, scratch) must carry nothing
from one list to the next: same kernels on the same values, so the tolerance is zero."""
import numpy as np
import pytest

from tests.test_gpu_schedule import ALPHA, BETA, markers

pytestmark = pytest.mark.gpu

LENGTHS = (500, 500, 3000, 3000, 1500, 6000, 6000, 0, 2000, 1000, 5000, 5000)


def outputs(cu):
    return cu.read_force(), cu.read_touched(), cu.read_markers()


@pytest.mark.parametrize("double", [False, True])
def test_lists_of_changing_length(gpu, double):
    tb = gpu
    dims = (20, 14, 22)
    cu = tb.ComputeUnit(x=dims[0], y=dims[1], z=dims[2], nu=1e-3)
    cu.initialise(1.0)
    if double:
        cu.forcing(markers(tb, np.random.default_rng(1), 1200, dims), ALPHA, BETA)
        cu.forcing(markers(tb, np.random.default_rng(2), 900, dims), ALPHA, BETA)
        cu.doubleResolutionFullCU()
        dims = (cu.x, cu.y, cu.z)
    rng = np.random.default_rng(7)
    for n in LENGTHS:
        mk = markers(tb, rng, n, dims)
        if n == 1500:   # a longer list that is refused leaves everything in place
            wrong = markers(tb, rng, 8000, dims)
            wrong["j"][7000] = dims[1]
            with pytest.raises(tb.TdlbError, match="marker 7000 at"):
                cu.set_markers(wrong)
        cu.initialise(1.0)
        cu.forcing(mk, ALPHA, BETA)
        cu.forcing_resident(ALPHA, BETA)
        fresh = tb.ComputeUnit(x=dims[0], y=dims[1], z=dims[2], nu=1e-3)
        fresh.initialise(1.0)
        fresh.forcing(mk, ALPHA, BETA)
        fresh.forcing_resident(ALPHA, BETA)
        for got, want in zip(outputs(cu), outputs(fresh)):
            np.testing.assert_array_equal(got, want, err_msg=f"{n} markers")
        np.testing.assert_array_equal(cu.read_markers(), mk)
        fresh.close()
    cu.close()
