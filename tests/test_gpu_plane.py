"""The XZ plane dump's records against the fields read back: the same kernels'
moments and force, so the tolerance is zero. Sizes around the 256-cell blocks."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CX = (1, -1, 0, 0)
CY = (0, 0, 1, -1)


def tank(tb, dims, streaming, steps):
    x, y, z = dims
    rng = np.random.default_rng(2)
    mk = np.zeros(60, tb.MARKER_DTYPE)
    for name, hi in zip("ijk", dims):
        mk[name] = rng.integers(0, hi, len(mk))
    for name in ("uDelta", "wDelta"):
        mk[name] = rng.uniform(-0.05, 0.05, len(mk))
    cu = tb.ComputeUnit(x=x, y=y, z=z, nu=1e-3, cs0=0.1, useLES=1, streaming=streaming)
    cu.set_markers(mk)
    cu.initialise(1.0)
    cu.forcing_resident(0.97, 1.9)
    for _ in range(steps):
        cu.step(0.97, 1.9)
    return cu, mk


def slots(cu, j, streaming):
    m = cu.read_moments()
    if streaming == "Simple":
        return m[:, j, :, :4]
    out = []
    for s in range(4):
        d = s if cu.evenStep else s ^ 1
        out.append(np.roll(m[..., d], (int(CX[d] < 0), int(CY[d] < 0), 0), (0, 1, 2))[:, j])
    return np.stack(out, -1)


@pytest.mark.parametrize("streaming,steps", [("Simple", 3), ("Esotwist", 3), ("Esotwist", 4)])
@pytest.mark.parametrize("dims,excluded", [((16, 5, 16), 0), ((15, 4, 17), 30), ((3, 2, 5), 4), ((33, 3, 40), 60)])
def test_records_equal_the_fields(gpu, streaming, steps, dims, excluded):
    tb = gpu
    x, y, z = dims
    cu, mk = tank(tb, dims, streaming, steps)
    out = np.zeros((x, y, z), bool)
    if excluded:
        cu.set_output_exclude(mk[:excluded])
        out[mk["i"][:excluded], mk["j"][:excluded], mk["k"][:excluded]] = True
    force = cu.read_force()
    for j in range(y):
        q, f = cu.plane_xz(j)
        i, k = np.nonzero(~out[:, j])
        np.testing.assert_array_equal(q["iGrid"], i)
        np.testing.assert_array_equal(q["kGrid"], k)
        assert (q["jGrid"] == j).all()
        np.testing.assert_array_equal(q["q"], slots(cu, j, streaming)[i, k])
        i, k = np.nonzero(~out[:, j] & (force[:, j] != 0).any(-1))
        np.testing.assert_array_equal(f["iGrid"], i)
        np.testing.assert_array_equal(f["kGrid"], k)
        assert (f["jGrid"] == j + 1).all()
        np.testing.assert_array_equal(f["q"], force[i, j, k])
    cu.close()


def test_counts_and_capacity(gpu):
    tb = gpu
    cu, _ = tank(tb, (15, 4, 17), "Simple", 2)
    nq, nf = ctypes.c_size_t(), ctypes.c_size_t()
    call = lambda q, nqc, f, nfc: cu.lib.tdlb_plane_xz(cu.h, 1, q, nqc, ctypes.byref(nq), f, nfc, ctypes.byref(nf))  # noqa: E731
    assert call(None, 0, None, 0) == 0 and nq.value == 15 * 17
    q = np.zeros(100, tb.DISK_GRID4_DTYPE)
    assert call(tb._p(q), len(q), None, 0) == -1          # too small: the records that fit, and the count
    assert nq.value == 15 * 17
    np.testing.assert_array_equal(q, cu.plane_xz(1)[0][:100])
    cu.close()
