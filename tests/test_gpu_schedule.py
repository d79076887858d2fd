"""The device's marker scheduler (csrc/schedule.cu): force, touched flags and list
checks against the CPU restatement, which applies the markers one by one in
list order.

A marker's update rounds as the restatement's does up to fused multiply-adds:
about 20 FP32 operations, relative error at most 20 * 2^-24 = 1.2e-6 of the
cell's largest term per update; updates of a cell shrink earlier errors by
alpha (0.97), so a chain of any length stays within 1.2e-6 / 0.03 = 4e-5 of the
field's norm.
"""
import numpy as np
import pytest

from tests.test_gpu_parity import rel_l2

pytestmark = pytest.mark.gpu

ALPHA, BETA = 0.97, 1.9
TOL = 4e-5


def markers(tb, rng, n, dims, **fixed):
    m = np.zeros(n, tb.MARKER_DTYPE)
    for name, hi in zip("ijk", dims):
        m[name] = fixed.get(name, rng.integers(0, hi, n))
    for name in ("iCartFraction", "kCartFraction"):
        m[name] = rng.uniform(-0.5, 0.5, n)
    for name in ("uDelta", "vDelta", "wDelta"):
        m[name] = rng.uniform(-0.05, 0.05, n)
    return m


def ring(tb, rng, dims, planes):
    """Markers along a ring in ring order: each overlaps the one before it."""
    x, _, z = dims
    r = min(x, z) / 2 - 3
    th = np.arange(0, 2 * np.pi, 1 / r)
    out = []
    for j in planes:
        m = markers(tb, rng, len(th), dims, j=j)
        a, c = (x - 1) / 2 + r * np.cos(th), (z - 1) / 2 + r * np.sin(th)
        m["i"], m["k"] = np.rint(a), np.rint(c)
        out.append(m)
    return np.concatenate(out)


def lists(tb):
    rng = np.random.default_rng(11)
    return {
        "empty": ((9, 4, 8), markers(tb, rng, 0, (9, 4, 8))),
        "one": ((3, 1, 3), markers(tb, rng, 1, (3, 1, 3))),
        "narrow": ((2, 3, 1), markers(tb, rng, 40, (2, 3, 1))),
        "one chunk and one more": ((12, 33, 17), markers(tb, rng, 1025, (12, 33, 17))),
        "chains": ((40, 5, 36), ring(tb, rng, (40, 5, 36), [0, 2, 4])),
        "a crowded plane": ((80, 6, 90), markers(tb, rng, 9000, (80, 6, 90), j=3)),
        "a pile beyond the rounds": ((8, 3, 8), np.concatenate([markers(tb, rng, 4200, (8, 3, 8), i=4, j=1, k=4),
                                                                markers(tb, rng, 60, (8, 3, 8))])),
        "a plane beyond shared memory": ((840, 2, 800), markers(tb, rng, 3000, (840, 2, 800))),
    }


@pytest.mark.parametrize("name", ["empty", "one", "narrow", "one chunk and one more", "chains", "a crowded plane",
                                  "a pile beyond the rounds", "a plane beyond shared memory"])
def test_forcing_of_a_list_equals_list_order(gpu, port_oracle, name):
    tb, po = gpu, port_oracle
    (x, y, z), mk = lists(tb)[name]
    cu = tb.ComputeUnit(x=x, y=y, z=z, nu=1e-3, cs0=0.1, useLES=1)
    lat = po.CpuLattice("port", x, y, z, po.Flow(initialRho=1.0, nu=1e-3, cs0=0.1, useLES=True), "Simple", 4)
    cu.initialise(1.0)
    lat.initialise(1.0)
    for _ in range(2):   # the second pass starts from the first one's force
        cu.forcing(mk, ALPHA, BETA)
        lat.forcing(mk, ALPHA, BETA)
    got, want = cu.read_force(), lat.interior(lat.get_f())
    assert np.isfinite(got).all()
    assert rel_l2(got, want) <= TOL
    # the same list kept resident gives the same bits
    cu.initialise(1.0)
    cu.set_markers(mk)
    for _ in range(2):
        cu.forcing_resident(ALPHA, BETA)
    np.testing.assert_array_equal(cu.read_force(), got)
    touched = np.zeros((x, y, z), np.uint8)
    for di in (-1, 0, 1):
        for dk in (-1, 0, 1):
            touched[(mk["i"] + di) % x, mk["j"], (mk["k"] + dk) % z] = 1
    np.testing.assert_array_equal(cu.read_touched(), touched)
    cu.close()


def test_a_list_with_a_marker_outside_leaves_the_resident_one(gpu):
    tb = gpu
    dims = (12, 7, 11)
    good = markers(tb, np.random.default_rng(3), 300, dims)
    cu = tb.ComputeUnit(x=dims[0], y=dims[1], z=dims[2], nu=1e-3)
    cu.initialise(1.0)
    cu.set_markers(good)
    for name, bad in (("i", 12), ("j", -1), ("k", 11)):
        wrong = good.copy()
        wrong[name][170] = bad
        with pytest.raises(tb.TdlbError, match="marker 170 at"):
            cu.set_markers(wrong)
        np.testing.assert_array_equal(cu.read_markers(), good)
    cu.forcing_resident(ALPHA, BETA)
    cu.close()
