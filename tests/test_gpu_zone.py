"""Split steps word by word: the outer launch (every word outside the zone), the
inner launch (the zone's words, without the residual box's cells) and the box
launch together store every cell once, with the arithmetic of the unsplit
step. So the tolerance is zero, whatever the cells per thread, the row length
against the 32-cell words and the 4-cell granule, and the box's place."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ALPHA, BETA = 0.97, 1.9


def run(tb, dims, streaming, storage, vec, box, overlap, steps=6):
    x, y, z = dims
    rng = np.random.default_rng(5)
    mk = np.zeros(14, tb.MARKER_DTYPE)
    for name, hi in (("i", x), ("j", y), ("k", z)):
        mk[name] = rng.integers(0, hi, len(mk))
    for name in ("iCartFraction", "kCartFraction"):
        mk[name] = rng.uniform(-0.5, 0.5, len(mk))
    for name in ("uDelta", "vDelta", "wDelta"):
        mk[name] = rng.uniform(-0.05, 0.05, len(mk))
    cu = tb.ComputeUnit(x=x, y=y, z=z, nu=1e-3, cs0=0.1, useLES=1, streaming=streaming, storage=storage)
    if vec:
        cu.set_cells_per_thread(vec)
    if storage != "fp32":
        cu.set_residual_box(*box)
    cu.set_overlap(overlap)
    cu.set_markers(mk)
    cu.initialise(1.0)
    cu.forcing_resident(ALPHA, BETA)
    for _ in range(steps):
        cu.step(ALPHA, BETA)
    rho, u = cu.read_velocity_density()
    out = dict(rho=rho, u=u, nu=cu.read_nu(), force=cu.read_force(), touched=cu.read_touched())
    cu.close()
    return out


@pytest.mark.parametrize("streaming", ["Simple", "Esotwist"])
@pytest.mark.parametrize("dims", [(12, 31, 20), (11, 64, 13), (9, 70, 12), (20, 6, 17), (14, 3, 33), (10, 97, 9)])
@pytest.mark.parametrize("storage,vec", [("fp32", 1), ("fp16", 1), ("fp16", 2), ("bf16", 4)])
def test_split_parts_store_every_cell_once(gpu, streaming, dims, storage, vec):
    x, y, z = dims
    box = (3, min(7, x), 1, min(max(2, y // 2), y), 2, min(8, z))
    a = run(gpu, dims, streaming, storage, vec, box, "always")
    b = run(gpu, dims, streaming, storage, vec, box, False)
    for key in a:
        np.testing.assert_array_equal(a[key], b[key], err_msg=key)


@pytest.mark.parametrize("streaming", ["Simple", "Esotwist"])
@pytest.mark.parametrize("storage", ["fp16", "bf16"])
def test_box_cells_left_out_of_the_plain_launch(gpu, streaming, storage):
    """A box against none over one step from rest: the cells away from the box
    and from the markers hold the same values."""
    dims = (16, 40, 16)
    a = run(gpu, dims, streaming, storage, 0, (5, 9, 8, 30, 5, 9), False, steps=1)
    b = run(gpu, dims, streaming, storage, 0, (0, 0, 0, 0, 0, 0), False, steps=1)
    far = np.ones(dims, bool)
    far[3:11, 6:32, :] = False
    np.testing.assert_array_equal(a["touched"], b["touched"])
    np.testing.assert_array_equal(a["rho"][far], b["rho"][far])
    np.testing.assert_array_equal(a["u"][far], b["u"][far])
