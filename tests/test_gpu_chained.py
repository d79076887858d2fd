"""The launches of a step that are set up while the one before them drains do
what they do one at a time: the same calls, once with a wait for the device
after each of them and once without, give the same values. So the tolerance is
zero. The sizes give a few blocks and several waves of them; rotated and
uploaded blades, and `always`, which adds the inner words and the box."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ALPHA, BETA = 0.97, 1.9


def run(tb, dims, streaming, storage, overlap, host_blades, wait):
    x, y, z = dims
    rt = tb.RushtonTurbine(x, y, z, tip_speed=0.1, startup_steps=0)
    d = rt.increment(1)
    cu = tb.ComputeUnit(x=x, y=y, z=z, nu=1e-3, cs0=0.1, useLES=1, streaming=streaming, storage=storage)
    cu.set_overlap(overlap)
    then = cu.synchronize if wait else (lambda: None)
    cu.attach_rushton(rt, d, d, d)
    cu.initialise(1.0)
    then()
    cu.forcing_resident(ALPHA, BETA)
    then()
    angle, loads = d, []
    for s in range(2, 12):
        dd = rt.increment(s)
        angle += dd
        if host_blades:
            cu.set_rotating_markers(rt.rotating(angle, dd))
        else:
            cu.rotate_impeller(angle, dd)
        then()
        cu.collision()
        then()
        cu.forcing_resident(ALPHA, BETA)
        then()
        if s % 4 == 0:
            loads.append(cu.impeller_load())
    rho, u = cu.read_velocity_density()
    out = dict(rho=rho, u=u, nu=cu.read_nu(), force=cu.read_force(), touched=cu.read_touched(), loads=np.array(loads))
    cu.close()
    return out


@pytest.mark.parametrize("streaming", ["Simple", "Esotwist"])
@pytest.mark.parametrize("dims,overlap,host_blades", [((20, 20, 20), False, False), ((24, 24, 24), False, True),
                                                      ((41, 70, 41), False, False), ((41, 70, 41), "always", True)])
@pytest.mark.parametrize("storage", ["fp32", "fp16", "bf16"])
def test_close_launches_give_the_values_of_separate_ones(gpu, streaming, dims, overlap, host_blades, storage):
    a = run(gpu, dims, streaming, storage, overlap, host_blades, False)
    b = run(gpu, dims, streaming, storage, overlap, host_blades, True)
    for key in a:
        np.testing.assert_array_equal(a[key], b[key], err_msg=key)
