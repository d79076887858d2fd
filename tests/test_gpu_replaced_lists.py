"""Markers replaced between a forcing pass and the next step, the reference's own
order of work (main.cpp:409-454: geometry, collision, forcing).

A step uses the force of the last pass, whichever list that pass applied, so
setting the new markers before the collision or after it is the same run, and so
is splitting the steps or not: the tolerance is zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ALPHA, BETA = 0.97, 1.9
EDGE = 96                 # above 2^19 cells: steps split unasked


def unit(tb, streaming, storage, overlap):
    cu = tb.ComputeUnit(x=EDGE, y=EDGE, z=EDGE, nu=1e-3, cs0=0.1, useLES=1, streaming=streaming, storage=storage)
    if overlap is not None:
        cu.set_overlap(overlap)
    return cu


def outputs(cu):
    rho, u = cu.read_velocity_density()
    out = dict(rho=rho, u=u, nu=cu.read_nu(), force=cu.read_force(), touched=cu.read_touched())
    cu.close()
    return out


def same(a, b):
    for key in a:
        np.testing.assert_array_equal(a[key], b[key], err_msg=key)


def sphere(tb, at, r=9):
    """Markers of a small ball about `at`: a few words of the lattice."""
    g = np.stack(np.meshgrid(*[np.arange(-r, r + 1, 3)] * 3, indexing="ij"), -1).reshape(-1, 3)
    g = g[(g ** 2).sum(1) <= r * r]
    m = np.zeros(len(g), tb.MARKER_DTYPE)
    for q, name in enumerate("ijk"):
        m[name] = at[q] + g[:, q]
    m["uDelta"], m["wDelta"] = 0.05, -0.03
    return m


@pytest.mark.parametrize("streaming", ["Simple", "Esotwist"])
@pytest.mark.parametrize("storage,box", [("fp32", False), ("fp16", False), ("fp16", True)])
def test_a_moving_geometry(gpu, streaming, storage, box):
    """A ball set anew each step, before the collision, against after it."""
    tb = gpu

    def run(early, overlap):
        cu = unit(tb, streaming, storage, overlap)
        if box:
            cu.set_residual_box(30, 50, 30, 50, 30, 50)
        cu.initialise(1.0)
        cu.set_markers(sphere(tb, (30, 40, 40)))
        cu.forcing_resident(ALPHA, BETA)
        for s in range(1, 6):
            new = sphere(tb, (30 + 7 * s, 40, 40 + 5 * (s % 2)))
            if early:
                cu.set_markers(new)
            cu.collision()
            if not early:
                cu.set_markers(new)
            for _ in range(2):        # the second pass finds a list that stays
                cu.forcing_resident(ALPHA, BETA)
                cu.collision()
            cu.forcing_resident(ALPHA, BETA)
        return outputs(cu)

    want = run(False, False)
    for early in (True, False):
        for overlap in (None, False, "always"):
            same(run(early, overlap), want)


@pytest.mark.parametrize("streaming", ["Simple", "Esotwist"])
def test_another_impeller(gpu, streaming):
    """Attaching another tank's impeller, or one after a plain list, before the collision."""
    tb = gpu
    rts = [tb.RushtonTurbine(EDGE, EDGE, EDGE, tip_speed=0.1, startup_steps=0, impeller_diameter=dia, clearance=c)
           for dia, c in ((32.0, 32.0), (44.0, 60.0))]
    d = rts[0].increment(1)

    def run(early, overlap):
        cu = unit(tb, streaming, "fp32", overlap)
        cu.initialise(1.0)
        cu.forcing(sphere(tb, (48, 20, 48)), ALPHA, BETA)
        for rt in (*rts, rts[0]):
            if early:
                cu.attach_rushton(rt, d, 0.1, d)
            cu.collision()
            if not early:
                cu.attach_rushton(rt, d, 0.1, d)
            for s in range(3):
                cu.rotate_impeller(0.1 + d * s, d)
                cu.forcing_resident(ALPHA, BETA)
                cu.collision()
            cu.forcing_resident(ALPHA, BETA)
        return outputs(cu)

    want = run(False, False)
    for early in (True, False):
        for overlap in (None, False, "always"):
            same(run(early, overlap), want)


@pytest.mark.parametrize("streaming,storage", [("Simple", "fp32"), ("Esotwist", "fp32"), ("Esotwist", "fp16")])
def test_host_blades_that_come_back_into_the_swept_volume(gpu, streaming, storage):
    tb = gpu
    rt = tb.RushtonTurbine(EDGE, EDGE, EDGE, tip_speed=0.1, startup_steps=0)
    d = rt.increment(1)

    def run(early, overlap):
        cu = unit(tb, streaming, storage, overlap)
        cu.attach_rushton(rt, d, 0.0, d)
        cu.initialise(1.0)
        cu.forcing_resident(ALPHA, BETA)
        for s in range(1, 9):
            blades = rt.rotating(d * s, d)
            if s % 3 == 0:            # outside: towards the wall, in planes without blades too
                blades["i"] = (blades["i"] + 30) % EDGE
                blades["j"] = (blades["j"] + 17) % EDGE
            if early:
                cu.set_rotating_markers(blades)
            cu.collision()
            if not early:
                cu.set_rotating_markers(blades)
            cu.forcing_resident(ALPHA, BETA)
        return outputs(cu)

    want = run(False, False)
    for early in (True, False):
        for overlap in (None, False, "always"):
            same(run(early, overlap), want)


@pytest.mark.parametrize("streaming", ["Simple", "Esotwist"])
@pytest.mark.parametrize("first", [0, 1, 2, 3, 4])
def test_host_blades_in_other_planes(gpu, streaming, first):
    """Blades that the host moves to other planes at step `first`, before or after
    the zone of the attached ones was planned."""
    tb = gpu
    rt = tb.RushtonTurbine(EDGE, EDGE, EDGE, tip_speed=0.1, startup_steps=0)
    d = rt.increment(1)

    def run(early, overlap):
        cu = unit(tb, streaming, "fp32", overlap)
        cu.attach_rushton(rt, d, 0.0, d)
        cu.initialise(1.0)
        cu.forcing_resident(ALPHA, BETA)
        for s in range(8):
            def blades():
                if s < first:
                    cu.rotate_impeller(d * s, d)
                else:
                    moved = rt.rotating(d * s, d)
                    if s % 3 == first % 3:
                        moved["j"] = (moved["j"] + 30) % EDGE
                    cu.set_rotating_markers(moved)
            if early:
                blades()
            cu.collision()
            if not early:
                blades()
            cu.forcing_resident(ALPHA, BETA)
        return outputs(cu)

    want = run(False, False)
    for early in (True, False):
        for overlap in (None, "always"):
            same(run(early, overlap), want)
