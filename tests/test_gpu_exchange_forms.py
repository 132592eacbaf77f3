"""The forms of dem_step_exchange that share the steps' launch: every launch
shape with the split integrator at any size, input in pageable memory, input
fields left out, calls of more steps than a launch takes.  Each leaves the
buffers as uninterrupted stepping does, bit for bit, and counts as direct."""
import ctypes as C

import numpy as np
import pytest

from taichi_dem_julia_port_gb300 import GlobalData, _abi, scenes

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "omega", "quat", "force", "moment", "wall_shear")
INPUT = ("pos", "vel", "omega", "quat", "wall_shear")


def exchange(g, arrays, steps, buf):
    """One call with the named input arrays (the others NULL) and buf's output."""
    addr = {k: a.ctypes.data for k, a in arrays.items()}
    state = _abi.DemParticleState(g.n, *(addr.get(k) for k in FIELDS))
    assert g.lib.dem_step_exchange(g.h, C.byref(state), steps, C.byref(buf._out)) == _abi.DEM_OK


def plain(sc, steps, lead=0):
    with GlobalData(sc.cfg, sc.particles) as g:
        g.initialize()
        g.simulate(lead + steps)
        return g.particles()


def same(buf, want, what):
    for k in FIELDS:
        np.testing.assert_array_equal(getattr(buf, k), want[k], err_msg=f"{k} {what}")


@pytest.mark.parametrize("per_call", [1, 7])
@pytest.mark.parametrize("shape", [dict(integrate_lanes=4), dict(list_lanes=1), dict(list_lanes=4),
                                   dict(dependent_launch=1), dict(dependent_launch=2),
                                   dict(list_lanes=1, integrate_lanes=4, dependent_launch=1)])
def test_every_split_launch_shape(gpu, shape, per_call):
    """Into a wall impact, exchanged and plain steps in turn."""
    sc = scenes.bonded_cube(8, speed=30.0, steps=0, seed=2)
    want = plain(sc, 280)
    with GlobalData(sc.cfg, sc.particles) as g:
        g.set_launch_shape(**shape)
        g.initialize()
        g.simulate(140)
        buf = g.state_buffers(forces=True)
        for _ in range(70 // per_call):
            buf.step(per_call)
        g.simulate(35)
        buf.download()
        for _ in range(35 // per_call):
            buf.step(per_call)
        same(buf, want, f"{shape}")
        assert g.stats()["exchanges_direct"] == 105 // per_call
        buf.close()
    assert np.any(want["wall_shear"] != 0.0)


@pytest.mark.parametrize("side,calls", [(34, [1, 2, 3, 1]), (47, [1, 3, 2])])
def test_split_integrator_of_a_larger_scene(gpu, side, calls):
    """integrate_lanes = 4 above 256 and 512 spheres per SM: the steps' launch
    for calls of one or two steps, the separate kernels for longer ones."""
    sc = scenes.bonded_cube(side, speed=30.0, steps=0, seed=3)
    want = plain(sc, sum(calls), lead=45)
    with GlobalData(sc.cfg, sc.particles) as g:
        g.set_launch_shape(integrate_lanes=4)
        g.initialize()
        g.simulate(45)
        buf = g.state_buffers(forces=True)
        for k in calls:
            buf.step(k)
        same(buf, want, f"{side}")
        assert g.stats()["exchanges_direct"] == sum(k <= 2 for k in calls)
        buf.close()


@pytest.mark.parametrize("paged", [INPUT, ("vel",), ("pos", "quat")])
@pytest.mark.parametrize("steps", [1, 5])
def test_pageable_input(gpu, paged, steps):
    """Some or all input fields in pageable memory, output page-locked."""
    sc = scenes.bonded_cube(8, speed=30.0, steps=0, seed=2)
    want = plain(sc, 3 * steps, lead=300)
    with GlobalData(sc.cfg, sc.particles) as g:
        g.initialize()
        g.simulate(300)
        buf = g.state_buffers(forces=True)
        for _ in range(3):
            given = {k: getattr(buf, k).copy() if k in paged else getattr(buf, k) for k in INPUT}
            exchange(g, given, steps, buf)
        same(buf, want, f"{paged} {steps}")
        assert g.stats()["exchanges_direct"] == 3
        buf.close()


@pytest.mark.parametrize("given", [("pos",), ("pos", "omega"), ("pos", "vel", "wall_shear")])
@pytest.mark.parametrize("steps", [1, 2])
def test_input_fields_left_out(gpu, given, steps):
    """NULL input fields keep the device's values; every output is written."""
    sc = scenes.bonded_cube(8, speed=30.0, steps=0, seed=2)
    want = plain(sc, steps, lead=300)
    with GlobalData(sc.cfg, sc.particles) as g:
        g.initialize()
        g.simulate(300)
        buf = g.state_buffers(forces=True)
        for k in FIELDS:
            if k not in given:
                getattr(buf, k)[:] = -7.0
        exchange(g, {k: getattr(buf, k) for k in given}, steps, buf)
        same(buf, want, f"{given} {steps}")
        assert g.stats()["exchanges_direct"] == 1
        buf.close()


@pytest.mark.parametrize("steps", [64, 65, 130])
def test_calls_longer_than_a_launch(gpu, steps):
    """The first launch of a call reads the input, its last writes the output."""
    sc = scenes.bonded_cube(8, speed=30.0, steps=0, seed=2)
    want = plain(sc, steps, lead=250)
    with GlobalData(sc.cfg, sc.particles) as g:
        g.initialize()
        g.simulate(250)
        buf = g.state_buffers(forces=True)
        for k in ("force", "moment"):
            getattr(buf, k)[:] = -7.0
        buf.step(steps)
        same(buf, want, f"{steps}")
        assert g.stats()["exchanges_direct"] == 1
        buf.close()


def test_autotuned_scene_keeps_its_exchange(gpu):
    """The autotuner leaves a scene whose steps share a launch as it is; a
    forced layout or a larger scene does have knobs."""
    from taichi_dem_julia_port_gb300.autotune import autotune
    sc = scenes.bonded_cube(8, speed=30.0, steps=0, seed=2)
    with GlobalData(sc.cfg, sc.particles) as g:
        g.initialize()
        before = g.launch_shape()
        assert g.steps_in_one_launch(152) and not g.steps_in_one_launch(1)
        r = autotune(g, steps=2)
        assert r.shape == before == g.launch_shape() and r.ms_per_step > 0.0
        g.set_launch_shape(dependent_launch=1)
        assert not g.steps_in_one_launch(152)
