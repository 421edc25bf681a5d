"""The paths that a rigid or mixed frame takes by its size, bit for bit against
the oracle: one CTA, four, eight or sixteen or a launch per color for the
iterations; one block, a cluster or launched passes for the coloring; a frame
that needs more colors than its graph was built for; manifolds of one to eight
points shared out to the lanes; and, for particles, colors of more blocks than
the device holds and elements that do not fit the staged tables."""
import math

import numpy as np
import pytest

from avbd_b200 import demos
from avbd_b200.scene import PhysicsScene, SceneSpring, SceneTet
from avbd_b200.solver import GPUSolver

pytestmark = pytest.mark.gpu


def _same(g, o, what):
    for a, b in zip(g.positions(), o.positions()):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), what


def _run(scene, oracle_lib, frames, every=1):
    g, o = GPUSolver(scene), oracle_lib.OracleSolver(scene, threads=8)
    for f in range(0, frames, every):
        g.step(every)
        assert o.step(every) == 0
        _same(g, o, f"frame {f + every}")
    return g


def pile(count, layers=4):
    """Boxes in columns, a little apart: colors appear as they land."""
    s = PhysicsScene("pile")
    demos.add_ground(s, friction=0.6)
    side = max(1, int(math.ceil(math.sqrt(count / layers))))
    for k in range(count):
        col, layer = k % (side * side), k // (side * side)
        s.add_body((0.3, 0.3, 0.3), 500.0, 0.6, ((col % side) * 0.32, (col // side) * 0.32, 0.18 + 0.34 * layer))
    s.settings.iterations = 6
    return s


@pytest.mark.parametrize("count", [1, 32, 33, 64, 65, 128, 129, 300, 511, 512, 513])
def test_iteration_paths(cuda_lib, oracle_lib, count):
    _run(pile(count), oracle_lib, 24, every=4)


@pytest.mark.parametrize("count", [1022, 1023, 1024, 4096])
def test_coloring_sizes(cuda_lib, oracle_lib, count):
    # with the ground, 1,023 boxes are the last scene of the one-block coloring
    # and 4,095 the last of the four-CTA cluster
    _run(pile(count), oracle_lib, 12, every=6)


@pytest.mark.parametrize("count,length", [(10239, 12), (10240, 12), (10240, 40), (32768, 40)])
def test_coloring_passes(cuda_lib, oracle_lib, count, length):
    """Rows of touching boxes, all of one color at first: a pass settles one box
    of each row.  With the ground, 10,239 boxes are the last scene of the eight-CTA
    cluster; above it the passes are launched, rows of 12 settle in the passes that
    follow the launched eight, and rows of 40 only in the repair.  Above 32,767
    boxes all twenty passes are launched."""
    s = PhysicsScene("rows")
    demos.add_ground(s, friction=0.6)
    for k in range(count):
        s.add_body((0.3, 0.3, 0.3), 500.0, 0.6, ((k % length) * 0.298, (k // length) * 0.5, 0.15))
    s.settings.iterations = 3
    _run(s, oracle_lib, 3)


def falling(count):
    """Four layers of boxes, each shifted against the one below: one color in
    the air (up to frame 16), four once they have landed (from frame 32)."""
    s = PhysicsScene("falling")
    demos.add_ground(s, friction=0.6)
    side = int(math.ceil(math.sqrt(count / 4)))
    for k in range(count):
        col, layer = k % (side * side), k // (side * side)
        s.add_body((0.3, 0.3, 0.3), 500.0, 0.6, ((col % side) * 0.34 + 0.15 * (layer % 2),
                                                 (col // side) * 0.34 + 0.15 * (layer // 2 % 2), 0.5 + 0.4 * layer))
    s.settings.iterations = 6
    return s


@pytest.mark.parametrize("count", [640, 2600])
def test_more_colors_than_launched(cuda_lib, oracle_lib, count):
    """The color bound is fitted while the boxes are apart; the frames in which
    they land are submitted without a retirement between, so that the launch of
    the only color solves all of them.  (Above 512 bodies: a launch per color.)"""
    import time
    import torch
    s = falling(count)
    g, o = GPUSolver(s), oracle_lib.OracleSolver(s, threads=8)
    g.step(9)                                    # seven of them time the block shapes
    assert o.step(9) == 0
    _same(g, o, "in the air")                    # retired: the bound is one color
    assert g.counters().used_colors == 1
    g.step(1)
    one = g.profile()["kernels_per_frame"]

    def burst():
        torch.cuda.synchronize()                 # waits without retiring
        t = time.perf_counter()
        g.step(20)
        torch.cuda.synchronize()
        return time.perf_counter() - t

    g.step(30)
    unfitted = burst()
    assert o.step(51) == 0
    _same(g, o, "landed")
    used = g.counters().used_colors
    assert used >= 3
    g.step(4)                                    # captures the graphs of the fitted bound
    assert g.profile()["kernels_per_frame"] >= one + s.settings.iterations * (used - 1)
    fitted = min(burst() for _ in range(3))
    # one block for the other colors takes 5 to 60 times a launch per color
    assert unfitted < 2.5 * fitted, (unfitted, fitted)


def test_shapes_between_the_paths(cuda_lib, oracle_lib):
    for count in (60, 140):
        _run(demos.shapes_scene(seed=3, count=count), oracle_lib, 60, every=10)


def test_staged_large_color(cuda_lib, oracle_lib):
    """Above 444 blocks of 16 bodies a color does not take its contacts ahead."""
    s = demos.soft_cube_scene(n=26)
    s.settings.iterations = 4
    g = _run(s, oracle_lib, 9, every=3)
    assert max(g.counters().color_counts) > 444 * 16


def rods(levers):
    """Hard and soft springs of particles under a cloth scene's kinds; with
    `levers`, anchors off the particles' centres."""
    s = demos.drape_scene(res=10)
    first = len(s.bodies)
    for k in range(12):
        s.add_particle(0.02, 0.05, position=(5.0 + 0.2 * k, 0.0, 1.0))
    for k in range(11):
        a = (0.01, 0.0, 0.0) if levers else (0, 0, 0)
        s.add_spring(SceneSpring(first + k, first + k + 1, a, (0, 0, 0), 200.0 if k % 2 else 1e5, hard=k % 2 == 0))
    return s


@pytest.mark.parametrize("levers", [False, True])
def test_staged_springs(cuda_lib, oracle_lib, levers):
    _run(rods(levers), oracle_lib, 20, every=5)


@pytest.mark.parametrize("tets", [80, 84, 90, 300])
def test_staged_reference_limit(cuda_lib, oracle_lib, tets):
    """A hub of `tets` tets refers to 3 tets + 1 bodies: 253 fit a byte with
    one to spare, 271 do not and take the grouped kernel, in one color with
    particles that are staged."""
    s = PhysicsScene("hub")
    s.settings.iterations = 8
    demos.add_ground(s, friction=0.5)
    hub = s.add_particle(0.02, 0.05, position=(0.0, 0.0, 2.0))
    for k in range(tets):
        z = 1.0 - 2.0 * (k + 0.5) / tets
        r, phi = math.sqrt(max(0.0, 1.0 - z * z)), k * 2.399963229728653
        d = np.array([r * math.cos(phi), r * math.sin(phi), z])
        u = np.cross(d, [0.0, 0.0, 1.0] if abs(z) < 0.9 else [1.0, 0.0, 0.0])
        u /= np.linalg.norm(u)
        c = np.array([0.0, 0.0, 2.0]) + 0.5 * d
        ids = [s.add_particle(0.01, 0.02, position=tuple(c + 0.04 * w)) for w in (u, np.cross(d, u), d)]
        s.add_tet(SceneTet((hub, *ids), 500.0, 2000.0))
    _run(s, oracle_lib, 10, every=2)
