"""Several steps in one launch (lbm_scheme_multi_step) against single steps.

The region kernel holds the values in the storage type and runs the same
generated collision, so the populations, ghost layer included, must be those
of single launches bit for bit: periodic grids (smaller than a region, odd,
wider than one), box walls, and boundary links of every method on obstacles,
for each region shape and for the rule's choice.
"""
import numpy as np
import pytest

from pylbm_gb300 import Simulation
from pylbm_gb300 import workloads as W

pytestmark = pytest.mark.gpu

FLOWS = {
    "shear8": lambda: W.shear_layer(n=8),
    "shear97": lambda: W.shear_layer(n=97),
    "shear128": lambda: W.shear_layer(n=128),
    "cavity33": lambda: W.cavity(n=33),
    "cavity96": lambda: W.cavity(n=96),
    "disc": lambda: W.cylinder(nx=131, ny=48, radius=3, center=(26, 25), re=18.75),
    "karman": lambda: W.karman(dx=1.0 / 64),
}
C0 = {"disc": [1.0, 0.05, 0.0], "karman": [1.0, 0.05, 0.0]}
# shape and margin; the last is the rule's choice
PLANS = [(0, 5), (0, 10), (1, 6), (2, 3), (2, 8), (-1, 0)]


def _populations(sim):
    return np.array([sim.F_halo[k] for k in range(sim.scheme.nv)])


@pytest.mark.parametrize("flow, dtype", [(f, "float32") for f in FLOWS] +
                         [("shear97", "float16"), ("shear128", "bfloat16"), ("cavity33", "float16")])
def test_multi_step_equals_single_steps(flow, dtype):
    def make():
        return Simulation(FLOWS[flow](), dtype=dtype, c0=C0.get(flow, [1.0, 0.0, 0.0]))

    single = make()
    single.multi_step = False
    single.run(23)
    ref = _populations(single)
    single.free()
    assert np.all(np.isfinite(ref))
    for shape, margin in PLANS:
        sim = make()
        mode = sim._multi_mode()
        assert mode is not None
        assert sim._multi_plan(mode, shape, margin) is not None
        sim.run(23)
        assert sim.nt == 23
        assert np.array_equal(_populations(sim), ref), (shape, margin)
        sim.free()


def _box3d(n, walls):
    """Taylor-Green vortex or cube on n[0] x n[1] x n[2] nodes."""
    d = W.cavity3d(n=n[0]) if walls else W.tgv3d(n=n[0])
    dx = d["space_step"]
    for axis, k in zip("xyz", n):
        d["box"][axis] = [0.0, k * dx]
    return d


def _advection3d():
    from demo_cases import advection_3d
    return advection_3d(dx=1.0 / 36)


BOXES = {
    "tgv24": lambda: _box3d((24, 24, 24), False),
    "tgv_flat": lambda: _box3d((9, 40, 71), False),
    "tgv_tall": lambda: _box3d((45, 6, 33), False),
    "cube17": lambda: _box3d((17, 17, 17), True),
    "cube_flat": lambda: _box3d((8, 23, 70), True),
    "cube_tall": lambda: _box3d((46, 13, 10), True),
    "d3q6": _advection3d,
}


@pytest.mark.parametrize("box", list(BOXES))
def test_two_steps_3d_equal_single_steps(box):
    """Every split of the outermost axis the rule can take, and its choice."""
    def make():
        d = BOXES[box]()
        return Simulation(d, dtype="float32", c0=None if box == "d3q6" else [1.0, 0.0, 0.0, 0.0])

    single = make()
    single.multi_step = False
    single.run(11)
    ref = _populations(single)
    n0 = single.domain.shape_in[0]
    single.free()
    assert np.all(np.isfinite(ref))
    splits = sorted({-(-n0 // t) for t in range(1, (n0 + 3) // 4 + 1)})
    for planes in splits:
        sim = make()
        multi = sim._multi_plan(sim._multi_mode(), planes, 0)
        assert multi is not None and multi[0].planes == planes
        sim.run(11)
        assert np.array_equal(_populations(sim), ref), (planes, multi[0].out[:], multi[0].tiles[:])
        sim.free()


@pytest.mark.parametrize("walls", [False, True])
def test_two_steps_3d_columns(walls):
    """Columns of the narrowest and widest cross-sections a block can hold."""
    from pylbm_gb300 import runtime

    n = (9, 64, 75)
    c0 = [1.0, 0.0, 0.0, 0.0]
    single = Simulation(_box3d(n, walls), dtype="float32", c0=c0)
    single.multi_step = False
    single.run(8)
    ref = _populations(single)
    single.free()
    for out in ((7, 69), (62, 8), (8, 57), (18, 30), (9, 55), (1, 1)):
        sim = Simulation(_box3d(n, walls), dtype="float32", c0=c0)
        mode = sim._multi_mode()
        plan, bnd = sim._multi_plan(mode, 5, 0)
        plan = runtime.TilePlan.from_buffer_copy(plan)
        for d in range(2):
            plan.out[d], plan.tiles[d] = out[d], -(-n[1 + d] // out[d])
        sim._multi[mode] = (plan, bnd)
        sim.run(8)
        assert np.array_equal(_populations(sim), ref), out
        sim.free()


def test_captured_launches_continue_the_run():
    runs = []
    for multi in (True, False):
        sim = Simulation(W.shear_layer(n=97), dtype="float32", c0=[1.0, 0.0, 0.0])
        sim.multi_step = multi
        for steps in (500, 3, 700, 2):
            sim.run(steps)
        assert sim.nt == 1205
        runs.append(_populations(sim))
        sim.free()
    assert np.array_equal(*runs)


@pytest.mark.parametrize("flow", ["cavity33", "karman"])
def test_captured_single_steps_equal_calls(flow):
    """Runs long enough for the graph of sixteen steps, its remainder and an odd step."""
    runs = []
    for captured in (True, False):
        sim = Simulation(FLOWS[flow]())
        for steps in (37, 35, 5):
            if captured:
                sim.run(steps)
            else:
                for _ in range(steps):
                    sim.one_time_step()
        assert sim.nt == 77
        runs.append((_populations(sim), sim.t))
        sim.free()
    assert np.array_equal(runs[0][0], runs[1][0]) and runs[0][1] == runs[1][1]


def test_single_steps_remain_where_they_must():
    sim = Simulation(W.cavity(n=32))   # FP64
    assert sim._multi_mode() is None
    sim.free()
    sim = Simulation(W.karman(dx=1.0 / 64), dtype="float32", c0=C0["karman"], halo="full")
    assert sim._multi_mode() is None
    sim.free()
    sim = Simulation(W.tgv3d(n=16), dtype="float16")   # 3D in 16 bits, and small 3D grids
    assert sim._multi_plan(sim._multi_mode()) is None
    sim.free()
    sim = Simulation(W.tgv3d(n=16), dtype="float32")
    assert sim._multi_plan(sim._multi_mode()) is None
    sim.free()
