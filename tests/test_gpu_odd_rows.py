"""16-bit storage with rows of odd length: the last pair of a row holds one node.

The two-node kernels (periodic, ghost layer, box walls) must give the
populations of the one-node kernels bit for bit, at the shortest
rows, at a row of one full block and one node, and between.
"""
import numpy as np
import pytest

from pylbm_gb300 import Simulation
from pylbm_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _tgv(n0, n1, n2):
    d = W.tgv3d(n=n0)
    for axis, k in zip("xyz", (n0, n1, n2)):
        d["box"][axis] = [0.0, k * d["space_step"]]
    return d


FLOWS = {
    "tgv5": lambda: _tgv(6, 5, 5),
    "tgv35": lambda: _tgv(9, 8, 35),
    "tgv257": lambda: _tgv(4, 5, 257),
    "shear33": lambda: W.shear_layer(n=33),
    "cavity35": lambda: W.cavity(n=35),
    "cube17": lambda: W.cavity3d(n=17),
    "disc": lambda: W.cylinder(nx=131, ny=47, radius=3, center=(26, 25), re=18.75),
}


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("flow", list(FLOWS))
def test_odd_rows_equal_single_nodes(flow, dtype):
    if dtype == "bfloat16" and flow not in ("tgv35", "cube17"):
        pytest.skip("one periodic and one walled grid in BF16")
    out = []
    for pairs in (True, False):
        for fold in ((True, False) if flow in ("cavity35", "cube17") else (True,)):
            d = FLOWS[flow]()
            c0 = [1.0, 0.05 if flow == "disc" else 0.0, 0.0] + ([0.0] if "z" in d["box"] else [])
            sim = Simulation(d, dtype=dtype, c0=c0, node_pairs=pairs)
            sim.fold_walls = fold
            for _ in range(9):
                sim.one_time_step()
            out.append(np.array([sim.F[k] for k in range(sim.scheme.nv)]))
            sim.free()
    assert np.all(np.isfinite(out[0]))
    for other in out[1:]:
        assert np.array_equal(out[0], other)
