"""Boundary links by tiles (boundary.tile_links) against the batched launch.

A NumPy restatement of the multi-step launch -- regions in the plain and the
swapped layout, links by their element offsets, poisoned with NaN wherever a
region holds no value -- must give, after several steps, what the batched
boundary launch and the pull give one step at a time on the whole grid.  The
collision is an arbitrary linear mixing of a node's populations: only the
movement of values is checked, and it must be exact.
"""
import types

import numpy as np
import pytest

from pylbm_gb300 import workloads as W
from pylbm_gb300.boundary import Boundary, batch_entries, observed_ghost_copies, tile_links
from pylbm_gb300.codegen import opposite_populations
from pylbm_gb300.domain import Domain
from pylbm_gb300.scheme import Scheme

FLOWS = {
    "disc": lambda: W.cylinder(nx=67, ny=37, radius=5, center=(20, 19), re=31.25),
    "karman": lambda: W.karman(dx=1.0 / 32),
    "cavity": lambda: W.cavity(n=29),
}


def _value(kind, g0, g1, rhs, dist):
    if kind.startswith("bouzidi"):
        return (1.0 - dist) * g1 + (-dist * g0 if "anti" in kind else dist * g0) + rhs
    return (-g0 if kind == "anti_bounce_back" else g0) + rhs


def _setup(flow):
    dico = FLOWS[flow]()
    scheme = Scheme(dico)
    dom = Domain(dico, scheme.stencil)
    bc = Boundary(dom, dico)
    for m in bc.methods:
        m.set_iload()
        m.fix_iload()
    vel = np.asarray(scheme.stencil.get_all_velocities())
    ghost = observed_ghost_copies(dom.shape_in, dom.halo, vel, bc.methods)
    ghost = ghost if ghost is not None and len(ghost[0]) else None
    ext = [scheme.nv] + [n + 2 * int(h) for n, h in zip(dom.shape_in, dom.halo)]
    entries, joined = batch_entries(bc.methods, ext, ghost)
    assert ghost is None or joined
    rng = np.random.default_rng(7)
    for e in entries:
        e["rhs"] = rng.integers(-8, 8, len(e["istore"])).astype(np.float32)
        e["dist"] = rng.choice([0.25, 0.5, 1.0], len(e["istore"])).astype(np.float32)
    wrap = [int(dom.box_label[2 * d]) == -1 for d in range(2)]
    return dom, vel, entries, ghost, wrap, rng


def _collide(g, mix):
    return np.tensordot(mix, g, axes=1)


def _whole_grid(f, steps, dom, vel, entries, ghost, mix):
    n = dom.shape_in
    for _ in range(steps):
        new = f.copy()
        if ghost is not None:
            new[tuple(ghost[0].T)] = f[tuple(ghost[1].T)]
        for e in entries:
            load = [f[tuple(np.asarray(il).T)] for il in e["iload"]]
            new[tuple(np.asarray(e["istore"]).T)] = _value(e["kind"], load[0], load[-1], e["rhs"], e["dist"])
        pulled = np.array([new[k, 1 - v[0]:1 - v[0] + n[0], 1 - v[1]:1 - v[1] + n[1]] for k, v in enumerate(vel)])
        f = new
        f[:, 1:-1, 1:-1] = _collide(pulled, mix)
    return f[:, 1:-1, 1:-1]


def _tiles(f, steps, dom, vel, entries, ghost, wrap, plan, mix):
    n, q = dom.shape_in, len(vel)
    opp = opposite_populations(vel)
    lists = tile_links(entries, ghost, n, dom.halo, wrap, vel, opp, plan)
    assert lists is not None
    first, links = lists
    m, out = plan.margin, plan.out
    rows, cols = out[0] + 2 * m, out[1] + 2 * m
    kind_of = {0: "bounce_back", 1: "anti_bounce_back", 2: "bouzidi_bounce_back", 3: "bouzidi_anti_bounce_back"}
    result = np.full((q,) + tuple(n), np.nan)
    for t in range(plan.tiles[0] * plan.tiles[1]):
        o0 = t // plan.tiles[1] * out[0] - m
        o1 = t % plan.tiles[1] * out[1] - m
        sm = np.full(q * plan.plane, np.nan)
        where = lambda k, r, c: k * plan.plane + (r + 1) * plan.pitch + c + 1  # noqa: E731
        grid = {}
        for r in range(rows):
            for c in range(cols):
                g = [o0 + r, o1 + c]
                g = [x % s if w else x for x, s, w in zip(g, n, wrap)]
                if all(0 <= x < s for x, s in zip(g, n)):
                    grid[r, c] = g
                    for k in range(q):
                        sm[where(k, r, c)] = f[k, g[0] + 1, g[1] + 1]
        mine = links[first[t]:first[t + 1]]
        for s in range(1, steps + 1):
            swapped = (s + 1) % 2
            new = {}
            for rec in mine:
                value = _value(kind_of[int(rec["flags"])], sm[rec["load0"][swapped]],
                               sm[rec["load1"][swapped]] if rec["flags"] & 2 else 0.0, rec["rhs"], rec["dist"])
                new[int(rec["store"][swapped])] = value
            assert len(new) == len(mine)
            for at, value in new.items():
                sm[at] = value
            nodes = [(r, c) for r, c in grid if s <= r < rows - s and s <= c < cols - s]
            slots = {(r, c): [where(opp[k], r, c) if swapped else where(k, r - v[0], c - v[1])
                              for k, v in enumerate(vel)] for r, c in nodes}
            old = sm.copy()
            for r, c in nodes:
                g = _collide(old[slots[r, c]], mix)
                for k, v in enumerate(vel):
                    sm[where(k, r, c) if swapped else where(opp[k], r + v[0], c + v[1])] = g[k]
                    if s == steps and 0 <= r - m < out[0] and 0 <= c - m < out[1]:
                        i, j = o0 + r, o1 + c
                        if i < n[0] and j < n[1]:
                            result[k, i, j] = g[k]
    return result


@pytest.mark.parametrize("region, margin, steps", [((16, 32), 3, 3), ((16, 32), 3, 2), ((20, 24), 5, 4)])
@pytest.mark.parametrize("flow", ["disc", "karman", "cavity"])
def test_tiles_equal_the_batched_launch(flow, region, margin, steps):
    dom, vel, entries, ghost, wrap, rng = _setup(flow)
    n = dom.shape_in
    plan = types.SimpleNamespace(margin=margin, pitch=region[1] + 2, plane=(region[0] + 2) * (region[1] + 2))
    room = [s - 2 * margin for s in region]
    plan.tiles = [-(-n[d] // room[d]) for d in range(2)]
    plan.out = [-(-n[d] // plan.tiles[d]) for d in range(2)]
    f = rng.integers(-64, 64, (9, n[0] + 2, n[1] + 2)).astype(float)
    mix = rng.integers(-2, 3, (9, 9)).astype(float)
    ref = _whole_grid(f.copy(), steps, dom, vel, entries, ghost, mix)
    got = _tiles(f, steps, dom, vel, entries, ghost, wrap, plan, mix)
    assert np.array_equal(got, ref)


def test_links_that_do_not_fit_are_refused():
    dom, vel, entries, ghost, wrap, _ = _setup("disc")
    plan = types.SimpleNamespace(margin=2, pitch=34, plane=18 * 34, tiles=[6, 2], out=[12, 28])
    args = (dom.shape_in, dom.halo, wrap, vel, opposite_populations(vel), plan)
    assert tile_links(entries, ghost, *args) is not None
    # a ghost copy that is not the periodic image of its source
    moved = np.array(ghost[1])
    moved[0, 1] += 1
    assert tile_links(entries, (ghost[0], moved), *args) is None
    # a load that lies far from the node it feeds
    far = [dict(e) for e in entries]
    far[0]["iload"] = [np.array(il) for il in far[0]["iload"]]
    far[0]["iload"][0][:, 1] = (far[0]["iload"][0][:, 1] + 10) % dom.shape_in[0] + 1
    assert tile_links(far, ghost, *args) is None
    # periodic copies on an axis that the tiles do not wrap
    assert tile_links(entries, ghost, dom.shape_in, dom.halo, [False, False], vel, opposite_populations(vel), plan) is None


def test_opposite_populations():
    vel = np.array([[0, 0], [1, 0], [-1, 0], [1, 0], [-1, 0]])
    assert opposite_populations(vel) == [0, 2, 1, 4, 3]
    assert opposite_populations(np.array([[0, 0], [1, 0]])) is None
