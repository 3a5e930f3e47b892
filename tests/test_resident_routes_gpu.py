"""Which plans of path 0 the resident kernel takes, and its rarer forms, against
the general kernels.  Bounds as in test_resident_gpu.py."""
import time

import numpy as np
import pytest

from tests.test_mesher import jittered_quads
from tests.test_resident_gpu import TOL, config, plate, rel

pytestmark = pytest.mark.gpu


def quads(pkg, nex, ney, seed):
    q, pos = jittered_quads(nx=nex + 1, ny=ney + 1, Lx=nex * 6.25e-3, Ly=ney * 6.25e-3, amp=6e-4, seed=seed, flip=(1,))
    nodes, coords, _ = pkg.mesher.quad2spectral(pkg.mesher.change_turn_quad(q, pos), pos, 5)
    sc = plate(pkg, nex, ney, seed)
    sc.mesh = dict(nodes=nodes, coords=coords, structured=False)
    return sc


@pytest.mark.parametrize("wrong", ["swapped", "doubled"])
def test_basket_maps_that_disagree_with_the_nodes(pkg, wrong):
    """Maps with the right number of entries per node, but the forces of two inner
    element nodes exchanged, or one copy of a shared node listed twice: the
    element + node kernels gather as the maps say, and so does path 0."""
    from oracle import ref_setup as R
    sc = quads(pkg, 9, 7, 11)
    nodes, nn = sc.mesh["nodes"], sc.mesh["coords"].shape[0]
    IG, IL = (np.array(a) for a in R.nodes_maps_fiborek(nodes.astype(np.int32), nn, 5, 1))
    count = np.bincount(nodes.ravel(), minlength=nn + 1)
    if wrong == "swapped":
        a, b = (np.argwhere(IG == g)[0] for g in np.nonzero(count == 1)[0][[3, 70]])
        IL[tuple(a)], IL[tuple(b)] = IL[tuple(b)], IL[tuple(a)]
    else:
        a, b = np.argwhere(IG == np.nonzero(count == 2)[0][5])
        IL[tuple(a)] = IL[tuple(b)]
    sc.mesh.update(I_G=IG.astype(np.int32), I_L=IL.astype(np.int32))
    run = config(pkg, 12)
    sc.signal = np.ones(12)
    got = []
    for path in (0, 1):
        plan = pkg.Plan([sc], run, precision=64, path=path)
        plan.forward()
        got.append(plan.get_state()[0])
        plan.close()
    assert np.abs(got[1]).max() > 0 and rel(*got) <= TOL[64]


def test_more_rows_per_task_than_the_plate_has(pkg):
    """Any number of rows is one task per strip, at the price of one: nothing is
    sized or counted by a number that the caller only meant as "all of them"."""
    sc, run = plate(pkg, 37, 9, 5, nft=30), config(pkg, 30)
    got, took = [], []
    for rows in (9, 9, 400_000_000):
        t = time.perf_counter()
        plan = pkg.Plan([sc], run, precision=32, path=2, rows_per_block=rows)
        took.append(time.perf_counter() - t)
        assert plan.info["rows_per_block"] == rows
        got.append(plan.forward()[0]["displ"])
        plan.close()
    np.testing.assert_array_equal(got[1], got[2])
    assert took[2] <= 0.5 + 5 * took[1]


@pytest.mark.parametrize("precision", [64, 32])
def test_a_named_split_is_what_the_plan_runs(pkg, precision):
    """path 0 with tile_elems or rows_per_block: that split of the structured
    kernel, as path 2; where there is none to split, path 0 as ever."""
    sc, run = plate(pkg, 37, 9, 5, nft=30), config(pkg, 30)
    for kw in (dict(tile_elems=16), dict(rows_per_block=3), dict(tile_elems=32, rows_per_block=5)):
        got = []
        for path in (0, 2):
            plan = pkg.Plan([sc], run, precision=precision, path=path, **kw)
            assert plan.info["path"] == 2 and plan.info["launches_per_step"] == 1
            got.append((plan.forward()[0]["displ"], plan.info["tile"], plan.info["rows_per_block"]))
            plan.close()
        np.testing.assert_array_equal(got[0][0], got[1][0])
        assert got[0][1:] == got[1][1:]
    plan = pkg.Plan([quads(pkg, 9, 7, 3)], run, precision=precision, tile_elems=16)
    assert plan.info["launches_per_step"] == 0
    plan.close()


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("n", [8, 9, 12])
def test_a_node_of_many_elements(pkg, n, precision):
    """n kites around one node that is forced and read: up to eight copies have their
    codes at the node, more stand in its list."""
    a = np.arange(n) * 2 * np.pi / n
    r = 6.25e-3
    ring, tips = (r * np.stack([np.cos(t), np.sin(t)], 1) for t in (a, a + np.pi / n))
    pos = np.zeros((1 + 2 * n, 3))
    pos[1:, :2] = np.concatenate([ring, 1.2 * tips])
    i = np.arange(n)
    q = np.stack([np.ones(n, int), 2 + i, 2 + n + i, 2 + (i + 1) % n], 1).astype(np.int32)
    nodes, coords, _ = pkg.mesher.quad2spectral(pkg.mesher.change_turn_quad(q, pos), pos, 5)
    centre = int(np.argmin(np.hypot(*coords[:, :2].T))) + 1
    assert (nodes == centre).sum() == n
    sc = plate(pkg, n, 1, 6)
    sc.mesh = dict(nodes=nodes, coords=coords, structured=False)
    sc.force_dof = np.array([5 * centre, 5 * centre - 4, 5 * int(nodes[3, 8])])
    sc.out_dof = np.array([5 * centre, 5 * centre - 3, 5 * int(nodes[1, 20])])
    run = config(pkg)
    run.dt = 1e-8
    got = {}
    for path, prec in ((0, precision), (1, 64)):
        plan = pkg.Plan([sc], run, precision=prec, path=path)
        assert (plan.info["launches_per_step"] == 0) == (path == 0)
        got[path] = plan.forward()[0]["displ"], plan.get_state()[0]
        plan.close()
    for x, y in zip(got[0], got[1]):
        assert np.isfinite(y).all() and np.abs(y).max() > 0 and rel(x, y) <= TOL[precision]


@pytest.mark.parametrize("precision", [64, 32])
def test_plan_facts_name_the_kernel(pkg, precision):
    """A plan on the resident kernel has no split of the structured one and is not
    persistent; one that left it has and is what it was set to."""
    sc, run = plate(pkg, 37, 9, 5, nft=60), config(pkg, 60)
    plan = pkg.Plan([sc], run, precision=precision)
    facts = lambda: tuple(plan.info[k] for k in ("resident", "persistent", "launches_per_step"))
    assert facts() == (True, False, 0) and plan.info["tile"] == plan.info["rows_per_block"] == 0
    best = plan.autotune(10)
    assert (best["tile"], best["rows_per_block"]) == (plan.info["tile"], plan.info["rows_per_block"]) or plan.info["path"] == 1
    assert best["persistent"] == plan.info["persistent"]
    assert plan.info["resident"] == (best["rows_per_block"] == 0)
    again = pkg.Plan([sc], run, precision=precision, tile_elems=best["tile"], rows_per_block=best["rows_per_block"])
    if plan.info["resident"]:  # the reported choice, named to a new plan
        assert again.info["resident"]
    again.close()
    plan.set_persistent(False)
    if plan.info["path"] == 2:
        assert facts() == (False, False, 1) and plan.info["tile"] in (16, 32) and plan.info["rows_per_block"] > 0
        if precision == 32:
            plan.set_persistent(True)
            assert facts() == (False, True, 0) and plan.info["tile"] in (16, 32)
    plan.close()
    plan = pkg.Plan([quads(pkg, 9, 7, 3)], run, precision=precision)
    assert facts() == (True, False, 0)
    plan.set_persistent(False)
    assert facts() == (False, False, 2)
    plan.close()
