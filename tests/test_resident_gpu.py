"""Resident stepping (plans of path 0 whose elements fit on the chip) against
the general element + node kernels, which the other tests pin to the oracle.

Bounds as in test_flat_shell_gpu.py: FP64 1e-10 relative L2 (summation order,
and the derivative blocks of even and odd values in place of the 6x6 matrix:
a few hundred roundings of 1e-16 per step over at most 250 steps), FP32 1e-3
against the FP64 general kernels."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {64: 1e-10, 32: 1e-3}


def rel(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / max(np.linalg.norm(b), 1e-300)


def plate(pkg, nex, ney, seed, nft=160, edge=6.25e-3):
    """Damaged plate of two laminates (one unsymmetric) with a force, outputs, two sensors and frames."""
    from tests.test_oracle_physics import _materials
    rng = np.random.default_rng(seed)
    mesh = pkg.mesh.structured_plate(nex * edge, ney * edge * 1.1, nex, ney)
    fen = nex * ney
    nodes = rng.integers(1, mesh["coords"].shape[0] + 1, 6)
    _, st = pkg.hanning_signal(4e-8, nft, 1e5, 5e5)
    sc = pkg.Scenario(mesh=mesh, mat_table=np.stack([pkg.materials.table_row(l) for l in _materials(pkg)]),
                      elem_mat=rng.integers(0, 2, fen).astype(np.int32), elem_keep=rng.uniform(0.2, 1.0, fen),
                      force_dof=np.array([5 * nodes[0], 5 * nodes[0] - 4, 5 * nodes[1] - 3]), force_val=np.array([1.0, -0.5, 1e-3]),
                      out_dof=np.concatenate([5 * nodes, 5 * nodes[:2] - 2, 5 * nodes[:1]]), signal=st)
    sc.sensors = [np.array([0], np.int32), np.arange(max(1, fen // 2), fen, dtype=np.int32)][:1 + (fen > 1)]
    sc.pzt = dict(pzt_thickness=0.2e-3, g33=1.5e-8, e31=-5.4, e32=-3.4)
    return sc


def config(pkg, nft=160):
    return pkg.RunConfig(dt=4e-8, nft=nft, nn_first=2, eta_xy=4e2, eta_z=4e3, h=3.9e-3, frm_int=45, frame_dof=0, frame_kind=0)


def solve(pkg, scs, run, precision, path, pieces=None):
    plan = pkg.Plan(scs, run, precision=precision, path=path)
    assert (plan.info["launches_per_step"] == 0) == (path == 0)
    if pieces is None:
        res = plan.forward(want_frames=True)
    else:
        plan.set_signal()
        left = run.nft - run.nn_first + 1
        for n in pieces:
            plan.advance(min(n, left))
            left -= min(n, left)
        plan.advance(left)
        res = plan.read_outputs(want_frames=True)
    state = plan.get_state()
    plan.close()
    return res, state


def compare(pkg, scs, run, precision):
    got, state = solve(pkg, scs, run, precision, 0)
    ref, rstate = solve(pkg, scs, run, 64, 1)
    for a, b in zip(got, ref):
        assert np.abs(b["displ"]).max() > 0
        for key in ("displ", "voltage", "frames"):
            if key in b and np.size(b[key]):
                assert rel(a[key], b[key]) <= TOL[precision], key
    for a, b in zip(state, rstate):
        assert rel(a, b) <= TOL[precision]


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("nex,ney", [(1, 1), (1, 7), (5, 2), (19, 8), (39, 31), (61, 57)])
def test_rectangles_match_general_kernels(pkg, nex, ney, precision):
    """One element (no neighbour), strips, counts around the passes and the SM count."""
    compare(pkg, [plate(pkg, nex, ney, 7)], config(pkg), precision)


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("nex,ney", [(2, 2), (9, 8), (41, 29)])
def test_quads_match_general_kernels(pkg, nex, ney, precision):
    """Distorted elements (direct form) in the mesher's numbering."""
    from tests.test_mesher import jittered_quads
    q, pos = jittered_quads(nx=nex + 1, ny=ney + 1, Lx=nex * 6.25e-3, Ly=ney * 6.25e-3, amp=6e-4, seed=5, flip=(1,))
    nodes, coords, _ = pkg.mesher.quad2spectral(pkg.mesher.change_turn_quad(q, pos), pos, 5)
    sc = plate(pkg, nex, ney, 9)
    sc.mesh = dict(nodes=nodes, coords=coords, structured=False)
    compare(pkg, [sc], config(pkg), precision)


@pytest.mark.parametrize("precision", [64, 32])
def test_batch_delamination_and_pressure(pkg, precision):
    compare(pkg, [plate(pkg, 7, 5, 1), plate(pkg, 12, 9, 2, edge=5e-3), plate(pkg, 3, 4, 3)], config(pkg), precision)
    scs, run = pkg.workloads.plate_delamination(nex=14, ney=11, L=0.2, zone=(0.1, 0.1, 0.04, 0.03, 0.4), nft=200, radius=0.02)
    run.frm_int = 60
    compare(pkg, scs, run, precision)
    scs, run = pkg.workloads.plate_pressure(nft=250)
    run.frm_int = 60
    compare(pkg, scs, run, precision)


@pytest.mark.parametrize("precision", [64, 32])
def test_pieces_and_threads_give_the_same_bits(pkg, precision):
    """One advance, uneven pieces, and two plans stepping at the same time
    from two threads."""
    scs = [[plate(pkg, 23, 17, 4)], [plate(pkg, 31, 30, 6)]]
    run = config(pkg)
    whole = [solve(pkg, s, run, precision, 0) for s in scs]
    parts = [solve(pkg, s, run, precision, 0, pieces=(1, 2, 57, 33)) for s in scs]
    both = [None, None]

    def work(k):
        for _ in range(3):
            both[k] = solve(pkg, scs[k], run, precision, 0)

    th = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for k in range(2):
        for other in (parts[k], both[k]):
            for key in ("displ", "voltage", "frames"):
                np.testing.assert_array_equal(whole[k][0][0][key], other[0][0][key])
            np.testing.assert_array_equal(whole[k][1][0], other[1][0])
            np.testing.assert_array_equal(whole[k][1][1], other[1][1])


def test_elements_that_do_not_fit_keep_the_structured_kernel(pkg):
    """The same bits as the kernel named by path 2 (in FP32 path 0 may advance
    in one persistent launch of it)."""
    sc = plate(pkg, 130, 120, 8, nft=20)
    for precision in (64, 32):
        got = []
        for path in (0, 2):
            plan = pkg.Plan([sc], config(pkg, 20), precision=precision, path=path)
            assert plan.info["path"] == 2
            got.append((plan.forward()[0]["displ"], plan.get_state()[0]))
            plan.close()
        for a, b in zip(*got):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("per_sm", [66, 74])
def test_fullest_meshes(pkg, per_sm):
    """FP32 quads with as many elements per SM as two CTAs and as one CTA of short
    passes hold (152 SMs)."""
    from tests.test_mesher import jittered_quads
    q, pos = jittered_quads(nx=153, ny=per_sm + 1, Lx=0.95, Ly=per_sm * 6.25e-3, amp=6e-4, seed=6, flip=(1,))
    nodes, coords, _ = pkg.mesher.quad2spectral(pkg.mesher.change_turn_quad(q, pos), pos, 5)
    sc = plate(pkg, 152, per_sm, 9)
    sc.mesh = dict(nodes=nodes, coords=coords, structured=False)
    compare(pkg, [sc], config(pkg), 32)


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("kind,nex,ney", [("plate", 1, 1), ("plate", 8, 5), ("plate", 37, 21), ("batch", 6, 4), ("quads", 9, 8),
                                          ("quads", 33, 27)])
def test_adjoint_matches_general_kernels(pkg, kind, nex, ney, precision):
    """Misfit and gradient against the per-step kernels, an undamaged, a damaged
    and a fully lost element among them; the same bits however many segments are
    stored, a last segment of one step among the intervals."""
    from tests.test_mesher import jittered_quads
    scs = [plate(pkg, nex, ney, 21)] + ([plate(pkg, ney, nex, 22)] if kind == "batch" else [])
    if kind == "quads":
        q, pos = jittered_quads(nx=nex + 1, ny=ney + 1, Lx=nex * 6.25e-3, Ly=ney * 6.25e-3, amp=6e-4, seed=7, flip=(1,))
        nodes, coords, _ = pkg.mesher.quad2spectral(pkg.mesher.change_turn_quad(q, pos), pos, 5)
        scs[0].mesh = dict(nodes=nodes, coords=coords, structured=False)
    run = config(pkg)
    rng = np.random.default_rng(23)
    for sc in scs:
        sc.elem_keep[0] = 1.0
        if nex * ney > 1:
            sc.elem_keep[nex // 2] = 0.0
    ref = pkg.Plan(scs, run, precision=64, path=1)
    peak = [np.abs(r["displ"]).max(axis=0) for r in ref.forward()]
    targets = [rng.normal(size=(run.nft, len(sc.out_dof))) * m for sc, m in zip(scs, peak)]
    mis, grad = ref.forward_backward(targets, ckpt_every=40)
    ref.close()
    plan = pkg.Plan(scs, run, precision=precision, path=0)
    assert plan.info["launches_per_step"] == 0
    got = []
    for k, part in ((40, 0), (40, 2), (40, None), (run.nft, None), (79, 0)):
        plan.set_adjoint_store(None if part is None else part * k * plan.info["nnode"] * 5 * precision // 8)
        got.append(plan.forward_backward(targets, ckpt_every=k))
    plan.close()
    assert (run.nft - run.nn_first + 1) % 79 == 1
    for m, g in got:
        for a, b in zip(m, got[0][0]):
            assert a == b
        for a, b in zip(g, got[0][1]):
            np.testing.assert_array_equal(a, b)
    for a, b in zip(got[0][0], mis):
        assert abs(a - b) <= TOL[precision] * b
    for a, b in zip(got[0][1], grad):
        assert np.abs(b).max() > 0 and rel(a, b) <= TOL[precision]


@pytest.mark.parametrize("kind", ["solid", "plate"])
def test_fp32_is_no_further_from_64_bits_than_per_step_kernels(pkg, kind):
    """A wave that has only just reached the outputs, its source on an element
    corner: the displacements there are orders below the source's, and rounding
    that an element spreads from one corner to the others shows.  Half as much
    again is allowed for the chance in single roundings."""
    if kind == "solid":
        scs, run = pkg.workloads.solid_plate(nex=12, L=0.05, seed=3, radius=5e-3, nft=80)
        make = pkg.SolidPlan
        scs[0].signal = pkg.hanning_signal(run.dt, run.nft, 2e4, 1e5, 0.0)[1]
    else:
        scs, run = pkg.workloads.plate_force(nex=24, ney=24, L=0.24, T=1e-4, f=100e3, n_out=8, radius=0.03)
        make = pkg.Plan
        run.nft = 80
        scs[0].signal = scs[0].signal[:80]
    out = {}
    for name, precision, resident in (("exact", 64, False), ("resident", 32, True), ("steps", 32, False)):
        plan = make(scs, run, precision=precision)
        if not resident:
            plan.set_persistent(False)
        assert (plan.info["launches_per_step"] == 0) == resident
        out[name] = plan.forward()[0]["displ"]
        plan.close()
    assert rel(out["resident"], out["exact"]) <= 1.5 * rel(out["steps"], out["exact"])


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("nex", [1, 5, 9])
def test_solid_boxes_match_per_step_kernels(pkg, nex, precision):
    """3D solid laminates: one column of elements (no neighbour in plane), a
    few, and more than one pass per CTA; delaminated interface, frames, damage,
    several forces, against the same plan stepped by the element and node kernels."""
    rng = np.random.default_rng(nex)
    scs, run = pkg.workloads.solid_plate(nex=nex, L=nex * 0.5 / 120, seed=3, radius=0.4 * nex * 0.5 / 120, nft=120)
    sc = scs[0]
    nn = sc.mesh["coords"].shape[0]
    sc.elem_keep = rng.uniform(0.3, 1.0, sc.mesh["nodes"].shape[0])
    sc.force_dof = np.concatenate([sc.force_dof, rng.integers(1, 3 * nn + 1, 3)]).astype(np.int32)
    sc.force_val = np.array([1.0, 0.5, -2.0, 0.3])
    sc.out_dof = rng.integers(1, 3 * nn + 1, 40).astype(np.int32)
    run.frm_int, run.frame_dof, run.frame_kind = 30, 0, 3
    got = []
    for on in (True, False):
        plan = pkg.SolidPlan(scs, run, precision=precision if on else 64)
        assert plan.info["launches_per_step"] == 0
        if not on:
            plan.set_persistent(False)
            assert plan.info["launches_per_step"] == 2
        res = plan.forward(want_frames=True)[0]
        got.append((res["displ"], res["frames"][:, 3:6], res["frames"][:, 6:], *plan.get_state()))
        if on:
            plan.reset()
            plan.set_signal()
            for n in (1, 50, 2, run.nft - run.nn_first + 1 - 53):
                plan.advance(n)
            again = plan.read_outputs(want_frames=True)[0]
            np.testing.assert_array_equal(again["displ"], res["displ"])
            np.testing.assert_array_equal(again["frames"], res["frames"])
        plan.close()
    for a, b in zip(*got):
        assert np.abs(b).max() > 0 and rel(a, b) <= TOL[precision]
