"""(U, uold) of shm_get_state is the whole state of a resident plan: a run that is
read and set again in a new plan gives the bits of the run in one piece, as the
other paths do (test_flat_shell_gpu.py)."""
import numpy as np
import pytest

from tests.test_resident_gpu import config, plate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("kind", ["plate", "quads", "solid"])
def test_resume_is_bit_identical(pkg, kind, precision):
    run = config(pkg)
    make = pkg.Plan
    if kind == "solid":
        scs, run = pkg.workloads.solid_plate(nex=5, L=5 * 0.5 / 120, seed=3, radius=6e-3, nft=120)
        make = pkg.SolidPlan
    else:
        scs = [plate(pkg, 17, 13, 4)]
        if kind == "quads":
            from tests.test_mesher import jittered_quads
            q, pos = jittered_quads(nx=18, ny=14, Lx=17 * 6.25e-3, Ly=13 * 6.25e-3, amp=6e-4, seed=5, flip=(1,))
            nodes, coords, _ = pkg.mesher.quad2spectral(pkg.mesher.change_turn_quad(q, pos), pos, 5)
            scs[0].mesh = dict(nodes=nodes, coords=coords, structured=False)
    whole = make(scs, run, precision=precision)
    assert whole.info["launches_per_step"] == 0
    ref = whole.forward()[0]["displ"]
    state = whole.get_state()
    whole.close()
    assert np.abs(ref).max() > 0
    cut = [run.nn_first, run.nn_first + 1, 50, 51, run.nft - 3, run.nft + 1]
    U = Uo = None
    for a, b in zip(cut[:-1], cut[1:]):
        part = make(scs, run, precision=precision)
        part.set_signal()
        if U is not None:
            part.set_state(U, Uo, a)
            for got, want in zip(part.get_state(), (U, Uo)):
                np.testing.assert_array_equal(got, want)
        part.advance(b - a)
        U, Uo = part.get_state()
        displ = part.read_outputs()[0]["displ"]
        part.close()
        np.testing.assert_array_equal(displ[a - 1:b - 1], ref[a - 1:b - 1])
    np.testing.assert_array_equal(U, state[0])
    np.testing.assert_array_equal(Uo, state[1])
