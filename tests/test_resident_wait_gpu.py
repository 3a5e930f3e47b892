"""The resident kernel's bounded wait: one that runs out is an error that the host
reads, and the plan steps on after it."""
import numpy as np
import pytest

from tests.test_resident_gpu import config, plate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
def test_a_wait_that_runs_out_is_reported(pkg, precision):
    """One poll allowed: of hundreds of CTAs some wait for longer, in the forward kernel,
    in shm_advance and in the gradient; with the default limit again, the same bits."""
    sc, run = plate(pkg, 20, 17, 4), config(pkg)
    plan = pkg.Plan([sc], run, precision=precision)
    assert plan.info["launches_per_step"] == 0
    ref = plan.forward(want_frames=True)[0]
    target = [0.5 * ref["displ"]]
    mis, grad = plan.forward_backward(target, ckpt_every=30)

    def gives_up(call):
        with pytest.raises(pkg.native.ShmError) as ei:
            call()
        assert ei.value.status == pkg.native.SHM_ERR_TIMEOUT and "resident exchange" in str(ei.value)

    plan.set_exchange_limit(0)
    gives_up(plan.forward)
    plan.reset()
    plan.set_signal()
    gives_up(lambda: plan.advance(5))
    gives_up(lambda: plan.forward_backward(target, ckpt_every=30))
    plan.set_exchange_limit()
    assert plan.info["launches_per_step"] == 0
    again = plan.forward(want_frames=True)[0]
    for key in ("displ", "voltage", "frames"):
        np.testing.assert_array_equal(again[key], ref[key])
    mis2, grad2 = plan.forward_backward(target, ckpt_every=30)
    plan.close()
    np.testing.assert_array_equal(mis2, mis)
    np.testing.assert_array_equal(grad2[0], grad[0])


def test_a_plan_without_neighbours_never_waits(pkg):
    """One element: no records, so the limit changes nothing."""
    sc, run = plate(pkg, 1, 1, 4), config(pkg)
    plan = pkg.Plan([sc], run)
    ref = plan.forward()[0]["displ"]
    plan.set_exchange_limit(0)
    got = plan.forward()[0]["displ"]
    plan.close()
    np.testing.assert_array_equal(got, ref)
