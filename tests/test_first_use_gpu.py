"""Buffers that a call allocates on its first use are cleared before the call's own
work reaches them: the first frames, gradient and stepping of a new plan are those of
every later call."""
import numpy as np
import pytest

from tests.test_resident_gpu import config, plate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32])
def test_first_calls_of_new_plans(pkg, precision):
    sc, run = plate(pkg, 24, 21, 4), config(pkg)
    run.frm_int = 2   # 80 frames, 5 fields: 50 MB
    want = None
    for k in range(6):
        plan = pkg.Plan([sc], run, precision=precision, path=(0, 1, 2)[k % 3])
        res = plan.forward(want_frames=True)[0]
        target = [0.5 * res["displ"]]
        mis, grad = plan.forward_backward(target, ckpt_every=40)
        again = plan.forward(want_frames=True)[0]
        np.testing.assert_array_equal(res["frames"], again["frames"])
        assert np.abs(res["frames"][-1]).max() > 0
        mis2, grad2 = plan.forward_backward(target, ckpt_every=40)
        np.testing.assert_array_equal(mis, mis2)
        np.testing.assert_allclose(grad2[0], grad[0], rtol=1e-9, atol=1e-12 * np.abs(grad[0]).max())
        plan.close()
        if k % 3 == 0:
            if want is not None:
                np.testing.assert_array_equal(res["frames"], want)
            want = res["frames"]


def test_state_set_and_stepped_at_once(pkg):
    """The copies of shm_set_state are complete when shm_advance starts on another stream."""
    import torch
    sc, run = plate(pkg, 40, 33, 4), config(pkg)
    plan = pkg.Plan([sc], run, precision=32, path=1)
    plan.set_signal()
    plan.advance(60)
    U, Uo = plan.get_state()
    plan.advance(1)
    want = plan.get_state()[0]
    stream = torch.cuda.Stream()
    for _ in range(20):
        plan.set_state(np.zeros_like(U), np.zeros_like(U), run.nn_first + 60)
        plan.set_state(U, Uo, run.nn_first + 60)
        assert plan.lib.shm_advance(plan.handle, 1, stream.cuda_stream) == pkg.native.SHM_OK
        np.testing.assert_array_equal(plan.get_state()[0], want)
    plan.close()
