"""Device memory that plans and grids hold between calls: bounded for the process,
not per object, given back with the object, and the same results whoever's
buffer was freed in between, also with several threads."""
import gc
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def plan_of(pkg, seed, nft):
    """A plate whose states of all steps take about 7 GB (FP32)."""
    scs, run = pkg.workloads.plate_force(nex=130, ney=130, L=130 * 6.25e-3, T=1e-4, nft=nft)
    scs[0].signal = np.random.default_rng(seed).standard_normal(nft)
    return pkg.Plan(scs, run, precision=32), [np.zeros((nft, len(scs[0].out_dof)))]


def test_adjoint_stores_are_bounded_together(pkg):
    torch = pytest.importorskip("torch")
    free = lambda: torch.cuda.mem_get_info()[0]
    gc.collect()
    nft = 820
    limit = torch.cuda.mem_get_info()[1] // 8
    plans = [plan_of(pkg, 0, nft)]
    states = plans[0][0].info["nnode"] * 5 * 4 * (nft - 1)
    assert 2 * states < limit
    plans += [plan_of(pkg, s, nft) for s in range(1, limit // states + 2)]
    for p, t in plans:   # allocates what every call needs
        p.set_adjoint_store(0)
        p.forward_backward(t)
        p.set_adjoint_store(None)
    base = free()
    first = [p.forward_backward(t) for p, t in plans]
    assert [p.stored_segments() for p, _ in plans] == [5] * len(plans)
    held = base - free()
    assert limit // 2 < held <= limit
    got = [None] * len(plans)

    def work(k):
        for _ in range(2):
            got[k] = plans[k][0].forward_backward(plans[k][1])

    th = [threading.Thread(target=work, args=(k,)) for k in range(len(plans))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for (ma, ga), (mb, gb) in zip(first, got):
        np.testing.assert_array_equal(ma, mb)
        np.testing.assert_array_equal(ga[0], gb[0])
    assert base - free() <= limit
    # a smaller allowance gives the larger store back
    p, t = plans[0]
    p.forward_backward(t)
    before = free()
    p.set_adjoint_store(states // 4)
    p.forward_backward(t)
    assert free() - before > states // 2
    for p, _ in plans:
        p.close()
    assert free() - base > -(64 << 20)


@pytest.mark.parametrize("precision", [64, 32])
def test_a_plan_without_memory_for_the_resident_arrays(pkg, precision):
    """Device memory for the element and node kernels but not for the resident
    kernel's arrays beside them: the plan steps on the former, as path 1."""
    torch = pytest.importorskip("torch")
    from tests.test_resident_gpu import config
    from tests.test_resident_routes_gpu import quads
    free = lambda: torch.cuda.mem_get_info()[0]
    sc, run = quads(pkg, 60, 60, 3), config(pkg, 20)
    run.frm_int, took, ref = 0, {}, None
    gc.collect()
    for path in (0, 1):   # (twice: what the first plan of a process allocates besides)
        for _ in range(2):
            before = free()
            plan = pkg.Plan([sc], run, precision=precision, path=path)
            took[path] = before - free()
            assert (plan.info["launches_per_step"] == 0) == (path == 0)
            ref = plan.forward()[0]["displ"]
            plan.close()
    assert took[0] - took[1] > 12 << 20
    torch.cuda.empty_cache()
    fill = torch.empty(free() - (took[0] + took[1]) // 2, dtype=torch.uint8, device="cuda:0")
    try:
        plan = pkg.Plan([sc], run, precision=precision)
        assert plan.info["launches_per_step"] == 2
        got = plan.forward()[0]["displ"]
        plan.close()
    finally:
        del fill
        torch.cuda.empty_cache()
    np.testing.assert_array_equal(got, ref)
