"""shm_stiffness_static at the edges of its launch: one element, counts around
the elements per CTA (1..7 by element count) and the SM count, other meshes
through the same arrays in between, nodes that no element uses, and the longer
path for nodes beyond the slot array; against the plan's operator.  FP64 bound
as in test_zz_no_alloc.py (1e-11: summation order)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nex,ney,spare", [(1, 1, 0), (19, 8, 0), (17, 9, 5), (61, 15, 0), (64, 64, 0), (2, 3, 0),
                                           (3, 2, 150000)])
def test_static_force_of_any_size(pkg, nex, ney, spare):
    torch = pytest.importorskip("torch")
    from tests.test_zz_no_alloc import StaticCase
    lib = pkg.native.load()
    case = StaticCase(pkg, torch, nex, ney, seed=nex)
    n0, n1 = case.nnode, case.nnode + spare
    rng = np.random.default_rng(nex)
    U = np.zeros(5 * n1)
    U[:5 * n0] = rng.standard_normal(5 * n0) * 1e-9
    co = torch.zeros(3, n1, dtype=torch.float64, device="cuda:0")
    co[:, :n0] = case.t["coords"]
    case.t["coords"], case.nnode = co, n1
    t_U = torch.tensor(U, device="cuda:0")
    t_F = torch.full((5 * n1,), np.nan, dtype=torch.float64, device="cuda:0")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert case.call(lib, t_U, t_F, stream) == pkg.native.SHM_OK
    torch.cuda.synchronize()
    F = t_F.cpu().numpy()
    assert np.array_equal(F[5 * n0:], np.zeros(5 * spare))
    case.check(F[:5 * n0], U[:5 * n0], (nex, ney))
    case.plan.close()
