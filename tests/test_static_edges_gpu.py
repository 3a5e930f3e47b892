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


@pytest.mark.parametrize("pad", ["zero", "beyond"])
def test_maps_padded_with_a_node_number(pkg, pad):
    """Rows that name a node but no element node are empty, whatever else the basket
    says of that node; before and after the rows that count."""
    torch = pytest.importorskip("torch")
    from tests.test_zz_no_alloc import StaticCase
    lib = pkg.native.load()
    case = StaticCase(pkg, torch, 9, 8, seed=3)
    rng = np.random.default_rng(5)
    ig, il = (case.t[k].cpu().numpy().reshape(12, -1) for k in ("ig", "il"))
    none = 0 if pad == "zero" else case.fen * 36 + 1
    more = 700
    big_g, big_l = np.zeros((12, ig.shape[1] + 2 * more), np.int32), np.zeros((12, il.shape[1] + 2 * more), np.int32)
    big_g[:, more:-more], big_l[:, more:-more] = ig, il
    empty = big_g == 0
    big_g[empty] = rng.integers(1, case.nnode + 1, empty.sum())
    big_l[empty] = none
    case.rows = big_g.shape[1]
    case.t["ig"], case.t["il"] = (torch.tensor(a, device="cuda:0") for a in (big_g, big_l))
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for k in range(3):
        U = rng.standard_normal(5 * case.nnode) * 1e-9
        t_U = torch.tensor(U, device="cuda:0")
        t_F = torch.full((5 * case.nnode,), np.nan, dtype=torch.float64, device="cuda:0")
        assert case.call(lib, t_U, t_F, stream) == pkg.native.SHM_OK
        torch.cuda.synchronize()
        case.check(t_F.cpu().numpy(), U, (pad, k))
    case.plan.close()
