"""The 3D solid's element and node kernels (plans too large for the chip, or of
elements that are no boxes) against the FP64 oracle.  Bounds as in test_solid_gpu.py:
FP64 1e-10 relative L2, FP32 1e-3."""
import numpy as np
import pytest

from oracle.oracle import OracleSolid
from tests.test_solid_gpu import rel

pytestmark = pytest.mark.gpu

TOL = {64: 1e-10, 32: 1e-3}


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("boxes", [True, False])
@pytest.mark.parametrize("nex", [1, 4, 5])
def test_element_and_node_kernels_match_oracle(pkg, nex, boxes, precision):
    """8, 128 and 200 elements (the FP32 kernel takes 12 to a CTA), the larger ones with
    a delamination; boxes, and in-plane jittered node columns."""
    L = 0.005 * nex
    scs, run = pkg.workloads.solid_plate(nex=nex, L=L, T=6e-6, f=800e3, n_out=4, radius=0.3 * L, delam=False)
    sc = scs[0]
    base = sc.mesh["base"]["coords"]
    if nex > 1:
        mid = nex * (nex // 2) + nex // 2 + 1
        sc.mesh = pkg.mesh.split_interface(sc.mesh, 3, [mid - 1, mid])
    run.nft = min(run.nft, 160)
    sc.signal = sc.signal[:run.nft]
    fen = sc.mesh["nodes"].shape[0]
    assert fen == 8 * nex * nex
    sc.elem_keep = np.linspace(0.6, 1.0, fen)
    if not boxes:  # every copy of a column moves alike
        coords = np.array(sc.mesh["coords"])
        key = np.round(coords[:, :2] / L, 9)
        rng = np.random.default_rng(9)
        columns = np.unique(np.round(base[:, :2] / L, 9), axis=0)
        jit = dict(zip(map(tuple, columns), rng.uniform(-0.04, 0.04, columns.shape) * (L / nex / 5)))
        coords[:, :2] += np.array([jit[tuple(k)] for k in key])
        sc.mesh = {**sc.mesh, "coords": coords}
    ref = OracleSolid(sc.mesh["nodes"], sc.mesh["coords"], sc.mat_table[:, :13], sc.mat_table[:, 13], sc.elem_mat,
                      sc.elem_keep).run(run.dt, run.nft, sc.signal, nn_first=run.nn_first, eta_xy=run.eta_xy,
                                        eta_z=run.eta_z, force_dof=sc.force_dof, force_val=sc.force_val,
                                        out_dof=sc.out_dof)
    assert np.abs(ref["displ"]).max() > 0 and np.abs(ref["U"]).max() > 0
    plan = pkg.SolidPlan([sc], run, precision=precision)
    plan.set_persistent(False)
    assert plan.info["launches_per_step"] == 2
    got = plan.forward()[0]["displ"]
    U, _ = plan.get_state()
    plan.close()
    assert rel(got, ref["displ"]) <= TOL[precision]
    assert rel(U, ref["U"]) <= TOL[precision]
