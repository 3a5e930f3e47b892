"""Image tiles at their edges: fewer points than elements (a tile is full at 32
elements), more than 256 points per element (several tiles on one element),
widths that leave a partial tile, one frame and more frames than runs, and
both data orders of the C ABI; against the tensor-product sum in numpy from
the grid's own (owner, ksi, eta).  FP64, 36 products of weights below about 10:
1e-12 of the largest value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nex,ney,nx,ny,nframes", [(9, 7, 3, 2, 1), (13, 11, 12, 10, 2), (2, 1, 45, 37, 3), (1, 1, 2, 300, 1),
                                                   (6, 5, 64, 31, 40)])
def test_tiles(pkg, nex, ney, nx, ny, nframes):
    mesh = pkg.mesh.structured_plate(nex * 0.01, ney * 0.012, nex, ney)
    nn = mesh["coords"].shape[0]
    frames = np.random.default_rng(nx).standard_normal((nframes, 5, nn))
    g = pkg.wavefield.Grid(mesh, nx, ny, "top")
    P = g.points()
    x, _ = pkg.mesh.gll_points(6)

    def weights(t):
        return np.stack([np.prod([(t - x[m]) / (x[i] - x[m]) for m in range(6) if m != i], axis=0) for i in range(6)], 1)

    wx, wy = weights(P["ksi"]), weights(P["eta"])
    nodes = mesh["nodes"][P["owner"]].reshape(-1, 6, 6) - 1
    h = 4e-3
    for motion in (3, 9):
        u, fx, v, fy, w = (frames[:, k] for k in range(5))
        val = w if motion == 3 else np.sqrt((u + h / 2 * fx) ** 2 + (v + h / 2 * fy) ** 2 + w ** 2)
        want = np.einsum("pj,pi,npji->np", wy, wx, val[:, nodes])
        img = g.interpolate(frames, [0, 1, 2, 3, 4], motion, h)
        assert img.shape == (nframes, ny, nx)
        err = np.abs(img - want.reshape(nframes, nx, ny).transpose(0, 2, 1)).max()
        assert err <= 1e-12 * np.abs(want).max()
    # the ABI's default order: point p = iy + ny*ix
    flat = np.zeros((nframes, nx * ny))
    lib, ptr = g.lib, pkg.native.ptr
    assert lib.shm_grid_image_order(g.handle, 0) == pkg.native.SHM_OK
    df = np.arange(5, dtype=np.int32)
    assert lib.shm_grid_interpolate(g.handle, ptr(frames), nframes, 5, ptr(df, pkg.native.I32P), 9, 0, h, ptr(flat),
                                    None) == pkg.native.SHM_OK
    assert np.array_equal(flat.reshape(nframes, nx, ny).transpose(0, 2, 1), img)
    g.close()
