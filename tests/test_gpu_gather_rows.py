"""The gather from the stored H (rows of two samples) at the sizes where it can go wrong.

Every coil width (1 to 8, two passes, odd counts beyond a pass), grids smaller
than a padded tile, tiles that wrap around the grid edge, tiles with one sample
and tiles with more rows than a record, 2-D.  Compared with the FP64 oracle and
with the same plan evaluating the weights: the taps and their FP32 weights are
the same, so the results differ by the order of about 113 additions, below
1e-6 of the result's norm.
"""
import numpy as np
import pytest

from oracle.nufft_ref import NufftRef

pytestmark = pytest.mark.gpu


def _case(N, om, nc, opts, seed=5):
    import torch

    from nufft_3d_gb300 import nufft_3d
    rng = np.random.default_rng(seed)
    on = nufft_3d(om, N, density_iters=0, tap_table=1, spread_table=0, **opts)
    off = nufft_3d(om, N, density_iters=0, tap_table=0, **opts)
    assert on.tap_table_bytes > 0 and off.tap_table_bytes == 0
    ref = NufftRef(om, N, density_iters=0, **opts)
    n = tuple(int(v) for v in on.N)
    x = rng.standard_normal(n + (nc,)) + 1j * rng.standard_normal(n + (nc,))
    xt = torch.from_numpy(np.ascontiguousarray(x.transpose(3, 2, 1, 0)).astype(np.complex64)).cuda()
    a, b = on.fNUFT(xt).cpu().numpy().T, off.fNUFT(xt).cpu().numpy().T
    for _ in range(3):  # the sums have a fixed order: a race would show as a difference
        assert np.array_equal(on.fNUFT(xt).cpu().numpy().T, a)
    r = ref.fNUFT(x)
    for c in range(nc):  # per coil: a coil that is missed or swapped does not hide in the norm of all
        nrm = np.linalg.norm(r[:, c])
        assert np.linalg.norm(a[:, c] - r[:, c]) < 1e-5 * nrm
        assert np.linalg.norm(a[:, c] - b[:, c]) < 1e-6 * nrm
    w = torch.from_numpy(rng.random(on.M).astype(np.float32)).cuda()  # the weighted form (normal operator)
    ya, yb = on.iprojection(xt, 0.1, w), off.iprojection(xt, 0.1, w)
    # (both spread by the fixed-point kernel: about 22 bits per product)
    assert float((ya - yb).abs().norm() / yb.abs().norm()) < 5e-6


@pytest.mark.parametrize("nc", [1, 2, 3, 4, 5, 6, 7, 9, 11, 12, 16])
def test_coil_widths(nc):
    rng = np.random.default_rng(nc)
    om = rng.uniform(-9, 8, (3, 3001))
    _case(18, om, nc, dict(J=6, u=2))


@pytest.mark.parametrize("N,opts", [
    (4, dict(J=6, u=2)),                       # grid 8: the padded tile (14) is wider than the grid
    ((6, 20, 10), dict(J=5, u=1.5, radial=0)),  # ... on one axis; K not a multiple of the tile
    (14, dict(J=2, u=2)),
    ((16, 12, 22), dict(J=4, u=2)),
    ((36, 20, 1), dict(J=6, u=2)),
    ((64, 48, 1), dict(J=4, u=2, radial=0)),
])
@pytest.mark.parametrize("nc", [1, 3, 8])
def test_grids(N, opts, nc):
    rng = np.random.default_rng(7)
    n = np.resize(np.asarray(N), 3)
    om = np.stack([rng.uniform(-v / 2, v / 2 - 1, 2500) if v > 1 else np.zeros(2500) for v in n])
    _case(N, om, nc, opts)


@pytest.mark.parametrize("counts", [(1,), (2,), (3,), (127,), (128,), (129, 1, 515), (4000, 3)])
@pytest.mark.parametrize("nc", [1, 8])
def test_samples_of_a_slab(counts, nc):
    """Clusters of the given numbers of samples inside one slab each (a record holds 128), the last at the grid edge."""
    rng = np.random.default_rng(3)
    pts = []
    for i, c in enumerate(counts):
        centre = np.array([3.0 - 5 * i, -2.0, 1.0]) if i + 1 < len(counts) or len(counts) == 1 else np.array([7.2, 7.5, -7.7])
        pts.append(centre[:, None] + rng.uniform(-0.2, 0.2, (3, c)))
    _case(16, np.concatenate(pts, axis=1), nc, dict(J=6, u=2))


@pytest.mark.parametrize("nc", [1, 2, 3, 4, 5, 6, 7, 8])
def test_one_producer(nc):
    """A grid of 40 x 40 tiles a plane, nine tenths of them inside: bulk copies by a single warp at every width."""
    rng = np.random.default_rng(nc)
    om = np.stack([rng.uniform(-n / 2, n / 2 - 1, 20000) for n in (160, 160, 6)])
    _case((160, 160, 6), om, nc, dict(J=6, u=2))


@pytest.mark.parametrize("nc", [1, 8])
def test_rows_move_samples_between_small_pieces(nc):
    """Pieces of 64 samples, half a record of the stored H, on a dense cluster: the record's rows are sorted across
    the pieces, and the fixed-point spread scales by what each piece then holds."""
    import torch

    from nufft_3d_gb300 import nufft_3d
    rng = np.random.default_rng(11)
    om = np.concatenate([rng.normal(0, 0.6, (3, 9000)), rng.uniform(-8, 7, (3, 4000))], axis=1)
    obj = nufft_3d(om, 16, J=6, density_iters=0, tap_table=1, spread_table=0, samples_per_block=64)
    assert obj.tap_table_bytes > 0 and obj.spread_table_bytes == 0
    ref = NufftRef(om, 16, J=6, density_iters=0)
    y = np.abs(rng.standard_normal((om.shape[1], nc))) + 1j * np.abs(rng.standard_normal((om.shape[1], nc)))
    a = obj.aNUFT(torch.from_numpy(np.ascontiguousarray(y.T).astype(np.complex64)).cuda()).cpu().numpy()
    r = ref.aNUFT(y)
    a = a.transpose(3, 2, 1, 0)
    assert np.linalg.norm(a - r.reshape(a.shape)) < 1e-5 * np.linalg.norm(r)


@pytest.mark.parametrize("nc", [1, 2, 3, 4, 5, 6, 7, 8, 9, 16])
@pytest.mark.parametrize("N,opts", [
    ((14, 18, 22), dict(J=6, u=2)),               # one to three tiles an axis, every column at the edge
    ((12, 26, 10), dict(J=5, u=1.5, radial=0)),   # tiles cut short by the grid
    ((36, 20, 12), dict(J=2, u=2)),               # odd tile origins moved by one
    ((50, 44, 1), dict(J=4, u=2)),
])
def test_tiles_that_wrap(N, opts, nc):
    """Samples in the outermost cells of both ends of every axis: rows that wrap in x, in y and in both."""
    rng = np.random.default_rng(nc)
    n = np.asarray(N)
    m = 3000
    om = np.stack([np.where(rng.random(m) < 0.5, -v / 2 + rng.random(m), v / 2 - 1 - rng.random(m)) if v > 1
                   else np.zeros(m) for v in n])
    om[:, ::3] = np.stack([rng.uniform(-v / 2, v / 2 - 1, om[:, ::3].shape[1]) if v > 1
                           else np.zeros(om[:, ::3].shape[1]) for v in n])
    _case(N, om, nc, opts)
