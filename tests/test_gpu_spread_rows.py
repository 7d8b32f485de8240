"""The spread from the stored H' (rows of 2 x 2 points) at the sizes where it can go wrong.

Every coil width, odd coil counts beyond a pass, a slab with more samples than
a piece, runs of slabs that end at the longest piece, grids smaller than a
padded tile, 2-D.  Against the FP64 oracle per coil: FP32 sums of at most a few
thousand products of both signs, below 1e-5 (the operators' tolerance).
"""
import numpy as np
import pytest

from oracle.nufft_ref import NufftRef

pytestmark = pytest.mark.gpu


def _case(N, om, nc, opts, seed=5):
    import torch

    from nufft_3d_gb300 import nufft_3d
    rng = np.random.default_rng(seed)
    obj = nufft_3d(om, N, density_iters=0, tap_table=1, spread_table=1, **opts)
    assert obj.spread_table_bytes > 0
    ref = NufftRef(om, N, density_iters=0, **opts)
    y = rng.standard_normal((om.shape[1], nc)) + 1j * rng.standard_normal((om.shape[1], nc))
    yt = torch.from_numpy(np.ascontiguousarray(y.T).astype(np.complex64)).cuda()
    r = ref.aNUFT(y)
    for _ in range(2):
        a = obj.aNUFT(yt).cpu().numpy().transpose(3, 2, 1, 0)
        for c in range(nc):
            assert np.linalg.norm(a[..., c] - r[..., c]) < 1e-5 * np.linalg.norm(r[..., c])


@pytest.mark.parametrize("nc", [1, 2, 3, 4, 5, 6, 7, 8, 9, 11, 12])
def test_coil_widths(nc):
    rng = np.random.default_rng(nc)
    _case(18, rng.uniform(-9, 8, (3, 33001)), nc, dict(J=6, u=2))  # above the size where narrow passes use H'


@pytest.mark.parametrize("N,opts", [
    (4, dict(J=6, u=2)),
    ((6, 20, 10), dict(J=5, u=1.5, radial=0)),
    (14, dict(J=2, u=2)),
    ((12, 10, 60), dict(J=4, u=2)),   # columns longer than a piece
    ((36, 20, 1), dict(J=6, u=2)),
])
@pytest.mark.parametrize("nc", [1, 8])
def test_grids(N, opts, nc):
    rng = np.random.default_rng(7)
    n = np.resize(np.asarray(N), 3)
    om = np.stack([rng.uniform(-v / 2, v / 2 - 1, 33000) if v > 1 else np.zeros(33000) for v in n])
    _case(N, om, nc, opts)


@pytest.mark.parametrize("nc", [2, 8])
def test_dense_slab(nc):
    """6000 samples at nearly one point (shares of a slab, equal terms) beside a sparse rest."""
    rng = np.random.default_rng(3)
    om = np.concatenate([rng.normal(0, 1e-3, (3, 6000)), rng.uniform(-8, 7, (3, 30000))], axis=1)
    _case(16, om, nc, dict(J=6, u=2))
