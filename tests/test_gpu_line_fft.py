"""The line FFTs at every pair of register factors, on every axis, with ragged runs of lines.

Oversampled lengths that are products of two factors of up to 32 points, and
lengths that are not (a prime factor squared times another), against the FP64
oracle: FP32 FFTs of a few hundred points stay below 1e-6, the operators'
tolerance of 1e-5 covers the interpolation too.
"""
import numpy as np
import pytest

from oracle.nufft_ref import NufftRef

pytestmark = pytest.mark.gpu

# oversampled lengths: the smallest, each radix as the larger factor, remainders of threads per column, no split
LENGTHS = [12, 20, 22, 26, 36, 54, 56, 66, 70, 98, 110, 126, 130, 150, 156, 168, 182, 192, 196, 200, 208, 210, 240, 242,
           250, 256, 286, 308, 338, 364, 378, 420, 484, 512, 540, 572, 686, 700, 840, 896, 900, 1024]


@pytest.mark.parametrize("K", LENGTHS)
def test_lengths(K):
    import torch

    from nufft_3d_gb300 import nufft_3d
    rng = np.random.default_rng(K)
    for axis, nc in ((0, 3), (1, 5), (2, 1), (2, 16)):
        N = [10, 8 if axis else 6, 6]
        N[axis] = 2 * round(K / 4)
        u = K / N[axis] - 1e-9
        om = np.stack([rng.uniform(-n / 2, n / 2 - 1, 1500) for n in N])
        obj = nufft_3d(om, tuple(N), J=4, u=u, density_iters=0)
        ref = NufftRef(om, tuple(N), J=4, u=u, density_iters=0)
        assert ref.K[axis] == K
        x = rng.standard_normal((*N, nc)) + 1j * rng.standard_normal((*N, nc))
        y = rng.standard_normal((1500, nc)) + 1j * rng.standard_normal((1500, nc))
        f = obj.fNUFT(torch.from_numpy(x.transpose(3, 2, 1, 0).astype(np.complex64)).cuda()).cpu().numpy()
        a = obj.aNUFT(torch.from_numpy(np.ascontiguousarray(y.T).astype(np.complex64)).cuda()).cpu().numpy()
        fr, ar = ref.fNUFT(x), ref.aNUFT(y)
        f = f.reshape(nc, -1).T
        a = a.transpose(3, 2, 1, 0)
        assert np.linalg.norm(f - fr.reshape(f.shape)) < 1e-5 * np.linalg.norm(fr)
        assert np.linalg.norm(a - ar.reshape(a.shape)) < 1e-5 * np.linalg.norm(ar)


@pytest.mark.parametrize("N,u,nc", [((256, 250, 1), 2, 8), ((42, 100, 1), 1.5, 7), ((28, 34, 46), 1.4, 2)])
def test_other_oversampling(N, u, nc):
    import torch

    from nufft_3d_gb300 import nufft_3d
    rng = np.random.default_rng(1)
    om = np.stack([rng.uniform(-n / 2, n / 2 - 1, 3000) if n > 1 else np.zeros(3000) for n in N])
    obj = nufft_3d(om, N, J=5, u=u, density_iters=0)
    ref = NufftRef(om, N, J=5, u=u, density_iters=0)
    x = rng.standard_normal((*N, nc)) + 1j * rng.standard_normal((*N, nc))
    f = obj.fNUFT(torch.from_numpy(x.transpose(3, 2, 1, 0).astype(np.complex64)).cuda()).cpu().numpy()
    fr = ref.fNUFT(x)
    f = f.reshape(nc, -1).T
    assert np.linalg.norm(f - fr.reshape(f.shape)) < 1e-5 * np.linalg.norm(fr)


@pytest.mark.parametrize("N,u,nc", [((10, 6, 500), 2, 1), ((6, 8, 500), 2, 3), ((6, 500, 8), 2, 4),
                                    ((8, 6, 454), 910 / 454 - 1e-9, 1), ((6, 6, 528), 2, 2)])
def test_long_lengths_without_a_split(N, u, nc):
    """K = 1000, 910, 1056 on the y and z axes: 16 lines of two Stockham buffers would not fit in shared memory."""
    import torch

    from nufft_3d_gb300 import nufft_3d
    rng = np.random.default_rng(N[2])
    om = np.stack([rng.uniform(-n / 2, n / 2 - 1, 1500) for n in N])
    obj = nufft_3d(om, N, J=4, u=u, density_iters=0)
    ref = NufftRef(om, N, J=4, u=u, density_iters=0)
    x = rng.standard_normal((*N, nc)) + 1j * rng.standard_normal((*N, nc))
    y = rng.standard_normal((1500, nc)) + 1j * rng.standard_normal((1500, nc))
    f = obj.fNUFT(torch.from_numpy(x.transpose(3, 2, 1, 0).astype(np.complex64)).cuda()).cpu().numpy()
    a = obj.aNUFT(torch.from_numpy(np.ascontiguousarray(y.T).astype(np.complex64)).cuda()).cpu().numpy()
    fr, ar = ref.fNUFT(x), ref.aNUFT(y)
    f = f.reshape(nc, -1).T
    a = a.transpose(3, 2, 1, 0)
    assert np.linalg.norm(f - fr.reshape(f.shape)) < 1e-5 * np.linalg.norm(fr)
    assert np.linalg.norm(a - ar.reshape(a.shape)) < 1e-5 * np.linalg.norm(ar)


@pytest.mark.parametrize("K", [132, 150, 168, 182, 196, 200, 210, 242, 308, 338, 420, 484, 512, 572, 700, 896, 1024])
def test_x_lengths_with_many_lines(K):
    """x passes of at least 768 lines take the two register phases at every length; with fewer the block-a-row form."""
    import torch

    from nufft_3d_gb300 import nufft_3d
    rng = np.random.default_rng(K)
    n = 2 * -(-K // 4)
    u = K / n - 1e-9
    for N, nc in (((n, 16, 16), 3), ((n, 14, 10), 5)):  # 768 and 700 lines
        om = np.stack([rng.uniform(-v / 2, v / 2 - 1, 1200) for v in N])
        obj = nufft_3d(om, N, J=4, u=u, density_iters=0)
        ref = NufftRef(om, N, J=4, u=u, density_iters=0)
        assert ref.K[0] == K
        x = rng.standard_normal((*N, nc)) + 1j * rng.standard_normal((*N, nc))
        y = rng.standard_normal((1200, nc)) + 1j * rng.standard_normal((1200, nc))
        f = obj.fNUFT(torch.from_numpy(x.transpose(3, 2, 1, 0).astype(np.complex64)).cuda()).cpu().numpy()
        a = obj.aNUFT(torch.from_numpy(np.ascontiguousarray(y.T).astype(np.complex64)).cuda()).cpu().numpy()
        fr, ar = ref.fNUFT(x), ref.aNUFT(y)
        assert np.linalg.norm(f.T - fr.reshape(f.T.shape)) < 1e-5 * np.linalg.norm(fr)
        a = a.transpose(3, 2, 1, 0)
        assert np.linalg.norm(a - ar.reshape(a.shape)) < 1e-5 * np.linalg.norm(ar)
