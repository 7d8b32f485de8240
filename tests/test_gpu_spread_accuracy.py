"""The rounding of the spread's long sums.

k-space data fall by orders of magnitude from their centre, which every spoke
of a radial trajectory samples: the adjoint's error against FP64 is the
rounding of the sums of those few grid points, and grows with the number of
partial sums that meet there.  A spread whose rows reach those points in few
pieces stays near the error of the FP32 FFT passes, 1e-7.
"""
import numpy as np
import pytest

from oracle.cpu_bench import adjoint_per_coil
from oracle.nufft_ref import NufftRef

pytestmark = pytest.mark.gpu


def _blob_samples(om, nc, rng):
    """Transform of 16 Gaussian blobs at om, with noise at 30 dB."""
    centre, sigma = rng.uniform(-0.3, 0.3, (16, 3)), np.exp(rng.uniform(np.log(0.008), np.log(0.12), 16))
    gain = rng.standard_normal((16, nc)) + 1j * rng.standard_normal((16, nc))
    r2 = np.sum(om * om, axis=0)
    k = sum((np.sqrt(2 * np.pi) * s) ** 3 * np.exp(-2 * np.pi ** 2 * s * s * r2 - 2j * np.pi * (c @ om))[:, None] * g
            for c, s, g in zip(centre, sigma, gain))
    power = np.mean(np.abs(k) ** 2, axis=0) * 1e-3 / 2
    return k + np.sqrt(power) * (rng.standard_normal(k.shape) + 1j * rng.standard_normal(k.shape))


def _koosh(n, nr, ns, rng):
    d = rng.standard_normal((3, ns))
    d /= np.linalg.norm(d, axis=0)
    return (d[:, :, None] * np.linspace(0, n / 2 - 1, nr)).reshape(3, -1)


@pytest.mark.parametrize("nc", [1, 8])
def test_radial_data(nc):
    """64^3, 64 x 4096 centre-out spokes: at most 1.6e-7 on average, a quarter above the worst of the sums of whole
    tiles with 1664 samples a share (1.28e-7; shares of 431 samples gave 2.2e-7)."""
    import torch

    from nufft_3d_gb300 import nufft_3d
    errs = []
    for seed in range(3):
        rng = np.random.default_rng(seed)
        om = _koosh(64, 64, 4096, rng)
        y = _blob_samples(om, nc, rng).astype(np.complex64)
        obj = nufft_3d(om, 64, J=6, u=2, density_iters=0, tap_table=1, spread_table=1)
        ref = NufftRef(om, 64, J=6, u=2, density_iters=0, matrix=False)
        r = adjoint_per_coil(ref, y.astype(np.complex128))
        yt = torch.from_numpy(np.ascontiguousarray(y.T)).cuda()
        for _ in range(2):
            a = obj.aNUFT(yt).cpu().numpy().transpose(3, 2, 1, 0)
            errs.append(np.linalg.norm(a.reshape(r.shape) - r) / np.linalg.norm(r))
    assert np.mean(errs) < 1.6e-7, errs
