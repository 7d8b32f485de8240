"""GPU parity of the batched (multi-volume) operators: every volume of a batch
equals its own single-plan fNUFT / aNUFT / CG iNUFT (rel L2 <= 1e-5 for the
operators, <= 1e-4 for the iterative images)."""
import numpy as np
import pytest

from nufft_3d_gb300 import NufftBatch, nufft_3d, synth

pytestmark = pytest.mark.gpu
TOL_OP = 1e-5
TOL_IMG = 1e-4


def rel(a, b):
    return float((a - b).abs().norm() / b.abs().norm())


def volumes():
    specs = [(16, "koosh", 3), (24, "random", 1), (32, "koosh", 8), (20, "spiral", 4), (32, "koosh", 2)]
    out = []
    for i, (N, kind, nc) in enumerate(specs):
        if kind == "koosh":
            om = synth.koosh_ball(N, N, 40 * N)
        elif kind == "random":
            om = synth.random_uniform(N, 3 * N ** 3 // 2, seed=i)
        else:
            om = synth.stack_of_spirals(N, n_interleaves=4, n_samples=256, n_partitions=N)
        out.append((om, N, nc))
    return out


def test_batch_matches_single(cuda):
    torch = cuda
    vols = volumes()
    objs = [nufft_3d(om, N, "J", 6) for om, N, _ in vols]
    objs[4] = objs[2].share() if vols[4][1] == vols[2][1] and vols[4][0].shape == vols[2][0].shape else objs[4]
    ncs = [nc for _, _, nc in vols]
    g = torch.Generator(device="cuda").manual_seed(0)
    xs = [torch.randn((nc,) + (int(o.N[2]), int(o.N[1]), int(o.N[0])), dtype=torch.complex64, device="cuda",
                      generator=g) for o, nc in zip(objs, ncs)]
    ys = [torch.randn((nc, o.M), dtype=torch.complex64, device="cuda", generator=g) for o, nc in zip(objs, ncs)]
    single_k = [o.fNUFT(x) for o, x in zip(objs, xs)]
    single_a = [o.aNUFT(y) for o, y in zip(objs, ys)]
    single_i = [o.iNUFT(y, 8, 0.05, solver="cg", tol=0) for o, y in zip(objs, ys)]
    batch = NufftBatch(objs, ncs)
    ks = batch.forward(xs)
    xa = batch.adjoint(ys)
    xi, its = batch.inverse(ys, 8, 0.05, tol=0, return_iters=True)
    torch.cuda.synchronize()
    for v in range(len(objs)):
        assert rel(ks[v], single_k[v]) < TOL_OP, v
        assert rel(xa[v], single_a[v]) < TOL_OP, v
        assert rel(xi[v], single_i[v]) < TOL_IMG, v
    assert all(i == 8 for i in its)
    batch.close()
    for o in objs:
        o.close()


def test_batch_rejects_mixed_kernels(cuda):
    om = synth.koosh_ball(16, 16, 200)
    a = nufft_3d(om, 16, "J", 6)
    b = nufft_3d(om, 16, "J", 4)
    with pytest.raises(Exception, match="share"):
        NufftBatch([a, a], [1, 1])
    with pytest.raises(Exception, match="kernel"):
        NufftBatch([a, b], [1, 1])
    c = nufft_3d(om, 16, "J", 6, "u", 1.5)   # same ceil(J/2), different alpha
    with pytest.raises(Exception, match="kernel"):
        NufftBatch([a.share(), c], [1, 1])


def test_objects_closed_before_their_batch(cuda):
    """Objects closed before their batch, as at the end of a program: the batch frees what is its own."""
    om = synth.koosh_ball(16, 16, 200)
    objs = [nufft_3d(om, 16, "J", 6, density_iters=0) for _ in range(2)]
    batch = NufftBatch(objs, [1, 2])
    ks = batch.forward([cuda.randn(c, 16, 16, 16, dtype=cuda.complex64, device="cuda") for c in (1, 2)])
    for o in objs:
        o.close()
    batch.close()
    assert all(bool(cuda.isfinite(cuda.view_as_real(k)).all()) for k in ks)


@pytest.mark.parametrize("shape,nvol,ncs", [
    ((16, 16, 16), 9, (1, 2, 8)),      # small volumes: narrow passes share a launch, 8-coil ones are their own
    ((24, 20, 30), 11, (1, 3, 12)),    # more volumes than side streams, a pass of each kind in one volume
    ((40, 36, 1), 10, (1, 8)),         # 2-D: few tiles, all shared
    ((140, 128, 1), 3, (2, 8, 9)),     # 2-D: 8-coil passes of their own, ranges of records merged
])
def test_many_volumes(cuda, shape, nvol, ncs):
    """Volumes with both tables, with the stored H alone and with none, in one batch on a stream of its own: each
    equals its own object."""
    torch = cuda
    rng = np.random.default_rng(nvol)
    tables = [dict(tap_table=1, spread_table=1), dict(tap_table=1, spread_table=0), dict(tap_table=0)]
    objs, xs, ys = [], [], []
    for v in range(nvol):
        m = 1500 + 977 * v
        om = np.stack([rng.uniform(-n / 2, n / 2 - 1, m) if n > 1 else np.zeros(m) for n in shape])
        if v % 2:  # a dense centre
            om = om * rng.random(m) ** 2
        objs.append(nufft_3d(om, shape, "J", 6, density_iters=3, **(tables[v % 3] if v > 4 else tables[0])))
        nc = ncs[v % len(ncs)]
        xs.append(torch.randn(nc, *shape[::-1], dtype=torch.complex64, device="cuda"))
        ys.append(torch.randn(nc, m, dtype=torch.complex64, device="cuda"))
    single_k = [o.fNUFT(x) for o, x in zip(objs, xs)]
    single_a = [o.aNUFT(y) for o, y in zip(objs, ys)]
    single_i = [o.iNUFT(y, 4, 0.05, solver="cg", tol=0.0) for o, y in zip(objs, ys)]
    batch = NufftBatch(objs, [x.shape[0] for x in xs])
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        for _ in range(2):
            ks, xa, xi = batch.forward(xs), batch.adjoint(ys), batch.inverse(ys, 4, 0.05, tol=0.0)
    stream.synchronize()
    for v in range(nvol):
        assert rel(ks[v], single_k[v]) < TOL_OP, v
        assert rel(xa[v], single_a[v]) < TOL_OP, v
        assert rel(xi[v], single_i[v]) < TOL_IMG, v
        objs[v].check_status(stream)
    batch.close()
