"""The work that a user of nufft_3d_gb300 has it do, as cases that can be timed.

A case names an operation, a volume, a trajectory, a kernel and a coil count.
The listed sizes are this repository's own: the single-coil 64^3 koosh ball
(forward, adjoint, CG), the 128^3 x 8-coil koosh ball of bench.py,
uneven batched volumes, the 192^3 x 16-coil normal operator that its CG
iterates, 2-D radial slices, and the uneven sizes, coil counts and kernels
that the tests cover.  ``draw`` gives others of the same ranges.

Images and samples are a sum of Gaussian blobs and its analytic transform plus
noise at 30 dB, so both have the dynamic range of real data (k-space falls by
orders of magnitude from its centre), and trajectories are rotated by the seed.
"""
import math

import numpy as np
import torch

from nufft_3d_gb300 import NufftBatch, nufft_3d

DEV = "cuda"
BLOBS = 16


def _case(name, op, n, traj, nr, ns, nc, J=6, u=2.0, radial=True, iters=0, solver="cg", given_d=False, mix=0):
    c = {"op": op, "n1": n[0], "n2": n[1], "n3": n[2], "traj": traj, "nr": nr, "ns": ns, "nc": nc, "J": J,
         "u": u, "radial": radial, "iters": iters, "solver": solver, "given_d": given_d, "mix": mix}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest calls: a navigator or a test volume, where launches and latency are what counts
        _case("forward_32_c1", "forward", (32, 32, 32), "koosh", 32, 512, 1),
        # the repository's plain configuration: one coil at 64^3, 64 x 4096 koosh ball
        _case("forward_64_c1", "forward", (64, 64, 64), "koosh", 64, 4096, 1),
        _case("adjoint_64_c1", "adjoint", (64, 64, 64), "koosh", 64, 4096, 1),
        # ... and its reconstruction, 8 CG iterations (damp 1e-3, density weights from the plan)
        _case("cg_64_c1", "solve", (64, 64, 64), "koosh", 64, 4096, 1, iters=8),
        # one 2-D slice, golden-angle radial, 8 coils
        _case("adjoint_2d_256_c8", "adjoint", (256, 256, 1), "radial2d", 512, 402, 8),
        # numpy arrays in, numpy arrays out: the host program that the class mirrors
        _case("host_forward_64_c8", "host_forward", (64, 64, 64), "koosh", 128, 4096, 8),
        # an uneven volume, an odd coil count, a separable kernel at low oversampling, random samples
        _case("forward_uneven_c5", "forward", (88, 112, 100), "random", 1000003, 1, 5, J=5, u=1.5, radial=False),
        # the constructor's default kernel width on another uneven volume, three coils
        _case("adjoint_uneven_c3", "adjoint", (100, 84, 60), "spirals", 1000, 704, 3, J=4),
        # the benchmark's single large forward and adjoint: 8.4 M samples, 8 coils
        _case("forward_128_c8", "forward", (128, 128, 128), "koosh", 256, 32768, 8),
        _case("adjoint_128_c8", "adjoint", (128, 128, 128), "koosh", 256, 32768, 8),
        # uneven volumes reconstructed together, CG on all of them
        _case("batch_cg", "batch", (64, 64, 64), "mixed", 4, 1, 12, iters=4, mix=3),
        # the largest: one application of the normal operator of the 192^3 x 16-coil reconstruction
        _case("normal_192_c16", "normal", (192, 192, 192), "koosh", 384, 60000, 16, given_d=True),
    ]


# ------------------------------------------------------------- other cases
def _smooth(k):
    for p in (2, 3, 5, 7, 11, 13):
        while k % p == 0:
            k //= p
    return k == 1


def _side(rng, lo, hi, u):
    """An even volume side between lo and hi (spread over its logarithm) whose oversampled length the library takes."""
    while True:
        n = 2 * int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2))
        if _smooth(2 * math.ceil(n * u / 2)):
            return n


def draw(rng):
    op = rng.choice(["forward", "adjoint", "forward", "adjoint", "normal", "solve", "host_forward", "batch"])
    if op == "batch":
        return _case(None, op, (64, 64, 64), "mixed", rng.randint(2, 4), 1, rng.randint(2, 12), iters=rng.randint(2, 4),
                     mix=rng.randrange(1 << 20))
    J, u = rng.choice([(6, 2.0), (6, 2.0), (4, 2.0), (5, 1.5), (6, 1.5)])
    radial = rng.random() < 0.7
    small = op in ("solve", "host_forward")
    if rng.random() < 0.15 and not small:
        n1, n2 = _side(rng, 64, 512, u), _side(rng, 64, 512, u)
        nr = rng.randint(n1 // 2, 2 * n1)
        return _case(None, op, (n1, n2, 1), "radial2d", nr, rng.randint(n1 // 2, 2 * n1), rng.randint(1, 16), J, u,
                     radial, given_d=op == "normal")
    if rng.random() < 0.5:
        n = (_side(rng, 24, 96 if small else 176, u),) * 3
    else:
        n = tuple(_side(rng, 24, 96 if small else 176, u) for _ in range(3))
    nc = rng.choice([1, 2, 3, 4, 5, 6, 7, 8, 8, 8, 10, 12, 16])
    # 0.3 to 4 samples a voxel, at most 2e8 samples over all coils (half of that for the separable kernel, which has
    # twice the taps) and 2e6 where a whole solve or a host call is drawn
    m = int(n[0] * n[1] * n[2] * math.exp(rng.uniform(math.log(0.3), math.log(4))))
    m = max(1001, min(m, int((2e6 if small else 2e8 if radial else 1e8) / nc)))
    traj = rng.choice(["koosh", "koosh", "spirals", "random"])
    if traj == "random":
        nr, ns = m, 1
    else:
        nr = rng.randint(max(n) // 2, 2 * max(n))
        ns = max(2, m // nr)
    return _case(None, op, n, traj, nr, ns, nc, J, u, radial, iters=rng.randint(3, 6) if op == "solve" else 0,
                 solver=rng.choice(["cg", "minres"]), given_d=op == "normal")


# ------------------------------------------------------------------ inputs
def _rotation(rng):
    a = rng.standard_normal(4)
    a, b, c, d = a / np.linalg.norm(a)
    return np.array([[a * a + b * b - c * c - d * d, 2 * (b * c - a * d), 2 * (b * d + a * c)],
                     [2 * (b * c + a * d), a * a - b * b + c * c - d * d, 2 * (c * d - a * b)],
                     [2 * (b * d - a * c), 2 * (c * d + a * b), a * a - b * b - c * c + d * d]])


def _stack(n, ns):
    """Partitions and interleaves of a stack of spirals of about ns shots."""
    parts = max(1, min(64, n[2], ns))
    return parts, max(1, ns // parts)


def _count(n, traj, nr, ns):
    parts, inter = _stack(n, ns)
    return nr * (parts * inter if traj == "spirals" else ns)


def _trajectory(traj, n, nr, ns, seed):
    """om [3, nr*ns] in cycles/FOV."""
    rng = np.random.default_rng([seed, 1])
    half = np.array([v / 2 - 1 if v > 1 else 0 for v in n], dtype=np.float64)
    if traj == "koosh":  # centre-out spokes on a golden-angle sphere
        t = np.linspace(0.0, 1.0, nr)
        k = np.arange(ns, dtype=np.float64)
        polar = np.arccos(np.clip(1 - 2 * k / max(ns - 1, 1), -1, 1))
        azim = k * math.pi * (3 - math.sqrt(5))
        d = np.stack([np.cos(azim) * np.sin(polar), np.sin(azim) * np.sin(polar), np.cos(polar)])
        d = (_rotation(rng) @ d) * half[:, None]
        return (d[:, :, None] * t[None, None, :]).reshape(3, -1)
    if traj == "radial2d":  # full spokes, golden angle
        t = np.linspace(-1.0, 1.0, nr)
        a = rng.uniform(0, math.pi) + np.arange(ns) * math.pi * (math.sqrt(5) - 1) / 2
        d = np.stack([np.cos(a), np.sin(a), np.zeros(ns)]) * half[:, None]
        return (d[:, :, None] * t[None, None, :]).reshape(3, -1)
    if traj == "spirals":  # spiral interleaves, stacked in kz
        parts, inter = _stack(n, ns)
        t = np.linspace(0.0, 1.0, nr)
        a = 2 * math.pi * (max(1.0, max(n[0], n[1]) / (2 * inter)) * t + np.arange(inter)[:, None] / inter)
        a = a + rng.uniform(0, 2 * math.pi)
        xy = np.stack([half[0] * t * np.cos(a), half[1] * t * np.sin(a)]).reshape(2, 1, -1)
        z = np.linspace(-n[2] / 2, n[2] / 2 - 1, parts)
        xy, z = np.broadcast_arrays(xy, z[None, :, None])
        return np.concatenate([xy, z[:1]]).reshape(3, -1)
    lo = np.array([[-v / 2] if v > 1 else [0] for v in n])  # uniform over k-space
    return lo + rng.random((3, nr * ns)) * np.maximum(np.array([[v - 1] for v in n]), 0)


def _blobs(seed, nc, three_d):
    g = np.random.default_rng([seed, 2])
    centre = g.uniform(-0.3, 0.3, (BLOBS, 3))
    sigma = np.exp(g.uniform(math.log(0.008), math.log(0.12), BLOBS))
    if not three_d:
        centre[:, 2] = 0
    gain = g.standard_normal((BLOBS, nc)) + 1j * g.standard_normal((BLOBS, nc))
    return centre, sigma, gain * np.exp(g.uniform(-1, 1, (1, nc)))


def _noise(shape, power, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(shape, dtype=torch.complex64, device=DEV, generator=g) * math.sqrt(power * 1e-3)


def _image(n, nc, seed):
    """(nc, n3, n2, n1) complex64."""
    centre, sigma, gain = _blobs(seed, nc, n[2] > 1)
    axes = [(torch.arange(v, device=DEV, dtype=torch.float32) - v // 2) / v for v in n]
    rows = []
    for b in range(BLOBS):
        e = [torch.exp(-(axes[a] - float(centre[b, a])) ** 2 / (2 * float(sigma[b]) ** 2)) for a in range(3)]
        if n[2] == 1:
            e[2] = torch.ones(1, device=DEV)
        rows.append((e[2][:, None, None] * e[1][None, :, None] * e[0][None, None, :]).reshape(-1))
    im = torch.as_tensor(gain.T, dtype=torch.complex64, device=DEV) @ torch.stack(rows).to(torch.complex64)
    im = im.reshape(nc, n[2], n[1], n[0])
    return im + _noise(im.shape, float(torch.view_as_real(im).square().mean()) * 2, seed)


def _samples(om, n, nc, seed):
    """(nc, M) complex64: the blobs' transform at om."""
    centre, sigma, gain = _blobs(seed, nc, n[2] > 1)
    dim = 3 if n[2] > 1 else 2
    m = om.shape[1]
    out = torch.empty((nc, m), dtype=torch.complex64, device=DEV)
    gt = torch.as_tensor(gain.T, dtype=torch.complex64, device=DEV)
    for lo in range(0, m, 1 << 21):
        o = torch.as_tensor(np.ascontiguousarray(om[:, lo:lo + (1 << 21)]), dtype=torch.float32, device=DEV)
        r2 = o.square().sum(0)
        c = torch.as_tensor(centre, dtype=torch.float32, device=DEV)
        s = torch.as_tensor(sigma, dtype=torch.float32, device=DEV)[:, None]
        mag = (math.sqrt(2 * math.pi) * s) ** dim * torch.exp(-2 * math.pi ** 2 * s * s * r2)
        out[:, lo:lo + (1 << 21)] = gt @ torch.polar(mag, -2 * math.pi * (c @ o))
    return out + _noise(out.shape, float(torch.view_as_real(out).square().mean()) * 2, seed)


def _volumes(case):
    """(n, traj, nr, ns, nc) of a batch: sides 64 or 96, trajectories in turn, 4 to 12 coils."""
    r = np.random.default_rng(case["mix"])
    vols = []
    for v in range(case["nr"]):
        side = int(r.choice([64, 96]))
        count = int(r.uniform(0.5, 1.5) * side ** 3)
        traj = ("koosh", "spirals", "random")[v % 3]
        nr, ns = {"koosh": (side, count // side), "spirals": (max(64, count // 1024), 1024), "random": (count, 1)}[traj]
        vols.append(((side,) * 3, traj, nr, ns, int(r.integers(min(4, case["nc"]), case["nc"] + 1))))
    return vols


def _parts(case):
    if case["op"] == "batch":
        return _volumes(case)
    return [((case["n1"], case["n2"], case["n3"]), case["traj"], case["nr"], case["ns"], case["nc"])]


def _analytic_d(om):
    r2 = np.sum(om * om, axis=0)
    r2 = r2 + r2.max() * 1e-4
    return (r2 / r2.mean()).astype(np.float32)


def _options(case, om):
    o = {"J": case["J"], "u": case["u"], "radial": case["radial"]}
    if case["given_d"]:
        o["d"] = _analytic_d(om)
    return o


def prepare(case, seed):
    objs, ins = [], []
    for v, (n, traj, nr, ns, nc) in enumerate(_parts(case)):
        om = _trajectory(traj, n, nr, ns, seed + v)
        objs.append(nufft_3d(om, list(n), **_options(case, om)))
        if case["op"] in ("adjoint", "solve", "batch"):
            ins.append(_samples(om, n, nc, seed + v))
        else:
            ins.append(_image(n, nc, seed + v))
    st = {"case": case, "objs": objs, "ins": ins}
    if case["op"] == "batch":
        st["batch"] = NufftBatch(objs, [k.shape[0] for k in ins])
    if case["op"] == "host_forward":
        st["ins"] = [np.asfortranarray(ins[0].cpu().numpy().transpose(3, 2, 1, 0))]
    return st


def run(state):
    case, obj, x = state["case"], state["objs"][0], state["ins"][0]
    op = case["op"]
    if op in ("forward", "host_forward"):
        return obj.fNUFT(x)
    if op == "adjoint":
        return obj.aNUFT(x)
    if op == "normal":
        return obj.iprojection(x, 0.1)
    if op == "solve":
        return obj.iNUFT(x, case["iters"], 1e-3, solver=case["solver"], tol=0.0)
    return state["batch"].inverse(state["ins"], case["iters"], 1e-3, tol=0.0)


def work(case):
    """Inputs (data, 12 bytes of coordinates a sample, weights) read once and outputs written once; the flops of the
    taps (4 per coil and tap: a real weight times a complex value, added) and of the oversampled FFTs."""
    nbytes = flops = 0.0
    for n, traj, nr, ns, nc in _parts(case):
        m = _count(n, traj, nr, ns)
        vox = float(n[0] * n[1] * n[2])
        grid = 1.0
        for v in n:
            grid *= 2 * math.ceil(v * case["u"] / 2) if v > 1 else 1
        h = case["J"] / 2
        if n[2] == 1:
            taps = math.pi * h ** 2 if case["radial"] else case["J"] ** 2
        else:
            taps = 4 / 3 * math.pi * h ** 3 if case["radial"] else case["J"] ** 3
        one = m * nc * taps * 4 + nc * 5 * grid * math.log2(grid)
        nbytes += 12.0 * m
        if case["op"] == "normal":
            nbytes += 2 * 8 * vox * nc + 4 * m
            flops += 2 * one
        else:
            nbytes += 8.0 * nc * (vox + m) + (4 * m if case["iters"] else 0)
            flops += one * (2 * case["iters"] + 1 if case["iters"] else 1)
    return {"bytes": nbytes, "flops": flops}


# --------------------------------------------------- the same in 64 bits
class _Plain:
    """The operators with dense torch arithmetic in 64 bits: zero-padded FFTs and, for each of the (2R+1)^3 grid
    offsets, one gather or scatter over all samples."""

    SMALL = (1.0, 3.5156229, 3.0899424, 1.2067492, 0.2659732, 0.360768e-1, 0.45813e-2)
    LARGE = (0.39894228, 0.1328592e-1, 0.225319e-2, -0.157565e-2, 0.916281e-2, -0.2057706e-1, 0.2635537e-1,
             -0.1647633e-1, 0.392377e-2)

    def __init__(self, om, n, case, density):
        self.n, self.J, self.u, self.radial = n, float(case["J"]), float(case["u"]), case["radial"]
        self.R = math.ceil(self.J / 2)
        self.K = [2 * math.ceil(v * self.u / 2) if v > 1 else 1 for v in n]
        q = (self.J * (1 - 0.5 / self.u)) ** 2
        self.alpha = math.pi * math.sqrt(q - 0.6 * self.u if self.radial else q - 0.8)
        self.i0a = float(self._i0(torch.tensor([self.alpha], dtype=torch.complex128))[0].real)
        og = torch.as_tensor(om, dtype=torch.float64, device=DEV) * self.u
        self.M = og.shape[1]
        ok = torch.ones(self.M, dtype=torch.bool, device=DEV)
        if n[2] > 1:
            for a in range(3):
                ok &= (og[a] >= -self.K[a] / 2) & (og[a] <= self.K[a] / 2 - 1)
        self.keep = ok.nonzero()[:, 0]
        self.og = og[:, self.keep]
        self.base = torch.sign(self.og) * torch.floor(self.og.abs() + 0.5)  # rounds halves away from zero
        self.nnz = self.keep.numel()
        rz = range(-self.R, self.R + 1) if n[2] > 1 else (0,)
        xy = range(-self.R, self.R + 1)
        low = lambda d: max(abs(d) - 0.5, 0.0) ** 2  # noqa: E731
        self.offsets = [(dx, dy, dz) for dz in rz for dy in xy for dx in xy
                        if not self.radial or low(dx) + low(dy) + low(dz) <= (self.J / 2) ** 2 + 1e-9]
        self.U = self._deap()
        self.d = None
        if density is not None:
            self.d = torch.as_tensor(density, dtype=torch.float64, device=DEV)[self.keep]
        elif case["op"] in ("solve", "batch", "normal"):
            d = torch.ones(self.nnz, dtype=torch.float64, device=DEV)
            for _ in range(20):
                hh = self.gather(self.spread(d[:, None]))[:, 0]
                d = d / torch.clamp(hh, min=2.220446049250313e-16)
            self.d = d / (d.sum() / self.nnz)

    def _i0(self, ax):
        out = torch.empty_like(ax)
        s = ax.abs() < 3.75
        for sel, cs in ((s, self.SMALL), (~s, self.LARGE)):
            a = ax[sel]
            y = (a / 3.75) ** 2 if cs is self.SMALL else 3.75 / a
            acc = torch.full_like(a, cs[-1])
            for c in cs[-2::-1]:
                acc = c + y * acc
            if cs is self.LARGE:
                acc = acc * torch.exp(a) / torch.sqrt(a)
                if a.is_complex():
                    acc = torch.where(a.real == 0, 2 * acc, acc)
            out[sel] = acc
        return out

    def _kernel(self, d2):
        t = 1 - d2 / (self.J / 2) ** 2
        return self._i0(self.alpha * torch.sqrt(torch.clamp(t, min=0.0))) / self.i0a

    def _deap(self):
        nj = int(math.floor(self.J)) + 1
        nz = nj if self.n[2] > 1 else 1
        d = torch.arange(nj, dtype=torch.float64) / 2
        dz = d[:nz]

        def table(d2):
            t = 1 - d2 / (self.J / 2) ** 2
            arg = torch.where(t >= 0, torch.sqrt(t.abs()).to(torch.complex128), 1j * torch.sqrt(t.abs()))
            return (self._i0(self.alpha * arg) / self.i0a).real
        if self.radial:
            T = table(d[:, None, None] ** 2 + d[None, :, None] ** 2 + dz[None, None, :] ** 2)
        else:
            T = table(d ** 2)[:, None, None] * table(d ** 2)[None, :, None] * table(dz ** 2)[None, None, :]
        for a in range(3 if nz > 1 else 2):
            p = torch.arange(self.n[a], dtype=torch.float64) - self.n[a] // 2
            j = torch.arange(T.shape[0], dtype=torch.float64)
            c = torch.cos(math.pi * j[None, :] * p[:, None] / self.K[a])
            c[:, 0] = 0.5
            T = torch.tensordot(T, c, dims=([0], [1]))  # the next axis comes to the front
        if nz == 1:
            T = T.permute(1, 2, 0)
        return (1.0 / T).permute(2, 1, 0).contiguous().to(DEV)

    def _taps(self, lo, hi):
        og, base = self.og[:, lo:hi], self.base[:, lo:hi]
        h2 = (self.J / 2) ** 2
        for off in self.offsets:
            e = [(base[a] + off[a] - og[a]) ** 2 for a in range(3)]
            if self.radial:
                d2 = e[0] + e[1] + e[2]
                w = torch.where(d2 <= h2, self._kernel(d2), 0.0)
            else:
                w = 1.0
                for a in range(3 if self.n[2] > 1 else 2):
                    w = w * torch.where(e[a] <= h2, self._kernel(e[a]), 0.0)
            ix = [torch.remainder(base[a] + off[a], self.K[a]).long() for a in range(3)]
            yield w, (ix[2] * self.K[1] + ix[1]) * self.K[0] + ix[0]

    def _chunk(self, nc):
        return max(1 << 18, (1 << 25) // nc)

    def gather(self, g):
        """[K3 K2 K1, nc] -> [nnz, nc]"""
        out = torch.zeros((self.nnz, g.shape[1]), dtype=g.dtype, device=DEV)
        step = self._chunk(g.shape[1])
        for lo in range(0, self.nnz, step):
            for w, i in self._taps(lo, lo + step):
                out[lo:lo + step] += w[:, None] * g[i]
        return out

    def spread(self, k):
        """[nnz, nc] -> [K3 K2 K1, nc]"""
        real = torch.view_as_real(k).flatten(1) if k.is_complex() else k
        g = torch.zeros((self.K[0] * self.K[1] * self.K[2], real.shape[1]), dtype=torch.float64, device=DEV)
        step = self._chunk(k.shape[1])
        for lo in range(0, self.nnz, step):
            for w, i in self._taps(lo, lo + step):
                g.index_add_(0, i, w[:, None] * real[lo:lo + step])
        return torch.view_as_complex(g.reshape(g.shape[0], -1, 2)) if k.is_complex() else g

    def forward(self, x, scatter=True):
        """(nc, n3, n2, n1) -> [nnz, nc]"""
        x = x.to(torch.complex128) * self.U
        pad = []
        for a in range(3):
            pad += [(self.K[a] - self.n[a]) // 2] * 2
        x = torch.fft.fftn(torch.fft.fftshift(torch.nn.functional.pad(x, pad), dim=(1, 2, 3)), dim=(1, 2, 3))
        return self.gather(x.reshape(x.shape[0], -1).T.contiguous()) / math.sqrt(self.nnz)

    def adjoint(self, k):
        """[nnz, nc] -> (nc, n3, n2, n1)"""
        g = self.spread(k.to(torch.complex128)).T.reshape(k.shape[1], self.K[2], self.K[1], self.K[0])
        g = torch.fft.ifftshift(torch.fft.ifftn(g, dim=(1, 2, 3), norm="forward"), dim=(1, 2, 3))
        lo = [(self.K[a] - self.n[a]) // 2 for a in range(3)]
        g = g[:, lo[2]:self.K[2] - lo[2], lo[1]:self.K[1] - lo[1], lo[0]:self.K[0] - lo[0]]
        return g * self.U / math.sqrt(self.nnz)

    def normal(self, x, damp):
        return self.adjoint(self.d[:, None] * self.forward(x)) + damp ** 2 * x

    def solve(self, raw, iters, damp, solver):
        b = self.adjoint(self.d[:, None] * raw.T[self.keep].to(torch.complex128))
        dot = lambda p, q: (p.conj() * q).sum(dim=(1, 2, 3)).real.reshape(-1, 1, 1, 1)  # noqa: E731
        x = torch.zeros_like(b)
        if solver == "cg":
            r, p, rr = b, b, dot(b, b)
            for _ in range(iters):
                q = self.normal(p, damp)
                step = rr / dot(p, q)
                x, r = x + step * p, r - step * q
                new = dot(r, r)
                p, rr = r + (new / rr) * p, new
            return x
        beta = dot(b, b).sqrt()  # MINRES (Paige and Saunders): Lanczos vectors, one rotation a step
        v, v_old, w1, w2 = b / beta, torch.zeros_like(b), torch.zeros_like(b), torch.zeros_like(b)
        cs, sn, dbar, eps, phibar = -torch.ones_like(beta), *(torch.zeros_like(beta) for _ in range(3)), beta
        for _ in range(iters):
            p = self.normal(v, damp) - beta * v_old
            a = dot(v, p)
            p = p - a * v
            beta = dot(p, p).sqrt()
            old, delta, gbar = eps, cs * dbar + sn * a, sn * dbar - cs * a
            eps, dbar = sn * beta, -cs * beta
            gamma = torch.sqrt(gbar ** 2 + beta ** 2)
            cs, sn = gbar / gamma, beta / gamma
            phi, phibar = cs * phibar, sn * phibar
            w = (v - old * w1 - delta * w2) / gamma
            x = x + phi * w
            w1, w2, v_old, v = w2, w, v, p / beta
        return x


def exact(case, seed):
    outs, cost = [], 0.0
    for n, traj, nr, ns, nc in _parts(case):
        passes = {"normal": 2}.get(case["op"], 2 * case["iters"] + 1 if case["iters"] else 1)
        cost += (case["J"] + 1) ** (3 if n[2] > 1 else 2) * float(nr) * ns * (nc + 4) * passes
    if cost > 4e11:
        return None
    for v, (n, traj, nr, ns, nc) in enumerate(_parts(case)):
        om = _trajectory(traj, n, nr, ns, seed + v)
        plain = _Plain(om, n, case, _analytic_d(om) if case["given_d"] else None)
        if case["op"] in ("adjoint", "solve", "batch"):
            k = _samples(om, n, nc, seed + v)
            if case["op"] == "adjoint":
                outs.append(plain.adjoint(k.T[plain.keep]))
            else:
                outs.append(plain.solve(k, case["iters"], 1e-3, case["solver"]))
            continue
        x = _image(n, nc, seed + v)
        if case["op"] == "normal":
            outs.append(plain.normal(x.to(torch.complex128), 0.1))
            continue
        k = torch.zeros((nc, plain.M), dtype=torch.complex128, device=DEV)
        k[:, plain.keep] = plain.forward(x).T
        outs.append(k if case["op"] == "forward" else np.ascontiguousarray(k.T.cpu().numpy()))
    return outs if case["op"] == "batch" else outs[0]
