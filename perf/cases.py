"""Performance cases of the table NUFFT and of the solvers on top of it.

A case is one call sequence of a user's program on the GPU: ``prepare`` makes
what the program holds (plan, images, data, weights), ``run`` is one pass
through the public entry points, ``work`` the bytes and operations that a pass
cannot do without, and ``exact`` the same outputs in 64 bits by plain torch.

Kinds
  nufft    a NufftPlan's forward and adjoint (min-max:KB tables), 2D or 3D
  newfft   the same through newfft's default: real KB tables, 1st order
  dcf      Pipe-Menon density compensation of a batch of trajectories
  learned  learned density compensation: features and regressor
  sense    CG-SENSE (qpwls_pcg1), a NUFFT pair or the Toeplitz Gram operator per
           iteration
  grad     loss and gradient of the density-compensation regressor

Trajectories are golden-angle radial (2D) and kooshball (3D).  Images are sums
of Gaussian blobs seen by coils; k-space data are the blobs' Fourier transforms
at the sample locations plus noise, so that they have the large dynamic range
of measured data (a strong centre and a noise floor).
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

import mirt_b200 as mb
from mirt_b200 import sense as mbs

DEV = "cuda"
BLOBS = 16


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _nufft(kind, n, k, coils, slices, spokes, readout, j=6):
    """A NUFFT case: image n, grid k (1st dimension first), `spokes` a range."""
    n3, k3 = (n[2], k[2]) if len(n) == 3 else (0, 0)
    return dict(kind=kind, n1=n[0], n2=n[1], n3=n3, k1=k[0], k2=k[1], k3=k3, j=j, coils=coils,
                slices=slices, spokes_lo=spokes[0], spokes_hi=spokes[1], readout=readout)


def _sense(n, k, coils, problems, spokes, readout, niter, gram):
    return dict(kind="sense", n1=n[0], n2=n[1], k1=k[0], k2=k[1], j=6, coils=coils,
                slices=problems, spokes_lo=spokes, spokes_hi=spokes, readout=readout, niter=niter,
                gram=gram)


def listed():
    return [
        # one small image, one coil: the benchmark's smallest configuration (a
        # phantom, a unit test, one dynamic frame); launches and latency
        dict(name="image_64", **_nufft("nufft", (64, 64), (128, 128), 1, 1, (64, 64), 128)),
        # one image of odd, unequal extents through newfft with its defaults
        # (real tables, linear table interpolation, K = 2 N: no power of two)
        dict(name="image_odd", **_nufft("newfft", (201, 175), (402, 350), 1, 1, (157, 157), 402)),
        # one fully sampled multicoil slice with the scanner's usual 16 channels
        # at N = 192 (K = 384), the plan's default launch shapes
        dict(name="coils_16", **_nufft("nufft", (192, 192), (384, 384), 16, 1, (302, 302), 384)),
        # the benchmark's batch: 64 uneven slices of 32 coils
        dict(name="batch_32", **_nufft("nufft", (256, 256), (512, 512), 32, 64, (100, 400), 512)),
        # a 3D kooshball of 8 coils (the benchmark's 3D configuration)
        dict(name="koosh_8", **_nufft("nufft", (128, 128, 128), (256, 256, 256), 8, 1,
                                      (16384, 16384), 256)),
        # one 3D volume with one column, as the reference's 3D gateways take it
        dict(name="volume_1", **_nufft("nufft", (72, 60, 48), (144, 120, 96), 1, 1, (1500, 1500),
                                       144)),
        # density compensation of uneven trajectories in one batch, 30 updates
        # (the targets of the learned regressor, and a user's weights)
        dict(name="dcf_pipe", kind="dcf", n1=256, n2=256, k1=512, k2=512, j=6, slices=6,
             spokes_lo=64, spokes_hi=256, readout=512, niter=29),
        # the learned weights of a batch of undersampled trajectories (R = 4)
        dict(name="dcf_learned", kind="learned", n1=256, n2=256, k1=512, k2=512, slices=8,
             spokes_lo=101, spokes_hi=101, readout=512),
        # CG-SENSE at R = 4: 24 coils at N = 192 with the NUFFT pair, 16 coils
        # at N = 256 on the Toeplitz normal equations; the iterations between
        # two looks at the image (few, so that the iterates of one operator in
        # other roundings stay comparable)
        dict(name="sense_nufft", **_sense((192, 192), (384, 384), 24, 5, 76, 384, 4, False)),
        dict(name="sense_gram", **_sense((256, 256), (512, 512), 16, 6, 101, 512, 4, True)),
        # one gradient of the regressor over a training set's rows (backward)
        dict(name="mlp_grad", kind="grad", rows=65536),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _extent(rng, n):
    """n, or now and then another extent near it (rectangular, odd images)."""
    return n if rng.random() < 0.6 else max(8, int(n * rng.uniform(0.75, 1.1)))


def draw(rng):
    kind = rng.choice(["nufft2", "nufft2", "nufft2", "nufft3", "nufft3", "newfft", "dcf", "learned",
                       "sense", "sense", "grad"])
    if kind in ("nufft2", "newfft"):
        n0 = rng.choice([64, 128, 192, 256]) if rng.random() < 0.5 else _log_int(rng, 40, 288)
        n = (n0, _extent(rng, n0))
        over = 2.0 if rng.random() < 0.85 else 1.5
        k = tuple(int(math.ceil(over * v)) for v in n)
        coils = rng.choice([1, 1, 1, 2, 4, 6, 8, 8, 12, 16, 20, 24, 32, 32, 48])
        readout = 2 * n0 - rng.choice([0, 0, 1])
        spokes = _log_int(rng, 24, 1.6 * n0)
        slices = min(_log_int(rng, 1, 16), max(1, int(6e7 / (spokes * readout * coils))))
        return _nufft("nufft" if kind == "nufft2" else "newfft", n, k, coils, slices,
                      (max(8, spokes // 2) if slices > 1 else spokes, spokes), readout,
                      j=rng.choice([6, 6, 6, 6, 5, 4, 7]))
    if kind == "nufft3":
        n0 = rng.choice([32, 64, 96]) if rng.random() < 0.4 else _log_int(rng, 24, 96)
        n = (n0, _extent(rng, n0), _extent(rng, n0))
        k = tuple(2 * v for v in n)
        coils = rng.choice([1, 1, 1, 2, 4, 8, 8, 12, 16])
        spokes = min(_log_int(rng, 200, 6000), int(4e6 / (2 * n0 * coils)))
        return _nufft("nufft", n, k, coils, 1, (spokes, spokes), 2 * n0,
                      j=rng.choice([6, 6, 6, 5, 4]))
    if kind in ("dcf", "learned"):
        n0 = rng.choice([128, 192, 256])
        hi = _log_int(rng, 48, 320)
        c = dict(kind=kind, n1=n0, n2=n0, k1=2 * n0, k2=2 * n0, slices=rng.randint(1, 8),
                 spokes_lo=max(24, hi // 3), spokes_hi=hi, readout=2 * n0 - rng.choice([0, 1]))
        if kind == "dcf":
            c.update(j=6, niter=rng.choice([9, 19, 29]))
        else:
            # the shipped regressor is trained for the 256 / 512 grid
            c.update(n1=256, n2=256, k1=512, k2=512)
        return c
    if kind == "sense":
        n0 = rng.choice([128, 192, 256]) if rng.random() < 0.6 else rng.randint(96, 256)
        n = (n0, n0)
        return _sense(n, (2 * n0, 2 * n0), rng.choice([4, 8, 12, 16, 24, 32]), rng.randint(1, 6),
                      int(math.ceil(math.pi * n0 / 2 / rng.choice([2, 3, 4]))), 2 * n0,
                      rng.randint(2, 4), rng.random() < 0.5)
    return dict(kind="grad", rows=_log_int(rng, 2048, 262144))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _dims(case):
    n = [case["n1"], case["n2"]] + ([case["n3"]] if case.get("n3") else [])
    k = [case["k1"], case["k2"]] + ([case["k3"]] if case.get("k3") else [])
    return n, k


def _trajectory(case, seed):
    """(om [M, D] radians FP64, slice offsets): golden-angle radial slices of
    uneven length, or one kooshball with a random rotation about its axis."""
    rng = np.random.default_rng([seed, 11])
    nro = case["readout"]
    rho = (np.arange(nro) - (nro // 2 - 1)) / nro * 2 * np.pi
    if case.get("n3"):
        ns = case["spokes_lo"]
        z = 1 - 2 * (np.arange(ns) + 0.5) / ns
        r = np.sqrt(1 - z * z)
        th = np.pi * (1 + np.sqrt(5)) * (np.arange(ns) + 0.5) + rng.uniform(0, 2 * np.pi)
        d = np.stack([r * np.cos(th), r * np.sin(th), z], 1)
        return (d[:, None, :] * rho[None, :, None]).reshape(-1, 3), np.array([0, ns * nro])
    # every seed has the same (uneven) slice sizes: spokes_lo .. spokes_hi, shuffled
    spokes = np.linspace(case["spokes_lo"], case["spokes_hi"], case["slices"]).astype(int)
    spokes = spokes[np.random.default_rng(case["slices"]).permutation(case["slices"])]
    oms = []
    for s in spokes:
        a = np.arange(s) * np.pi * (np.sqrt(5) - 1) / 2 + rng.uniform(0, np.pi)
        oms.append(np.stack([np.outer(np.cos(a), rho).ravel(), np.outer(np.sin(a), rho).ravel()], 1))
    return np.concatenate(oms), np.concatenate([[0], np.cumsum(spokes * nro)]).astype(np.int64)


class _Scene:
    """Gaussian blobs of one slice: centres and widths in pixels, amplitudes,
    and each coil's (complex) sensitivity at each blob."""

    def __init__(self, case, seed, s):
        n, _ = _dims(case)
        rng = np.random.default_rng([seed, 23, s])
        self.n = n
        self.centre = np.stack([rng.uniform(0.25, 0.75, BLOBS) * m for m in n], 1)
        self.width = rng.uniform(0.01, 0.08, BLOBS) * min(n)
        amp = rng.uniform(0.2, 1, BLOBS) * np.exp(1j * rng.uniform(-np.pi, np.pi, BLOBS))
        coils = case.get("coils", 1)
        u = (self.centre / n - 0.5) * 2
        ang = 2 * np.pi * np.arange(coils) / coils
        d2 = (u[:, :1] - 1.2 * np.cos(ang)) ** 2 + (u[:, 1:2] - 1.2 * np.sin(ang)) ** 2
        self.amp = amp[:, None] * np.exp(-d2 / 2 + 1j * ang)           # [blob, coil]

    def image(self):
        """[.., N2, N1, C] complex64 on the GPU."""
        g = [torch.exp(-(torch.arange(m, device=DEV)[None, :] - _dev(self.centre[:, d:d + 1])) ** 2
                       / (2 * _dev(self.width[:, None] ** 2))).float()
             for d, m in enumerate(self.n)]
        a = _dev(self.amp).to(torch.complex64)
        p = g[1][:, :, None] * g[0][:, None, :]
        if len(g) == 3:
            p = g[2][:, :, None, None] * p[:, None]
        flat = p.reshape(BLOBS, -1).t().to(torch.complex64)
        return (flat @ a).reshape(*self.n[::-1], -1)

    def data(self, om):
        """The blobs' Fourier transform at om (FP64, on the GPU): [M, C]."""
        e = torch.zeros(om.shape[0], BLOBS, dtype=torch.complex128, device=DEV)
        w2 = _dev(self.width ** 2)
        shift = _dev(self.centre - np.array(self.n) / 2)
        e.imag = -(om @ shift.t())
        e.real = -(om * om).sum(1)[:, None] * w2[None, :] / 2
        vol = (2 * np.pi * self.width ** 2) ** (len(self.n) / 2)
        return torch.exp(e) @ _dev(self.amp * vol[:, None])


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def _noise(shape, seed, scale):
    g = torch.Generator(device=DEV).manual_seed(1000003 * seed + 7)
    return scale * torch.randn(shape, dtype=torch.complex64, device=DEV, generator=g)


def _images(case, seed):
    x = torch.stack([_Scene(case, seed, s).image() for s in range(case["slices"])])
    return (x + _noise(x.shape, seed, 0.01)).contiguous()


def _samples(case, seed, om, moff):
    y = torch.empty(om.shape[0], case["coils"], dtype=torch.complex64, device=DEV)
    for s in range(case["slices"]):
        o = _dev(om[moff[s]:moff[s + 1]])
        y[moff[s]:moff[s + 1]] = _Scene(case, seed, s).data(o).to(torch.complex64)
    scale = float(y.abs().pow(2).mean().sqrt())
    return (y + _noise(y.shape, seed + 1, 0.03 * scale)).contiguous()


def _coil_maps(case, seed):
    """[S, N2, N1, C] complex64 smooth Gaussian-bump sensitivities."""
    n1, n2, C, S = case["n1"], case["n2"], case["coils"], case["slices"]
    rng = np.random.default_rng([seed, 31])
    u1 = torch.linspace(-1, 1, n1, device=DEV)[None, :, None]
    u2 = torch.linspace(-1, 1, n2, device=DEV)[:, None, None]
    out = torch.empty(S, n2, n1, C, dtype=torch.complex64, device=DEV)
    ang = 2 * np.pi * np.arange(C) / C
    for s in range(S):
        w = _dev(rng.uniform(0.6, 1.2, C)).float()
        ph = _dev(rng.uniform(-np.pi, np.pi, C)).float() + 0.5 * u1 * _dev(rng.uniform(-1, 1, C)).float()
        d2 = (u1 - _dev(1.2 * np.cos(ang)).float()) ** 2 + (u2 - _dev(1.2 * np.sin(ang)).float()) ** 2
        out[s] = torch.polar(torch.exp(-d2 / (2 * w ** 2)), ph.expand(n2, n1, C).contiguous())
    return out


def _beta(moff, sens):
    """The Reg1 weights: 2^-8 times the mean diagonal of A'A per problem."""
    p = (sens.abs() ** 2).sum(-1).double().flatten(1).mean(1).cpu().numpy()
    return 2.0 ** -8 * np.diff(moff) * p


def _rows(case, seed):
    """Regressor rows: radius, angle, log1p neighbour counts; standardised targets."""
    rng = np.random.default_rng([seed, 41])
    n = case["rows"]
    x = np.empty((n, 18), np.float32)
    x[:, 0] = rng.uniform(0, 1, n)
    x[:, 1] = rng.uniform(-1, 1, n)
    dens = 2.0 / (0.05 + x[:, :1])
    x[:, 2:] = np.log1p(rng.poisson(dens * (0.2 + 0.1 * np.arange(16))))
    y = (np.log(0.02 + x[:, 0]) + 0.1 * rng.standard_normal(n)).astype(np.float32)
    return x, (y - y.mean()) / y.std()


def _mlp_params(seed):
    """He-uniform weights and small biases of the 18-64-64-64-1 regressor."""
    rng = np.random.default_rng([seed, 43])
    parts = []
    for fi, fo in ((18, 64), (64, 64), (64, 64), (64, 1)):
        lim = math.sqrt(6.0 / fi)
        parts += [rng.uniform(-lim, lim, fo * fi), rng.uniform(-0.1, 0.1, fo)]
    return np.concatenate(parts).astype(np.float32)


# ---------------------------------------------------------------------------
# what a program holds, and one pass
# ---------------------------------------------------------------------------
def _plan(case, om, moff, coils):
    n, k = _dims(case)
    shift = [v / 2 for v in n]
    mo = moff if case["slices"] > 1 else None
    if case["kind"] == "newfft":
        return mb.newfft(om, n, Jd=[case["j"]] * len(n), Kd=k, n_shift=shift, ncol=coils,
                         slice_moff=mo)
    return mb.NufftPlan(om, n, [case["j"]] * len(n), k, n_shift=shift, Ld=1024, ncol=coils,
                        slice_moff=mo)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "grad":
        x, y = _rows(case, seed)
        return dict(kind=kind, x=_dev(x), y=_dev(y), mlp=mb.DcfMLP(params=_mlp_params(seed)))
    om, moff = _trajectory(case, seed)
    if kind in ("nufft", "newfft"):
        return dict(kind=kind, G=_plan(case, om, moff, case["coils"]), x=_images(case, seed),
                    y=_samples(case, seed, om, moff))
    if kind == "dcf":
        return dict(kind=kind, G=_plan(case, om, moff, 1), niter=case["niter"])
    if kind == "learned":
        return dict(kind=kind, om=_dev(om), moff=moff, model=mb.LearnedDCF.pretrained())
    sens = _coil_maps(case, seed)
    A = mbs.SenseSystem(_plan(case, om, moff, case["coils"]), sens, _beta(moff, sens))
    if case["gram"]:
        A.toeplitz()
    return dict(kind=kind, A=A, y=_samples(case, seed, om, moff), niter=case["niter"],
                gram=case["gram"])


def run(state):
    kind = state["kind"]
    if kind in ("nufft", "newfft"):
        return state["G"].forward(state["x"]), state["G"].adjoint(state["y"])
    if kind == "dcf":
        # FP32 weights, as the solvers' data weights take them
        return mb.dcf_pipe(state["G"], niter=state["niter"], thresh=0.0).to(torch.float32)
    if kind == "learned":
        return state["model"].predict(state["om"], slice_moff=state["moff"]).to(torch.float32)
    if kind == "sense":
        x = torch.zeros(state["A"].image_shape, dtype=torch.complex64, device=DEV)
        state["A"].pcg(x, state["y"], state["niter"], gram=state["gram"])
        return x
    return state["mlp"].grad(state["x"], state["y"])


def _mean_samples(case):
    return 0.5 * (case["spokes_lo"] + case["spokes_hi"]) * case["readout"] * case["slices"]


def work(case):
    """Inputs read once and outputs written once; the taps' multiply-adds (the
    innermost dimension's complex ones, 8 flops per tap and column, outer
    dimensions' partial sums included) and 5 K log2 K per FFT."""
    kind = case["kind"]
    if kind == "grad":
        n = case["rows"]
        p = 18 * 64 + 2 * 64 * 64 + 64
        return dict(bytes=4.0 * (19 * n + 2 * 9601), flops=n * (6.0 * p - 2 * 18 * 64))
    M = _mean_samples(case)
    if kind == "learned":
        return dict(bytes=M * (16 + 4), flops=M * 2.0 * (18 * 64 + 2 * 64 * 64 + 64))
    n, k = _dims(case)
    D, S, C = len(n), case["slices"], case.get("coils", 1)
    npix, ngrid = float(np.prod(n)), float(np.prod(k))
    j = case["j"]
    taps = M * C * 8.0 * sum(j ** d for d in range(1, D + 1))
    fft = 5.0 * S * C * ngrid * math.log2(ngrid)
    if kind in ("nufft", "newfft"):
        return dict(bytes=2 * (8 * S * C * npix + 8 * C * M + 8 * D * M), flops=2 * (taps + fft))
    if kind == "dcf":
        return dict(bytes=8 * D * M + 4 * M, flops=2 * (case["niter"] + 1) * taps)
    once = 8 * S * C * npix + 8 * C * M + 8 * S * npix
    gfft = 10.0 * S * C * 4 * npix * math.log2(4 * npix)
    it = case["niter"]
    return dict(bytes=once, flops=it * gfft if case["gram"] else 2 * it * (taps + fft))


# ---------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------
# nufft/param-data/kaiser,m=0.mat: the optimised KB shape per unit J for K/N = 2
_KB_ZN = {4: 2.31, 5: 2.34, 6: 2.32, 7: 2.32}


def _kb_ft(u, J, alpha):
    """Fourier transform of the KB kernel of order 0 (nufft/kaiser_bessel_ft.m)."""
    z = np.sqrt((np.pi * J * u) ** 2 - alpha ** 2 + 0j)
    return (J * np.sin(z) / z).real / np.i0(alpha)


def _minmax_kb(N, J, K, L):
    """Table (nufft/nufft_table_init.m) and 1D scaling factors of 'minmax:kb'."""
    alpha = float("%g" % (_KB_ZN[J] * J if K == 2 * N else 2.34 * J))
    nl = np.arange(N) - (N - 1) / 2
    gam = 2 * np.pi / K
    nc = 13 if N > 40 else -(-N // 3)
    X = np.cos(gam * nl[:, None] * np.arange(nc + 1)[None, :])
    c = np.linalg.lstsq(X, 1.0 / _kb_ft(nl / K, J, alpha), rcond=None)[0]
    al = np.concatenate([c[:1], c[1:] / 2])
    ls = np.arange(-nc, nc + 1)
    a = al[np.abs(ls)]
    sn = (a[None, :] * np.exp(1j * gam * nl[:, None] * ls[None, :])).sum(1)
    jj = np.arange(1, J + 1)
    diric = lambda t: np.sinc(t * N / K)                            # noqa: E731
    arg4 = (jj[None, :, None, None] - jj[:, None, None, None] + ls[None, None, :, None]
            - ls[None, None, None, :])
    T = np.linalg.inv((a[:, None] * a[None, :] * diric(arg4)).sum((2, 3)))
    arg = -jj[:, None] + (J / 2 + np.arange(L) / L)[None, :]
    r = (a[:, None, None] * diric(arg[None] + ls[:, None, None])).sum(0)
    p = np.conj(np.exp(1j * gam * (N - 1) / 2 * arg) * (T @ r))
    return np.concatenate([p[::-1].ravel(), [0]]), np.conj(sn)


def _kb_real(N, J, K, L):
    """Table and 1D scaling factors of newfft's 'kb:minmax' (nufft/newfft.m)."""
    alpha = 2.34 * J
    t = (np.arange(J * L + 1) - J * L / 2) / L
    f = np.sqrt(np.maximum(0, 1 - (2 * t / J) ** 2))
    a = float("%g" % alpha)
    h = np.where(np.abs(t) < J / 2, np.i0(a * f) / np.i0(a), 0)
    return h.astype(complex), 1.0 / _kb_ft((np.arange(N) - N // 2) / K, J, alpha) + 0j


class _Nufft64:
    """The table NUFFT of one slice in complex128 (nufft/nufft.m, nufft_adj.m)."""

    def __init__(self, n, k, j, om, shift, newfft=False):
        self.n, self.k, self.j, self.D = n, k, j, len(n)
        self.order, L = (1, 512) if newfft else (0, 1024)
        self.L = L
        make = _kb_real if newfft else _minmax_kb
        tabs = [make(n[d], j, k[d], L) for d in range(self.D)]
        self.h = [_dev(t[0]) for t in tabs]
        sn = np.ones(1)
        for t in tabs:
            sn = np.outer(t[1], sn.ravel()).reshape(len(t[1]), *np.shape(sn))  # last dimension first
        self.sn = _dev(sn.reshape(n[::-1]).astype(complex))[..., None]
        self.pb = None
        if newfft:
            shift = [shift[d] - n[d] // 2 for d in range(self.D)]
            pb = torch.ones((), dtype=torch.complex128, device=DEV)
            for d in range(self.D):
                a = 2 * np.pi * (np.arange(k[d]) * (n[d] // 2) % k[d]) / k[d]
                pb = _dev(np.exp(1j * a)).reshape([-1] + [1] * d) * pb
            self.pb = pb[..., None]
        self.om = _dev(om)
        ph = self.om @ torch.tensor(shift, dtype=torch.float64, device=DEV)
        self.phase = torch.polar(torch.ones_like(ph), ph)[:, None]

    def _taps(self, m0, m1):
        """Per dimension: grid indices [m, J] and coefficients [m, J]."""
        out = []
        for d in range(self.D):
            gam = torch.tensor(2 * np.pi / self.k[d], dtype=torch.float64, device=DEV)
            t = self.om[m0:m1, d] / gam
            kk = (1 + torch.floor(t - self.j / 2))[:, None] + torch.arange(self.j, device=DEV)
            p = (t[:, None] - kk) * self.L
            h, nc = self.h[d], self.j * self.L // 2
            if self.order == 0:
                w = h[(nc + torch.floor(p + 0.5)).long().clamp(0, len(h) - 1)]
            else:
                f = torch.floor(p)
                i = (nc + f).long()
                w = (1 - (p - f)) * h[i] + (p - f) * h[(i + 1).clamp(max=len(h) - 1)]
            out.append((kk.long() % self.k[d], w))
        return out

    def _each(self, chunk=1 << 19):
        """(samples, flat grid index, coefficient) of every tap."""
        M = self.om.shape[0]
        for m0 in range(0, M, chunk):
            m1 = min(M, m0 + chunk)
            taps = self._taps(m0, m1)
            sel = [()]
            for _ in range(self.D):
                sel = [(*s, q) for s in sel for q in range(self.j)]
            for q in sel:
                idx, w = 0, 1.0
                for d in reversed(range(self.D)):
                    idx = idx * self.k[d] + taps[d][0][:, q[d]]
                    w = w * taps[d][1][:, q[d]]
                yield slice(m0, m1), idx, w[:, None]

    def gather(self, ck):
        """[prod K, C] -> [M, C]"""
        out = torch.zeros(self.om.shape[0], ck.shape[1], dtype=torch.complex128, device=DEV)
        for s, idx, w in self._each():
            out[s] += w * ck[idx]
        return out * self.phase

    def spread(self, y):
        """[M, C] -> [prod K, C]"""
        y = y * self.phase.conj()
        g = torch.zeros(int(np.prod(self.k)), y.shape[1], 2, dtype=torch.float64, device=DEV)
        for s, idx, w in self._each():
            g.index_add_(0, idx, torch.view_as_real(w.conj() * y[s]))
        return torch.view_as_complex(g)

    def forward(self, x):
        dims = list(range(self.D))
        g = torch.fft.fftn(x.to(torch.complex128) * self.sn, s=self.k[::-1], dim=dims)
        return self.gather((g if self.pb is None else g * self.pb).reshape(-1, x.shape[-1]))

    def adjoint(self, y):
        g = self.spread(y.to(torch.complex128)).reshape(*self.k[::-1], y.shape[1])
        if self.pb is not None:
            g = g * self.pb.conj()
        x = torch.fft.ifftn(g, dim=list(range(self.D)), norm="forward")
        return x[tuple(slice(0, v) for v in self.n[::-1])] * self.sn.conj()


def _exact_dcf(case, om, moff):
    n, k = _dims(case)
    out = []
    for s in range(case["slices"]):
        G = _Nufft64(n, k, case["j"], om[moff[s]:moff[s + 1]], [v / 2 for v in n])
        w = torch.ones(G.om.shape[0], dtype=torch.float64, device=DEV)
        for _ in range(case["niter"] + 1):
            w = w / G.gather(G.spread(w[:, None].to(torch.complex128)))[:, 0].real
        psf = G.adjoint(w[:, None].to(torch.complex128)).real.sum()
        out.append(w * (float(np.prod(n)) / psf))
    return torch.cat(out)


def _exact_learned(case, om, moff):
    path = os.path.join(os.path.dirname(mb.__file__), "data", "learned_dcf_n256_k512.npz")
    z = np.load(path)
    feats = []
    for s in range(case["slices"]):
        o = _dev(om[moff[s]:moff[s + 1]])
        t = o * torch.tensor(512 / (2 * np.pi), dtype=torch.float64, device=DEV)
        M = len(o)
        f = torch.empty(M, 18, dtype=torch.float64, device=DEV)
        f[:, 0] = o.square().sum(1).sqrt() / np.pi
        f[:, 1] = torch.atan2(o[:, 1], o[:, 0]) / np.pi
        step = max(1, int(1.5e8 // M))
        for m in range(0, M, step):
            d2 = (t[None, :, 0] - t[m:m + step, None, 0]).square_()
            d2 += (t[None, :, 1] - t[m:m + step, None, 1]).square_()
            cum = [(d2 < (e / 8) ** 2).sum(1) for e in range(17)]
            cum[0] += 1                          # the sample itself is not counted
            for b in range(16):
                f[m:m + step, 2 + b] = torch.log1p((cum[b + 1] - cum[b]).double())
        feats.append(f)
    out = _mlp64(_dev(z["params"]), torch.cat(feats))
    return torch.exp(float(z["sigma"]) * out + float(z["mu"]))


def _mlp64(params, x):
    """The regressor in FP64 at the BF16 rounding of its parameters."""
    p = params.to(torch.bfloat16).double() if not params.requires_grad else params
    at = 0
    for li, (fi, fo) in enumerate(((18, 64), (64, 64), (64, 64), (64, 1))):
        W = p[at:at + fi * fo].reshape(fo, fi)
        b = p[at + fi * fo:at + fi * fo + fo]
        at += fi * fo + fo
        x = x @ W.t() + b
        if li < 3:
            x = torch.relu(x)
    return x[:, 0]


def _exact_grad(case, seed):
    x, y = _rows(case, seed)
    p = _dev(_mlp_params(seed)).to(torch.bfloat16).double().requires_grad_(True)
    loss = (_mlp64(p, _dev(x).double()) - _dev(y).double()).square().mean()
    loss.backward()
    return float(loss.detach()), p.grad.detach()


def _reg64(x, beta):
    """C'C x of the first-order differences at [1 nx nx+1 nx-1] (penalty/Reg1.m)."""
    out = torch.zeros_like(x)
    n1 = x.shape[1]
    for d1, d2, w in ((1, 0, 1.0), (0, 1, 1.0), (1, 1, 2 ** -0.5), (-1, 1, 2 ** -0.5)):
        a, b = max(d1, 0), n1 + min(d1, 0)
        d = w * beta * (x[d2:, a:b] - x[:x.shape[0] - d2, a - d1:b - d1])
        out[d2:, a:b] += d
        out[:x.shape[0] - d2, a - d1:b - d1] -= d
    return out


def _gram64(n, k, j, om):
    """Spectrum [2 N2, 2 N1] of the Hermitian circulant embedding of G'G
    (systems/Gnufft_gram.m)."""
    n1, n2 = n
    one = torch.ones(len(om), 1, dtype=torch.complex128, device=DEV)
    b1, b2 = (_Nufft64(n, k, j, o, [0, 0]).adjoint(one)[..., 0] for o in (om, om * [-1, 1]))
    c = torch.zeros(2 * n2, 2 * n1, dtype=torch.complex128, device=DEV)
    c[:n2, :n1] = b1
    c[:n2, n1 + 1:] = b2[:, 1:].flip(1)
    c[n2 + 1:, 0] = b1[1:, 0].conj().flip(0)
    c[n2 + 1:, 1:n1] = b2[1:, 1:].conj().flip(0)
    c[n2 + 1:, n1 + 1:] = b1[1:, 1:].conj().flip(0, 1)
    mirror = torch.roll(c.flip(0, 1), (1, 1), (0, 1)).conj()
    return torch.fft.fft2((c + mirror) / 2)


def _exact_sense(case, seed, om, moff):
    n, k = _dims(case)
    n1, n2 = n
    sens, y = _coil_maps(case, seed), _samples(case, seed, om, moff)
    beta = _beta(moff, sens)
    dot = lambda a, b: (a.conj() * b).real.sum()                      # noqa: E731
    out = []
    for s in range(case["slices"]):
        o = om[moff[s]:moff[s + 1]]
        G = _Nufft64(n, k, case["j"], o, [n1 / 2, n2 / 2])
        H = _gram64(n, k, case["j"], o)[..., None] if case["gram"] else None
        sm = sens[s].to(torch.complex128)
        ys = y[moff[s]:moff[s + 1]].to(torch.complex128)

        def T(v):
            f = torch.fft.fftn(sm * v[..., None], s=(2 * n2, 2 * n1), dim=(0, 1))
            return (sm.conj() * torch.fft.ifftn(H * f, dim=(0, 1))[:n2, :n1]).sum(-1)

        A = lambda v: G.forward(sm * v[..., None])                      # noqa: E731
        At = lambda v: (sm.conj() * G.adjoint(v)).sum(-1)               # noqa: E731
        x = torch.zeros(n2, n1, dtype=torch.complex128, device=DEV)
        rhs = At(ys) if case["gram"] else ys
        Ax, Rx = torch.zeros_like(rhs), torch.zeros_like(x)
        old, d = None, None
        for _ in range(case["niter"]):
            g = rhs - Ax - Rx if case["gram"] else At(rhs - Ax) - Rx
            new = dot(g, g)
            d = g if d is None else g + (new / old) * d
            old = new
            Ad, Rd = (T if case["gram"] else A)(d), _reg64(d, beta[s])
            cur = dot(d, Ad) if case["gram"] else dot(Ad, Ad)
            step = dot(d, g) / (cur + dot(d, Rd))
            x, Ax, Rx = x + step * d, Ax + step * Ad, Rx + step * Rd
        out.append(x)
    return torch.stack(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "grad":
        return _exact_grad(case, seed)
    om, moff = _trajectory(case, seed)
    if kind == "dcf":
        return _exact_dcf(case, om, moff)
    if kind == "learned":
        return _exact_learned(case, om, moff)
    if kind == "sense":
        return _exact_sense(case, seed, om, moff)
    n, k = _dims(case)
    x, y = _images(case, seed), _samples(case, seed, om, moff)
    X = torch.empty(y.shape, dtype=torch.complex128, device=DEV)
    xa = torch.empty(x.shape, dtype=torch.complex128, device=DEV)
    for s in range(case["slices"]):
        m = slice(int(moff[s]), int(moff[s + 1]))
        G = _Nufft64(n, k, case["j"], om[m], [v / 2 for v in n], kind == "newfft")
        X[m] = G.forward(x[s])
        xa[s] = G.adjoint(y[m])
    return X, xa
