"""The framework's workloads, for timing it and for comparing two builds of it.

Every case goes through the public entry points on device tensors, as a
program that calls the framework does: the NUFFT's forward and adjoint, the
CG-SENSE solve (on a kept model, with the model's set-up, with and without
the Toeplitz operator, in 3D), a batch of uneven solves, one training pass of
the learned preconditioner and the ESPIRiT calibration. All data are
complex64 (the network's layers bfloat16), synthetic and made from the seed.

``exact`` computes the same results in float64 with plain torch: the
Kaiser-Bessel gridding (width 6, 2x oversampling, the 1001-entry table), the
Toeplitz PSF, the data scaling, CG and PCG, the network, the calibration.
"""

from __future__ import annotations

import math

import numpy as np
import torch

GOLDEN = (1.0 + math.sqrt(5.0)) / 2.0
WIDTH = 6.0
TABLE = 1000


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # one slice of a real-time or interactive scan: launches and latency are all of it
        _nufft("nufft2d_64_c1", 64, 64, 1, 1, 101, 128),
        # the 2D single-channel operator pair at the benchmark's size
        _nufft("nufft2d_256_c1", 256, 256, 1, 1, 402, 512),
        # a multi-channel slice of a rectangular, not power-of-two matrix, odd readout, density weights
        _nufft("nufft2d_200x180_c12_weights", 200, 180, 1, 12, 150, 399, weights=True),
        # the bit-reproducible gridding mode, odd channel count
        _nufft("nufft2d_160_c5_deterministic", 160, 160, 1, 5, 120, 320, deterministic=True),
        # the 3D kooshball at the benchmark's size: the operator pair of a volume
        _nufft("nufft3d_128_c8", 128, 128, 128, 8, 20000, 256),
        # the reference's solve (plain CG, its 30 iterations) of the next frame on a kept model
        _recon("recon2d_256_c16_cg30", 256, 256, 1, 16, 96, 512, iters=30),
        # one slice from nothing: model set-up with the PSF, the preconditioned solve, release
        _recon("recon2d_256_c16_pcg_setup", 256, 256, 1, 16, 96, 512, iters=12, precond=3, setup=True),
        # the solve without the Toeplitz operator: gridding in every iteration, not a power of two
        _recon("recon2d_192_c8_explicit", 192, 192, 1, 8, 64, 384, iters=5, toeplitz=False),
        # a small volume
        _recon("recon3d_64_c8_pcg", 64, 64, 64, 8, 6000, 128, iters=8, precond=3),
        # a stack of slices of uneven matrix, spoke and channel counts in one graph launch
        {"name": "batch2d_24", "kind": "batch", "stack": 1, "problems": 24, "iters": 20},
        # one gradient pass of the learned preconditioner on a problem's seven residuals
        {"name": "precnet_grad_256_n7", "kind": "train", "X": 256, "Y": 256, "n": 7},
        # coil maps of one slice
        {"name": "ecalib2d_256_c16", "kind": "ecalib", "X": 256, "Y": 256, "C": 16},
    ]


def _nufft(name, X, Y, Z, C, spokes, samples, weights=False, deterministic=False):
    c = {"kind": "nufft", "X": X, "Y": Y, "Z": Z, "C": C, "spokes": spokes, "samples": samples,
         "weights": weights, "deterministic": deterministic}
    return {"name": name, **c} if name else c


def _recon(name, X, Y, Z, C, spokes, samples, iters, precond=0, toeplitz=True, setup=False):
    c = {"kind": "recon", "X": X, "Y": Y, "Z": Z, "C": C, "spokes": spokes, "samples": samples, "iters": iters,
         "precond": precond, "toeplitz": toeplitz, "setup": setup}
    return {"name": name, **c} if name else c


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def even(lo, hi):
        return 2 * logint(lo // 2, hi // 2)

    kind = rng.choice(["nufft2d"] * 4 + ["nufft3d"] * 2 + ["recon2d"] * 4 + ["recon3d", "batch", "train", "ecalib"])

    if kind == "nufft2d":
        X = even(48, 320)
        Y = X if rng.random() < 0.5 else max(48, 2 * int(X * rng.uniform(0.3, 0.5)))
        opt = rng.random()
        return _nufft(None, X, Y, 1, logint(1, 32), logint(16, 402), int(X * rng.uniform(1.0, 2.0)),
                      weights=opt < 0.25, deterministic=opt > 0.85)
    if kind == "nufft3d":
        X = even(24, 128)
        return _nufft(None, X, X, X, logint(1, 8), logint(200, 20000), int(X * rng.uniform(1.0, 2.0)))
    if kind == "recon2d":
        X = even(64, 320)
        Y = X if rng.random() < 0.7 else max(64, 2 * int(X * rng.uniform(0.35, 0.5)))
        how = rng.choice(["cg", "cg", "pcg", "fcg", "explicit"])
        iters = {"cg": rng.randint(20, 30), "pcg": rng.randint(6, 12), "fcg": rng.randint(8, 17),
                 "explicit": rng.randint(2, 5)}[how]
        return _recon(None, X, Y, 1, rng.randint(4, 32), rng.randint(32, 160), 2 * X, iters,
                      precond={"pcg": 3, "fcg": 1}.get(how, 0), toeplitz=how != "explicit", setup=rng.random() < 0.4)
    if kind == "recon3d":
        X = even(32, 72)
        return _recon(None, X, X, X, rng.randint(2, 8), rng.randint(1500, 6000), 2 * X, rng.randint(4, 8), precond=3,
                      setup=rng.random() < 0.4)
    if kind == "batch":
        return {"kind": "batch", "stack": rng.randint(2, 10 ** 6), "problems": rng.randint(3, 20), "iters": 20}
    if kind == "train":
        X = even(64, 256)
        return {"kind": "train", "X": X, "Y": X if rng.random() < 0.5 else even(64, 256), "n": rng.randint(1, 7)}
    X = even(96, 256)
    return {"kind": "ecalib", "X": X, "Y": even(96, 256), "C": rng.randint(4, 16)}


# the solves' l2 regularisation (the operators' norms are some hundreds)
LAMBDA = 0.5


def _axes(case):
    return [n for n in (case["X"], case["Y"], case["Z"]) if n > 1]


def work(case):
    if case["kind"] == "batch":
        parts = [work(c) for c in _batch_list(case)]
        return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}
    if case["kind"] == "train":
        pix = case["X"] * case["Y"] * case["n"]
        macs = 9 * (2 * 32 + 4 * 32 * 32 + 32 * 2)      # per pixel, forward; backward twice that (no input gradient)
        return {"bytes": 2 * 8 * pix, "flops": 2.0 * pix * (3 * macs - 9 * 2 * 32)}
    if case["kind"] == "ecalib":
        pix, C = case["X"] * case["Y"], case["C"]
        return {"bytes": 8 * (24 * 24 * C + pix * C + pix), "flops": 8.0 * pix * C * C * 30}
    C, M, ax = case["C"], case["spokes"] * case["samples"], _axes(case)
    pix, grid = math.prod(ax), math.prod(2 * n for n in ax)
    fft, interp = 5.0 * grid * math.log2(grid) * C, 4.0 * 6 ** len(ax) * M * C
    if case["kind"] == "nufft":
        return {"bytes": 2 * 8 * C * (pix + M) + 2 * 24 * M, "flops": 2 * (fft + interp)}
    per = 2 * fft + (6.0 * grid * C if case["toeplitz"] else 2 * interp) + 16.0 * pix * C
    if case["precond"]:
        per += 2 * fft / C
    return {"bytes": 8 * C * (pix + M) + 24 * M + 8 * pix, "flops": fft + interp + case["iters"] * per}


def tolerance(case):
    """About four times what was seen against float64, or (solves) between two orders of the float32 sums."""
    if case["kind"] == "nufft":         # 1.9e-7 .. 3.2e-7, largest 1.8e-6
        return {"rel": 1.5e-6, "max": 1e-5}
    if case["kind"] == "train":         # bfloat16 layers: 4.2e-3 on the gradient
        return {"rel": 1.7e-2, "max": 0.9}
    if case["kind"] == "ecalib":        # 2e-6 .. 1.1e-5, largest 7e-4
        return {"rel": 1e-4, "max": 3e-3}
    if case["kind"] == "recon" and case["precond"]:     # 5e-5 .. 1e-4
        return {"rel": 4e-4, "max": 4e-3}
    if case["kind"] == "recon" and not case["toeplitz"]:        # at most 5 iterations: 2e-6 .. 1e-5
        return {"rel": 4e-5, "max": 4e-4}
    # plain CG loses the orthogonality of its directions: up to 2e-3 between two summation orders
    return {"rel": 8e-3, "max": 0.2}


# ---------------------------------------------------------------------------
# inputs. Arrays are column-major [X, Y, Z, C]: torch shapes [C, Z, Y, X].
# ---------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed), np.random.default_rng(seed)


def _gauss(gen, *shape):
    return torch.view_as_complex(torch.randn(*shape, 2, generator=gen, device="cuda"))


def _traj(case, rng):
    """Golden-angle radial (2D) or golden-means kooshball (3D) trajectory [M, 3] in cycles per FOV, started at a random
    spoke; complex64 as the entry points take it."""
    D, S, X, Y, Z = case["samples"], case["spokes"], case["X"], case["Y"], case["Z"]
    s = np.arange(S) + int(rng.integers(0, 1000))
    if Z == 1:
        a = s * (math.pi / GOLDEN)
        d = np.stack([X * np.cos(a), Y * np.sin(a), 0.0 * a], axis=1)
    else:
        z = 2.0 * np.mod(s * 0.465571231876768, 1.0) - 1.0
        a = 2.0 * math.pi * np.mod(s * 0.682327803828019, 1.0)
        rxy = np.sqrt(np.maximum(0.0, 1.0 - z * z))
        d = np.stack([X * rxy * np.cos(a), Y * rxy * np.sin(a), Z * z], axis=1)
    t = ((np.arange(D) + 0.5) / D - 0.5)[None, :, None] * d[:, None, :]
    return torch.from_numpy(t.reshape(-1, 3).astype(np.complex64)).cuda()


def _coords(case):
    n = (case["Z"], case["Y"], case["X"])
    return torch.meshgrid(*[torch.linspace(-1.0, 1.0, k, device="cuda", dtype=torch.float64) if k > 1
                            else torch.zeros(1, device="cuda", dtype=torch.float64) for k in n], indexing="ij")


def _maps(case, rng):
    """exp of random complex 2nd-order polynomials, unit root sum of squares over the channels [C, Z, Y, X]."""
    z, y, x = _coords(case)
    terms = torch.stack([torch.ones_like(x), x, y, z, x * x, x * y, y * y, x * z, y * z, z * z]).to(torch.complex128)
    c = torch.from_numpy((rng.standard_normal((case["C"], 10)) + 1j * rng.standard_normal((case["C"], 10))) * 0.5).cuda()
    s = torch.exp(torch.einsum("ct,tzyx->czyx", c, terms))
    return (s / torch.sqrt((s.abs() ** 2).sum(0))).to(torch.complex64)


def _phantom(case, rng):
    """Twenty random ellipses or ellipsoids of constant phase [Z, Y, X]."""
    q = _coords(case)
    img = torch.zeros_like(q[0], dtype=torch.complex64)
    for _ in range(20):
        ctr, rad = rng.uniform(-0.6, 0.6, 3), rng.uniform(0.04, 0.47, 3)
        a = rng.uniform(0.0, math.pi)
        dx, dy, dz = q[2] - ctr[0], q[1] - ctr[1], q[0] - (ctr[2] if case["Z"] > 1 else 0.0)
        u, v = dx * math.cos(a) + dy * math.sin(a), dy * math.cos(a) - dx * math.sin(a)
        inside = (u / rad[0]) ** 2 + (v / rad[1]) ** 2 + (dz / rad[2]) ** 2 <= 1.0
        img += inside * complex(rng.uniform(0.1, 1.0) * np.exp(2j * math.pi * rng.uniform()))
    return img


def _noisy(gen, y, snr_db=40.0):
    sigma = torch.sqrt((y.abs() ** 2).mean() / 10.0 ** (snr_db / 10.0) / 2.0)
    return (y + sigma * _gauss(gen, *y.shape)).to(torch.complex64)


def _problem(case, seed):
    """Trajectory, maps and noisy k-space [C, M] of a SENSE problem."""
    gen, rng = _gen(seed)
    traj, sens = _traj(case, rng), _maps(case, rng)
    op = _Exact(traj, (case["X"], case["Y"], case["Z"]))
    return traj, sens, _noisy(gen, op.forward((_phantom(case, rng) * sens).to(torch.complex128)))


def _batch_list(case):
    """The stack's slices: matrix sizes spread over 64..320, coils 4..32, spokes 16..256."""
    rng = np.random.default_rng(case["stack"])
    got = []
    for i in range(case["problems"]):
        N = 2 * int(round(32 + 128 * (i + rng.uniform(0.3, 0.7)) / case["problems"]))
        got.append(_recon(None, N, N, 1, int(rng.integers(4, 33)), int(rng.integers(16, 257)), 2 * N, case["iters"]))
    return got


def _pics(case, traj, sens):
    from bart_b200.pics import Pics, PicsConf
    dims = [case["X"], case["Y"], case["Z"], case["C"]]
    return Pics(traj, sens, conf=PicsConf(lam=LAMBDA, maxiter=case["iters"], precond=case["precond"],
                                          toeplitz=case["toeplitz"]),
                traj_dims=[3, case["samples"], case["spokes"]], sens_dims=dims,
                ksp_dims=[1, case["samples"], case["spokes"], case["C"]])


def _train_inputs(case, seed):
    from bart_b200.precnet import init_params
    gen, rng = _gen(seed)
    pix = case["X"] * case["Y"]
    x, t = _gauss(gen, case["n"], pix), _gauss(gen, case["n"], pix)
    par = init_params(seed)
    k = np.flatnonzero(par == 0)                      # biases and the last layer, as some training leaves them
    par[k] = 0.05 * rng.standard_normal(k.size).astype(np.float32)
    return x / torch.linalg.vector_norm(x, dim=1, keepdim=True), t / torch.linalg.vector_norm(t, dim=1, keepdim=True), par


def _calib_ksp(case, seed):
    """Cartesian k-space [C, 1, Y, X]: every second line, 24 x 24 fully sampled centre lines, 40 dB."""
    gen, rng = _gen(seed)
    c = {**case, "Z": 1}
    img = (_phantom(c, rng) * _maps(c, rng)).to(torch.complex128)
    k = torch.fft.fftshift(torch.fft.fft2(torch.fft.ifftshift(img, dim=(2, 3)), norm="ortho"), dim=(2, 3))
    j = torch.arange(case["Y"], device="cuda")
    keep = ((j - case["Y"] // 2).abs() <= 12) | (j % 2 == 0)
    return _noisy(gen, k) * keep[:, None]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "nufft":
        from bart_b200.nufft import NufftConf, nufft_create2
        gen, rng = _gen(seed)
        kd, td = [1, case["samples"], case["spokes"], case["C"]], [3, case["samples"], case["spokes"]]
        cd = [case["X"], case["Y"], case["Z"], case["C"]]
        M = case["samples"] * case["spokes"]
        wgt = _weights(case) if case["weights"] else None
        op = nufft_create2(kd, cd, td, _traj(case, rng), [1] + td[1:] if case["weights"] else None, wgt,
                           conf=NufftConf(toeplitz=False, deterministic=case["deterministic"]))
        return {"kind": kind, "op": op, "img": _gauss(gen, math.prod(cd)), "ksp": _gauss(gen, M * case["C"])}
    if kind == "recon":
        traj, sens, ksp = _problem(case, seed)
        model = None if case["setup"] else _pics(case, traj, sens)
        return {"kind": kind, "case": case, "traj": traj, "sens": sens, "ksp": ksp, "model": model}
    if kind == "batch":
        from bart_b200.batch import BatchRecon
        probs = []
        for i, c in enumerate(_batch_list(case)):
            t, s, y = _problem(c, 100 * seed + i)
            host = [a.cpu().numpy().ravel() for a in (t, s, y)]
            probs.append({"traj": host[0].reshape(3, c["samples"], c["spokes"], order="F"),
                          "sens": host[1].reshape(c["X"], c["Y"], 1, c["C"], order="F"),
                          "ksp": host[2].reshape(1, c["samples"], c["spokes"], c["C"], order="F")})
        return {"kind": kind, "batch": BatchRecon(probs, torch.device("cuda", 0), lam=LAMBDA, maxiter=case["iters"]).build()}
    if kind == "train":
        from bart_b200.precnet import PrecNet
        x, t, par = _train_inputs(case, seed)
        return {"kind": kind, "case": case, "net": PrecNet(par), "x": x, "t": t, "grads": np.empty(par.size, np.float32)}
    return {"kind": kind, "case": case, "ksp": _calib_ksp(case, seed)}


def run(state):
    kind = state["kind"]
    if kind == "nufft":
        return state["op"].forward(state["img"]), state["op"].adjoint(state["ksp"])
    if kind == "recon":
        p = state["model"] or _pics(state["case"], state["traj"], state["sens"])
        x = p.run(state["ksp"])
        if state["model"] is None:
            p.free()
        return x
    if kind == "batch":
        state["batch"].run()
        return list(state["batch"].img)
    c = state["case"]
    if kind == "train":
        loss = state["net"].train_step(state["x"], state["t"], c["X"], c["Y"], c["n"], 0.0, grads=state["grads"])
        return {"loss": loss, "grads": state["grads"]}
    from bart_b200.espirit import EcalibConf, ecalib
    sens, ev, info = ecalib(state["ksp"], EcalibConf(maps=1, softcrop=True), dims=[c["X"], c["Y"], 1, c["C"]])
    return {"sens": sens, "eigenvalues": ev, "nkernels": info["nkernels"]}


def _weights(case):
    """Ramp density compensation along the readout, [M] complex64."""
    r = (torch.arange(case["samples"], device="cuda") + 0.5) / case["samples"] - 0.5
    return (2.0 * r.abs()).repeat(case["spokes"]).to(torch.complex64)


# ---------------------------------------------------------------------------
# the same results in float64
# ---------------------------------------------------------------------------

def _table():
    beta = float(np.float32(math.pi * math.sqrt((WIDTH / 2.0 * 1.5) ** 2 - 0.8)))
    x = np.arange(TABLE + 1) / (TABLE - 1) / 2.0
    kb = np.where(x < 0.5, np.i0(beta * np.sqrt(np.maximum(0.0, 1.0 - (2.0 * x) ** 2))) / np.i0(beta), 0.0)
    return beta, torch.from_numpy(kb).cuda()


def _rolloff(n, beta):
    if n == 1:
        return torch.ones(1, dtype=torch.float64, device="cuda")
    p = (torch.arange(n, dtype=torch.float64, device="cuda") - n // 2) / (2 * n) * WIDTH * math.pi
    a = torch.sqrt((beta * beta - p * p).to(torch.complex128))
    return float(np.i0(beta)) / (torch.sinh(a) / a).real / WIDTH


class _Exact:
    """The NUFFT of [C, Z, Y, X] images and [C, M] k-space in float64: roll-off, 2x zero-padded transform, interpolation
    with the Kaiser-Bessel table at float32 sample positions, and the adjoint."""

    def __init__(self, traj, dims, periodic=False, weights=None):
        self.N, self.G = dims, tuple(2 * n if n > 1 else 1 for n in dims)
        self.traj, self.periodic, self.w = traj.real.contiguous(), periodic, weights
        beta, self.kb = _table()
        rx, ry, rz = (_rolloff(n, beta) for n in dims)
        self.roll = rz[:, None, None] * ry[:, None] * rx / math.sqrt(math.prod(dims))
        self.scale = math.prod(self.G)

    def lookup(self, d):
        s = 2.0 * d * (TABLE - 1)
        i = s.long().clamp(max=TABLE - 1)
        f = s - i
        return (1.0 - f) * self.kb[i] + f * self.kb[i + 1]

    def taps(self, k, a):
        """Cells [m, 6] and weights of axis a for positions k (float32)."""
        n = self.N[a]
        if n == 1:
            zero = torch.zeros(k.numel(), 1, device="cuda")
            return zero.long(), self.lookup(zero.double())
        cells, wts = [], []
        for s in (0, 1):
            pos = k + (-0.5 * s) + float(n // 2)
            lo = pos.double() - 1.5
            t = torch.floor(lo).long()[:, None] + torch.arange(1, 4, device="cuda")
            w = self.lookup(((t - pos.double()[:, None]).abs() / 3.0).clamp(max=0.5))
            if not self.periodic:
                w = w * ((t >= 0) & (t < n))
            cells.append((2 * t + s + n) % (2 * n))
            wts.append(w)
        return torch.cat(cells, 1), torch.cat(wts, 1)

    def chunks(self):
        size = 1 << (15 if self.N[2] > 1 else 16)
        for m0 in range(0, self.traj.shape[0], size):
            k = self.traj[m0:m0 + size]
            (cx, wx), (cy, wy), (cz, wz) = (self.taps(k[:, a].contiguous(), a) for a in range(3))
            idx = (cz[:, :, None, None] * self.G[1] + cy[:, None, :, None]) * self.G[0] + cx[:, None, None, :]
            w = wz[:, :, None, None] * wy[:, None, :, None] * wx[:, None, None, :]
            yield slice(m0, m0 + k.shape[0]), idx.flatten(1), w.flatten(1)

    def place(self, x):
        """[C, Z, Y, X] centred input in the zero-padded, DFT-ordered grid."""
        g = torch.zeros((x.shape[0],) + self.G[::-1], dtype=torch.complex128, device="cuda")
        z, y, xx = (n for n in x.shape[1:])
        g[:, :z, :y, :xx] = x
        return torch.roll(g, (-(z // 2), -(y // 2), -(xx // 2)), (1, 2, 3))

    def crop(self, g):
        x, y, z = self.N
        return torch.roll(g, (z // 2, y // 2, x // 2), (1, 2, 3))[:, :z, :y, :x]

    def forward(self, x):
        g = torch.fft.fftn(self.place(x * self.roll), dim=(1, 2, 3)).flatten(1).T.contiguous()
        g = torch.view_as_real(g).flatten(1)
        out = torch.empty(self.traj.shape[0], g.shape[1], dtype=torch.float64, device="cuda")
        for m, idx, w in self.chunks():
            out[m] = torch.bmm(w[:, None, :], g[idx])[:, 0]
        y = torch.view_as_complex(out.view(out.shape[0], -1, 2)).T.contiguous()
        return y if self.w is None else y * self.w

    def adjoint(self, y):
        y = y if self.w is None else y * self.w.conj()
        v = torch.view_as_real(y.to(torch.complex128).T.contiguous()).flatten(1)
        g = torch.zeros(self.scale, v.shape[1], dtype=torch.float64, device="cuda")
        for m, idx, w in self.chunks():
            g.index_add_(0, idx.flatten(), (w[:, :, None] * v[m][:, None, :]).flatten(0, 1))
        g = torch.view_as_complex(g.view(self.scale, -1, 2)).T.reshape((-1,) + self.G[::-1])
        return self.crop(torch.fft.ifftn(g, dim=(1, 2, 3)) * self.scale) * self.roll

    def psf(self):
        """Toeplitz spectrum: the adjoint of ones on the doubled image (periodic gridding), transformed."""
        inner = _Exact(2.0 * self.traj.to(torch.complex64), self.G, periodic=True)
        ones = torch.ones(1, self.traj.shape[0], dtype=torch.complex128, device="cuda")
        h = inner.adjoint(ones)
        h = torch.roll(h, tuple(-(n // 2) for n in h.shape[1:]), (1, 2, 3))
        return torch.fft.fftn(h, dim=(1, 2, 3)) / math.sqrt(self.scale) / math.prod(self.N)


def _exact_recon(case, seed):
    traj, sens, ksp = _problem(case, seed)
    sens = sens.to(torch.complex128)
    op = _Exact(traj, (case["X"], case["Y"], case["Z"]))
    psf = op.psf() if case["toeplitz"] else None

    def toeplitz(v, p):
        return op.crop(torch.fft.ifftn(torch.fft.fftn(op.place(v), dim=(1, 2, 3)) * p, dim=(1, 2, 3)) * op.scale)

    def normal(x):
        v = x * sens
        v = toeplitz(v, psf) if case["toeplitz"] else op.adjoint(op.forward(v))
        return (sens.conj() * v).sum(0) + LAMBDA * x

    if case["precond"] == 3:            # the padded circulant
        mu = max(2.5 * LAMBDA * 4.0 ** len(_axes(case)) / op.scale, 1e-3 * float(psf[0, 0, 0, 0].abs()))
        prec = lambda r: toeplitz(r[None], 1.0 / (psf.abs() + mu))[0]  # noqa: E731
    elif case["precond"] == 1:          # the circulant of the PSF's kernel on the image grid
        h = op.crop(torch.fft.ifftn(psf, dim=(1, 2, 3)) * op.scale)[0]
        pre = torch.fft.fftn(torch.roll(h, tuple(-(n // 2) for n in h.shape), (0, 1, 2))).abs()
        pre = pre / math.sqrt(h.numel()) + 1e-3
        prec = lambda r: torch.fft.ifftn(torch.fft.fftn(r) / pre)  # noqa: E731
    else:
        prec = lambda r: r  # noqa: E731

    b = (sens.conj() * op.adjoint(ksp)).sum(0)
    mag = torch.sort(b.abs().flatten()).values
    n = mag.numel()
    med, p90, top = (float(mag[i]) for i in (n // 2, int(n * 0.9), n - 1))
    b = b / (p90 if (top - p90) < 2 * (p90 - med) else top)
    x, r = torch.zeros_like(b), b.clone()
    z = prec(r)
    p, rz = z.clone(), torch.vdot(r.flatten(), z.flatten()).real
    for _ in range(case["iters"]):
        q = normal(p)
        a = rz / torch.vdot(p.flatten(), q.flatten()).real
        x, r = x + a * p, r - a * q
        z = prec(r)
        rz, old = torch.vdot(r.flatten(), z.flatten()).real, rz
        p = z + (rz / old) * p
    return x.flatten()


def _exact_train(case, seed):
    x, t, par = _train_inputs(case, seed)
    par = torch.from_numpy(par).cuda().double().requires_grad_()
    shape = (case["n"], case["Y"], case["X"], 2)
    act = torch.view_as_real(x.to(torch.complex128)).reshape(shape).permute(0, 3, 1, 2)
    want = torch.view_as_real(t.to(torch.complex128)).reshape(shape).permute(0, 3, 1, 2)
    o = 0
    for layer in range(6):
        ci, co = 2 if layer == 0 else 32, 2 if layer == 5 else 32
        w = par[o:o + co * 9 * ci].reshape(co, 3, 3, ci).permute(0, 3, 1, 2)
        b = par[o + co * 9 * ci:o + co * 9 * ci + co]
        o += co * 9 * ci + co
        cols = torch.nn.functional.pad(act, (1, 1, 1, 1)).unfold(2, 3, 1).unfold(3, 3, 1)
        act = torch.einsum("nchwyx,ocyx->nohw", cols, w) + b[:, None, None]
        if layer < 5:
            act = torch.relu(act)
    loss = ((act - want) ** 2).sum() / case["n"]
    loss.backward()
    return {"loss": float(loss.detach()), "grads": par.grad}


def _exact_ecalib(case, seed):
    k = _calib_ksp(case, seed).to(torch.complex128)[:, 0]
    C, Y, X = k.shape
    y0 = (Y - 24) // 2
    lines = k[:, y0:y0 + 24]
    energy = torch.stack([(lines[:, :, r:r + 24].abs() ** 2).sum() for r in range(X - 23)])
    x0 = int(torch.argmax(energy))
    cal = lines[:, :, x0:x0 + 24]
    # Casorati rows [361, C 36], kernel index x + 6 y + 36 c
    A = cal.unfold(1, 6, 1).unfold(2, 6, 1).permute(1, 2, 0, 3, 4).reshape(361, C * 36)
    _, s, vh = torch.linalg.svd(A, full_matrices=False)
    nk = int((s / s[0] > math.sqrt(np.float32(0.001))).sum())
    # the reference decomposes the conjugate matrix: its kernels are the conjugates of the right singular vectors
    kern = vh[:nk].reshape(nk, C, 6, 6)

    def basis(n):       # centred DFT of 6 kernel taps at the 12-point grid, then sinc interpolation to n points
        up = torch.zeros(n, 12, dtype=torch.complex128, device="cuda")
        u = torch.arange(12, device="cuda", dtype=torch.float64) - 6
        x = torch.arange(n, device="cuda", dtype=torch.float64) - n // 2
        f = torch.arange(12, device="cuda", dtype=torch.float64) - 6
        up = torch.exp(2j * math.pi * x[:, None] * f[None, :] / n) @ torch.exp(-2j * math.pi * f[:, None] * u[None, :] / 12)
        return up

    u = torch.arange(12, device="cuda", dtype=torch.float64) - 6
    t = torch.arange(6, device="cuda", dtype=torch.float64) - 3
    F = torch.exp(2j * math.pi * u[:, None] * t[None, :] / 12)          # centred inverse DFT of the padded kernel
    img = torch.einsum("yt,nctv,xv->ncyx", F, kern, F)
    cov = torch.einsum("niyx,njyx->ijyx", img.conj(), img) / (36.0 * 144.0)
    cov = torch.einsum("Yy,ijyx,Xx->YXij", basis(Y), cov, basis(X))
    H = torch.tril(cov)
    H = H + torch.tril(cov, -1).transpose(-1, -2).conj()
    v = torch.zeros(Y, X, C, dtype=torch.complex128, device="cuda")
    v[..., 0] = 1.0
    for _ in range(30):
        v = torch.einsum("yxi,yxij->yxj", v, H)
        ev = torch.linalg.vector_norm(v, dim=-1)
        v = v / ev[..., None]
    w = (torch.sqrt(ev) - 0.8) / 0.2
    v = v * ((w >= 1.0).double() + (w >= -1.0) * (w / (w * w + 1.0) + 0.5))[..., None]
    D = cal.reshape(C, -1).T
    r = torch.linalg.eigh((D.conj().T @ D).conj())[1][:, -1]
    r = r * (r[-1].conj() / r[-1].abs())
    ph = (v * r.conj()).sum(-1)
    v = v * torch.where(ph.abs() > 0, ph.conj() / ph.abs(), torch.ones_like(ph))[..., None]
    return {"sens": v.permute(2, 0, 1).flatten(), "eigenvalues": ev.to(torch.complex128).flatten(), "nkernels": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "nufft":
        gen, rng = _gen(seed)
        op = _Exact(_traj(case, rng), (case["X"], case["Y"], case["Z"]),
                    weights=_weights(case) if case["weights"] else None)
        shape = (case["C"], case["Z"], case["Y"], case["X"])
        img = _gauss(gen, math.prod(shape))
        ksp = _gauss(gen, case["samples"] * case["spokes"] * case["C"])
        y = op.forward(img.reshape(shape).to(torch.complex128)).flatten()
        return y, op.adjoint(ksp.reshape(case["C"], -1)).flatten()
    if kind == "recon":
        return _exact_recon(case, seed)
    if kind == "batch":
        return [_exact_recon(c, 100 * seed + i) for i, c in enumerate(_batch_list(case))]
    if kind == "train":
        return _exact_train(case, seed)
    return _exact_ecalib(case, seed)
