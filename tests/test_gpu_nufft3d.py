"""3D radial kooshball NUFFT on the GPU: the reference's outputs at 32^3, the
oracle at 64^3 with 8 coils, and size-independent properties at the full
128^3 / 8-coil / 20000 x 256 configuration.

Bar: relative L2 <= 1e-5 per operator apply against the reference and the
oracle; at full size, adjointness <A x, y> = <x, A^H y> to 1e-5 and the
default (output-stationary) scatter against the global-atomic scatter to
1e-6 (same sums, other float32 order).
"""

import hashlib
import os
import subprocess
import sys

import numpy as np
import pytest

from bart_b200 import synth
from bart_b200.nufft import NufftConf, nufft_create2
from conftest import golden, rel
from oracle import nufft_oracle as orc

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _cplx(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


def _sha(a):
    return hashlib.sha256(np.ascontiguousarray(a).tobytes(order="F")).hexdigest()


def test_kooshball_32_vs_reference():
    g = golden("nufft3d_n32_c2")
    rng = np.random.default_rng(int(g["seed"]))
    traj = synth.kooshball_traj(32, 400)
    img = _cplx(rng, (32, 32, 32, 2))
    ksp = _cplx(rng, (1, 64, 400, 2))
    assert _sha(img) == str(g["img_sha256"]) and _sha(ksp) == str(g["ksp_sha256"])
    cd, kd = [32, 32, 32, 2], [1, 64, 400, 2]
    op = nufft_create2(kd, cd, list(traj.shape), traj, conf=NufftConf(toeplitz=True))
    try:
        assert rel(op.forward(img), g["fwd"]) < TOL
        assert rel(op.adjoint(ksp), g["adj"]) < TOL
        assert rel(op.normal(img), g["normal"]) < TOL
    finally:
        op.free()


def test_kooshball_64_eight_coils_vs_oracle():
    """64^3, 8 coils, 1000 spokes x 128: the multi-coil 3D scatter (the
    output-stationary kernel) and gather against the FP64 oracle."""
    import torch
    rng = np.random.default_rng(64)
    N, C = 64, 8
    traj = synth.kooshball_traj(N, 1000)
    M = traj.shape[1] * traj.shape[2]
    img = _cplx(rng, (N, N, N, C))
    y = _cplx(rng, (1, traj.shape[1], traj.shape[2], C))
    cd, kd = [N, N, N, C], [1, traj.shape[1], traj.shape[2], C]
    dev = torch.device("cuda:0")

    def d(a):
        return torch.from_numpy(np.asfortranarray(a).ravel(order="F").copy()).to(dev)

    op = nufft_create2(kd, cd, list(traj.shape), d(traj), conf=NufftConf(toeplitz=False))
    try:
        fwd = op.forward(d(img)).cpu().numpy()
        adj = op.adjoint(d(y)).cpu().numpy()
    finally:
        op.free()
    o = orc.NufftOracle(traj.real.reshape(3, -1, order="F"), (N, N, N))
    assert rel(fwd, o.forward(img)) < TOL
    assert rel(adj, o.adjoint(y.reshape(M, C, order="F")).ravel(order="F")) < TOL


def test_kooshball_full_size_properties(monkeypatch):
    """The config's own size: 128^3, 8 coils, 20000 x 256 golden-means
    kooshball (5.12 M samples per coil). <A x, y> = <x, A^H y> in float64
    sums of the GPU's float32 outputs, and the default scatter equals the
    global-atomic one (an explicit bin edge selects it) to float32 order."""
    import torch
    rng = np.random.default_rng(128)
    N, C = 128, 8
    traj = synth.kooshball_traj(N, 20000)
    dev = torch.device("cuda:0")
    t_d = torch.from_numpy(np.asfortranarray(traj).ravel(order="F").copy()).to(dev)
    M = traj.shape[1] * traj.shape[2]
    cd, kd = [N, N, N, C], [1, traj.shape[1], traj.shape[2], C]
    gen = torch.Generator(device=dev).manual_seed(5)
    x = torch.randn(N ** 3 * C, dtype=torch.complex64, device=dev, generator=gen)
    y = torch.randn(M * C, dtype=torch.complex64, device=dev, generator=gen)
    monkeypatch.delenv("BNUFFT_GRIDDING", raising=False)
    op = nufft_create2(kd, cd, list(traj.shape), t_d, conf=NufftConf(toeplitz=False))
    ref = nufft_create2(kd, cd, list(traj.shape), t_d, conf=NufftConf(toeplitz=False, bin=16))
    try:
        ax = op.forward(x)
        ahy = op.adjoint(y)
        ahy_atomic = ref.adjoint(y)
        lhs = torch.vdot(y.to(torch.complex128), ax.to(torch.complex128))
        rhs = torch.vdot(ahy.to(torch.complex128), x.to(torch.complex128))
        assert abs(complex(lhs - rhs)) / abs(complex(lhs)) < TOL
        assert float(torch.linalg.vector_norm(ahy - ahy_atomic) / torch.linalg.vector_norm(ahy_atomic)) < 1e-6
    finally:
        op.free()
        ref.free()


_MEMORY = """
import sys
import torch
from bart_b200.nufft import NufftConf, nufft_create2
M, C, N = int(sys.argv[1]), int(sys.argv[2]), 64
t = ((torch.rand(M, 3, device="cuda") - 0.5) * N).to(torch.complex64)
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
op = nufft_create2([1, 1024, M // 1024, C], [N, N, N, C], [3, 1024, M // 1024], t, conf=NufftConf(toeplitz=False))
torch.cuda.synchronize()
print((free - torch.cuda.mem_get_info()[0]) / M)
"""


def _plan_bytes_per_sample(M, C):
    """Device memory that a new process's first plan takes, per sample."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _MEMORY, str(M), str(C)], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    return float(r.stdout)


def test_plan_memory_of_many_samples():
    """Hit lists as long as counted: of 2^23 uniform samples a footprint of six
    cells a side meets (8 + 5)(4 + 5)(4 + 5) / 128 = 8.2 tiles, 33 bytes, and a
    sample further holds 96 bytes of footprint, 4 of order, 16 of trajectory and
    16 of two channels' k-space: 165. The set-up's own arrays (order, its sort and
    the start cells) stay below 32. (At the bound of 18 hits: 204 and those.)"""
    assert _plan_bytes_per_sample(1 << 23, 2) < 165 + 32


def test_plan_memory_of_many_samples_one_channel():
    """Plans without tiles keep the footprints of 2^25 samples, 96 bytes each: of
    2^26 samples 48 bytes a sample, and 4 of order, 16 of trajectory and less
    than 28 of the set-up's own arrays. (96 with all footprints.)"""
    assert _plan_bytes_per_sample(1 << 26, 1) < 68 + 28


def test_more_samples_than_footprints():
    """2^25 + 3 * 2^20 samples in one channel, with weights, more than a plan keeps
    footprints of: forward has the same bits as a plan of the last 2^21 samples,
    and the adjoint is the sum of those of the first and the other 2^25. Some
    1200 terms in a cell of the grid: 1200^(1/2) 2^-24 = 2.1e-6."""
    import torch
    N, M, last, first = 512, (1 << 25) + 3 * (1 << 20), 1 << 21, 1 << 25
    gen = torch.Generator(device="cuda").manual_seed(5)
    t = torch.zeros(M, 3, dtype=torch.complex64, device="cuda")
    t[:, :2] = (torch.rand(M, 2, generator=gen, device="cuda") - 0.5) * N
    y = torch.view_as_complex(torch.randn(M, 2, generator=gen, device="cuda"))
    w = torch.rand(M, generator=gen, device="cuda").to(torch.complex64)
    x = torch.view_as_complex(torch.randn(N * N, 2, generator=gen, device="cuda"))

    def plan(sel):
        n = t[sel].shape[0] // 1024
        return nufft_create2([1, 1024, n, 1], [N, N, 1, 1], [3, 1024, n], t[sel].contiguous(), [1, 1024, n],
                             w[sel].contiguous(), conf=NufftConf(toeplitz=False))

    op = plan(slice(0, M))
    fwd, adj = op.forward(x), op.adjoint(y).to(torch.complex128)
    op.free()
    parts = []
    for sel in (slice(0, first), slice(first, M)):
        op = plan(sel)
        parts.append(op.adjoint(y[sel].contiguous()).to(torch.complex128))
        op.free()
    op = plan(slice(M - last, M))
    assert torch.equal(torch.view_as_real(op.forward(x)), torch.view_as_real(fwd[M - last:].contiguous()))
    op.free()
    want = parts[0] + parts[1]
    assert float(torch.linalg.vector_norm(adj - want) / torch.linalg.vector_norm(want)) < 2.1e-6


@pytest.mark.parametrize("dims,spokes,chunk,periodic", [((64, 64, 64), 2000, None, False), ((64, 64, 64), 9000, None, True),
                                                        ((128, 64, 80), 2000, 32, False), ((128, 72, 84), 2000, 32, True)])
def test_plans_of_many_tiles(dims, spokes, chunk, periodic, monkeypatch):
    """More tiles than one block plans (16384 in two segments, 40960 in five, 48384
    in six): the tile scatter and its deterministic form against the
    single-channel scatter, with hits that fit one work item a tile and with
    several. Tiles listed by warps (330, 130 and 110 candidates on average, more than
    a warp takes at the centre, and where a periodic grid wraps around tiles cut
    short) and by blocks (1500; their lists are counted before they are made). Two orders of the same float32
    sums of some hundred terms."""
    rng = np.random.default_rng(dims[0] + spokes)
    if chunk:
        monkeypatch.setenv("BNUFFT_GRID_CHUNK", str(chunk))
    t = rng.uniform(-0.55, 0.55, (3, 100, spokes)) * np.array(dims)[:, None, None]
    t[:, :, :spokes // 5] *= 0.1            # dense towards the centre
    t = t.astype(np.complex64)
    y = _cplx(rng, (1, 100, spokes, 2))
    kd, cd = [1, 100, spokes, 2], list(dims) + [2]
    out = []
    for det in (False, True):
        op = nufft_create2(kd, cd, list(t.shape), t, conf=NufftConf(toeplitz=False, deterministic=det, periodic=periodic))
        out.append(np.asarray(op.adjoint(y)).copy().reshape(cd, order="F"))
        op.free()
    op = nufft_create2(kd[:3] + [1], list(dims) + [1], list(t.shape), t, conf=NufftConf(toeplitz=False, periodic=periodic))
    one = [np.asarray(op.adjoint(np.asfortranarray(y[..., c:c + 1]))).copy().reshape(dims, order="F") for c in range(2)]
    op.free()
    for c in range(2):
        assert rel(out[0][..., c], one[c]) < 1e-6
        assert rel(out[1][..., c], one[c]) < 1e-6
