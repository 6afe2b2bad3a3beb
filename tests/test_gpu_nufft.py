"""GPU NUFFT through the C ABI against the reference's outputs and the oracle.

Bar: relative L2 <= 1e-5 per operator apply (forward, adjoint, Toeplitz
normal, PSF), on the golden fixtures (reference outputs) and on fresh seeded
inputs against the oracle.
"""

import numpy as np
import pytest

from bart_b200 import synth
from bart_b200.nufft import NufftConf, nufft_create2
from conftest import golden, rel
from oracle import nufft_oracle as orc

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _dims(img_shape):
    s = list(img_shape) + [1] * (4 - len(img_shape))
    return s


def _plan(g, periodic=False, toeplitz=True):
    img = g["img"]
    cd = _dims(img.shape)
    td = list(g["traj"].shape)
    kd = [1, td[1], td[2], cd[3]]
    w = g.get("pattern")
    wd = None if w is None else list(w.shape)
    return nufft_create2(kd, cd, td, g["traj"], wd, w, conf=NufftConf(toeplitz=toeplitz, periodic=periodic)), cd, kd


# image sides that are not powers of two: grid DFTs by Bluestein's algorithm
UNEVEN = [("nufft2d_n40", False), ("nufft2d_n40_periodic", True), ("nufft3d_n12", False)]


@pytest.mark.parametrize("name,periodic", [("nufft2d_n64", False), ("nufft2d_n64_periodic", True),
                                           ("nufft3d_n16", False), ("nufft2d_n32_coils3", False),
                                           ("nufft2d_n64_weights", False)] + UNEVEN)
def test_forward_adjoint_vs_reference(name, periodic):
    g = golden(name)
    op, cd, kd = _plan(g, periodic, toeplitz=False)
    fwd = op.forward(g["img"].reshape(cd, order="F"))
    assert rel(fwd, g["fwd"]) < TOL
    adj = op.adjoint(g["ksp"].reshape(kd, order="F"))
    assert rel(adj, g["adj"]) < TOL
    op.free()


@pytest.mark.parametrize("name,periodic", [("nufft2d_n64", False), ("nufft2d_n64_periodic", True),
                                           ("nufft3d_n16", False), ("nufft2d_n64_weights", False)] + UNEVEN)
def test_toeplitz_normal_and_psf_vs_reference(name, periodic):
    g = golden(name)
    op, cd, kd = _plan(g, periodic, toeplitz=True)
    n = op.normal(g["img"].reshape(cd, order="F"))
    assert rel(n, g["normal"]) < TOL
    psf = op.psf()
    assert rel(psf, g["psf"].reshape(psf.shape, order="F")) < TOL
    op.free()
    op, cd, kd = _plan(g, periodic, toeplitz=False)
    n = op.normal(g["img"].reshape(cd, order="F"))     # explicit adjoint(forward)
    assert rel(n, g["normal_explicit"]) < TOL
    op.free()


def _basis_plan(g, toeplitz):
    w = g.get("pattern")
    return nufft_create2(list(g["fwd"].shape), list(g["img"].shape), list(g["traj"].shape), g["traj"],
                         None if w is None else list(w.shape), w, list(g["basis"].shape), g["basis"],
                         conf=NufftConf(toeplitz=toeplitz))


@pytest.mark.parametrize("name", ["nufft2d_n32_basis", "nufft2d_n32_basis_shared"])
def test_basis_vs_reference(name):
    """Subspace basis (nufft -B): forward, adjoint, block-Toeplitz normal and
    the explicit normal against the reference's outputs; frames with their
    own trajectories, or one trajectory with a per-frame sampling pattern."""
    g = golden(name)
    op = _basis_plan(g, toeplitz=True)
    cd, kd = list(g["img"].shape), list(g["fwd"].shape)
    assert rel(op.forward(g["img"]), g["fwd"]) < TOL
    assert rel(op.adjoint(g["ksp"].reshape(kd, order="F")), g["adj"]) < TOL
    assert rel(op.normal(g["img"]), g["normal"]) < TOL
    op.free()
    op = _basis_plan(g, toeplitz=False)
    assert rel(op.normal(g["img"].reshape(cd, order="F")), g["normal_explicit"]) < TOL
    op.free()


def test_basis_uneven_size_and_3d_vs_oracle():
    """The basis on a non-power-of-two side (Bluestein spectra, block PSF on
    the 2N grid) and in 3D, against the oracle."""
    rng = np.random.default_rng(41)
    T, K, C = 3, 2, 2
    for N, ndim, spokes in ((40, 2, 30), (12, 3, 60)):
        t = synth.radial_traj(N, spokes) if ndim == 2 else synth.kooshball_traj(N, spokes)
        S = t.shape[2] // T
        tf = np.stack([t[:, :, f * S:(f + 1) * S] for f in range(T)], axis=-1).reshape(3, t.shape[1], S, 1, 1, T,
                                                                                    order="F")
        B = (rng.standard_normal((1, 1, 1, 1, 1, T, K)) + 1j * rng.standard_normal((1, 1, 1, 1, 1, T, K))).astype(
            np.complex64)
        Z = N if ndim == 3 else 1
        cd = [N, N, Z, C, 1, 1, K]
        kd = [1, t.shape[1], S, C, 1, T]
        x = (rng.standard_normal(cd) + 1j * rng.standard_normal(cd)).astype(np.complex64)
        op = nufft_create2(kd, cd, list(tf.shape), tf, None, None, list(B.shape), B, conf=NufftConf(toeplitz=True))
        o = orc.BasisNufftOracle([tf[..., 0, 0, f].real.reshape(3, -1, order="F") for f in range(T)], (N, N, Z),
                                 B.reshape(T, K, order="F"))
        xo = x.reshape(N, N, Z, C, K, order="F")
        assert rel(op.forward(x), o.forward(xo)) < TOL, (N, ndim)
        assert rel(op.normal(x), o.normal_toeplitz(xo)) < TOL, (N, ndim)
        op.free()


@pytest.mark.parametrize("N,spokes,coils", [(128, 64, 1), (64, 40, 2), (256, 402, 1), (512, 100, 1),
                                            (66, 30, 2), (200, 64, 1), (318, 90, 1), (320, 40, 2)])
def test_2d_vs_oracle(N, spokes, coils):
    rng = np.random.default_rng(N + spokes)
    t = synth.radial_traj(N, spokes)
    img = (rng.standard_normal((N, N, 1, coils)) + 1j * rng.standard_normal((N, N, 1, coils))).astype(np.complex64)
    cd = [N, N, 1, coils]
    kd = [1, t.shape[1], t.shape[2], coils]
    op = nufft_create2(kd, cd, list(t.shape), t, conf=NufftConf(toeplitz=True))
    o = orc.NufftOracle(t.real.reshape(3, -1, order="F"), (N, N, 1))
    assert rel(op.forward(img), o.forward(img)) < TOL
    y = (rng.standard_normal((t.shape[1] * t.shape[2], coils)) + 1j * rng.standard_normal((t.shape[1] * t.shape[2], coils))).astype(np.complex64)
    assert rel(op.adjoint(y.reshape(kd, order="F")), o.adjoint(y)) < TOL
    assert rel(op.normal(img), o.normal_toeplitz(img)) < TOL
    op.free()


def test_3d_vs_oracle():
    rng = np.random.default_rng(5)
    N = 32
    t = synth.kooshball_traj(N, 300)
    img = (rng.standard_normal((N, N, N, 1)) + 1j * rng.standard_normal((N, N, N, 1))).astype(np.complex64)
    cd = [N, N, N, 1]
    kd = [1, t.shape[1], t.shape[2], 1]
    op = nufft_create2(kd, cd, list(t.shape), t, conf=NufftConf(toeplitz=True))
    o = orc.NufftOracle(t.real.reshape(3, -1, order="F"), (N, N, N))
    assert rel(op.forward(img), o.forward(img)) < TOL
    y = (rng.standard_normal(kd[1] * kd[2]) + 1j * rng.standard_normal(kd[1] * kd[2])).astype(np.complex64)
    assert rel(op.adjoint(y.reshape(kd, order="F")), o.adjoint(y[:, None])) < TOL
    assert rel(op.normal(img), o.normal_toeplitz(img)) < TOL
    op.free()


def test_device_and_host_pointers_agree(cuda):
    import torch
    g = golden("nufft2d_n64")
    op, cd, kd = _plan(g, toeplitz=False)
    x = g["img"].reshape(cd, order="F").astype(np.complex64)
    host = op.forward(x)
    xd = torch.from_numpy(np.asfortranarray(x).ravel(order="F")).to(cuda)
    dev = op.forward(xd)
    torch.cuda.synchronize()
    assert np.array_equal(dev.cpu().numpy(), np.asarray(host).ravel(order="F"))
    op.free()


def test_adjointness_full_size():
    """<A x, y> = <x, A^H y> at the 256^2, 402x512 single-coil size."""
    rng = np.random.default_rng(11)
    t = synth.radial_traj(256, 402)
    cd = [256, 256, 1, 1]
    kd = [1, 512, 402, 1]
    op = nufft_create2(kd, cd, list(t.shape), t, conf=NufftConf(toeplitz=False))
    x = (rng.standard_normal(cd) + 1j * rng.standard_normal(cd)).astype(np.complex64)
    y = (rng.standard_normal(kd) + 1j * rng.standard_normal(kd)).astype(np.complex64)
    ax = np.asarray(op.forward(x)).astype(np.complex128)
    ay = np.asarray(op.adjoint(y)).astype(np.complex128)
    lhs = np.vdot(ax.ravel(order="F"), y.astype(np.complex128).ravel(order="F"))
    rhs = np.vdot(x.astype(np.complex128).ravel(order="F"), ay.ravel(order="F"))
    assert abs(lhs - rhs) / abs(lhs) < 1e-5
    op.free()


def test_unsupported_options_fail_loudly():
    """Options outside what is built are refused with a status, not run: an
    oversampled grid of odd length (os 1.25 on 34 pixels: 42.5 -> 42 is even,
    on 30: 37.5 -> 38 even, on 26: 32.5 -> 33 odd), os beyond 4, odd image
    sides, deterministic gridding with os != 2."""
    from bart_b200._lib import BnufftError
    t = synth.radial_traj(32, 8)
    with pytest.raises(BnufftError):
        nufft_create2([1, 64, 8, 1], [26, 26, 1, 1], list(t.shape), t, conf=NufftConf(os=1.25))
    with pytest.raises(BnufftError):
        nufft_create2([1, 64, 8, 1], [32, 32, 1, 1], list(t.shape), t, conf=NufftConf(os=5.0))
    with pytest.raises(BnufftError):
        nufft_create2([1, 64, 8, 1], [33, 33, 1, 1], list(t.shape), t)
    with pytest.raises(BnufftError):
        nufft_create2([1, 64, 8, 1], [32, 32, 1, 1], list(t.shape), t, conf=NufftConf(os=1.5, deterministic=True))


@pytest.mark.parametrize("name,periodic", [("nufft2d_n64", False), ("nufft2d_n64_periodic", True),
                                           ("nufft3d_n16", False), ("nufft2d_n32_coils3", False)])
def test_deterministic_mode_vs_reference(name, periodic):
    """Fixed-order (atomic-free) gridding: same parity bar as the default."""
    g = golden(name)
    img = g["img"]
    cd = _dims(img.shape)
    td = list(g["traj"].shape)
    kd = [1, td[1], td[2], cd[3]]
    toep = "normal" in g
    op = nufft_create2(kd, cd, td, g["traj"], conf=NufftConf(toeplitz=toep, periodic=periodic, deterministic=True))
    assert rel(op.forward(img.reshape(cd, order="F")), g["fwd"]) < TOL
    assert rel(op.adjoint(g["ksp"].reshape(kd, order="F")), g["adj"]) < TOL
    if toep:
        assert rel(op.normal(img.reshape(cd, order="F")), g["normal"]) < TOL
    op.free()


def test_deterministic_mode_is_bit_identical():
    """Two plans, two adjoints (and PSFs) of the same data: identical bits."""
    rng = np.random.default_rng(9)
    t = synth.radial_traj(256, 402)
    kd = [1, 512, 402, 4]
    cd = [256, 256, 1, 4]
    y = (rng.standard_normal(kd) + 1j * rng.standard_normal(kd)).astype(np.complex64)
    outs = []
    for _ in range(2):
        op = nufft_create2(kd, cd, list(t.shape), t, conf=NufftConf(toeplitz=True, deterministic=True))
        outs.append((np.asarray(op.adjoint(y)).copy(), op.psf().copy()))
        op.free()
    assert np.array_equal(outs[0][0].view(np.uint32), outs[1][0].view(np.uint32))
    assert np.array_equal(outs[0][1].view(np.uint32), outs[1][1].view(np.uint32))


@pytest.mark.parametrize("key,kw", [("inv_m5", dict(maxiter=5)), ("inv_m5_l", dict(maxiter=5, lam=0.1)),
                                    ("inv_m5_c", dict(maxiter=5, precond=True)),
                                    ("inv_m5_c_l", dict(maxiter=5, precond=True, lam=0.1))])
def test_nufft_inverse_vs_reference(key, kw):
    """bart nufft -i [-c] [-l] -m5 on three coil images."""
    g = golden("inverse2d_n32_coils3")
    td = list(g["traj"].shape)
    kd = [1, td[1], td[2], 3]
    op = nufft_create2(kd, [32, 32, 1, 3], td, g["traj"], conf=NufftConf(toeplitz=True))
    x = op.inverse(g["ksp"].reshape(kd, order="F"), **kw)
    op.free()
    assert rel(x, g[key]) < TOL


def test_nufft_inverse_30_iterations_precond():
    g = golden("inverse2d_n32_coils3")
    td = list(g["traj"].shape)
    kd = [1, td[1], td[2], 3]
    op = nufft_create2(kd, [32, 32, 1, 3], td, g["traj"], conf=NufftConf(toeplitz=True))
    x = op.inverse(g["ksp"].reshape(kd, order="F"), maxiter=30, precond=True)
    op.free()
    assert rel(x, g["inv_m30_c"]) < 1e-3


def test_lowmem_matches_default():
    """--lowmem (one coil's grid at a time) gives the default's results
    (deterministic gridding: identical bits)."""
    rng = np.random.default_rng(21)
    N, C = 48, 3
    t = synth.radial_traj(N, 20)
    img = (rng.standard_normal((N, N, 1, C)) + 1j * rng.standard_normal((N, N, 1, C))).astype(np.complex64)
    cd, kd = [N, N, 1, C], [1, t.shape[1], t.shape[2], C]
    out = {}
    for low in (False, True):
        op = nufft_create2(kd, cd, list(t.shape), t, conf=NufftConf(toeplitz=True, lowmem=low, deterministic=True))
        k = np.asarray(op.forward(img))
        out[low] = (k, np.asarray(op.adjoint(k.reshape(kd, order="F"))), np.asarray(op.normal(img)))
        op.free()
    for a, b in zip(out[False], out[True]):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("deterministic", [True, False])
def test_update_traj_equals_fresh_plan(deterministic):
    """nufft_update_traj (src/noncart/nufft.c:2041-2054): a plan created with
    one trajectory and updated to another gives the same forward, adjoint,
    Toeplitz normal and PSF as a plan created with the second one (bit for
    bit in the deterministic mode; with atomic gridding to float32 rounding),
    and those match the reference's outputs for that trajectory."""
    g = golden("nufft2d_n64")
    cd, td = [64, 64, 1, 1], list(g["traj"].shape)
    kd = [1, td[1], td[2], 1]
    other = synth.radial_traj(64, td[2]).reshape(td)        # uniform spacing, different angles
    other[0] *= 0.9
    conf = NufftConf(toeplitz=True, deterministic=deterministic)
    fresh = nufft_create2(kd, cd, td, g["traj"], conf=conf)
    upd = nufft_create2(kd, cd, td, other, conf=conf)
    x = g["img"].reshape(cd, order="F")
    y = g["ksp"].reshape(kd, order="F")
    before = np.asarray(upd.normal(x)).copy()
    upd.update_traj(g["traj"])
    outs = {}
    for name, op in (("fresh", fresh), ("upd", upd)):
        outs[name] = (np.asarray(op.forward(x)), np.asarray(op.adjoint(y)), np.asarray(op.normal(x)), op.psf())
    for a, b in zip(outs["fresh"], outs["upd"]):
        if deterministic:
            assert np.array_equal(np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32))
        else:
            assert rel(b, a) < 1e-6
    fwd, adj, nrm, psf = outs["upd"]
    assert rel(fwd, g["fwd"]) < TOL
    assert rel(adj, g["adj"]) < TOL
    assert rel(nrm, g["normal"]) < TOL
    assert rel(psf, g["psf"]) < TOL
    assert rel(before, g["normal"]) > 1e-2      # the PSF really followed the trajectory
    fresh.free()
    upd.free()


@pytest.mark.parametrize("N,spokes,coils,nd,periodic", [(256, 96, 16, 2, False), (256, 402, 1, 2, False),
                                                         (128, 64, 3, 2, False), (64, 40, 2, 2, True),
                                                         (40, 30, 6, 2, False), (32, 300, 8, 3, False),
                                                         (32, 200, 1, 3, True), (48, 300, 4, 3, False)])
def test_tiled_scatter_matches_atomic(N, spokes, coils, nd, periodic, monkeypatch):
    """The output-stationary adjoint gridding (tiles with register
    accumulation and plain stores; the default for 3D multi-coil problems,
    BNUFFT_GRIDDING=lines everywhere) against the global-atomic scatter
    (selected by an explicit bin edge) and the oracle, on 2D and 3D,
    periodic and not, single- and multi-coil problems, dense centres
    included."""
    rng = np.random.default_rng(N * 7 + coils)
    t = synth.radial_traj(N, spokes) if nd == 2 else synth.kooshball_traj(N, spokes)
    cd = [N, N, 1 if nd == 2 else N, coils]
    kd = [1, t.shape[1], t.shape[2], coils]
    y = (rng.standard_normal(kd) + 1j * rng.standard_normal(kd)).astype(np.complex64)
    outs = []
    monkeypatch.setenv("BNUFFT_GRIDDING", "lines")
    for b in (0, 32):
        op = nufft_create2(kd, cd, list(t.shape), t, conf=NufftConf(toeplitz=False, periodic=periodic, bin=b))
        outs.append(np.asarray(op.adjoint(y)))
        op.free()
    monkeypatch.delenv("BNUFFT_GRIDDING")
    assert rel(outs[0], outs[1]) < 1e-6
    o = orc.NufftOracle(t.real.reshape(3, -1, order="F"), tuple(cd[:3]), periodic=periodic)
    want = o.adjoint(y.reshape(-1, coils, order="F"))
    assert rel(outs[0], want.reshape(cd, order="F")) < TOL


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("dims,samples,spokes,coils,periodic,weights", [
    ((8, 8, 1), 16, 5, 1, False, False),        # a side of the quads' window twice over
    ((2, 4, 1), 16, 5, 1, False, False),        # shorter than the window, the smallest of all
    ((2, 4, 1), 16, 5, 3, True, False),         # the same, wrapping around several times
    ((6, 40, 1), 60, 9, 2, True, True),
    ((40, 6, 4), 60, 30, 4, False, True),       # a thin volume
    ((40, 4, 2), 60, 30, 3, True, False),       # the same, the footprint longer than an axis
    ((4, 6, 16), 40, 30, 8, True, False),       # four coils side by side on a short x
    ((50, 26, 1), 71, 33, 3, False, True),      # tiles cut short on both axes, odd coils, weights
    ((50, 50, 1), 100, 40, 2, True, False),     # the same, wrapping around
    ((100, 60, 1), 200, 300, 13, False, False),  # several chunks per tile, two coil jobs, the second partial
    ((24, 30, 26), 48, 120, 5, False, False),   # 3D, partial tiles
    ((26, 26, 26), 52, 80, 2, True, False)])    # 3D, wrapping around a partial tile
def test_gridding_edges_vs_oracle(dims, samples, spokes, coils, periodic, weights, deterministic):
    """Forward and adjoint where the tile lists, the quads' windows and the coil
    groups of the width-6 kernels end, with samples beyond the band edge (their
    taps are clipped or wrap), against the float64 oracle. Sums of at most a few
    thousand float32 products: TOL covers them as for the other sizes."""
    rng = np.random.default_rng(sum(dims) + coils)
    t = rng.uniform(-0.52, 0.52, (3, samples, spokes)) * np.array(dims)[:, None, None]
    t *= (np.arange(samples) / samples)[None, :, None]      # dense towards the centre
    t[np.array(dims) == 1] = 0.0
    t = t.astype(np.complex64)
    cd, kd = list(dims) + [coils], [1, samples, spokes, coils]
    w = (rng.uniform(0.5, 1.5, kd[:3]) * np.exp(1j * rng.uniform(0, 6, kd[:3]))).astype(np.complex64) if weights else None
    op = nufft_create2(kd, cd, list(t.shape), t, None if w is None else list(w.shape), w,
                       conf=NufftConf(toeplitz=False, periodic=periodic, deterministic=deterministic))
    o = orc.NufftOracle(t.real.reshape(3, -1, order="F"), dims, periodic=periodic, weights=w)
    x = (rng.standard_normal(cd) + 1j * rng.standard_normal(cd)).astype(np.complex64)
    y = (rng.standard_normal(kd) + 1j * rng.standard_normal(kd)).astype(np.complex64)
    fwd, adj = np.asarray(op.forward(x)), np.asarray(op.adjoint(y))
    if deterministic:
        assert np.array_equal(adj, np.asarray(op.adjoint(y)))
    op.free()
    assert rel(fwd.reshape(-1, coils, order="F"), o.forward(x)) < TOL
    assert rel(adj, o.adjoint(y.reshape(-1, coils, order="F"))) < TOL


@pytest.mark.parametrize("dims,coils,periodic,weights", [
    ((8, 8, 8), 4, False, False),       # the shortest z transform, one group of four
    ((10, 14, 16), 8, True, True),      # a block for each of two groups, wrapping around, weights
    ((18, 22, 32), 12, False, True),     # three groups
    ((16, 12, 96), 20, False, False),   # a mixed z length, several groups
    ((12, 10, 64), 6, True, False)])    # coils not in fours: the plain grid
def test_forward_of_coil_fours_vs_oracle(dims, coils, periodic, weights):
    """3D forward with four coils of a cell side by side in the grid, with
    samples beyond the band edge, against the float64 oracle and, channel by
    channel, the plain grid's gather: two orders of the same 216 float32
    products per sample, each within 216 eps of their absolute sum at worst and
    sqrt(216) eps = 9e-7 of its norm for independent roundings."""
    rng = np.random.default_rng(sum(dims) + coils)
    t = rng.uniform(-0.55, 0.55, (3, 40, 30)) * np.array(dims)[:, None, None]
    t = t.astype(np.complex64)
    cd, kd = list(dims) + [coils], [1, 40, 30, coils]
    w = (rng.uniform(0.5, 2.0, kd[:3]) * np.exp(1j * rng.uniform(0, 6, kd[:3]))).astype(np.complex64) if weights else None
    wd = None if w is None else list(w.shape)
    conf = NufftConf(toeplitz=False, periodic=periodic)
    op = nufft_create2(kd, cd, list(t.shape), t, wd, w, conf=conf)
    one = nufft_create2([1, 40, 30, 1], list(dims) + [1], list(t.shape), t, wd, w, conf=conf)
    o = orc.NufftOracle(t.real.reshape(3, -1, order="F"), dims, periodic=periodic, weights=w)
    x = (rng.standard_normal(cd) + 1j * rng.standard_normal(cd)).astype(np.complex64)
    fwd = np.asarray(op.forward(x))
    single = np.concatenate([np.asarray(one.forward(np.asfortranarray(x[..., c:c + 1]))) for c in range(coils)], axis=-1)
    op.free()
    one.free()
    assert rel(fwd, single) < 9e-7
    assert rel(fwd.reshape(-1, coils, order="F"), o.forward(x)) < TOL


@pytest.mark.parametrize("coils,periodic,weights", [(8, True, True), (12, False, True), (12, True, False), (20, False, True)])
def test_forward_of_two_coil_fours_at_once(coils, periodic, weights):
    """As above with samples enough (76000 and more) for blocks that take all
    channels, eight at a time and the last four after them, against the plain
    grid's gather channel by channel."""
    dims, M = (12, 14, 16), 400 * 200
    rng = np.random.default_rng(coils)
    t = (rng.uniform(-0.55, 0.55, (3, 400, 200)) * np.array(dims)[:, None, None]).astype(np.complex64)
    w = (rng.uniform(0.5, 2.0, (1, 400, 200)) * np.exp(1j * rng.uniform(0, 6, (1, 400, 200)))).astype(np.complex64) if weights else None
    wd = list(w.shape) if weights else None
    conf = NufftConf(toeplitz=False, periodic=periodic)
    op = nufft_create2([1, 400, 200, coils], list(dims) + [coils], list(t.shape), t, wd, w, conf=conf)
    one = nufft_create2([1, 400, 200, 1], list(dims) + [1], list(t.shape), t, wd, w, conf=conf)
    x = (rng.standard_normal(dims + (coils,)) + 1j * rng.standard_normal(dims + (coils,))).astype(np.complex64)
    fwd = np.asarray(op.forward(x)).reshape(M, coils, order="F")
    for c in range(coils):
        assert rel(fwd[:, c], np.asarray(one.forward(np.asfortranarray(x[..., c:c + 1])))) < 9e-7
    op.free()
    one.free()


@pytest.mark.parametrize("dims,coils", [
    ((96, 160, 1), 2), ((192, 224, 1), 1), ((288, 320, 1), 1), ((384, 62, 1), 2),      # the mixed lengths
    ((70, 132, 1), 3), ((104, 90, 1), 5), ((154, 54, 1), 1),    # radices 2 to 13
    ((228, 34, 1), 1),                                          # 456 = 8 3 19 and 68 = 4 17: Bluestein
    ((250, 500, 1), 1),                                         # four sequences per block
    ((210, 60, 1), 3), ((210, 60, 1), 25), ((60, 200, 1), 3),   # embedded on 512 points: rows of few channels, columns
    ((36, 40, 50), 2)])
def test_grid_lengths_vs_oracle(dims, coils):
    """Forward, adjoint and Toeplitz normal on grids of mixed lengths (64 times
    3, 5, 6, 7, 9, 10, 12), of smooth lengths (products of radices up to 13)
    and of lengths with a larger prime factor, on the two sides of a
    rectangle, against the float64 oracle. Transforms of at most 1000 points
    per axis add less than 1e-6 to the gridding's float32 sums."""
    rng = np.random.default_rng(sum(dims))
    t = rng.uniform(-0.5, 0.5, (3, 60, 50)) * np.array(dims)[:, None, None]
    t[np.array(dims) == 1] = 0.0
    t = t.astype(np.complex64)
    cd, kd = list(dims) + [coils], [1, 60, 50, coils]
    op = nufft_create2(kd, cd, list(t.shape), t, conf=NufftConf(toeplitz=True))
    o = orc.NufftOracle(t.real.reshape(3, -1, order="F"), dims)
    x = (rng.standard_normal(cd) + 1j * rng.standard_normal(cd)).astype(np.complex64)
    y = (rng.standard_normal(kd) + 1j * rng.standard_normal(kd)).astype(np.complex64)
    fwd, adj, nrm = (np.asarray(v).copy() for v in (op.forward(x), op.adjoint(y), op.normal(x)))
    op.free()
    assert rel(fwd.reshape(-1, coils, order="F"), o.forward(x)) < TOL
    assert rel(adj, o.adjoint(y.reshape(-1, coils, order="F"))) < TOL
    assert rel(nrm, o.normal_toeplitz(x)) < TOL


@pytest.mark.parametrize("N", [96, 160, 192, 224])
def test_mixed_lengths_are_as_exact_as_their_roundings(N):
    """Toeplitz normal on sides of 2N = 192, 320, 384 and 448 points (no
    embedding) against the float64 oracle, tighter than TOL: the transforms of
    the mixed lengths round no more often than their stages do. With u = 2^-24
    a float32 transform of L points with rounded twiddles has an rms error of
    about 0.7 u sqrt(log2 L). The normal has four of them along the two axes,
    the PSF four more (of 2L points) and its 36-product sums, about 2 u: together
    u sqrt(8 * 0.49 log2 L + 4), at most 2.12 u sqrt(log2 L) here. Bound: a tenth
    more, 2.35."""
    rng = np.random.default_rng(N)
    ang = np.arange(60) * np.pi * (np.sqrt(5.0) - 1.0) / 2.0
    r = ((np.arange(2 * N) + 0.5) / (2 * N) - 0.5) * N
    t = np.stack([r[:, None] * np.cos(ang), r[:, None] * np.sin(ang), 0.0 * r[:, None] * ang]).astype(np.complex64)
    op = nufft_create2([1, 2 * N, 60, 4], [N, N, 1, 4], list(t.shape), t, conf=NufftConf(toeplitz=True, deterministic=True))
    x = (rng.standard_normal((N, N, 1, 4)) + 1j * rng.standard_normal((N, N, 1, 4))).astype(np.complex64)
    y = np.asarray(op.normal(x)).copy()
    op.free()
    want = orc.NufftOracle(t.real.reshape(3, -1, order="F"), (N, N, 1)).normal_toeplitz(x)
    assert rel(y, want) < 2.35 * 2.0 ** -24 * np.sqrt(np.log2(2 * N))


@pytest.mark.parametrize("name", ["nufft2d_n64_chain", "nufft2d_n64_chain_weights", "nufft3d_n16_chain"])
def test_chain_vs_reference(name):
    """Oversampling other than 2 (nufft -o 1.25 / 1.5 / 2.5: the reference's
    chained NUFFT on a grid of lround(os N) cells, Bluestein transforms):
    forward, adjoint and the normal (adjoint of the forward, as the chain
    has no Toeplitz form) against the reference's outputs."""
    g = golden(name)
    cd = _dims(g["img"].shape)
    td = list(g["traj"].shape)
    kd = [1, td[1], td[2], cd[3]]
    w = g.get("pattern")
    for i, os_ in enumerate(g["oss"]):
        op = nufft_create2(kd, cd, td, g["traj"], None if w is None else list(w.shape), w,
                           conf=NufftConf(toeplitz=True, os=float(os_)))
        img = g["img"].reshape(cd, order="F")
        assert rel(op.forward(img), g[f"fwd_{i}"]) < TOL, os_
        assert rel(op.adjoint(g["ksp"].reshape(kd, order="F")), g[f"adj_{i}"]) < TOL, os_
        o = orc.ChainNufftOracle(g["traj"].real.reshape(3, -1, order="F"), cd[:3], float(os_), weights=w)
        assert rel(op.normal(img), o.adjoint(o.forward(img))) < TOL, os_
        op.free()


def test_cli_nufft_basis(tmp_path):
    """python -m bart_b200 nufft -B (forward, then adjoint with -x) on the
    basis fixture, as the reference's `bart nufft -B`."""
    from bart_b200.__main__ import main_nufft
    from bart_b200.cfl import readcfl, writecfl
    g = golden("nufft2d_n32_basis")
    for n in ("traj", "img", "ksp", "basis"):
        writecfl(str(tmp_path / n), g[n])
    p = lambda n: str(tmp_path / n)     # noqa: E731
    assert 0 == main_nufft(["-B", p("basis"), p("traj"), p("img"), p("k")])
    assert rel(readcfl(p("k")), g["fwd"]) < TOL
    assert 0 == main_nufft(["-a", "-B", p("basis"), "-x", "32:32:1", p("traj"), p("ksp"), p("a")])
    assert rel(readcfl(p("a")), g["adj"]) < TOL


def test_memory_pool_is_the_librarys_own(cuda):
    """Plans and models leave the release threshold of the device's default
    memory pool as the application set it, and what they leave mapped is given
    back on request."""
    import ctypes
    import torch
    from bart_b200 import _lib
    from bart_b200.pics import Pics, PicsConf
    lib = _lib.load()               # (with the symbols of the CUDA runtime that it links)
    pool, keep, now, before = ctypes.c_void_p(), ctypes.c_uint64(3 << 20), ctypes.c_uint64(0), ctypes.c_uint64(0)
    threshold = 4                   # cudaMemPoolAttrReleaseThreshold
    assert 0 == lib.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0)
    assert 0 == lib.cudaMemPoolGetAttribute(pool, threshold, ctypes.byref(before))
    try:
        assert 0 == lib.cudaMemPoolSetAttribute(pool, threshold, ctypes.byref(keep))
        rng = np.random.default_rng(2)
        t = synth.radial_traj(128, 60)
        free = torch.cuda.mem_get_info()[0]
        op = nufft_create2([1, 256, 60, 64], [128, 128, 1, 64], list(t.shape), t, conf=NufftConf(toeplitz=True))
        op.normal((rng.standard_normal((128, 128, 1, 64)) + 0j).astype(np.complex64))
        model = Pics(t, synth.coil_maps(128, 4, rng), conf=PicsConf(maxiter=2))
        model.run((rng.standard_normal((1, 256, 60, 4)) + 0j).astype(np.complex64))
        op.free()
        model.free()
        torch.cuda.synchronize()
        assert 0 == lib.cudaMemPoolGetAttribute(pool, threshold, ctypes.byref(now))
        assert now.value == keep.value
        _lib.check(lib.bnufft_release_memory())
        assert free - torch.cuda.mem_get_info()[0] < 64 << 20       # of some 200 MB of grids
    finally:
        lib.cudaMemPoolSetAttribute(pool, threshold, ctypes.byref(before))
