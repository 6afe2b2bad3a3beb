"""GPU CG-SENSE (pics -l2) through the C ABI against the reference and the oracle."""

import os

import numpy as np
import pytest

from bart_b200 import synth
from bart_b200.pics import Pics, PicsConf
from conftest import golden, rel
from oracle import nufft_oracle as orc

pytestmark = pytest.mark.gpu


def _run(g, **kw):
    p = Pics(g["traj"], g["sens"], ksp_dims=list(g["ksp"].shape), conf=PicsConf(lam=0.01, **kw))
    x = p.run(g["ksp"])
    st = p.stats()
    p.free()
    return np.asarray(x), st


# Reconstructions: the bar is 1e-4 (per operator apply 1e-5). The 2D cases
# hold 1e-5; in 3D each sample has 216 taps and float32 atomics add them in
# an arbitrary order, measured 1.2e-5 after 5 iterations.
@pytest.mark.parametrize("name,tol", [("pics2d_n64_c4", 1e-5), ("pics2d_n48_c3", 1e-5), ("pics3d_n16_c2", 5e-5)])
def test_pics_5_iterations_vs_reference(name, tol):
    g = golden(name)
    x, st = _run(g, maxiter=5, scaling=1.0)
    assert st[0] == 5
    assert rel(x, g["x5_w1"]) < tol
    x, st = _run(g, maxiter=5, scaling=1.0, toeplitz=False)
    assert rel(x, g["x5_w1_notoep"]) < tol


def test_pics_30_iterations_vs_reference():
    """30 unconverged iterations at 64^2 (4 coils) stay within the 1e-4
    reconstruction bar of the reference's pics (measured 4.9e-5; the
    reference's own runs at 1..8 threads differ by ~2.5e-5). Scaling must
    match to the last bit of the adjoint's order statistics."""
    g = golden("pics2d_n64_c4")
    x, st = _run(g, maxiter=30)
    xw, _ = _run(g, maxiter=30, scaling=1.0)
    x64, _ = _run(g, maxiter=30, ref_scalars=False)
    print(f"30 it: float32 scalars {rel(x, g['x30']):.2e} (w1 {rel(xw, g['x30_w1']):.2e}), "
          f"float64 scalars {rel(x64, g['x30']):.2e}")
    assert rel(x, g["x30"]) < 1e-4
    assert rel(xw, g["x30_w1"]) < 1e-4
    xs, st2 = _run(g, maxiter=30, rescale=True)
    # gridding adds with atomics, so the adjoint's p90 moves in the last bit
    assert abs(st2[2] - st[2]) <= 1e-6 * st[2]
    assert rel(xs, g["x30_rescale"]) < 1e-4


@pytest.mark.parametrize("lam,tol", [(0.1, 1e-4), (0.01, 5e-4)])
def test_pics_converged_vs_fp64_oracle(lam, tol):
    """Run to a tight CG tolerance: GPU (FP32 vectors, FP64 scalars) and the
    FP64 oracle converge to the same solution. The bar is the problem's own
    sensitivity to float32 operator rounding: perturbing the FP64 normal
    operator by 2e-7 relative moves the solution by 2.6e-5 (lambda 0.1) and
    2.2e-4 (lambda 0.01, condition ~1e3), so any float32 implementation,
    the reference's included, lands within that distance."""
    g = golden("pics2d_n64_c4")
    traj = g["traj"].real.reshape(3, -1, order="F")
    C = g["sens"].shape[3]
    y = g["ksp"].reshape(-1, C, order="F")
    A = orc.SenseOracle(traj, g["sens"])
    b = A.adjoint(y)
    xo, _ = orc.conjgrad(A.normal, b, lam, 500, tol=1e-10)
    p = Pics(g["traj"], g["sens"], ksp_dims=list(g["ksp"].shape),
             conf=PicsConf(lam=lam, maxiter=400, scaling=1.0, tol=1e-6))
    x = np.asarray(p.run(g["ksp"]))
    st = p.stats()
    p.free()
    assert st[1] <= 1e-6
    assert rel(x, xo) < tol
    assert orc.normal_residual(A, x.reshape(xo.shape, order="F"), b, lam) < 1e-4


def test_sense_normal_vs_oracle():
    g = golden("pics2d_n64_c4")
    p = Pics(g["traj"], g["sens"], ksp_dims=list(g["ksp"].shape), conf=PicsConf(lam=0.01))
    rng = np.random.default_rng(3)
    x = (rng.standard_normal((64, 64)) + 1j * rng.standard_normal((64, 64))).astype(np.complex64)
    n = np.asarray(p.normal(np.asfortranarray(x.reshape(64, 64, 1))))
    p.free()
    A = orc.SenseOracle(g["traj"].real.reshape(3, -1, order="F"), g["sens"])
    assert rel(n, A.normal(x.reshape(64, 64, 1, 1))) < 1e-5


def test_pics_deterministic_mode_bit_identical():
    """Deterministic mode: two full reconstructions give identical bits, and
    the result still matches the reference at 5 iterations."""
    g = golden("pics2d_n64_c4")
    x1, st1 = _run(g, maxiter=30, deterministic=True)
    x2, st2 = _run(g, maxiter=30, deterministic=True)
    assert np.array_equal(np.asarray(x1).view(np.uint32), np.asarray(x2).view(np.uint32))
    assert st1 == st2
    x5, _ = _run(g, maxiter=5, scaling=1.0, deterministic=True)
    assert rel(x5, g["x5_w1"]) < 1e-5


@pytest.mark.parametrize("tol", [0.0, 1e-4])
def test_cg_loop_graph_matches_host_loop(tol):
    """The CG loop as one graph (a while node over one iteration) and the
    host-driven loop run the same kernels: identical bits in deterministic
    mode, the same stopping iteration, and the graph runs no kernels past
    convergence."""
    g = golden("pics2d_n64_c4")
    res = {}
    for mode in ("1", "0"):
        os.environ["BNUFFT_CG_GRAPH"] = mode
        try:
            p = Pics(g["traj"], g["sens"], ksp_dims=list(g["ksp"].shape),
                     conf=PicsConf(lam=0.01, maxiter=200 if tol else 12, tol=tol, deterministic=True))
            x = np.asarray(p.run(g["ksp"]))
            res[mode] = (x, p.stats(), p.kernels())
            p.free()
        finally:
            os.environ.pop("BNUFFT_CG_GRAPH", None)
    (xg, sg, kg), (xh, sh, kh) = res["1"], res["0"]
    assert np.array_equal(xg.view(np.uint32), xh.view(np.uint32))
    assert sg == sh
    if tol:
        assert 10 < sg[0] < 200 and sg[1] <= tol
        assert kg < kh / 2      # the host loop launches all 200 iterations
    else:
        assert sg[0] == 12 and kg == kh + sg[0]    # plus one loop-advance kernel per iteration


def test_cg_loop_graph_reused_across_models():
    """A freed model hands its loop graph to the next one, which captures its
    own iteration into it and updates the executable in place (or, when that
    fails, instantiates its own): a chain of models of two sizes and two
    solvers, each built after the last was freed, solves bit-identically to
    the host-driven loop."""
    gs = {"a": golden("pics2d_n64_c4"), "b": golden("pics2d_n48_c3")}

    def solve(name, pc, graph):
        g = gs[name]
        os.environ["BNUFFT_CG_GRAPH"] = graph
        try:
            p = Pics(g["traj"], g["sens"], ksp_dims=list(g["ksp"].shape),
                     conf=PicsConf(lam=0.01, maxiter=60, tol=1e-6, scaling=1.0, precond=pc, deterministic=True))
            x = np.asarray(p.run(g["ksp"]))
            st = p.stats()
            p.free()
        finally:
            os.environ.pop("BNUFFT_CG_GRAPH", None)
        return x, st

    chain = [("a", 0), ("a", 0), ("b", 0), ("a", 1), ("a", 1), ("b", 1), ("b", 1), ("a", 0)]
    ref = {k: solve(*k, "0") for k in set(chain)}
    for k in chain:
        x, st = solve(*k, "1")
        assert np.array_equal(x.view(np.uint32), ref[k][0].view(np.uint32)), k
        assert st == ref[k][1], k


def test_fcg_circulant_converges_faster():
    """Flexible CG with the circulant PSF preconditioner reaches the same
    tolerance in fewer iterations than plain CG, to the same solution (the
    FP64 oracle's), with a true normal-equation residual at the tolerance;
    graph and host loops agree bit for bit in deterministic mode."""
    g = golden("pics2d_n64_c4")
    traj = g["traj"].real.reshape(3, -1, order="F")
    C = g["sens"].shape[3]
    A = orc.SenseOracle(traj, g["sens"])
    b = A.adjoint(g["ksp"].reshape(-1, C, order="F"))
    xo, _ = orc.conjgrad(A.normal, b, 0.01, 500, tol=1e-10)
    out = {}
    for pc in (0, 1):
        for mode in ("1", "0"):
            os.environ["BNUFFT_CG_GRAPH"] = mode
            try:
                p = Pics(g["traj"], g["sens"], ksp_dims=list(g["ksp"].shape),
                         conf=PicsConf(lam=0.01, maxiter=400, tol=1e-6, scaling=1.0, precond=pc, deterministic=True))
                x = np.asarray(p.run(g["ksp"]))
                out[pc, mode] = (x, p.stats())
                p.free()
            finally:
                os.environ.pop("BNUFFT_CG_GRAPH", None)
    for pc in (0, 1):
        assert np.array_equal(out[pc, "1"][0].view(np.uint32), out[pc, "0"][0].view(np.uint32))
        assert out[pc, "1"][1] == out[pc, "0"][1]
    it_cg, it_fcg = out[0, "1"][1][0], out[1, "1"][1][0]
    assert it_fcg < it_cg, (it_fcg, it_cg)
    x = out[1, "1"][0].reshape(xo.shape, order="F")
    assert orc.normal_residual(A, x, b, 0.01) < 1e-5
    assert rel(x, xo) < 5e-4      # the problem's float32 sensitivity (see the converged test)


@pytest.mark.parametrize("name", ["pics2d_n48_c3", "pics3d_n16_c2"])
def test_fcg_circulant_uneven_and_3d(name):
    """Flexible CG with the circulant preconditioner on a non-power-of-two 2D
    size (Bluestein grid DFTs, power-of-two Toeplitz embedding) and in 3D:
    converges to the FP64 oracle's solution in fewer iterations than CG."""
    g = golden(name)
    traj = g["traj"].real.reshape(3, -1, order="F")
    C = g["sens"].shape[3]
    A = orc.SenseOracle(traj, g["sens"])
    b = A.adjoint(g["ksp"].reshape(-1, C, order="F"))
    its = {}
    for pc in (0, 1):
        p = Pics(g["traj"], g["sens"], ksp_dims=list(g["ksp"].shape),
                 conf=PicsConf(lam=0.01, maxiter=400, tol=1e-6, scaling=1.0, precond=pc))
        x = np.asarray(p.run(g["ksp"]))
        its[pc] = p.stats()[0]
        p.free()
        xr = x.reshape(b.shape, order="F")
        assert orc.normal_residual(A, xr, b, 0.01) < 2e-5, pc
    assert its[1] < its[0], its


@pytest.mark.parametrize("N", [64, 128, 256])
def test_precond_cluster_matches_three_passes(N):
    """The circulant preconditioner in one launch on a thread-block cluster
    (square 2D images of 64, 128, 256 pixels) runs the three-pass form's
    arithmetic: z bit-identical, and a solve stops at the same iteration."""
    from bart_b200.problems import cgsense_problem
    prob = cgsense_problem(np.random.default_rng(N), N=N, coils=4, spokes=max(16, N // 4))
    r = (np.random.default_rng(1).standard_normal((N, N)) + 1j * np.random.default_rng(2).standard_normal((N, N)))
    r = np.asfortranarray(r.astype(np.complex64))
    out = {}
    for mode in ("1", "0"):
        os.environ["BNUFFT_PRECOND_CLUSTER"] = mode
        try:
            p = Pics(prob["traj"], prob["sens"], ksp_dims=list(prob["ksp"].shape),
                     conf=PicsConf(lam=0.01, maxiter=100, tol=1e-5, scaling=1.0, precond=1, deterministic=True))
            z = np.asarray(p.precond(r))
            p.run(prob["ksp"])
            out[mode] = (z, p.stats())
            p.free()
        finally:
            os.environ.pop("BNUFFT_PRECOND_CLUSTER", None)
    assert np.array_equal(out["1"][0].view(np.uint32), out["0"][0].view(np.uint32))
    assert np.abs(out["1"][0]).max() > 0
    # the <A p, z> partials are summed in another grouping: the stopping
    # iteration may move by one near the tolerance
    assert abs(out["1"][1][0] - out["0"][1][0]) <= 1 and out["1"][1][1] <= 1e-5


@pytest.mark.parametrize("name", ["pics2d_n64_c4", "pics2d_n48_c3", "pics3d_n16_c2"])
def test_fcg_padded_precond(name):
    """precond 3, the padded-circulant preconditioner (the Toeplitz
    operator's own circulant inverted on the padded image): converges to the
    FP64 oracle's normal-equation residual, in fewer iterations than plain
    CG and no more than the reference's Strang circulant (precond 1); on a
    power-of-two, a Bluestein-embedded and a 3D problem; graph and host
    loops agree bit for bit in deterministic mode."""
    g = golden(name)
    traj = g["traj"].real.reshape(3, -1, order="F")
    C = g["sens"].shape[3]
    A = orc.SenseOracle(traj, g["sens"])
    b = A.adjoint(g["ksp"].reshape(-1, C, order="F"))
    its, xs = {}, {}
    for pc, mode in ((0, "1"), (1, "1"), (3, "1"), (3, "0")):
        os.environ["BNUFFT_CG_GRAPH"] = mode
        try:
            p = Pics(g["traj"], g["sens"], ksp_dims=list(g["ksp"].shape),
                     conf=PicsConf(lam=0.01, maxiter=400, tol=1e-6, scaling=1.0, precond=pc, deterministic=True))
            x = np.asarray(p.run(g["ksp"]))
            its[pc, mode] = p.stats()[0]
            xs[pc, mode] = x
            p.free()
        finally:
            os.environ.pop("BNUFFT_CG_GRAPH", None)
        assert orc.normal_residual(A, x.reshape(b.shape, order="F"), b, 0.01) < 2e-5, (pc, mode)
    assert np.array_equal(xs[3, "1"].view(np.uint32), xs[3, "0"].view(np.uint32))
    assert its[3, "1"] == its[3, "0"]
    assert its[3, "1"] < its[0, "1"] and its[3, "1"] <= its[1, "1"], its


def test_padded_precond_matches_oracle():
    """z = M(r) of precond 3 on the device equals the FP64 oracle's
    padded-circulant preconditioner (its npix^2 normalisation, see
    oracle.padded_precond) on a power-of-two problem."""
    g = golden("pics2d_n64_c4")
    traj = g["traj"].real.reshape(3, -1, order="F")
    N = g["sens"].shape[0]
    A = orc.SenseOracle(traj, g["sens"])
    p = Pics(g["traj"], g["sens"], ksp_dims=list(g["ksp"].shape), conf=PicsConf(lam=0.01, precond=3))
    rng = np.random.default_rng(3)
    r = (rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))).astype(np.complex64)
    z = np.asarray(p.precond(np.asfortranarray(r))).reshape(N, N, order="F")
    p.free()
    zo = orc.padded_precond(A.nufft, 0.01)(r.astype(np.complex128).reshape(N, N, 1, 1))[:, :, 0, 0]
    assert rel(z, (N * N) ** 2 * zo) < 1e-5


@pytest.mark.parametrize("N", [72, 100])
def test_padded_precond_keeps_power_of_two_grid(N):
    """Where the normal operator runs on a shorter grid than the power of two
    (2N = 144 on 192; 2N = 200 on 256, the same), the padded-circulant
    preconditioner is still the power-of-two circulant's: its application
    against the float64 one from the oracle's PSF, and the normal operator on
    its own grid against the oracle."""
    rng = np.random.default_rng(N)
    traj = synth.radial_traj(N, 40)
    sens = synth.coil_maps(N, 3, rng)
    lam, L, E = 0.01, 2 * N, 256
    p = Pics(traj, sens, conf=PicsConf(lam=lam, precond=3))
    r = (rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))).astype(np.complex64)
    z = np.asarray(p.precond(np.asfortranarray(r))).reshape(N, N, order="F")
    y = np.asarray(p.normal(np.asfortranarray(r))).reshape(N, N, order="F")
    p.free()
    A = orc.SenseOracle(traj.real.reshape(3, -1, order="F"), sens)
    q = np.fft.ifft2(np.fft.ifftshift(A.nufft.psf()[:, :, 0])) / (N * N)
    d = np.arange(-N + 1, N)
    qe = np.zeros((E, E), dtype=np.complex128)
    qe[np.ix_(d % E, d % E)] = q[np.ix_(d % L, d % L)]
    P = np.abs(np.fft.fft2(qe)) * (L / E) ** 2
    mu = max(2.5 * lam * 16.0 / E ** 2, 1e-3 * P[0, 0])
    want = E * E * np.fft.ifft2(np.fft.fft2(r.astype(np.complex128), (E, E)) / (P + mu))[:N, :N]
    assert rel(z, want) < 1e-5
    s = sens[:, :, 0].astype(np.complex128)
    cim = (r.astype(np.complex128)[:, :, None] * s)[:, :, None, :]
    full = np.sum(np.conj(s) * A.nufft.normal_toeplitz(cim)[:, :, 0, :], axis=2)
    assert rel(y, full) < 1e-5


def test_fcg_folded_launches_match_unfolded():
    """The folded circulant flexible CG (dot products from the
    preconditioner's last pass, convergence test in the next direction
    update) solves like the unfolded one: about the same iterations, the
    same solution to the problem's float32 sensitivity at this tolerance,
    fewer launches."""
    g = golden("pics2d_n64_c4")
    res = {}
    for fold in ("1", "0"):
        os.environ["BNUFFT_FCG_FOLD"] = fold
        try:
            p = Pics(g["traj"], g["sens"], ksp_dims=list(g["ksp"].shape),
                     conf=PicsConf(lam=0.01, maxiter=300, tol=1e-5, scaling=1.0, precond=1))
            x = np.asarray(p.run(g["ksp"]))
            res[fold] = (x, p.stats(), p.kernels())
            p.free()
        finally:
            os.environ.pop("BNUFFT_FCG_FOLD", None)
    (xf, sf, kf), (xu, su, ku) = res["1"], res["0"]
    # float32 rounding in another summation order moves the stopping
    # iteration by a few near the tolerance
    assert abs(sf[0] - su[0]) <= max(3, su[0] // 10) and sf[1] <= 1e-5 and su[1] <= 1e-5
    assert rel(xf, xu) < 2e-3
    assert kf < ku


def test_pics_gpu_gridding_case_vs_reference():
    """Counterpart of the reference's GPU-gridding test (tests/gpu.mk:27-37,
    test-pics-gpu-noncart-gridding): the reference's own traj / scale /
    phantom -t / ones inputs and its CPU pics -S -r0.001 (30 iterations) as
    the fixture. The reference accepts its GPU gridding within nrmse 0.007 of
    its CPU result; here all gridding runs on the GPU, and with the
    reference's float32 CG scalars the result lies within the reference's own
    1-vs-all-thread spread (stored in the fixture) of its CPU output."""
    g = golden("pics2d_gpu_gridding_n128")
    traj, ksp = g["traj"], g["ksp"]
    sens = np.ones((128, 128, 1, 1), dtype=np.complex64)
    p = Pics(traj, sens, ksp_dims=list(ksp.shape), conf=PicsConf(lam=0.001, maxiter=30, rescale=True))
    x = np.asarray(p.run(ksp))
    p.free()
    e = rel(x, g["reco"])
    print(f"GPU-gridding case: {e:.2e} (reference spread {float(g['spread']):.2e})")
    assert e < 0.007
