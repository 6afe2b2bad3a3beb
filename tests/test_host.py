"""Host-side logic: .cfl I/O, synthetic inputs, CLI dimension rules."""

import os
import stat

import numpy as np
import pytest

from bart_b200 import build as builder
from bart_b200 import synth
from bart_b200.__main__ import estimate_im_dims
from bart_b200.cfl import readcfl, writecfl


def test_cfl_roundtrip(tmp_path):
    a = (np.arange(24) + 1j * np.arange(24)).astype(np.complex64).reshape(2, 3, 4, order="F")
    writecfl(str(tmp_path / "a"), a)
    b = readcfl(str(tmp_path / "a"))
    assert b.shape[:3] == (2, 3, 4) and all(d == 1 for d in b.shape[3:])
    assert np.array_equal(b.reshape(2, 3, 4, order="F"), a)
    hdr = open(str(tmp_path / "a.hdr")).read().split("\n")
    assert hdr[0] == "# Dimensions" and len(hdr[1].split()) == 16


def test_radial_traj_layout():
    t = synth.radial_traj(256, 402)
    assert t.shape == (3, 512, 402)
    assert np.isclose(t.real.max(), 127.75, atol=1e-3) and np.isclose(t.real.min(), -127.75, atol=1e-3)
    assert np.all(t.imag == 0) and np.all(t[2] == 0)


def test_synthetic_problem_is_seeded():
    a = synth.coil_maps(32, 4, np.random.default_rng(1))
    b = synth.coil_maps(32, 4, np.random.default_rng(1))
    assert np.array_equal(a, b)
    rss = np.sqrt(np.sum(np.abs(a) ** 2, axis=-1))
    assert np.allclose(rss, 1.0, atol=1e-5)
    p = synth.ellipse_phantom(64, 20, np.random.default_rng(2))
    assert p.shape == (64, 64, 1) and np.abs(p).max() > 0


def test_kooshball_directions_are_unit():
    t = synth.kooshball_traj(16, 100)
    d = t.real[:, -1, :] / np.abs(t.real[:, -1, :]).max()
    n = np.linalg.norm(t.real[:, -1, :], axis=0)
    assert np.allclose(n, n[0], rtol=1e-5)


def test_estimate_im_dims():
    t = synth.radial_traj(64, 8)
    assert estimate_im_dims(t) == [2 * int(np.ceil(np.abs(t.real[0]).max())), 2 * int(np.ceil(np.abs(t.real[1]).max())), 1]


def test_stream_reader_on_the_reference_stream():
    """bart_b200.stream reads a stream the reference wrote (copy --stream
    8192 | tee -b: header, settings, then index / raw / break per slice):
    every slice arrives once, at its position, with the array's values."""
    import io
    from bart_b200.stream import StreamReader
    from conftest import golden
    g = golden("stream_ksp_c4_s3")
    r = StreamReader(io.BytesIO(g["stream"].tobytes()))
    assert r.binary and r.flags == 8192 and r.dims[13] == 3
    seen = []
    for index, pos, block in r:
        seen.append(index)
        assert np.array_equal(block[..., 0, 0].reshape(block.shape[:4], order="F"),
                              g["ksp"][..., pos[0]].reshape(block.shape[:4], order="F"))
    assert seen == [0, 1, 2]


@pytest.fixture
def fake_nvcc(tmp_path, monkeypatch):
    """The build with a compiler that logs its arguments and writes its output file;
    with the word fail among the flags it leaves half a file and fails."""
    log = tmp_path / "log"
    nvcc = tmp_path / "nvcc"
    nvcc.write_text('#!/bin/sh\n[ "$1" = --version ] && echo one && exit\necho "$@" >> ' + str(log) + '\n'
                    'fail=0\nfor a in "$@"; do [ "$a" = fail ] && fail=1; [ "$p" = -o ] && echo out > "$a"; p="$a"; done\nexit $fail\n')
    nvcc.chmod(nvcc.stat().st_mode | stat.S_IXUSR)
    for name, value in (("NVCC", str(nvcc)), ("OBJ", str(tmp_path / "obj")), ("LIB", str(tmp_path / "lib" / "lib.so")),
                        ("STAMP", str(tmp_path / "obj" / "command")), ("FLAGS", ["-O3"])):
        monkeypatch.setattr(builder, name, value, raising=False)
    log.touch()
    return lambda: log.read_text().splitlines()


def test_build_follows_its_command_and_sources(fake_nvcc, monkeypatch):
    """Objects and the library are made again when a flag, an environment's compiler or
    a source changed, and not otherwise."""
    builder.build()
    n = len(fake_nvcc())
    assert n == len(builder.UNITS) + 1
    builder.build()
    assert len(fake_nvcc()) == n
    monkeypatch.setattr(builder, "FLAGS", ["-O2"])
    builder.build()
    assert len(fake_nvcc()) == 2 * n and all("-O2" in c for c in fake_nvcc()[n:2 * n - 1])
    later = os.path.getmtime(builder.LIB) + 1000
    inputs = builder._inputs
    monkeypatch.setattr(builder, "_inputs", lambda u: inputs(u) + (["changed"] if u == "passes_1" else []))
    getmtime = os.path.getmtime
    monkeypatch.setattr(os.path, "getmtime", lambda f: later if f == "changed" else getmtime(f))
    builder.build()
    assert len(fake_nvcc()) == 2 * n + 2


def test_build_that_fails_leaves_no_object(fake_nvcc, monkeypatch):
    monkeypatch.setattr(builder, "FLAGS", ["fail"])
    with pytest.raises(RuntimeError):
        builder.build()
    assert not os.path.exists(builder.LIB) and not os.listdir(builder.OBJ)


def test_objects_are_kept_in_the_checkout():
    """No folder of a predictable name that other users of the machine can make first."""
    assert builder.OBJ.startswith(builder.ROOT + os.sep)
