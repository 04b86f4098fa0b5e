"""Vertices and signs in pairs of floats (csrc/pair_float.cuh), built for the host
with g++ (tests/pair_float_host.cpp), against extended precision: each
coordinate of an accepted vertex is its exact value rounded to float, whatever
its size against the others, up to what less than 2^-30 of it can move a
rounding (half an ulp and a fiftieth)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import PKG_DIR, ROOT


@pytest.fixture(scope="module")
def pair_bin(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    out = tmp_path_factory.mktemp("pair_float") / "pair_float_host"
    r = subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(PKG_DIR / "csrc"), "-I",
                        os.path.join(cuda, "include"), str(ROOT / "tests" / "pair_float_host.cpp"), "-o", str(out)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return out


def bisectors(kind, m, rng):
    """(m, 4, 4) planes (-b, |b|^2 / 2) of neighbours b."""
    b = rng.normal(0.0, 10.0, (m, 4, 3))
    if kind == "mirrored":  # vertices near the plane x = 0
        b[:, 1] = b[:, 0] * [-1, 1, 1] + rng.normal(0.0, 0.05, (m, 3))
    if kind == "lattice":
        b = 62.5 * rng.integers(-2, 3, (m, 4, 3)) + rng.uniform(-2e-3, 2e-3, (m, 4, 3))
    b = b.astype(np.float32)
    w = np.float32(0.5) * (b * b).sum(-1, dtype=np.float32)
    return np.concatenate([-b, w[..., None]], -1)


@pytest.mark.parametrize("kind,accepted", [("random", 0.97), ("mirrored", 0.2), ("lattice", 0.3)])
def test_accepted_vertices_are_rounded_once(pair_bin, tmp_path, kind, accepted):
    m = 300_000
    rows = np.ascontiguousarray(bisectors(kind, m, np.random.default_rng(5)), np.float32)
    src, dst = tmp_path / "r.f32", tmp_path / "o.f32"
    rows.tofile(src)
    r = subprocess.run([str(pair_bin), str(src), str(m), str(dst)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = np.fromfile(dst, dtype=np.float32).reshape(m, 5)
    ok = out[:, 0] == 1
    assert accepted < ok.mean() < 1
    q = rows[ok].astype(np.longdouble)
    n, w = q[:, :3, :3], q[:, :3, 3]
    bc, ca, ab = (np.cross(n[:, i], n[:, (i + 1) % 3]) for i in (1, 2, 0))
    det = (n[:, 0] * bc).sum(-1)
    x = -(w[:, :1] * bc + w[:, 1:2] * ca + w[:, 2:] * ab) / det[:, None]
    ulp = np.spacing(np.abs(x).astype(np.float32)).astype(np.longdouble)
    assert (np.abs(out[ok, 1:4].astype(np.longdouble) - x) / ulp).max() < 0.52
    # the fourth plane's side, where the pairs tell it
    at = (q[:, 3, :3] * x).sum(-1) + q[:, 3, 3]
    side = out[ok, 4]
    told = (side != 0) & (np.abs(at) > 1e-15 * np.abs(q[:, 3, 3]))
    assert told.mean() > 0.9
    assert np.array_equal(np.sign(at[told]).astype(np.float32), side[told])
