"""CPU check of the register form of the DMC vertex representative (repr::vertex_point,
tmc_gb300/csrc/dmc_repr.cuh): built as host code by nvcc, every contour it answers must get the same
floats as the float64 restatement of the reference (cpp_dmc/DualMarchingCubes.cpp:194-326)."""
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

from tmc_gb300 import volumes as V

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = tmp_path_factory.mktemp("point") / "point_check"
    subprocess.run([nvcc, "-std=c++17", "-O2", "-x", "cu", "-Xcompiler", "-ffp-contract=off", "-fmad=false", "-o",
                    str(exe), os.path.join(ROOT, "tests", "cpp", "point_check.cpp")], check=True, capture_output=True)
    return exe


def _saddles(n):
    rng = np.random.Generator(np.random.PCG64(5))
    d = V.periodic(n, n, n, 6 * math.pi)
    V.seed_saddles(d, rng, frac=0.5)
    return d


def _levels(n, step):
    """Whole numbers (a scan's), isovalue one of them: corners at the isovalue, exact ties."""
    d = V.small_noise_volume(n, seed=4, coarse=6).data
    return np.round(d * step).astype(np.float32)


CASES = {
    "noise": (V.small_noise_volume(40, seed=5, coarse=7).data, 0.0),
    "noise_iso": (V.small_noise_volume(32, seed=3).data, 0.1234567),
    "blobs": (V.blobs_volume(48, seed=0).data, 0.5),
    "saddles": (_saddles(25), 0.0),
    "periodic": (V.periodic(41, 37, 33, 5 * math.pi), 0.1),
    # the in-plane pruning and the exact sample coordinates at the ends of their ranges
    "levels": (_levels(33, 20.0), 3.0),
    "levels_between": (_levels(33, 200.0), 2.5),
    "binary": ((V.small_noise_volume(24, seed=8).data > 0).astype(np.float32), 0.5),
    "tiny_values": (V.small_noise_volume(24, seed=9).data * np.float32(1e-38), 0.0),
    "huge_values": (V.small_noise_volume(24, seed=9).data * np.float32(3e38), 0.0),
    "steep": (np.sign(V.small_noise_volume(24, seed=9).data) * 10.0 ** (7 * V.small_noise_volume(24, seed=2).data),
              0.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_vertex_point_matches_the_reference_arithmetic(checker, tmp_path, name):
    data, iso = CASES[name]
    f = tmp_path / "f.raw"
    data.astype(np.float32).tofile(f)
    nz, ny, nx = data.shape
    r = subprocess.run([str(checker), str(f), str(nx), str(ny), str(nz), repr(iso)], capture_output=True, text=True,
                       check=True)
    contours, mism, redone, w64, excluded, searched = (int(x) for x in r.stdout.split())
    assert contours > 0
    assert mism == 0, r.stderr
    if name in ("noise", "noise_iso", "blobs", "periodic"):
        assert redone < 0.02 * contours  # generic fields: the rest takes the whole search
        assert searched == contours
