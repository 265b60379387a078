"""The kernels' viscosity, one Newton-Raphson inverse square root (mu_nr, nsf_physics.cuh; tests/host/viscosity.cu),
against x^1.5 sc1 / (re (T + sc1)) in extended precision.

Largest error, in units of u = 2^-53: x = 1 + T is rounded (1.5), d = re + T re / sc1 (1, and its rounded coefficient by
|T / (T + sc1)|), x d and (x d) d under the root (1), the root's last correction (1), the two products by x (2): at most
6.5 + |T / (T + sc1)|, taken as 8 + |T / (T + sc1)|. Over the flows' range of T, |T| <= 0.2, its rms is no larger than that of the quotient
form it stands for."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
U = 2.0 ** -53


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    nvcc = shutil.which("nvcc") or os.path.join(CUDA, "bin", "nvcc")
    out = str(tmp_path_factory.mktemp("viscosity") / "viscosity")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(ROOT, "3d-ns-fsi_b200", "csrc"),
                    os.path.join(ROOT, "tests", "host", "viscosity.cu"), "-o", out], check=True)
    return out


# (Reynolds number, sc1 = 1 + C2 / T0, range of T): the flows' range, hot and cold gas, the smallest and largest Reynolds
# numbers that are not clamped, negative denominators
CASES = [(1600.0, 1.4034, -0.2, 0.2), (100.0, 1.368, -0.2, 0.2), (0.37, 1.4034, -0.9, 5.0), (1e-100, 1.4, -0.2, 0.2),
         (1e100, 1.4, -0.2, 0.2), (-50.0, 1.4, -0.2, 0.2), (75.0, 0.5, -0.95, -0.6)]


@pytest.mark.gpu
@pytest.mark.parametrize("re,sc1,lo,hi", CASES)
def test_viscosity_against_extended_precision(exe, re, sc1, lo, hi, tmp_path):
    n = 200000
    T = np.random.default_rng(11).uniform(lo, hi, n)
    src, dst = str(tmp_path / "in"), str(tmp_path / "out")
    np.concatenate([[re, sc1], T]).tofile(src)
    subprocess.run([exe, src, dst], check=True, timeout=120)
    got = np.fromfile(dst).reshape(2, n).astype(np.longdouble)
    t, s = T.astype(np.longdouble), np.longdouble(sc1)
    ref = (1 + t) * np.sqrt(1 + t) * s / (np.longdouble(re) * (t + s))
    err = (got - ref) / ref
    rms = [float(np.sqrt(np.mean(e * e))) for e in err]
    print("re %g sc1 %g T %g .. %g: rms %.3g (quotient form %.3g), largest %.3g (%.3g)" % (
        re, sc1, lo, hi, rms[0], rms[1], float(np.abs(err[0]).max()), float(np.abs(err[1]).max())))
    assert np.all(np.abs(err[0]) <= (8 + np.abs(T / (T + sc1))) * U)
    if max(abs(lo), abs(hi)) <= 0.2:
        assert rms[0] <= rms[1]
