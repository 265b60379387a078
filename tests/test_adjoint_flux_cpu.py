"""The flux-form transposed RHS of the discrete adjoint (nsf_rhs_adjoint_flux.cuh), compiled for the host, against the
term table's transposed stencil (gen_rhs_adjoint.py) at every node of small grids, faces and corners included."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from test_adjoint_cpu import consts, gen

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NAMES = ["ax", "ay", "az", "h0", "pf", "e_xx23", "e_xx12", "e_yx6", "e_zx6", "e_yx4", "e_zx4", "e_yy12", "e_yy23", "e_zy6",
         "e_zy4", "e_zz12", "e_zz23"]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("flux") / "flux.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wno-unknown-pragmas", "-I",
                    os.path.join(ROOT, "3d-ns-fsi_b200", "csrc"),
                    os.path.join(ROOT, "tests", "host", "rhs_adjoint_flux.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("shape,d", [((7, 7, 7), (0.11, 0.13, 0.17)), ((5, 8, 3), (0.3, 0.02, 0.5)),
                                     ((3, 4, 9), (1.0, 2.0, 0.1))])
def test_flux_form_matches_the_term_table(lib, shape, d):
    rng = np.random.default_rng(sum(shape))
    pf = 1 / (0.4 * 0.71)
    fields = {q: rng.uniform(-1.0, 1.5, shape) for q in gen.VARS}
    fields["ka"] = pf * fields["mu"]
    C = consts(*d, 1.4)
    inner = np.zeros(shape, bool)
    inner[1:-1, 1:-1, 1:-1] = True
    lam = np.stack([rng.standard_normal(shape) * inner for _ in range(5)])
    ref = gen.adjoint(gen.adjoint_terms(gen.rhs_polys()), fields, list(lam), C)
    ref["mu"] = ref["mu"] + pf * ref["ka"]  # kappa = pf mu
    names = gen.VARS[:10]
    inp = np.ascontiguousarray(np.stack([fields[q] for q in names]))
    out = np.empty_like(inp)
    dp = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))  # noqa: E731
    cs = np.array([dict(C, pf=pf)[n] for n in NAMES])
    lib.rhs_adjoint_flux(dp(cs), np.array(shape, np.int32).ctypes.data_as(ctypes.POINTER(ctypes.c_int)),
                         dp(np.ascontiguousarray(lam)), dp(inp), dp(out))
    for q, name in enumerate(names):
        scale = max(1.0, np.abs(ref[name]).max())
        assert np.abs(out[q] - ref[name]).max() <= 1e-12 * scale, name
