"""Rounding of nsf_step_metrics_noalloc, on data where every other operation is exact or spelled out.

The dt limits divide by 1 + rho and by the viscosity's denominator. A quotient that is corrected by its residual is
rounded as a division except next to a midpoint, and so is the refined square root: dt equals the IEEE evaluation in all
but a rare case (1 % allowed), where the plain product with a reciprocal is off by one in the last place for every few
values. A block adds its warps' sums in pairs: terms that vanish one by one against the largest survive together."""
import ctypes
import math

import numpy as np
import pytest

import nsfsi


def config(n, lengths, re):
    cfg = nsfsi.config_load(nsfsi.case_path("tgv256"))
    cfg.NI, cfg.NJ, cfg.NK = n
    cfg.lx, cfg.ly, cfg.lz = lengths
    cfg.gamma, cfg.pr, cfg.re = 2.0, 1.0, re  # gamma - 1 = 1, gamma p exact, viscous factor max(4/3, 2) = 2
    return cfg


def metrics(cfg, old, new, types, out):
    import torch

    st = nsfsi.lib().nsf_step_metrics_noalloc(ctypes.byref(cfg), old.data_ptr(), new.data_ptr(),
                                              None if types is None else types.data_ptr(), out.data_ptr(),
                                              torch.cuda.current_stream().cuda_stream)
    assert st == 0


@pytest.mark.gpu
@pytest.mark.parametrize("limit", ["convective", "viscous"])
def test_time_step_is_rounded_as_by_divisions(limit):
    import torch

    cfg = config((3, 3, 3), (1.0, 1.0, 1.0), 1e9 if limit == "convective" else 0.37)
    m = 2000
    rng = np.random.default_rng(3)
    rho = rng.uniform(-0.2, 0.2, m)
    # gas at rest: p = rho_E, 1 + gamma p = 1 + 2 rho_E; the viscous case at T = 0, where 2 p = rho
    E = rng.uniform(0.3, 0.6, m) if limit == "convective" else rho / 2
    states = torch.zeros((m, 5, 27), dtype=torch.float64)
    states[:, 0] = torch.from_numpy(rho)[:, None]
    states[:, 4] = torch.from_numpy(E)[:, None]
    states = states.cuda()
    out = torch.zeros((m, 6), dtype=torch.float64, device="cuda")
    for q in range(m):
        metrics(cfg, states[q], states[q], None, out[q])
    c = np.sqrt((1 + 2 * E) / (1 + rho))
    conv = abs(cfg.conv_stability_limit) / ((c + c) + c)
    sc = 1 + cfg.sutherlands_c2 / cfg.t0
    visc = abs(cfg.visc_stability_limit) / ((sc / (cfg.re * sc) / (1 + rho) * 2) * 3)
    ref = conv if limit == "convective" else visc
    assert np.all(conv < visc) if limit == "convective" else np.all(visc < conv)
    got = out[:, 5].cpu().numpy()
    assert np.all(np.abs(got - ref) <= 2 * np.spacing(ref))
    assert np.mean(got == ref) >= 0.99, np.mean(got == ref)


@pytest.mark.gpu
def test_warps_are_added_in_pairs():
    import torch

    cfg = config((8, 8, 4), (6.0, 6.0, 2.0), 1600.0)  # unit spacing, 256 nodes: one block
    new = torch.zeros((5, 256), dtype=torch.float64)
    old = new.clone()
    old[0, 0] = 1.0
    for w in range(1, 8):
        old[0, 32 * w] = old[0, 32 * w + 1] = 2.0 ** -27  # 2^-53 a warp: half an ulp of the first warp's sum
    out = torch.zeros(6, dtype=torch.float64, device="cuda")
    metrics(cfg, old.cuda(), new.cuda(), torch.zeros(256, dtype=torch.uint8, device="cuda"), out)
    norm, exact = float(out[0]), np.sqrt(np.longdouble(1) + 7 * np.longdouble(2) ** -53)
    assert abs(np.longdouble(norm) - exact) <= np.longdouble(2) ** -52
    assert math.isfinite(norm) and float(out[1]) == 0.0
