"""nsf_step_metrics_noalloc over grid sizes around its block and stride edges, against plain torch in 64 bits.

Norms are sums of squares in another order, the dt limit holds a few reciprocals and square roots: both agree with
the 64-bit reference within 1e-12."""
import ctypes

import pytest

import nsfsi

SIZES = [(3, 3, 3), (4, 8, 8), (3, 5, 17), (8, 8, 4), (9, 7, 37), (64, 64, 37), (61, 83, 95), (5, 400, 401), (400, 401, 3)]


@pytest.mark.gpu
@pytest.mark.parametrize("types", [False, True], ids=["faces", "types"])
@pytest.mark.parametrize("n", SIZES, ids=["%dx%dx%d" % n for n in SIZES])
def test_matches_torch(n, types):
    import torch

    cfg = nsfsi.config_load(nsfsi.case_path("tgv256"))
    cfg.NI, cfg.NJ, cfg.NK = n
    g = torch.Generator(device="cuda").manual_seed(sum(n))
    N = n[0] * n[1] * n[2]
    new = 0.03 * torch.randn((5, N), dtype=torch.float64, device="cuda", generator=g)
    old = new + 1e-3 * torch.randn((5, N), dtype=torch.float64, device="cuda", generator=g)
    inside = torch.zeros(n, dtype=torch.bool, device="cuda")
    if types:
        t = torch.randint(0, 5, (N,), device="cuda", generator=g).to(torch.uint8)
        inside = t == 0
    else:
        t = None
        inside[1:-1, 1:-1, 1:-1] = True
        inside = inside.reshape(-1)
    out = torch.full((6,), -1.0, dtype=torch.float64, device="cuda")
    st = nsfsi.lib().nsf_step_metrics_noalloc(ctypes.byref(cfg), old.data_ptr(), new.data_ptr(),
                                              t.data_ptr() if types else None, out.data_ptr(),
                                              torch.cuda.current_stream().cuda_stream)
    assert st == 0
    d = [L / (m - 2) for L, m in zip((cfg.lx, cfg.ly, cfg.lz), n)]
    norms = torch.sqrt(d[0] * d[1] * d[2] * torch.where(inside, (old - new) ** 2, 0.0).sum(1))
    r = 1 + new[0]
    v = new[1:4] / r
    p = (cfg.gamma - 1) * (new[4] - 0.5 * r * (v * v).sum(0))
    T = (cfg.gamma * p - new[0]) / r
    sc = 1 + cfg.sutherlands_c2 / cfg.t0
    mu = (1 + T) ** 1.5 * sc / (cfg.re * (T + sc))
    c = torch.sqrt((1 + cfg.gamma * p) / r)
    conv = abs(cfg.conv_stability_limit) / sum((c + v[a].abs()).max() / d[a] for a in range(3))
    nu = (mu / r).max() * max(4 / 3, cfg.gamma / cfg.pr)
    visc = abs(cfg.visc_stability_limit) / (nu * sum(1 / h ** 2 for h in d))
    ref = torch.cat([norms, torch.stack([torch.minimum(conv, visc)])])
    assert torch.all((out - ref).abs() <= 1e-12 * ref.abs()), (out, ref)
