"""Compile-time pass kernels at the large sizes with a factor 3: N = 384 in FP64, and N = 768, whose FP32 y/z plan alone has
the stages 8, 4, 24 and whose FP64 tiles alone are 4 columns wide by default.  Against the run-time plans
(MLQ_PASS_KERNELS=reg) and against transforms of the whole box in 64 bits."""
import numpy as np
import pytest

import maxlq_b200 as mlq

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.abs(np.subtract(a, b)).max() / max(np.abs(b).max(), 1e-300))


# tolerances of test_gpu_sizes.py
@pytest.mark.parametrize("n,precision,iters", [(384, "fp64", 2), (768, "mixed", 0)])
def test_match_run_time_plans(n, precision, iters, monkeypatch):
    monkeypatch.setenv("MLQ_AUTOTUNE", "0")
    u, out = None, {}
    for kernels in ("reg", "compile-time"):
        monkeypatch.setenv("MLQ_PASS_KERNELS", kernels)
        with mlq.MaxLq(n, 4.0, 1.0, precision=precision, optim_tol=1e-14) as c:
            assert (c.kernel_config()["pass_kernels"] == "compile-time") == (kernels != "reg")
            if u is None:
                u = c.seed_field(1, 2.0, n / 16)
            out[kernels] = c.calc_global_dLqdt_inclParts(u), c.calc_global_Lq_norm(u), c.GradL2ForLq(u)
            if iters:
                c.state_load(u)
                _, st, rec = c.state_iterate(iters)
                assert st == 0
                out[kernels] += ([r["J1"] for r in rec],)
    a, b = out["reg"], out["compile-time"]
    assert rel(b[0], a[0]) < (1e-12 if precision == "fp64" else 2e-6)
    assert b[1] == pytest.approx(a[1], rel=1e-12 if precision == "fp64" else 2e-6)
    assert rel(b[2], a[2]) < (1e-10 if precision == "fp64" else 1e-3)
    if iters:
        assert b[3] == pytest.approx(a[3], rel=1e-10)


def test_dealias_and_gradient_at_768_in_fp64():
    import torch

    n = 768
    f = torch.randn((n, n, n), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    k = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device="cuda")
    kx = torch.arange(n // 2 + 1, dtype=torch.float64, device="cuda")

    def error(got, want):
        got = torch.from_numpy(got).cuda()
        e = float((got - want).abs().max() / want.abs().max())
        del got, want
        torch.cuda.empty_cache()
        return e

    host = f.cpu().numpy()
    h = torch.fft.rfftn(f)
    del f
    with mlq.MaxLq(n, 4.0, 1.0) as c:
        assert c.kernel_config()["pass_kernels"] == "compile-time"
        for order in (2.0, 1.5):
            cut = mlq.band_cut(n, order)
            keep = (k.abs() <= cut)[:, None, None] & (k.abs() <= cut)[None, :, None] & (kx <= cut)
            assert error(c.dealias_scalar(host, order), torch.fft.irfftn(h * keep, s=(n, n, n))) < 1e-12
            del keep
        g = c.gradient(host)
        odd = k.clone()
        odd[n // 2] = 0.0  # a first derivative has no Nyquist mode
        oddx = kx.clone()
        oddx[-1] = 0.0
        for i, w in enumerate((oddx[None, None, :], odd[None, :, None], odd[:, None, None])):
            assert error(g[i], torch.fft.irfftn(h * (2j * np.pi * w), s=(n, n, n))) < 1e-12
    del h
    torch.cuda.empty_cache()
