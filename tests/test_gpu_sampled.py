"""Sampled fields by folding the spectrum against the general route (window, full inverse, nearest cells)
and float64, over sampling ratios with and without a middle alias, one included."""
import numpy as np
import pytest

from conftest import module

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import ic_oracle as IO  # noqa: E402


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize("dim,hii", [(64, 64), (64, 16), (96, 32), (160, 32), (128, 64), (512, 256)])
@pytest.mark.parametrize("filt,compat", [(0, False), (0, True), (2, False)])
def test_folding_matches_the_general_route(dim, hii, filt, compat):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ini = module("initial")
    with ini.InitialConditions(dim, hii, 1.7 * dim) as ic:
        assert ic._small is not None
        H = ic.spectrum(*ic.normals(dim + hii))
        got = ic._sampled(H, -1, 4, ic.norm, filt, compat)
        for c, box in zip((-1, 0, 1, 2), got):
            ref = ic.subsample(ic._fft.fft_c2r(ic.shaped(H, c, filt, compat)), ic.norm)
            # two float32 routes: windows good to ~1e-6 of the field, transforms to ~3e-7
            assert _rel(box, ref) < 4e-6, (c, _rel(box, ref))
        v = ic.velocities(H, ic.norm, filt, compat)
        assert all(torch.equal(v[k], b) for k, b in zip(("vx", "vy", "vz"), got[1:]))


def test_ratio_that_is_not_whole_takes_the_general_route():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ini = module("initial")
    n, sw, L = 64, 48, 80.0
    with ini.InitialConditions(n, sw, L) as ic:
        assert ic._small is None
        out = ic.generate(seed=1)
        H, R = out["spectrum"].cpu().numpy(), ic.smooth_R
    ref = IO.boxes(H, L, sw, R, 0, False)
    for name in ("deltax", "smoothed", "vx", "vy", "vz"):
        assert _rel(out[name].cpu(), torch.from_numpy(np.asarray(ref[name]))) < 2e-5, name


def test_transform_plans_refuse_everything_else():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    eng, _lib = module("engine"), module("_lib")
    x = torch.randn((32,) * 3, device="cuda")
    with eng.FftPlan(32, 50.0) as p:
        assert _rel(p.fft_c2r(p.fft_r2c(x), scale=1.0 / 32 ** 3), x) < 1e-6
        with pytest.raises(_lib.EngineError):
            p.forward(x)
        with pytest.raises(_lib.EngineError):
            p.delta_T(x, x, 1.0)
        with pytest.raises(_lib.EngineError):
            p.power_spectrum(x, torch.ones(1, device="cuda"), [1.0, 2.0])
        p.check()
    with pytest.raises(_lib.EngineError):
        eng.FftPlan(100, 50.0)
