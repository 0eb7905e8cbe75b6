"""Warp-per-columns column passes (sizes 256 and 512): transforms against cuFFT in float64, the filtered
inverse against the other tile shapes, and a wait that runs out."""
import pytest

from conftest import module

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from parity_util import PARTIAL_ATOL  # noqa: E402

cos = module("cosmology")
sch = module("schedule")
grf = module("grf")


@pytest.fixture(scope="module")
def eng():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return module("engine")


@pytest.mark.parametrize("n", [256, 512])
def test_transforms_match_float64(eng, n):
    # 3-D float32 transforms of unit-variance noise: rounding of ~3 log2(n) stages, far below 1e-6 in the 2-norm
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn((n, n, n), device="cuda", generator=g)
    with eng.ExcursionSetPlan(n, 300.0, max_radii=1) as p:
        ref = torch.fft.rfftn(x.double())
        X = p.fft_r2c(x)
        assert ((X - ref).abs().norm() / ref.abs().norm()).item() < 1e-6
        del X
        y = p.fft_c2r(ref.to(torch.complex64))
        assert ((y / n ** 3 - x).norm() / x.norm()).item() < 1e-6
        p.check()


@pytest.mark.parametrize("n,kw", [(256, dict()), (256, dict(filter_type=1)), (256, dict(ref_compat=True)),
                                  (256, dict(filter_type=2)), (512, dict(R_max=4.0))])
def test_filtered_inverse_matches_other_shapes(eng, n, kw):
    L, z = 1.2 * n, 8.5
    g = torch.Generator(device="cuda").manual_seed(5)
    d = torch.randn((n, n, n), device="cuda", generator=g) * 0.4
    st = sch.ionize_setup(n, L, z, zeta=30.0, t_vir_min=1e4, cosmo=cos.BASELINE_COSMO, **{"R_max": 8.0, **kw})
    outs = []
    with eng.ExcursionSetPlan(n, L) as p:
        for tile, overlap in ((0, 0), (0, 1), (1, 0)):
            p.set_option(2, tile)                        # ES_OPT_COL_TILE
            p.set_option(7, overlap)                     # ES_OPT_OVERLAP
            xh, nf = p.run(d, st)
            outs.append((xh.clone(), nf.item()))
        p.check()
    assert 0.01 < outs[0][1] < 0.999
    for xh, nf in outs[1:]:
        assert ((xh - outs[0][0]).abs() > PARTIAL_ATOL).float().mean().item() <= 1e-5
        assert abs(nf - outs[0][1]) <= 1e-6


def test_timed_out_wait_reports_and_plan_recovers(eng):
    _lib = module("_lib")
    n, L, z = 256, 300.0, 8.0
    g = torch.Generator(device="cuda").manual_seed(2)
    d = torch.randn((n, n, n), device="cuda", generator=g) * 0.3
    st = sch.ionize_setup(n, L, z, zeta=30.0, t_vir_min=1e4, R_max=2.0, cosmo=cos.BASELINE_COSMO)
    with eng.ExcursionSetPlan(n, L) as p:
        good = p.run(d, st)[0].clone()
        p.check()
        p.set_option(_lib.OPT_WAIT_LOG2, 12)
        p.set_option(_lib.OPT_DEBUG_STALL, _lib.STALL_COL_Z_INV)
        p.run(d, st)
        with pytest.raises(_lib.EngineError) as ei:
            p.check()
        assert ei.value.code == _lib.ES_E_DEVICE
        p.set_option(_lib.OPT_DEBUG_STALL, 0)
        p.set_option(_lib.OPT_WAIT_LOG2, 0)
        again = p.run(d, st)[0]
        p.check()
        assert torch.equal(again, good)
