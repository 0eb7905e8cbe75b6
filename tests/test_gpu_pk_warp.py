"""P(k) by the warp-per-columns z pass (256^3, 512^3; the default tile shape) against the CTA-wide one (the
other shapes): counts equal, sums of the same float32 terms in another order (each term within 1 ulp of the
other's, partial sums in float32: 1e-5 is 80 ulp)."""
import numpy as np
import pytest

from conftest import module

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

sch = module("schedule")


@pytest.mark.parametrize("n,bins", [(256, 1), (256, 20), (256, 128), (512, 2), (512, 100)])
@pytest.mark.parametrize("dimensional", [False, True])
def test_warp_form_matches_the_cta_wide_form(n, bins, dimensional):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    eng, L = module("engine"), 1.3 * n
    g = torch.Generator("cuda").manual_seed(n + bins)
    x = 5.0 + torch.randn((n, n, n), generator=g, device="cuda")
    ave = x.double().mean().float().reshape(1)
    edges = sch.pk_edges(n, L, bins)
    with eng.ExcursionSetPlan(n, L, max_radii=1) as p:
        got = [p.power_spectrum(x, ave, edges, dimensional=dimensional).cpu().numpy().astype(np.float64) for _ in range(2)]
        p.set_option(2, 1)                               # ES_OPT_COL_TILE
        ref = p.power_spectrum(x, ave, edges, dimensional=dimensional).cpu().numpy().astype(np.float64)
        p.check()
    assert np.array_equal(got[0], got[1])                # deterministic, counters left ready
    assert np.array_equal(got[0][2], ref[2])
    assert np.allclose(got[0], ref, rtol=1e-5, atol=0)
