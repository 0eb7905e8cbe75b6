"""The warp-per-rows R2C pass (tile shape 0 at 512; 256 takes the older form) against the CTA-wide one (shape 1): the same
arithmetic in the same order, so the same bits, with either prologue."""
import pytest

from conftest import module

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

sch = module("schedule")


@pytest.mark.parametrize("n", [256, 512])
def test_same_bits_as_the_cta_wide_form(n):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn((n, n, n), device="cuda", generator=g) + 3.0
    ave, edges = x.double().mean().float().reshape(1), sch.pk_edges(n, 1.5 * n, 20)
    with module("engine").ExcursionSetPlan(n, 1.5 * n, max_radii=1) as p:
        out = []
        for tile in (0, 1):
            p.set_option(3, tile)                        # ES_OPT_ROW_TILE
            out.append((torch.view_as_real(p.fft_r2c(x)),
                        p.power_spectrum(x, ave, edges), p.power_spectrum(x, ave, edges, dimensional=True)))
        assert all(torch.equal(a, b) for a, b in zip(*out))
        p.check()
