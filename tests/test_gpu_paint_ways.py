"""Sphere painting by either way (dilation, ball by ball) against a float64 convolution of the centres with the ball,
on both sides of the line between them, up to 512^3, with balls of one cell to more rows than the kernel's table."""
import dataclasses
import math

import pytest

from conftest import module

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

sch = module("schedule")
cos = module("cosmology")

STD = 0.4                                        # of the filtered field; the threshold is nsigma of them, below delta_c


def _reach(n, R, periodic, device):
    """Indicator of the ball |d| < R (cells) around the origin on the periodic grid (twice n if it is not)."""
    m = torch.arange(n if periodic else 2 * n, device=device)
    m = torch.minimum(m, len(m) - m)
    r2 = (m ** 2)[:, None, None] + (m ** 2)[None, :, None] + (m ** 2)[None, None, :]
    return (r2.double() < R * R).double()


def _painted(centres, R, periodic):
    n = centres.shape[0]
    ball = _reach(n, R, periodic, centres.device)
    x = torch.zeros_like(ball)
    x[:n, :n, :n] = centres
    hits = torch.fft.irfftn(torch.fft.rfftn(x) * torch.fft.rfftn(ball), s=ball.shape)
    return hits[:n, :n, :n] > 0.5, float(ball.sum())


# R: the filter's radius in cells, and the ball's; with ref_compat the ball's is R in Mpc (`scale` to the cell)
@pytest.mark.parametrize("n,R,nsigma,compat,scale", [
    (16, 5.3, 1.5, False, 1.5), (48, 6.3, 2.9, False, 1.5), (48, 6.3, 1.0, True, 1.5), (48, 2.1, 2.4, True, 30.0),
    (96, 9.2, 1.4, True, 1.5), (96, 9.2, 2.0, False, 1.5), (96, 60.0, 0.1, False, 1.5), (128, 1.2, 1.8, False, 1.5),
    (128, 30.0, 3.0, False, 1.5), (160, 4.3, 2.4, False, 1.5), (160, 4.3, 1.9, True, 1.5), (256, 0.9, 2.6, False, 1.5),
    (256, 0.9, 1.0, False, 1.5), (256, 7.4, 3.3, False, 1.5), (256, 7.4, 1.0, False, 1.5), (512, 3.2, 2.5, False, 1.5),
    (512, 3.2, 1.0, False, 1.5), (512, 12.3, 3.6, False, 1.5), (512, 28.0, 3.5, False, 1.5)])
def test_painting_matches_the_convolution(n, R, nsigma, compat, scale):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    L = scale * n
    g = torch.Generator(device="cuda").manual_seed(int(n + 10 * R + 100 * nsigma))
    cells = max(1.0, 4.0 / 3.0 * math.pi * R ** 3)
    d = torch.randn((n, n, n), device="cuda", generator=g) * (STD * math.sqrt(cells))
    st = sch.ionize_setup(n, L, 8.0, zeta=30.0, t_vir_min=1e4, R_max=10.0 * scale, cosmo=cos.BASELINE_COSMO, ref_compat=compat)
    t, delta_c = nsigma * STD, 1.686
    # centres: delta_R >= t at the first radius; the second ionises nothing that is no centre
    first = dataclasses.replace(st.steps[0], R=R * scale, denom=1.0)
    st = dataclasses.replace(st, steps=[first, dataclasses.replace(first, denom=1e-3)], normalize_mean=False,
                             delta_c=delta_c, zeta=1.0 / math.erfc(delta_c - t), growth_scale=1.0)
    with module("engine").ExcursionSetPlan(n, L, max_radii=2) as p:
        centres = (p.run(d, st, output="ionized")[0] == 1.0).clone()
        got = p.run(d, dataclasses.replace(st, update=1), output="ionized")[0] == 1.0
        p.check()
    count = int(centres.sum())
    assert 0 < count < n ** 3
    want, volume = _painted(centres.double(), R * scale if compat else R, not compat)
    # the first run carries its flags in delta_R's last bit, which can move a cell by one unit in the last place
    # (2^-23 at most) across the threshold: the density of cells there, at most 0.4 / STD, times half of that
    flips = n ** 3 * (0.4 / STD) * 2.0 ** -23 * 0.5
    assert int((got != want).sum()) <= math.floor(flips + 6.0 * math.sqrt(flips)) * volume
