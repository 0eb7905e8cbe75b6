"""Smoothed boxes in the plan's own layout against the general route: the window on numpy's layout, the plain
inverse and a multiply.  The same expressions in the same order, so the same bits."""
import ctypes as C

import pytest

from conftest import module

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 48, 64, 96, 128, 160, 256, 512])
def test_smoothing_keeps_the_bits_of_the_general_route(n):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    eng, lib = module("engine"), module("_lib").load()
    radii = (0.4, 2.0, n / 3.0)
    g = torch.Generator("cuda").manual_seed(n)
    delta = torch.randn((n, n, n), generator=g, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    with eng.ExcursionSetPlan(n, float(n), max_radii=1) as plan:
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        got = torch.empty((len(radii), n, n, n), device="cuda")
        plan.forward(delta)
        assert lib.es_smooth(plan.handle, (C.c_float * len(radii))(*radii), len(radii), p(got), stream) == 0
        X = plan.fft_r2c(delta)
        Y = torch.empty_like(X)
        for j, R in enumerate(radii):
            assert lib.ic_shape(n, C.c_float(float(n)), p(X), -1, 0, C.c_float(R), 0, p(Y), stream) == 0
            assert torch.equal(got[j], plan.fft_c2r(Y) * (1.0 / float(n) ** 3))
        # a bad call is refused before any launch
        assert lib.es_smooth(plan.handle, None, 1, p(got), stream) != 0
