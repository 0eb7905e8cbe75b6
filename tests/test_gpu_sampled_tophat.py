"""Sampled fields with the k-space top hat (filter 1, a cut of the spectrum at an integer |k|^2): the folded route against
the window, the full inverse and the nearest cells."""
import pytest

from conftest import module

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,hii", [(64, 64), (64, 32), (96, 32), (128, 16), (256, 128)])
def test_folding_matches_the_general_route(dim, hii):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    with module("initial").InitialConditions(dim, hii, 1.7 * dim) as ic:
        H = ic.spectrum(*ic.normals(dim + hii))
        for c, box in zip((-1, 0, 1, 2), ic._sampled(H, -1, 4, ic.norm, 1, False)):
            ref = ic.subsample(ic._fft.fft_c2r(ic.shaped(H, c, 1, False)), ic.norm)
            # the same modes with the same weights: transforms good to ~3e-7 either way
            assert float((box.double() - ref.double()).norm() / ref.double().norm()) < 2e-6, c
