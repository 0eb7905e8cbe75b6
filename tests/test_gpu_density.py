"""The density box made with its spectrum against the two calls it stands for: the same bits."""
import pytest

from conftest import module

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,hii", [(16, 16), (48, 32), (96, 32), (160, 160), (256, 64), (512, 128)])
def test_density_matches_spectrum_and_inverse(dim, hii):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    with module("initial").InitialConditions(dim, hii, 1.7 * dim) as ic:
        nre, nim = ic.normals(dim)
        H, box = ic._density(nre, nim)
        ref = ic.spectrum(nre, nim)
        assert torch.equal(torch.view_as_real(H), torch.view_as_real(ref))
        assert torch.equal(box, ic._fft.fft_c2r(ref, scale=ic.norm))
