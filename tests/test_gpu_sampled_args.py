"""Sampled fields: calls whose inputs or outputs lie in the small plan's own spectra are refused before any launch."""
import ctypes as C

import pytest

from conftest import module

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_overlapping_arguments_are_refused():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    eng, _lib = module("engine"), module("_lib")
    n, h, L = 32, 16, 50.0
    lib = _lib.load()
    x = torch.randn((n, n, n), device="cuda")
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def call(big, half, small, out):
        return lib.ic_sampled_fields(big.handle, half, small.handle, 0, 2.0, 0, -1, 1, 1.0, (C.c_void_p * 1)(out), stream)

    with eng.FftPlan(n, L) as big, eng.FftPlan(h, L, spectra=4) as small, eng.FftPlan(n, L, spectra=4) as same_size:
        big.forward_spectrum(x)
        out = torch.empty((n, n, n), device="cuda")
        base = small._ws.data_ptr()
        assert call(big, None, small, out.data_ptr()) == 0
        # one plan as both; half at the start, the middle and across the end of the spectra; an output there
        assert call(same_size, None, same_size, out.data_ptr()) == _lib.ES_E_ARG
        for at in (base, base + small.workspace_bytes() // 2, base - 1024):
            assert call(big, C.c_void_p(at), small, out.data_ptr()) == _lib.ES_E_ARG
        for at in (base, base + small.workspace_bytes() // 2):
            assert call(big, None, small, at) == _lib.ES_E_ARG
        ref = eng.sampled_fields(big, None, small, -1, 1, 2.0, 1.0)[0]
        assert torch.equal(out[:].flatten()[: h ** 3], ref.flatten())
        big.check()
        small.check()
