"""The initial spectrum from tables of any spacing: bit for bit a float32 restatement with a sorted search, and about as
fast as from a log-spaced one."""
import ctypes as C

import numpy as np
import pytest

from conftest import module

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _tables(n, L, count):
    dk = 2 * np.pi / L
    lo, hi = dk / 10, dk * np.sqrt(3.0) * n
    t = np.linspace(0.0, 1.0, count)
    yield "log", lo * (hi / lo) ** t
    yield "linear", lo + (hi - lo) * t
    yield "quadratic", lo + (hi - lo) * t ** 2
    yield "short", lo + (dk * n / 4 - lo) * t                         # ends below the largest |k|
    yield "clustered", np.sort(np.concatenate([[lo], np.full(count - 2, 5 * dk) + 1e-3 * dk * np.arange(count - 2), [hi]]))


def _call(lib, n, L, nre, nim, K, P, out):
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    rc = lib.ic_spectrum(n, C.c_float(L), p(nre), p(nim), p(K), p(P), len(K), p(out),
                         C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0


@pytest.mark.parametrize("count", [2, 3, 513, 3000])
def test_any_table(count):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    lib, n, L = module("_lib").load(), 32, 41.0
    g = torch.Generator(device="cuda").manual_seed(count)
    nre, nim = (torch.randn((n, n, n // 2 + 1), device="cuda", generator=g) for _ in range(2))
    out = torch.empty((n, n, n // 2 + 1), dtype=torch.complex64, device="cuda")
    f = np.float32
    dk, vol = f(2.0 * np.pi / float(f(L))), f(f(f(L) * f(L)) * f(L))
    m = np.fft.fftfreq(n, 1.0 / n)
    k1 = (m.astype(f) * dk) ** 2
    kz = (np.arange(n // 2 + 1).astype(f) * dk) ** 2
    k = np.sqrt((k1[:, None, None] + k1[None, :, None]) + kz[None, None, :])
    for name, table in _tables(n, L, count):
        K = np.unique(table.astype(f)) if count > 3 else table.astype(f)
        P = (1e3 / (1.0 + K.astype(np.float64) ** 2)).astype(f)
        _call(lib, n, L, nre, nim, torch.from_numpy(K).cuda(), torch.from_numpy(P).cuda(), out)
        i = np.clip(np.searchsorted(K, k, side="left"), 1, len(K) - 1)
        with np.errstate(invalid="ignore"):
            ps = P[i - 1] + ((P[i] - P[i - 1]) * (k - K[i - 1])) / (K[i] - K[i - 1])
            a = np.sqrt(ps * vol) * f(0.70710678118654752)
        got = out.cpu().numpy()[:, :, 1:-1]
        assert np.array_equal(got.real, (a * nre.cpu().numpy())[:, :, 1:-1], equal_nan=True), name
        assert np.array_equal(got.imag, (a * nim.cpu().numpy())[:, :, 1:-1], equal_nan=True), name


def test_spacing_costs_little():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    lib, n, L = module("_lib").load(), 128, 150.0
    nre, nim = (torch.randn((n, n, n // 2 + 1), device="cuda") for _ in range(2))
    out = torch.empty((n, n, n // 2 + 1), dtype=torch.complex64, device="cuda")
    ms = {}
    for name, table in _tables(n, L, 4096):
        K = torch.from_numpy(table.astype(np.float32)).cuda()
        P = 1e3 / (1.0 + K ** 2)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        for _ in range(3):
            _call(lib, n, L, nre, nim, K, P, out)
        a.record()
        for _ in range(10):
            _call(lib, n, L, nre, nim, K, P, out)
        b.record()
        torch.cuda.synchronize()
        ms[name] = a.elapsed_time(b)
    assert max(ms.values()) < 10.0 * ms["log"], ms
