"""NaN, infinite and out-of-range masses in the mass move: the kernel that takes a whole HII cell per thread
(aligned input) against the cell-by-cell one (unaligned input), bit for bit."""
import numpy as np
import pytest

from conftest import module

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,sw", [(32, 16), (64, 16), (64, 8)])
@pytest.mark.parametrize("first,second", [(np.nan, None), (np.inf, None), (-np.inf, None), (1e6, np.nan), (np.inf, np.nan),
                                          (np.nan, np.nan)])
@pytest.mark.parametrize("place", ["first", "middle", "last"])
def test_same_bits_as_cell_by_cell(dim, sw, first, second, place):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(dim + sw)
    P = dim // sw
    delta = (rng.standard_normal((dim,) * 3) * 1.5).astype(np.float32)
    # cells of one HII cell in the order a thread reads them; `second` comes right after `first`
    cells = [(a, b, c) for a in range(P) for b in range(P) for c in range(P)]
    at = {"first": 0, "middle": len(cells) // 2, "last": len(cells) - (1 if second is None else 2)}[place]
    for h in ((0, 0, 0), (1, sw // 2, sw - 1)):
        for q, value in ((at, first), (at + 1, second)):
            if value is not None:
                delta[tuple(h[a] * P + cells[q][a] for a in range(3))] = value
    v = [torch.from_numpy((rng.standard_normal((sw,) * 3) * 40.0).astype(np.float32)).cuda() for _ in range(3)]
    out = []
    with module("perturb").PerturbPlan(dim, sw) as plan:
        for offset in (0, 1):
            d = torch.empty(dim ** 3 + offset, dtype=torch.float32, device="cuda")[offset:].view(dim, dim, dim)
            d.copy_(torch.from_numpy(delta))
            out.append(plan.move_mass(d, *v, init_growth=0.1, disp_scale=0.01, mass_factor=float(P ** 3)))
    assert torch.equal(out[0].view(torch.int32), out[1].view(torch.int32))


@pytest.mark.parametrize("dim,sw", [(256, 128), (256, 64), (512, 64)])
def test_large_masses_are_no_slower_than_cell_by_cell(dim, sw):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    g = torch.Generator(device="cuda").manual_seed(dim + sw)
    buf = torch.randn(dim ** 3 + 1, device="cuda", generator=g)
    v = [torch.randn((sw,) * 3, device="cuda", generator=g) * 0.5 for _ in range(3)]
    ms = []
    with module("perturb").PerturbPlan(dim, sw) as plan:
        for offset in (0, 1):                            # whole HII cells, cell by cell
            d = buf[offset:offset + dim ** 3].view(dim, dim, dim)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            for q in range(14):
                if q == 4:
                    a.record()
                plan.move_mass(d, *v, init_growth=1e3, disp_scale=1.0 / sw, mass_factor=1.0)
            b.record()
            torch.cuda.synchronize()
            ms.append(a.elapsed_time(b))
    assert ms[0] <= 1.1 * ms[1], ms
