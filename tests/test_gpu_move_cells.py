"""The mass move where a thread takes a whole HII cell: bit for bit the CPU restatement, at every ratio that
has a kernel, with masses and displacements that leave the fast way, and on unaligned input."""
import numpy as np
import pytest

from conftest import module

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import pf_oracle as PO  # noqa: E402

cos = module("cosmology")


@pytest.mark.parametrize("dim,sw,cells,amp", [(32, 16, 1.0, 1.5), (64, 16, 2.5, 1.5), (128, 16, 0.2, 1.5), (64, 8, 3.0, 60.0),
                                              (96, 24, 0.0, 1.5), (64, 16, 900.0, 3000.0), (80, 40, 700.0, 1e5)])
@pytest.mark.parametrize("offset", [0, 1])
def test_move_is_bit_exact(dim, sw, cells, amp, offset):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    pt = module("perturb")
    rng = np.random.default_rng(dim + sw)
    g0 = np.float32(cos.growth_factor(8.0, cos.PLANCK13))
    ds = np.float32(0.01)
    delta = (rng.standard_normal((dim,) * 3) * amp).astype(np.float32)
    v = [(rng.standard_normal((sw,) * 3) * (cells / sw / float(ds))).astype(np.float32) for _ in range(3)]
    pf = np.float32(dim) / np.float32(sw)
    mf = np.float32(pf ** 3.0)
    ref = PO.move_mass(delta, *v, g0, ds, pf, mf)
    buf = torch.empty(dim ** 3 + offset, dtype=torch.float32, device="cuda")
    d = buf[offset:].view(dim, dim, dim)                 # offset 1: contiguous, 4-byte aligned only
    d.copy_(torch.from_numpy(delta))
    with pt.PerturbPlan(dim, sw) as plan:
        vs = [torch.from_numpy(x).cuda() for x in v]
        kw = dict(init_growth=float(g0), disp_scale=float(ds), mass_factor=float(mf))
        got = plan.move_mass(d, *vs, **kw).cpu().numpy()
        again = plan.move_mass(d, *vs, **kw).cpu().numpy()
    assert np.array_equal(got, ref)
    assert np.array_equal(got, again)
