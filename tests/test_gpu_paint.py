"""Sphere painting (both ways of the painting kernel) against the float64 oracle, at row lengths whose
words are whole, partial and straddling, for every row-pass layout that writes the centre bitmap."""
import numpy as np
import pytest

from conftest import module

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import es_oracle as O  # noqa: E402
from parity_util import FLAG_TOL, compare_ionized  # noqa: E402

cos = module("cosmology")
sch = module("schedule")
grf = module("grf")

CASES = [
    # (n, L, z, zeta, R_max, ref_compat): dense centres unless noted
    (16, 24.0, 8.0, 30.0, 12.0, False),       # half a word per row, balls wider than half the box
    (48, 72.0, 8.0, 25.0, 12.0, False),       # 1.5 words, rows straddling the 64-voxel flag words
    (48, 72.0, 8.0, 25.0, 20.0, True),        # clipped at the edges
    (96, 144.0, 8.0, 25.0, 60.0, False),      # widths beyond a word
    (64, 96.0, 11.0, 30.0, 10.0, False),      # few centres: one warp per centre
]


@pytest.mark.parametrize("case", CASES, ids=[f"{c[0]}-{i}" for i, c in enumerate(CASES)])
def test_painting_matches_oracle(case):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    eng, at = module("engine"), module("autotune")
    n, L, z, zeta, R_max, compat = case
    d = grf.density_box(n, L, seed=n, z=z)
    st = sch.ionize_setup(n, L, z, zeta=zeta, t_vir_min=1e4, R_max=R_max, cosmo=cos.BASELINE_COSMO, update=1,
                          ref_compat=compat)
    ref = O.conv_bubbles(d, st, tol=FLAG_TOL)
    assert ref["flags"].any()
    with eng.ExcursionSetPlan(n, L) as p:
        for cfg in [(1, 0, t, 0, rr) for t in range(4) for rr in range(2)] + [(0, 0, 0, 0, 0)]:
            at.apply(p, cfg)
            out, _ = p.run(torch.from_numpy(d).cuda(), st, output="ionized")
            compare_ionized(out.cpu().numpy().astype(np.float64), ref, f"{case} {cfg}")
        p.check()
