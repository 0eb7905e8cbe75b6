"""P(k) binning against the float64 oracle from one bin to the most, for lines shorter than a column's
threads and longer, on every tile shape (counts exact, values to the engine's 1e-4)."""
import numpy as np
import pytest

from conftest import module

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import es_oracle as O  # noqa: E402
from parity_util import PK_RTOL  # noqa: E402

sch = module("schedule")


@pytest.mark.parametrize("n,bins", [(16, 1), (16, 128), (48, 3), (96, 128), (128, 100), (160, 5)])
def test_pk_matches_oracle(n, bins):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    eng, L = module("engine"), 1.3 * n
    rng = np.random.default_rng(n + bins)
    x = (5.0 + rng.standard_normal((n, n, n))).astype(np.float32)
    edges = sch.pk_edges(n, L, bins)
    ave = np.float32(x.mean(dtype=np.float64))
    _, k_ref, ps_ref, cnt = O.power_spectrum(x, ave, L, edges)
    with eng.ExcursionSetPlan(n, L) as p:
        d, a = torch.from_numpy(x).cuda(), torch.full((1,), float(ave), device="cuda")
        for tile in range(3):
            p.set_option(2, tile)                        # ES_OPT_COL_TILE
            for _ in range(2):                           # the group counters are left ready for the next call
                ps, k, c = p.power_spectrum(d, a, edges).cpu().numpy()
                assert np.array_equal(c, cnt)
                nz = cnt > 0
                assert np.allclose(ps[nz], ps_ref[nz], rtol=PK_RTOL) and np.allclose(k[nz], k_ref[nz], rtol=PK_RTOL)
        p.check()
