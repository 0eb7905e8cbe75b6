"""P(k) thresholds: the integers of the definition, edge by edge, and the edges that are refused."""
import math
import timeit

import numpy as np
import pytest

from conftest import module

sch = module("schedule")


@pytest.mark.parametrize("bad,error", [(math.nan, ValueError), (math.inf, OverflowError), (-math.inf, OverflowError),
                                       (1e200, OverflowError), (-1e200, OverflowError)])
@pytest.mark.parametrize("count", [1, 60])
def test_edges_without_a_square_are_refused(bad, error, count):
    edges = np.linspace(0.1, 2.0, count)
    edges[-1] = bad
    with pytest.raises(error):
        sch.pk_k2_thresholds(64, 96.0, edges)


@pytest.mark.parametrize("n", [16, 128, 1024])
@pytest.mark.parametrize("count", [1, 2, 15, 55, 56, 57, 128])
def test_thresholds_are_those_of_the_definition(n, count):
    rng = np.random.default_rng(n + count)
    L = 1.37 * n
    dk = float(sch.delta_k(L))
    kmax2 = 3 * (n // 2) ** 2
    for edges in (sch.pk_edges(n, L, count), dk * np.sqrt(rng.integers(0, kmax2 + 40, count)),
                  rng.uniform(-2.0 * dk, 3.0 * dk * n, count), np.zeros(count), np.full(count, 1e12)):
        out = sch.pk_k2_thresholds(n, L, edges)
        assert out.dtype == np.int32 and out.shape == (count,)
        for t, e in zip(out.tolist(), np.asarray(edges, dtype=np.float64).tolist()):
            assert -1 <= t <= kmax2
            assert t == -1 or dk * math.sqrt(t) <= e
            assert t == kmax2 or dk * math.sqrt(t + 1) > e


def test_no_edges():
    assert sch.pk_k2_thresholds(32, 50.0, np.zeros(0)).shape == (0,)


def test_one_edge_costs_less_than_a_hundred():
    def time(count):
        edges = sch.pk_edges(64, 96.0, count)
        return min(timeit.repeat(lambda: sch.pk_k2_thresholds(64, 96.0, edges), number=100, repeat=5))

    assert time(1) < 0.5 * time(100)
