"""The smoother's default degree on either side of its rule (CPU)."""

from types import SimpleNamespace

import pytest


@pytest.mark.parametrize("n,degree", [
    ((4, 4, 4), 1), ((64, 64, 64), 1), ((48, 32, 40), 1), ((18, 18, 18), 1),
    ((2, 4, 4), 2), ((5, 7, 9), 2), ((37, 50, 23), 2), ((32, 32, 33), 2), ((39, 39, 39), 2),
    ((40, 39, 39), 1), ((63, 61, 59), 1)])
def test_default_degree(n, degree):
    from hippymfem_b200.sparse import default_smoothing_degree

    ndof = (2 * n[0] + 1) * (2 * n[1] + 1) * (2 * n[2] + 1)
    assert default_smoothing_degree(SimpleNamespace(n=n, ndof=ndof)) == degree
