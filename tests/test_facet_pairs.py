"""The facet grid's antipodal symmetry, on which the matrix-free kernels rest:
for every number of rows a problem may have, each facet normal's negative is a
facet normal too (to rounding, far closer than any other facet)."""
import numpy as np
import pytest


@pytest.mark.parametrize("nrows", [1, 2, 3, 5, 8, 13, 21, 34, 47, 64])
def test_every_facet_has_an_antipode(oracle_lib, nrows):
    o = oracle_lib.Oracle.geometry(1, 1, nrows, 1.05, 1.0, 0.95)
    n = o.array("nor").reshape(-1, 3)[: 8 * nrows * nrows]
    o.close()
    assert np.all(n[:, 2] != 0)
    key = lambda x: x[np.lexsort(np.round(x, 9).T)]  # noqa: E731
    assert np.abs(key(n) - key(-n)).max() <= 1e-12
    assert int((n[:, 2] > 0).sum()) == 4 * nrows * nrows
