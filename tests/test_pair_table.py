"""The host's table of antipodal facet pairs, which the matrix-free calls need:
for every number of rows a problem may have it holds each facet once, and a pair's
normals cancel."""
import numpy as np
import pytest

from conftest import golden_path


@pytest.mark.parametrize("nrows", range(1, 65))
def test_pair_table(native, tmp_path, nrows):
    lines = open(golden_path("tiny")).read().splitlines(True)
    lines[4], lines[5] = "1 1\n", "%d\n" % nrows
    path = tmp_path / "period_search_in"
    path.write_text("".join(lines))
    h = native.PeriodSearch(str(path), host_only=True)
    f = h.array("pairs").astype(int)
    n = h.array("nor").reshape(-1, 3)
    h.close()
    assert n.shape[0] == 8 * nrows * nrows
    assert np.array_equal(np.sort(f), np.arange(n.shape[0]))
    f = f.reshape(-1, 2)
    assert np.all(n[f[:, 0], 2] > 0)
    assert np.abs(n[f[:, 0]] + n[f[:, 1]]).max() <= 1e-12
