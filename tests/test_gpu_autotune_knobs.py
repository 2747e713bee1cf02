"""A calibration tries the knobs that the batch's solver reads."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("large", [False, True])
def test_ctas_per_sm_only_where_it_is_read(cuda_ok, tmp_path, large):
    """The grid-wide solver reads it; 68,121 rows do not fit on chip."""
    from lapy_gb300 import TriaMesh, autotune, meshes

    ms = meshes.deformed_icospheres([3, 3], [1, 2])
    if large:
        grid = meshes.square_grid(260)
        ms.append(TriaMesh(grid.v * 10, grid.t))
    _, report = autotune.calibrate(ms, k=4, sample=3, cache=autotune.TuneCache(tmp_path / "tune.json"))
    tried = {c["ctas_per_sm"] for c, _ in report}
    assert (len(tried) > 1) == large
    # every other knob is tried in both
    for key, values in autotune.CANDIDATES.items():
        if key != "ctas_per_sm":
            assert {c[key] for c, _ in report} == set(values)
