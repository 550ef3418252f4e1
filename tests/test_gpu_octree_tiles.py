"""The octree's levels numbered together, at the edges of its tiles and key widths, against the oracle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

FIELDS = ("depth", "morton", "parent", "child_start", "child_count", "point_leaf")


@pytest.fixture(scope="module", autouse=True)
def device():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def cloud(count, kind):
    rng = np.random.default_rng(count)
    pts = rng.random((count, 3))
    if kind == "clumped":  # many equal codes, long runs that cross warps and tiles
        pts = 0.5 + 0.001 * np.floor(4 * pts) / 4
    if kind == "corners":  # cells of the last index on every level, and the first
        pts = np.where(pts < 0.5, 0.0, 1.0)
    return pts


@pytest.mark.parametrize("kind", ("spread", "clumped", "corners"))
@pytest.mark.parametrize("depth", (0, 1, 10, 11, 19))
@pytest.mark.parametrize("count", (1, 31, 33, 1023, 1024, 1025, 2049, 70001))
def test_levels_match_the_oracle(oracle, count, depth, kind):
    import mojo_poissonrecon_b200 as mpr

    pts = cloud(count, kind)
    got, want = mpr.build_octree(pts, depth), oracle.build_octree(pts, depth)
    for k in FIELDS:
        assert np.array_equal(getattr(got, k), getattr(want, k)), k


def test_two_tile_sizes_of_the_sort_agree(oracle):
    import mojo_poissonrecon_b200 as mpr

    pts = cloud((1 << 20) + 777, "spread")  # 2,048-item tiles; up to 2^20 items they hold 1,024
    for count in (len(pts), 1 << 20):
        got, want = mpr.build_octree(pts[:count], 9), oracle.build_octree(pts[:count], 9)
        for k in FIELDS:
            assert np.array_equal(getattr(got, k), getattr(want, k)), k


@pytest.mark.parametrize("bad", (np.nan, np.inf, -np.inf, -1e-300, 1.0 + 2.0 ** -52))
def test_points_outside_are_refused(bad):
    import mojo_poissonrecon_b200 as mpr

    pts = cloud(3000, "spread")
    pts[2049, 1] = bad
    with pytest.raises(ValueError, match="finite and inside"):
        mpr.build_octree(pts, 8)
